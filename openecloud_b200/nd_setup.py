"""Host-side setup of the nested-dissection Poisson solve, numpy only.

A = S diag(eps0 dsi dst~) S^T over the inside nodes (poissonSolver.pyx:41-58)
is symmetric and couples grid neighbours only.  The unknowns are split by
grid lines into a binary tree (oec_nd_dissect); runs of consecutive depths of
that tree are taken together as the levels of fronts.  A front has s pivots (its
separators, or the whole set at the bottom) and b boundary unknowns (the
neighbours of everything below it, pivots of fronts above).  Eliminating level
by level from the bottom, with F the front's matrix after its children,

    F = [[A11, A21^T], [A21, A22]],   X = A11^-1,   G = A21 X,

the Schur complement A22 - G A21^T goes to the parent.  The device keeps X and G
of every front: forward, a front sums the updates u of its children into v, and
y = X v1, u = v2 - G v1; backward, x1 = y - G^T x2.  Both are products of dense
blocks with a vector, so a solve takes two passes over the levels with no
dependent chain inside one.
"""
import ctypes

import numpy as np

from . import _lib

MAX_LEVELS = 16       # oec_nd_t's array of levels
MAX_FRONT = 6144      # pivots or boundary unknowns of one front (the device keeps them in shared memory)
WARP_IN = 32          # fronts of at most this many inputs may be taken by one warp each
QUARTER_IN = 512      # and of this many by a quarter of a CTA
CTAS = 296            # CTAs of 512 threads that solve together: 2 on each of a B200's 148 SMs
LEAF = 12             # unknowns below which a set is not split


class NdPass_t(ctypes.Structure):
    _fields_ = [(k, ctypes.c_int32) for k in ("tile", "tiles", "width", "group")]


class NdLevel_t(ctypes.Structure):
    _fields_ = [("fwd", NdPass_t), ("bwd", NdPass_t), ("has_children", ctypes.c_int32), ("pad", ctypes.c_int32)]


class Nd_t(ctypes.Structure):
    _P = ctypes.c_void_p
    _fields_ = [("n", ctypes.c_int32), ("n_nodes", ctypes.c_int32), ("n_bnd", ctypes.c_int32),
                ("n_outside", ctypes.c_int32), ("n_levels", ctypes.c_int32), ("max_front", ctypes.c_int32),
                ("n_tiles", ctypes.c_int32), ("ctas", ctypes.c_int32), ("n_mat", ctypes.c_int64),
                ("level", NdLevel_t * MAX_LEVELS), ("tiles", _P), ("piv_node", _P), ("piv_src", _P),
                ("bnd_node", _P), ("bnd_src", _P), ("outside", _P), ("mat", _P)]


TILE = np.dtype([("mat", np.int64)] + [(k, np.int32) for k in ("n_in", "n_out", "ld", "o0", "piv0", "bnd0")])

_lib.OTHER_DECLARED.update({"oec_nd_dissect"})


def _declare():
    L = _lib.lib()
    if not getattr(L, "_nd_declared", False):
        P = ctypes.c_void_p
        L.oec_nd_dissect.restype = ctypes.c_int
        L.oec_nd_dissect.argtypes = [ctypes.c_int64, P, P, ctypes.c_int32, ctypes.c_int32, P]
        L._nd_declared = True
    return L


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def dissect(ix, iy, max_depth, leaf=LEAF):
    """Tree node (root 1, children 2h and 2h + 1) of every unknown."""
    ix, iy = np.ascontiguousarray(ix, np.int32), np.ascontiguousarray(iy, np.int32)
    out = np.empty(ix.size, np.int64)
    rc = _declare().oec_nd_dissect(ix.size, _ptr(ix), _ptr(iy), int(max_depth), int(leaf), _ptr(out))
    if rc:
        raise _lib.OecError("oec_nd_dissect", rc)
    return out


# Model of a solve's time (B200, us) by which the levels and the tiles are
# chosen.  A pass over one level costs a barrier.  A tile costs its chain of
# dependent loads, a round of loads per GT inputs that its group of GT threads
# gathers and one per 4 x GT pairs of outputs of its block; the pass takes as many
# rounds of tiles as the groups need, and at least the time of the bytes that
# the busiest SM reads.
PHASE_US, TILE_US, GATHER_US, BLOCK_US, WARP_US, GBS_SM = 2.0, 2.0, 1.2, 0.8, 3.0, 44.0
SMS = CTAS // 2


def pass_plan(ins, outs):
    """(modelled time, outputs per tile, threads per group) of one direction of
    a level for fronts with `ins` inputs and `outs` outputs."""
    if not outs.size or not outs.any():
        return 0.0, 8, 512
    n_in, n_out = int(ins.max()), int(outs.max())
    best = None
    for group, widths in ((512, (256, 128, 64, 32, 16, 8)), (128, (128, 64, 32, 16, 8))):
        if group == 128 and n_in > QUARTER_IN:
            continue
        for w in widths:
            tiles = int((-(-outs // w)).sum())
            t = -(-tiles * group // (512 * CTAS)) * (TILE_US + GATHER_US * -(-n_in // group) +
                                                     BLOCK_US * -(-n_in * w // (8 * group)))
            t = max(t, -(-tiles // SMS) * n_in * min(w, n_out) * 8e-3 / GBS_SM)
            if best is None or t < best[0]:
                best = (t, w, group)
    if n_in <= WARP_IN:
        lanes = 32 if n_out > 32 else 16 if n_out > 16 else 8
        t = -(-outs.size // (16 * CTAS)) * (WARP_US + BLOCK_US * -(-n_out // (2 * lanes)) * -(-n_in * lanes // 128))
        t = max(t, -(-outs.size // SMS) * n_in * n_out * 8e-3 / GBS_SM)
        if t < best[0]:
            best = (t, 8, 32)
    return best[0] + PHASE_US, best[1], best[2]


def choose_levels(hid, dep, w, v, n):
    """Depths [d_0 = 0, d_1, ...] at which the levels start: level k takes the
    tree's depths d_k .. d_k+1 - 1, the last one everything from there down.
    Minimises the modelled time over all choices.  (w, v) are the coupled
    pairs of unknowns."""
    top = int(dep.max())
    size, bnd = [], []
    for d in range(top + 1):
        anc = np.where(dep >= d, hid >> np.maximum(dep - d, 0), 0)
        size.append(np.bincount(anc[anc > 0] - (1 << d), minlength=1 << d))
        m = (anc[w] > 0) & (anc[v] != anc[w])
        key = np.unique(anc[w][m] * np.int64(n) + v[m])
        bnd.append(np.bincount(key // n - (1 << d), minlength=1 << d))
    end = top + 1
    best = {end: (0.0, [], 0)}
    for d in range(end - 1, -1, -1):
        cand = None
        for d2 in range(d + 1, end + 1):
            if best[d2] is None or best[d2][2] + 1 > MAX_LEVELS:
                continue
            s = size[d] if d2 == end else size[d] - size[d2].reshape(1 << d, -1).sum(1)
            b = bnd[d]
            if s.max() > MAX_FRONT or b.max() > MAX_FRONT:
                continue
            ok = s > 0
            t = pass_plan(s[ok], s[ok] + b[ok])[0] + best[d2][0]
            if d:
                t += pass_plan(b[ok], s[ok])[0]
            if cand is None or t < cand[0]:
                cand = (t, [d] + best[d2][1], best[d2][2] + 1)
        best[d] = cand
    return None if best[0] is None else best[0][1]


def host_inverse(A):
    """Inverses of a stack of symmetric blocks (LinAlgError when one is singular),
    with a Newton step (error of a solve at 200 x 131: 3.6e-15 -> 2.0e-15)."""
    X = np.linalg.inv(A)
    X = X + X @ (np.eye(A.shape[1]) - A @ X)
    return 0.5 * (X + X.transpose(0, 2, 1))


def nd_host_arrays(a, inside, nx, n_nodes, inverse=host_inverse):
    """oec_nd_t's arrays for the CSC matrix `a` over the nodes `inside` of an
    extended grid nx nodes wide, or None when A is not a matrix of this form
    (couplings beyond grid neighbours, not symmetric, a singular front): the
    level-scheduled factors take it, or refuse it.  `inverse` replaces
    host_inverse (the cubic part of the work on large grids)."""
    n = int(a.shape[0])
    inside = np.asarray(inside, np.int64)
    coo = a.tocoo()
    r, c, val = coo.row.astype(np.int64), coo.col.astype(np.int64), coo.data
    dist = np.abs(inside[r] - inside[c])
    if n < 1 or 4 * n > 2 ** 31 - 1 or np.any((dist != 0) & (dist != 1) & (dist != nx)) or \
            not np.all(np.isfinite(val)) or abs(a - a.T).max() > 0.0:
        return None
    off = r != c
    w, v = r[off], c[off]
    ix, iy = inside % nx, inside // nx
    depth = max(0, int(np.ceil(np.log2(max(n, 2) / LEAF))))
    hid = dissect(ix, iy, depth)
    dep = np.frexp(hid.astype(np.float64))[1].astype(np.int64) - 1
    cuts = choose_levels(hid, dep, w, v, n)
    if cuts is None:
        return None
    K = len(cuts)
    level = np.searchsorted(cuts, dep, side="right") - 1
    heap = hid >> (dep - np.asarray(cuts)[level])     # tree node of the unknown's front
    # fronts: level by level from the root, by tree node inside a level
    key = level * (np.int64(1) << 42) + heap
    order = np.lexsort((np.arange(n), key))           # unknowns by (front, node)
    ukey, first, s = np.unique(key[order], return_index=True, return_counts=True)
    front = np.empty(n, np.int64)
    front[order] = np.repeat(np.arange(ukey.size), s)
    pos = np.empty(n, np.int64)
    pos[order] = np.arange(n)                         # place of an unknown among all pivots
    flevel = (ukey >> 42).astype(np.int64)
    fheap = ukey & ((np.int64(1) << 42) - 1)
    nf = ukey.size
    # boundary of every front: the neighbours outside of all unknowns below it
    bkeys = []
    for k in range(K):
        d = cuts[k]
        anc = np.where(dep >= d, hid >> np.maximum(dep - d, 0), 0)
        m = (anc[w] > 0) & (anc[v] != anc[w])
        u = np.unique(anc[w][m] * np.int64(n) + v[m])
        f = np.searchsorted(ukey, k * (np.int64(1) << 42) + u // n)
        bkeys.append(f * np.int64(n) + u % n)
    bkey = np.concatenate(bkeys)                      # (front, unknown), ascending
    bfront, bunk = bkey // n, bkey % n
    b = np.bincount(bfront, minlength=nf)
    bnd0 = np.concatenate([[0], np.cumsum(b)])
    piv0 = np.concatenate([[0], np.cumsum(s)])
    # parent front (a tree node without unknowns of its own has no front: its children go further up)
    parent = np.full(nf, -1, np.int64)
    for k in range(1, K):
        f = np.nonzero(flevel == k)[0]
        for up in range(k - 1, -1, -1):
            f = f[parent[f] < 0]
            cand = up * (np.int64(1) << 42) + (fheap[f] >> (cuts[k] - cuts[up]))
            q = np.minimum(np.searchsorted(ukey, cand), nf - 1)
            hit = ukey[q] == cand
            parent[f[hit]] = q[hit]

    def local(f, unk):
        """Index of unknown `unk` in front f's vector [pivots, boundary]."""
        q = np.searchsorted(bkey, f * np.int64(n) + unk)
        q = np.minimum(q, bkey.size - 1) if bkey.size else q
        return np.where(front[unk] == f, pos[unk] - piv0[f], s[f] + q - bnd0[f])

    # contributions: entry e of the children's updates goes to the parent's entry
    tgt_front = parent[bfront]
    tgt = local(tgt_front, bunk) if bkey.size else np.zeros(0, np.int64)
    is_piv = tgt < s[tgt_front] if bkey.size else np.zeros(0, bool)
    slot_of = np.where(is_piv, piv0[tgt_front] + tgt, n + bnd0[tgt_front] + tgt - s[tgt_front])
    src = np.full((n + bkey.size, 4), -1, np.int32)
    e_order = np.argsort(slot_of, kind="stable")
    so = slot_of[e_order]
    rank = np.arange(so.size) - np.searchsorted(so, so)
    if rank.size and rank.max() > 3:
        return None
    src[so, rank] = e_order
    # the blocks
    ldf, ldb = (s + b + 1) // 2 * 2, (s + 1) // 2 * 2
    mf = np.concatenate([[0], np.cumsum(s * ldf + b * ldb)])
    mat = np.zeros(int(mf[-1]))
    # A as couplings and row sums: a front's matrix gets its diagonal as row sum
    # minus couplings, and a Schur complement's row sums are formed from row sums.
    # All couplings are negative and no row sum is, so nothing cancels (after Grassmann,
    # Taksar and Heyman's elimination; Alfa, Xue and Ye, Math. Comp. 71, 2002).  Error of
    # a solve: 512^2 ellipse 2.2e-13 -> 3e-15, 1024^2 7.8e-13 -> 5e-15
    # (SuperLU 9.2e-14 and 8.6e-12).
    excess = np.zeros(n, np.longdouble)  # exact: the sums themselves cancel
    np.add.at(excess, r, val.astype(np.longdouble))
    excess = excess.astype(np.float64)
    r, c, val = w, v, val[off]
    own = np.where(level[r] >= level[c], front[r], front[c])
    li, lj = local(own, r), local(own, c)
    by_front = np.argsort(own, kind="stable")
    own_ptr = np.searchsorted(own[by_front], np.arange(nf + 1))
    kids = np.argsort(parent, kind="stable")
    kid_ptr = np.searchsorted(parent[kids], np.arange(nf + 1))
    schur, schur_sum = {}, {}

    def eliminate(fs):
        """Fronts fs (of one level, similar size): their blocks into `mat`,
        their Schur complements into `schur`."""
        S, B = int(s[fs].max()), int(b[fs].max())
        T = S + B
        idx, vals = [], []
        rs = np.zeros((fs.size, T))  # row sums; 1 on the padding
        for k, f in enumerate(fs):
            rs[k, :s[f]] = excess[order[piv0[f]:piv0[f] + s[f]]]
            rs[k, s[f]:S] = 1.0
            e = by_front[own_ptr[f]:own_ptr[f + 1]]
            i, j = li[e], lj[e]
            i, j = np.where(i < s[f], i, i - s[f] + S), np.where(j < s[f], j, j - s[f] + S)
            idx.append((k * T + i) * T + j)
            vals.append(val[e])
            for ch in kids[kid_ptr[f]:kid_ptr[f + 1]]:
                t = tgt[bnd0[ch]:bnd0[ch + 1]]
                t = np.where(t < s[f], t, t - s[f] + S)
                idx.append(((k * T + t)[:, None] * T + t).ravel())
                vals.append(schur.pop(int(ch)).ravel())
                rs[k, t] += schur_sum.pop(int(ch))
        F = np.bincount(np.concatenate(idx), weights=np.concatenate(vals), minlength=fs.size * T * T)
        F = F.reshape(fs.size, T, T).astype(np.float64, copy=False)  # (no couplings: whole numbers)
        d = np.arange(T)
        F[:, d, d] = 0.0
        F[:, d, d] = rs - F.sum(2)
        X = inverse(F[:, :S, :S])
        A21 = F[:, S:, :S]
        G = A21 @ X
        C = F[:, S:, S:] - G @ A21.transpose(0, 2, 1) if B else None
        CS = rs[:, S:] - (G @ rs[:, :S, None])[:, :, 0]
        for k, f in enumerate(fs):
            sf, bf, o = int(s[f]), int(b[f]), int(mf[f])
            fw = mat[o:o + sf * ldf[f]].reshape(sf, ldf[f])
            fw[:, :sf] = X[k, :sf, :sf]
            if bf:
                fw[:, sf:sf + bf] = G[k, :bf, :sf].T
                o += sf * int(ldf[f])
                mat[o:o + bf * ldb[f]].reshape(bf, ldb[f])[:, :sf] = G[k, :bf, :sf]
                schur[int(f)] = np.ascontiguousarray(C[k, :bf, :bf])
                schur_sum[int(f)] = CS[k, :bf]

    # one after another: BLAS threads the large fronts by itself
    for k in range(K - 1, -1, -1):
        fs = np.nonzero(flevel == k)[0]
        fs = fs[np.lexsort((b[fs], s[fs]))]
        # chunks of up to ~4 M matrix entries
        chunk = np.cumsum((s[fs] + b[fs]) ** 2) // 4_000_000
        for part in np.split(fs, np.nonzero(np.diff(chunk))[0] + 1):
            try:
                eliminate(part)
            except np.linalg.LinAlgError:
                return None
    out = {"n": n, "n_nodes": int(n_nodes), "n_bnd": int(bkey.size), "n_levels": K, "cuts": list(cuts),
           "level_of_front": flevel, "s": s, "b": b, "piv0": piv0, "bnd0": bnd0, "ldf": ldf, "ldb": ldb,
           "mf": mf[:-1], "mb": mf[:-1] + s * ldf}
    mask = np.ones(int(n_nodes), bool)
    mask[inside] = False
    out["outside"] = np.nonzero(mask)[0].astype(np.int32)
    out["piv_node"] = inside[order].astype(np.int32)
    out["bnd_node"] = inside[bunk].astype(np.int32)
    out["piv_src"], out["bnd_src"] = np.ascontiguousarray(src[:n]), np.ascontiguousarray(src[n:])
    out["mat"] = mat
    tiles, lv = [], []
    count, widest = 0, 16 * WARP_IN
    for k in range(K):
        fs = np.nonzero(flevel == k)[0]
        rec = {"has_children": int(np.any(np.isin(parent, fs)))}
        for tag in ("fwd", "bwd"):
            fwd = tag == "fwd"
            outs = s[fs] + b[fs] if fwd else s[fs] if k else 0 * s[fs]
            ins = s[fs] if fwd else b[fs]
            _, wd, group = pass_plan(ins, outs)
            per = np.where(outs > 0, 1, 0) if group == 32 else -(-outs // wd)
            t = np.zeros(int(per.sum()), TILE)
            f = np.repeat(fs, per)
            t["o0"] = (np.arange(t.size) - np.repeat(np.cumsum(per) - per, per)) * wd
            t["n_in"] = np.repeat(ins, per)
            left = np.repeat(outs, per) - t["o0"]
            t["n_out"] = left if group == 32 else np.minimum(left, wd)
            t["ld"] = (ldf if fwd else ldb)[f]
            t["mat"] = (out["mf"] if fwd else out["mb"])[f] + t["o0"]
            t["piv0"], t["bnd0"] = piv0[f], bnd0[f]
            rec[tag] = {"tile": count, "tiles": t.size, "width": wd, "group": group}
            count += t.size
            if group > 32 and t.size:
                widest = max(widest, int(t["n_in"].max()) * 512 // group)
            tiles.append(t)
        lv.append(rec)
    out["max_front"] = -(-widest // 4) * 4
    out["tiles"] = np.ascontiguousarray(np.concatenate(tiles))
    out["level"] = lv
    return out


def nd_struct(a, ptr):
    """An Nd_t over the arrays of nd_host_arrays; ptr(name) gives the address
    of array `name` (host or device copy)."""
    t = Nd_t()
    for k in ("n", "n_nodes", "n_bnd", "n_levels", "max_front"):
        setattr(t, k, a[k])
    t.n_outside, t.n_tiles, t.n_mat = a["outside"].size, a["tiles"].size, a["mat"].size
    for k, rec in enumerate(a["level"]):
        t.level[k].has_children = rec["has_children"]
        for tag in ("fwd", "bwd"):
            for name, x in rec[tag].items():
                setattr(getattr(t.level[k], tag), name, x)
    for name in ("tiles", "piv_node", "piv_src", "bnd_node", "bnd_src", "outside", "mat"):
        setattr(t, name, ptr(name))
    return t


def nd_solve_host(a, q):
    """The device's solve restated with numpy: phi on all nodes, tile by tile."""
    y, u, phi = np.zeros(a["n"]), np.zeros(a["n_bnd"] + 1), np.zeros(a["n_nodes"])
    mat = a["mat"]

    def gathered(src):
        return u[src].sum(1)  # -1 is the zero behind the last update

    def product(t, v):
        """The tile's outputs (its rows of the block start ld apart)."""
        i = t["mat"] + np.arange(t["n_in"])[:, None] * t["ld"] + np.arange(t["n_out"])
        return v @ mat[i]

    def tiles_of(k, tag):
        p = a["level"][k][tag]
        return a["tiles"][p["tile"]:p["tile"] + p["tiles"]]

    for k in range(a["n_levels"] - 1, -1, -1):
        for t in tiles_of(k, "fwd"):
            s, p0, o0 = int(t["n_in"]), int(t["piv0"]), int(t["o0"])
            o = product(t, q[a["piv_node"][p0:p0 + s]] + gathered(a["piv_src"][p0:p0 + s]))
            m = min(max(s - o0, 0), o.size)  # outputs that are pivots
            y[p0 + o0:p0 + o0 + m] = o[:m]
            e = int(t["bnd0"]) + np.arange(o0 + m - s, o0 + o.size - s)
            u[e] = gathered(a["bnd_src"][e]) - o[m:]
    for k in range(a["n_levels"]):
        if k == 0:
            for t in tiles_of(0, "fwd"):
                i = int(t["piv0"]) + int(t["o0"]) + np.arange(t["n_out"])
                phi[a["piv_node"][i]] = y[i]
            continue
        for t in tiles_of(k, "bwd"):
            i = int(t["piv0"]) + int(t["o0"]) + np.arange(t["n_out"])
            e = int(t["bnd0"]) + np.arange(t["n_in"])
            phi[a["piv_node"][i]] = y[i] - product(t, phi[a["bnd_node"][e]])
    return phi
