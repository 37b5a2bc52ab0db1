"""The direct solve on nested-dissection fronts, against a sparse solve of the
assembled matrix.

Tolerance: both sides are backward stable up to small factors, so they differ
by at most about eps times the condition number, which for the 5-point
operator on nx x ny cells is below nx^2 + ny^2 (times the squared aspect ratio
of a cell); 16 eps of that."""
import numpy as np
import pytest
import scipy.sparse as spsp
import scipy.sparse.linalg as spla

# nx, ny, lx, ly, boundType: a single unknown row, one front, several levels, odd and elongated grids
GRIDS = [(3, 3, 0.04, 0.04, 0), (5, 4, 0.04, 0.03, 0), (33, 25, 0.04, 0.03, 0), (24, 200, 0.02, 0.1, 0),
         (64, 48, 0.04, 0.04, 1), (131, 97, 0.06, 0.05, 1), (200, 151, 0.09, 0.036, 1)]


def _case(p):
    from openecloud_b200.grid import Grid
    from openecloud_b200.lu_setup import assemble
    g = Grid(*p)
    a, _, _, inside = assemble(g)
    q = np.zeros(g.getNpExt())
    q[inside] = np.random.default_rng(p[0]).normal(size=inside.size) * 1e-9
    r = g.getDx() / g.getDy()
    tol = 16 * 2.3e-16 * (p[0] ** 2 + p[1] ** 2) * max(r, 1 / r) ** 2
    phi = np.zeros(q.size)
    phi[inside] = spla.spsolve(a.tocsc(), q[inside])
    return g, a, inside, q, phi, tol


@pytest.mark.parametrize("levels", ["model", "many"])
@pytest.mark.parametrize("p", GRIDS)
def test_fronts_on_the_host(p, levels, monkeypatch):
    """The setup's fronts, replayed with numpy, solve the matrix; with a phase
    that costs nothing the tree is cut at (nearly) every depth."""
    from openecloud_b200 import nd_setup
    if levels == "many":
        for k in ("PHASE_US", "TILE_US", "GATHER_US", "BLOCK_US", "WARP_US"):
            monkeypatch.setattr(nd_setup, k, 0.0)
    g, a, inside, q, phi, tol = _case(p)
    h = nd_setup.nd_host_arrays(a, inside, g.getNxExt(), g.getNpExt())
    x = nd_setup.nd_solve_host(h, q)
    assert np.linalg.norm(x - phi) <= tol * np.linalg.norm(phi)
    assert h["piv_node"].size == np.unique(h["piv_node"]).size == inside.size
    if levels == "many" and inside.size > 1000:
        assert h["n_levels"] >= 5


@pytest.mark.parametrize("p", [(96, 96, 0.04, 0.04, 1), (200, 131, 0.06, 0.05, 1), (150, 120, 0.09, 0.036, 0)])
def test_fronts_keep_the_accuracy_of_row_sums(p):
    """Charges of one sign (nothing cancels in the solve itself): the error, against
    a solve refined with residuals in long double, stays at 64 eps whatever the
    condition number, as couplings and row sums determine the inverse's entries
    to a few eps per level of the elimination."""
    from openecloud_b200 import nd_setup
    g, a, inside, q, *_ = _case(p)
    q = np.abs(q)
    csr, lu = a.tocsr(), spla.splu(a.tocsc())
    x = lu.solve(q[inside]).astype(np.longdouble)
    for _ in range(4):
        r = q[inside] - np.add.reduceat(csr.data.astype(np.longdouble) * x[csr.indices], csr.indptr[:-1])
        x += lu.solve(r.astype(np.float64))
    h = nd_setup.nd_host_arrays(a, inside, g.getNxExt(), g.getNpExt())
    d = nd_setup.nd_solve_host(h, q)[inside] - x
    assert np.sqrt((d * d).sum()) <= 64 * 2.3e-16 * np.sqrt((x * x).sum())


def test_other_matrices_are_left_to_the_factors():
    """A matrix that couples other than grid neighbours, is not symmetric or
    has a singular front gets no fronts."""
    from openecloud_b200 import nd_setup
    g, a, inside, *_ = _case(GRIDS[2])
    args = (inside, g.getNxExt(), g.getNpExt())
    far = a.tolil()
    far[0, 40] = far[40, 0] = -1e-12
    assert nd_setup.nd_host_arrays(far.tocsc(), *args) is None
    skew = a.tolil()
    skew[0, 1] = 2 * a[0, 1]
    assert nd_setup.nd_host_arrays(skew.tocsc(), *args) is None
    assert nd_setup.nd_host_arrays(spsp.csc_matrix((inside.size, inside.size)), *args) is None


@pytest.mark.gpu
@pytest.mark.parametrize("levels", ["model", "many"])
@pytest.mark.parametrize("p", GRIDS + [(402, 301, 0.09, 0.036, 1)])
def test_fronts_on_the_device(gpu, p, levels, monkeypatch):
    """One solve per grid and choice of levels (one front, CTA tiles of every
    width, a warp per front), twice: the same bits, and zero outside."""
    from openecloud_b200 import nd_setup
    from openecloud_b200.poissonSolver import PoissonSolver
    if levels == "many":
        for k in ("PHASE_US", "TILE_US", "GATHER_US", "BLOCK_US", "WARP_US"):
            monkeypatch.setattr(nd_setup, k, 0.0)
    g, a, inside, q, phi, tol = _case(p)
    ps = PoissonSolver(g)
    assert ps._lu_t.nd
    ps.phi.fill_(3.0)
    ps.solve(q)
    x = ps.getPhi()
    assert np.linalg.norm(x - phi) <= tol * np.linalg.norm(phi)
    ps.phi.fill_(-1.0)
    ps.solve(q)
    assert np.array_equal(ps.getPhi(), x)
    assert np.all(np.delete(x, inside) == 0.0)


def test_parts_of_the_device_for_the_solves_of_a_batch():
    from openecloud_b200.batch import solve_ctas
    assert solve_ctas(1000, 1000, 1) == 0
    assert [solve_ctas(1000, 1000, b) for b in (2, 3, 4, 64)] == [148, 98, 74, 74]
    assert solve_ctas(9000, 3000, 4) == 0 and solve_ctas(4000, 3000, 4) == 98 and solve_ctas(10, 3000, 4) == 74


@pytest.mark.gpu
@pytest.mark.parametrize("p", [(64, 48, 0.04, 0.04, 1), (128, 128, 0.04, 0.04, 1), (402, 301, 0.09, 0.036, 1)])
def test_solve_on_a_part_of_the_device(gpu, p):
    """Fewer CTAs (several tiles to each, down to all of them to one) give the
    bits of the whole device."""
    from openecloud_b200.poissonSolver import PoissonSolver
    g, a, inside, q, phi, tol = _case(p)
    ps = PoissonSolver(g)
    ps.solve(q)
    x = ps.getPhi()
    assert np.linalg.norm(x - phi) <= tol * np.linalg.norm(phi)
    s = ps.sibling()
    for ctas in (1, 7, 74, 148, 295, 10000, 0):
        ps.shareSolve(ctas)
        s.phi.fill_(-1.0)
        s.solve(q)
        assert np.array_equal(s.getPhi(), x), ctas


@pytest.mark.gpu
@pytest.mark.parametrize("levels", ["model", "many"])
@pytest.mark.parametrize("p", GRIDS + [(402, 301, 0.09, 0.036, 1)])
def test_solve_over_its_own_charge(gpu, p, levels, monkeypatch):
    """phi in the charge's memory, and shifted against it both ways: the bits of a solve into
    an array of its own."""
    import ctypes
    import torch
    from openecloud_b200 import device as D
    from openecloud_b200 import nd_setup
    from openecloud_b200.poissonSolver import PoissonSolver, _declare
    if levels == "many":
        for k in ("PHASE_US", "TILE_US", "GATHER_US", "BLOCK_US", "WARP_US"):
            monkeypatch.setattr(nd_setup, k, 0.0)
    g, a, inside, q, *_ = _case(p)
    ps = PoissonSolver(g)
    ps.solve(q)
    want = ps.getPhi()
    ps.phi.copy_(torch.as_tensor(q))
    ps.solveDevice(ps.getPhiDevice())
    assert np.array_equal(ps.getPhi(), want)
    n = q.size
    for shift in (-g.getNxExt(), -1, 1, n // 2, n - 1):
        buf = D.zeros(3 * n, torch.float64)
        buf[n:2 * n] = torch.as_tensor(q, device="cuda")
        phi = buf[n + shift:2 * n + shift]
        rc = _declare().oec_lu_solve(ctypes.byref(ps._lu_t), buf[n:].data_ptr(), phi.data_ptr(), ps._work.data_ptr(),
                                     D.stream())
        assert rc == 0 and np.array_equal(phi.cpu().numpy(), want), shift


def test_dissection_without_the_memory_for_it_returns_an_error():
    """No exception crosses the C entry: positions that span two thousand million lines (the
    counts per line take 8 GB) in a process that may not have that, and more unknowns than
    an index has, give a status; the spans at the ends of int32 are told right."""
    import subprocess
    import sys
    code = """
import ctypes, resource
import numpy as np
from openecloud_b200 import _lib, nd_setup
L, p = nd_setup._declare(), lambda a: a.ctypes.data_as(ctypes.c_void_p)
out = np.zeros(4, np.int64)
far = np.array([0, 2 ** 31 - 2, 5, 9], np.int32)
ends = np.array([-2 ** 31, 2 ** 31 - 1, 5, 9], np.int32)
zero = np.zeros(4, np.int32)
resource.setrlimit(resource.RLIMIT_AS, (3 << 30, 3 << 30))
print(L.oec_nd_dissect(4, p(far), p(zero), 3, 1, p(out)), L.oec_nd_dissect(4, p(ends), p(zero), 3, 1, p(out)),
      L.oec_nd_dissect(2 ** 31, p(far), p(zero), 3, 1, p(out)), L.oec_nd_dissect(4, p(zero), p(zero), 3, 1, p(out)))
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]
    assert r.stdout.split() == ["6", "6", "1", "0"]  # OEC_ERR_HOST, OEC_ERR_INVALID, OEC_OK


QUARTERS = [(150, 120, 0.09, 0.036, 0), (192, 192, 0.04, 0.04, 1), (300, 240, 0.044, 0.036, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("p", QUARTERS)
def test_tiles_by_quarters_of_a_cta(gpu, p):
    """Grids whose lowest level goes to groups of 128 threads: the whole device, and parts of
    it that leave several tiles to a group, give the same bits."""
    from openecloud_b200.poissonSolver import PoissonSolver
    g, a, inside, q, phi, tol = _case(p)
    ps = PoissonSolver(g)
    low = ps._nd_t.level[ps._nd_t.n_levels - 1]
    assert low.fwd.group == 128 and low.fwd.tiles > 600
    ps.solve(q)
    x = ps.getPhi()
    assert np.linalg.norm(x - phi) <= tol * np.linalg.norm(phi)
    for ctas in (1, 7, 74, 148):
        ps.shareSolve(ctas)
        ps.phi.fill_(-1.0)
        ps.solve(q)
        assert np.array_equal(ps.getPhi(), x), ctas


@pytest.mark.gpu
@pytest.mark.parametrize("p", [(96, 96, 0.04, 0.04, 1), (200, 131, 0.06, 0.05, 1), (512, 512, 0.09, 0.036, 1)])
def test_device_keeps_the_accuracy_of_row_sums(gpu, p):
    """test_fronts_keep_the_accuracy_of_row_sums with the blocks inverted on the device and
    the solve made there, up to 512^2: the same 64 eps."""
    from openecloud_b200.poissonSolver import PoissonSolver
    g, a, inside, q, *_ = _case(p)
    q = np.abs(q)
    csr, lu = a.tocsr(), spla.splu(a.tocsc())
    x = lu.solve(q[inside]).astype(np.longdouble)
    for _ in range(4):
        r = q[inside] - np.add.reduceat(csr.data.astype(np.longdouble) * x[csr.indices], csr.indptr[:-1])
        x += lu.solve(r.astype(np.float64))
    ps = PoissonSolver(g)
    ps.solve(q)
    d = ps.getPhi()[inside] - x
    assert np.sqrt((d * d).sum()) <= 64 * 2.3e-16 * np.sqrt((x * x).sum())


def test_front_structures_follow_the_header(tmp_path, monkeypatch):
    """The ctypes structures of the fronts, and the numpy records of their tiles, have the
    layout of include/oec.h."""
    import ctypes
    import test_abi_layout
    from openecloud_b200 import nd_setup
    ct = {np.dtype(np.int64): ctypes.c_int64, np.dtype(np.int32): ctypes.c_int32}
    Tile = type("Tile", (ctypes.Structure,), {"_fields_": [(k, ct[nd_setup.TILE[k]]) for k in nd_setup.TILE.names]})
    assert ctypes.sizeof(Tile) == nd_setup.TILE.itemsize
    assert all(getattr(Tile, k).offset == nd_setup.TILE.fields[k][1] for k in nd_setup.TILE.names)
    classes = {"oec_nd_pass_t": nd_setup.NdPass_t, "oec_nd_level_t": nd_setup.NdLevel_t, "oec_nd_t": nd_setup.Nd_t,
               "oec_nd_tile_t": Tile}
    monkeypatch.setattr(test_abi_layout, "_classes", lambda: classes)
    test_abi_layout.test_ctypes_structures_follow_the_header(tmp_path)
