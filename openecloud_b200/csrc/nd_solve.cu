// nd_solve.cu -- the direct FP64 Poisson solve on nested-dissection fronts.
//
// Reference: poissonSolver.pyx:85 (phi[inside] = lu.solve(q[inside])).  The
// setup (nd_setup.py) eliminates the unknowns front by front and keeps, per
// front of s pivots and b boundary unknowns, X = A11^-1 and G = A21 X.  With
// v the front's right-hand side (q on the pivots plus the updates u of the
// fronts below),
//
//   forward  (bottom to top):  y = X v1,   u = v2 - G v1
//   backward (top to bottom):  x1 = y - G^T x2
//
// The triangular factors' chain of dependent rows is gone: what is left between
// two levels is one grid barrier, and inside a level every front is a dense
// block times a vector.  The bytes of the blocks bound large grids, the
// barriers and the dependent loads around them small ones.  Measured (warm,
// per solve) against the level-scheduled factors with their dense tail:
// 33 x 25 rectangle 6.2 against 270 us, 128^2 circle 20.5 against 146 us, 512^2
// ellipse 111 against 1400 us, 1024^2 ellipse 312 us against 9.1 ms; the blocks
// take 4, 44, 264 and 1049 MB (the 1024^2 tail inverses alone took 4.3 GB).
// Tried and dropped: only 128-thread CTAs, eight to an SM (45 us at 128^2: every
// CTA gathers a long front's inputs anew); fetching the next pass's first blocks
// into L1 or L2 ahead of the barrier (1024^2 330 -> 344 us); fetching a warp's or a
// group's next block into L2 behind the current one (with E, 1024^2 330 -> 328 us, but
// 512^2 119 -> 121 and 1000 x 700 274 -> 277 us).
#include <stdint.h>

#include <cooperative_groups.h>

#include <algorithm>

#include "oec_common.cuh"

namespace oec {
namespace {

constexpr int kNdThreads = 512, kNdWarps = kNdThreads / 32;
constexpr int kNdPerSm = 2;       // resident CTAs per SM
constexpr int kNdQuarter = 128;   // threads of a group that is a quarter of a CTA
constexpr int kNdWarpVec = OEC_ND_WARP_IN;

struct NdArgs {
    oec_nd_t nd;
    const double *q;
    double *phi, *y, *u;
    bool staged;  // q shares memory with phi: the root's part of q lies in y (k_nd_stage)
};

__device__ __forceinline__ double2 load_mat(const double *p) { return __ldg(reinterpret_cast<const double2 *>(p)); }

__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

__device__ __forceinline__ oec_nd_tile_t load_tile(const oec_nd_tile_t *p) {
    union {
        int4 v[2];
        oec_nd_tile_t t;
    } x;
    x.v[0] = __ldg(reinterpret_cast<const int4 *>(p));
    x.v[1] = __ldg(reinterpret_cast<const int4 *>(p) + 1);
    return x.t;
}

// Sum of the (at most four) child updates that go to one entry.  The order is
// the setup's, so the sum does not depend on the launch.
__device__ __forceinline__ double child_sum(const int4 k, const double *u) {
    const double a = k.x >= 0 ? __ldcg(u + k.x) : 0.0, b = k.y >= 0 ? __ldcg(u + k.y) : 0.0;
    const double c = k.z >= 0 ? __ldcg(u + k.z) : 0.0, d = k.w >= 0 ? __ldcg(u + k.w) : 0.0;
    return ((a + b) + c) + d;
}

// Partial products of 2 outputs with the inputs i0, i0 + step, ... < n; M at the
// outputs' place in input 0.  The block is stored input by input, so the lanes of
// a warp read neighbouring outputs of one input and no product needs a
// reduction inside a row.
template <int U>  // loads in flight per lane
__device__ __forceinline__ double2 partial(const double *__restrict__ M, int ld, int i0, int step, int n,
                                           const double *vec) {
    double2 a = make_double2(0.0, 0.0);
    const double *p = M + (int64_t)i0 * ld;
    const int64_t d = (int64_t)step * ld;
    int i = i0;
    for (; i + (U - 1) * step < n; i += U * step, p += U * d) {
        double2 m[U];
#pragma unroll
        for (int k = 0; k < U; ++k) m[k] = load_mat(p + k * d);
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const double v = vec[i + k * step];
            a.x += m[k].x * v;
            a.y += m[k].y * v;
        }
    }
    // the last ones, loaded together
    double2 m[U - 1];
#pragma unroll
    for (int k = 0; k < U - 1; ++k) m[k] = i + k * step < n ? load_mat(p + k * d) : make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < U - 1; ++k)
        if (i + k * step < n) {
            const double v = vec[i + k * step];
            a.x += m[k].x * v;
            a.y += m[k].y * v;
        }
    return a;
}

// The inputs of a tile into v: forward the pivots' right-hand side with the
// children's updates, backward phi on the boundary.
template <bool FWD>
__device__ __forceinline__ void gather(const NdArgs &a, const oec_nd_tile_t &t, bool children, bool root, int first,
                                       int step, double *v) {
    const bool staged = FWD && root && a.staged;
    const int4 *src = reinterpret_cast<const int4 *>(a.nd.piv_src) + t.piv0;
    const int32_t *node = FWD ? a.nd.piv_node + t.piv0 : a.nd.bnd_node + t.bnd0;
#pragma unroll 2
    for (int i = first; i < t.n_in; i += step) {
        const int k = __ldg(node + i);
        if (FWD) {
            double x = staged ? __ldcg(a.y + t.piv0 + i) : __ldg(a.q + k);
            if (children) x += child_sum(__ldg(src + i), a.u);
            v[i] = x;
        } else {
            v[i] = __ldcg(a.phi + k);
        }
    }
}

// What a product at output o is combined with, read before the product is
// there: y of the backward direction, the children's updates to a boundary entry
// of the forward one.
template <bool FWD>
__device__ __forceinline__ double out_base(const NdArgs &a, const oec_nd_tile_t &t, int o, bool children) {
    if (o >= t.o0 + t.n_out) return 0.0;
    if (!FWD) return __ldcg(a.y + t.piv0 + o);
    if (!children || o < t.n_in) return 0.0;
    return child_sum(__ldg(reinterpret_cast<const int4 *>(a.nd.bnd_src) + t.bnd0 + o - t.n_in), a.u);
}

template <bool FWD>
__device__ __forceinline__ void put_out(const NdArgs &a, const oec_nd_tile_t &t, int o, double base, double val,
                                        bool root) {
    if (o >= t.o0 + t.n_out) return;
    if (!FWD)
        a.phi[__ldg(a.nd.piv_node + t.piv0 + o)] = base - val;
    else if (o >= t.n_in)
        a.u[t.bnd0 + o - t.n_in] = base - val;
    else if (root)
        a.phi[__ldg(a.nd.piv_node + t.piv0 + o)] = val;
    else
        a.y[t.piv0 + o] = val;
}

// A barrier of a group of GT threads: the CTA's, or one of its quarters'.
template <int GT>
__device__ __forceinline__ void group_sync() {
    if (GT == kNdThreads)
        __syncthreads();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / GT), "n"(GT) : "memory");
}

// The tiles of one direction of one level by groups of GT threads.  A tile is
// `width` outputs of a front; its inputs are split over the lanes that the
// outputs leave (summed in a fixed order).  What a tile costs is its chain of
// dependent loads (tile, indices, values, block): quarter CTAs have four times
// as many chains under way, whole ones gather long inputs faster.
template <bool FWD, int GT>
__device__ __forceinline__ void run_tiles(const NdArgs &a, const oec_nd_tile_t *__restrict__ tiles, int n_tiles,
                                          int width, bool children, bool root, double *vec, double *red) {
    constexpr int kGroups = kNdThreads / GT, kWarps = GT / 32;
    const int lane = threadIdx.x & 31, group = threadIdx.x / GT, tid = threadIdx.x % GT;
    const int L = width >> 1, parts = GT / L;  // L lanes across the outputs, two each
    const int part = tid / L, col = tid & (L - 1);
    const int slots = L < 32 ? kWarps : parts, slot = L < 32 ? tid >> 5 : part;
    vec += group * (a.nd.max_front / kGroups);
    red += group * 2 * GT;
    // with several tiles to a CTA: neighbouring ones, so that the front's inputs
    // are gathered once (quarters, with short inputs, lost by the uneven tiles that
    // lie together: 1024^2 312 -> 328 us)
    const int gid = blockIdx.x + group * gridDim.x, groups = gridDim.x * kGroups;
    int k = gid, end = n_tiles, step = groups, front = -1;
    if (GT == kNdThreads && n_tiles > groups) {
        k = (int)((int64_t)n_tiles * gid / groups);
        end = (int)((int64_t)n_tiles * (gid + 1) / groups);
        step = 1;
    }
    for (; k < end; k += step) {
        const oec_nd_tile_t t = load_tile(tiles + k);
        if (tid == 0 && k + step < end) prefetch_l1(tiles + k + step);
        if (GT != kNdThreads || t.piv0 != front) gather<FWD>(a, t, children, root, tid, GT, vec);
        front = t.piv0;
        const int oa = t.o0 + tid;  // this thread's output
        const bool has = tid < width;
        const double base = has ? out_base<FWD>(a, t, oa, children) : 0.0;
        group_sync<GT>();
        double2 s = make_double2(0.0, 0.0);
        if (t.o0 + 2 * col < t.ld) s = partial<4>(a.nd.mat + t.mat + 2 * col, t.ld, part, parts, t.n_in, vec);
        for (int m = 16; m >= L; m >>= 1) {
            s.x += __shfl_xor_sync(kFullMask, s.x, m);
            s.y += __shfl_xor_sync(kFullMask, s.y, m);
        }
        if (L >= 32 || lane < L) *reinterpret_cast<double2 *>(red + slot * width + 2 * col) = s;
        group_sync<GT>();
        if (has) {
            double v = 0.0;
            for (int m = 0; m < slots; ++m) v += red[m * width + tid];
            put_out<FWD>(a, t, oa, base, v, root);
        }
        // red is written again only behind the next tile's first barrier, vec behind this one's last read
    }
}

// The tiles by single warps: whole fronts of at most kNdWarpVec inputs.
template <bool FWD>
__device__ __forceinline__ void run_fronts(const NdArgs &a, const oec_nd_tile_t *__restrict__ tiles, int n_tiles,
                                           bool children, bool root, double *vec) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *v = vec + warp * kNdWarpVec;
    const int step = gridDim.x * kNdWarps;
    for (int k = blockIdx.x * kNdWarps + warp; k < n_tiles; k += step) {
        const oec_nd_tile_t t = load_tile(tiles + k);
        if (k + step < n_tiles) prefetch_l1(tiles + k + step);
        __syncwarp();
        gather<FWD>(a, t, children, root, lane, 32, v);
        __syncwarp();
        const int L = t.n_out > 32 ? 32 : t.n_out > 16 ? 16 : 8;  // lanes across the outputs, two each
        const int R = 32 / L, sub = lane / L, ol = 2 * (lane & (L - 1));
        for (int o0 = 0; o0 < t.n_out; o0 += 2 * L) {
            const int o = o0 + ol;
            const double b0 = sub == 0 ? out_base<FWD>(a, t, o, children) : 0.0;
            const double b1 = sub == 0 ? out_base<FWD>(a, t, o + 1, children) : 0.0;
            double2 s = make_double2(0.0, 0.0);
            if (o < t.ld) s = partial<6>(a.nd.mat + t.mat + o, t.ld, sub, R, t.n_in, v);
            for (int m = 16; m >= L; m >>= 1) {
                s.x += __shfl_xor_sync(kFullMask, s.x, m);
                s.y += __shfl_xor_sync(kFullMask, s.y, m);
            }
            if (sub == 0) {
                put_out<FWD>(a, t, o, b0, s.x, root);
                put_out<FWD>(a, t, o + 1, b1, s.y, root);
            }
        }
    }
}

template <bool FWD>
__device__ __forceinline__ void run_level(const NdArgs &a, const oec_nd_pass_t &p, bool children, bool root,
                                          double *vec, double *red) {
    if (p.group == kNdThreads)
        run_tiles<FWD, kNdThreads>(a, a.nd.tiles + p.tile, p.tiles, p.width, children, root, vec, red);
    else if (p.group == kNdQuarter)
        run_tiles<FWD, kNdQuarter>(a, a.nd.tiles + p.tile, p.tiles, p.width, children, root, vec, red);
    else
        run_fronts<FWD>(a, a.nd.tiles + p.tile, p.tiles, children, root, vec);
}

__global__ void __launch_bounds__(kNdThreads, kNdPerSm) k_nd_solve(const __grid_constant__ NdArgs a) {
    extern __shared__ __align__(16) double vec[];
    __shared__ __align__(16) double red[2 * kNdThreads];  // (split of the inputs) x width
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    for (int k = a.nd.n_levels - 1; k >= 0; --k) {
        const oec_nd_level_t &l = a.nd.level[k];
        run_level<true>(a, l.fwd, l.has_children != 0, k == 0, vec, red);
        if (a.nd.n_levels > 1) grid.sync();
    }
    // phi is written from the root on, when q has been read (it may be the same memory)
    for (int i = blockIdx.x * kNdThreads + threadIdx.x; i < a.nd.n_outside; i += gridDim.x * kNdThreads)
        a.phi[a.nd.outside[i]] = 0.0;
    for (int k = 1; k < a.nd.n_levels; ++k) {
        run_level<false>(a, a.nd.level[k].bwd, false, false, vec, red);
        if (k + 1 < a.nd.n_levels) grid.sync();
    }
}

// q on the pivots into y, before a solve whose q and phi share memory: the tiles of
// the root read q while others of them write phi.  (The fronts below overwrite their
// part of y, and have read q before anything of phi is written.)
__global__ void k_nd_stage(int n, const int32_t *__restrict__ piv_node, const double *q, double *__restrict__ y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = q[piv_node[i]];
}

// A pass fits the kernel: its tiles exist, its group is one of the three and its
// width a power of two that the group's lanes can take.
bool pass_ok(const oec_nd_pass_t &p, int n_tiles) {
    if (p.tile < 0 || p.tiles < 0 || (int64_t)p.tile + p.tiles > n_tiles) return false;
    if (p.group == 32) return true;
    return (p.group == kNdThreads || p.group == kNdQuarter) && p.width >= 8 && (p.width & (p.width - 1)) == 0 &&
           p.width <= (p.group == kNdThreads ? 256 : 128);
}

int64_t pass_ctas(const oec_nd_pass_t &p) {
    const int groups = kNdThreads / p.group;
    return (p.tiles + groups - 1) / groups;
}

}  // namespace

int nd_solve(const oec_nd_t *nd, const double *q, double *phi, double *work, cudaStream_t s) {
    if (nd->n <= 0 || nd->n_levels < 1 || nd->n_levels > OEC_ND_MAX_LEVELS || nd->max_front < kNdWarps * kNdWarpVec ||
        nd->max_front > OEC_ND_MAX_FRONT || nd->max_front % 4 || nd->n_bnd < 0 || nd->n_outside < 0 || nd->ctas < 0 || !nd->tiles || !nd->piv_node ||
        !nd->mat || (nd->n_levels > 1 && (!nd->piv_src || !nd->bnd_node || !nd->bnd_src)) ||
        (nd->n_outside > 0 && !nd->outside))
        return OEC_ERR_INVALID;
    int64_t need = 1;
    for (int k = 0; k < nd->n_levels; ++k) {
        const oec_nd_level_t &l = nd->level[k];
        if (!pass_ok(l.fwd, nd->n_tiles) || !pass_ok(l.bwd, nd->n_tiles)) return OEC_ERR_INVALID;
        need = std::max(need, std::max(pass_ctas(l.fwd), pass_ctas(l.bwd)));
    }
    const size_t smem = sizeof(double) * (size_t)nd->max_front;
    static std::atomic<int> attr[kMaxDevices];
    const int ok = per_device_cached(attr, [] {
        return cudaFuncSetAttribute(k_nd_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(sizeof(double) * OEC_ND_MAX_FRONT)) == cudaSuccess
                   ? 1
                   : 0;
    });
    if (!ok) return OEC_ERR_CUDA;
    const uintptr_t q0 = reinterpret_cast<uintptr_t>(q), p0 = reinterpret_cast<uintptr_t>(phi);
    const uintptr_t bytes = sizeof(double) * (uintptr_t)nd->n_nodes;
    NdArgs a{*nd, q, phi, work, work + nd->n, q0 < p0 + bytes && p0 < q0 + bytes};
    if (a.staged) {
        k_nd_stage<<<persistent_grid((nd->n + 255) / 256, 4), 256, 0, s>>>(nd->n, nd->piv_node, q, a.y);
        OEC_LAUNCH_CHECK();
    }
    if (nd->n_levels == 1) {  // no barrier: an ordinary launch
        k_nd_solve<<<(unsigned)need, kNdThreads, smem, s>>>(a);
        OEC_LAUNCH_CHECK();
        return OEC_OK;
    }
    // every CTA resident at once: the barrier between levels is the grid's
    int per_sm = 0;
    OEC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_nd_solve, kNdThreads, smem));
    int64_t most = (int64_t)sm_count() * std::min(per_sm, kNdPerSm);
    if (nd->ctas > 0) most = std::min<int64_t>(most, nd->ctas);
    const int grid = (int)std::min(need, most);
    if (grid < 1) return OEC_ERR_CUDA;
    void *args[] = {&a};
    OEC_CUDA_TRY(cudaLaunchCooperativeKernel((void *)k_nd_solve, dim3(grid), dim3(kNdThreads), args, smem, s));
    return OEC_OK;
}

}  // namespace oec
