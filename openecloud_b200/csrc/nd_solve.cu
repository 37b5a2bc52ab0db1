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
// 33 x 25 rectangle 11.5 against 270 us, 128^2 circle 31 against 146 us, 512^2
// ellipse 168 against 1400 us, 1024^2 ellipse 451 us against 9.1 ms; the blocks
// take 4, 44, 318 and 1144 MB (the 1024^2 tail inverses alone took 4.3 GB).
#include <stdint.h>

#include <cooperative_groups.h>

#include <algorithm>

#include "oec_common.cuh"

namespace oec {
namespace {

constexpr int kNdThreads = 512, kNdWarps = kNdThreads / 32;
constexpr int kNdPerSm = 2;       // resident CTAs per SM
constexpr int kNdWarpVec = 256;   // inputs of a front that one warp takes
constexpr int kNdWidth = 64;      // widest tile of a CTA

struct NdArgs {
    oec_nd_t nd;
    const double *q;
    double *phi, *y, *u;
};

__device__ __forceinline__ double2 load_mat(const double *p) { return __ldg(reinterpret_cast<const double2 *>(p)); }

// Sum of the (at most four) child updates that go to one entry.  The order is
// the setup's, so the sum does not depend on the launch.
__device__ __forceinline__ double child_sum(const int4 *__restrict__ src, int e, const double *u) {
    const int4 k = __ldg(src + e);
    double a = 0.0;
    if (k.x >= 0) a = __ldcg(u + k.x);
    if (k.y >= 0) a += __ldcg(u + k.y);
    if (k.z >= 0) a += __ldcg(u + k.z);
    if (k.w >= 0) a += __ldcg(u + k.w);
    return a;
}

// Partial products of 2 outputs at o with the inputs i0, i0 + step, ... < n.
// The block is stored input by input, so the lanes of a warp read neighbouring
// outputs of one input and no product needs a reduction inside a row.
__device__ __forceinline__ double2 partial(const double *__restrict__ M, int ld, int o, int i0, int step, int n,
                                           const double *vec) {
    double2 a = make_double2(0.0, 0.0);
    const double *p = M + (int64_t)i0 * ld + o;
    const int64_t d = (int64_t)step * ld;
    int i = i0;
    for (; i + 3 * step < n; i += 4 * step, p += 4 * d) {
        const double2 m0 = load_mat(p), m1 = load_mat(p + d), m2 = load_mat(p + 2 * d), m3 = load_mat(p + 3 * d);
        const double v0 = vec[i], v1 = vec[i + step], v2 = vec[i + 2 * step], v3 = vec[i + 3 * step];
        a.x += m0.x * v0;
        a.y += m0.y * v0;
        a.x += m1.x * v1;
        a.y += m1.y * v1;
        a.x += m2.x * v2;
        a.y += m2.y * v2;
        a.x += m3.x * v3;
        a.y += m3.y * v3;
    }
    for (; i < n; i += step, p += d) {
        const double2 m = load_mat(p);
        const double v = vec[i];
        a.x += m.x * v;
        a.y += m.y * v;
    }
    return a;
}

template <bool FWD>
__device__ __forceinline__ double gather_in(const NdArgs &a, const oec_nd_front_t &f, int i, bool children) {
    if (FWD) {
        double v = __ldg(a.q + __ldg(a.nd.piv_node + f.piv0 + i));
        if (children) v += child_sum(reinterpret_cast<const int4 *>(a.nd.piv_src), f.piv0 + i, a.u);
        return v;
    }
    return __ldcg(a.phi + __ldg(a.nd.bnd_node + f.bnd0 + i));
}

template <bool FWD>
__device__ __forceinline__ void put_out(const NdArgs &a, const oec_nd_front_t &f, int o, double val, bool children,
                                        bool root) {
    if (FWD) {
        if (o < f.s) {
            if (root)
                a.phi[__ldg(a.nd.piv_node + f.piv0 + o)] = val;
            else
                a.y[f.piv0 + o] = val;
        } else if (o < f.s + f.b) {
            const int e = f.bnd0 + o - f.s;
            const double v = children ? child_sum(reinterpret_cast<const int4 *>(a.nd.bnd_src), e, a.u) : 0.0;
            a.u[e] = v - val;
        }
    } else if (o < f.s) {
        a.phi[__ldg(a.nd.piv_node + f.piv0 + o)] = __ldcg(a.y + f.piv0 + o) - val;
    }
}

// One direction of one level.  width > 0: a tile is `width` outputs of a front,
// its inputs split over the 16 warps of a CTA (summed in a fixed order);
// width 0: a tile is a whole front, one warp's work.
template <bool FWD>
__device__ __forceinline__ void run_level(const NdArgs &a, const int2 *__restrict__ tiles, int n_tiles, int width,
                                          bool children, bool root, double *vec, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (width == 0) {
        double *v = vec + warp * kNdWarpVec;
        for (int t = blockIdx.x * kNdWarps + warp; t < n_tiles; t += gridDim.x * kNdWarps) {
            const oec_nd_front_t f = a.nd.fronts[__ldg(&tiles[t].x)];
            const int n_in = FWD ? f.s : f.b, n_out = FWD ? f.s + f.b : f.s, ld = FWD ? f.ldf : f.ldb;
            const double *M = a.nd.mat + (FWD ? f.mf : f.mb);
            __syncwarp();
            for (int i = lane; i < n_in; i += 32) v[i] = gather_in<FWD>(a, f, i, children);
            __syncwarp();
            const int L = n_out > 32 ? 32 : n_out > 16 ? 16 : 8;  // lanes across the outputs, two each
            const int R = 32 / L, sub = lane / L, ol = 2 * (lane & (L - 1));
            for (int o0 = 0; o0 < n_out; o0 += 2 * L) {
                const int o = o0 + ol;
                double2 s = make_double2(0.0, 0.0);
                if (o < ld) s = partial(M, ld, o, sub, R, n_in, v);
                for (int k = 16; k >= L; k >>= 1) {
                    s.x += __shfl_xor_sync(kFullMask, s.x, k);
                    s.y += __shfl_xor_sync(kFullMask, s.y, k);
                }
                if (sub == 0) {
                    put_out<FWD>(a, f, o, s.x, children, root);
                    put_out<FWD>(a, f, o + 1, s.y, children, root);
                }
            }
        }
        return;
    }
    const int L = width >> 1, R = 32 / L, sub = lane / L, ol = 2 * (lane & (L - 1));
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int2 tile = __ldg(tiles + t);
        const oec_nd_front_t f = a.nd.fronts[tile.x];
        const int n_in = FWD ? f.s : f.b, ld = FWD ? f.ldf : f.ldb;
        const double *M = a.nd.mat + (FWD ? f.mf : f.mb);
        for (int i = threadIdx.x; i < n_in; i += kNdThreads) vec[i] = gather_in<FWD>(a, f, i, children);
        __syncthreads();
        const int o = tile.y + ol;
        double2 s = make_double2(0.0, 0.0);
        if (o < ld) s = partial(M, ld, o, warp * R + sub, kNdWarps * R, n_in, vec);
        for (int k = 16; k >= L; k >>= 1) {
            s.x += __shfl_xor_sync(kFullMask, s.x, k);
            s.y += __shfl_xor_sync(kFullMask, s.y, k);
        }
        if (sub == 0) *reinterpret_cast<double2 *>(red + warp * kNdWidth + ol) = s;
        __syncthreads();
        if (threadIdx.x < width) {
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < kNdWarps; ++k) v += red[k * kNdWidth + threadIdx.x];
            put_out<FWD>(a, f, tile.y + threadIdx.x, v, children, root);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kNdThreads, kNdPerSm) k_nd_solve(const __grid_constant__ NdArgs a) {
    extern __shared__ double vec[];
    __shared__ __align__(16) double red[kNdWarps * kNdWidth];
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const int2 *tiles = reinterpret_cast<const int2 *>(a.nd.tiles);
    for (int i = blockIdx.x * kNdThreads + threadIdx.x; i < a.nd.n_outside; i += gridDim.x * kNdThreads)
        a.phi[a.nd.outside[i]] = 0.0;
    for (int k = a.nd.n_levels - 1; k >= 0; --k) {
        const oec_nd_level_t &l = a.nd.level[k];
        run_level<true>(a, tiles + l.fwd_tile, l.fwd_tiles, l.fwd_width, l.has_children != 0, k == 0, vec, red);
        if (a.nd.n_levels > 1) grid.sync();
    }
    for (int k = 1; k < a.nd.n_levels; ++k) {
        const oec_nd_level_t &l = a.nd.level[k];
        run_level<false>(a, tiles + l.bwd_tile, l.bwd_tiles, l.bwd_width, false, false, vec, red);
        if (k + 1 < a.nd.n_levels) grid.sync();
    }
}

bool width_ok(int w) { return w == 0 || w == 8 || w == 16 || w == 32 || w == 64; }

}  // namespace

int nd_solve(const oec_nd_t *nd, const double *q, double *phi, double *work, cudaStream_t s) {
    if (nd->n <= 0 || nd->n_levels < 1 || nd->n_levels > OEC_ND_MAX_LEVELS || nd->max_front < 1 ||
        nd->max_front > OEC_ND_MAX_FRONT || nd->n_bnd < 0 || nd->n_outside < 0 || !nd->fronts || !nd->tiles ||
        !nd->piv_node || !nd->mat || (nd->n_levels > 1 && (!nd->piv_src || !nd->bnd_node || !nd->bnd_src)) ||
        (nd->n_outside > 0 && !nd->outside))
        return OEC_ERR_INVALID;
    int64_t need = 1;
    for (int k = 0; k < nd->n_levels; ++k) {
        const oec_nd_level_t &l = nd->level[k];
        if (!width_ok(l.fwd_width) || !width_ok(l.bwd_width) || l.fwd_tile < 0 || l.bwd_tile < 0 ||
            l.fwd_tile + (int64_t)l.fwd_tiles > nd->n_tiles || l.bwd_tile + (int64_t)l.bwd_tiles > nd->n_tiles)
            return OEC_ERR_INVALID;
        need = std::max<int64_t>(need, l.fwd_width ? l.fwd_tiles : (l.fwd_tiles + kNdWarps - 1) / kNdWarps);
        need = std::max<int64_t>(need, l.bwd_width ? l.bwd_tiles : (l.bwd_tiles + kNdWarps - 1) / kNdWarps);
    }
    const size_t smem = sizeof(double) * (size_t)std::max(nd->max_front, kNdWarps * kNdWarpVec);
    static std::atomic<int> attr[kMaxDevices];
    const int ok = per_device_cached(attr, [] {
        return cudaFuncSetAttribute(k_nd_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(sizeof(double) * OEC_ND_MAX_FRONT)) == cudaSuccess
                   ? 1
                   : 0;
    });
    if (!ok) return OEC_ERR_CUDA;
    NdArgs a{*nd, q, phi, work, work + nd->n};
    const int grid = (int)std::min<int64_t>(need, (int64_t)sm_count() * kNdPerSm);
    if (nd->n_levels == 1) {
        k_nd_solve<<<grid, kNdThreads, smem, s>>>(a);
        OEC_LAUNCH_CHECK();
    } else {
        void *args[] = {&a};
        OEC_CUDA_TRY(cudaLaunchCooperativeKernel((void *)k_nd_solve, dim3(grid), dim3(kNdThreads), args, smem, s));
    }
    return OEC_OK;
}

}  // namespace oec
