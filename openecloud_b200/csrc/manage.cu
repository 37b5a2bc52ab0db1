// manage.cu -- macro-particle management on the device: stable radix sort
// (sortByColumn, cell ordering), Russian roulette (globalRandom) and the
// cell-binned phase-space merge (localRandom).
//
// Reference: particles.pyx sortByColumn (:49-50, :431-459),
// particleManagement.pyx globalRandom (:35-67) and localRandom (:74-238).
//  * Sorting is a stable least-significant-digit radix sort of 32-bit keys
//    (8-bit digits): per pass a per-tile digit histogram, one launch that scans
//    each digit's tile counts (a CTA per digit), and a stable scatter in which
//    a tile ranks its elements by warp votes and puts them in order in shared
//    memory before they are written.
//  * globalRandom removes n - target particles chosen uniformly without
//    replacement (each thread throws darts at free slots with atomicOr on the
//    removal bitmask, as the reference redraws until it hits a particle it has
//    not removed), or appends target - n copies of particles drawn with
//    replacement; weights are scaled by n/target in both cases.
//  * localRandom keeps the reference's bookkeeping (weight thresholds, split
//    and merge counts, typical velocity, phase-space metric with
//    lambda = ds / v_typical) but replaces the sequential kd-tree search by
//    binning: the merge candidates (the lightest particles) are ordered along
//    a 5-D Morton curve of (x, y, lambda v) and neighbours in that order are
//    merged when their phase-space distance passes the reference's test.
#include <math.h>
#include <stdint.h>

#include "oec_common.cuh"
#include "specfun.cuh"

namespace oec {
namespace {

constexpr int kSortThreads = 512;                      // threads per sort CTA (16 warps)
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kPerLane = 8;                             // keys per thread (16 with 256 threads: 231 -> 217 us)
constexpr int kTile = kSortThreads * kPerLane;          // keys per sort tile (one CTA): 4096
constexpr int kWarpKeys = 32 * kPerLane;                // a warp's consecutive keys in the tile

__device__ __forceinline__ int blk_scan(int v, int *tot, int *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(kFullMask, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(kFullMask, s, o);
            if (lane >= o) s += y;
        }
        sh[lane] = s;
    }
    __syncthreads();
    int ex = (wid > 0 ? sh[wid - 1] : 0) + x - v;
    if (tot) *tot = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return ex;
}

// ----------------------------------------------------------- radix sort

// Digit counts of one tile (kTile keys): per-warp counters in shared memory
// (fewer same-address conflicts), summed per digit at the end; written
// digit-major, hist[d * ntiles + tile].
__global__ void __launch_bounds__(kSortThreads) k_digit_hist(const uint32_t *__restrict__ keys, const int32_t *n_p,
                                                             int shift, int ntiles, int *__restrict__ hist) {
    __shared__ int h[kSortWarps][256];  // 16 KB
    const int n = *n_p;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int d = threadIdx.x; d < kSortWarps * 256; d += kSortThreads) (&h[0][0])[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kTile + w * kWarpKeys + lane;
#pragma unroll 4
    for (int r = 0; r < kPerLane; ++r) {
        const int64_t i = base + r * 32;
        if (i < n) atomicAdd(&h[w][(keys[i] >> shift) & 255u], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += kSortThreads) {
        int c = 0;
#pragma unroll
        for (int k = 0; k < kSortWarps; ++k) c += h[k][d];
        hist[d * ntiles + blockIdx.x] = c;
    }
}

// Exclusive scan of the tiles' counts of one digit per CTA, in place, and the
// digit's total; the scatter scans the 256 totals itself.
constexpr int kDigitScanT = 512;
__global__ void __launch_bounds__(kDigitScanT) k_digit_scan(int *__restrict__ hist, int ntiles, int *__restrict__ total) {
    __shared__ int sh[32];
    int *row = hist + (int64_t)blockIdx.x * ntiles;
    int carry = 0;
    for (int base = 0; base < ntiles; base += kDigitScanT) {  // same trip count in every thread
        const int i = base + threadIdx.x;
        int tot;
        const int ex = blk_scan(i < ntiles ? row[i] : 0, &tot, sh);
        if (i < ntiles) row[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// The lanes of the warp that hold a key (`mine`) with this lane's digit, by a vote
// per bit.  __match_any_sync takes a step per distinct value, some 30 of them in
// a round of random digits (sort of 2.2e6 by weight with 16 keys a thread 244 -> 231 us).
__device__ __forceinline__ unsigned warp_peers(unsigned mine, int d) {
    unsigned peers = mine;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1;
        const unsigned set = __ballot_sync(kFullMask, bit);
        peers &= bit ? set : ~set;
    }
    return peers;
}

// Stable scatter of one tile (kTile keys) by the digit at `shift`.  Warp w
// owns the tile's keys w*256 .. w*256+255 and walks them in 8 rounds of 32
// consecutive keys (coalesced loads); a key's place among the equal digits
// of its warp is the warp's running count of that digit (shared memory, one
// counter row per warp) plus the lanes below it in the round with the same
// digit (warp_peers).  After the rounds the counts of the lower warps give
// each warp's start inside the tile's run of a digit, and the scanned tile
// histogram the run's start in the output, so the order is (digit, tile,
// warp, round, lane) = stable.  The tile is put in that order in shared memory
// first and written from there, so that a digit's keys leave in one run: written
// from the registers every key was a sector of its own (2.2e6 pairs per pass
// 38 -> 27 us).
__global__ void __launch_bounds__(kSortThreads, 3) k_scatter(const uint32_t *__restrict__ keys,
                                                          const int32_t *__restrict__ vals, const int32_t *n_p,
                                                          int shift, int ntiles, const int *__restrict__ offs,
                                                          const int *__restrict__ total,
                                                          uint32_t *__restrict__ okeys, int32_t *__restrict__ ovals) {
    static_assert(kSortThreads >= 256 && kTile < 1 << 16, "a thread per digit, 16-bit counts");
    __shared__ uint32_t sk[kTile];
    __shared__ int32_t sv[kTile];
    __shared__ int first[256];  // output place of a digit's first key minus its place in the tile
    __shared__ int sh[32];
    __shared__ uint16_t cnt[kSortWarps][256];  // running digit counts, then each warp's start in a digit's run
    const int n = *n_p;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    for (int e = threadIdx.x; e < kSortWarps * 256; e += kSortThreads) (&cnt[0][0])[e] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kTile + w * kWarpKeys + lane;
    uint32_t k[kPerLane];
    int32_t v[kPerLane];
    int dr[kPerLane];  // digit << 16 | rank among the warp's equal digits, -1: no key
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
        const int64_t i = base + r * 32;
        const bool valid = i < n;
        k[r] = valid ? keys[i] : 0u;
        v[r] = valid ? vals[i] : 0;
    }
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
        const bool valid = base + r * 32 < n;
        const int d = (int)((k[r] >> shift) & 255u);
        const unsigned peers = warp_peers(__ballot_sync(kFullMask, valid), d);
        int rank = 0;
        if (valid) rank = cnt[w][d] + __popc(peers & below);
        __syncwarp();
        if (valid && (peers & below) == 0) cnt[w][d] = (uint16_t)(rank + __popc(peers));
        __syncwarp();
        dr[r] = valid ? (d << 16 | rank) : -1;
    }
    __syncthreads();
    // digit d's run in the tile: its start, and in it each warp's start (the
    // counts of the lower warps)
    const int d0 = threadIdx.x;
    const bool digit = d0 < 256;
    int run = 0;
    if (digit) {
#pragma unroll
        for (int q = 0; q < kSortWarps; ++q) run += cnt[q][d0];
    }
    const int out0 = blk_scan(digit ? total[d0] : 0, nullptr, sh);
    int nk;
    int at = blk_scan(run, &nk, sh);
    if (digit) {
        first[d0] = out0 + offs[d0 * ntiles + blockIdx.x] - at;
#pragma unroll
        for (int q = 0; q < kSortWarps; ++q) {
            const int c = cnt[q][d0];
            cnt[q][d0] = (uint16_t)at;
            at += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPerLane; ++r) {
        if (dr[r] < 0) continue;
        const int at_tile = cnt[w][dr[r] >> 16] + (dr[r] & 0xffff);
        sk[at_tile] = k[r];
        sv[at_tile] = v[r];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nk; e += kSortThreads) {
        const uint32_t key = sk[e];
        const int dst = first[(key >> shift) & 255u] + e;
        okeys[dst] = key;
        ovals[dst] = sv[e];
    }
}

// float -> order-preserving uint32
__device__ __forceinline__ uint32_t float_key(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void k_make_keys(oec_particles_t p, int column, uint32_t *__restrict__ keys, int32_t *__restrict__ vals) {
    int n = *p.count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t k;
        switch (column) {
            case 6: k = (uint32_t)p.cell[i]; break;  // cell order
            case 2: k = float_key(p.vx[i]); break;
            case 3: k = float_key(p.vy[i]); break;
            case 4: k = float_key(p.vz[i]); break;
            case 5: k = float_key(p.w[i]); break;
            default: k = (uint32_t)p.cell[i]; break;
        }
        keys[i] = k;
        vals[i] = i;
    }
}

// gather every SoA array through the permutation into `q`
__global__ void k_permute(oec_particles_t p, const int32_t *__restrict__ perm, oec_particles_t q) {
    int n = *p.count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int s = perm[i];
        q.cell[i] = p.cell[s];
        q.ox[i] = p.ox[s];
        q.oy[i] = p.oy[s];
        q.vx[i] = p.vx[s];
        q.vy[i] = p.vy[s];
        q.vz[i] = p.vz[s];
        q.w[i] = p.w[s];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *q.count = n;
}

// The same through rows of 32 bytes: a particle in random order is then one
// sector instead of seven (2.2e6 particles by weight 94 -> 60 us with the
// packing).  An order close to the stored one is faster field by field.
__device__ __forceinline__ void pack_row(const oec_particles_t &p, int i, float4 *__restrict__ rows) {
    rows[2 * (int64_t)i] = make_float4(__int_as_float(p.cell[i]), p.ox[i], p.oy[i], p.vx[i]);
    rows[2 * (int64_t)i + 1] = make_float4(p.vy[i], p.vz[i], p.w[i], 0.f);
}

__global__ void k_pack_rows(oec_particles_t p, float4 *__restrict__ rows) {
    const int n = *p.count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) pack_row(p, i, rows);
}

__global__ void k_permute_rows(const float4 *__restrict__ rows, const int32_t *__restrict__ perm, const int32_t *count,
                               oec_particles_t q) {
    const int n = *count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int64_t s = perm[i];
        const float4 a = __ldg(rows + 2 * s), b = __ldg(rows + 2 * s + 1);
        q.cell[i] = __float_as_int(a.x);
        q.ox[i] = a.y;
        q.oy[i] = a.z;
        q.vx[i] = a.w;
        q.vy[i] = b.x;
        q.vz[i] = b.y;
        q.w[i] = b.z;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *q.count = n;
}

// ------------------------------------------------------- weight search
// _searchSorted (particleManagement.pyx:244-262) on the weight-sorted store:
// 0 when w[0] >= value, else the first index with w[i] > value.  A warp per
// threshold takes 32 probes a round, five rounds of dependent loads for 2^24
// weights where the reference's bisection has 24.
__global__ void k_search_sorted2(const float *__restrict__ w, const int32_t *count, double lo, double hi,
                                 int32_t *out) {
    const int lane = threadIdx.x & 31;
    const double value = threadIdx.x < 32 ? lo : hi;
    const int n = *count;
    int r;
    if (n <= 0) {
        r = 0;
    } else if ((double)w[n - 1] <= value) {
        r = n;
    } else if ((double)w[0] >= value) {
        r = 0;
    } else {
        // w[i0] <= value < w[i2]
        int i0 = 0, i2 = n - 1;
        while (i2 - i0 > 1) {
            const int step = (i2 - i0 + 32) / 33, i = min(i0 + (lane + 1) * step, i2);
            const unsigned above = __ballot_sync(kFullMask, (double)w[i] > value);
            const int below = above ? __ffs(above) - 1 : 32;  // probes before the first one above
            const int a = i0;
            if (below < 32) i2 = min(a + (below + 1) * step, i2);
            i0 = min(a + below * step, i2 - 1);
        }
        r = i0 + 1;
    }
    if (lane == 0) out[threadIdx.x >> 5] = r;
}

// -------------------------------------------------------------- roulette

__global__ void k_scale_w(oec_particles_t p, double factor) {
    int n = *p.count;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        p.w[i] = (float)((double)p.w[i] * factor);
}

__global__ void k_zero_words(uint32_t *m, int nwords) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nwords; i += gridDim.x * blockDim.x) m[i] = 0u;
}

// Mark `k` distinct uniformly chosen indices in [0, n) in `mask`.
__global__ void k_darts(int n, int k, uint32_t *mask, uint2 key, uint32_t call, int max_tries, int *fails) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < k; t += gridDim.x * blockDim.x) {
        bool done = false;
        for (int a = 0; a < max_tries && !done; ++a) {
            uint4 r = sf::philox4x32_10(make_uint4((uint32_t)t, call, (uint32_t)a, 0x7011u), key);
            uint32_t idx = (uint32_t)(((uint64_t)r.x * (uint64_t)n) >> 32);
            uint32_t bit = 1u << (idx & 31);
            uint32_t old = atomicOr(&mask[idx >> 5], bit);
            done = (old & bit) == 0u;
        }
        if (!done) atomicAdd(fails, 1);
    }
}

// mask = ~mask on [0, n)
__global__ void k_invert_valid(uint32_t *mask, int n) {
    int nw = (n + 31) >> 5;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += gridDim.x * blockDim.x) {
        uint32_t valid = (w * 32 + 32 <= n) ? 0xffffffffu : ((1u << (n - w * 32)) - 1u);
        mask[w] = (~mask[w]) & valid;
    }
}

// rows of particles drawn with replacement (clone step of globalRandom)
__global__ void k_clone_rows(oec_particles_t p, int n, int k, uint2 key, uint32_t call, int nx, float inv_nx,
                             double dx, double dy, double lxh, double lyh, double *rows) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < k; t += gridDim.x * blockDim.x) {
        uint4 r = sf::philox4x32_10(make_uint4((uint32_t)t, call, 0u, 0xc10eu), key);
        int s = (int)(((uint64_t)r.x * (uint64_t)n) >> 32);
        int ix, iy;
        split_cell(p.cell[s], nx, inv_nx, ix, iy);
        double *q = rows + 6 * (int64_t)t;
        q[0] = abs_coord(ix, p.ox[s], dx, lxh);
        q[1] = abs_coord(iy, p.oy[s], dy, lyh);
        q[2] = p.vx[s];
        q[3] = p.vy[s];
        q[4] = p.vz[s];
        q[5] = p.w[s];
    }
}

// ------------------------------------------------------------ local merge

// Sums over a store's particles, sum w and sum |v|^2 w^2 (f64): those of one CTA, in
// threads 0 and 1.  Which CTA takes which particles depends on their number alone.
constexpr int kStatThreads = 256, kStatCtas = OEC_WEIGHT_SUMS_CTAS;

// CTAs with particles, of at most `ctas`.
__device__ __forceinline__ int stat_ctas(int n, int ctas) {
    return (int)min((int64_t)ctas, ((int64_t)n + kStatThreads - 1) / kStatThreads);
}

__device__ __forceinline__ double stat_cta(const oec_particles_t &p, int n) {
    __shared__ double sh[2][kStatThreads / 32];
    double sw = 0, sv = 0;
    for (int i = blockIdx.x * kStatThreads + threadIdx.x; i < n; i += stat_ctas(n, gridDim.x) * kStatThreads) {
        double w = p.w[i], vx = p.vx[i], vy = p.vy[i], vz = p.vz[i];
        sw += w;
        sv += (vx * vx + vy * vy + vz * vz) * w * w;
    }
    for (int o = 16; o > 0; o >>= 1) {
        sw += __shfl_xor_sync(kFullMask, sw, o);
        sv += __shfl_xor_sync(kFullMask, sv, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = sw;
        sh[1][threadIdx.x >> 5] = sv;
    }
    __syncthreads();
    double t = 0;
    if (threadIdx.x < 2)
        for (int w = 0; w < kStatThreads / 32; ++w) t += sh[threadIdx.x][w];
    return t;
}

// Added to acc, one atomic per sum and CTA: in the order of arrival.
__global__ void __launch_bounds__(kStatThreads) k_wstats(oec_particles_t p, double *acc) {
    const int n = *p.count;
    if ((int)blockIdx.x >= stat_ctas(n, gridDim.x)) return;
    const double t = stat_cta(p, n);
    if (threadIdx.x < 2) atomicAdd(&acc[threadIdx.x], t);
}

// Left in part (all of sum w, then all of sum |v|^2 w^2) for k_wsums.
__global__ void __launch_bounds__(kStatThreads) k_wparts(oec_particles_t p, double *part) {
    const int n = *p.count;
    if ((int)blockIdx.x >= stat_ctas(n, gridDim.x)) return;
    const double t = stat_cta(p, n);
    if (threadIdx.x < 2) part[threadIdx.x * kStatCtas + blockIdx.x] = t;
}

// The CTAs' sums in a fixed order, a warp per sum.  The thresholds of a merge follow
// from them, so that two runs of one store must agree to the last bit.
__global__ void __launch_bounds__(64) k_wsums(const int32_t *count, int ctas, const double *__restrict__ part,
                                              double *__restrict__ acc) {
    const int parts = stat_ctas(*count, ctas);
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    double t = 0;
    for (int i = lane; i < parts; i += 32) t += part[k * kStatCtas + i];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFullMask, t, o);
    if (lane == 0) acc[k] = t;
}

struct MergeArgs {
    oec_particles_t p;         // weight-sorted store
    int n_cand;                // merge candidates: the lightest n_cand particles
    int n_merge_target;        // merges wanted
    const int32_t *order;      // candidates in Morton order
    const float4 *rows;        // candidates packed as k_pack_rows does, in store order
    uint32_t *qual;            // a bit per pair: it passes the test
    double lam2;               // (ds / v_typical)^2 * lambda_factor^2
    double limit;              // factorDisLimit * ds (compared with the squared distance, as the reference)
    double dx, dy;
    int nx;
    float inv_nx;
    uint2 key;
    uint32_t call;
    int scheme;
    uint32_t *mask;            // removal bits
    int *counters;             // [0] qualifying pairs, [1] merges done
};

// Pair (2k, 2k+1) of the ordered candidates: qualifies when the weighted
// phase-space distance passes the reference's test.  The two lie anywhere in the
// store, so they are read from packed rows, one sector each where the arrays
// would take six, and the outcome is kept for k_pair_merge.  Bound by these
// sectors.
__global__ void k_pair_count(MergeArgs a) {
    const int npairs = a.n_cand / 2, lane = threadIdx.x & 31;
    int q = 0;
    for (int k0 = blockIdx.x * blockDim.x + threadIdx.x - lane; k0 < npairs; k0 += gridDim.x * blockDim.x) {
        const int k = k0 + lane;
        bool near = false;
        if (k < npairs) {
            const int i = __ldg(a.order + 2 * k), j = __ldg(a.order + 2 * k + 1);
            const float4 *ri = a.rows + 2 * (int64_t)i, *rj = a.rows + 2 * (int64_t)j;
            const float4 pi = __ldg(ri), pj = __ldg(rj);
            const float2 vi = __ldg(reinterpret_cast<const float2 *>(ri + 1));
            const float2 vj = __ldg(reinterpret_cast<const float2 *>(rj + 1));
            int ix, iy, jx, jy;
            split_cell(__float_as_int(pi.x), a.nx, a.inv_nx, ix, iy);
            split_cell(__float_as_int(pj.x), a.nx, a.inv_nx, jx, jy);
            const double ddx = ((double)(ix - jx) + ((double)pi.y - pj.y)) * a.dx;
            const double ddy = ((double)(iy - jy) + ((double)pi.z - pj.z)) * a.dy;
            const double dvx = (double)pi.w - pj.w, dvy = (double)vi.x - vj.x, dvz = (double)vi.y - vj.y;
            const double d2 = ddx * ddx + ddy * ddy + a.lam2 * (dvx * dvx + dvy * dvy + dvz * dvz);
            near = d2 < a.limit;
        }
        const unsigned m = __ballot_sync(kFullMask, near);
        if (lane == 0) {
            a.qual[k0 >> 5] = m;
            q += __popc(m);
        }
    }
    if (lane == 0 && q) atomicAdd(&a.counters[0], q);
}

__global__ void k_pair_merge(MergeArgs a) {
    int npairs = a.n_cand / 2;
    int qual = a.counters[0];
    double paccept = qual > 0 ? fmin(1.0, (double)a.n_merge_target / (double)qual) : 0.0;
    int done = 0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < npairs; k += gridDim.x * blockDim.x) {
        if (!(a.qual[k >> 5] >> (k & 31) & 1u)) continue;
        uint4 r = sf::philox4x32_10(make_uint4((uint32_t)k, a.call, 0u, 0x3e59u), a.key);
        double u0 = r.x * (1.0 / 4294967296.0), u1 = r.y * (1.0 / 4294967296.0);
        if (u0 >= paccept) continue;
        const int i = a.order[2 * k], j = a.order[2 * k + 1];
        double wi = a.p.w[i], wj = a.p.w[j];
        int keep = (u1 < wi / (wi + wj)) ? i : j;  // keep with probability proportional to weight
        int drop = keep == i ? j : i;
        if (a.scheme == 1) {
            // scale the kept velocity to conserve kinetic energy (particleManagement.pyx:200-236)
            double wk = a.p.w[keep], wd = a.p.w[drop];
            double vk2 = (double)a.p.vx[keep] * a.p.vx[keep] + (double)a.p.vy[keep] * a.p.vy[keep] +
                         (double)a.p.vz[keep] * a.p.vz[keep];
            double vd2 = (double)a.p.vx[drop] * a.p.vx[drop] + (double)a.p.vy[drop] * a.p.vy[drop] +
                         (double)a.p.vz[drop] * a.p.vz[drop];
            double f = vk2 > 0 ? wk / (wk + wd) + vd2 / vk2 * wd / (wk + wd) : 1.0;
            a.p.vx[keep] = (float)(a.p.vx[keep] * f);
            a.p.vy[keep] = (float)(a.p.vy[keep] * f);
            a.p.vz[keep] = (float)(a.p.vz[keep] * f);
        }
        a.p.w[keep] = (float)(wi + wj);
        atomicOr(&a.mask[drop >> 5], 1u << (drop & 31));
        ++done;
    }
    for (int o = 16; o > 0; o >>= 1) done += __shfl_xor_sync(kFullMask, done, o);
    if ((threadIdx.x & 31) == 0 && done) atomicAdd(&a.counters[1], done);
}

// The candidates' count, the empty bounding box and the zeroed counters.
__global__ void k_merge_begin(int n_cand, int32_t *ncand, uint32_t *bbox, int32_t *counters) {
    const int t = threadIdx.x;
    if (t == 0) *ncand = n_cand;
    if (t < 10) bbox[t] = t < 5 ? 0xffffffffu : 0u;
    if (t < 2) counters[t] = 0;
}

// Weighted phase-space coordinates of the merge metric (localRandom :166-171):
// (x, y, lambda vx, lambda vy, lambda vz), positions relative to the grid corner.
__device__ __forceinline__ void phase5(const oec_particles_t &p, int i, int nx, float inv_nx, double dx, double dy,
                                       double lam, float c[5]) {
    int ix, iy;
    split_cell(p.cell[i], nx, inv_nx, ix, iy);
    c[0] = (float)(((double)ix + p.ox[i]) * dx);
    c[1] = (float)(((double)iy + p.oy[i]) * dy);
    c[2] = (float)(lam * p.vx[i]);
    c[3] = (float)(lam * p.vy[i]);
    c[4] = (float)(lam * p.vz[i]);
}

// Bounding box of the candidates' weighted coordinates (order-preserving
// float keys, atomic min / max): bbox[0..4] minima, bbox[5..9] maxima.
__global__ void k_cand_bbox(oec_particles_t p, int n_cand, int nx, float inv_nx, double dx, double dy, double lam,
                            uint32_t *bbox) {
    __shared__ uint32_t wmn[8][5], wmx[8][5];  // 256 threads
    uint32_t mn[5], mx[5];
    for (int d = 0; d < 5; ++d) {
        mn[d] = 0xffffffffu;
        mx[d] = 0u;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_cand; i += gridDim.x * blockDim.x) {
        float c[5];
        phase5(p, i, nx, inv_nx, dx, dy, lam, c);
        for (int d = 0; d < 5; ++d) {
            uint32_t k = float_key(c[d]);
            mn[d] = min(mn[d], k);
            mx[d] = max(mx[d], k);
        }
    }
    for (int d = 0; d < 5; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = min(mn[d], __shfl_xor_sync(kFullMask, mn[d], o));
            mx[d] = max(mx[d], __shfl_xor_sync(kFullMask, mx[d], o));
        }
        if ((threadIdx.x & 31) == 0) {
            wmn[threadIdx.x >> 5][d] = mn[d];
            wmx[threadIdx.x >> 5][d] = mx[d];
        }
    }
    __syncthreads();
    if (threadIdx.x < 5) {  // one atomic per bound and CTA
        const int d = threadIdx.x;
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            wmn[0][d] = min(wmn[0][d], wmn[w][d]);
            wmx[0][d] = max(wmx[0][d], wmx[w][d]);
        }
        atomicMin(&bbox[d], wmn[0][d]);
        atomicMax(&bbox[5 + d], wmx[0][d]);
    }
}

__device__ __forceinline__ float key_float(uint32_t k) {
    uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// Candidate keys: 5-D Morton order (6 bits per axis, one common scale for all
// axes so that the order follows the isotropic weighted metric): neighbours in
// key order are close in (x, y, lambda v).  The candidates also go into packed
// rows for k_pair_count.
__global__ void k_cand_keys(oec_particles_t p, int n_cand, int nx, float inv_nx, double dx, double dy, double lam,
                            const uint32_t *bbox, uint32_t *keys, int32_t *vals, float4 *rows) {
    float lo[5], span = 0.f;
    for (int d = 0; d < 5; ++d) {
        lo[d] = key_float(bbox[d]);
        span = fmaxf(span, key_float(bbox[5 + d]) - lo[d]);
    }
    float inv = span > 0.f ? 64.0f / span : 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_cand; i += gridDim.x * blockDim.x) {
        float c[5];
        phase5(p, i, nx, inv_nx, dx, dy, lam, c);
        uint32_t q[5];
        for (int d = 0; d < 5; ++d) q[d] = (uint32_t)fminf(fmaxf((c[d] - lo[d]) * inv, 0.f), 63.f);
        uint32_t key = 0;
        for (int b = 5; b >= 0; --b)
            for (int d = 0; d < 5; ++d) key = (key << 1) | ((q[d] >> b) & 1u);
        keys[i] = key;
        vals[i] = i;
        pack_row(p, i, rows);
    }
}

// rows: duplicates at half weight of the heaviest `k` (the last k in weight order)
__global__ void k_split_rows(oec_particles_t p, int n, int k, int nx, float inv_nx, double dx, double dy, double lxh,
                             double lyh, double *rows) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < k; t += gridDim.x * blockDim.x) {
        int s = n - k + t;
        p.w[s] = p.w[s] * 0.5f;
        int ix, iy;
        split_cell(p.cell[s], nx, inv_nx, ix, iy);
        double *q = rows + 6 * (int64_t)t;
        q[0] = abs_coord(ix, p.ox[s], dx, lxh);
        q[1] = abs_coord(iy, p.oy[s], dy, lyh);
        q[2] = p.vx[s];
        q[3] = p.vy[s];
        q[4] = p.vz[s];
        q[5] = p.w[s];
    }
}

}  // namespace
}  // namespace oec

using namespace oec;

static bool vp2(const oec_particles_t *p) {
    return p && p->cell && p->ox && p->oy && p->vx && p->vy && p->vz && p->w && p->count && p->capacity > 0;
}

extern "C" int64_t oec_cell_sort_work_bytes(int64_t capacity) {
    int64_t tiles = (capacity + kTile - 1) / kTile;
    // keys, vals (twice) | histogram | 256-byte slack (merge counters) | digit totals
    return 4 * capacity * 4 + 256 * tiles * 4 + 256 + 4 * 256;
}

extern "C" int64_t oec_sort_work_bytes(int64_t capacity) {
    return oec_cell_sort_work_bytes(capacity) + 32 * capacity + 256;  // rows of 32 bytes, aligned
}

// The digit totals, behind the histogram and its 256-byte slack.
static int *digit_totals(int *hist, int64_t ntiles) { return hist + 256 * ntiles + 64; }

// The packed rows, behind the digit totals.
static float4 *packed_rows(int *hist, int64_t cap) {
    const uintptr_t end = reinterpret_cast<uintptr_t>(digit_totals(hist, (cap + kTile - 1) / kTile) + 256);
    return reinterpret_cast<float4 *>((end + 31) & ~uintptr_t(31));
}

// Stable radix sort of (keys, vals) pairs, keys in work; `bits` significant key bits.
static int radix_sort(uint32_t *keys, int32_t *vals, uint32_t *k2, int32_t *v2, int *hist, const int32_t *n_dev,
                      int64_t cap, int bits, cudaStream_t s, uint32_t **kout, int32_t **vout) {
    int ntiles = (int)((cap + kTile - 1) / kTile);
    int *total = digit_totals(hist, ntiles);
    for (int shift = 0; shift < bits; shift += 8) {
        k_digit_hist<<<ntiles, kSortThreads, 0, s>>>(keys, n_dev, shift, ntiles, hist);
        k_digit_scan<<<256, kDigitScanT, 0, s>>>(hist, ntiles, total);
        k_scatter<<<ntiles, kSortThreads, 0, s>>>(keys, vals, n_dev, shift, ntiles, hist, total, k2, v2);
        uint32_t *tk = keys;
        keys = k2;
        k2 = tk;
        int32_t *tv = vals;
        vals = v2;
        v2 = tv;
    }
    *kout = keys;
    *vout = vals;
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_sort_particles(oec_particles_t *p, oec_particles_t *tmp, int32_t column, void *work_dev,
                                  void *stream) {
    if (!vp2(p) || !vp2(tmp) || !work_dev || tmp->capacity < p->capacity) return OEC_ERR_INVALID;
    if (column < 2 || column > 6) return OEC_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    int64_t cap = p->capacity;
    uint32_t *keys = static_cast<uint32_t *>(work_dev);
    int32_t *vals = reinterpret_cast<int32_t *>(keys + cap);
    uint32_t *k2 = reinterpret_cast<uint32_t *>(vals + cap);
    int32_t *v2 = reinterpret_cast<int32_t *>(k2 + cap);
    int *hist = reinterpret_cast<int *>(v2 + cap);
    int g = persistent_grid((cap + 255) / 256, 8);
    k_make_keys<<<g, 256, 0, s>>>(*p, column, keys, vals);
    OEC_LAUNCH_CHECK();
    int bits = 32;
    if (column == 6) {
        // cell keys: only as many digits as the largest cell index needs
        bits = 24;
    }
    uint32_t *kout;
    int32_t *vout;
    int rc = radix_sort(keys, vals, k2, v2, hist, p->count, cap, bits, s, &kout, &vout);
    if (rc != OEC_OK) return rc;
    if (column == 6) {
        k_permute<<<g, 256, 0, s>>>(*p, vout, *tmp);
    } else {
        float4 *rows = packed_rows(hist, cap);
        k_pack_rows<<<g, 256, 0, s>>>(*p, rows);
        k_permute_rows<<<g, 256, 0, s>>>(rows, vout, p->count, *tmp);
    }
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_weight_thresholds(const oec_particles_t *p, double lo, double hi, int32_t *out_dev,
                                     void *stream) {
    if (!vp2(p) || !out_dev) return OEC_ERR_INVALID;
    k_search_sorted2<<<1, 64, 0, as_stream(stream)>>>(p->w, p->count, lo, hi, out_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_scale_weights(oec_particles_t *p, double factor, void *stream) {
    if (!vp2(p)) return OEC_ERR_INVALID;
    k_scale_w<<<persistent_grid((p->capacity + 255) / 256, 8), 256, 0, as_stream(stream)>>>(*p, factor);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_roulette_select(int32_t n, int32_t n_remove, uint32_t *mask_dev, int64_t mask_words,
                                   uint64_t seed, uint32_t call, int32_t *fails_dev, void *stream) {
    if (n < 0 || n_remove < 0 || n_remove > n || !mask_dev || !fails_dev || mask_words * 32 < n)
        return OEC_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    int nw = (n + 31) / 32;
    k_zero_words<<<persistent_grid((mask_words + 255) / 256, 8), 256, 0, s>>>(mask_dev, (int)mask_words);
    OEC_CUDA_TRY(cudaMemsetAsync(fails_dev, 0, sizeof(int32_t), s));
    // choose the smaller of the removed and the kept sets by darts
    bool invert = n_remove > n / 2;
    int k = invert ? n - n_remove : n_remove;
    if (k > 0)
        k_darts<<<persistent_grid((k + 255) / 256, 8), 256, 0, s>>>(n, k, mask_dev, key, call, 4096, fails_dev);
    if (invert) k_invert_valid<<<persistent_grid((nw + 255) / 256, 8), 256, 0, s>>>(mask_dev, n);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_clone_rows(const oec_grid_t *grid, const oec_particles_t *p, int32_t n, int32_t k, uint64_t seed,
                              uint32_t call, double *rows_dev, void *stream) {
    if (!grid || !vp2(p) || n <= 0 || k < 0 || !rows_dev) return OEC_ERR_INVALID;
    GridConst gc = make_grid_const(*grid);
    uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    if (k > 0)
        k_clone_rows<<<persistent_grid((k + 255) / 256, 8), 256, 0, as_stream(stream)>>>(
            *p, n, k, key, call, gc.nx, 1.0f / (float)gc.nx, gc.dx, gc.dy, gc.lxh, gc.lyh, rows_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_weight_stats(const oec_particles_t *p, double *acc_dev, void *stream) {
    if (!vp2(p) || !acc_dev) return OEC_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    OEC_CUDA_TRY(cudaMemsetAsync(acc_dev, 0, 2 * sizeof(double), s));
    k_wstats<<<persistent_grid((p->capacity + kStatThreads - 1) / kStatThreads, 4), kStatThreads, 0, s>>>(*p, acc_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_weight_sums(const oec_particles_t *p, double *acc_dev, double *scratch_dev, void *stream) {
    if (!vp2(p) || !acc_dev || !scratch_dev) return OEC_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    const int ctas = std::min(persistent_grid((p->capacity + kStatThreads - 1) / kStatThreads, 4), kStatCtas);
    k_wparts<<<ctas, kStatThreads, 0, s>>>(*p, scratch_dev);
    k_wsums<<<1, 64, 0, s>>>(p->count, ctas, scratch_dev, acc_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_split_rows(const oec_grid_t *grid, oec_particles_t *p, int32_t n, int32_t k, double *rows_dev,
                              void *stream) {
    if (!grid || !vp2(p) || k < 0 || k > n || (k > 0 && !rows_dev)) return OEC_ERR_INVALID;
    GridConst gc = make_grid_const(*grid);
    if (k > 0)
        k_split_rows<<<persistent_grid((k + 255) / 256, 8), 256, 0, as_stream(stream)>>>(
            *p, n, k, gc.nx, 1.0f / (float)gc.nx, gc.dx, gc.dy, gc.lxh, gc.lyh, rows_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_cell_merge(const oec_grid_t *grid, oec_particles_t *p, int32_t n_cand, int32_t n_merge,
                              double lambda, double limit, int32_t scheme, uint64_t seed, uint32_t call,
                              double vscale, uint32_t *mask_dev, int32_t *counters_dev, void *work_dev,
                              void *stream) {
    if (!grid || !vp2(p) || n_cand < 0 || n_cand > p->capacity || n_merge < 0 || !mask_dev || !counters_dev ||
        !work_dev)
        return OEC_ERR_INVALID;
    GridConst gc = make_grid_const(*grid);
    (void)vscale;
    cudaStream_t s = as_stream(stream);
    int64_t cap = p->capacity;
    uint32_t *keys = static_cast<uint32_t *>(work_dev);
    int32_t *vals = reinterpret_cast<int32_t *>(keys + cap);
    uint32_t *k2 = reinterpret_cast<uint32_t *>(vals + cap);
    int32_t *v2 = reinterpret_cast<int32_t *>(k2 + cap);
    int *hist = reinterpret_cast<int *>(v2 + cap);
    int32_t *ncand_dev = reinterpret_cast<int32_t *>(hist + 256 * ((cap + kTile - 1) / kTile));
    uint32_t *bbox = reinterpret_cast<uint32_t *>(ncand_dev + 1);  // 10 words (inside the 256-byte slack)
    float4 *rows = packed_rows(hist, cap);
    k_merge_begin<<<1, 32, 0, s>>>(n_cand, ncand_dev, bbox, counters_dev);
    int g = persistent_grid((n_cand + 255) / 256 + 1, 8);
    k_cand_bbox<<<g, 256, 0, s>>>(*p, n_cand, gc.nx, 1.0f / (float)gc.nx, gc.dx, gc.dy, lambda, bbox);
    k_cand_keys<<<g, 256, 0, s>>>(*p, n_cand, gc.nx, 1.0f / (float)gc.nx, gc.dx, gc.dy, lambda, bbox, keys, vals,
                                rows);
    uint32_t *kout;
    int32_t *vout;
    int rc = radix_sort(keys, vals, k2, v2, hist, ncand_dev, cap, 32, s, &kout, &vout);
    if (rc != OEC_OK) return rc;
    MergeArgs a{};
    a.p = *p;
    a.n_cand = n_cand;
    a.n_merge_target = n_merge;
    a.order = vout;
    a.rows = rows;
    a.qual = kout == keys ? k2 : keys;  // the sort's other key buffer
    a.lam2 = lambda * lambda;
    a.limit = limit;
    a.dx = gc.dx;
    a.dy = gc.dy;
    a.nx = gc.nx;
    a.inv_nx = 1.0f / (float)gc.nx;
    a.key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    a.call = call;
    a.scheme = scheme;
    a.mask = mask_dev;
    a.counters = counters_dev;
    k_pair_count<<<g, 256, 0, s>>>(a);
    k_pair_merge<<<g, 256, 0, s>>>(a);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}
