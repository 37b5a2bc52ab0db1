// emit.cu -- Furman-Pivi secondary emission and the uniform loader.
//
// Reference: particleEmitter.pyx FurmanEmitter.generateSecondaries (:154-308)
// and homoLoader (:41-72).  Two passes over the absorbed rows:
//  pass 1: primary energy and incidence angle, elastic/rediffused/true yields
//          and the number of secondaries drawn from P_n (:180-229);
//          summed per 32 rows;
//  emit:   energies (single secondary: elastic/rediffused/true split;
//          several: the joint energy split through I_x and P inverses,
//          :232-278) and cos-law directions about the wall normal (:280-302).
// Every absorbed particle draws from its own Philox stream, so the emitted
// set depends on the absorbed set, the run seed and the step only.
#include <math.h>
#include <stdint.h>

#include "oec_common.cuh"
#include "specfun.cuh"

namespace oec {
namespace {

constexpr int kDraws = 32;  // replay stride: uniforms per absorbed particle

struct Rec {
    double e0, dE, dR, pN1;
    int nsec;
};

// An absorbed row emits only with a finite position, energy and wall normal.
// A non-finite one (the reference would draw ten secondaries from NaN
// yields, each as non-finite, and so on at every step) emits nothing and is
// counted in status->n_emit_skipped.
__device__ __forceinline__ bool row_emits(const double *r, double e0, double n0, double n1) {
    return isfinite(r[0]) && isfinite(r[1]) && isfinite(e0) && isfinite(n0) && isfinite(n1);
}

__device__ __forceinline__ double clip(double x, double lo, double hi) {
    // particleEmitter.pyx:33-39 -- a NaN falls through to `hi`
    if (x <= hi && x >= lo) return x;
    if (x < lo) return lo;
    return hi;
}

constexpr int kSlots = 10;
constexpr int kTileRows = 32;  // rows whose secondaries pass 1 sums
constexpr int kClasses = kSlots * (kSlots + 1) / 2;  // (n, k), k < n: n (n - 1) / 2 + k

// The constants of the inverses of k_furman_emit, by (n, k).
struct SplitConst {
    sf::BetaConst beta[kClasses - kSlots];  // k < n - 1: (n - 1) (n - 2) / 2 + k
    sf::GammaConst gamma[kSlots];           // k = n - 1: n - 1
    sf::GammaConst gamma1[kSlots];          // P(pSmallN[n-1], .): n - 1
};

// The blocks behind the first `row_blocks` lay out the constants of one class
// (n, k) each for the next kernels, beside the rows' work.
__global__ void __launch_bounds__(128)
    k_furman_pass1(oec_furman_t f, const double *__restrict__ rows, const double *__restrict__ normals,
                   const int32_t *n_abs, int cap, const int32_t *__restrict__ ids, uint2 key, uint32_t step,
                   const int32_t *step_dev, const double *__restrict__ replay, Rec *__restrict__ rec,
                   int32_t *__restrict__ tile_sum, oec_status_t *status, int row_blocks,
                   SplitConst *__restrict__ consts) {
    const int na = min(*n_abs, cap);
    if (na <= 0) return;
    if ((int)blockIdx.x >= row_blocks) {
        const int c = blockIdx.x - row_blocks;
        int n = 1, k;
        if (c < kClasses) {
            while (n * (n + 1) / 2 <= c) ++n;
            k = c - n * (n - 1) / 2;
        } else {
            n = k = c - kClasses + 1;
        }
        const double P = f.pSmallN[n - 1];
        if (k == n)  // the blocks behind the classes
            sf::gamma_const(P, consts->gamma1[n - 1]);
        else if (k == n - 1)
            sf::gamma_const(n * P, consts->gamma[n - 1]);
        else
            sf::beta_const(P * (n - k - 1), P, consts->beta[(n - 1) * (n - 2) / 2 + k]);
        return;
    }
    const double eFactor = 0.5 * f.particle_mass / 1.602176565e-19;
    int wd = 0, wt = 0;
    __shared__ double lfac[11];  // lgamma(j + 1), j <= m <= 10
    if ((int)(blockIdx.x * blockDim.x) >= na) return;
    if (threadIdx.x <= f.m) lfac[threadIdx.x] = sf::lgam((double)threadIdx.x + 1.0);
    __syncthreads();
    int skipped = 0;
    // the number of secondaries of row i
    auto row = [&](int i) -> int {
        const double *r = rows + 6 * (int64_t)i;
        const double n0 = normals[2 * i], n1 = normals[2 * i + 1];
        double v0 = sqrt(r[2] * r[2] + r[3] * r[3] + r[4] * r[4]);
        double e0 = eFactor * v0 * v0;
        if (!row_emits(r, e0, n0, n1)) {
            rec[i] = Rec{0., 0., 0., 1., 0};
            ++skipped;
            return 0;
        }
        double th = acos((r[2] * n0 + r[3] * n1) / v0);
        if (th > 0.5 * sf::kPi) th = sf::kPi - th;
        th = clip(th, 0., f.theta0max);
        double ct = cos(th);
        double dE = (f.p1EInf + (f.p1Ehat - f.p1EInf) * exp(-pow(fabs(e0 - f.eEHat) / f.w, f.p) / f.p)) *
                    (1 + f.e1 * (1 - pow(ct, f.e2)));
        double dR = f.p1RInf * (1 - exp(-pow(e0 / f.eR, f.r))) * (1 + f.r1 * (1 - pow(ct, f.r2)));
        double eHat = f.eHat0 * (1 + f.t3 * (1 - pow(ct, f.t4)));
        double dTS0 = f.deltaTSHat * f.s * e0 / eHat / (f.s - 1 + pow(e0 / eHat, f.s));
        double dTS = dTS0 * (1 + f.t1 * (1 - pow(ct, f.t2)));
        double sum = dE + dR;
        if (sum >= f.deltaERmax) {
            dE = dE / sum * f.deltaERmax;
            dR = dR / sum * f.deltaERmax;
            ++wd;
        }
        double dTSp = dTS / (1 - dE - dR);
        if (dTSp >= f.m) {
            dTSp = f.m;
            ++wt;
        } else if (dTSp < 0) {
            dTSp = 0;
        }
        double pr = dTSp / f.m;
        double keep = 1 - dE - dR;
        sf::Draws dr{key, ids ? (uint32_t)ids[i] : (uint32_t)i, step + (step_dev ? (uint32_t)*step_dev : 0u),
                     replay ? replay + (int64_t)i * kDraws : nullptr};
        double u = dr.next();
        // P_n = binom(n; m, pr) (1 - dE - dR), P_1 += dE + dR (:217-221);
        // inverse-CDF draw over n < m, default m (:222-229)
        // binom_pdf(k; m, pr) with lgamma(j+1) and the logs of pr evaluated once
        // (the same values as sf::binom_pdf)
        const double lp = log(pr), l1p = log1p(-pr);
        auto pdf = [&](unsigned k) -> double {
            const unsigned m = (unsigned)f.m;
            if (pr == 0.0) return k == 0 ? 1.0 : 0.0;
            if (pr == 1.0) return k == m ? 1.0 : 0.0;
            const double lc = lfac[m] - lfac[k] - lfac[m - k];
            return exp(lc + k * lp + (double)(m - k) * l1p);
        };
        const double pN1 = pdf(1u) * keep + (dE + dR);
        int n = f.m;
        double cum = 0.0;
        for (int k = 0; k < f.m; ++k) {
            cum += (k == 1) ? pN1 : pdf((unsigned)k) * keep;
            if (u <= cum) {
                n = k;
                break;
            }
        }
        rec[i] = Rec{e0, dE, dR, pN1, n};
        return n;
    };
    // a warp takes kTileRows consecutive rows and leaves their sum for the next kernel's places
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; (i & ~31) < na; i += row_blocks * blockDim.x) {
        const int sum = __reduce_add_sync(kFullMask, i < na ? row(i) : 0);
        if ((i & 31) == 0) tile_sum[i >> 5] = sum;
    }
    if (wd) atomicAdd(&status->warn_derm, wd);
    if (wt) atomicAdd(&status->warn_tsprime, wt);
    if (skipped) atomicAdd(&status->n_emit_skipped, skipped);
}

// A secondary's direction: cos-law about the normal (:280-302), draws dr.d and
// dr.d + 1.  sin(asin u) = u and cos(asin u) = sqrt(1 - u^2).
__device__ __forceinline__ void put_secondary(const double *r, double n0, double n1, double vs, sf::Draws &dr,
                                              double *q) {
    const double sT = dr.next(), cT = sqrt((1. - sT) * (1. + sT));
    double sP, cP;
    sincos(dr.next() * sf::kPi * 2., &sP, &cP);
    const double t1 = cT * n0 - sT * n1;
    const double t2 = sT * n0 + cT * n1;
    q[0] = r[0];
    q[1] = r[1];
    q[2] = vs * ((cP + n0 * n0 * (1 - cP)) * t1 + n0 * n1 * (1 - cP) * t2);
    q[3] = vs * ((cP + n1 * n1 * (1 - cP)) * t2 + n0 * n1 * (1 - cP) * t1);
    q[4] = vs * (-sP * n1 * t1 + sP * n0 * t2);
    q[5] = r[5];
}

// Energies and directions of all secondaries (particleEmitter.pyx:232-302).
// A lone one splits into elastic, rediffused and true.  n > 1 share the energy:
// slot k < n-1 takes B_k = I^-1_u(P(n-k-1), P) from draw 1+k, slot n-1 takes y =
// sqrt(P^-1(nP, u p0)) from draw n, and with sin(theta_k)^2 = B_k secondary k
// gets eps (y cos(theta_k) prod_{t<k} sin(theta_t))^2, the last one without
// the cosine.
//
// The inverses are most of the work.  They differ in their branch and their
// length by (n, k) above all, and most of a row's kSlots slots are empty, so a
// CTA takes a chunk of rows, sorts its secondaries by function and (n, k) in
// shared memory and works them off in that order, a warp taking the next (at
// most) 32 of one function when it is free: the lanes of a warp run the same
// branch of the same function, with the constants of (n, k) from pass 1
// (specfun.cuh), and with few rows the functions run side by side.  Which lane takes which
// does not enter its value.  106,457 absorbed rows of 200 eV electrons (179,048
// secondaries) on a B200: 3340 us for a thread per (row, slot) with the plain
// inverses and a thread per row for the directions, 95 us this way; 250 secondaries
// (one buildup step): 25 us, the latency of one inverse.
constexpr int kSplitT = 256, kSplitRows = 1024;
constexpr int kKinds = 9;  // lone, gamma, and the kinds of sf::BetaConst

struct SplitShared {
    SplitConst c;
    int first[kSplitRows];                  // a row's first secondary, from the chunk's first
    int warp_sum[2][kSplitT / 32];
    unsigned char kind[kClasses];           // the function a class is inverted by
    unsigned char rank[kClasses];           // a class's place in the order of the kinds
    int kind_first[kKinds + 1];             // first rank of a kind
    int count[kClasses + 1];                // per rank: secondaries, then the place after the last one put
    int batch[kKinds][3];                   // per kind: batches before it, first and last place
    int next[2];                            // batches handed out to the warps, per phase
    unsigned char nsec[kSplitRows];
    unsigned task[kSplitRows * kSlots];     // row in the chunk | n << 16 | k << 24
};

// The next batch of this warp, at most 32 secondaries of one kind: this lane's
// place, or -1.  False when none are left.
__device__ __forceinline__ bool next_batch(SplitShared &sh, int *t) {
    int first = -1, last = 0;
    if ((threadIdx.x & 31) == 0) {
        const int b = atomicAdd(&sh.next[0], 1);
        for (int g = 0; g < kKinds; ++g) {
            const int k = b - sh.batch[g][0], at = sh.batch[g][1] + 32 * k;
            if (k >= 0 && at < sh.batch[g][2]) {
                first = at;
                last = min(at + 32, sh.batch[g][2]);
            }
        }
    }
    first = __shfl_sync(kFullMask, first, 0);
    last = __shfl_sync(kFullMask, last, 0);
    *t = first + (int)(threadIdx.x & 31);
    if (*t >= last) *t = -1;
    return first >= 0;
}

// The next 32 secondaries for this warp; this lane's one, or -1.  False when
// none are left.
__device__ __forceinline__ bool next_task(int *next, int total, int *t) {
    int b = 0;
    if ((threadIdx.x & 31) == 0) b = atomicAdd(next, 32);
    b = __shfl_sync(kFullMask, b, 0);
    *t = b + (int)(threadIdx.x & 31);
    if (*t >= total) *t = -1;
    return b < total;
}

__global__ void __launch_bounds__(kSplitT)
    k_furman_emit(oec_furman_t f, const double *__restrict__ rows, const double *__restrict__ normals,
                  const int32_t *n_abs, int cap, const int32_t *__restrict__ ids, uint2 key, uint32_t step,
                  const int32_t *step_dev, const double *__restrict__ replay, const Rec *__restrict__ rec,
                  const SplitConst *__restrict__ consts, double *__restrict__ split,
                  const int32_t *__restrict__ tile_sum, double *__restrict__ out, int out_cap, int32_t *n_out,
                  oec_status_t *status) {
    extern __shared__ __align__(16) unsigned char split_smem[];
    SplitShared &sh = *reinterpret_cast<SplitShared *>(split_smem);
    const int na = min(*n_abs, cap);
    // rows per chunk: all CTAs busy before the chunks reach full size
    const int per = (na + (int)gridDim.x - 1) / (int)gridDim.x;
    const int chunk = min(kSplitRows, max(32, (per + 31) & ~31));
    if (na <= 0 && blockIdx.x == 0 && threadIdx.x == 0) *n_out = 0;
    if ((int)blockIdx.x * chunk >= na) return;
    const uint32_t st = step + (step_dev ? (uint32_t)*step_dev : 0u);
    const int tid = threadIdx.x;
    const double eFactorInv = 1.0 / (0.5 * f.particle_mass / 1.602176565e-19);
    const Rec last = rec[na - 1];
    static_assert(sizeof(SplitConst) % sizeof(int4) == 0, "copied by 16 bytes");
    for (int i = tid; i < (int)(sizeof(SplitConst) / sizeof(int4)); i += kSplitT)
        reinterpret_cast<int4 *>(&sh.c)[i] = __ldg(reinterpret_cast<const int4 *>(consts) + i);
    int dropped = 0;
    const int lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    if (tid < kClasses) {
        int n = 1;
        while (n * (n + 1) / 2 <= tid) ++n;
        const int k = tid - n * (n - 1) / 2;
        sh.kind[tid] = (unsigned char)(n == 1 ? 0 : k == n - 1 ? 1 : 2 + sh.c.beta[(n - 1) * (n - 2) / 2 + k].kind);
    }
    __syncthreads();
    if (tid < kClasses || (tid >= 64 && tid <= 64 + kKinds)) {
        const int key = tid < kClasses ? sh.kind[tid] * 64 + tid : (tid - 64) * 64;
        int r = 0;
        for (int c = 0; c < kClasses; ++c) r += sh.kind[c] * 64 + c < key ? 1 : 0;
        if (tid < kClasses)
            sh.rank[tid] = (unsigned char)r;
        else
            sh.kind_first[tid - 64] = r;
    }
    __syncthreads();
    int before = 0, summed = 0;  // secondaries of the rows before the chunk; tiles in `before`
    for (int r0 = blockIdx.x * chunk; r0 < na; r0 += gridDim.x * chunk) {
        const int nrows = min(chunk, na - r0);
        for (int c = tid; c <= kClasses; c += kSplitT) sh.count[c] = 0;
        if (tid < 2) sh.next[tid] = 0;
        __syncthreads();
        // a thread's kPer consecutive rows: their counts and, by a scan over the
        // CTA, the place of their first secondaries; with them the sum of the
        // tiles between the last chunk and this one
        constexpr int kPer = kSplitRows / kSplitT;
        int cnt[kPer], mine = 0, tiles = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int r = tid * kPer + j;
            cnt[j] = r < nrows ? rec[r0 + r].nsec : 0;
            sh.nsec[r] = (unsigned char)cnt[j];
            for (int k = 0; k < cnt[j]; ++k) atomicAdd(&sh.count[sh.rank[cnt[j] * (cnt[j] - 1) / 2 + k]], 1);
            mine += cnt[j];
        }
        for (int q = summed + tid; q < r0 / kTileRows; q += kSplitT) tiles += tile_sum[q];
        summed = r0 / kTileRows;
        tiles = __reduce_add_sync(kFullMask, tiles);
        int scan = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFullMask, scan, o);
            if (lane >= o) scan += y;
        }
        if (lane == 31) sh.warp_sum[0][warp] = scan;
        if (lane == 0) sh.warp_sum[1][warp] = tiles;
        __syncthreads();
        int at = scan - mine;
        for (int w = 0; w < kSplitT / 32; ++w) {
            if (w < warp) at += sh.warp_sum[0][w];
            before += sh.warp_sum[1][w];
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            sh.first[tid * kPer + j] = at;
            at += cnt[j];
        }
        if (r0 + nrows == na && tid == kSplitT - 1) *n_out = before + at;
        if (tid < 32) {  // exclusive scan of the counts by one warp
            int carry = 0;
            for (int c0 = 0; c0 <= kClasses; c0 += 32) {
                const int c = c0 + tid, v = c < kClasses ? sh.count[c] : 0;
                int x = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFullMask, x, o);
                    if (tid >= o) x += y;
                }
                if (c <= kClasses) sh.count[c] = carry + x - v;
                carry += __shfl_sync(kFullMask, x, 31);
            }
        }
        __syncthreads();
        const int total = sh.count[kClasses], lone = sh.count[1];  // class 0 comes first
        if (tid == 0)
            for (int g = 0, nb = 0; g < kKinds; ++g) {
                const int a = sh.count[sh.kind_first[g]], b = sh.count[sh.kind_first[g + 1]];
                sh.batch[g][0] = nb;
                sh.batch[g][1] = a;
                sh.batch[g][2] = b;
                nb += (b - a + 31) / 32;
            }
        __syncthreads();
        for (int r = tid; r < nrows; r += kSplitT) {
            const int n = sh.nsec[r];
            for (int k = 0; k < n; ++k) sh.task[atomicAdd(&sh.count[sh.rank[n * (n - 1) / 2 + k]], 1)] = r | n << 16 | k << 24;
        }
        __syncthreads();
        // the inverses; a lone secondary is finished here
        int t;
        while (next_batch(sh, &t)) {
            if (t < 0) continue;
            const unsigned w = sh.task[t];
            const int row = r0 + (int)(w & 0xffff), n = (w >> 16) & 0xff, k = w >> 24;
            sf::Draws dr{key, ids ? (uint32_t)ids[row] : (uint32_t)row, st,
                         replay ? replay + (int64_t)row * kDraws : nullptr};
            dr.d = 1 + k;  // draw 0 was the secondary count
            const double u = dr.next();
            if (k < n - 1) {
                split[(int64_t)row * kSlots + k] = sf::betaincinv_t(sh.c.beta[(n - 1) * (n - 2) / 2 + k], sh.c.gamma1[n - 1], u);
                continue;
            }
            const sf::GammaConst &G = sh.c.gamma[n - 1];
            const double e0 = rec[row].e0;
            if (n > 1) {
                split[(int64_t)row * kSlots + k] = sf::gammaincinv_t(G, u * sf::gammainc_of(G, e0 / f.epsN[n - 1]));
                continue;
            }
            // compat: the reference reads the split of the LAST absorbed particle
            // of pass 1 (stale loop variables, particleEmitter.pyx:245-246)
            const Rec S = f.compat_last ? last : rec[row];
            const double aE = S.dE / S.pN1, aR = S.dR / S.pN1;
            double e;
            if (u < aE) {
                const double sig = f.scaleSigmaE ? f.sigmaE * sqrt(e0 / 300) : f.sigmaE;
                e = e0 - fabs(sig * dr.normal());
                if (e < 0.) e = dr.next() * e0;
            } else if (u < aE + aR) {
                e = e0 * pow(dr.next(), 1. / (1. + f.q));
            } else {
                e = f.epsN[0] * sf::gammaincinv_t(G, dr.next() * sf::gammainc_of(G, e0 / f.epsN[0]));
            }
            const int o = before + sh.first[row - r0];
            if (o < out_cap)
                put_secondary(rows + 6 * (int64_t)row, normals[2 * row], normals[2 * row + 1], sqrt(eFactorInv * e), dr,
                              out + 6 * (int64_t)o);
            else
                ++dropped;
        }
        __syncthreads();
        // the shared energies and the directions
        while (next_task(&sh.next[1], total - lone, &t)) {
            if (t < 0) continue;
            const unsigned w = sh.task[lone + t];
            const int row = r0 + (int)(w & 0xffff), n = (w >> 16) & 0xff, k = w >> 24;
            const int o = before + sh.first[row - r0] + k;
            if (o >= out_cap) {
                ++dropped;
                continue;
            }
            const double *B = split + (int64_t)row * kSlots;
            double e = B[n - 1];
            for (int j = 0; j < k; ++j) e *= B[j];
            if (k < n - 1) e *= 1. - B[k];
            sf::Draws dr{key, ids ? (uint32_t)ids[row] : (uint32_t)row, st,
                         replay ? replay + (int64_t)row * kDraws : nullptr};
            dr.d = n + 1 + 2 * k;
            put_secondary(rows + 6 * (int64_t)row, normals[2 * row], normals[2 * row + 1],
                          sqrt(eFactorInv * (f.epsN[n - 1] * e)), dr, out + 6 * (int64_t)o);
        }
        __syncthreads();
        // the rows of this chunk are part of the tiles that the next one sums
    }
    if (dropped) atomicAdd(&status->n_capacity_drop, dropped);
}

// ------------------------------------------------------------------ scan

constexpr int kScanT = 1024;
constexpr int kMaxAbsorbedRows = 1 << 26;

// Blocks of the two-level count scan (at least kScanT partial slots).
inline int scan_blocks(int cap) {
    const int nb = (cap + kScanT - 1) / kScanT;
    return nb > kScanT ? nb : kScanT;
}

__device__ __forceinline__ int block_scan_excl(int v, int *tot, int *sh) {
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
    int before = (wid > 0 ? sh[wid - 1] : 0) + x - v;
    if (tot) *tot = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before;
}

__global__ void k_scan_blocks(const int32_t *in, const int32_t *n_p, int cap, int32_t *out, int *partial) {
    __shared__ int sh[32];
    int n = min(*n_p, cap);
    int i = blockIdx.x * kScanT + threadIdx.x;
    int v = i < n ? in[i] : 0;
    int tot;
    int ex = block_scan_excl(v, &tot, sh);
    if (i < cap) out[i] = ex;
    if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

// Exclusive scan of the nb block totals by one CTA, kScanT at a time with a
// running carry.
__global__ void k_scan_partials(int *partial, int nb, int32_t *total) {
    __shared__ int sh[32];
    int carry = 0;
    for (int base = 0; base < nb; base += kScanT) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? partial[i] : 0;
        int tot;
        const int ex = block_scan_excl(v, &tot, sh);
        if (i < nb) partial[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_scan_add(int32_t *out, const int32_t *n_p, int cap, const int *partial) {
    int n = min(*n_p, cap);
    int i = blockIdx.x * kScanT + threadIdx.x;
    if (i < n) out[i] += partial[blockIdx.x];
}

// The same scan in one CTA when the row capacity is small (a buildup step
// absorbs a few hundred rows of a capacity of tens of thousands): the first
// n rows, kScanT at a time with a running carry, one launch instead of three.
// Rows past n keep what they held; the emission passes read only rows < n.
constexpr int kSmallScanBlocks = 32;

__global__ void __launch_bounds__(kScanT)
    k_scan_small(const int32_t *in, const int32_t *n_p, int cap, int32_t *out, int32_t *total) {
    __shared__ int sh[32];
    const int n = min(*n_p, cap);
    int carry = 0;
    for (int base = 0; base < n; base += kScanT) {  // same trip count in every thread
        const int i = base + threadIdx.x;
        const int v = i < n ? in[i] : 0;
        int tot;
        const int ex = block_scan_excl(v, &tot, sh);
        if (i < n) out[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) *total = carry;
}

// offsets of the rows' secondaries and their total
void scan_counts(const int32_t *nsec, const int32_t *n_abs_dev, int cap, int32_t *off, int *partial,
                 int32_t *n_out_dev, cudaStream_t s) {
    const int nblocks = (cap + kScanT - 1) / kScanT;
    if (nblocks <= kSmallScanBlocks) {
        k_scan_small<<<1, kScanT, 0, s>>>(nsec, n_abs_dev, cap, off, n_out_dev);
        return;
    }
    k_scan_blocks<<<nblocks, kScanT, 0, s>>>(nsec, n_abs_dev, cap, off, partial);
    k_scan_partials<<<1, kScanT, 0, s>>>(partial, nblocks, n_out_dev);
    k_scan_add<<<nblocks, kScanT, 0, s>>>(off, n_abs_dev, cap, partial);
}

// ------------------------------------------- simplified emitters
// SecElecEmitter (particleEmitter.pyx:355-484) and SimpleSecEmitter
// (:506-597): pass 1 draws the elastic / rediffused / true counts (draws
// 0, 1, 2), the scan places each row's secondaries, pass 2 writes them
// (draws from 3 on, in the reference's order).
constexpr int kSecDraws = 64;  // replay stride: uniforms per absorbed row

struct SRec {
    double e0;
    int nE, nR, nT, pad;
};

__global__ void k_secelec_pass1(oec_secelec_t f, const double *__restrict__ rows, const double *__restrict__ normals,
                                const int32_t *n_abs, int cap, const int32_t *__restrict__ ids, uint2 key,
                                uint32_t step, const int32_t *step_dev, const double *__restrict__ replay,
                                SRec *__restrict__ rec, int32_t *__restrict__ nsec, oec_status_t *status) {
    const int na = min(*n_abs, cap);
    const double mass = f.model == 1 ? 9.10938291e-31 : f.particle_mass;
    const double eF = 0.5 * mass / 1.602176565e-19;
    int capped = 0, skipped = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < na; i += gridDim.x * blockDim.x) {
        const double *r = rows + 6 * (int64_t)i;
        const double v0 = sqrt(r[2] * r[2] + r[3] * r[3] + r[4] * r[4]);
        const double e0 = eF * v0 * v0;
        if (!row_emits(r, e0, normals[2 * i], normals[2 * i + 1])) {
            rec[i] = SRec{0., 0, 0, 0, 0};
            nsec[i] = 0;
            ++skipped;
            continue;
        }
        double dE, dR, dTS;
        if (f.model == 1) {
            const double s = 1.813, eHat = 310;
            dE = 0.05;
            dR = 0.5;
            dTS = 1.4 * s * e0 / eHat / (s - 1 + pow(e0 / eHat, s));
        } else {
            double th = acos((r[2] * normals[2 * i] + r[3] * normals[2 * i + 1]) / v0);
            if (th > 0.5 * sf::kPi) th = sf::kPi - th;
            th = clip(th, 0., f.theta0max);
            const double ct = cos(th);
            dE = (f.p1EInf + (f.p1Ehat - f.p1EInf) * exp(-pow(fabs(e0 - f.eEHat) / f.w, f.p) / f.p)) *
                 (1 + f.e1 * (1 - pow(ct, f.e2)));
            dR = f.p1RInf * (1 - exp(-pow(e0 / f.eR, f.r))) * (1 + f.r1 * (1 - pow(ct, f.r2)));
            const double eHat = f.eHat0 * (1 + f.t3 * (1 - pow(ct, f.t4)));
            dTS = f.deltaTSHat * f.s * e0 / eHat / (f.s - 1 + pow(e0 / eHat, f.s)) * (1 + f.t1 * (1 - pow(ct, f.t2)));
            const double t = dE + dR;
            if (t >= f.deltaERmax) {
                dE = dE / t * f.deltaERmax;
                dR = dR / t * f.deltaERmax;
            }
        }
        sf::Draws dr{key, ids ? (uint32_t)ids[i] : (uint32_t)i, step + (step_dev ? (uint32_t)*step_dev : 0u),
                     replay ? replay + (int64_t)i * kSecDraws : nullptr};
        const int nE = dr.next() <= dE ? 1 : 0;
        const int nR = dr.next() <= dR ? 1 : 0;
        // <unsigned int> truncation of the reference (:391, :553), then +1
        // with the probability of the fraction; a huge yield is capped below
        int nT = dTS >= 1e9 ? 1000000000 : (dTS > 0.0 ? (int)dTS : 0);
        if (dr.next() <= dTS - nT) ++nT;
        if (nT > f.max_ts) {
            nT = f.max_ts;
            ++capped;
        }
        rec[i] = SRec{e0, nE, nR, nT, 0};
        nsec[i] = nE + nR + nT;
    }
    if (capped) atomicAdd(&status->warn_tsprime, capped);
    if (skipped) atomicAdd(&status->n_emit_skipped, skipped);
}

__device__ __forceinline__ void put_row(double *q, const double *r, double vx, double vy, double vz) {
    q[0] = r[0];
    q[1] = r[1];
    q[2] = vx;
    q[3] = vy;
    q[4] = vz;
    q[5] = r[5];
}

__global__ void k_secelec_pass2(oec_secelec_t f, const double *__restrict__ rows, const double *__restrict__ normals,
                                const int32_t *n_abs, int cap, const int32_t *__restrict__ ids, uint2 key,
                                uint32_t step, const int32_t *step_dev, const double *__restrict__ replay,
                                const SRec *__restrict__ rec, const int32_t *__restrict__ offset,
                                double *__restrict__ out, int out_cap, oec_status_t *status) {
    const int na = min(*n_abs, cap);
    const double mass = f.model == 1 ? 9.10938291e-31 : f.particle_mass;
    const double eFi = 1.0 / (0.5 * mass / 1.602176565e-19);
    int dropped = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < na; i += gridDim.x * blockDim.x) {
        const SRec R = rec[i];
        if (R.nE + R.nR + R.nT == 0) continue;
        const double *r = rows + 6 * (int64_t)i;
        sf::Draws dr{key, ids ? (uint32_t)ids[i] : (uint32_t)i, step + (step_dev ? (uint32_t)*step_dev : 0u),
                     replay ? replay + (int64_t)i * kSecDraws : nullptr};
        dr.d = 3;  // draws 0..2 were the counts
        int o = offset[i];
        auto slot = [&](void) -> double * {
            if (o >= out_cap) {
                ++dropped;
                ++o;
                return nullptr;
            }
            return out + 6 * (int64_t)(o++);
        };
        if (R.nE) {
            if (double *q = slot()) put_row(q, r, -r[2], -r[3], -r[4]);
        }
        if (R.nR) {
            const double u = dr.next();
            const double vF = f.model == 1 ? sqrt(u) : sqrt(pow(u, 1. / (1. + f.q)));
            if (double *q = slot()) put_row(q, r, -r[2] * vF, -r[3] * vF, -r[4] * vF);
        }
        const int n = R.nT;
        if (n <= 0) continue;
        double eSec[10];
        if (f.model == 1) {
            for (int k = 0; k < n; ++k) eSec[k] = dr.next() * 5;
            for (int k = 0; k < n; ++k) {
                const double vF = sqrt(eSec[k] / R.e0);
                if (double *q = slot()) put_row(q, r, -r[2] * vF, -r[3] * vF, -r[4] * vF);
            }
            continue;
        }
        double eSum = 0.;
        for (int k = 0; k < n; ++k) {
            eSec[k] = exp(f.sigmaETS * dr.normal() + f.muETS);
            eSum += eSec[k];
        }
        if (eSum > R.e0)
            for (int k = 0; k < n; ++k) eSec[k] = dr.next() * R.e0 / n;
        const double n0 = normals[2 * i], n1 = normals[2 * i + 1];
        for (int k = 0; k < n; ++k) {
            const double vs = sqrt(eFi * eSec[k]);
            const double thS = asin(dr.next());
            const double cT = cos(thS), sT = sin(thS);
            const double phS = dr.next() * sf::kPi * 2.;
            const double cP = cos(phS), sP = sin(phS);
            const double t1 = cT * n0 - sT * n1, t2 = sT * n0 + cT * n1;
            if (double *q = slot())
                put_row(q, r, vs * ((cP + n0 * n0 * (1 - cP)) * t1 + n0 * n1 * (1 - cP) * t2),
                        vs * ((cP + n1 * n1 * (1 - cP)) * t2 + n0 * n1 * (1 - cP) * t1),
                        vs * (-sP * n1 * t1 + sP * n0 * t2));
        }
    }
    if (dropped) atomicAdd(&status->n_capacity_drop, dropped);
}

// ---------------------------------------------------------- homoLoader

// Rejection sampling of uniform positions inside the boundary
// (particleEmitter.pyx:52-63) with Philox draws: particle i tries
// candidate points until one is inside (at most `max_tries`).
__global__ void k_homo_load(oec_particles_t p, int64_t n, int kind, double lx, double ly, const uint16_t *faces,
                           const double *bpts, const int32_t *cpi, double lxh_ext, double lyh_ext, double dx,
                           double dy, int nx, int ny, double w0, double vsigma, int randomize_weight, uint2 key,
                           int max_tries, int32_t *failed) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        sf::Draws dr{key, (uint32_t)i, 0xffffffffu, nullptr};
        double x = 0, y = 0;
        bool ok = false;
        for (int t = 0; t < max_tries && !ok; ++t) {
            x = (dr.next() - 0.5) * lx;
            y = (dr.next() - 0.5) * ly;
            if (kind == OEC_BOUNDARY_RECT) {
                ok = !(x < -lx * 0.5 || x > lx * 0.5 || y < -ly * 0.5 || y > ly * 0.5);
            } else if (kind == OEC_BOUNDARY_ELLIPSE) {
                ok = !(x * x * (4. / (lx * lx)) + y * y * (4. / (ly * ly)) >= 1.);
            } else {
                int ix = (int)((x + lxh_ext) * (1. / dx)), iy = (int)((y + lyh_ext) * (1. / dy));
                int c = ix + iy * nx;
                unsigned fc = faces[c];
                if (fc == 8) ok = true;
                else if (fc == 0) ok = false;
                else {
                    int a = cpi[2 * c], b = cpi[2 * c + 1];
                    ok = a >= 0 && b >= 0 &&
                         (bpts[2 * a] - x) * (bpts[2 * b + 1] - y) > (bpts[2 * b] - x) * (bpts[2 * a + 1] - y);
                }
            }
        }
        if (!ok) atomicAdd(failed, 1);
        double ux = (x + lxh_ext) * (1. / dx), uy = (y + lyh_ext) * (1. / dy);
        int ix = (int)fmax(fmin(floor(ux), (double)(nx - 2)), 0.0);
        int iy = (int)fmax(fmin(floor(uy), (double)(ny - 2)), 0.0);
        p.cell[i] = ix + iy * nx;
        p.ox[i] = fminf(fmaxf((float)(ux - ix), 0.f), 0x1.fffffep-1f);
        p.oy[i] = fminf(fmaxf((float)(uy - iy), 0.f), 0x1.fffffep-1f);
        p.vx[i] = (float)(dr.normal() * vsigma);
        p.vy[i] = (float)(dr.normal() * vsigma);
        p.vz[i] = (float)(dr.normal() * vsigma);
        p.w[i] = (float)(randomize_weight ? w0 * (0.5 + dr.next()) : w0);
    }
}

}  // namespace
}  // namespace oec

using namespace oec;

extern "C" int oec_furman_emit(const oec_furman_t *params, const double *rows_dev, const double *normals_dev,
                               const int32_t *n_abs_dev, int32_t cap, const int32_t *ids_dev, uint64_t seed,
                               uint32_t step, const int32_t *step_dev, const double *replay_uniforms_dev,
                               void *work_dev,
                               double *out_rows_dev, int32_t out_cap, int32_t *n_out_dev, oec_status_t *status_dev,
                               void *stream) {
    if (!params || !rows_dev || !normals_dev || !n_abs_dev || !work_dev || !out_rows_dev || !n_out_dev ||
        !status_dev || cap < 0 || out_cap < 0 || params->m < 1 || params->m > 10)
        return OEC_ERR_INVALID;
    if (cap > kMaxAbsorbedRows) return OEC_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    // work layout: SplitConst | Rec[cap] | split[cap * kSlots] (f64) | tile_sum[cap / kTileRows], from the
    // first multiple of 16 bytes on (SplitConst is read 16 bytes at a time; the work bytes have the slack)
    char *w = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(work_dev) + 15) & ~uintptr_t(15));
    SplitConst *consts = reinterpret_cast<SplitConst *>(w);
    Rec *rec = reinterpret_cast<Rec *>(w + sizeof(SplitConst));
    double *split = reinterpret_cast<double *>(rec + cap);
    int32_t *tile_sum = reinterpret_cast<int32_t *>(split + (size_t)cap * kSlots);
    uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    const int g = persistent_grid((cap + 127) / 128, 8);
    k_furman_pass1<<<g + kClasses + kSlots, 128, 0, s>>>(*params, rows_dev, normals_dev, n_abs_dev, cap, ids_dev, key, step,
                                                         step_dev, replay_uniforms_dev, rec, tile_sum, status_dev, g,
                                                         consts);
    static std::atomic<int> attr[kMaxDevices];
    const int ok = per_device_cached(attr, [] {
        return cudaFuncSetAttribute(k_furman_emit, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(SplitShared)) == cudaSuccess
                   ? 1
                   : 0;
    });
    if (!ok) return OEC_ERR_CUDA;
    k_furman_emit<<<persistent_grid((cap + 31) / 32, 2), kSplitT, sizeof(SplitShared), s>>>(
        *params, rows_dev, normals_dev, n_abs_dev, cap, ids_dev, key, step, step_dev, replay_uniforms_dev, rec, consts,
        split, tile_sum, out_rows_dev, out_cap, n_out_dev, status_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int oec_secelec_emit(const oec_secelec_t *params, const double *rows_dev, const double *normals_dev,
                                const int32_t *n_abs_dev, int32_t cap, const int32_t *ids_dev, uint64_t seed,
                                uint32_t step, const int32_t *step_dev, const double *replay_uniforms_dev,
                                void *work_dev, double *out_rows_dev, int32_t out_cap, int32_t *n_out_dev,
                                oec_status_t *status_dev, void *stream) {
    if (!params || !rows_dev || !normals_dev || !n_abs_dev || !work_dev || !out_rows_dev || !n_out_dev ||
        !status_dev || cap < 0 || out_cap < 0 || params->model < 0 || params->model > 1 || params->max_ts < 1 ||
        params->max_ts > 10 || cap > kMaxAbsorbedRows)
        return OEC_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    // work layout: SRec[cap] | nsec[cap] | offset[cap] | partial[scan_blocks(cap)]
    char *w = static_cast<char *>(work_dev);
    SRec *rec = reinterpret_cast<SRec *>(w);
    int32_t *nsec = reinterpret_cast<int32_t *>(w + sizeof(SRec) * (size_t)cap);
    int32_t *off = nsec + cap;
    int *partial = off + cap;
    const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    const int g = persistent_grid((cap + 127) / 128, 8);
    k_secelec_pass1<<<g, 128, 0, s>>>(*params, rows_dev, normals_dev, n_abs_dev, cap, ids_dev, key, step, step_dev,
                                      replay_uniforms_dev, rec, nsec, status_dev);
    if (cap > 0) {
        scan_counts(nsec, n_abs_dev, cap, off, partial, n_out_dev, s);
    } else {
        OEC_CUDA_TRY(cudaMemsetAsync(n_out_dev, 0, sizeof(int32_t), s));
    }
    k_secelec_pass2<<<g, 128, 0, s>>>(*params, rows_dev, normals_dev, n_abs_dev, cap, ids_dev, key, step, step_dev,
                                      replay_uniforms_dev, rec, off, out_rows_dev, out_cap, status_dev);
    OEC_LAUNCH_CHECK();
    return OEC_OK;
}

extern "C" int64_t oec_secelec_work_bytes(int32_t cap) {
    if (cap < 0 || cap > kMaxAbsorbedRows) return -1;
    return (int64_t)sizeof(SRec) * cap + 2 * sizeof(int32_t) * (int64_t)cap + sizeof(int) * (int64_t)scan_blocks(cap) +
           256;
}

extern "C" int64_t oec_furman_work_bytes(int32_t cap) {
    if (cap < 0 || cap > kMaxAbsorbedRows) return -1;
    return (int64_t)sizeof(SplitConst) + (int64_t)sizeof(Rec) * cap + (int64_t)sizeof(double) * kSlots * cap +
           sizeof(int32_t) * ((int64_t)cap / kTileRows + 1) + 256;
}

extern "C" int oec_homo_load(const oec_grid_t *grid, const oec_boundary_t *boundary, oec_particles_t *p, int64_t n,
                             double weight, double vsigma, int32_t randomize_weight, uint64_t seed,
                             int32_t *failed_dev, void *stream) {
    if (!grid || !boundary || !p || n < 0 || n > p->capacity || !failed_dev) return OEC_ERR_INVALID;
    GridConst gc = make_grid_const(*grid);
    cudaStream_t s = as_stream(stream);
    int32_t cnt = (int32_t)n;
    OEC_CUDA_TRY(cudaMemsetAsync(failed_dev, 0, sizeof(int32_t), s));
    uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    k_homo_load<<<persistent_grid((n + 255) / 256, 8), 256, 0, s>>>(
        *p, n, boundary->kind, gc.lx, gc.ly, boundary->inside_faces_dev, boundary->boundary_points_dev,
        boundary->cut_cell_points_ind_dev, gc.lxh, gc.lyh, gc.dx, gc.dy, gc.nx, gc.ny, weight, vsigma,
        randomize_weight, key, 1000, failed_dev);
    OEC_LAUNCH_CHECK();
    OEC_CUDA_TRY(cudaMemcpyAsync(p->count, &cnt, sizeof(int32_t), cudaMemcpyHostToDevice, s));
    OEC_CUDA_TRY(cudaStreamSynchronize(s));  // `cnt` lives on this stack frame
    return OEC_OK;
}
