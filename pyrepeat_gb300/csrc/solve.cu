// Constraints and the bordered solve, on the device in FP64.
//
// Replaces repeat.py:2278-2313: symmetry folding (repeat.py:2445-2470: columns
// of every group into its base, then rows, linked atoms dropped), RESP
// restraints on the folded diagonal (repeat.py:2511-2520), the (n+1) bordered
// total-charge system [[A, w],[w^T, 0]] [q; l] = [b; Q] (repeat.py:2296-2304)
// solved by LU with partial pivoting (scipy.linalg.solve / repeat_cpu_omp.cpp:
// 466-495), then charges expanded to the linked atoms (repeat.py:2472-2489).
//
// For disjoint groups (each atom in at most one group) folding is the gather
//   A_red[r][c] = sum_{i in G(r)} sum_{j in G(c)} A[i][j],  b_red[r] = sum_{i in G(r)} b[i],
//   w[r] = |G(r)|
// which equals the reference's sequential column-then-row folding.  Groups
// that overlap are folded on the host with the reference's sequential rules.
//
// One CTA solves one system (so a batch of systems is one launch).  It factors the
// bordered matrix in FP32 (LU with partial pivoting) and refines x += LU32^{-1}(b - A x)
// with FP64 residuals until the backward error |b - A x| <= n eps64 |A| |x| (the
// classic mixed-precision iterative refinement; FP64 runs at a small fraction of
// the FP32 rate on this part).  If the FP32 factorisation meets a zero pivot or the
// refinement stalls (a step that does not halve the residual, or kRefineMax steps:
// cond(A) near 1/eps32), the system is factored again in FP64 with one step of FP64
// refinement.  Either way the refined residual and the pivot range are reported.
// Systems of kLUWideMin or more unknowns are factored and refined across the whole GPU instead of by
// their CTA (lu_wide_factor, refine_across), in FP32 and, when that stalls, in FP64
// (factor_refine_wide64).  Those of kLUHost64Min or more are refined across it too, and factored
// across it when single; several of a launch are factored in their CTAs, to the same bits.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <set>
#include <utility>

#include <cooperative_groups.h>

#include "common.cuh"

namespace rp {

namespace {

// Folded bordered matrices of many systems in one launch: blockIdx.y picks the system (from
// `sys`, the ones with disjoint groups), the blocks along x stride over its (n+1)^2 entries.
__global__ void build_bordered_kernel(const SolveDesc *__restrict__ descs, const int *__restrict__ sys) {
    const SolveDesc d = descs[sys[blockIdx.y]];
    const int n1 = d.n + 1;
    long long total = (long long)n1 * n1;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        int r = (int)(t / n1), c = (int)(t - (long long)r * n1);
        double v;
        if (r < d.n && c < d.n) {
            v = 0.0;
            for (int p = d.mem_ptr[r]; p < d.mem_ptr[r + 1]; ++p) {
                const double *row = d.A + (size_t)d.mem_idx[p] * d.N;
                for (int q = d.mem_ptr[c]; q < d.mem_ptr[c + 1]; ++q) v += row[d.mem_idx[q]];
            }
            if (r == c && d.resp_s) v += d.resp_s[r];
        } else if (r < d.n) {
            v = (double)(d.mem_ptr[r + 1] - d.mem_ptr[r]);
        } else if (c < d.n) {
            v = (double)(d.mem_ptr[c + 1] - d.mem_ptr[c]);
        } else {
            v = 0.0;
        }
        d.A0[t] = v;
        if (c == 0) {
            double bv;
            if (r < d.n) {
                bv = 0.0;
                for (int p = d.mem_ptr[r]; p < d.mem_ptr[r + 1]; ++p) bv += d.b[d.mem_idx[p]];
                if (d.resp_s) bv += d.resp_s[r] * d.resp_t[r];
            } else {
                bv = d.qtot;
            }
            d.bs[r] = bv;
        }
    }
}

// A warp per row of a system to be solved in its CTA: the FP32 copy of the bordered matrix (into the
// first half of As) and the row sums of |K| (into r) and of |A|, A the folded normal matrix
// without the border (into x), for the solve kernel's norms.  Across the GPU because FP64
// conversions and additions run at 1/64 of the FP32 rate: in the system's own CTA they took 45
// (copy) + 69 + 68 us (norms) at 425 unknowns.
__global__ void __launch_bounds__(256) prepare_kernel(const SolveDesc *__restrict__ descs) {
    const SolveDesc d = descs[blockIdx.y];
    const int n1 = d.n + 1, r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (d.wide64 || d.host32 || r >= n1) return;
    const double *row = d.A0 + (size_t)r * n1;
    float *L = reinterpret_cast<float *>(d.As) + (size_t)r * n1;
    double s = 0.0;
    for (int c = lane; c < n1; c += 32) {
        const double v = row[c];
        if (!d.across) L[c] = (float)v;  // (factors from across the GPU stay)
        s += c < d.n ? fabs(v) : 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        d.r[r] = s + fabs(row[d.n]);
        d.x[r] = r < d.n ? s : 0.0;
    }
}

constexpr int kLU = 1024;    // threads of a panel CTA of the factorisation across the GPU
constexpr int kSolve = 768;  // most threads of a solve CTA (solve_threads): 80 registers each

__device__ void block_argmax(double v, int idx, double *sv, int *si, double *out_v, int *out_i) {
    // max |v| with lowest index on ties (deterministic)
    for (int o = 16; o > 0; o >>= 1) {
        double ov = __shfl_down_sync(0xffffffffu, v, o);
        int oi = __shfl_down_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { sv[w] = v; si[w] = idx; }
    __syncthreads();
    if (w == 0) {
        v = (lane < (int)(blockDim.x >> 5)) ? sv[lane] : -1.0;
        idx = (lane < (int)(blockDim.x >> 5)) ? si[lane] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) {
            double ov = __shfl_down_sync(0xffffffffu, v, o);
            int oi = __shfl_down_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
        }
        if (lane == 0) { *out_v = v; *out_i = idx; }
    }
    __syncthreads();
}

// max of non-negative doubles over the block (their bits order like the values, so no FP64
// instruction runs: one holds that pipe for 16 cycles per warp); every thread gets the
// result.  `active`: the threads that may hold a non-zero value, a prefix.
__device__ double block_max(double v, int active, double *sv) {
    const int warp = threadIdx.x >> 5, nw = min((active + 31) >> 5, (int)(blockDim.x >> 5));
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    auto warp_max = [](unsigned long long x) {
        const unsigned hi = (unsigned)(x >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)x : 0u);
        return ((unsigned long long)mh << 32) | ml;
    };
    unsigned long long *sb = reinterpret_cast<unsigned long long *>(sv);
    __syncthreads();
    if (warp < nw) {
        b = warp_max(b);
        if ((threadIdx.x & 31) == 0) sb[warp] = b;
    }
    __syncthreads();
    b = warp_max((threadIdx.x & 31) < nw ? sb[threadIdx.x & 31] : 0ull);
    return __longlong_as_double((long long)b);
}

// sum over the block in a fixed order; every thread gets the result.  `active` as above.
__device__ double block_sum(double v, int active, double *sv) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31,
              nw = min((active + 31) >> 5, (int)(blockDim.x >> 5));
    __syncthreads();
    if (warp < nw) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sv[warp] = v;
    }
    __syncthreads();
    if (warp == 0) {
        double t = lane < nw ? sv[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sv[32] = t;
    }
    __syncthreads();
    return sv[32];
}

__device__ void lu_apply(const double *__restrict__ LU, const int *__restrict__ perm, int n1, double *y, double *ysh) {
    // solve (P L U) z = y in place (y global; ysh: n1 doubles of shared memory, or y itself), blocked by 32
    // columns: the diagonal block is solved by one warp with shuffles, then every thread
    // updates one remaining row with the block's 32 values (a warp instruction covers 32 rows:
    // the FP64 pipe takes as long for one lane as for 32).  The row interchanges run in
    // shared memory.  Three barriers per 32 columns.
    __shared__ double blk[32][33];
    __shared__ double yb[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    for (int t = threadIdx.x; t < n1; t += blockDim.x) ysh[t] = y[t];
    __syncthreads();
    if (threadIdx.x == 0) {
        int k = 0;
        for (; k + 8 <= n1; k += 8) {  // the interchanges' indices are independent loads
            int p[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) p[u] = perm[k + u];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (p[u] != k + u) { const double t = ysh[k + u]; ysh[k + u] = ysh[p[u]]; ysh[p[u]] = t; }
        }
        for (; k < n1; ++k) {
            const int p = perm[k];
            if (p != k) { const double t = ysh[k]; ysh[k] = ysh[p]; ysh[p] = t; }
        }
    }
    __syncthreads();
    for (int c0 = 0; c0 < n1; c0 += 32) {  // forward: L, unit diagonal
        const int bs = min(32, n1 - c0);
        for (int t = threadIdx.x; t < bs * 32; t += blockDim.x) {
            const int r = t >> 5, c = t & 31;
            blk[r][c] = c < bs ? LU[(size_t)(c0 + r) * n1 + c0 + c] : 0.0;
        }
        __syncthreads();
        if (warp == 0) {
            double yv = lane < bs ? ysh[c0 + lane] : 0.0;
            for (int c = 0; c < bs - 1; ++c) {
                const double yc = __shfl_sync(0xffffffffu, yv, c);
                if (lane > c && lane < bs) yv -= blk[lane][c] * yc;
            }
            if (lane < bs) ysh[c0 + lane] = yv;
            yb[lane] = lane < bs ? yv : 0.0;
        }
        __syncthreads();
        for (int r = c0 + bs + threadIdx.x; r < n1; r += blockDim.x) {
            const double *row = LU + (size_t)r * n1 + c0;
            double t = 0.0;
            for (int c = 0; c < bs; ++c) t += row[c] * yb[c];
            ysh[r] -= t;
        }
        __syncthreads();
    }
    for (int c1 = n1; c1 > 0; c1 -= 32) {  // backward: U
        const int c0 = max(0, c1 - 32), bs = c1 - c0;
        for (int t = threadIdx.x; t < bs * 32; t += blockDim.x) {
            const int r = t >> 5, c = t & 31;
            blk[r][c] = c < bs ? LU[(size_t)(c0 + r) * n1 + c0 + c] : 0.0;
        }
        __syncthreads();
        if (warp == 0) {
            double yv = lane < bs ? ysh[c0 + lane] : 0.0;
            for (int c = bs - 1; c >= 0; --c) {
                if (lane == c) yv = yv / blk[c][c];
                const double xc = __shfl_sync(0xffffffffu, yv, c);
                if (lane < c) yv -= blk[lane][c] * xc;
            }
            if (lane < bs) ysh[c0 + lane] = yv;
            yb[lane] = lane < bs ? yv : 0.0;
        }
        __syncthreads();
        for (int r = threadIdx.x; r < c0; r += blockDim.x) {
            const double *row = LU + (size_t)r * n1 + c0;
            double t = 0.0;
            for (int c = 0; c < bs; ++c) t += row[c] * yb[c];
            ysh[r] -= t;
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < n1; t += blockDim.x) y[t] = ysh[t];
    __syncthreads();
}

// max |v| with the lowest index on ties (deterministic), FP32: the FP32 factorisation's
// pivot search stays off the FP64 pipe (a warp-wide FP64 compare holds that pipe for
// 16 cycles, and every warp of the CTA runs this at every column)
__device__ void block_argmax_f(float v, int idx, float *sv, int *si, int *out_i) {
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_down_sync(0xffffffffu, v, o);
        const int oi = __shfl_down_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { sv[w] = v; si[w] = idx; }
    __syncthreads();
    if (w == 0) {
        v = (lane < (int)(blockDim.x >> 5)) ? sv[lane] : -1.0f;
        idx = (lane < (int)(blockDim.x >> 5)) ? si[lane] : 0x7fffffff;
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_down_sync(0xffffffffu, v, o);
            const int oi = __shfl_down_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
        }
        if (lane == 0) *out_i = idx;
    }
    __syncthreads();
}

// FP32 LU with partial pivoting, in place; false on a zero or non-finite pivot
__device__ bool lu_factor_f32(float *A, int *perm, int n1, double *sv, int *si, double *piv_v, int *piv_i,
                              double &pmin, double &pmax) {
    float *svf = reinterpret_cast<float *>(sv);
    float fmin_p = 3.0e38f, fmax_p = 0.f;
    for (int k = 0; k < n1; ++k) {
        float best = -1.0f;
        int bi = 0x7fffffff;
        for (int r = k + threadIdx.x; r < n1; r += blockDim.x) {
            const float v = fabsf(A[(size_t)r * n1 + k]);
            if (v > best || (v == best && r < bi)) { best = v; bi = r; }
        }
        block_argmax_f(best, bi, svf, si, piv_i);
        const int p = *piv_i < n1 ? *piv_i : k;  // no candidate (NaN): stay
        if (threadIdx.x == 0) perm[k] = p;
        if (p != k)
            for (int c = threadIdx.x; c < n1; c += blockDim.x) {
                const float t = A[(size_t)k * n1 + c];
                A[(size_t)k * n1 + c] = A[(size_t)p * n1 + c];
                A[(size_t)p * n1 + c] = t;
            }
        __syncthreads();
        const float pv = A[(size_t)k * n1 + k];
        const float apv = fabsf(pv);
        if (!(apv > 0.f) || !isfinite(pv)) return false;
        fmin_p = fminf(fmin_p, apv);
        fmax_p = fmaxf(fmax_p, apv);
        const float inv = 1.0f / pv;
        for (int r = k + 1 + threadIdx.x; r < n1; r += blockDim.x) A[(size_t)r * n1 + k] *= inv;
        __syncthreads();
        // rank-1 update: a warp per row, lanes along the row (coalesced, no index division)
        const float *prow = A + (size_t)k * n1;
        for (int rr = k + 1 + (threadIdx.x >> 5); rr < n1; rr += (int)(blockDim.x >> 5)) {
            float *row = A + (size_t)rr * n1;
            const float l = row[k];
            for (int cc = k + 1 + (threadIdx.x & 31); cc < n1; cc += 32) row[cc] -= l * prow[cc];
        }
        __syncthreads();
    }
    pmin = fmin(pmin, (double)fmin_p);
    pmax = fmax(pmax, (double)fmax_p);
    (void)piv_v;
    return true;
}

// Blocked FP32 LU with partial pivoting (right-looking, panels of 32 columns), in place, for systems
// of at most one row per thread; false on a zero or non-finite pivot.  Every element takes
// its updates one column at a time in column order (as an unblocked factorisation), so the
// factors do not depend on the blocking.
// What bounded the first form of it (panel rows in shared memory, one output per thread in the
// trailing update): two shared-memory reads per multiply-add and four barriers per column,
// 3.0 us per column at 425 unknowns.  Here a thread holds its row of the panel in registers;
// a column costs two barriers (the pivot search's partial results, then the pivot row); rows
// change places by their position numbers only, and the panel's net permutation is applied
// to the other columns through shared memory in one pass; the trailing update computes 8 rows x
// 4 columns per thread (6 shared-memory reads per 32 multiply-adds).
// orig[i]: the row of the input that ends up as row i.  work: 64 n1 floats of shared memory.
constexpr int kLUNB = 32;
constexpr int kLUBlockedMax = kSolve;
struct LuShared {
    unsigned key[2][32];                 // per warp: the largest |value| of the column (bits)
    int pos[2][32];                      // and the lowest position that has it
    float prow[2][kLUNB];                // the pivot row
    __align__(16) float l11[kLUNB][kLUNB + 4];  // L11 by columns
    int src[2 * kLUNB], dst[2 * kLUNB];  // rows of the panel's net permutation
    int moved;                           // entries beyond the first kLUNB
};
template <int NI>
__device__ __forceinline__ void lu_trailing_tile(float *A, int n1, const float *L, const float *U, int nb, int r,
                                                 int nr, int c, int nc, int ld) {
    // rows r .. r+7 (nr of them exist), columns c + 32 i (lane-strided; nc of the warp's 32 NI exist)
    float acc[8][NI];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k)
            acc[k][i] = (k < nr && lane + 32 * i < nc) ? A[(size_t)(r + k) * n1 + c + 32 * i] : 0.f;
#pragma unroll 4
    for (int j = 0; j < nb; ++j) {
        const float4 la = *reinterpret_cast<const float4 *>(L + (size_t)j * ld),
                     lb = *reinterpret_cast<const float4 *>(L + (size_t)j * ld + 4);
        const float l[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const float u = U[(size_t)j * ld + 32 * i];
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k][i] = fmaf(-l[k], u, acc[k][i]);
        }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k < nr && lane + 32 * i < nc) A[(size_t)(r + k) * n1 + c + 32 * i] = acc[k][i];
}
__device__ bool lu_factor_f32_blocked(float *A, int *orig, int n1, float *work, LuShared &sh, double &pmin,
                                      double &pmax) {
    const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    const int ld = (n1 + 3) & ~3;            // work rows: 16-byte aligned
    float *S = work, *LT = work + (size_t)kLUNB * ld;  // [32][ld] each: the top rows / U12, and L21 by columns
    float fmin_p = 3.0e38f, fmax_p = 0.f;
    for (int t = tid; t < n1; t += nt) orig[t] = t;
    bool ok = true;
    for (int k0 = 0; k0 < n1; k0 += kLUNB) {
        const int nb = min(kLUNB, n1 - k0), m = n1 - k0, c1 = k0 + nb;
        const bool own = tid < m;  // this thread's row of the panel: position tid at first
        // 1. the panel's rows, coalesced through shared memory, into registers
        __syncthreads();
        for (int r = warp; r < m; r += nw) work[r * 33 + lane] = lane < nb ? A[(size_t)(k0 + r) * n1 + k0 + lane] : 0.f;
        __syncthreads();
        float a[kLUNB];
#pragma unroll
        for (int c = 0; c < kLUNB; ++c) a[c] = own ? work[tid * 33 + c] : 0.f;
        const int my_orig = own ? orig[k0 + tid] : 0;
        int pos = own ? tid : 0x7fffffff;
        // 2. factor it
#pragma unroll
        for (int j = 0; j < kLUNB; ++j) {
            if (j < nb && ok) {
                const int b = j & 1;
                const bool in = own && pos >= j;
                const float v = fabsf(a[j]);
                // a NaN never wins the search, as in a comparison
                const unsigned bits = in && v == v ? __float_as_uint(v) + 1u : 0u;  // 0: no candidate
                unsigned best = __reduce_max_sync(0xffffffffu, bits);
                int at = __reduce_min_sync(0xffffffffu, bits == best ? pos : 0x7fffffff);
                if (lane == 0) {
                    sh.key[b][warp] = best;
                    sh.pos[b][warp] = at;
                }
                __syncthreads();
                const unsigned kb = lane < nw ? sh.key[b][lane] : 0u;
                best = __reduce_max_sync(0xffffffffu, kb);
                at = __reduce_min_sync(0xffffffffu, kb == best && lane < nw ? sh.pos[b][lane] : 0x7fffffff);
                const float apv = __uint_as_float(best - 1u);
                if (best <= 1u || !(apv <= 3.402823466e38f)) {
                    ok = false;  // uniform: zero, infinite or no pivot
                } else {
                    fmin_p = fminf(fmin_p, apv);
                    fmax_p = fmaxf(fmax_p, apv);
                    if (pos == at) {  // the pivot row: publish it, and trade places with position j
#pragma unroll
                        for (int c = j; c < kLUNB; ++c) sh.prow[b][c] = a[c];
                        pos = j;
                    } else if (pos == j) {
                        pos = at;
                    }
                    __syncthreads();
                    if (own && pos > j) {
                        const float l = a[j] * (1.0f / sh.prow[b][j]);
                        a[j] = l;
#pragma unroll
                        for (int c = j + 1; c < kLUNB; ++c) a[c] = fmaf(-l, sh.prow[b][c], a[c]);
                    }
                }
            }
        }
        if (!ok) break;
        // 3. the factored panel back, rows in their new places; the permutation's entries
        __syncthreads();
        if (own) {
            orig[k0 + pos] = my_orig;
#pragma unroll
            for (int c = 0; c < kLUNB; ++c) work[pos * 33 + c] = a[c];
            if (pos < nb) {
                sh.src[pos] = k0 + tid;
                sh.dst[pos] = k0 + pos;
#pragma unroll
                for (int c = 0; c < kLUNB; ++c) sh.l11[c][pos] = a[c];
            }
        }
        if (tid == 0) sh.moved = kLUNB;
        __syncthreads();
        for (int r = warp; r < m; r += nw)
            if (lane < nb) A[(size_t)(k0 + r) * n1 + k0 + lane] = work[r * 33 + lane];
        if (own && pos >= nb && pos != tid) {
            const int e = atomicAdd(&sh.moved, 1);  // at most nb rows leave the top
            sh.src[e] = k0 + tid;
            sh.dst[e] = k0 + pos;
        }
        __syncthreads();
        // 4. the permutation on the other columns, through shared memory
        const int moved = sh.moved;
        for (int e = warp; e < moved; e += nw) {
            if (e >= nb && e < kLUNB) continue;
            const bool same = sh.src[e] == sh.dst[e];
            const float *row = A + (size_t)sh.src[e] * n1;
            for (int c = (same ? c1 : 0) + lane; c < n1; c += 32)
                if (c < k0 || c >= c1) S[(size_t)e * ld + c] = row[c];
        }
        __syncthreads();
        for (int e = warp; e < moved; e += nw) {
            if ((e >= nb && e < kLUNB) || sh.src[e] == sh.dst[e]) continue;
            float *row = A + (size_t)sh.dst[e] * n1;
            const int hi = e < kLUNB ? k0 : n1;  // the top rows' right part is U12, below
            for (int c = lane; c < hi; c += 32)
                if (c < k0 || c >= c1) row[c] = S[(size_t)e * ld + c];
        }
        if (c1 >= n1) break;
        __syncthreads();  // the displaced rows' copies are no longer needed: L21 takes their place
        if (own && pos >= nb)
#pragma unroll
            for (int j = 0; j < kLUNB; ++j) LT[(size_t)j * ld + pos - nb] = a[j];
        // 5. U12 = L11^-1 A12 (unit lower L11), a thread per column
        for (int c = c1 + tid; c < n1; c += nt) {
            float u[kLUNB];
#pragma unroll
            for (int j = 0; j < kLUNB; ++j) u[j] = j < nb ? S[(size_t)j * ld + c] : 0.f;
#pragma unroll
            for (int j = 0; j < kLUNB; ++j)
#pragma unroll
                for (int i = j + 1; i < kLUNB; ++i) u[i] = fmaf(-sh.l11[j][i], u[j], u[i]);
#pragma unroll
            for (int j = 0; j < kLUNB; ++j)
                if (j < nb) {
                    S[(size_t)j * ld + c] = u[j];
                    A[(size_t)(k0 + j) * n1 + c] = u[j];
                }
        }
        __syncthreads();
        // 6. A22 -= L21 U12
        const int mr = m - nb, mc = n1 - c1;
        const int tiles_r = (mr + 7) / 8, tiles_c = (mc + 127) / 128;
        for (int t = warp; t < tiles_r * tiles_c; t += nw) {
            const int tc = t / tiles_r, r = (t - tc * tiles_r) * 8, c = tc * 128;
            const float *l = LT + r, *u = S + c1 + c + lane;
            const int nc = min(128, mc - c), nr = min(8, mr - r), row = c1 + r, col = c1 + c + lane;
            if (nc > 96) lu_trailing_tile<4>(A, n1, l, u, nb, row, nr, col, nc, ld);
            else if (nc > 64) lu_trailing_tile<3>(A, n1, l, u, nb, row, nr, col, nc, ld);
            else if (nc > 32) lu_trailing_tile<2>(A, n1, l, u, nb, row, nr, col, nc, ld);
            else lu_trailing_tile<1>(A, n1, l, u, nb, row, nr, col, nc, ld);
        }
    }
    pmin = fmin(pmin, (double)fmin_p);
    pmax = fmax(pmax, (double)fmax_p);
    __syncthreads();
    return ok;
}

// x = K^-1 y in FP32 with the factors (unit lower L, upper U, both in LU; row i of the factors is
// row orig[i] of K), blocked by 32 columns: the 32x32 diagonal block (fetched to shared memory
// during the step before) is solved by one warp with shuffles, then every warp updates the
// remaining rows with the block's 32 values, four rows at a time (coalesced).  Two barriers
// per 32 columns.
__device__ void lu_apply_f32(const float *__restrict__ LU, const int *__restrict__ orig, int n1,
                             const float *__restrict__ y, float *__restrict__ x) {
    __shared__ float blk[2][32][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, nt = blockDim.x;
    auto fetch = [&](int b, int c0) {
        if (c0 < 0 || c0 >= n1) return;
        const int bs = min(32, n1 - c0);
        for (int t = threadIdx.x; t < bs * 32; t += nt) {
            const int r = t >> 5, c = t & 31;
            blk[b][r][c] = c < bs ? LU[(size_t)(c0 + r) * n1 + c0 + c] : 0.f;
        }
    };
    // rows r0 .. r1 - 1 less LU[r][c0 ..] times x[c0 .. c0 + bs - 1]: eight rows' products are summed
    // over the lanes together (each exchange halves the rows a lane keeps), each in the order of
    // a plain exchange by 16, 8, 4, 2, 1
    auto update = [&](int r0, int r1, int c0, int bs) {
        const float xv = lane < bs ? x[c0 + lane] : 0.f;
        const float *base = LU + c0 + lane;
        const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
        for (int r = r0 + 8 * warp; r < r1; r += 8 * nw) {
            float t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = (lane < bs && r + k < r1) ? base[(size_t)(r + k) * n1] : 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] *= xv;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float give = u16 ? t[k] : t[k + 4], keep = u16 ? t[k + 4] : t[k];
                t[k] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float give = u8 ? t[k] : t[k + 2], keep = u8 ? t[k + 2] : t[k];
                t[k] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
            float v = (u4 ? t[1] : t[0]) + __shfl_xor_sync(0xffffffffu, u4 ? t[0] : t[1], 4);
            for (int o = 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int row = r + (u16 ? 4 : 0) + (u8 ? 2 : 0) + (u4 ? 1 : 0);
            if ((lane & 3) == 0 && row < r1) x[row] -= v;
        }
    };
    // the diagonal block b: its rows' values ahead of the serial chain, in registers
    auto solve_lower = [&](int b, int c0, int bs) {
        if (bs < 32) {  // the short block at the end
            float v = lane < bs ? x[c0 + lane] : 0.f;
            for (int c = 0; c < bs - 1; ++c) {
                const float vc = __shfl_sync(0xffffffffu, v, c);
                if (lane > c && lane < bs) v -= blk[b][lane][c] * vc;
            }
            if (lane < bs) x[c0 + lane] = v;
            return;
        }
        float l[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) l[c] = blk[b][lane][c];
        float v = x[c0 + lane];
#pragma unroll
        for (int c = 0; c < 31; ++c) {
            const float vc = __shfl_sync(0xffffffffu, v, c);
            if (lane > c) v -= l[c] * vc;
        }
        x[c0 + lane] = v;
    };
    auto solve_upper = [&](int b, int c0, int bs) {
        if (bs < 32) {
            float v = lane < bs ? x[c0 + lane] : 0.f;
            for (int c = bs - 1; c >= 0; --c) {
                if (lane == c) v = v / blk[b][c][c];
                const float xc = __shfl_sync(0xffffffffu, v, c);
                if (lane < c) v -= blk[b][lane][c] * xc;
            }
            if (lane < bs) x[c0 + lane] = v;
            return;
        }
        float u[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) u[c] = blk[b][lane][c];
        const float dg = blk[b][lane][lane];
        float v = x[c0 + lane];
#pragma unroll
        for (int c = 31; c >= 0; --c) {
            if (lane == c) v = v / dg;
            const float xc = __shfl_sync(0xffffffffu, v, c);
            if (lane < c) v -= u[c] * xc;
        }
        x[c0 + lane] = v;
    };
    const int nblk = (n1 + 31) / 32;
    __syncthreads();
    fetch(0, 0);
    for (int t = threadIdx.x; t < n1; t += nt) x[t] = y[orig[t]];
    __syncthreads();
    for (int s = 0; s < nblk; ++s) {  // forward: L (unit diagonal)
        const int c0 = 32 * s, bs = min(32, n1 - c0);
        if (warp == 0) solve_lower(s & 1, c0, bs);
        if (s + 1 < nblk) fetch((s + 1) & 1, c0 + 32);
        __syncthreads();
        update(c0 + bs, n1, c0, bs);
        __syncthreads();
    }
    // backward: U; the blocks end at n1, n1 - 32, ... (the first one, at the top, may be short)
    fetch(0, max(0, n1 - 32));
    __syncthreads();
    for (int s = 0; s < nblk; ++s) {
        const int e = n1 - 32 * s, c0 = max(0, e - 32), bs = e - c0;
        if (warp == 0) solve_upper(s & 1, c0, bs);
        if (s + 1 < nblk) {
            const int e2 = e - 32, d0 = max(0, e2 - 32);
            for (int t = threadIdx.x; t < (e2 - d0) * 32; t += nt) {
                const int r = t >> 5, c = t & 31;
                blk[(s + 1) & 1][r][c] = c < e2 - d0 ? LU[(size_t)(d0 + r) * n1 + d0 + c] : 0.f;
            }
        }
        __syncthreads();
        update(0, c0, c0, bs);
        __syncthreads();
    }
}

// d.r <- K^{-1} d.r with the factors that solved the system: FP32 (in the first half of As,
// through the FP32 vectors ys/xs) or FP64 (in As, through y64).  Non-finite FP32 results (a system
// far beyond FP32) read as 1e300.
__device__ void apply_inverse(const SolveDesc &d, int n1, bool f32, float *ys, float *xs, const int *orig, double *y64) {
    if (f32) {
        __syncthreads();
        for (int t = threadIdx.x; t < n1; t += blockDim.x) ys[t] = (float)d.r[t];
        lu_apply_f32(reinterpret_cast<const float *>(d.As), orig, n1, ys, xs);
        for (int t = threadIdx.x; t < n1; t += blockDim.x) {
            const float v = xs[t];
            d.r[t] = isfinite(v) ? (double)v : 1e300;
        }
        __syncthreads();
    } else {
        lu_apply(d.As, d.perm, n1, d.r, y64);
        __syncthreads();
    }
}

// Estimate of ||K^{-1}||_1 for the symmetric bordered matrix K (so K^{-T} = K^{-1}):
// Hager's method (W. W. Hager, "Condition estimates", SIAM J. Sci. Stat. Comput. 5 (1984)
// 311-316) with Higham's extra test vector (N. J. Higham, ACM TOMS 14 (1988) 381-396),
// at most four sign iterations.  A lower bound that is almost always within a small factor.
// Uses d.r as the work vector.
__device__ double inverse_norm1_estimate(const SolveDesc &d, int n1, bool f32, float *ys, float *xs, const int *orig, double *y64,
                                         double *sv, int *si, double *piv_v, int *piv_i) {
    for (int t = threadIdx.x; t < n1; t += blockDim.x) d.r[t] = 1.0 / (double)n1;
    apply_inverse(d, n1, f32, ys, xs, orig, y64);
    double a = 0.0;
    for (int t = threadIdx.x; t < n1; t += blockDim.x) a += fabs(d.r[t]);
    double est = block_sum(a, n1, sv);
    int jprev = -1;
    for (int it = 0; it < 4; ++it) {
        for (int t = threadIdx.x; t < n1; t += blockDim.x) d.r[t] = d.r[t] >= 0.0 ? 1.0 : -1.0;
        apply_inverse(d, n1, f32, ys, xs, orig, y64);  // z = K^{-T} sign(y)
        double best = -1.0, zsum = 0.0;
        int bi = 0x7fffffff;
        for (int t = threadIdx.x; t < n1; t += blockDim.x) {
            const double v = fabs(d.r[t]);
            zsum += d.r[t];
            if (v > best || (v == best && t < bi)) { best = v; bi = t; }
        }
        zsum = block_sum(zsum, n1, sv);
        block_argmax(best, bi, sv, si, piv_v, piv_i);
        const double zmax = *piv_v;
        const int j = *piv_i;
        const double ztx = jprev < 0 ? zsum / (double)n1 : d.r[jprev];
        __syncthreads();
        if (!(zmax > ztx)) break;  // uniform: every thread read the same values
        for (int t = threadIdx.x; t < n1; t += blockDim.x) d.r[t] = t == j ? 1.0 : 0.0;
        apply_inverse(d, n1, f32, ys, xs, orig, y64);
        double b = 0.0;
        for (int t = threadIdx.x; t < n1; t += blockDim.x) b += fabs(d.r[t]);
        b = block_sum(b, n1, sv);
        if (!(b > est)) break;
        est = b;
        jprev = j;
    }
    for (int t = threadIdx.x; t < n1; t += blockDim.x)
        d.r[t] = ((t & 1) ? -1.0 : 1.0) * (1.0 + (double)t / (double)max(n1 - 1, 1));
    apply_inverse(d, n1, f32, ys, xs, orig, y64);
    double c = 0.0;
    for (int t = threadIdx.x; t < n1; t += blockDim.x) c += fabs(d.r[t]);
    c = 2.0 * block_sum(c, n1, sv) / (3.0 * (double)n1);
    est = fmax(est, c);
    return est < 1e300 ? est : 1e300;
}

constexpr int kRefineMax = 30;  // and stop early once a step no longer halves the residual
// systems factored across the GPU (FP32 first by our panels, the bound being the panel rows
// that fit shared memory at 4 columns; FP64 by cuSOLVER when the FP32 refinement does not
// converge): n1 in [kLUWideMin, kLUWideMax]
constexpr int kLUWideMin = 768;
// systems of kLUHost64Min to kLUWideMin unknowns are refined with the wide ones' rounds, and their FP64
// factors come from across the GPU too (an in-CTA FP64 LU of 425 unknowns takes ~13 ms on one SM's FP64
// pipe); their FP32 factors come from their CTA when a launch holds several
constexpr int kLUHost64Min = 256;
// least unknowns for two systems of a launch, or one beside smaller ones, to be factored across the GPU one after
// the other: 0.88 ms for two against 1.06 side by side in their CTAs at 521 unknowns, 0.70 against
// 0.69 at 421; and a system of 255 takes 0.69 ms in its CTA anyway
constexpr int kAcrossTwo = 512;
constexpr int kLUWideMax = (int)((225 * 1024) / (sizeof(float) * 5));

// r = bs - A0 x in FP64: a warp per eight rows, lanes along the row.  The rows' sums over the lanes
// are reduced together (each exchange halves the rows a lane keeps), in the order of a plain
// exchange by 16, 8, 4, 2, 1: 9 additions for 8 rows instead of 40 on the slow FP64 pipe.
__device__ void residual(const SolveDesc &d, int n1) {
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
    for (int r = 8 * (threadIdx.x >> 5); r < n1; r += 8 * (blockDim.x >> 5)) {
        double s[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = 0.0;
        const double *row = d.A0 + (size_t)r * n1;
        for (int c = lane; c < n1; c += 32) {
            const double xv = d.x[c];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (r + k < n1) s[k] += row[(size_t)k * n1 + c] * xv;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double give = u16 ? s[k] : s[k + 4], keep = u16 ? s[k + 4] : s[k];
            s[k] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double give = u8 ? s[k] : s[k + 2], keep = u8 ? s[k + 2] : s[k];
            s[k] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
        }
        double v = (u4 ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, u4 ? s[0] : s[1], 4);
        for (int o = 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int rr = r + (u16 ? 4 : 0) + (u8 ? 2 : 0) + (u4 ? 1 : 0);
        if ((lane & 3) == 0 && rr < n1) d.r[rr] = d.bs[rr] - v;
    }
    __syncthreads();
}

// BIG: a launch with a system beyond kLUWideMax, whose vectors do not fit shared memory: they follow the FP32
// factors in the work matrix (3 n1 of its n1^2 words there), or the FP64 solves run on the vector itself.
template <bool BIG>
__global__ void __launch_bounds__(kSolve) lu_solve_refine_kernel(const SolveDesc *__restrict__ descs) {
    const SolveDesc d = descs[blockIdx.x];
    if (d.wide64 || d.host32) return;  // factor_refine_wide64, refine_across
    const int n1 = d.n + 1;
    // [2 n1] right-hand side / correction in FP32 (or n1 doubles), [n1] row order, then the work
    // area of the blocked factorisation
    extern __shared__ __align__(16) float fsh[];
    const bool big = BIG && d.big;
    float *ys = big ? reinterpret_cast<float *>(d.As) + (size_t)n1 * n1 : fsh, *xs = ys + n1;
    int *orig = reinterpret_cast<int *>(xs + n1);
    __shared__ double sv[33];
    __shared__ int si[kLU / 32];
    __shared__ double piv_v;
    __shared__ int piv_i;
    __shared__ LuShared lus;
    double pmin = 1e308, pmax = 0.0, res = 0.0;
    int singular = 0, steps = 0;
    bool done = false;

    // ---- FP32 LU + FP64-residual refinement
    double an, anorm;  // max row sums of |K| and |A| (prepare_kernel)
    {
        double u = 0.0, v = 0.0;
        for (int t = threadIdx.x; t < n1; t += blockDim.x) {
            u = fmax(u, d.r[t]);
            v = fmax(v, d.x[t]);
        }
        an = block_max(u, n1, sv);
        anorm = block_max(v, n1, sv);
    }
    {
        float *L = reinterpret_cast<float *>(d.As);  // the first half of the FP64 work matrix (prepare_kernel's copy)
        for (int t = threadIdx.x; t < n1; t += blockDim.x) {
            d.x[t] = 0.0;
            d.r[t] = d.bs[t];
        }
        bool factored;
        if (d.across) {  // factored across the GPU before this launch
            factored = d.pre[0] == 0.0;
            pmin = d.pre[1];
            pmax = d.pre[2];
            for (int t = threadIdx.x; t < n1; t += blockDim.x) orig[t] = factored ? d.perm[t] : t;
            __syncthreads();
        } else if (n1 <= kLUBlockedMax && !big) {
            float *work = fsh + ((3 * n1 + 3) & ~3);
            factored = lu_factor_f32_blocked(L, orig, n1, work, lus, pmin, pmax);
            if (d.factor_only) {  // the rounds refine it
                for (int t = threadIdx.x; t < n1; t += blockDim.x) d.perm[t] = orig[t];
                if (threadIdx.x == 0) {
                    d.pre[0] = factored ? 0.0 : 1.0;
                    d.pre[1] = pmin;
                    d.pre[2] = pmax;
                }
                return;
            }
        } else {
            factored = lu_factor_f32(L, d.perm, n1, sv, si, &piv_v, &piv_i, pmin, pmax);
            if (threadIdx.x == 0) {  // the interchanges as a row order
                for (int k = 0; k < n1; ++k) orig[k] = k;
                for (int k = 0; factored && k < n1; ++k) {
                    const int p = d.perm[k], o = orig[k];
                    orig[k] = orig[p];
                    orig[p] = o;
                }
            }
            __syncthreads();
        }
        if (factored) {
            double rprev = 1e308;
            for (int it = 0; it < kRefineMax && !done; ++it) {
                double rm = 0.0;
                for (int t = threadIdx.x; t < n1; t += blockDim.x) rm = fmax(rm, fabs(d.r[t]));
                rm = block_max(rm, n1, sv);
                if (rm == 0.0) {
                    done = true;
                    break;
                }
                const double inv = 1.0 / rm;
                ++steps;
                for (int t = threadIdx.x; t < n1; t += blockDim.x) ys[t] = (float)(d.r[t] * inv);
                lu_apply_f32(L, orig, n1, ys, xs);
                for (int t = threadIdx.x; t < n1; t += blockDim.x) d.x[t] += (double)xs[t] * rm;
                __syncthreads();
                double rn = 0.0, xn = 0.0;
                residual(d, n1);
                for (int rr = threadIdx.x; rr < n1; rr += blockDim.x) {
                    rn = fmax(rn, fabs(d.r[rr]));
                    xn = fmax(xn, fabs(d.x[rr]));
                }
                rn = block_max(rn, n1, sv);
                xn = block_max(xn, n1, sv);
                res = rn;
                if (rn <= (double)n1 * 1.1102230246251565e-16 * an * xn) done = true;
                // stalled (cond(A) near 1/eps32 or beyond): no use refining further, FP64 takes over
                else if (it >= 2 && rn > 0.5 * rprev) break;
                rprev = rn;
            }
        }
        __syncthreads();
    }

    // A wide (or mid-size) system whose FP32 factors did not converge is factored in FP64 and
    // refined by the host path (factor_refine_wide64); nothing is written here.
    if (!done && d.pre) {
        if (threadIdx.x == 0) d.pre[0] = 2.0;
        return;
    }

    // ---- fallback: FP64 LU with one step of FP64 refinement
    const bool f32_solved = done;
    if (!done) {
        double *A = d.As;
        {
        for (long long t = threadIdx.x; t < (long long)n1 * n1; t += blockDim.x) A[t] = d.A0[t];
        __syncthreads();
        pmin = 1e308;
        pmax = 0.0;
        for (int k = 0; k < n1; ++k) {
            double best = -1.0;
            int bi = 0x7fffffff;
            for (int r = k + threadIdx.x; r < n1; r += blockDim.x) {
                double v = fabs(A[(size_t)r * n1 + k]);
                if (v > best || (v == best && r < bi)) { best = v; bi = r; }
            }
            block_argmax(best, bi, sv, si, &piv_v, &piv_i);
            const int p = piv_i < n1 ? piv_i : k;  // no candidate (NaN): stay
            if (threadIdx.x == 0) d.perm[k] = p;
            if (p != k)
                for (int c = threadIdx.x; c < n1; c += blockDim.x) {
                    double t = A[(size_t)k * n1 + c];
                    A[(size_t)k * n1 + c] = A[(size_t)p * n1 + c];
                    A[(size_t)p * n1 + c] = t;
                }
            __syncthreads();
            double pv = A[(size_t)k * n1 + k];
            double apv = fabs(pv);
            pmin = fmin(pmin, apv);
            pmax = fmax(pmax, apv);
            if (!(apv > 1e-300)) {  // exactly singular: keep going with a tiny pivot, flag it
                singular = 1;
                pv = (pv < 0 ? -1e-300 : 1e-300);
                if (threadIdx.x == 0) A[(size_t)k * n1 + k] = pv;
            }
            __syncthreads();
            const double inv = 1.0 / pv;
            for (int r = k + 1 + threadIdx.x; r < n1; r += blockDim.x) A[(size_t)r * n1 + k] *= inv;
            __syncthreads();
            const double *prow = A + (size_t)k * n1;
            for (int rr = k + 1 + (threadIdx.x >> 5); rr < n1; rr += (blockDim.x >> 5)) {
                double *row = A + (size_t)rr * n1;
                const double l = row[k];
                for (int cc = k + 1 + (threadIdx.x & 31); cc < n1; cc += 32) row[cc] -= l * prow[cc];
            }
            __syncthreads();
        }
        }
        for (int t = threadIdx.x; t < n1; t += blockDim.x) d.x[t] = d.bs[t];
        lu_apply(A, d.perm, n1, d.x, big ? d.x : reinterpret_cast<double *>(fsh));
        for (int rr = threadIdx.x; rr < n1; rr += blockDim.x) {
            double s = d.bs[rr];
            const double *row = d.A0 + (size_t)rr * n1;
            for (int c = 0; c < n1; ++c) s -= row[c] * d.x[c];
            d.r[rr] = s;
        }
        lu_apply(A, d.perm, n1, d.r, big ? d.r : reinterpret_cast<double *>(fsh));
        for (int t = threadIdx.x; t < n1; t += blockDim.x) d.x[t] += d.r[t];
        __syncthreads();
        double rmax = 0.0;
        for (int rr = threadIdx.x; rr < n1; rr += blockDim.x) {
            double s = d.bs[rr];
            const double *row = d.A0 + (size_t)rr * n1;
            for (int c = 0; c < n1; ++c) s -= row[c] * d.x[c];
            rmax = fmax(rmax, fabs(s));
        }
        res = block_max(rmax, n1, sv);
    }
    // ---- conditioning: kappa = ||A||_1 ||K^{-1}||_1 with A the folded normal matrix (RESP
    // included, the border excluded) and K the bordered matrix.  A relative error e in A moves
    // the solution by about e * kappa * |q| at worst, so kappa says how much of the Gram's
    // rounding reaches the charges (the fit escalates a mixed-precision cube beyond a limit).
    const double kinv = inverse_norm1_estimate(d, n1, f32_solved, ys, xs, orig, big ? d.r : reinterpret_cast<double *>(fsh), sv, si, &piv_v, &piv_i);
    if (threadIdx.x == 0) {
        d.info[0] = res;
        d.info[1] = pmin;
        d.info[2] = pmax;
        d.info[3] = singular;
        d.info[4] = fmin(anorm * kinv, 1e300);
        d.info[5] = n1;
        d.info[6] = steps;
        d.info[7] = f32_solved ? 0.0 : 2.0;
    }
    __syncthreads();
    // expand to all atoms
    for (int i = threadIdx.x; i < d.N; i += blockDim.x) d.q[i] = d.x[d.map[i]];
}

// ---------------------------------------------------------------------------
// FP32 factorisation of one system beyond kLUAcrossMax unknowns across the whole GPU, before its
// refinement.  One CTA factoring n1^3 / 3 FMAs alone is SM-bound (20 ms at n1 = 1456); here only the
// panels are serial.  A0 is copied into As in FP32, then per panel of nb columns (32, or 16 / 8 / 4
// when the panel's rows do not fit shared memory at 32):
//   lu_panel_kernel   one CTA: the panel in shared memory, factored with the partial pivoting
//                     of the one-CTA factorisations (perm[k] = pivot row, full-row swaps),
//                     written back, its swaps applied to every other column;
//   lu_trsm_kernel    U12 = L11^-1 A12, a thread per column over many CTAs;
//   cuBLAS SGEMM      A22 -= L21 U12 (a plain product).
// pre = {flag, min|pivot|, max|pivot|}: flag 1 = zero or non-finite pivot (the later panels return at
// once).  refine_across refines; refine_wide32 by substitution or factor_refine_wide64 in FP64 take
// over when it says so.
constexpr size_t kPanelSmem = 225 * 1024;

int wide_panel_nb(int m) {
    for (int nb = 32; nb >= 4; nb /= 2)
        if (sizeof(float) * (size_t)m * (nb + 1) <= kPanelSmem) return nb;
    return 0;
}

template <typename T>
__global__ void lu_copy_kernel(const double *__restrict__ A0, T *__restrict__ L, long long n,
                               double *__restrict__ pre) {
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long t = t0; t < n; t += (long long)gridDim.x * blockDim.x) L[t] = (T)A0[t];
    if (t0 == 0) {
        pre[0] = 0.0;
        pre[1] = 1e308;
        pre[2] = 0.0;
    }
}

__global__ void __launch_bounds__(kLU) lu_panel_kernel(float *__restrict__ A, int *__restrict__ perm, int n1, int k0,
                                                       int NB, double *__restrict__ pre) {
    if (pre[0] != 0.0) return;  // an earlier panel met a zero pivot
    extern __shared__ __align__(16) float P[];  // [m][NB + 1] panel rows k0..n1-1
    __shared__ double sv[kLU / 32];
    __shared__ int si[kLU / 32];
    __shared__ int piv_i;
    const int m = n1 - k0, nb = min(NB, m), ld = NB + 1;
    for (int t = threadIdx.x; t < m * NB; t += kLU) {
        const int r = t / NB, c = t - r * NB;
        P[r * ld + c] = c < nb ? A[(size_t)(k0 + r) * n1 + k0 + c] : 0.f;
    }
    __syncthreads();
    double pmin_l = 1e308, pmax_l = 0.0;
    for (int j = 0; j < nb; ++j) {
        float best = -1.f;
        int bi = 0x7fffffff;
        for (int r = j + threadIdx.x; r < m; r += kLU) {
            const float v = fabsf(P[r * ld + j]);
            if (v > best || (v == best && r < bi)) { best = v; bi = r; }
        }
        block_argmax_f(best, bi, reinterpret_cast<float *>(sv), si, &piv_i);
        const int p = piv_i < m ? piv_i : j;  // no candidate (NaN): stay
        if (threadIdx.x == 0) perm[k0 + j] = k0 + p;
        if (p != j && threadIdx.x < NB) {
            const float t = P[j * ld + threadIdx.x];
            P[j * ld + threadIdx.x] = P[p * ld + threadIdx.x];
            P[p * ld + threadIdx.x] = t;
        }
        __syncthreads();
        const float pv = P[j * ld + j], apv = fabsf(pv);
        if (!(apv > 0.f) || !isfinite(pv)) {  // uniform: every thread read the same pivot
            if (threadIdx.x == 0) pre[0] = 1.0;
            return;
        }
        pmin_l = fmin(pmin_l, (double)apv);
        pmax_l = fmax(pmax_l, (double)apv);
        const float inv = 1.f / pv;
        const float *pj = P + j * ld;
        for (int r = j + 1 + threadIdx.x; r < m; r += kLU) {  // a thread per row
            float *row = P + r * ld;
            const float l = row[j] * inv;
            row[j] = l;
            for (int c = j + 1; c < nb; ++c) row[c] -= l * pj[c];
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < m * NB; t += kLU) {
        const int r = t / NB, c = t - r * NB;
        if (c < nb) A[(size_t)(k0 + r) * n1 + k0 + c] = P[r * ld + c];
    }
    for (int c = threadIdx.x; c < n1; c += kLU) {
        if (c >= k0 && c < k0 + nb) continue;
        for (int j = 0; j < nb; ++j) {
            const int p = perm[k0 + j];
            if (p != k0 + j) {
                const float t = A[(size_t)(k0 + j) * n1 + c];
                A[(size_t)(k0 + j) * n1 + c] = A[(size_t)p * n1 + c];
                A[(size_t)p * n1 + c] = t;
            }
        }
    }
    if (threadIdx.x == 0) {
        pre[1] = fmin(pre[1], pmin_l);
        pre[2] = fmax(pre[2], pmax_l);
    }
}

template <int NB>
__global__ void __launch_bounds__(256) lu_trsm_kernel(float *__restrict__ A, int n1, int k0,
                                                      const double *__restrict__ pre) {
    if (pre[0] != 0.0) return;
    __shared__ float Ls[NB][NB + 1];
    const int nb = min(NB, n1 - k0), c1 = k0 + nb;
    for (int t = threadIdx.x; t < NB * NB; t += blockDim.x) {
        const int i = t / NB, j = t - i * NB;
        Ls[i][j] = (i < nb && j < nb) ? A[(size_t)(k0 + i) * n1 + k0 + j] : 0.f;
    }
    __syncthreads();
    const int c = c1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n1) return;
    float u[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) u[j] = j < nb ? A[(size_t)(k0 + j) * n1 + c] : 0.f;
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int i = j + 1; i < NB; ++i) u[i] -= Ls[i][j] * u[j];
#pragma unroll
    for (int j = 0; j < NB; ++j)
        if (j < nb) A[(size_t)(k0 + j) * n1 + c] = u[j];
}

// ---------------------------------------------------------------------------
// FP32 factorisation of one system across the whole GPU, for systems of kLUHost64Min unknowns (where
// one CTA's n1^3 / 3 multiply-adds are SM-bound) to kLUAcrossMax.  Per panel of NB columns:
//   lu_panel_across_kernel<R>  one CTA: the panel's rows in registers (R rows of NB = 64 / R columns
//                    per thread, so up to 512 R rows), one barrier per column.  It writes the panel's rows in their new order
//                    (LP, for the update), each row to the factors' row of its input row's number
//                    (F), and the order itself: no row ever moves.
//   lu_update_across_kernel   64 x 64 tiles over the GPU: U12 = L11^-1 A12 of the tile's columns
//                    (by every tile of a column, cheaper than another launch), then
//                    A22 -= L21 U12 in place, the rows taken in the new order; the pivot rows,
//                    which every tile of a column reads, are not written again.
// lu_collect_kernel gathers F's rows into the final order.  d.perm receives that order (row i of
// the factors is row perm[i] of the input); pre = {flag, min|pivot|, max|pivot|}, flag 1 = zero or
// non-finite pivot (the later launches return at once).
// Bounded by the panels' chain of latencies, about 1200 cycles per column (search, publish, pick,
// update) and 5 us per panel of loads and stores; an update of 2001 x 2001 takes 8 us.  Two barriers
// per column took 5 % longer; eight columns at a time and panels wholly in line (their instruction
// fetch costs as much) were no faster.  Measured: 7.8 -> 3.05 ms at 2001 unknowns, 2.3 -> 0.67 at 768, 3.6 -> 1.2 at
// 1101 (against panels in shared memory with four barriers per column, interchanges on one CTA
// and a cuBLAS rank-32 update).
constexpr int kLUAcrossMax = 4096;
constexpr int kPanelT = 512;  // threads of a panel: R rows each, 64 values in registers
struct LuStep {
    float *A;          // the matrix, updated in place: row id stays where it is
    float *F;          // factors by input row
    float *LP;         // [rows from k0][32] the panel in its new order
    const int *id_o;   // position -> input row, before this panel
    int *id_n;         // and after it
    int *orig;         // final order
    double *pre;
    int n1, k0, nb;
};
//   The column loop is not unrolled (a whole panel in line is 60 KB of instructions run once, and
//   their fetch took 0.7 us per column): column j is always register 0, and the update that
//   leaves a row shifts it by one.  What is final of a row goes to shared memory on the way.
// Launches of one factorisation or refinement overlap their start-up with the end of the kernel before
// (programmatic dependent launch): each lets its successor begin when all its CTAs run, and waits
// for its predecessor's end, and so for all before it, ahead of its first access to memory.
// (A factorisation is two short launches per panel: 3.5 -> 3.1 ms at 2001 unknowns, 0.44 -> 0.38 at 425.)
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
void launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    RP_CUDA(cudaLaunchKernelEx(&c, kernel, P(args)...));
    RP_LAUNCH_CHECK();
}

template <int R>
__global__ void __launch_bounds__(kPanelT) lu_panel_across_kernel(LuStep p) {
    constexpr int NB = 64 / R, LD = NB + 1;
    extern __shared__ __align__(16) float pst[];  // [m][LD] the panel's rows, then their positions and input rows
    __shared__ unsigned key[2][16];  // each warp's candidate: its value, position, row of pst ...
    __shared__ int at_[2][16], row_[2][16];
    __shared__ __align__(16) float cand[2][16][NB + 4];  // ... and its row from this column on, 1 / pivot for the pivot, which is at NB
    const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    const int n1 = p.n1, k0 = p.k0, nb = p.nb, m = n1 - k0;
    int *posr = reinterpret_cast<int *>(pst + (size_t)m * LD), *ids = posr + m;
    chain_begin();
    if (k0 > 0 && p.pre[0] != 0.0) return;  // an earlier panel met a zero pivot
    const int sc = lane % NB, sr = warp * (32 / NB) + lane / NB, sn = nw * (32 / NB);  // staging: column, first row, step
    constexpr int RB = 32 / NB;  // rows of a staging step; a lane holds the input row of NB steps ahead
    int idl[64 / NB];
#pragma unroll
    for (int h = 0; h < 64 / NB; ++h) {
        const int r = warp * RB + lane % RB + (h * NB + lane / RB) * sn;
        idl[h] = r < m ? p.id_o[k0 + r] : 0;
    }
#pragma unroll
    for (int h = 0; h < 64 / NB; ++h) {
        const int own = warp * RB + lane % RB + (h * NB + lane / RB) * sn;
        if (own < m) ids[own] = idl[h];
        for (int it = 0; it < NB && warp * RB + (h * NB + it) * sn < m; ++it) {
            const int id = __shfl_sync(0xffffffffu, idl[h], it * RB + lane / NB), r = sr + (h * NB + it) * sn;
            if (r < m && sc < nb)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(pst + r * LD + sc)),
                             "l"(p.A + (size_t)id * n1 + k0 + sc) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    int pos[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int t = tid + q * nt;
        pos[q] = t < m ? t : -1;  // -1: no row
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float a[R][NB];
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
        for (int c = 0; c < NB; ++c) a[q][c] = pos[q] >= 0 && c < nb ? pst[pos[q] * LD + c] : 0.f;
    float pmin = 3.0e38f, pmax = 0.f;
    bool ok = true;
#pragma unroll
    for (int seg = 0; seg < NB / 8; ++seg) {
        const int W = NB - 8 * seg;  // live columns at the segment's start: registers 0 .. W-1
#pragma unroll 1
        for (int j = 8 * seg; j < min(8 * seg + 8, nb) && ok; ++j) {
            const int b = j & 1;
            unsigned bits = 0u;  // 0: no candidate; a NaN never wins
            int at = 0x7fffffff;
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const float v = fabsf(a[q][0]);
                const unsigned u = pos[q] >= j && v == v ? __float_as_uint(v) + 1u : 0u;
                if (u > bits || (u == bits && u != 0u && pos[q] < at)) {
                    bits = u;
                    at = pos[q];
                }
            }
            unsigned best = __reduce_max_sync(0xffffffffu, bits);
            unsigned who = __ballot_sync(0xffffffffu, bits == best);
            bool mine = bits == best;
            if (__popc(who) != 1) {  // ties: the lowest position
                const int low = __reduce_min_sync(0xffffffffu, mine ? at : 0x7fffffff);
                mine = mine && at == low;
            }
            if (mine) {  // (with no candidate, any of the lanes: at is the same)
                key[b][warp] = best;
                at_[b][warp] = at;
#pragma unroll
                for (int q = 0; q < R; ++q)
                    if (pos[q] == at) {
                        float *to = cand[b][warp];
#pragma unroll
                        for (int c = 4; c < W; c += 4)
                            *reinterpret_cast<float4 *>(to + c) = make_float4(a[q][c], a[q][c + 1], a[q][c + 2], a[q][c + 3]);
                        *reinterpret_cast<float4 *>(to) = make_float4(1.0f / a[q][0], a[q][1], a[q][2], a[q][3]);
                        to[NB] = a[q][0];
                        row_[b][warp] = tid + q * nt;
                    }
            }
            __syncthreads();
            const unsigned kb = lane < nw ? key[b][lane] : 0u;
            best = __reduce_max_sync(0xffffffffu, kb);
            who = __ballot_sync(0xffffffffu, kb == best);
            const float apv = __uint_as_float(best - 1u);
            if (best <= 1u || !(apv <= 3.402823466e38f)) {
                ok = false;  // uniform: zero, infinite or no pivot
                break;
            }
            if (__popc(who) != 1) {
                const int ka = kb == best ? at_[b][lane] : 0x7fffffff;  // (best > 1: such lanes are below nw)
                const int low = __reduce_min_sync(0xffffffffu, ka);
                who = __ballot_sync(0xffffffffu, ka == low);
            }
            const int w = __ffs(who) - 1;
            const float *prow = cand[b][w];
            at = at_[b][w];
            pmin = fminf(pmin, apv);
            pmax = fmaxf(pmax, apv);
            float4 pv[NB / 4];  // the pivot row, by vector loads (word by word: 3.1 ms at 2001 unknowns)
#pragma unroll
            for (int c = 0; c < W / 4; ++c) pv[c] = reinterpret_cast<const float4 *>(prow)[c];
            const float inv = pv[0].x;
            float l[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                l[q] = a[q][0] * inv;
                if (pos[q] == at) pos[q] = j;  // the pivot row and position j trade places
                else if (pos[q] == j) pos[q] = at;
                if (pos[q] > j) pst[(tid + q * nt) * LD + j] = l[q];
            }
#pragma unroll
            for (int c = 1; c < W; ++c) {  // (rows that are done take part: nothing reads them again)
                const float4 &v4 = pv[c / 4];
                const float pc = c % 4 == 0 ? v4.x : c % 4 == 1 ? v4.y : c % 4 == 2 ? v4.z : v4.w;
#pragma unroll
                for (int q = 0; q < R; ++q) a[q][c - 1] = fmaf(-l[q], pc, a[q][c]);
            }
            if (warp == j % nw && lane < NB - j) pst[row_[b][w] * LD + j + lane] = prow[lane ? lane : NB];
        }
    }
    if (!ok) {
        if (tid == 0) p.pre[0] = 1.0;
        return;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        if (pos[q] < 0) continue;
        const int t = tid + q * nt, id = ids[t];
        posr[t] = pos[q];
        p.id_n[k0 + pos[q]] = id;
        if (pos[q] < nb) p.orig[k0 + pos[q]] = id;
    }
    if (tid == 0) {
        p.pre[1] = k0 == 0 ? (double)pmin : fmin(p.pre[1], (double)pmin);
        p.pre[2] = k0 == 0 ? (double)pmax : fmax(p.pre[2], (double)pmax);
    }
    __syncthreads();
    if (sc < nb)
#pragma unroll 8
        for (int r = sr; r < m; r += sn) {
            const float v = pst[r * LD + sc];
            p.LP[(size_t)posr[r] * 32 + sc] = v;
            p.F[(size_t)ids[r] * n1 + k0 + sc] = v;
        }
}

constexpr int kUpd = 64;  // tile edge of the update
// SUM: the 32 products are summed and subtracted once, as a matrix product rounds (the wide
// systems); otherwise subtracted one by one, as the factorisation in one CTA rounds.
template <bool SUM>
__global__ void __launch_bounds__(256, 3) lu_update_across_kernel(LuStep p) {
    __shared__ __align__(16) float lt[kLUNB][kUpd + 4];    // L21 of the tile's rows, by columns
    __shared__ __align__(16) float l11[kLUNB][kLUNB + 4];  // L11 by columns
    __shared__ float u[kLUNB][kUpd];
    const int n1 = p.n1, k0 = p.k0, nb = p.nb, c1 = k0 + nb;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r0 = c1 + blockIdx.y * kUpd, q0 = c1 + blockIdx.x * kUpd;  // the tile's rows and columns
    const int tr = (tid >> 4) * 4, tc = tid & 15;  // rows tr .. tr+3, columns tc + 16 i
    chain_begin();
    const double flag = p.pre[0];
    const int top = lane < nb ? p.orig[k0 + lane] : 0;
    int fr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) fr[k] = p.id_n[min(r0 + tr + k, n1 - 1)];
#pragma unroll
    for (int t = tid; t < kLUNB * kLUNB; t += 256) {
        const int i = t >> 5, j = t & 31;
        l11[j][i] = i < nb && j < nb ? p.LP[(size_t)i * 32 + j] : 0.f;
    }
#pragma unroll
    for (int r = warp; r < kUpd; r += 8) lt[lane][r] = r0 + r < n1 && lane < nb ? p.LP[(size_t)(r0 + r - k0) * 32 + lane] : 0.f;
    if (flag != 0.0) return;  // (the row order is whole only after a whole panel)
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const int j = warp + 8 * h;
        const float *row = p.A + (size_t)__shfl_sync(0xffffffffu, top, j) * n1 + q0;
        u[j][lane] = j < nb && q0 + lane < n1 ? row[lane] : 0.f;
        u[j][lane + 32] = j < nb && q0 + lane + 32 < n1 ? row[lane + 32] : 0.f;
    }
    __syncthreads();
    // the tile's own values are in flight while U12 is formed
    float old[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float *row = p.A + (size_t)fr[k] * n1 + q0;
#pragma unroll
        for (int i = 0; i < 4; ++i) old[k][i] = r0 + tr + k < n1 && q0 + tc + 16 * i < n1 ? row[tc + 16 * i] : 0.f;
    }
    if (tid < kUpd) {  // U12 = L11^-1 A12 (unit lower L11), a thread per column
        float v[kLUNB];
#pragma unroll
        for (int j = 0; j < kLUNB; ++j) v[j] = u[j][tid];
#pragma unroll
        for (int j = 0; j < kLUNB; ++j)
#pragma unroll
            for (int i = j + 1; i < kLUNB; ++i) v[i] = fmaf(-l11[j][i], v[j], v[i]);
#pragma unroll
        for (int j = 0; j < kLUNB; ++j) u[j][tid] = v[j];
    }
    __syncthreads();
    if (blockIdx.y == 0)
        for (int j = warp; j < nb; j += 8) {
            float *row = p.F + (size_t)p.orig[k0 + j] * n1;
            for (int c = lane; c < kUpd && q0 + c < n1; c += 32) row[q0 + c] = u[j][c];
        }
    float acc[4][4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[k][i] = SUM ? 0.f : old[k][i];
#pragma unroll 4
    for (int j = 0; j < nb; ++j) {
        const float4 l4 = *reinterpret_cast<const float4 *>(&lt[j][tr]);
        const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float w = u[j][tc + 16 * i];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k][i] = fmaf(SUM ? l[k] : -l[k], w, acc[k][i]);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = r0 + tr + k, c = q0 + tc + 16 * i;
            if (r < n1 && c < n1) p.A[(size_t)fr[k] * n1 + c] = SUM ? old[k][i] - acc[k][i] : acc[k][i];
        }
}

__global__ void lu_collect_kernel(const float *__restrict__ F, const int *__restrict__ orig, int n1,
                                  const double *__restrict__ pre, float *__restrict__ LU) {
    chain_begin();
    if (pre[0] != 0.0) return;
    const int i = blockIdx.x;
    const float *src = F + (size_t)orig[i] * n1;
    for (int c = threadIdx.x; c < n1; c += blockDim.x) LU[(size_t)i * n1 + c] = src[c];
}
__global__ void iota_kernel(int *__restrict__ v, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) v[t] = t;
}

// The FP32 matrix is in the first half of d.As; the second half takes the factors by input row.  (A buffer of
// n1^2 floats more, so that rows can move with their positions, was up to 5 % faster (2.9 against 3.05 ms at
// 2001 unknowns), but a system would then be factored one way or another by what the scratch budget
// has left.)
void lu_factor_across(rp_ctx *ctx, const SolveDesc &d, int n1, const std::string &tag, cudaStream_t stream) {
    LuStep p{};
    p.A = reinterpret_cast<float *>(d.As);
    p.F = p.A + (size_t)n1 * n1;
    p.LP = ctx->buf_t<float>("s_luLP" + tag, (size_t)n1 * 32);
    int *idx = ctx->buf_t<int>("s_luidx" + tag, 2 * (size_t)n1);  // the rows' order, two generations
    p.orig = d.perm;
    p.pre = d.pre;
    p.n1 = n1;
    iota_kernel<<<ceil_div(n1, 256), 256, 0, stream>>>(idx, n1);
    RP_LAUNCH_CHECK();
    const size_t most = sizeof(float) * 4096 * 11;  // (8 columns of 4096 rows; 16 of 2048 and 32 of 1024 take less)
    smem_optin((const void *)lu_panel_across_kernel<2>, most);
    smem_optin((const void *)lu_panel_across_kernel<4>, most);
    smem_optin((const void *)lu_panel_across_kernel<8>, most);
    int step = 0;
    for (int k0 = 0; k0 < n1; ++step) {
        const int m = n1 - k0, R = m <= 2 * kPanelT ? 2 : m <= 4 * kPanelT ? 4 : 8, NB = 64 / R;
        p.id_o = idx + (size_t)(step & 1) * n1;
        p.id_n = idx + (size_t)((step + 1) & 1) * n1;
        p.k0 = k0;
        p.nb = std::min(NB, m);
        const int nt = (int)ceil_div(ceil_div(m, R), 32) * 32;
        const size_t smem = sizeof(float) * (size_t)m * (NB + 3);
        launch_chained(R == 2 ? lu_panel_across_kernel<2> : R == 4 ? lu_panel_across_kernel<4> : lu_panel_across_kernel<8>, dim3(1), nt, smem,
                       stream, p);
        k0 += p.nb;
        if (k0 < n1) {
            const unsigned t = ceil_div(n1 - k0, kUpd);
            launch_chained(n1 >= kLUWideMin ? lu_update_across_kernel<true> : lu_update_across_kernel<false>, dim3(t, t), 256, 0, stream, p);
        }
    }
    launch_chained(lu_collect_kernel, dim3(n1), 256, 0, stream, p.F, d.perm, n1, d.pre, p.A);
}

// dynamic shared memory of lu_solve_refine_kernel: the right-hand side, the correction and the row
// order, and for the blocked factorisation 64 rows of a panel's neighbours (or its own rows,
// 33 floats each); none beyond kLUWideMax (BIG)
size_t solve_smem_bytes(int n1, bool big = false) {
    if (big) return 0;
    size_t f = (3 * (size_t)n1 + 3) & ~(size_t)3;
    if (n1 <= kLUBlockedMax) f += 64 * (((size_t)n1 + 3) & ~(size_t)3);
    return sizeof(float) * f;
}
// threads: at least a row each for the blocked factorisation; 24 warps from 100 unknowns on (0.33
// against 0.38 ms at 151 unknowns, 1.37 against 1.48 at 425), 8 below (fewer to a barrier: 0.06
// against 0.09 ms at 10)
int solve_threads(int n1) { return n1 <= 100 ? 256 : kSolve; }

// the launch's shared memory opt-in, raised once to the largest the kernel is launched with
void lu_smem_optin() {
    smem_optin((const void *)lu_solve_refine_kernel<false>, solve_smem_bytes(kLUWideMin - 1));
    smem_optin((const void *)lu_solve_refine_kernel<true>, solve_smem_bytes(kLUWideMin - 1));
}

// ---- FP64 wide factorisation by cuSOLVER's getrf
// The bordered matrix K is symmetric, so its row-major image is also K read column-major and
// cuSOLVER's getrf factors it in place (P K = L U, column-major), with its panels across the
// GPU instead of in one CTA each (an FP64 panel of 1851 x 32 costs ~0.25 ms on one SM's FP64
// pipe).  The refinement's residuals use A0 itself, so a Gram that is symmetric only to
// rounding costs nothing.
// pivot rows to 0-based interchanges, the pivots' range, and an exactly zero pivot replaced by
// 1e-300 and flagged (the in-CTA FP64 factorisation's rule); one CTA
__global__ void __launch_bounds__(1024) getrf_finish_kernel(double *__restrict__ LU, int n,
                                                            const int *__restrict__ ipiv, int *__restrict__ perm,
                                                            double *__restrict__ pre) {
    __shared__ double smin[32], smax[32];
    __shared__ int ssing[32];
    double mn = 1e308, mx = 0.0;
    int sing = 0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        perm[k] = ipiv[k] - 1;
        double *dk = LU + (size_t)k * n + k;
        const double a = fabs(*dk);
        if (!(a > 1e-300)) {
            sing = 1;
            *dk = (*dk < 0.0) ? -1e-300 : 1e-300;
        }
        mn = fmin(mn, a);
        mx = fmax(mx, a);
    }
    for (int o = 16; o > 0; o >>= 1) {
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sing |= __shfl_xor_sync(0xffffffffu, sing, o);
    }
    if ((threadIdx.x & 31) == 0) {
        smin[threadIdx.x >> 5] = mn;
        smax[threadIdx.x >> 5] = mx;
        ssing[threadIdx.x >> 5] = sing;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            mn = fmin(mn, smin[w]);
            mx = fmax(mx, smax[w]);
            sing |= ssing[w];
        }
        pre[0] = sing ? 1.0 : 0.0;
        pre[1] = mn;
        pre[2] = mx;
    }
}

// vectors of the refinement and of Hager's estimate: mode 0 fills 1/n, 1 takes the signs of v,
// 2 the unit vector e_j, 3 Higham's alternating vector (-1)^t (1 + t/(n-1)), 4 ones
__global__ void vec_fill_kernel(double *__restrict__ v, int n, int mode, int j) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    if (mode == 0) v[t] = 1.0 / (double)n;
    else if (mode == 1) v[t] = v[t] >= 0.0 ? 1.0 : -1.0;
    else if (mode == 2) v[t] = t == j ? 1.0 : 0.0;
    else if (mode == 3) v[t] = ((t & 1) ? -1.0 : 1.0) * (1.0 + (double)t / (double)max(n - 1, 1));
    else v[t] = 1.0;
}

// ||A||_1 of the folded normal matrix (the first n rows and columns of the bordered A0)
__global__ void anorm1_kernel(const double *__restrict__ A0, int n, int n1, unsigned long long *__restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double s = 0.0;
    for (int r = 0; r < n; ++r) s += fabs(A0[(size_t)r * n1 + c]);
    atomicMax(out, (unsigned long long)__double_as_longlong(s));  // s >= 0: bits order like values
}

__global__ void expand_kernel(const double *__restrict__ x, const int *__restrict__ map, int N, double *__restrict__ q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) q[i] = x[map[i]];
}

// A system whose FP32 refinement cannot converge (or an escalated fit's, at once): FP64 factors
// from cuSOLVER's getrf (K is symmetric, so its row-major image read column-major is K itself),
// one step of FP64 refinement, the residual and Hager's estimate of ||K^-1||_1 (the same steps
// and vectors as lu_solve_refine_kernel's, with getrs solves and cuBLAS reductions across the
// GPU instead of triangular solves in one CTA), then the info words and the charges.  Waits.
void factor_refine_wide64(rp_ctx *ctx, const SolveDesc &d, int n1, cudaStream_t stream) {
    double *LU = d.As;
    const long long nn = (long long)n1 * n1;
    {
        StageTimer tt(ctx, "solve_lu_wide64", stream);
        lu_copy_kernel<double><<<(int)std::min<long long>(ceil_div(nn, 256), 4096), 256, 0, stream>>>(d.A0, LU, nn,
                                                                                                        d.pre);
        RP_LAUNCH_CHECK();
    }
    cusolverDnHandle_t hs = ctx->solver();
    if (cusolverDnSetStream(hs, stream) != CUSOLVER_STATUS_SUCCESS) fail(RP_E_CUDA, "cusolverDnSetStream failed");
    cublasHandle_t hb = ctx->blas();
    RP_CUBLAS(cublasSetStream(hb, stream));
    int lwork = 0;
    if (cusolverDnDgetrf_bufferSize(hs, n1, n1, LU, n1, &lwork) != CUSOLVER_STATUS_SUCCESS)
        fail(RP_E_CUDA, "cusolverDnDgetrf_bufferSize failed");
    double *work = ctx->buf_t<double>("s_getrf_work", (size_t)std::max(lwork, 1));
    int *ipiv = ctx->buf_t<int>("s_getrf_ipiv", (size_t)n1 + 1);  // [n1] pivots, then the info word
    unsigned long long *anorm_bits = ctx->buf_t<unsigned long long>("s_anorm", 1);
    {
        StageTimer tt(ctx, "solve_lu_wide64", stream);
        if (cusolverDnDgetrf(hs, n1, n1, LU, n1, work, ipiv, ipiv + n1) != CUSOLVER_STATUS_SUCCESS)
            fail(RP_E_CUDA, "cusolverDnDgetrf failed");
        getrf_finish_kernel<<<1, 1024, 0, stream>>>(LU, n1, ipiv, d.perm, d.pre);
        RP_LAUNCH_CHECK();
    }
    StageTimer tt(ctx, "solve_refine64", stream);
    auto solve = [&](double *v) {
        if (cusolverDnDgetrs(hs, CUBLAS_OP_N, n1, 1, LU, n1, ipiv, v, n1, ipiv + n1) != CUSOLVER_STATUS_SUCCESS)
            fail(RP_E_CUDA, "cusolverDnDgetrs failed");
    };
    const double one = 1.0, minus_one = -1.0;
    auto residual = [&]() {  // r = bs - A0 x (A0 row-major: its transpose in cuBLAS's terms)
        RP_CUDA(cudaMemcpyAsync(d.r, d.bs, sizeof(double) * n1, cudaMemcpyDeviceToDevice, stream));
        RP_CUBLAS(cublasDgemv(hb, CUBLAS_OP_T, n1, n1, &minus_one, d.A0, n1, d.x, 1, &one, d.r, 1));
    };
    const int nb = (int)ceil_div(n1, 256);
    RP_CUDA(cudaMemcpyAsync(d.x, d.bs, sizeof(double) * n1, cudaMemcpyDeviceToDevice, stream));
    solve(d.x);
    residual();
    solve(d.r);
    RP_CUBLAS(cublasDaxpy(hb, n1, &one, d.r, 1, d.x, 1));
    residual();
    int im = 0;
    RP_CUBLAS(cublasIdamax(hb, n1, d.r, 1, &im));  // 1-based
    double res = 0.0, pre[3];
    RP_CUDA(cudaMemcpyAsync(&res, d.r + (im - 1), sizeof(double), cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaMemcpyAsync(pre, d.pre, sizeof(pre), cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaMemsetAsync(anorm_bits, 0, sizeof(unsigned long long), stream));
    anorm1_kernel<<<(int)ceil_div(std::max(d.n, 1), 256), 256, 0, stream>>>(d.A0, d.n, n1, anorm_bits);
    RP_LAUNCH_CHECK();
    unsigned long long abits = 0;
    RP_CUDA(cudaMemcpyAsync(&abits, anorm_bits, sizeof(abits), cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaStreamSynchronize(stream));
    res = std::fabs(res);
    double anorm;
    std::memcpy(&anorm, &abits, sizeof(anorm));
    // Hager's estimate of ||K^-1||_1 (K symmetric: K^-T = K^-1), on d.r
    auto asum = [&]() {
        double v = 0.0;
        RP_CUBLAS(cublasDasum(hb, n1, d.r, 1, &v));
        return v;
    };
    double *ones = ctx->buf_t<double>("s_ones", (size_t)n1);
    vec_fill_kernel<<<nb, 256, 0, stream>>>(ones, n1, 4, 0);
    vec_fill_kernel<<<nb, 256, 0, stream>>>(d.r, n1, 0, 0);
    solve(d.r);
    double est = asum();
    int jprev = -1;
    for (int it = 0; it < 4; ++it) {
        vec_fill_kernel<<<nb, 256, 0, stream>>>(d.r, n1, 1, 0);
        solve(d.r);
        int jm = 0;
        RP_CUBLAS(cublasIdamax(hb, n1, d.r, 1, &jm));
        const int j = jm - 1;
        double zj = 0.0, ztx = 0.0;
        RP_CUDA(cudaMemcpyAsync(&zj, d.r + j, sizeof(double), cudaMemcpyDeviceToHost, stream));
        if (jprev >= 0) RP_CUDA(cudaMemcpyAsync(&ztx, d.r + jprev, sizeof(double), cudaMemcpyDeviceToHost, stream));
        double zsum = 0.0;
        RP_CUBLAS(cublasDdot(hb, n1, d.r, 1, ones, 1, &zsum));
        RP_CUDA(cudaStreamSynchronize(stream));
        if (jprev < 0) ztx = zsum / (double)n1;
        if (!(std::fabs(zj) > ztx)) break;
        vec_fill_kernel<<<nb, 256, 0, stream>>>(d.r, n1, 2, j);
        solve(d.r);
        const double bval = asum();
        if (!(bval > est)) break;
        est = bval;
        jprev = j;
    }
    vec_fill_kernel<<<nb, 256, 0, stream>>>(d.r, n1, 3, 0);
    solve(d.r);
    est = std::max(est, 2.0 * asum() / (3.0 * (double)n1));
    const double kinv = est < 1e300 ? est : 1e300;
    double *hinfo = static_cast<double *>(ctx->host_buf("s_info64", sizeof(double) * kSolveInfo));
    hinfo[0] = res;
    hinfo[1] = pre[1];
    hinfo[2] = pre[2];
    hinfo[3] = pre[0];
    hinfo[4] = std::fmin(anorm * kinv, 1e300);
    hinfo[5] = n1;
    hinfo[6] = 1;
    hinfo[7] = 3.0;  // FP64 factors from across the GPU
    RP_CUDA(cudaMemcpyAsync(d.info, hinfo, sizeof(double) * kSolveInfo, cudaMemcpyHostToDevice, stream));
    expand_kernel<<<(int)ceil_div(d.N, 256), 256, 0, stream>>>(d.x, d.map, d.N, d.q);
    RP_LAUNCH_CHECK();
    RP_CUDA(cudaStreamSynchronize(stream));  // the pinned info words are reused by the next system
}

// ---- refinement across the GPU with FP32 factors
// The refinement of lu_solve_refine_kernel for systems of kLUHost64Min or more unknowns: the same steps
// (scaled FP32 corrections, FP64 residuals, the backward-error stop) and the same condition
// estimate, as rounds of three launches that decide on the device and return at once when there is
// nothing left to do, for up to kAcSystems systems:
//   across_control_kernel   one CTA per system: what the last round's results mean for the refinement
//                           and for Hager's estimate, and the next right-hand sides;
//   across_apply_kernel     (P L U)^-1 of all of these at once, in one cluster per system;
//   across_residual_kernel  x += correction and r = bs - A0 x in FP64, rows over the GPU.
// The refinement, the estimate and its extra test vector do not depend on one another, so
// round k carries correction k, the estimate's vector k and (round 0) the extra vector: four
// rounds instead of eight triangular solves one after the other.
// Measured, refinement and estimate: 2.46 -> 0.95 ms at 2001 unknowns and 1.3 -> 0.38 at 768 (against
// cuBLAS solves and residuals with a look by the host after each), 1.56 -> 0.39 at 767 and 0.70 ->
// 0.28 at 425 (against one CTA, whose FP64 residual alone takes 154 us per step at 767).
constexpr int kAcB = 128;     // unknowns of a block, whose diagonal blocks of L and U are inverted once
constexpr int kAcCTAs = 8;    // CTAs of the cluster, 16 rows of each block each
constexpr int kAcT = 512;     // their threads
constexpr int kAcRounds = 6;  // rounds launched ahead of a look at the outcome
// When a system goes to substitution instead.  What the last correction leaves of itself, its largest
// element times the rate at which the residual fell, says how far the solution still depends on
// how the triangular solves round: at 3 steps the charges differ from substitution's by up to 4 times
// that (1e-10 to 2e-10 at the triclinic cells' 2e-11 to 1.4e-10, 3.5e-10 to 7.6e-8 at 4e-10 to 2e-7 of
// dense cells of 830 to 920 unknowns), at 2 steps by up to 0.45 times (QEq systems of 479 to 2001).
constexpr double kInvLeft2 = 1e-9, kInvLeft = 2e-10;
constexpr double kInvRate = 1e-2;  // a slower system is not waited for

struct AcrossState {
    unsigned long long an_bits, anorm_bits;  // max row sums of |K| and of |A|
    unsigned long long rn_bits, xn_bits;     // max |r|, max |x| of the round's residual
    double rm, rprev, res, est, alt;
    int steps, phase;       // phase 0: refining, 1: converged, 2: left to substitution, 3: zero pivot
    int hstate, hit, jprev, jcur;  // 0: uniform vector under way, 1: signs, 2: a unit vector, 3: estimate done
    int xsel, finished;     // which x holds the solution; nothing left to do
};
struct AcrossRun {
    const float *LU;        // factors, row i of them row perm[i] of K
    float *inv;             // inverses of their diagonal blocks, L's then U's, and behind them the blocks
    float *V, *Y;           // [3][n1] right-hand sides and solutions
    double *x[2];           // solution before and after a round
    AcrossState *st;
    const double *A0, *bs;  // SolveDesc's
    double *r, *q, *info, *pre;
    const int *perm, *map;
    int N, n1, nblk;
};
// The systems of a launch, one to a row of its grid.  Nothing of one system's work depends on the others, so
// its results are the same bits in any company.
constexpr int kAcSystems = 16;
struct AcrossLaunch {
    AcrossRun run[kAcSystems];
};

// max row sums of |K| and |A| (K symmetric), a warp per row; st cleared before
__global__ void __launch_bounds__(256) across_norms_kernel(const __grid_constant__ AcrossLaunch L) {
    const AcrossRun &p = L.run[blockIdx.y];
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, n1 = p.n1;
    if (r >= n1) return;
    const double *row = p.A0 + (size_t)r * n1;
    double s = 0.0;
    for (int c = lane; c < n1 - 1; c += 32) s += fabs(row[c]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {  // (non-negative: the bits order like the values)
        atomicMax(&p.st->an_bits, (unsigned long long)__double_as_longlong(s + fabs(row[n1 - 1])));
        if (r < n1 - 1) atomicMax(&p.st->anorm_bits, (unsigned long long)__double_as_longlong(s));
    }
}

// Inverses of the diagonal blocks: blockIdx.x the block, blockIdx.y 0 for L (unit), 1 for U, taken
// with rows and columns reversed, as a lower triangle too.  Four threads per column of the inverse
// hold 32 of its rows each in registers (rows 16 g + 4 q + 0..3), column by column of the triangle: 16
// steps in line, then the registers move up by 16 rows, so the code stays small.  (Dot products
// from shared memory, row by row, took 100 us at any size.)  Rows past the end: identity.
constexpr int kInvLD = kAcB + 4, kInvCols = 64, kInvT = 4 * kInvCols;  // blockIdx.z: the system and which 64 columns
__global__ void __launch_bounds__(kInvT) across_invert_kernel(const __grid_constant__ AcrossLaunch L) {
    const AcrossRun &p = L.run[blockIdx.z / (kAcB / kInvCols)];
    extern __shared__ __align__(16) float ash[];
    float *B = ash, *dinv = ash + kAcB * kInvLD;  // B[k][i]: column k below the diagonal
    chain_begin();
    if ((int)blockIdx.x >= p.nblk || p.pre[0] != 0.0) return;
    const int half = blockIdx.z % (kAcB / kInvCols);
    const int n1 = p.n1, b0 = blockIdx.x * kAcB, tid = threadIdx.x, lane = tid & 31, c = half * kInvCols + (tid >> 2), q = tid & 3;
    const bool rev = blockIdx.y == 1;
#pragma unroll 16
    for (int t = tid; t < kAcB * kAcB; t += kInvT) {
        const int i = t / kAcB, j = t % kAcB;
        const float v = b0 + i < n1 && b0 + j < n1 ? p.LU[(size_t)(b0 + i) * n1 + b0 + j] : (i == j ? 1.f : 0.f);
        const int r = rev ? kAcB - 1 - i : i, k = rev ? kAcB - 1 - j : j;
        B[k * kInvLD + r] = r > k ? v : 0.f;
        if (r == k) dinv[k] = rev ? 1.f / v : 1.f;
    }
    __syncthreads();
    float x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = 16 * (j >> 2) + 4 * q + (j & 3) == c ? 1.f : 0.f;
    float *out = p.inv + ((size_t)blockIdx.y * p.nblk + blockIdx.x) * kAcB * kAcB;
    float *tri = out + 2 * (size_t)p.nblk * kAcB * kAcB;  // the block's own triangle, zeros elsewhere
    for (int t = tid; t < kAcB * kInvCols; t += kInvT) {
        const int i = t / kInvCols, j = half * kInvCols + t % kInvCols;
        float v = i == j ? 1.f : 0.f;
        if ((rev ? j >= i : j < i) && b0 + i < n1 && b0 + j < n1) v = p.LU[(size_t)(b0 + i) * n1 + b0 + j];
        tri[i * kAcB + j] = v;
    }
#pragma unroll 1
    for (int t = 0; t < 8; ++t) {
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const int k = 16 * t + kk;
            const float xk = __shfl_sync(0xffffffffu, x[kk & 3], (lane & ~3) | (kk >> 2)) * dinv[k];
            if (q == kk >> 2) out[(rev ? kAcB - 1 - k : k) * kAcB + (rev ? kAcB - 1 - c : c)] = xk;
#pragma unroll
            for (int g = 0; g < 8; ++g)
                if (t + g < 8) {
                    const float4 b = *reinterpret_cast<const float4 *>(B + k * kInvLD + 16 * (t + g) + 4 * q);
                    x[4 * g + 0] = fmaf(-b.x, xk, x[4 * g + 0]);
                    x[4 * g + 1] = fmaf(-b.y, xk, x[4 * g + 1]);
                    x[4 * g + 2] = fmaf(-b.z, xk, x[4 * g + 2]);
                    x[4 * g + 3] = fmaf(-b.w, xk, x[4 * g + 3]);
                }
        }
#pragma unroll
        for (int j = 0; j < 28; ++j) x[j] = x[j + 4];
    }
}

// pre[0] at the end (last): 0 solved, 2 zero pivot, 3 not finished, 4 substitution (with the estimate
// in info); 3 is taken back by the rounds that follow
__global__ void __launch_bounds__(1024) across_control_kernel(const __grid_constant__ AcrossLaunch L, int round, int last) {
    const AcrossRun &p = L.run[blockIdx.x];
    __shared__ double sv[33], piv_v;
    __shared__ int si[32], piv_i;
    __shared__ AcrossState st;
    const int tid = threadIdx.x, n1 = p.n1, nt = blockDim.x;
    chain_begin();
    if (tid == 0) st = *p.st;
    __syncthreads();
    if (st.finished) return;
    if (round == 0) {
        double m = 0.0;
        for (int t = tid; t < n1; t += nt) {
            const double b = p.bs[t];
            p.r[t] = b;
            p.x[0][t] = 0.0;
            m = fmax(m, fabs(b));
        }
        m = block_max(m, n1, sv);
        if (tid == 0) {
            st.rm = m;
            st.rprev = 1e308;
            st.res = 0.0;
            st.steps = st.hit = st.hstate = st.xsel = 0;
            st.jprev = -1;
            st.est = st.alt = 0.0;
            st.phase = p.pre[0] != 0.0 ? 3 : m == 0.0 ? 1 : 0;
        }
        for (int t = tid; t < n1; t += nt) {
            p.V[n1 + t] = (float)(1.0 / (double)n1);
            p.V[2 * (size_t)n1 + t] = (float)(((t & 1) ? -1.0 : 1.0) * (1.0 + (double)t / (double)max(n1 - 1, 1)));
        }
    } else {
        double ym = 0.0;  // the correction's largest element, in units of rm
        if (st.phase == 0) {
            for (int t = tid; t < n1; t += nt) ym = fmax(ym, fabs((double)p.Y[t]));
            ym = block_max(ym, n1, sv);
        }
        if (tid == 0 && st.phase == 0) {
            const double rn = __longlong_as_double((long long)st.rn_bits), xn = __longlong_as_double((long long)st.xn_bits),
                         an = __longlong_as_double((long long)st.an_bits);
            st.res = rn;
            ++st.steps;
            st.xsel = round & 1;
            if (rn <= (double)n1 * 1.1102230246251565e-16 * an * xn) {
                // (ym st.rm the correction, rn / st.rm the rate)
                st.phase = !(ym * rn > (st.steps <= 2 ? kInvLeft2 : kInvLeft) * xn) ? 1 : 2;
            } else if (!(rn < 1e300) || (st.steps >= 2 && rn > kInvRate * st.rprev)) {
                st.phase = 2;  // substitution takes over
            }
            st.rprev = st.rm = rn;
        }
        if (st.hstate != 3) {
            const float *y = p.Y + n1;
            auto val = [&](float v) { return isfinite(v) ? (double)v : 1e300; };
            if (st.hstate == 1) {
                double best = -1.0, sum = 0.0;
                int bi = 0x7fffffff;
                for (int t = tid; t < n1; t += nt) {
                    const double z = val(y[t]), v = fabs(z);
                    sum += z;
                    if (v > best || (v == best && t < bi)) {
                        best = v;
                        bi = t;
                    }
                }
                sum = block_sum(sum, n1, sv);
                block_argmax(best, bi, sv, si, &piv_v, &piv_i);
                if (tid == 0) {
                    const double ztx = st.jprev < 0 ? sum / (double)n1 : val(y[st.jprev]);
                    st.jcur = piv_i;
                    st.hstate = piv_v > ztx ? 2 : 3;
                }
            } else {
                double a = 0.0;
                for (int t = tid; t < n1; t += nt) a += fabs(val(y[t]));
                a = block_sum(a, n1, sv);
                if (tid == 0) {
                    if (st.hstate == 0) {
                        st.est = a;
                        st.hstate = 1;
                    } else if (a > st.est) {
                        st.est = a;
                        st.jprev = st.jcur;
                        st.hstate = ++st.hit < 4 ? 1 : 3;
                    } else {
                        st.hstate = 3;
                    }
                }
            }
            __syncthreads();
            for (int t = tid; t < n1; t += nt)
                p.V[n1 + t] = st.hstate == 2 ? (t == st.jcur ? 1.f : 0.f) : (y[t] >= 0.f || !isfinite(y[t])) ? 1.f : -1.f;
        }
        if (round == 1) {
            double a = 0.0;
            for (int t = tid; t < n1; t += nt) {
                const float v = p.Y[2 * (size_t)n1 + t];
                a += isfinite(v) ? fabs((double)v) : 1e300;
            }
            a = block_sum(a, n1, sv);
            if (tid == 0) st.alt = 2.0 * a / (3.0 * (double)n1);
        }
    }
    __syncthreads();
    if (st.phase == 0) {
        const double rm = st.rm;
        for (int t = tid; t < n1; t += nt) p.V[t] = (float)(p.r[t] / rm);
    }
    const bool solved = st.hstate == 3 && (st.phase == 1 || st.phase == 2);
    if (solved && st.phase == 1) {  // the solution, expanded to all atoms
        const double *x = p.x[st.xsel];
        for (int i = tid; i < p.N; i += nt) p.q[i] = x[p.map[i]];
    }
    if (tid == 0) {
        if (solved) {
            const double est = fmax(st.est, st.alt), kinv = est < 1e300 ? est : 1e300;
            p.info[0] = st.res;
            p.info[1] = p.pre[1];
            p.info[2] = p.pre[2];
            p.info[3] = 0.0;
            p.info[4] = fmin(__longlong_as_double((long long)st.anorm_bits) * kinv, 1e300);
            p.info[5] = n1;
            p.info[6] = st.steps;
            p.info[7] = 1.0;  // FP32 factors from across the GPU
        }
        st.finished = solved || st.phase == 3;
        if (st.phase == 3) p.pre[0] = 2.0;
        else if (solved) p.pre[0] = st.phase == 2 ? 4.0 : 0.0;
        else if (last) p.pre[0] = 3.0;
        st.rn_bits = st.xn_bits = 0;
        *p.st = st;
    }
}

// Y = U^-1 L^-1 P V for NR right-hand sides, in one cluster: a block of 128 unknowns at a time.  Each CTA
// keeps the whole solution; its 16 warps hold a row of the block each (of 128 rows, 16 per CTA),
// whose product with the unknowns known so far they form while the cluster waits for the
// previous block.  The rows' values go to every CTA's shared memory, and every CTA multiplies
// them by the inverted diagonal block: one cluster barrier per block.
// Bounded by those steps' latency (16 + 16 of them at 2001 unknowns) and by the factors' way from
// L2 to eight SMs (2 MB each there).
template <int NR>
__global__ void __cluster_dims__(kAcCTAs, 1, 1) __launch_bounds__(kAcT) across_apply_kernel(const __grid_constant__ AcrossLaunch L) {
    const AcrossRun &p = L.run[blockIdx.y];
    namespace cg = cooperative_groups;
    constexpr int NS = NR == 3 ? 4 : NR;  // floats per unknown in shared memory
    extern __shared__ __align__(16) float ash[];
    float *xs = ash;                                    // [nblk * 128][NS]
    float *wb = ash + (size_t)p.nblk * kAcB * NS;       // [2][128][NS] the block's rows
    float *rb = wb + 2 * kAcB * NS;                     // [128][NS] what they leave
    cg::cluster_group cl = cg::this_cluster();
    chain_begin();
    if (p.st->finished) return;  // (the same for the whole cluster)
    const int rank = (int)cl.block_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n1 = p.n1, nblk = p.nblk, rl = rank * (kAcB / kAcCTAs) + warp;  // the warp's row of each block
    for (int t = tid; t < nblk * kAcB; t += kAcT) {
        const int o = t < n1 ? p.perm[t] : 0;
#pragma unroll
        for (int q = 0; q < NR; ++q) xs[t * NS + q] = t < n1 ? p.V[(size_t)q * n1 + o] : 0.f;
    }
    cl.sync();  // every CTA runs and holds its right-hand sides
    const int mr = tid >> 2, mp = tid & 3;  // a diagonal block: a row's quarter of the columns
    auto times = [&](const float4 (&m)[8], const float *w, float (&v)[NR]) {  // its row times w, in all four threads
#pragma unroll
        for (int q = 0; q < NR; ++q) v[q] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float e[4] = {m[j].x, m[j].y, m[j].z, m[j].w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int q = 0; q < NR; ++q) v[q] = fmaf(e[i], w[(16 * j + 4 * mp + i) * NS + q], v[q]);
        }
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            v[q] += __shfl_xor_sync(0xffffffffu, v[q], 1);
            v[q] += __shfl_xor_sync(0xffffffffu, v[q], 2);
        }
    };
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
        const float *inv = p.inv + (size_t)dir * nblk * kAcB * kAcB + (size_t)mr * kAcB + 4 * mp;
        float acc[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) acc[q] = 0.f;
#pragma unroll 1
        for (int s = 0; s < nblk; ++s) {
            // (the buffers take turns over both sweeps: with an odd number of blocks, turns counted per
            // sweep would let a CTA that is ahead write the second sweep's first rows over the first's
            // last ones while another still reads them)
            const int b = dir ? nblk - 1 - s : s, nb_ = dir ? b - 1 : b + 1, buf = (dir * nblk + s) & 1;
            // this block's rows, to every CTA
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                float v = acc[q];
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                v = xs[(b * kAcB + rl) * NS + q] - v;
                if (lane < kAcCTAs) *cl.map_shared_rank(wb + (buf * kAcB + rl) * NS + q, lane) = v;
                acc[q] = 0.f;
            }
            __syncwarp();
            cg::cluster_group::arrival_token tok = cl.barrier_arrive();
            // while they travel: the inverted block, and the next block's rows times what is known
            float4 iv[8];
            {
                const float *src = inv + (size_t)b * kAcB * kAcB;
#pragma unroll
                for (int j = 0; j < 8; ++j) iv[j] = *reinterpret_cast<const float4 *>(src + 16 * j);
            }
            float near_[4] = {0.f, 0.f, 0.f, 0.f};  // the next rows' part of this block's columns
            const int nrow = nb_ * kAcB + rl;
            if (s + 1 < nblk && nrow < n1) {
                const float *row = p.LU + (size_t)nrow * n1;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = b * kAcB + lane + 32 * i;
                    near_[i] = c < n1 ? row[c] : 0.f;
                }
                const int c0 = dir ? (b + 1) * kAcB : 0, c1 = dir ? n1 : b * kAcB;
                for (int cc = c0 + lane; cc - lane < c1; cc += 512) {  // 16 loads in flight, none left over
                    float l[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) l[i] = cc + 32 * i < c1 ? row[cc + 32 * i] : 0.f;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float *x = xs + (cc + 32 * i < c1 ? cc + 32 * i : cc) * NS;
#pragma unroll
                        for (int q = 0; q < NR; ++q) acc[q] = fmaf(l[i], x[q], acc[q]);
                    }
                }
            }
            cl.barrier_wait(std::move(tok));
            // x = inv w, then once more on what w - B x leaves: as exact as substitution
            float v[NR], u[NR];
            times(iv, wb + buf * kAcB * NS, v);
            float4 bv[8];
            {
                const float *src = inv + (2 * (size_t)nblk + b) * kAcB * kAcB;
#pragma unroll
                for (int j = 0; j < 8; ++j) bv[j] = *reinterpret_cast<const float4 *>(src + 16 * j);
            }
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (mp == 0) xs[(b * kAcB + mr) * NS + q] = v[q];
            __syncthreads();
            times(bv, xs + b * kAcB * NS, u);
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (mp == 0) rb[mr * NS + q] = wb[(buf * kAcB + mr) * NS + q] - u[q];
            __syncthreads();
            times(iv, rb, u);
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (mp == 0) xs[(b * kAcB + mr) * NS + q] = v[q] + u[q];
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int q = 0; q < NR; ++q) acc[q] = fmaf(near_[i], xs[(b * kAcB + lane + 32 * i) * NS + q], acc[q]);
        }
    }
    for (int t = rank * kAcT + tid; t < n1; t += kAcCTAs * kAcT)
#pragma unroll
        for (int q = 0; q < NR; ++q) p.Y[(size_t)q * n1 + t] = xs[t * NS + q];
    cl.sync();  // no CTA leaves while another may still write to it
}

// x' = x + rm y (kept by the first CTA) and r = bs - A0 x' with its largest element, a warp per row
__global__ void __launch_bounds__(256) across_residual_kernel(const __grid_constant__ AcrossLaunch L, int round) {
    const AcrossRun &p = L.run[blockIdx.y];
    extern __shared__ double xd[];
    __shared__ unsigned long long top[2];
    chain_begin();
    if (p.st->finished || p.st->phase != 0) return;
    const int n1 = p.n1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double rm = p.st->rm, *xo = p.x[round & 1];
    double *xn = p.x[(round + 1) & 1];
    if (threadIdx.x < 2) top[threadIdx.x] = 0;
    __syncthreads();
    double m = 0.0;
    for (int t = threadIdx.x; t < n1; t += 256) {
        const double v = xo[t] + (double)p.Y[t] * rm;
        xd[t] = v;
        if (blockIdx.x == 0) {
            xn[t] = v;
            m = fmax(m, fabs(v));
        }
    }
    if (blockIdx.x == 0) atomicMax(&top[1], (unsigned long long)__double_as_longlong(m));
    __syncthreads();
    for (int r = blockIdx.x * 8 + warp; r < n1; r += gridDim.x * 8) {
        const double *row = p.A0 + (size_t)r * n1;
        double s = 0.0;
#pragma unroll 8
        for (int c = lane; c < n1; c += 32) s = fma(row[c], xd[c], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            const double v = p.bs[r] - s;
            p.r[r] = v;
            atomicMax(&top[0], (unsigned long long)__double_as_longlong(fabs(v)));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&p.st->rn_bits, top[0]);
        if (blockIdx.x == 0) p.st->xn_bits = top[1];
    }
}

// A system for the rounds, and the name of its buffers
struct AcrossSystem {
    const SolveDesc *d;
    std::string key;
};
// what a system needs beside its matrices when the second half of As does not hold it
size_t across_inv_bytes(int n1) { return sizeof(float) * (4 * (size_t)ceil_div(n1, kAcB) * kAcB * kAcB + 6 * (size_t)n1); }

// Launches rounds first .. first + rounds - 1 of up to kAcSystems systems (whose states are kept for the
// rounds that may follow), then looks at the outcome: pre[0] = 0 (solved: q and info written), 2
// (zero pivot: FP64 factors), 3 (not finished) or 4 (substitution).
void refine_across(rp_ctx *ctx, const std::vector<AcrossSystem> &sys, int first, int rounds, cudaStream_t stream) {
    StageTimer tt(ctx, "solve_refine32", stream);
    AcrossLaunch L{};
    int n1 = 0;  // the largest
    for (size_t k = 0; k < sys.size(); ++k) {
        const SolveDesc &d = *sys[k].d;
        AcrossRun &p = L.run[k];
        p.n1 = d.n + 1;
        p.nblk = (int)ceil_div(p.n1, kAcB);
        p.LU = reinterpret_cast<const float *>(d.As);
        p.A0 = d.A0; p.bs = d.bs; p.r = d.r; p.q = d.q; p.info = d.info; p.pre = d.pre; p.perm = d.perm; p.map = d.map;
        p.N = d.N;
        // inverses, blocks and vectors go to the second half of As, which is free once the factors are
        // collected, where they fit there
        const size_t need = across_inv_bytes(p.n1), half = sizeof(float) * (size_t)p.n1 * p.n1;
        const uintptr_t free_half = (reinterpret_cast<uintptr_t>(p.LU) + half + 255) & ~(uintptr_t)255;
        p.inv = need + 255 <= half ? reinterpret_cast<float *>(free_half)
                                   : static_cast<float *>(ctx->buf("s_ac_inv" + sys[k].key, need));
        p.V = p.inv + 4 * (size_t)p.nblk * kAcB * kAcB;
        p.Y = p.V + 3 * (size_t)p.n1;
        p.x[0] = d.x;
        p.x[1] = ctx->buf_t<double>("s_ac_x" + sys[k].key, (size_t)p.n1);
        p.st = ctx->buf_t<AcrossState>("s_ac_st" + sys[k].key, 1);
        n1 = std::max(n1, p.n1);
    }
    const unsigned ns = (unsigned)sys.size();
    const int nblk = (int)ceil_div(n1, kAcB);
    if (first == 0) {
        for (unsigned k = 0; k < ns; ++k) RP_CUDA(cudaMemsetAsync(L.run[k].st, 0, sizeof(AcrossState), stream));
        across_norms_kernel<<<dim3(ceil_div(n1, 8), ns), 256, 0, stream>>>(L);
        RP_LAUNCH_CHECK();
        const size_t inv_smem = sizeof(float) * (kAcB * kInvLD + kAcB);
        smem_optin((const void *)across_invert_kernel, inv_smem);
        launch_chained(across_invert_kernel, dim3(nblk, 2, ns * (kAcB / kInvCols)), kInvT, inv_smem, stream, L);
        launch_chained(across_control_kernel, dim3(ns), 1024, 0, stream, L, 0, 0);
    }
    const size_t np = (size_t)nblk * kAcB, res_smem = sizeof(double) * n1;
    const size_t most = sizeof(float) * 4 * (((size_t)kLUWideMax + kAcB - 1) / kAcB * kAcB + 3 * kAcB);
    smem_optin((const void *)across_apply_kernel<3>, most);
    smem_optin((const void *)across_apply_kernel<2>, most / 2);
    smem_optin((const void *)across_residual_kernel, sizeof(double) * kLUWideMax);
    const unsigned rows = (unsigned)std::min<long long>(ceil_div(n1, 8), std::max(304u / ns, 32u));
    for (int k = first; k < first + rounds; ++k) {
        if (k == 0) launch_chained(across_apply_kernel<3>, dim3(kAcCTAs, ns), kAcT, sizeof(float) * 4 * (np + 3 * kAcB), stream, L);
        else launch_chained(across_apply_kernel<2>, dim3(kAcCTAs, ns), kAcT, sizeof(float) * 2 * (np + 3 * kAcB), stream, L);
        launch_chained(across_residual_kernel, dim3(rows, ns), 256, res_smem, stream, L, k);
        launch_chained(across_control_kernel, dim3(ns), 1024, 0, stream, L, k + 1, (int)(k + 1 == first + rounds));
    }
}

// ---- the same by substitution, driven by the host
// For a system that the inverted blocks leave too far from it (kInvLeft, kInvRate): cuBLAS STRSV
// solves and DGEMV residuals across the GPU, a look at the outcome after each step.  Returns
// false when the refinement stalls: the caller then factors the system in FP64
// (factor_refine_wide64).  Waits.

__global__ void to_f32_kernel(const double *__restrict__ v, int n, double scale, float *__restrict__ y) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) y[t] = (float)(v[t] / scale);
}
__global__ void add_f32_kernel(const float *__restrict__ y, int n, double scale, double *__restrict__ x) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) x[t] += (double)y[t] * scale;
}
// y[i] = v[order[i]]: the factorisation's row order
__global__ void gather_rows_kernel(const float *__restrict__ v, const int *__restrict__ order, int n,
                                   float *__restrict__ y) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) y[t] = v[order[t]];
}
bool refine_wide32(rp_ctx *ctx, const SolveDesc &d, int n1, const std::string &key, cudaStream_t stream) {
    StageTimer tt(ctx, "solve_refine32", stream);
    const float *LU = reinterpret_cast<const float *>(d.As);
    cublasHandle_t hb = ctx->blas();
    RP_CUBLAS(cublasSetStream(hb, stream));
    float *ys = ctx->buf_t<float>("s_r32_y", (size_t)n1), *yv = ctx->buf_t<float>("s_r32_v", (size_t)n1);
    const int nb = (int)ceil_div(n1, 256);
    // pivot range of the factorisation, norms of the matrix and the estimate of refine_across
    double pre[3], kappa;
    AcrossState st{};
    RP_CUDA(cudaMemcpyAsync(pre, d.pre, sizeof(pre), cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaMemcpyAsync(&kappa, d.info + 4, sizeof(kappa), cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaMemcpyAsync(&st, ctx->buf_t<AcrossState>("s_ac_st" + key, 1), sizeof(st), cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaStreamSynchronize(stream));
    double an;
    std::memcpy(&an, &st.an_bits, sizeof(an));
    auto apply = [&]() {  // ys = (P L U)^-1 yv in FP32
        gather_rows_kernel<<<nb, 256, 0, stream>>>(yv, d.perm, n1, ys);
        RP_LAUNCH_CHECK();
        RP_CUBLAS(cublasStrsv(hb, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_T, CUBLAS_DIAG_UNIT, n1, LU, n1, ys, 1));
        RP_CUBLAS(cublasStrsv(hb, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_T, CUBLAS_DIAG_NON_UNIT, n1, LU, n1, ys, 1));
    };
    auto absmax = [&](const double *v) {
        int im = 0;
        RP_CUBLAS(cublasIdamax(hb, n1, v, 1, &im));
        double x = 0.0;
        RP_CUDA(cudaMemcpyAsync(&x, v + (im - 1), sizeof(double), cudaMemcpyDeviceToHost, stream));
        RP_CUDA(cudaStreamSynchronize(stream));
        return std::fabs(x);
    };
    const double one = 1.0, minus_one = -1.0;
    RP_CUDA(cudaMemsetAsync(d.x, 0, sizeof(double) * n1, stream));
    RP_CUDA(cudaMemcpyAsync(d.r, d.bs, sizeof(double) * n1, cudaMemcpyDeviceToDevice, stream));
    bool done = false;
    double res = 0.0, rprev = 1e308;
    int steps = 0;
    for (int it = 0; it < kRefineMax && !done; ++it) {
        const double rm = absmax(d.r);
        if (rm == 0.0) {
            done = true;
            break;
        }
        ++steps;
        to_f32_kernel<<<nb, 256, 0, stream>>>(d.r, n1, rm, yv);
        RP_LAUNCH_CHECK();
        apply();
        add_f32_kernel<<<nb, 256, 0, stream>>>(ys, n1, rm, d.x);
        RP_LAUNCH_CHECK();
        RP_CUDA(cudaMemcpyAsync(d.r, d.bs, sizeof(double) * n1, cudaMemcpyDeviceToDevice, stream));
        RP_CUBLAS(cublasDgemv(hb, CUBLAS_OP_T, n1, n1, &minus_one, d.A0, n1, d.x, 1, &one, d.r, 1));
        const double rn = absmax(d.r), xn = absmax(d.x);
        res = rn;
        if (rn <= (double)n1 * 1.1102230246251565e-16 * an * xn) done = true;
        else if (it >= 2 && rn > 0.5 * rprev) break;  // stalled: FP64 takes over
        rprev = rn;
    }
    if (!done) return false;
    double *hinfo = static_cast<double *>(ctx->host_buf("s_info32", sizeof(double) * kSolveInfo));
    hinfo[0] = res;
    hinfo[1] = pre[1];
    hinfo[2] = pre[2];
    hinfo[3] = 0.0;
    hinfo[4] = kappa;
    hinfo[5] = n1;
    hinfo[6] = steps;
    hinfo[7] = 1.0;  // FP32 factors from across the GPU
    RP_CUDA(cudaMemcpyAsync(d.info, hinfo, sizeof(double) * kSolveInfo, cudaMemcpyHostToDevice, stream));
    expand_kernel<<<(int)ceil_div(d.N, 256), 256, 0, stream>>>(d.x, d.map, d.N, d.q);
    RP_LAUNCH_CHECK();
    RP_CUDA(cudaStreamSynchronize(stream));  // the pinned info words are reused by the next system
    return true;
}

// interchanges in order (perm[k]: the row that came to k) to a row order, in place; one CTA.  After a
// zero pivot the later panels wrote no interchanges: nothing is read then.
__global__ void __launch_bounds__(1024) order_of_swaps_kernel(int *__restrict__ perm, int n,
                                                              const double *__restrict__ pre) {
    extern __shared__ int osm[];  // [n] interchanges, [n] order
    if (pre[0] != 0.0) return;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        osm[t] = perm[t];
        osm[n + t] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < n; ++k) {
            const int q = osm[k], o = osm[n + k];
            osm[n + k] = osm[n + q];
            osm[n + q] = o;
        }
    __syncthreads();
    for (int t = threadIdx.x; t < n; t += blockDim.x) perm[t] = osm[n + t];
}
void lu_wide_factor(rp_ctx *ctx, const SolveDesc &d, int n1, const std::string &tag, cudaStream_t stream) {
    float *L = reinterpret_cast<float *>(d.As);
    const long long nn = (long long)n1 * n1;
    lu_copy_kernel<float><<<(int)std::min<long long>(ceil_div(nn, 256), 4096), 256, 0, stream>>>(d.A0, L, nn, d.pre);
    RP_LAUNCH_CHECK();
    if (n1 <= kLUAcrossMax) {
        lu_factor_across(ctx, d, n1, tag, stream);
        return;
    }
    smem_optin((const void *)lu_panel_kernel, kPanelSmem);
    cublasHandle_t h = ctx->blas();
    RP_CUBLAS(cublasSetStream(h, stream));
    const float minus_one = -1.f, one = 1.f;
    for (int k0 = 0; k0 < n1;) {
        const int m = n1 - k0, NB = wide_panel_nb(m), nb = std::min(NB, m), c1 = k0 + nb;
        lu_panel_kernel<<<1, kLU, sizeof(float) * (size_t)m * (NB + 1), stream>>>(L, d.perm, n1, k0, NB, d.pre);
        RP_LAUNCH_CHECK();
        if (c1 < n1) {
            const int w = n1 - c1, grid = (int)ceil_div(w, 256);
            switch (NB) {
                case 32: lu_trsm_kernel<32><<<grid, 256, 0, stream>>>(L, n1, k0, d.pre); break;
                case 16: lu_trsm_kernel<16><<<grid, 256, 0, stream>>>(L, n1, k0, d.pre); break;
                case 8: lu_trsm_kernel<8><<<grid, 256, 0, stream>>>(L, n1, k0, d.pre); break;
                default: lu_trsm_kernel<4><<<grid, 256, 0, stream>>>(L, n1, k0, d.pre); break;
            }
            RP_LAUNCH_CHECK();
            // row-major A22 (w x w) -= L21 (w x nb) U12 (nb x w), as column-major C^T -= U12^T L21^T
            RP_CUBLAS(cublasSgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, w, w, nb, &minus_one, L + (size_t)k0 * n1 + c1, n1,
                                  L + (size_t)c1 * n1 + k0, n1, &one, L + (size_t)c1 * n1 + c1, n1));
        }
        k0 = c1;
    }
    smem_optin((const void *)order_of_swaps_kernel, 2 * sizeof(int) * kLUWideMax);
    order_of_swaps_kernel<<<1, 1024, 2 * sizeof(int) * (size_t)n1, stream>>>(d.perm, n1, d.pre);
    RP_LAUNCH_CHECK();
}

// the refinement of lu_solve_refine_kernel alone, on the FP32 factors that the rounds had; pre[0] = 2 where
// it stalls
void refine_in_cta(rp_ctx *ctx, const std::vector<const SolveDesc *> &sys, cudaStream_t stream) {
    StageTimer tt(ctx, "solve_refine32", stream);
    std::vector<SolveDesc> h;
    int n1 = 0;
    for (const SolveDesc *d : sys) {
        h.push_back(*d);
        h.back().host32 = h.back().factor_only = 0;
        h.back().across = 1;
        n1 = std::max(n1, d->n + 1);
        RP_CUDA(cudaMemsetAsync(d->pre, 0, sizeof(double), stream));
    }
    SolveDesc *dev = ctx->buf_t<SolveDesc>("s_desc_cta", h.size());
    RP_CUDA(cudaMemcpyAsync(dev, h.data(), sizeof(SolveDesc) * h.size(), cudaMemcpyHostToDevice, stream));
    lu_smem_optin();
    prepare_kernel<<<dim3(ceil_div(n1, 8), (unsigned)h.size()), 256, 0, stream>>>(dev);
    RP_LAUNCH_CHECK();
    lu_solve_refine_kernel<false><<<(unsigned)h.size(), solve_threads(n1), solve_smem_bytes(n1), stream>>>(dev);
    RP_LAUNCH_CHECK();
    RP_CUDA(cudaStreamSynchronize(stream));
}

}  // namespace

// Host side: reduced-index maps (repeat.py:2445-2470 semantics).
struct FoldPlan {
    int n = 0;
    std::vector<int> map, mem_ptr, mem_idx, ind;
    bool disjoint = true;
};

static FoldPlan make_plan(int N, int n_groups, const int *gptr, const int *gidx) {
    FoldPlan p;
    std::vector<char> linked((size_t)N, 0);
    std::vector<int> seen((size_t)N, 0);
    for (int g = 0; g < n_groups; ++g) {
        for (int t = gptr[g]; t < gptr[g + 1]; ++t) {
            int a = gidx[t];
            RP_REQUIRE(a >= 0 && a < N, "rp_solve: group atom index out of range");
            if (seen[a]++) p.disjoint = false;
            if (t > gptr[g]) linked[a] = 1;
        }
    }
    p.map.assign((size_t)N, -1);
    for (int i = 0; i < N; ++i)
        if (!linked[i]) {
            p.map[i] = (int)p.ind.size();
            p.ind.push_back(i);
        }
    p.n = (int)p.ind.size();
    std::vector<std::vector<int>> mem((size_t)p.n);
    for (int r = 0; r < p.n; ++r) mem[r].push_back(p.ind[r]);
    for (int g = 0; g < n_groups; ++g) {
        int base = gidx[gptr[g]];
        for (int t = gptr[g] + 1; t < gptr[g + 1]; ++t) {
            int l = gidx[t];
            if (p.map[base] >= 0) {
                mem[p.map[base]].push_back(l);
                p.map[l] = p.map[base];
            }
        }
    }
    // linked atoms whose base is itself linked (chains) take the final base's value
    for (int pass = 0; pass < n_groups + 1; ++pass) {
        bool changed = false;
        for (int g = 0; g < n_groups; ++g) {
            int base = gidx[gptr[g]];
            for (int t = gptr[g] + 1; t < gptr[g + 1]; ++t)
                if (p.map[gidx[t]] != p.map[base] && p.map[base] >= 0) {
                    p.map[gidx[t]] = p.map[base];
                    changed = true;
                }
        }
        if (!changed) break;
    }
    for (int i = 0; i < N; ++i)
        RP_REQUIRE(p.map[i] >= 0 && p.map[i] < p.n, "rp_solve: symmetry groups link atoms in a cycle");
    p.mem_ptr.push_back(0);
    for (auto &m : mem) {
        p.mem_idx.insert(p.mem_idx.end(), m.begin(), m.end());
        p.mem_ptr.push_back((int)p.mem_idx.size());
    }
    return p;
}

// Exact sequential folding on the host for overlapping groups.
static void host_fold(int N, const std::vector<double> &A, const std::vector<double> &b, int n_groups, const int *gptr,
                      const int *gidx, const FoldPlan &p, std::vector<double> &Ar, std::vector<double> &br,
                      std::vector<double> &w) {
    std::vector<double> AA(A), bb(b), ww((size_t)N, 1.0);
    for (int g = 0; g < n_groups; ++g) {
        int base = gidx[gptr[g]];
        for (int t = gptr[g] + 1; t < gptr[g + 1]; ++t) {
            int l = gidx[t];
            bb[base] += bb[l];
            ww[base] += 1.0;
            for (int r = 0; r < N; ++r) AA[(size_t)r * N + base] += AA[(size_t)r * N + l];
        }
    }
    for (int g = 0; g < n_groups; ++g) {
        int base = gidx[gptr[g]];
        for (int t = gptr[g] + 1; t < gptr[g + 1]; ++t) {
            int l = gidx[t];
            for (int c = 0; c < N; ++c) AA[(size_t)base * N + c] += AA[(size_t)l * N + c];
        }
    }
    Ar.assign((size_t)p.n * p.n, 0.0);
    br.assign((size_t)p.n, 0.0);
    w.assign((size_t)p.n, 0.0);
    for (int r = 0; r < p.n; ++r) {
        for (int c = 0; c < p.n; ++c) Ar[(size_t)r * p.n + c] = AA[(size_t)p.ind[r] * N + p.ind[c]];
        br[r] = bb[p.ind[r]];
        w[r] = ww[p.ind[r]];
    }
}

const double *solve_batch_async(rp_ctx *ctx, const std::vector<SolveJob> &jobs, cudaStream_t stream,
                                const std::string &tag, SolvePending *pend) {
    const int nj = (int)jobs.size();
    if (nj == 0) return nullptr;
    std::vector<FoldPlan> plans((size_t)nj);
    size_t n_map = 0, n_mptr = 0, n_midx = 0, n_red = 0, n_sq = 0;
    for (int j = 0; j < nj; ++j) {
        const SolveJob &J = jobs[j];
        RP_REQUIRE(J.A && J.b && J.q && J.N > 0, "rp_solve: null argument or N <= 0");
        RP_REQUIRE(J.n_groups == 0 || (J.group_ptr && J.group_idx), "rp_solve: groups given without arrays");
        plans[j] = make_plan(J.N, J.n_groups, J.group_ptr, J.group_idx);
        const size_t n1 = (size_t)plans[j].n + 1;
        n_map += J.N;
        n_mptr += plans[j].mem_ptr.size();
        n_midx += std::max<size_t>(plans[j].mem_idx.size(), 1);
        n_red += n1;
        n_sq += n1 * n1;
    }
    int *d_map = ctx->buf_t<int>("s_map" + tag, n_map);
    int *d_mptr = ctx->buf_t<int>("s_mptr" + tag, n_mptr);
    int *d_midx = ctx->buf_t<int>("s_midx" + tag, n_midx);
    double *d_rs = ctx->buf_t<double>("s_rs" + tag, n_red);
    double *d_rt = ctx->buf_t<double>("s_rt" + tag, n_red);
    double *As = ctx->buf_t<double>("s_As" + tag, n_sq);
    double *A0 = ctx->buf_t<double>("s_A0" + tag, n_sq);
    double *bs = ctx->buf_t<double>("s_bs" + tag, n_red);
    double *x = ctx->buf_t<double>("s_x" + tag, n_red);
    double *r = ctx->buf_t<double>("s_r" + tag, n_red);
    int *perm = ctx->buf_t<int>("s_perm" + tag, n_red);
    double *d_info = ctx->buf_t<double>("s_info" + tag, (size_t)nj * kSolveInfo);
    double *d_pre = ctx->buf_t<double>("s_pre" + tag, (size_t)nj * 3);
    SolveDesc *d_desc = ctx->buf_t<SolveDesc>("s_desc" + tag, (size_t)nj);
    // host staging of the small per-system tables, one upload each
    std::vector<int> h_map(n_map), h_mptr(n_mptr), h_midx(n_midx, 0);
    std::vector<double> h_rs(n_red, 0.0), h_rt(n_red, 0.0);
    std::vector<SolveDesc> descs((size_t)nj);
    size_t o_map = 0, o_mptr = 0, o_midx = 0, o_red = 0, o_sq = 0;
    for (int j = 0; j < nj; ++j) {
        const SolveJob &J = jobs[j];
        const FoldPlan &p = plans[j];
        const int n1 = p.n + 1;
        std::copy(p.map.begin(), p.map.end(), h_map.begin() + o_map);
        std::copy(p.mem_ptr.begin(), p.mem_ptr.end(), h_mptr.begin() + o_mptr);
        std::copy(p.mem_idx.begin(), p.mem_idx.end(), h_midx.begin() + o_midx);
        if (J.resp_s)
            for (int rr = 0; rr < p.n; ++rr) {
                h_rs[o_red + rr] = J.resp_s[p.ind[rr]];
                h_rt[o_red + rr] = J.resp_t ? J.resp_t[p.ind[rr]] : 0.0;
            }
        SolveDesc &d = descs[j];
        d.A = J.A; d.b = J.b; d.N = J.N; d.n = p.n;
        d.mem_ptr = d_mptr + o_mptr; d.mem_idx = d_midx + o_midx;
        d.resp_s = J.resp_s ? d_rs + o_red : nullptr; d.resp_t = J.resp_s ? d_rt + o_red : nullptr;
        d.map = d_map + o_map; d.qtot = J.qtot;
        d.As = As + o_sq; d.A0 = A0 + o_sq; d.bs = bs + o_red; d.x = x + o_red; d.r = r + o_red;
        d.big = n1 > kLUWideMax || (ctx->solve_in_memory && n1 >= 4);
        d.perm = perm + o_red; d.q = J.q; d.info = d_info + kSolveInfo * (size_t)j;
        o_map += J.N;
        o_mptr += p.mem_ptr.size();
        o_midx += std::max<size_t>(p.mem_idx.size(), 1);
        o_red += (size_t)n1;
        o_sq += (size_t)n1 * n1;
    }
    // wide systems are factored across the GPU before the refinement kernel: their flags
    std::vector<int> disjoint;
    for (int j = 0; j < nj; ++j) {
        const int n1 = plans[j].n + 1;
        if (n1 >= kLUHost64Min && n1 <= kLUWideMax) {
            descs[j].pre = d_pre + 3 * (size_t)j;
            if (jobs[j].fp64) descs[j].wide64 = 1;
            else if (n1 >= kLUWideMin) descs[j].host32 = 1;
        }
        if (plans[j].disjoint) disjoint.push_back(j);
    }
    // Between kLUHost64Min and kLUWideMin unknowns a system alone in its launch is factored across the GPU, from
    // kAcrossTwo also one or two beside smaller ones; others side by side with them, each in its CTA, to
    // the same factors bit for bit.  All of a launch are refined together by the rounds, so charges do not depend on the
    // batch.  (Factors and refinement of 16 systems: 0.71 ms at 256 unknowns, 1.2 at 420, 3.3 at 740, against
    // 0.76, 1.5 and 4.5 with each refined in its CTA; of one: 0.44, 0.64 and 1.1 against 0.71, 1.2 and 2.6.)
    std::vector<int> rounds;
    int least = kLUWideMin;
    for (int j = 0; j < nj; ++j) {
        const int n1 = plans[j].n + 1;
        if (!descs[j].pre || descs[j].wide64 || n1 >= kLUWideMin) continue;
        rounds.push_back(j);
        least = std::min(least, n1);
        descs[j].factor_only = 1;
    }
    if (nj == 1 || (rounds.size() <= 2 && least >= kAcrossTwo))
        for (int j : rounds) {
            descs[j].across = 1;
            descs[j].host32 = 1;
        }
    // the small tables go up from one pinned staging block per tag (asynchronous copies that
    // never wait for the stream; a later solve with another tag cannot overwrite them)
    const size_t st_bytes[7] = {sizeof(int) * n_map, sizeof(int) * n_mptr, sizeof(int) * n_midx,
                                sizeof(double) * n_red, sizeof(double) * n_red, sizeof(SolveDesc) * nj,
                                sizeof(int) * std::max<size_t>(disjoint.size(), 1)};
    size_t st_off[7], st_end = 0;
    for (int t = 0; t < 7; ++t) {
        st_off[t] = st_end;
        st_end += (st_bytes[t] + 15) / 16 * 16;
    }
    char *stage = static_cast<char *>(ctx->host_buf("s_stage" + tag, st_end));
    std::memcpy(stage + st_off[0], h_map.data(), st_bytes[0]);
    std::memcpy(stage + st_off[1], h_mptr.data(), st_bytes[1]);
    std::memcpy(stage + st_off[2], h_midx.data(), st_bytes[2]);
    std::memcpy(stage + st_off[3], h_rs.data(), st_bytes[3]);
    std::memcpy(stage + st_off[4], h_rt.data(), st_bytes[4]);
    RP_CUDA(cudaMemcpyAsync(d_map, stage + st_off[0], st_bytes[0], cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_mptr, stage + st_off[1], st_bytes[1], cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_midx, stage + st_off[2], st_bytes[2], cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_rs, stage + st_off[3], st_bytes[3], cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_rt, stage + st_off[4], st_bytes[4], cudaMemcpyHostToDevice, stream));
    std::memcpy(stage + st_off[5], descs.data(), st_bytes[5]);
    RP_CUDA(cudaMemcpyAsync(d_desc, stage + st_off[5], st_bytes[5], cudaMemcpyHostToDevice, stream));
    if (!disjoint.empty()) {  // every system with disjoint groups: one launch
        int *d_sys = ctx->buf_t<int>("s_sys" + tag, disjoint.size());
        std::memcpy(stage + st_off[6], disjoint.data(), st_bytes[6]);
        RP_CUDA(cudaMemcpyAsync(d_sys, stage + st_off[6], st_bytes[6], cudaMemcpyHostToDevice, stream));
        long long most = 1;
        for (int j : disjoint) most = std::max<long long>(most, (long long)(plans[j].n + 1) * (plans[j].n + 1));
        const dim3 grid((unsigned)std::min<long long>(ceil_div(most, 256), 1024), (unsigned)disjoint.size());
        build_bordered_kernel<<<grid, 256, 0, stream>>>(d_desc, d_sys);
        RP_LAUNCH_CHECK();
    }
    for (int j = 0; j < nj; ++j) {
        const SolveJob &J = jobs[j];
        const FoldPlan &p = plans[j];
        const int n1 = p.n + 1;
        if (!p.disjoint) {
            // overlapping groups: the reference's sequential folding on the host
            std::vector<double> hA((size_t)J.N * J.N), hb((size_t)J.N), Ar, br, w;
            RP_CUDA(cudaMemcpyAsync(hA.data(), J.A, sizeof(double) * hA.size(), cudaMemcpyDeviceToHost, stream));
            RP_CUDA(cudaMemcpyAsync(hb.data(), J.b, sizeof(double) * J.N, cudaMemcpyDeviceToHost, stream));
            RP_CUDA(cudaStreamSynchronize(stream));
            host_fold(J.N, hA, hb, J.n_groups, J.group_ptr, J.group_idx, p, Ar, br, w);
            std::vector<double> hs((size_t)n1 * n1, 0.0), hbs((size_t)n1, 0.0);
            for (int rr = 0; rr < p.n; ++rr) {
                for (int c = 0; c < p.n; ++c) hs[(size_t)rr * n1 + c] = Ar[(size_t)rr * p.n + c];
                double rsv = J.resp_s ? J.resp_s[p.ind[rr]] : 0.0;
                double rtv = (J.resp_s && J.resp_t) ? J.resp_t[p.ind[rr]] : 0.0;
                hs[(size_t)rr * n1 + rr] += rsv;
                hs[(size_t)rr * n1 + p.n] = w[rr];
                hs[(size_t)p.n * n1 + rr] = w[rr];
                hbs[rr] = br[rr] + rsv * rtv;
            }
            hbs[p.n] = J.qtot;
            RP_CUDA(cudaMemcpyAsync(descs[j].A0, hs.data(), sizeof(double) * hs.size(), cudaMemcpyHostToDevice, stream));
            RP_CUDA(cudaMemcpyAsync(descs[j].bs, hbs.data(), sizeof(double) * hbs.size(), cudaMemcpyHostToDevice, stream));
            RP_CUDA(cudaStreamSynchronize(stream));
        }
    }
    // large systems: factored across the GPU first, the wide ones refined behind their factors
    bool any_wide = false, any_pre = false;
    for (int j = 0; j < nj; ++j) any_pre |= descs[j].pre != nullptr;
    if (pend) *pend = SolvePending{};
    if (any_pre) RP_CUDA(cudaMemsetAsync(d_pre, 0, sizeof(double) * 3 * nj, stream));
    for (int j = 0; j < nj; ++j) {
        if (!descs[j].pre || descs[j].wide64) continue;  // wide64: factored and refined after the launch
        any_wide = true;  // its flag is read after the launch
        const bool wide = plans[j].n + 1 >= kLUWideMin;
        if (!wide && !descs[j].across) continue;
        {
            StageTimer tt(ctx, "solve_lu_wide", stream);
            lu_wide_factor(ctx, descs[j], plans[j].n + 1, tag, stream);
        }
        if (wide) refine_across(ctx, {{&descs[j], tag + "#" + std::to_string(j)}}, 0, kAcRounds, stream);
    }
    {
        StageTimer tt(ctx, "solve_lu", stream);
        int n1max = 0;  // of the systems solved in their CTAs
        size_t smem = 0;
        bool big = false;
        for (int j = 0; j < nj; ++j) {
            if (descs[j].wide64 || descs[j].host32) continue;
            n1max = std::max(n1max, descs[j].n + 1);
            smem = std::max(smem, solve_smem_bytes(descs[j].n + 1, descs[j].big));
            big |= descs[j].big != 0;
        }
        if (n1max > 0) {
            lu_smem_optin();
            prepare_kernel<<<dim3(ceil_div(n1max, 8), nj), 256, 0, stream>>>(d_desc);
            RP_LAUNCH_CHECK();
            auto kernel = big ? lu_solve_refine_kernel<true> : lu_solve_refine_kernel<false>;
            kernel<<<nj, solve_threads(n1max), smem, stream>>>(d_desc);
            RP_LAUNCH_CHECK();
        }
    }
    // the rounds of those below kLUWideMin: as many at a time as a launch takes and a quarter of the scratch left
    // holds, one set after the other in the same buffers
    size_t each = 1;
    for (int j : rounds) each = std::max(each, across_inv_bytes(plans[j].n + 1));
    const size_t set = std::max<size_t>(1, std::min<size_t>(kAcSystems, ctx->room({}) / 4 / each));
    std::vector<std::string> keys((size_t)nj);
    for (int j = 0; j < nj; ++j) keys[j] = tag + "#" + std::to_string(j);
    for (size_t k = 0; k < rounds.size(); ++k) keys[rounds[k]] = tag + "#m" + std::to_string(k % set);
    for (size_t k0 = 0; k0 < rounds.size(); k0 += set) {
        std::vector<AcrossSystem> sys;
        for (size_t k = k0; k < std::min(rounds.size(), k0 + set); ++k) sys.push_back({&descs[rounds[k]], keys[rounds[k]]});
        refine_across(ctx, sys, 0, kAcRounds, stream);
    }
    for (int j = 0; j < nj; ++j)  // systems known to need FP64 (an escalated fit): getrf, host-driven refinement
        if (descs[j].wide64) factor_refine_wide64(ctx, descs[j], plans[j].n + 1, stream);
    double *h_info = static_cast<double *>(ctx->host_buf("s_info" + tag, sizeof(double) * kSolveInfo * nj));
    if (any_wide) {
        // wide systems whose FP32 refinement did not converge (flag 2) are factored again in FP64:
        // their flags go to pinned memory, and solve_wide_fp64 (now, or, with `pend`, when the
        // caller's completion reaches it) reads them and redoes those systems
        double *h_pre = static_cast<double *>(ctx->host_buf("s_preh" + tag, sizeof(double) * 3 * nj));
        RP_CUDA(cudaMemcpyAsync(h_pre, d_pre, sizeof(double) * 3 * nj, cudaMemcpyDeviceToHost, stream));
        SolvePending local;
        SolvePending &pd = pend ? *pend : local;
        pd.any_wide = true;
        pd.tag = tag;
        pd.h_pre = h_pre;
        pd.h_info = h_info;
        pd.d_info = d_info;
        pd.descs = descs;
        pd.keys = keys;
        pd.shared = rounds.size() > set;
        pd.n1.resize((size_t)nj);
        for (int j = 0; j < nj; ++j) pd.n1[j] = plans[j].n + 1;
        if (!pend) {
            RP_CUDA(cudaStreamSynchronize(stream));
            solve_wide_fp64(ctx, pd, stream);
        }
    }
    RP_CUDA(cudaMemcpyAsync(h_info, d_info, sizeof(double) * kSolveInfo * nj, cudaMemcpyDeviceToHost, stream));
    return h_info;
}

void solve_wide_fp64(rp_ctx *ctx, SolvePending &pd, cudaStream_t stream) {
    if (!pd.any_wide) return;
    pd.any_wide = false;
    const int nj = (int)pd.descs.size();
    bool any = false;
    std::vector<double> flag((size_t)nj, 0.0);
    auto look = [&](int j) { RP_CUDA(cudaMemcpyAsync(&flag[j], pd.descs[j].pre, sizeof(double), cudaMemcpyDeviceToHost, stream)); };
    std::vector<int> cta;
    for (int j = 0; j < nj; ++j) {
        if (!pd.descs[j].pre || pd.h_pre[3 * j] < 2.0) continue;
        flag[j] = pd.h_pre[3 * j];
        any = true;
        const bool wide = pd.n1[j] >= kLUWideMin;
        for (int n = 4; flag[j] == 3.0; n += 4) {  // not finished: more rounds, from the start where a later set took the buffers
            const bool again = !wide && pd.shared;
            if (again) RP_CUDA(cudaMemsetAsync(pd.descs[j].pre, 0, sizeof(double), stream));
            refine_across(ctx, {{&pd.descs[j], pd.keys[j]}}, again ? 0 : kAcRounds + n - 4, again ? kAcRounds + n : 4, stream);
            look(j);
            RP_CUDA(cudaStreamSynchronize(stream));
        }
        if (flag[j] != 4.0) continue;  // 4: by substitution
        if (!wide) cta.push_back(j);
        else if (refine_wide32(ctx, pd.descs[j], pd.n1[j], pd.keys[j], stream)) flag[j] = 0.0;
    }
    if (!cta.empty()) {
        std::vector<const SolveDesc *> sys;
        for (int j : cta) sys.push_back(&pd.descs[j]);
        refine_in_cta(ctx, sys, stream);
        for (int j : cta) look(j);
        RP_CUDA(cudaStreamSynchronize(stream));
    }
    for (int j = 0; j < nj; ++j)
        if (flag[j] != 0.0) factor_refine_wide64(ctx, pd.descs[j], pd.n1[j], stream);
    if (!any) return;
    RP_CUDA(cudaMemcpyAsync(pd.h_info, pd.d_info, sizeof(double) * kSolveInfo * nj, cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaStreamSynchronize(stream));
}

void solve_batch(rp_ctx *ctx, const std::vector<SolveJob> &jobs, std::vector<double> &info, cudaStream_t stream) {
    const int nj = (int)jobs.size();
    info.assign((size_t)nj * kSolveInfo, 0.0);
    if (nj == 0) return;
    const double *h = solve_batch_async(ctx, jobs, stream, "");
    RP_CUDA(cudaStreamSynchronize(stream));
    std::copy(h, h + kSolveInfo * (size_t)nj, info.begin());
}

void solve_run(rp_ctx *ctx, const double *A_dev, const double *b_dev, int N, int n_groups, const int *group_ptr,
               const int *group_idx, const double *resp_s, const double *resp_t, double qtot, double *q_dev,
               double *info, cudaStream_t stream) {
    std::vector<SolveJob> jobs(1);
    jobs[0] = SolveJob{A_dev, b_dev, N, n_groups, group_ptr, group_idx, resp_s, resp_t, qtot, q_dev};
    std::vector<double> hinfo;
    solve_batch(ctx, jobs, hinfo, stream);
    if (info) {
        info[0] = hinfo[0];
        info[1] = hinfo[1];
        info[2] = hinfo[2];
        info[3] = hinfo[4];
    }
    if (hinfo[3] != 0.0) fail(RP_E_SINGULAR, "rp_solve: bordered system is singular (zero pivot)");
}

}  // namespace rp

// ---------------------------------------------------------------------------
// No-allocation variant of the constrained bordered solve.
//
// For callers that must not allocate device memory while they run: a serving
// loop that cannot afford the device-wide synchronisation cudaMalloc/cudaFree
// may cause, or an embedder whose device memory is owned entirely by its own
// allocator.  Its scratch is the file-scope array below (kNoAllocScratchBytes,
// enough for N <= kNoAllocMaxN atoms), which every GPU that loads this library
// keeps until the process exits.  Host code only sees a host-side stand-in for
// that symbol; the device address comes from cudaGetSymbolAddress, looked up once
// per device with that device current, on the first call made on it (make that
// first call before any stream capture).  With lazy module loading that first call
// may also be what loads the library's device code, and the array with it.  The
// address is kept for the life of the process: a cudaDeviceReset voids it, so do
// not call this entry point after resetting the device.  A call is synchronous: it
// returns once the solve on `stream` has finished.  All calls share the array and it
// keeps the last call's contents (every region is fully rewritten before it is read),
// so calls that overlap on the GPU race: serialise them on one stream.
namespace rp {
namespace {

constexpr int kNoAllocMaxN = 512;
constexpr size_t kNoAllocScratchBytes = 4718592;  // 4.5 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

unsigned char *noalloc_scratch_device() {
    static std::mutex mu;
    static unsigned char *addr[256] = {};
    int dev = 0;
    RP_CUDA(cudaGetDevice(&dev));
    RP_REQUIRE(dev >= 0 && dev < 256, "rp_solve_noalloc: device index out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) fail(RP_E_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        addr[dev] = static_cast<unsigned char *>(p);
    }
    return addr[dev];
}

// Bump allocator over the static array (256-byte aligned slices).
struct Carve {
    unsigned char *base;
    size_t off = 0;
    template <class T>
    T *take(size_t count) {
        size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
        if (off + bytes > kNoAllocScratchBytes) fail(RP_E_NOMEM, "rp_solve_noalloc: static scratch exhausted");
        T *p = reinterpret_cast<T *>(base + off);
        off += bytes;
        return p;
    }
};

}  // namespace
}  // namespace rp

extern "C" int rp_solve_noalloc(const double *A_dev, const double *b_dev, int N, int n_groups, const int *group_ptr,
                                const int *group_idx, const double *resp_s, const double *resp_t, double qtot,
                                double *q_dev, double *info, rp_stream_t stream_) {
    using namespace rp;
    cudaStream_t stream = (cudaStream_t)stream_;
    try {
        RP_REQUIRE(A_dev && b_dev && q_dev, "rp_solve_noalloc: null argument");
        if (N <= 0 || N > kNoAllocMaxN) return RP_E_ARG;  // N must be in 1..512
        RP_REQUIRE(n_groups == 0 || (group_ptr && group_idx), "rp_solve_noalloc: groups given without arrays");
        FoldPlan p = make_plan(N, n_groups, group_ptr, group_idx);
        const int n1 = p.n + 1;
        Carve cv{noalloc_scratch_device()};
        int *d_map = cv.take<int>((size_t)N);
        int *d_mptr = cv.take<int>(p.mem_ptr.size());
        int *d_midx = cv.take<int>(std::max<size_t>(p.mem_idx.size(), 1));
        double *d_rs = cv.take<double>((size_t)p.n);
        double *d_rt = cv.take<double>((size_t)p.n);
        double *As = cv.take<double>((size_t)n1 * n1);
        double *A0 = cv.take<double>((size_t)n1 * n1);
        double *bs = cv.take<double>((size_t)n1);
        double *x = cv.take<double>((size_t)n1);
        double *r = cv.take<double>((size_t)n1);
        int *perm = cv.take<int>((size_t)n1);
        double *d_info = cv.take<double>(kSolveInfo);
        SolveDesc *d_desc = cv.take<SolveDesc>(1);
        int *d_sys = cv.take<int>(1);
        std::vector<double> rs((size_t)p.n, 0.0), rt((size_t)p.n, 0.0);
        if (resp_s)
            for (int k = 0; k < p.n; ++k) {
                rs[k] = resp_s[p.ind[k]];
                rt[k] = resp_t ? resp_t[p.ind[k]] : 0.0;
            }
        RP_CUDA(cudaMemcpyAsync(d_map, p.map.data(), sizeof(int) * N, cudaMemcpyHostToDevice, stream));
        RP_CUDA(cudaMemcpyAsync(d_mptr, p.mem_ptr.data(), sizeof(int) * p.mem_ptr.size(), cudaMemcpyHostToDevice, stream));
        if (!p.mem_idx.empty())
            RP_CUDA(cudaMemcpyAsync(d_midx, p.mem_idx.data(), sizeof(int) * p.mem_idx.size(), cudaMemcpyHostToDevice,
                                    stream));
        if (p.n > 0) {
            RP_CUDA(cudaMemcpyAsync(d_rs, rs.data(), sizeof(double) * p.n, cudaMemcpyHostToDevice, stream));
            RP_CUDA(cudaMemcpyAsync(d_rt, rt.data(), sizeof(double) * p.n, cudaMemcpyHostToDevice, stream));
        }
        SolveDesc d{};
        d.A = A_dev; d.b = b_dev; d.N = N; d.n = p.n; d.mem_ptr = d_mptr; d.mem_idx = d_midx;
        d.resp_s = resp_s ? d_rs : nullptr; d.resp_t = resp_s ? d_rt : nullptr; d.map = d_map; d.qtot = qtot;
        d.As = As; d.A0 = A0; d.bs = bs; d.x = x; d.r = r; d.perm = perm; d.q = q_dev; d.info = d_info;
        RP_CUDA(cudaMemcpyAsync(d_desc, &d, sizeof(SolveDesc), cudaMemcpyHostToDevice, stream));
        if (p.disjoint) {
            RP_CUDA(cudaMemsetAsync(d_sys, 0, sizeof(int), stream));  // the one system
            const dim3 grid((unsigned)std::min<long long>(ceil_div((long long)n1 * n1, 256), 1024), 1u);
            build_bordered_kernel<<<grid, 256, 0, stream>>>(d_desc, d_sys);
            RP_LAUNCH_CHECK();
        } else {
            std::vector<double> hA((size_t)N * N), hb((size_t)N), Ar, br, w;
            RP_CUDA(cudaMemcpyAsync(hA.data(), A_dev, sizeof(double) * hA.size(), cudaMemcpyDeviceToHost, stream));
            RP_CUDA(cudaMemcpyAsync(hb.data(), b_dev, sizeof(double) * N, cudaMemcpyDeviceToHost, stream));
            RP_CUDA(cudaStreamSynchronize(stream));
            host_fold(N, hA, hb, n_groups, group_ptr, group_idx, p, Ar, br, w);
            std::vector<double> hs((size_t)n1 * n1, 0.0), hbs((size_t)n1, 0.0);
            for (int k = 0; k < p.n; ++k) {
                for (int c = 0; c < p.n; ++c) hs[(size_t)k * n1 + c] = Ar[(size_t)k * p.n + c];
                hs[(size_t)k * n1 + k] += rs[k];
                hs[(size_t)k * n1 + p.n] = w[k];
                hs[(size_t)p.n * n1 + k] = w[k];
                hbs[k] = br[k] + rs[k] * rt[k];
            }
            hbs[p.n] = qtot;
            RP_CUDA(cudaMemcpyAsync(A0, hs.data(), sizeof(double) * hs.size(), cudaMemcpyHostToDevice, stream));
            RP_CUDA(cudaMemcpyAsync(bs, hbs.data(), sizeof(double) * hbs.size(), cudaMemcpyHostToDevice, stream));
        }
        lu_smem_optin();
        prepare_kernel<<<dim3(ceil_div(n1, 8), 1), 256, 0, stream>>>(d_desc);
        RP_LAUNCH_CHECK();
        lu_solve_refine_kernel<false><<<1, solve_threads(n1), solve_smem_bytes(n1), stream>>>(d_desc);
        RP_LAUNCH_CHECK();
        double hinfo[kSolveInfo];
        RP_CUDA(cudaMemcpyAsync(hinfo, d_info, sizeof(hinfo), cudaMemcpyDeviceToHost, stream));
        RP_CUDA(cudaStreamSynchronize(stream));
        if (info) {
            info[0] = hinfo[0];
            info[1] = hinfo[1];
            info[2] = hinfo[2];
            info[3] = hinfo[4];
        }
        return hinfo[3] != 0.0 ? RP_E_SINGULAR : RP_OK;
    } catch (const rp::Error &e) {
        return e.code;
    } catch (const std::exception &) {
        return RP_E_ARG;
    }
}

// Diagnostics (not part of the public ABI): solve systems of any size in their CTA with the vectors in
// memory, as those beyond kLUWideMax are (on != 0)
extern "C" int rp_debug_solve_in_memory(rp_ctx *ctx, int on) {
    if (!ctx) return RP_E_ARG;
    ctx->solve_in_memory = on != 0;
    return RP_OK;
}
