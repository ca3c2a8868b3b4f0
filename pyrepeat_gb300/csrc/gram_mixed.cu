// Mixed-precision Phi -> normal equations on GB300.
//
// Replaces, on the device, the Phi build of EwaldCalculator._compute_gpu*
// (repeat.py:1199-1435) and the Gram accumulation of fit_charges
// (repeat.py:2246-2276).  Once per fit:
//
//  0. recip   E[r][a][n1] for every grid row r (separable reciprocal sum, stages A
//             and B in recip_sep.cu, on the FP32 pipe).
//
// Then per chunk of kept points (Phi exists for one chunk only):
//
//  1. Phi     Phi_t[a][m] = real-space erfc sum (FP32 terms from double-float
//             coordinates, FP64 at the cutoff, double-float per-pair sums)
//             + Re sum_n1 ex[n1][i_m] E[r_m][a][n1] (FP32), written once,
//             atom-major (phi_chunk_kernel).
//  2. split   X[a][m] = (Phi_t[a][m] - c_a) * 2^e_a cut into four 7-bit fixed-point
//             digits, plus a row for the centred ESP: c_a is the column mean of the
//             first chunk (a per-column shift corrected exactly later), 2^e_a a
//             power-of-two row scale.
//  3. Gram    G = X X^T on tcgen05 (kind::f16, FP32 accumulators in TMEM) with all
//             16 digit products kept: every partial sum is an integer below 2^24,
//             so the Gram of the staged Phi is exact; a persistent kernel (one CTA
//             per SM) takes work units (one point split of one tile) from a counter
//             and adds each unit's int64 sums to the tile's exact 64-bit totals with
//             atomics, which are rounded to FP64 once.
//  4. finish  A = G - s s^T/M, b = G[:,V] - s sum(V)/M with s = sum_m (Phi - c)
//             (FP64), i.e. repeat.py:2266-2276 for the shifted columns.
//
// Error budget: Phi carries the FP32 real-space terms and the FP32 reciprocal
// stages B and C (~1e-7 relative each, unbiased rounding) and the 28-bit digit
// quantisation of the Gram input (~2^-29 of each row's range, unbiased).  The
// tensor cores' FP32 accumulation truncates, which is why the Gram is done in
// exact integer digits instead of as an FP16/BF16 hi+lo product.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "df.cuh"
#include "f32x2.cuh"
#include "tc.cuh"

namespace rp {
namespace {

constexpr int kBM = 128;       // Gram tile rows (TMEM lanes)
constexpr int kKPad = 64;      // digit rows are padded to a multiple of 64 points (the tensor maps' unit)
constexpr int kBK = 32;        // points (K elements) per stage: 64 B of FP16 = one 64-byte swizzle row
constexpr int kTileBytes = kBM * kBK * 2;  // 8 KB per operand tile

// ---- GEMM-2 (Gram): exact integer products of four 7-bit fixed-point slices
// x = 2^-6 (x0 + 2^-7 x1 + 2^-14 x2 + 2^-21 x3), x_s integers with |x0| <= 32,
// |x1..x3| <= 64 (|x| <= 1/2; 28 bits below the row maximum, because a centred
// column's typical value sits orders of magnitude below its maximum).  All 16
// slice products are kept: for the many values far below their row's maximum the
// low digits carry the signal, not rounding noise (leaving out the three products of
// weight 5 and 6 moved the batch's charges from 4e-7 to 4e-6 e of FP64).  They are
// grouped by weight g = s+u into seven TMEM accumulators of a 128 x 64 tile.  Per
// point, a group's products sum to at most 12288 in magnitude (weight 3: x0 x3 +
// x3 x0 <= 2 * 32 * 64, x1 x2 + x2 x1 <= 2 * 64 * 64; weight 4: three products
// <= 64 * 64; the others less), so a stage of 32 points adds at most 393,216 =
// 3 * 2^17 to a group and kGramFlush = 32 stages (1024 points) stay below 2^24 (12.6 M):
// the FP32 sums are exact, and a work unit of kGramSplit = 32 stages drains them once, at
// its end.
// (A row whose |x| passed 1/2 is clamped, counted and its cube refitted from the
// staged Phi, whose own scale keeps |x| < 1/2.)  At each flush the epilogue folds the
// groups into one int64 per element (sum_g D_g 2^(7(6-g))), so the Gram carries no
// rounding bias (its diagonal is the most sensitive quantity of the fit).
constexpr int kGN = 64;          // Gram tile columns
constexpr int kGSlices = 4;
constexpr int kGroups = 2 * kGSlices - 1;
constexpr int kGramStages = 3;   // 3 x 48 KB: two stages in flight while one is multiplied
constexpr int kGramFlush = 32;
constexpr int kGramSplit = 32;   // stages per work unit: 1024 points, the int64 fold's headroom (2^52 per point)
constexpr int kStagesPer64 = kKPad / kBK;  // the autotuner's and the diagnostics' 64-point blocks, in stages
constexpr int kGramEpiWarps = 8;
constexpr int kEpiCols = kGN * 4 / kGramEpiWarps;  // Gram tile columns per epilogue warp (TMEM lane quarter)
constexpr int kGramThreads = 64 + 32 * kGramEpiWarps;  // 320
constexpr int kBTileBytes = kGN * kBK * 2;             // 4 KB
constexpr int kGramStageBytes = kGSlices * kTileBytes + kGSlices * kBTileBytes;
constexpr int kGramSmem = kGramStages * kGramStageBytes + 1024 + 256;

constexpr int kSched = 4;         // work-unit ring entries (producer -> MMA thread and epilogue)
// the barriers, the ring and the TMEM address after the stages, in the last 256 bytes
static_assert((2 * kGramStages + 3 + 2 * kSched) * 8 + kSched * 4 + 4 <= 256, "gram smem tail");

struct GramArgs {
    int nt, ntj, ntri, kb_total, kb_per_split, flush;  // flush: stages per exact FP32 run (<= kGramFlush)
    int unit0, nunits;  // this launch's work units unit0 .. unit0 + nunits - 1 of the ntri Gram
                        // tiles x ceil(kb_total / kb_per_split) point splits
    int *next_unit;     // this launch's work counter, zero at launch
    // exact tile sums [tri][col][row] as two's complement 64-bit halves: every unit adds the
    // high (acc >> 32) and low (acc & (2^32 - 1)) parts of its int64 partial (|acc| < 2^62)
    unsigned long long *out_hi, *out_lo;
    int *status;
    long long budget;  // clock budget of the pipeline's waits (tc::kWaitBudgetCycles; <= 0: give up at once)
};

__device__ __forceinline__ uint8_t *align1024(uint8_t *raw) {
    const uint32_t s = tc::smem_u32(raw);
    return raw + (((s + 1023u) & ~1023u) - s);
}

// Gram tile t -> (ti, tj): rows [128 ti, +128), columns [64 tj, +64), 2 ti <= tj < ntj,
// ntj = ceil(rows / 64): tiles wholly beyond the last row are never computed, and rows
// past the end of the digit arrays read as zeros (the tensor maps' out-of-bounds fill).
__device__ __forceinline__ void gram_tile_decode(int t, int ntj, int &ti, int &tj) {
    ti = 0;
    int len = ntj;
    while (t >= len) {
        t -= len;
        ++ti;
        len -= 2;
    }
    tj = 2 * ti + t;
}

// Work unit u = (tile u % ntri, point split u / ntri): consecutive units share their points,
// so the CTAs working at one time read the same digit columns through L2.
struct GramUnit {
    int tile, a_row0, b_row0, kb0, nkb;
};
__device__ __forceinline__ GramUnit gram_unit(const GramArgs &g, int unit) {
    GramUnit w;
    w.tile = unit % g.ntri;
    int ti, tj;
    gram_tile_decode(w.tile, g.ntj, ti, tj);
    w.a_row0 = ti * kBM;
    w.b_row0 = tj * kGN;
    w.kb0 = (unit / g.ntri) * g.kb_per_split;
    w.nkb = min(w.kb0 + g.kb_per_split, g.kb_total) - w.kb0;  // >= 1
    return w;
}

// Persistent: one CTA per SM takes work units from the launch's counter until none are left.
// Warp 0 (one thread) takes the units, posts each in a shared ring and streams its digit
// tiles by TMA through the stages, running ahead across unit boundaries; warp 1 (one
// thread) issues the MMAs; warps 2..9 drain the seven group accumulators from TMEM into
// int64 sums once per flush, 16 columns at a time, and add them to the tile's totals with
// 64-bit atomics (the last columns' while the MMAs of the next unit already run).
// At most 96 registers and 3 x 48 KB of stages: the SM keeps room for CTAs of other kernels
// (the Phi kernel of other cubes, bound by instruction issue, which this kernel barely uses).
__global__ void __maxnreg__(96) gram_exact_kernel(
    const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
    const __grid_constant__ CUtensorMap tm2, const __grid_constant__ CUtensorMap tm3,
    const __grid_constant__ CUtensorMap tb0, const __grid_constant__ CUtensorMap tb1,
    const __grid_constant__ CUtensorMap tb2, const __grid_constant__ CUtensorMap tb3, GramArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align1024(smem_raw);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kGramStages * kGramStageBytes);
    uint64_t *empty = full + kGramStages;
    uint64_t *accf = empty + kGramStages;  // accumulators ready for the epilogue
    uint64_t *acce = accf + 1;             // epilogue done reading them
    uint64_t *sfull = acce + 1;            // work unit posted in the ring
    uint64_t *sempty = sfull + kSched;     // ring entry read by the MMA thread and every epilogue warp
    uint64_t *fin = sempty + kSched;       // every MMA the CTA issued is complete
    volatile int *sched = reinterpret_cast<volatile int *>(fin + 1);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(const_cast<int *>(sched + kSched));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // B is loaded for every tile (also where its rows lie inside A's tile): the four B slices
    // then sit back to back and form one 256-row operand
    const uint32_t stage_tx = kGSlices * (kTileBytes + kBTileBytes);
    const CUtensorMap *ta[kGSlices] = {&tm0, &tm1, &tm2, &tm3};
    const CUtensorMap *tb[kGSlices] = {&tb0, &tb1, &tb2, &tb3};

    if (threadIdx.x == 0) {
        for (int s = 0; s < kGramStages; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(accf, 1);
        tc::mbar_init(acce, 32 * kGramEpiWarps);
        for (int r = 0; r < kSched; ++r) {
            tc::mbar_init(&sfull[r], 1);
            tc::mbar_init(&sempty[r], 1 + kGramEpiWarps);
        }
        tc::mbar_init(fin, 1);
        tc::fence_mbar_init();
    }
    if (warp == 1) tc::tmem_alloc(tmem_holder, 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_holder;

    if (warp == 0 && lane == 0) {
        int it = 0;  // stages issued
        bool ok = true;
        for (int j = 0; ok; ++j) {
            const int r = j % kSched;
            if (j >= kSched && !tc::mbar_wait(&sempty[r], ((j / kSched) - 1) & 1, g.status, g.budget)) break;
            const int k = atomicAdd(g.next_unit, 1);
            const int unit = k < g.nunits ? g.unit0 + k : -1;
            sched[r] = unit;
            tc::mbar_arrive(&sfull[r]);  // release: the entry is visible to the waiters
            if (unit < 0) break;
            const GramUnit w = gram_unit(g, unit);
            for (int kb = 0; kb < w.nkb; ++kb, ++it) {
                const int s = it % kGramStages, u = it / kGramStages;
                if (u > 0 && !tc::mbar_wait(&empty[s], (u - 1) & 1, g.status, g.budget)) {
                    ok = false;
                    break;
                }
                uint8_t *st = smem + s * kGramStageBytes;
                tc::mbar_arrive_expect_tx(&full[s], stage_tx);
                const int x = (w.kb0 + kb) * kBK;
#pragma unroll
                for (int q = 0; q < kGSlices; ++q) {
                    tc::tma_load_2d(st + q * kTileBytes, ta[q], x, w.a_row0, &full[s]);
                    tc::tma_load_2d(st + kGSlices * kTileBytes + q * kBTileBytes, tb[q], x, w.b_row0, &full[s]);
                }
            }
        }
        // after a timeout, the copies still in flight land before the CTA exits
        if (*reinterpret_cast<volatile int *>(g.status) != 0)
            for (int k = max(0, it - kGramStages); k < it; ++k)
                tc::mbar_wait(&full[k % kGramStages], (k / kGramStages) & 1, nullptr);
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = tc::idesc_f16_f32(kBM, kGN);
        const uint32_t idesc4 = tc::idesc_f16_f32(kBM, 4 * kGN);  // all four B slices, four adjacent groups
        uint32_t d[kGroups];  // group accumulators, 64 TMEM columns each
#pragma unroll
        for (int q = 0; q < kGroups; ++q) d[q] = tmem + (uint32_t)(q * kGN);
        int it = 0, fc = 0;  // stages consumed, flushes committed
        bool ok = true;
        for (int j = 0; ok; ++j) {
            const int r = j % kSched;
            if (!tc::mbar_wait(&sfull[r], (j / kSched) & 1, g.status, g.budget)) break;
            const int unit = sched[r];
            tc::mbar_arrive(&sempty[r]);
            if (unit < 0) break;
            const GramUnit w = gram_unit(g, unit);
            const int nflush = (w.nkb + g.flush - 1) / g.flush;
            for (int f = 0; f < nflush; ++f) {
                if (fc > 0 && !tc::mbar_wait(acce, (fc - 1) & 1, g.status, g.budget)) {  // sums drained
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const int kbf0 = f * g.flush, kbf1 = min(kbf0 + g.flush, w.nkb);
                for (int kb = kbf0; kb < kbf1; ++kb, ++it) {
                    const int s = it % kGramStages, u = it / kGramStages;
                    if (!tc::mbar_wait(&full[s], u & 1, g.status, g.budget)) {
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t st = tc::smem_u32(smem + s * kGramStageBytes);
                    uint64_t x[kGSlices], y[kGSlices];
#pragma unroll
                    for (int q = 0; q < kGSlices; ++q) {
                        x[q] = tc::sdesc_k_sw64(st + q * kTileBytes);
                        y[q] = tc::sdesc_k_sw64(st + kGSlices * kTileBytes + q * kBTileBytes);
                    }
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk) {
                        const uint64_t o = (uint64_t)(kk * 2);
                        if (kb == kbf0 && kk == 0) {
                            // the first products of a flush start each group's sum: one MMA per
                            // (slice a, slice b), the first into a group overwriting it
                            bool started[kGroups] = {false, false, false, false, false, false, false};
#pragma unroll
                            for (int a = 0; a < kGSlices; ++a)
#pragma unroll
                                for (int b = 0; b < kGSlices; ++b) {
                                    const int grp = a + b;
                                    const uint32_t acc = started[grp] ? 1u : 0u;
                                    started[grp] = true;
                                    tc::umma_f16(d[grp], x[a] + o, y[b] + o, idesc, acc);
                                }
                        } else {
                            // then N = 256: slice a against the four B slices back to back (a 256-row
                            // operand) writes the products of weights a .. a+3 into the four adjacent
                            // groups from d[a] (the same products, in the same order per group, as the
                            // pairs above), reading A once instead of four times
#pragma unroll
                            for (int a = 0; a < kGSlices; ++a) tc::umma_f16(d[a], x[a] + o, y[0] + o, idesc4, 1u);
                        }
                    }
                    tc::umma_commit(&empty[s]);
                }
                if (!ok) break;
                tc::umma_commit(accf);
                ++fc;
            }
        }
        tc::umma_commit(fin);  // tracks every MMA issued above
    } else if (warp >= 2) {
        const int ew = warp - 2;
        const int lane_base = (warp & 3) * 32;
        const int col0 = (ew >> 2) * kEpiCols;  // this warp's columns of the 64
        const uint32_t base = tmem + ((uint32_t)lane_base << 16) + (uint32_t)col0;
        int fc = 0;  // flushes drained
        bool ok = true;
        // every wait's outcome is made warp-uniform by a vote before the warp-wide
        // TMEM loads and the __syncwarp below
        for (int j = 0; ok; ++j) {
            const int r = j % kSched;
            if (!__all_sync(0xffffffffu, tc::mbar_wait(&sfull[r], (j / kSched) & 1, g.status, g.budget))) break;
            const int unit = sched[r];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&sempty[r]);
            if (unit < 0) break;
            const GramUnit w = gram_unit(g, unit);
            const int nflush = (w.nkb + g.flush - 1) / g.flush;
            const long long t0 = (long long)w.tile * (kBM * kGN);
            const int rr = lane_base + lane;
            for (int f = 0; f < nflush; ++f, ++fc) {
                if (!__all_sync(0xffffffffu, tc::mbar_wait(accf, fc & 1, g.status, g.budget)) ||
                    __any_sync(0xffffffffu, *reinterpret_cast<volatile int *>(g.status) != 0)) {
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                // the warp's columns 16 at a time (fewer live registers): the flush's int64 sums
                // of 16 columns go to the tile totals before the next 16 are loaded
#pragma unroll
                for (int h = 0; h < kEpiCols / 16; ++h) {
                    long long acc[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[i] = 0;
#pragma unroll
                    for (int q = 0; q < kGroups; ++q) {
                        float v[16];
                        tc::tmem_ld_32x16(base + (uint32_t)(q * kGN + 16 * h), v);
                        const int sh = 7 * (kGroups - 1 - q);
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[i] += (long long)__float2int_rn(v[i]) << sh;
                    }
                    if (h == kEpiCols / 16 - 1) {
                        tc::fence_before_sync();
                        tc::mbar_arrive(acce);
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const long long e = t0 + (col0 + 16 * h + i) * kBM + rr;
                        atomicAdd(g.out_hi + e, (unsigned long long)(acc[i] >> 32));
                        atomicAdd(g.out_lo + e, (unsigned long long)(acc[i] & 0xffffffffLL));
                    }
                }
            }
        }
    }
    // TMEM is freed only after every MMA of the CTA has completed (also after a timeout)
    if (warp == 1 && lane == 0) tc::mbar_wait(fin, 0, nullptr);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 1) tc::tmem_dealloc(tmem, 512);
}

// ESP row scale 2^(-e-1) with max|Vc| in [2^(e-1), 2^e), so |V * scale| < 1/2
__device__ __forceinline__ float vscale_of(double vmax) {
    int e = 0;
    if (vmax > 0.0) frexp(vmax, &e);
    return ldexpf(1.0f, -e - 1);
}

// Four 7-bit signed digits of an integer I = round(x 2^27), |x| <= 1:
// x ~ 2^-6 (s0 + 2^-7 s1 + 2^-14 s2 + 2^-21 s3), digits rounded half up so |s| <= 64,
// each exact in FP16.  Integer shifts only (no FP64 on the per-element path).
__device__ __forceinline__ void split4(int v, int &s0, int &s1, int &s2, int &s3) {
    s0 = (v + (1 << 20)) >> 21;
    int r = v - (s0 << 21);  // [-2^20, 2^20)
    s1 = (r + (1 << 13)) >> 14;
    r -= s1 << 14;           // [-2^13, 2^13)
    s2 = (r + (1 << 6)) >> 7;
    s3 = r - (s2 << 7);      // [-64, 64)
}

__device__ __forceinline__ void digits4(int v, __half *o0, __half *o1, __half *o2, __half *o3, long long idx) {
    int s0, s1, s2, s3;
    split4(v, s0, s1, s2, s3);
    o0[idx] = __int2half_rn(s0);
    o1[idx] = __int2half_rn(s1);
    o2[idx] = __int2half_rn(s2);
    o3[idx] = __int2half_rn(s3);
}

// round((h + l) * sc) for a double-float (h, l) and a power of two sc, |(h + l) sc| <= 2^27:
// rint of the high part is exact, the remainder (h sc - I1) is exact (Sterbenz), and the
// low part decides the last unit.
__device__ __forceinline__ int round_df(float h, float l, float sc) {
    const float H = h * sc, L = l * sc;
    const float I1 = rintf(H);
    const float I2 = rintf(__fadd_rn(__fadd_rn(H, -I1), L));
    return (int)I1 + (int)I2;
}

// Pairs closer than this radius (Bohr) get the FP64 real-space term; tunable with
// RP_REAL_FP64_R.  Default 0: with double-float image coordinates the FP32 terms
// keep the fitted charges within ~3e-7 e of the FP64 fit on the synthetic
// workloads, so FP64 is used only to decide images that sit at the cutoff.
float real_near2() {
    static float v = [] {
        const char *e = getenv("RP_REAL_FP64_R");
        double r = e ? atof(e) : 0.0;
        return (float)(r * r);
    }();
    return v;
}

// I = round(x 2^27) of one element of X (x = (Phi - c) scale, or the scaled ESP), |x| <= 1
__device__ __forceinline__ int x_fixed(float h, float l, float sc, int *clamped) {
    sc *= 134217728.0f;  // 2^27
    if (fabsf(h * sc) > 134217728.0f) {  // |x| beyond 1: clamp (counted; the fit reports it)
        atomicAdd(clamped, 1);
        return h > 0.f ? (1 << 27) : -(1 << 27);
    }
    return round_df(h, l, sc);
}

// ------------------------------------------------------------------ Phi of one chunk

// The approximate reciprocal, reciprocal square root and base-2 exponential of the
// multi-function unit, flushing subnormals (the arguments here are normal numbers), so
// that each is one instruction with no subnormal fix-up around it.
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// erfc(x), x >= 0, in FP32 by the Chebyshev fit "erfcc" of Press, Teukolsky, Vetterling
// and Flannery, Numerical Recipes in C (2nd ed., section 6.2): erfc(x) = t exp(-x^2 + P(t)),
// t = 1/(1 + x/2), fractional error below 1.2e-7.  It is evaluated in base 2: the argument
// comes pre-scaled, xs = sqrt(log2 e) x, and log2(e) is folded into the coefficients, so
//   erfc(x) = t 2^(-xs^2 + log2(e) P(t)),   t = 1 / (1 + xs / (2 sqrt(log2 e))),
// 14 instructions (one reciprocal, one exponential).  In FP32 the rounding of the exponent
// -xs^2 + p and of the reciprocal and exponential instructions dominates the error
// (measured against FP64 erfc and against CUDA's erfcf in the tests).  A degree-7 fit for
// the bounded range x <= pi (two FMAs fewer) was measured and dropped: its coefficients,
// up to 15 with alternating signs, lose bits in FP32 Horner evaluation (1.3e-6 for
// x < 1.5) and moved the batch's charges from 3.9e-7 to 4.6e-7 e of FP64.
constexpr double kLog2e = 1.4426950408889634074;
constexpr double kSqrtLog2e = 1.2011224087864498;  // sqrt(log2 e)
__device__ __forceinline__ float erfc_nr2(float xs) {
    const float t = rcp_ftz(fmaf((float)(0.5 / kSqrtLog2e), xs, 1.0f));
    float p = (float)(kLog2e * 0.17087277);
    p = fmaf(t, p, (float)(kLog2e * -0.82215223));
    p = fmaf(t, p, (float)(kLog2e * 1.48851587));
    p = fmaf(t, p, (float)(kLog2e * -1.13520398));
    p = fmaf(t, p, (float)(kLog2e * 0.27886807));
    p = fmaf(t, p, (float)(kLog2e * -0.18628806));
    p = fmaf(t, p, (float)(kLog2e * 0.09678418));
    p = fmaf(t, p, (float)(kLog2e * 0.37409196));
    p = fmaf(t, p, (float)(kLog2e * 1.00002368));
    p = fmaf(t, p, (float)(kLog2e * -1.26551223));
    return t * ex2_ftz(fmaf(-xs, xs, p));
}

__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, dup2(-1.0f), a); }  // one rounding, as a - b
// a + b as s + e exactly, both halves (dfa::two_sum)
__device__ __forceinline__ void two_sum2(f2 a, f2 b, f2 &s, f2 &e) {
    s = add2(a, b);
    const f2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

// erfc_nr2 of two arguments: the same operations in the same order.  The polynomial is carried with
// the opposite sign, which changes no rounding: xs^2 - p is then one packed multiply-add, and
// the exponential instruction negates its operand.  Its steps are scalar: a packed step issues
// once but holds its pipe as long as the two scalar ones, and its coefficients would take a
// register pair each, where the scalar steps carry them in the instruction (302 us against
// 308 us for 33 M pairs).
__device__ __forceinline__ f2 erfc_nr2x2(f2 xs) {
    float u, v, tu, tv;
    unpack2(fma2(dup2((float)(0.5 / kSqrtLog2e)), xs, dup2(1.0f)), u, v);
    tu = rcp_ftz(u);
    tv = rcp_ftz(v);
    float pu = -(float)(kLog2e * 0.17087277), pv = pu;
    auto step = [&](float c) {
        pu = fmaf(tu, pu, c);
        pv = fmaf(tv, pv, c);
    };
    step(-(float)(kLog2e * -0.82215223));
    step(-(float)(kLog2e * 1.48851587));
    step(-(float)(kLog2e * -1.13520398));
    step(-(float)(kLog2e * 0.27886807));
    step(-(float)(kLog2e * -0.18628806));
    step(-(float)(kLog2e * 0.09678418));
    step(-(float)(kLog2e * 0.37409196));
    step(-(float)(kLog2e * 1.00002368));
    step(-(float)(kLog2e * -1.26551223));
    unpack2(fma2(xs, xs, pack2(pu, pv)), u, v);
    return mul2(pack2(tu, tv), pack2(ex2_ftz(-u), ex2_ftz(-v)));
}
// min(m, |a|, |b|): the three-operand minimum
__device__ __forceinline__ float min3_abs(float m, float a, float b) {
    float r;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
    return r;
}

constexpr int kPhiPts = 128;                  // points per CTA, two consecutive ones per thread
constexpr int kPhiThreads = kPhiPts / 2;
constexpr int kPhiWarps = kPhiThreads / 32;
constexpr int kPhiAtoms = 32;    // most atoms per CTA (phi_atoms_per_cta)
// Staged E values (KMAX 7): 60 words for the four atoms of a run (a run: consecutive points of one
// grid row) while a tile has at most 32 runs, 28 words for two atoms up to 64 runs, else 14 for one.
// The strides put the reads of 8 (16 for one atom) consecutive runs on distinct banks.
constexpr int kEBytes = 7680;
constexpr int kMaxShifts = 128;  // pruned real-space shifts (checked on the host)

// The reference's FP64 cutoff decision for one (point, image) pair (repeat.py:944-966:
// r = |g - (a + s)| with g = (i a0 + j a1) + k a2, r <= Rc, the self image skipped at
// r <= 1e-10).  Returns 0 (outside), 1 (inside: the caller adds the FP32 term) or, with
// full = true, 2 and the FP64 term as a double-float (th, tl).  Not inlined on purpose:
// it runs for a few pairs in a million, and inlined the compiler may evaluate it
// speculatively for every pair on the slow FP64 pipe.
__device__ __noinline__ int fp64_pair(const double *axis, int i, int j, int k, const double *p,
                                      const double *shifts, int s, int zero_idx, double rc, double sa, bool full,
                                      float &th, float &tl) {
    double g[3];
    for (int d = 0; d < 3; ++d) g[d] = ((double)i * axis[d] + (double)j * axis[3 + d]) + (double)k * axis[6 + d];
    const double ex = g[0] - (p[0] + shifts[3 * s]), ey = g[1] - (p[1] + shifts[3 * s + 1]),
                 ez = g[2] - (p[2] + shifts[3 * s + 2]);
    const double r = sqrt(ex * ex + ey * ey + ez * ez);
    if (!(r <= rc) || (s == zero_idx && !(r > 1e-10))) return 0;
    if (!full) return 1;
    const double t = erfc(sa * r) / r;
    th = (float)t;
    tl = (float)(t - (double)th);
    return 2;
}

// Image positions atom + shift as double-float, [N][S] x {hi (x, y, z, shift index), lo}
__global__ void images_df_kernel(const double *__restrict__ atoms, int N, const double *__restrict__ shifts, int S,
                                 float4 *__restrict__ img) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * S) return;
    const int a = t / S, s = t - a * S;
    double q[3];
    for (int d = 0; d < 3; ++d) q[d] = atoms[3 * a + d] + shifts[3 * s + d];
    const float hx = (float)q[0], hy = (float)q[1], hz = (float)q[2];
    img[2 * t] = make_float4(hx, hy, hz, __int_as_float(s));
    img[2 * t + 1] = make_float4((float)(q[0] - (double)hx), (float)(q[1] - (double)hy), (float)(q[2] - (double)hz), 0.f);
}

// (ah + al) - (bh + bl) as a normalised double-float
__device__ __forceinline__ float2 df_sub(float ah, float al, float bh, float bl) {
    float s, e;
    dfa::two_sum(ah, -bh, s, e);
    e = __fadd_rn(e, __fadd_rn(al, -bl));
    const float h = __fadd_rn(s, e);
    return make_float2(h, __fadd_rn(e, -__fadd_rn(h, -s)));
}

// Phi_t[a][m] = sum over the images of atom a within Rc of erfc(sqrt(alpha) r)/r
//             + Re sum_n1 ex[n1][i_m] E[r_m][a][n1],   stored as double-float (hi, lo).
// Real space (repeat.py:944-966): the CTA first culls the images of its atoms to
// those within Rc + 1e-3 Bohr of the bounding box of its points, in shift order
// (warp-ballot compaction, so the summation order is fixed).  Distances are formed
// in FP32 from double-float coordinates relative to the CTA's first point; images
// within 2e-6 of Rc are decided in FP64 with the reference's expressions (the term
// is the FP32 one), pairs closer than sqrt(near2) are evaluated entirely in FP64,
// the rest with FP32 erfcf.  Reciprocal part: stage C of the
// separable sum in FP32.  `parts`: bit 0 real space, bit 1 reciprocal.
// With psum/pmax given, the CTA also writes each atom's sum and max |Phi| over its
// points (fixed-order reductions), the column statistics of the centring step.
// The grid step vectors as double-float (a[d] = h[d] + l[d]), passed by value.
struct AxisDF {
    float h[9], l[9];
};

// k * (ah + al) for two small integers k, each as an unevaluated pair (p, e)
__device__ __forceinline__ void int_times_df2(f2 k, float ah, float al, f2 &p, f2 &e) {
    p = mul2(k, dup2(ah));
    e = fma2(k, dup2(ah), mul2(p, dup2(-1.0f)));
    e = fma2(k, dup2(al), e);
}

// Digit output of the Phi kernel (single pass): instead of Phi_t, the kernel writes the
// four fixed-point digit slices of X rows a0..a0+na-1 (x = Phi * scale_a, centre 0) and,
// from the CTAs of the first atom block, the ESP row N (x = Vc * scale_V); columns
// rows..rows_kpad-1 get zero digits.  Exact row sums go to rowsum (one atomic per CTA
// and row), values beyond |x| = 1 are clamped and counted in *clamped.
struct PhiDigits {
    __half *X;            // slice 0, rows of rows_kpad points
    long long slice;      // elements from one slice to the next
    long long rows_kpad;  // points per row (the chunk padded to the Gram's K step)
    const float *scale;   // per atom, a power of two
    const double *Vc;     // the chunk's centred ESP
    const double *vmax_p; // max |Vc| (the ESP row scale)
    unsigned long long *rowsum;
    int *clamped;
    int N;
};

// The images of one atom that the real-space loop skipped for one point (half u of the packed
// coordinates): decided in FP64 (fp64_pair), in table order, added to the loop's sum `acc32`.
// Returns the sum as a double-float (s, e).  A few points in a million run it.
__device__ __noinline__ void real_special(int f, int u, const f2 (&gh)[3], const f2 (&gl)[3], const float4 *tab,
                                          const unsigned short *items, int nc, float fp64_below, float r2_in,
                                          float r2_out, float saf, const double *axis, int nx, int ny,
                                          const double *p, const double *shifts, int zero_idx, double rc, double sa,
                                          float acc32, float &s, float &e) {
    float h[3], lo[3];
    for (int d = 0; d < 3; ++d) {
        float a, b;
        unpack2(gh[d], a, b);
        h[d] = u ? b : a;
        unpack2(gl[d], a, b);
        lo[d] = u ? b : a;
    }
    const int row = f / nx, i = f - row * nx, l = row / ny, j = row - l * ny;
    float x64h = 0.f, x64l = 0.f;  // rare FP64 terms, folded in as double-float pairs
    for (int c = 0; c < nc; ++c) {
        const float4 t0 = tab[3 * c], t1 = tab[3 * c + 1], t2 = tab[3 * c + 2];
        const float dx = __fadd_rn(__fadd_rn(h[0], t0.x), __fadd_rn(lo[0], t1.z));
        const float dy = __fadd_rn(__fadd_rn(h[1], t0.z), __fadd_rn(lo[1], t2.x));
        const float dz = __fadd_rn(__fadd_rn(h[2], t1.x), __fadd_rn(lo[2], t2.z));
        const float r2 = fmaf(dz, dz, fmaf(dx, dx, __fmul_rn(dy, dy)));
        if (!(r2 < fp64_below || (r2 > r2_in && r2 <= r2_out))) continue;
        float th, tl;
        const int dec = fp64_pair(axis, i, j, l, p, shifts, items[c] & 127, zero_idx, rc, sa, r2 < fp64_below, th, tl);
        if (dec == 1) {  // inside the cutoff: the FP32 term
            const float rinv = rsqrt_ftz(r2);
            acc32 = fmaf(erfc_nr2(saf * (r2 * rinv)), rinv, acc32);
        } else if (dec == 2) {  // a point on top of an image: the large term in FP64
            float s2, e2;
            dfa::two_sum(x64h, th, s2, e2);
            x64h = s2;
            x64l = __fadd_rn(x64l, __fadd_rn(e2, tl));
        }
    }
    float s_, e_;
    dfa::two_sum(acc32, x64h, s_, e_);
    s = s_;
    e = __fadd_rn(e_, x64l);
}

// max(|a|, |b|), NaN if either is
__device__ __forceinline__ float max_abs_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(fabsf(a)), "f"(fabsf(b)));
    return r;
}

// The digits of two consecutive points of one row.  I = round(x 2^27), x = (h + l) sc, comes as
// hi 2^14 + lo without conversion instructions (a quarter of the rate): adding 1.5 2^37 and
// 1.5 2^23 rounds to multiples of 2^14 and of 1 (to nearest even, as rintf), and the integers
// are read off the sums' bits; the remainder after the integer part is exact, and the low
// part decides the last unit.  |hi|, |lo| <= 2^13 (+ 5), so with 64 (1 + 2^7) added each half
// holds two digits as a 7-bit field below an 8-bit one, every digit 64 too large: the digits
// of split4 up to a carry where that one gives another 64, the same value.  A field u under
// the bits of 1024 is the FP16 number 1024 + u, and subtracting 1088 gives the digit exactly.
// Returns the two biased sums hi, lo (without the points past the end) for the row sum.
constexpr int kHalfBias = 64 * (1 + (1 << 7));
__device__ __forceinline__ void digit_halves2(f2 h, f2 l, float sc, int full, bool valid0, bool valid1, int *clamped,
                                              int &hi0, int &hi1, int &lo0, int &lo1) {
    constexpr float kM1 = 206158430208.0f, kM0 = 12582912.0f;  // 1.5 2^37, 1.5 2^23
    constexpr int kB1 = 0x52400000, kB0 = 0x4b400000;          // their bits
    constexpr float kTop = 134217728.0f;                       // 2^27
    const f2 sc2 = dup2(sc * kTop);
    const f2 H = mul2(h, sc2), L = mul2(l, sc2);
    const f2 a1 = add2(H, dup2(kM1));
    const f2 r = sub2(H, add2(a1, dup2(-kM1)));
    const f2 a0 = add2(r, dup2(kM0));
    const f2 b0 = add2(add2(sub2(r, add2(a0, dup2(-kM0))), L), dup2(kM0));
    float hu, hv, pu, pv, qu, qv, ru, rv;
    unpack2(H, hu, hv);
    unpack2(a1, pu, pv);
    unpack2(a0, qu, qv);
    unpack2(b0, ru, rv);
    hi0 = __float_as_int(pu) + (kHalfBias - kB1);
    hi1 = __float_as_int(pv) + (kHalfBias - kB1);
    lo0 = __float_as_int(qu) + __float_as_int(ru) + (int)((unsigned)kHalfBias - 2u * (unsigned)kB0);
    lo1 = __float_as_int(qv) + __float_as_int(rv) + (int)((unsigned)kHalfBias - 2u * (unsigned)kB0);
    if (!full) {  // the last tile: points past the end are zero
        if (!valid0) hi0 = lo0 = kHalfBias;
        if (!valid1) hi1 = lo1 = kHalfBias;
    }
    if (!(max_abs_nan(hu, hv) <= kTop)) {  // |x| beyond 1: clamp (counted; the fit is redone); a NaN gives 0
        if (valid0 && !(fabsf(hu) <= kTop)) {
            hi0 = kHalfBias + (hu > 0.f ? 8192 : hu < 0.f ? -8192 : 0);
            lo0 = kHalfBias;
        }
        if (valid1 && !(fabsf(hv) <= kTop)) {
            hi1 = kHalfBias + (hv > 0.f ? 8192 : hv < 0.f ? -8192 : 0);
            lo1 = kHalfBias;
        }
        const int n = (valid0 && fabsf(hu) > kTop) + (valid1 && fabsf(hv) > kTop);
        if (n) atomicAdd(clamped, n);
    }
}
__device__ __forceinline__ void store_digits2(__half *x, long long slice, int hi0, int hi1, int lo0, int lo1) {
    const unsigned hp = __byte_perm(hi0, hi1, 0x5410), lp = __byte_perm(lo0, lo1, 0x5410);
    const __half2 off = __half2half2(__ushort_as_half((unsigned short)0x6440));  // 1088
    auto put = [&](int q, unsigned v) {
        *reinterpret_cast<__half2 *>(x + q * slice) = __hsub2(*reinterpret_cast<const __half2 *>(&v), off);
    };
    put(0, ((hp >> 7) & 0x00ff00ffu) | 0x64006400u);
    put(1, (hp & 0x007f007fu) | 0x64006400u);
    put(2, ((lp >> 7) & 0x00ff00ffu) | 0x64006400u);
    put(3, (lp & 0x007f007fu) | 0x64006400u);
}
// The warp's exact sum of I over its points from the biased halves (32-bit sums below 2^21)
__device__ __forceinline__ long long warp_sum_halves2(int hi0, int hi1, int lo0, int lo1) {
    const int shi = __reduce_add_sync(0xffffffffu, hi0 + hi1) - 64 * kHalfBias;
    const int slo = __reduce_add_sync(0xffffffffu, lo0 + lo1) - 64 * kHalfBias;
    return (long long)shi * 16384 + slo;
}

// x / d for 0 <= x < 2^31 by a multiplication (d's reciprocal rounded up, computed on the host)
struct FastDiv {
    unsigned mul;
    int shift;
};
__device__ __forceinline__ int fast_div(int x, FastDiv f) {
    return (int)(((unsigned long long)(unsigned)x * f.mul) >> f.shift);
}

// One thread handles two consecutive points (2t, 2t + 1 of the CTA's 128), packed where that
// helps: the table loads, the loop and the digit stores serve two points and most FP32
// operations of the real-space term issue once for both.  Each point's value is computed by
// the same operations in the same order as one at a time.
// What bounds it: the issue of instructions and the latencies between them (16 warps per SM at
// 128 registers; 96 registers and 20 warps spill and took 381 us against 302).  On 273 atoms x
// 121k points (33 M pairs): 287 us, 203 thread instructions per pair, against 360 us and 344 for
// one point per thread with the E values loaded per point and 16 atoms per CTA.
// NC = 7: the number of n1 terms (the reference's KMAX) is a compile-time constant: the points'
// phases ex stay in registers, and the E values of up to four atoms at a time are copied to
// shared memory (asynchronously, one stage ahead), once per run of points in the same grid
// row: loaded per point, they took 112 of ~160 L1 wavefronts per 64 points and atom.
// NC = 0: any KMAX, phases in shared memory and E read in the loop.
template <int NC, bool DIG>
__global__ void __launch_bounds__(kPhiThreads, 8) phi_chunk_kernel(
    const int32_t *__restrict__ kept, long long m0, long long rows, const double *__restrict__ axis, AxisDF adf,
    int nx, int ny,
    FastDiv dnx, FastDiv dny, const double *__restrict__ atoms, int N, const double *__restrict__ shifts, int S, int per_cta, int slots, int zero_idx,
    double rc, double sa, float rcf, float saf, float near2, const float4 *__restrict__ img,
    const float4 *__restrict__ EX,
    const float2 *__restrict__ E, int n1c, int parts, float2 *__restrict__ phit, long long ld,
    double *__restrict__ psum, float *__restrict__ pmax, PhiDigits dg) {
    static_assert(NC == 0 || NC == 7, "the E stages are laid out for KMAX 7");
    // Image table, `slots` entries (each warp fills one half): the negated double-float position
    // relative to the CTA origin with every value twice, (-x, -x, -y, -y), (-z, -z, -xl, -xl),
    // (-yl, -yl, -zl, -zl), the packed operands of both points; NC = 7: two stages of E values;
    // NC = 0: ex[n1][i] of the points, (re, re, im, im) per pair; then the entries'
    // (atom << 7) | shift.
    extern __shared__ ulonglong2 dsm[];
    ulonglong2 *tab = dsm;
    char *es = reinterpret_cast<char *>(tab + 3 * (size_t)slots);       // NC = 7: [2][kEBytes]
    float4 *exs = reinterpret_cast<float4 *>(tab + 3 * (size_t)slots);  // NC = 0: [n1c][kPhiThreads]
    unsigned short *items = reinterpret_cast<unsigned short *>(
        NC > 0 ? es + 2 * kEBytes : reinterpret_cast<char *>(exs + (size_t)n1c * kPhiThreads));
    __shared__ int start[kPhiAtoms];        // an atom's first entry
    __shared__ int cand[kPhiAtoms];         // (first entry << 9) | (near << 8) | entries
    __shared__ int close[kPhiAtoms];        // an image near or inside the points' box
    __shared__ int filled[kPhiWarps];  // end of each warp's entries
    __shared__ float scl[kPhiAtoms];        // digit scales (DIG)
    __shared__ float bb[2][3][kPhiWarps];
    __shared__ float wsum[kPhiPts / 32][DIG ? 1 : kPhiAtoms];
    __shared__ float wmax[kPhiPts / 32][DIG ? 1 : kPhiAtoms];
    __shared__ long long wrow[kPhiWarps][kPhiAtoms + 1];  // digit-row partial sums (DIG)
    __shared__ long long run_off[NC > 0 ? kPhiPts : 1];  // byte offset of each run's E row
    __shared__ int wruns[kPhiWarps];
    const long long mb = (long long)blockIdx.x * kPhiPts;
    const int a0 = blockIdx.y * per_cta;
    const int na = min(per_cta, N - a0);
    const int Ne = (N + 1) & ~1;  // E's columns per row
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long m = mb + 2 * threadIdx.x;
    const bool valid0 = m < rows, valid1 = m + 1 < rows;

    // CTA origin: the first point of the tile (FP64 once, shared as a double-float)
    __shared__ float org[6];
    __shared__ int org_idx[3];
    if (threadIdx.x < 3) {
        const int d = threadIdx.x, f0 = kept[m0 + mb];
        const int q = fast_div(f0, dnx), i0 = f0 - q * nx, l0 = fast_div(q, dny), j0 = q - l0 * ny;
        const double o = ((double)i0 * axis[d] + (double)j0 * axis[3 + d]) + (double)l0 * axis[6 + d];
        org[d] = (float)o;
        org[3 + d] = (float)(o - (double)org[d]);
        org_idx[d] = d == 0 ? i0 : d == 1 ? j0 : l0;
    }
    if (DIG && threadIdx.x < na) scl[threadIdx.x] = dg.scale[a0 + threadIdx.x];
    __syncthreads();
    // a point past the end repeats the tile's first point
    const int f0 = kept[m0 + (valid0 ? m : mb)], f1 = kept[m0 + (valid1 ? m + 1 : mb)];
    const int row0 = fast_div(f0, dnx), row1 = fast_div(f1, dnx);  // grid rows j + l ny
    // point - origin = di a0 + dj a1 + dl a2 with small integers: double-float on the FP32 pipe
    f2 gh[3], gl[3];
    {
        const int l0 = fast_div(row0, dny), l1 = fast_div(row1, dny);
        const f2 di = pack2((float)(f0 - row0 * nx - org_idx[0]), (float)(f1 - row1 * nx - org_idx[0])),
                 dj = pack2((float)(row0 - l0 * ny - org_idx[1]), (float)(row1 - l1 * ny - org_idx[1])),
                 dl = pack2((float)(l0 - org_idx[2]), (float)(l1 - org_idx[2]));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            f2 p0, e0, p1, e1, p2, e2, s, t, s2, t2;
            int_times_df2(di, adf.h[d], adf.l[d], p0, e0);
            int_times_df2(dj, adf.h[3 + d], adf.l[3 + d], p1, e1);
            int_times_df2(dl, adf.h[6 + d], adf.l[6 + d], p2, e2);
            two_sum2(p0, p1, s, t);
            two_sum2(s, p2, s2, t2);
            const f2 e = add2(add2(add2(e0, e1), e2), add2(t, t2));
            gh[d] = add2(s2, e);
            gl[d] = sub2(e, sub2(gh[d], s2));
            float u, v;
            unpack2(gh[d], u, v);
            float mn = fminf(u, v), mx = fmaxf(u, v);
            for (int o = 16; o > 0; o >>= 1) {
                mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if (lane == 0) {
                bb[0][d][warp] = mn;
                bb[1][d][warp] = mx;
            }
        }
    }
    f2 xr[NC > 0 ? NC : 1], xi[NC > 0 ? NC : 1];  // ex[n1][i] of both points (n1 > 0)
    int slot0 = 0, slot1 = 0, nruns = 0;          // the points' runs
    if (NC > 0) {
        if (parts & 2) {
            const int i0 = f0 - row0 * nx, i1 = f1 - row1 * nx;
#pragma unroll
            for (int n = 1; n < (NC > 0 ? NC : 1); ++n) {
                const float4 x = EX[(long long)n * nx + i0], y = EX[(long long)n * nx + i1];
                xr[n] = pack2(x.x, y.x);
                xi[n] = pack2(x.z, y.z);
            }
        }
        int prev = __shfl_up_sync(0xffffffffu, row1, 1);
        if (lane == 0) prev = -1;  // a warp starts a run of its own
        const unsigned b0 = __ballot_sync(0xffffffffu, row0 != prev), b1 = __ballot_sync(0xffffffffu, row1 != row0);
        const unsigned lt = (1u << lane) - 1u, le = lt | (1u << lane);
        if (lane == 0) wruns[warp] = __popc(b0) + __popc(b1);
        __syncthreads();
        int base = 0;
        for (int w = 0; w < kPhiWarps; ++w) {
            if (w < warp) base += wruns[w];
            nruns += wruns[w];
        }
        slot0 = base + __popc(b0 & le) + __popc(b1 & lt) - 1;
        slot1 = base + __popc(b0 & le) + __popc(b1 & le) - 1;
        if (row0 != prev) run_off[slot0] = (long long)row0 * Ne * 56;
        if (row1 != row0) run_off[slot1] = (long long)row1 * Ne * 56;
    } else if (parts & 2) {
        const int i0 = f0 - row0 * nx, i1 = f1 - row1 * nx;
        for (int n = 0; n < n1c; ++n) {
            const float4 x = EX[(long long)n * nx + i0], y = EX[(long long)n * nx + i1];
            exs[n * kPhiThreads + threadIdx.x] = make_float4(x.x, y.x, x.z, y.z);
        }
    }
    __syncthreads();

    // FP64 decides every image whose FP32 squared distance lies within +-4e-6 Rc^2 of the
    // cutoff: with coordinates exact to ~2^-48, dx carries <= 2^-23 relative error and
    // r2 <= 2^-21 (4.8e-7), so the band covers the FP32 error 8-fold.  Only the decision
    // r <= Rc is made in FP64 (the reference's expressions); the term itself, ~erfc(pi)/Rc
    // there, is the FP32 one.  FP64 runs at 1/64 of the FP32 rate per lane on this part,
    // and one lane in the band makes its whole warp run the FP64 code, so it stays short.
    const float rcc = rcf * rcf, band = 4e-6f * rcc;  // saf: sqrt(alpha log2 e), the argument scale of erfc_nr2
    const float r2_in = rcc - band, r2_out = rcc + band;
    const float fp64_below = fmaxf(near2, 1e-6f);

    // The images of atoms r0 .. r0 + nr - 1 within Rc + 1e-3 Bohr of the points' bounding box: an
    // FP32 test per image (1e-4 Bohr more covers its rounding), each warp over the images of half
    // of the atoms 32 at a time, which lists the survivors, an atom's in shift order; then
    // their table entries.  An atom with an image near or inside the box is marked: only there
    // can a point be closer than sqrt(fp64_below) to an image.  False when a warp's list
    // overflows its half of the table.
    auto cull = [&](int r0, int nr) -> bool {
        if (threadIdx.x < kPhiAtoms) close[threadIdx.x] = 0;
        __syncthreads();
        float bmin[3], bmax[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bmin[d] = fminf(bb[0][d][0], bb[0][d][1]) + org[d];
            bmax[d] = fmaxf(bb[1][d][0], bb[1][d][1]) + org[d];
        }
        const float reach = rcf + 1.1e-3f, reach2 = reach * reach, near = 4.f * fp64_below;
        const int half = slots >> 1, na0 = (nr + 1) >> 1;
        const int wa = warp ? r0 + na0 : r0, wn = warp ? nr - na0 : na0;  // the warp's atoms
        const int step_a = 32 / S, step_s = 32 - step_a * S;
        int a = lane / S, sh = lane - a * S, base = 0;
        const float4 *src = img + 2 * ((size_t)(a0 + wa) * S + lane);
        for (int k0 = 0; k0 < wn * S; k0 += 32, src += 64) {
            bool keep = false;
            if (a < wn) {
                const float4 ph = *src;
                const float dx = fmaxf(fmaxf(bmin[0] - ph.x, ph.x - bmax[0]), 0.f);
                const float dy = fmaxf(fmaxf(bmin[1] - ph.y, ph.y - bmax[1]), 0.f);
                const float dz = fmaxf(fmaxf(bmin[2] - ph.z, ph.z - bmax[2]), 0.f);
                const float d2 = dx * dx + dy * dy + dz * dz;
                keep = d2 <= reach2;
                if (d2 <= near) close[wa + a] = 1;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            const int pos = base + __popc(bal & ((1u << lane) - 1u));
            if (sh == 0 && a < wn) start[wa + a] = warp * half + pos;
            if (keep && pos < half) items[warp * half + pos] = (unsigned short)(((wa + a) << 7) | sh);
            base += __popc(bal);
            a += step_a;
            sh += step_s;
            if (sh >= S) {
                sh -= S;
                ++a;
            }
        }
        if (lane == 0) filled[warp] = warp * half + base;
        const bool ok = !__syncthreads_or(base > half);
        if (ok) {
            for (int t = threadIdx.x; t < nr; t += kPhiThreads) {
                const int b = start[r0 + t];
                const int e = t + 1 == na0 ? filled[0] : t + 1 == nr ? filled[1] : start[r0 + t + 1];
                cand[r0 + t] = (b << 9) | (close[r0 + t] << 8) | (e - b);
            }
            for (int k = warp * half + lane; k < warp * half + base; k += 32) {
                const int it = items[k];
                const float4 *ps = img + 2 * ((size_t)(a0 + (it >> 7)) * S + (it & 127));
                const float4 ph = ps[0], pl = ps[1];
                const float2 qx = df_sub(ph.x, pl.x, org[0], org[3]), qy = df_sub(ph.y, pl.y, org[1], org[4]),
                             qz = df_sub(ph.z, pl.z, org[2], org[5]);
                ulonglong2 *t = tab + 3 * k;
                t[0] = make_ulonglong2(dup2(-qx.x), dup2(-qy.x));
                t[1] = make_ulonglong2(dup2(-qz.x), dup2(-qx.y));
                t[2] = make_ulonglong2(dup2(-qy.y), dup2(-qz.y));
            }
        }
        return ok;
    };

    // E values of atoms a .. a + n - 1 for every run into stage buffer b, run by run (the stride
    // above): 16 bytes a lane, two runs of four atoms (four of two) per warp instruction; E's rows
    // have an even number of columns, so a stage that starts at an even atom is aligned, and an
    // odd last atom takes half of the next column along.  One atom per stage: 8 bytes a lane.
    const int eb = nruns <= 32 ? 4 : nruns <= 64 ? 2 : 1;
    const int e_stride = eb == 4 ? 240 : eb == 2 ? 112 : 56;
    const int e_run = eb == 4 ? (lane >= 14) : lane / 7, e_chunk = lane - e_run * (eb == 4 ? 14 : 7);
    const int e_runs = eb == 4 ? 2 : 4, e_run0 = warp * e_runs + e_run, e_step = kPhiWarps * e_runs;
    const char *e_src = reinterpret_cast<const char *>(E + (long long)a0 * 7) + e_chunk * (eb > 1 ? 16 : 8);
    const uint32_t e_dst = tc::smem_u32(es) + e_run0 * e_stride + e_chunk * (eb > 1 ? 16 : 8);
    auto stage_e = [&](int a, int n, int b) {
        if (lane >= 28 || (eb > 1 ? 2 * e_chunk >= 7 * n : n <= 0)) return;
        const char *src = e_src + a * 56;
        uint32_t dst = e_dst + b * kEBytes;
        if (eb > 1) {
#pragma unroll 2
            for (int r = e_run0; r < nruns; r += e_step, dst += e_step * e_stride)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + run_off[r]) : "memory");
        } else {
#pragma unroll 1
            for (int r = e_run0; r < nruns; r += e_step, dst += e_step * e_stride)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src + run_off[r]) : "memory");
        }
    };

    int round = na;  // atoms whose images share one table
    if ((parts & 1) && !cull(0, na)) round = 2 * ((slots >> 1) / S);
    const float2 *erow0 = E + ((long long)row0 * Ne + a0) * n1c, *erow1 = E + ((long long)row1 * Ne + a0) * n1c;
    const int full = mb + kPhiPts <= rows;
    __half *xp = DIG ? dg.X + a0 * dg.rows_kpad + m : nullptr;
    const bool stores = DIG && m < dg.rows_kpad;
    int e_buf = 0;
    if (NC > 0) {
        if (parts & 2) stage_e(0, min(eb, min(round, na)), 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int r0 = 0; r0 < na; r0 += round) {
        const int r1 = min(r0 + round, na);
        __syncthreads();  // the first round's table is complete; a later round: the one before has been read
        if (round < na && (parts & 1)) {
            cull(r0, r1 - r0);
            __syncthreads();
        }
      for (int e_lo = r0; e_lo < r1;) {
        const int e_hi = NC > 0 ? min(e_lo + eb, r1) : r1;
        if (NC > 0) {  // this stage has landed, and every warp is done with the buffer of the next
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (parts & 2) stage_e(e_hi, min(eb, (e_hi < r1 ? r1 : min(r1 + round, na)) - e_hi), e_buf ^ 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const char *ep = es + e_buf * kEBytes + slot0 * e_stride;
        const int eq = (slot1 - slot0) * e_stride;
        for (int a = e_lo; a < e_hi; ++a, ep += 56) {
            f2 acc = 0ull;
            float edge = 3e38f;  // the smallest | r^2 - Rc^2 |
            bool spec = false;
            const int ci = cand[a];
            const ulonglong2 *t = tab + 3 * (ci >> 9);
            // Branch-free over the candidates: most of them are inside the cutoff for some lane of
            // the warp, so the term is computed for all and selected.  Images whose decision needs
            // FP64 (within the band around Rc, or on top of the point) are skipped here and taken
            // in a second pass, which a warp runs only when one of its lanes met one.  (A per-warp
            // ballot mask over the tile's candidates, which skips images out of the warp's reach,
            // measured 3 % more instructions: the mask costs more than the images it drops.)
            auto real_space = [&](auto low) {
                const f2 saf2 = dup2(saf), rcc2 = dup2(-rcc);
#pragma unroll 2
                for (int c = ci & 255; c > 0; --c, t += 3) {
                    const ulonglong2 t0 = t[0], t1 = t[1], t2 = t[2];
                    const f2 dx = add2(add2(gh[0], t0.x), add2(gl[0], t1.y));
                    const f2 dy = add2(add2(gh[1], t0.y), add2(gl[1], t2.x));
                    const f2 dz = add2(add2(gh[2], t1.x), add2(gl[2], t2.y));
                    const f2 r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
                    float ra, rb, va, vb, aa, ab, da, db;
                    unpack2(r2, ra, rb);
                    unpack2(add2(r2, rcc2), da, db);
                    edge = min3_abs(edge, da, db);
                    bool oka = ra <= r2_in, okb = rb <= r2_in;
                    if (decltype(low)::value) {
                        oka = oka && ra >= fp64_below;
                        okb = okb && rb >= fp64_below;
                        spec |= ra < fp64_below || rb < fp64_below;
                    }
                    const f2 rinv = pack2(rsqrt_ftz(ra), rsqrt_ftz(rb));
                    const f2 v = fma2(erfc_nr2x2(mul2(saf2, mul2(r2, rinv))), rinv, acc);
                    unpack2(v, va, vb);
                    unpack2(acc, aa, ab);
                    acc = pack2(oka ? va : aa, okb ? vb : ab);
                }
            };
            if (parts & 1) {
                if (ci & 256) real_space(std::true_type{});
                else real_space(std::false_type{});
                spec |= edge <= band * 1.01f;  // every image of the band (r2_in, r2_out], and at most a few more
            }
            float ru = 0.f, rv = 0.f;  // stage C: Re sum_n1 ex[n1][i] E[row][a][n1]
            if (parts & 2) {
                if (NC > 0) {
                    const float2 *p = reinterpret_cast<const float2 *>(ep), *q = reinterpret_cast<const float2 *>(ep + eq);
                    ru = p[0].x;  // ex[0] = 1
                    rv = q[0].x;
#pragma unroll
                    for (int n = 1; n < (NC > 0 ? NC : 1); ++n) {
                        const float2 y = p[n], z = q[n];
                        float xa, xb, ya, yb;
                        unpack2(xr[n], xa, xb);
                        unpack2(xi[n], ya, yb);
                        ru = fmaf(xa, y.x, ru);
                        rv = fmaf(xb, z.x, rv);
                        ru = fmaf(-ya, y.y, ru);
                        rv = fmaf(-yb, z.y, rv);
                    }
                } else {
                    const float2 *p = erow0 + (long long)a * n1c, *q = erow1 + (long long)a * n1c;
                    for (int n = 0; n < n1c; ++n) {
                        const float4 x = exs[n * kPhiThreads + threadIdx.x];
                        const float2 y = p[n], z = q[n];
                        ru = fmaf(x.x, y.x, ru);
                        rv = fmaf(x.y, z.x, rv);
                        ru = fmaf(-x.z, y.y, ru);
                        rv = fmaf(-x.w, z.y, rv);
                    }
                }
            }
            f2 oh, ol;  // Phi as a double-float: the sum of the two parts, exactly
            two_sum2(acc, pack2(ru, rv), oh, ol);
            if (__any_sync(0xffffffffu, spec)) {
                float as[2], hh[2], ll[2];
                unpack2(acc, as[0], as[1]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    float s_, ve, s2, e2;
                    real_special(u ? f1 : f0, u, gh, gl, reinterpret_cast<const float4 *>(tab + 3 * (ci >> 9)),
                                 items + (ci >> 9), ci & 255, fp64_below, r2_in, r2_out, saf, axis, nx, ny,
                                 atoms + 3 * (a0 + a), shifts, zero_idx, rc, sa, as[u], s_, ve);
                    dfa::two_sum(s_, u ? rv : ru, s2, e2);
                    const float2 o = dfa::norm(dfa::acc{s2, __fadd_rn(ve, e2)});
                    hh[u] = o.x;
                    ll[u] = o.y;
                }
                oh = pack2(hh[0], hh[1]);
                ol = pack2(ll[0], ll[1]);
            }
            if (DIG) {
                int hi0, hi1, lo0, lo1;
                digit_halves2(oh, ol, scl[a], full, valid0, valid1, dg.clamped, hi0, hi1, lo0, lo1);
                const long long rsum = warp_sum_halves2(hi0, hi1, lo0, lo1);
                if (lane == 0) wrow[warp][a] = rsum;
                if (stores) store_digits2(xp, dg.slice, hi0, hi1, lo0, lo1);
                xp += dg.rows_kpad;
            } else {
                float h0, h1, l0, l1;
                unpack2(oh, h0, h1);
                unpack2(ol, l0, l1);
                float2 *p = phit + (long long)(a0 + a) * ld + m;
                if (valid0) p[0] = make_float2(h0, l0);
                if (valid1) p[1] = make_float2(h1, l1);
                if (psum) {  // column statistics for the centre and the scale: FP32 is enough (any
                             // centre is corrected exactly; the max is exact); 32 points at a time
                    float s0 = valid0 ? h0 : 0.f, s1 = valid1 ? h1 : 0.f;
                    float mx = fmaxf(valid0 ? fabsf(h0) : 0.f, valid1 ? fabsf(h1) : 0.f);
                    for (int o = 8; o > 0; o >>= 1) {
                        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    }
                    if ((lane & 15) == 0) {
                        wsum[2 * warp + (lane >> 4)][a] = s0 + s1;
                        wmax[2 * warp + (lane >> 4)][a] = mx;
                    }
                }
            }
        }
        e_lo = e_hi;
        e_buf ^= 1;
      }
    }
    if (DIG) {
        // the ESP row, from the CTAs of the first atom block
        if (blockIdx.y == 0) {
            float h[2] = {0.f, 0.f}, l[2] = {0.f, 0.f};
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (u ? valid1 : valid0) {
                    const double v = dg.Vc[m + u];
                    h[u] = (float)v;
                    l[u] = (float)(v - (double)h[u]);
                }
            int hi0, hi1, lo0, lo1;
            digit_halves2(pack2(h[0], h[1]), pack2(l[0], l[1]), vscale_of(*dg.vmax_p), full, valid0, valid1, dg.clamped,
                          hi0, hi1, lo0, lo1);
            const long long rsum = warp_sum_halves2(hi0, hi1, lo0, lo1);
            if (lane == 0) wrow[warp][kPhiAtoms] = rsum;
            if (stores) store_digits2(dg.X + dg.N * dg.rows_kpad + m, dg.slice, hi0, hi1, lo0, lo1);
        }
        __syncthreads();
        // exact row sums (two's complement int64 atomics: order-independent), one per CTA and row
        if (threadIdx.x < na || (blockIdx.y == 0 && threadIdx.x == kPhiAtoms)) {
            const int a = threadIdx.x;
            long long t = 0;
            for (int w = 0; w < kPhiWarps; ++w) t += wrow[w][a];
            if (t != 0) atomicAdd(dg.rowsum + (a == kPhiAtoms ? dg.N : a0 + a), (unsigned long long)t);
        }
    } else if (psum) {
        __syncthreads();
        if (threadIdx.x < na) {
            const int a = threadIdx.x;
            double s = 0.0;
            float mx = 0.f;
            for (int w = 0; w < kPhiPts / 32; ++w) {
                s += (double)wsum[w][a];
                mx = fmaxf(mx, wmax[w][a]);
            }
            psum[(size_t)(a0 + a) * gridDim.x + blockIdx.x] = s;
            pmax[(size_t)(a0 + a) * gridDim.x + blockIdx.x] = mx;
        }
    }
}

// Slots of the image table: about 1.4 times the images within Rc of a tile for all the CTA's
// atoms (a tile that reaches more goes through its atoms in rounds), at least one atom's S for
// each warp's half.
int phi_slots(int S, int at, double rc, double volume) {
    const double images = std::min<double>(S, 4.18879 * (rc + 3.0) * (rc + 3.0) * (rc + 3.0) / std::max(volume, 1.0));
    const double want = std::min(1.4 * at * images + 32.0, 640.0);
    return 2 * (int)(std::min<double>((double)at * S, std::max<double>(2.0 * S, want)) / 2.0 + 0.5);
}
// d's multiplier: ceil(2^(31 + s) / d), s = ceil(log2 d), exact for dividends below 2^31
FastDiv fast_div_of(int d) {
    int s = 0;
    while ((1ll << s) < d) ++s;
    return FastDiv{(unsigned)(((1ull << (31 + s)) + d - 1) / d), 31 + s};
}
size_t phi_smem_bytes(int n1c, bool regs, int slots) {
    const size_t e = regs ? 2 * (size_t)kEBytes : sizeof(float4) * (size_t)n1c * kPhiThreads;
    return sizeof(ulonglong2) * 3 * (size_t)slots + e + (sizeof(unsigned short) * (size_t)slots + 15) / 16 * 16;
}

// Atoms per CTA: the largest even split of the atoms into blocks of at most `cap` (32: a CTA's
// start costs as much as 2.5 atoms of its loop; 0.293 ms with 32 atoms, 0.308 with 16 and 0.334
// with 8 on 273 atoms and 121k points), into more blocks, of at least 8, while the CTAs
// would not fill the GPU four times over.
int phi_atoms_per_cta(int N, long long tiles, int cap, int resident) {
    int blocks = (int)ceil_div(N, cap);
    while (tiles * blocks < 4LL * resident && (int)ceil_div(N, blocks + 1) >= 8) ++blocks;
    const int a = (int)ceil_div(N, blocks);
    return (a + 1) & ~1;
}

// The instantiation for (KMAX 7 or any, digits or staged Phi)
using PhiKernel = decltype(&phi_chunk_kernel<7, false>);
PhiKernel phi_kernel(bool regs, bool dig) {
    return dig ? (regs ? phi_chunk_kernel<7, true> : phi_chunk_kernel<0, true>)
               : (regs ? phi_chunk_kernel<7, false> : phi_chunk_kernel<0, false>);
}

void launch_phi(const int32_t *kept, long long m0, long long rows, const double *d_axis, const double *h_axis,
                const double *h_box, int nx, int ny,
                const double *d_atoms, int N, const double *d_shifts, int S, int zero_idx, double rc, double sa,
                const float4 *img, const float4 *EX, const float2 *E, int n1c, int parts, float2 *phit, long long ld,
                double *psum, float *pmax, const PhiDigits *dig, cudaStream_t s, int cap, int sm_count) {
    if (cap != 8 && cap != 16) cap = 32;
    RP_REQUIRE(S >= 1 && S <= kMaxShifts, "more than 128 real-space shifts after pruning (cutoff too large for the cell)");
    const bool regs = (n1c == 7);  // KMAX 7: the specialised kernel
    const double *b = h_box;
    const double vol = std::fabs(b[0] * (b[4] * b[8] - b[5] * b[7]) - b[1] * (b[3] * b[8] - b[5] * b[6]) +
                                 b[2] * (b[3] * b[7] - b[4] * b[6]));
    const int at = phi_atoms_per_cta(N, ceil_div(rows, kPhiPts), cap, 8 * std::max(1, sm_count));
    const int slots = phi_slots(S, at, rc, vol);
    const size_t smem = phi_smem_bytes(n1c, regs, slots);
    RP_REQUIRE(smem <= 192 * 1024, "phi kernel: KMAX too large for shared memory");
    auto kern = phi_kernel(regs, dig != nullptr);
    smem_optin((const void *)kern, std::max<size_t>(smem, 96 * 1024));
    AxisDF adf;
    for (int q = 0; q < 9; ++q) {
        adf.h[q] = (float)h_axis[q];
        adf.l[q] = (float)(h_axis[q] - (double)adf.h[q]);
    }
    dim3 grd(ceil_div(rows, kPhiPts), ceil_div(N, at));
    const PhiDigits dg = dig ? *dig : PhiDigits{};
    kern<<<grd, kPhiThreads, smem, s>>>(kept, m0, rows, d_axis, adf, nx, ny, fast_div_of(nx), fast_div_of(ny), d_atoms, N, d_shifts, S, at,
                                        slots, zero_idx, rc, sa, (float)rc,
                                        (float)(sa * kSqrtLog2e), real_near2(), img, EX, E, n1c, parts, phit, ld, psum,
                                        pmax, dg);
    RP_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ column statistics and the split

// Per atom (one warp each), on the first chunk: the centre c (the chunk mean, as a
// double-float; cvec holds its exact FP64 value) and the power-of-two scale, from the
// phi kernel's per-CTA partial sums and maxima.  Any centre works: the mean correction
// uses the exact sums of the fixed-point rows (slice_rows_kernel).
__global__ void colstats_finish_kernel(const double *__restrict__ psum, const float *__restrict__ pmax, int nblk,
                                       int N, long long rows, double *__restrict__ c, float2 *__restrict__ cdf,
                                       float *__restrict__ scale) {
    const int a = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= N) return;  // whole warp
    double s = 0.0;
    float mx = 0.f;
    for (int k = lane; k < nblk; k += 32) {
        s += psum[(size_t)a * nblk + k];
        mx = fmaxf(mx, pmax[(size_t)a * nblk + k]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane != 0) return;
    const double mean = s / (double)rows;
    const float ch = (float)mean, cl = (float)(mean - (double)ch);
    cdf[a] = make_float2(ch, cl);
    c[a] = (double)ch + (double)cl;  // the shift actually applied, exactly
    // |Phi - c| <= 2 max|Phi| =: bound in [2^(e-1), 2^e); scale 2^(-e-1) puts |x| below 1/2,
    // so the fixed-point slices stay within |x_s| <= 64 (later chunks: colstats_scale_kernel)
    float bound = 2.f * mx;
    int e = 0;
    if (bound > 0.f) frexpf(bound, &e);
    scale[a] = ldexpf(1.f, -e - 1);
}

// Later chunks of a two-pass fit keep the first chunk's centre c and take a scale of their
// own: |Phi - c| <= 2 max(max|Phi|, |c|) =: bound in [2^(e-1), 2^e), scale 2^(-e-1).  Each
// chunk's Gram tiles and row sums are converted to Phi units with that chunk's scale
// (gram_finish_tiles_kernel, rowsum_flush_kernel), so chunks need not share one.
__global__ void colstats_scale_kernel(const float *__restrict__ pmax, int nblk, int N, const double *__restrict__ c,
                                      float *__restrict__ scale) {
    const int a = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= N) return;  // whole warp
    float mx = 0.f;
    for (int k = lane; k < nblk; k += 32) mx = fmaxf(mx, pmax[(size_t)a * nblk + k]);
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane != 0) return;
    float bound = 2.f * fmaxf(mx, (float)fabs(c[a]) * 1.0001f);
    int e = 0;
    if (bound > 0.f) frexpf(bound, &e);
    scale[a] = ldexpf(1.f, -e - 1);
}

// After each chunk: its exact fixed-point row sums, converted to Phi units with the chunk's
// scales (exact: an int64 below 2^53 times a power of two), are added to sums[Np] and
// the integer sums are cleared for the next chunk.
__global__ void rowsum_flush_kernel(unsigned long long *__restrict__ rowsum, const float *__restrict__ scale,
                                    const double *__restrict__ vmax_p, int N, double *__restrict__ sums) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a > N) return;
    const double sc = a < N ? (double)scale[a] : (double)vscale_of(*vmax_p);
    sums[a] += ldexp((double)(long long)rowsum[a], -27) / sc;
    rowsum[a] = 0ull;
}

constexpr int kSliceThreads = 256;

// X rows: a < N: (Phi_t[a][m] - c_a) * scale_a;  a == N: Vc[m] * scale_V;  rest zero.
// Each value x (|x| <= 1) becomes I = round(x 2^27) and four 7-bit digits
// x ~ 2^-6 (x0 + 2^-7 x1 + 2^-14 x2 + 2^-21 x3), x_s integers in [-64, 64], exact in FP16.
// One thread per two consecutive points of one row (16-B loads, 4-B stores).
__global__ void __launch_bounds__(kSliceThreads) slice_rows_kernel(const float2 *__restrict__ phit, long long ld, long long rows, long long rows_pad,
                                  int N, const float2 *__restrict__ cdf, const float *__restrict__ scale,
                                  const double *__restrict__ Vc, long long m0, const double *__restrict__ vmax_p,
                                  __half *__restrict__ X0, __half *__restrict__ X1, __half *__restrict__ X2,
                                  __half *__restrict__ X3, int *__restrict__ clamped,
                                  unsigned long long *__restrict__ rowsum) {
    const int a = blockIdx.y;  // uniform per CTA: the ESP row and the padding rows branch as a whole
    const long long m = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
    int I[2] = {0, 0};
    if (m >= rows_pad) {
        // lanes past the row end only join the shuffle
    } else if (a == N) {
        const float sc = vscale_of(*vmax_p);
        for (int u = 0; u < 2; ++u)
            if (m + u < rows) {
                const double v = Vc[m0 + m + u];
                const float h = (float)v;
                I[u] = x_fixed(h, (float)(v - (double)h), sc, clamped);
            }
    } else if (a < N) {
        const float2 c = cdf[a];
        const float sc = scale[a];
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m + 1 < rows) v = *reinterpret_cast<const float4 *>(phit + (long long)a * ld + m);
        else if (m < rows) {
            const float2 v0 = phit[(long long)a * ld + m];
            v.x = v0.x;
            v.y = v0.y;
        }
        if (m < rows) {
            const float2 d = df_sub(v.x, v.y, c.x, c.y);
            I[0] = x_fixed(d.x, d.y, sc, clamped);
        }
        if (m + 1 < rows) {
            const float2 d = df_sub(v.z, v.w, c.x, c.y);
            I[1] = x_fixed(d.x, d.y, sc, clamped);
        }
    }
    // exact sum of the row's fixed-point values (two's complement int64 atomics: exact and
    // order-independent, so the mean correction sees exactly the values the Gram sees)
    __shared__ long long wpart[kSliceThreads / 32];
    long long rs = (long long)I[0] + (long long)I[1];
    for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
    if ((threadIdx.x & 31) == 0) wpart[threadIdx.x >> 5] = rs;
    __syncthreads();
    if (threadIdx.x == 0 && a <= N) {
        long long t = 0;
        for (int w = 0; w < kSliceThreads / 32; ++w) t += wpart[w];
        if (t != 0) atomicAdd(rowsum + a, (unsigned long long)t);  // one per CTA and row
    }
    if (m >= rows_pad) return;
    __half d0[2], d1[2], d2[2], d3[2];
    for (int u = 0; u < 2; ++u) digits4(I[u], d0, d1, d2, d3, u);
    const long long idx = (long long)a * rows_pad + m;
    *reinterpret_cast<__half2 *>(X0 + idx) = __halves2half2(d0[0], d0[1]);
    *reinterpret_cast<__half2 *>(X1 + idx) = __halves2half2(d1[0], d1[1]);
    *reinterpret_cast<__half2 *>(X2 + idx) = __halves2half2(d2[0], d2[1]);
    *reinterpret_cast<__half2 *>(X3 + idx) = __halves2half2(d3[0], d3[1]);
}

// The Gram tiles' exact sums (high and low 64-bit halves accumulated by the Gram kernel's
// work units, whatever the points per unit) rounded to FP64 once, (hi 2^32 exactly) + lo after
// normalising lo to [0, 2^32), and added, unscaled, into G (Np x Np).  Tiles inside a
// 128-row block already hold both (a,b) and (b,a); the others are mirrored.
__global__ void gram_finish_tiles_kernel(const unsigned long long *__restrict__ th,
                                         const unsigned long long *__restrict__ tl, int ntj, int Np,
                                         const float *__restrict__ scale, const double *__restrict__ vmax_p, int N,
                                         double *__restrict__ G) {
    const float vscale = vscale_of(*vmax_p);
    const int tile = blockIdx.y;
    int ti, tj;
    gram_tile_decode(tile, ntj, ti, tj);
    const int e = blockIdx.x * blockDim.x + threadIdx.x;  // element in tile, column-major (c*128 + r)
    if (e >= kBM * kGN) return;
    const int c = e / kBM, r = e - c * kBM;
    const int a = ti * kBM + r, b = tj * kGN + c;
    if (a >= Np || b >= Np) return;
    const size_t k = (size_t)tile * (kBM * kGN) + e;
    long long hi = (long long)th[k], lo = (long long)tl[k];
    hi += lo >> 32;  // lo in [0, 2^32), |hi| < 2^53 (the total is below 2^85)
    lo &= 0xffffffffLL;
    double s = (double)hi * 4294967296.0 + (double)lo;
    const double sa = (a < N) ? (double)scale[a] : (double)vscale;
    const double sb = (b < N) ? (double)scale[b] : (double)vscale;
    s = ldexp(s, -54) / (sa * sb);
    G[(size_t)a * Np + b] += s;
    if (tj >= 2 * ti + 2) G[(size_t)b * Np + a] += s;
}

// A = G - s s^T / M, b = G[:, V] - s s_V / M with s the exact column sums of the
// fixed-point rows in Phi units (rowsum_flush_kernel), i.e. repeat.py:2266-2276 for the
// shifted, quantised columns; optionally sum_phi = s + M c.
__global__ void finish_mixed_kernel(const double *__restrict__ G, int Np, const double *__restrict__ sums,
                                    const double *__restrict__ c, long long M, int N, double *__restrict__ A,
                                    double *__restrict__ b, double *__restrict__ sum_phi) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const double invM = 1.0 / (double)M;
    const double sv = sums[N];
    if (t < (long long)N * N) {
        const int i = (int)(t / N), j = (int)(t - (long long)i * N);
        A[t] = G[(size_t)i * Np + j] - sums[i] * sums[j] * invM;
    }
    if (t < N) {
        const double si = sums[t];
        b[t] = G[(size_t)t * Np + N] - si * sv * invM;
        if (sum_phi) sum_phi[t] = si + (double)M * c[t];
    }
}

__global__ void df_to_double_kernel(const float2 *__restrict__ x, long long n, double *__restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = (double)x[t].x + (double)x[t].y;
}

__global__ void __launch_bounds__(1024) absmax_kernel(const double *__restrict__ x, long long n,
                                                     double *__restrict__ out) {
    __shared__ double sm[1024];
    double m = 0.0;
    for (long long i = threadIdx.x; i < n; i += 1024) m = fmax(m, fabs(x[i]));
    sm[threadIdx.x] = m;
    __syncthreads();
    for (int o = 512; o > 0; o >>= 1) {
        if (threadIdx.x < o) sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sm[0];
}

// ------------------------------------------------------------------ host helpers

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        RP_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess) fail(RP_E_CUDA, "cuTensorMapEncodeTiled not available");
        fn = reinterpret_cast<EncodeFn>(p);
    }
    return fn;
}

// 2-D FP16 tensor [rows][cols] (cols contiguous, multiple of 64), box 32 x box_rows, 64-B swizzle
CUtensorMap make_map(const void *ptr, long long rows, long long cols, int box_rows) {
    RP_REQUIRE(cols % kKPad == 0, "tensor map: columns must be a multiple of 64");
    RP_REQUIRE(((uintptr_t)ptr & 15) == 0, "tensor map: base must be 16-byte aligned");
    CUtensorMap m;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) fail(RP_E_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return m;
}

// Work units of a Gram: ntri tiles x ceil(kb_total / kb_per_split) point splits.
int gram_units_total(const GramArgs &g) {
    RP_REQUIRE(g.kb_per_split >= 1 && g.kb_per_split <= kGramSplit && g.flush >= 1 && g.flush <= kGramFlush,
               "gram: bad split");
    const long long u = (long long)g.ntri * ceil_div(g.kb_total, g.kb_per_split);
    RP_REQUIRE(u < (1LL << 30), "gram: too many work units");
    return (int)u;
}
// Units per launch: kGramRounds rounds of one unit per SM.  A larger Gram is cut into launches
// of that size, so that it holds the SMs for well under a millisecond at a time: between two
// launches the block scheduler hands whole SMs to the waiting CTAs of streams of higher
// priority (the small fits of a served stream), which a single persistent launch over a large
// cube's ~10^5 units would keep to the room left beside its CTAs for tens of milliseconds.
constexpr int kGramRounds = 16;
int gram_units_per_launch(const rp_ctx *ctx) { return std::max(1, ctx->sm_count) * kGramRounds; }

// Zeroed tile totals (high and low halves, 2 x ntri x 128 x 64 words) with one work counter
// per launch after them, in one buffer cleared by one memset on the stream
size_t gram_launches(const rp_ctx *ctx, const GramArgs &g) { return (size_t)ceil_div(gram_units_total(g), gram_units_per_launch(ctx)); }
size_t gram_totals_words(const rp_ctx *ctx, const GramArgs &g) {
    return 2 * (size_t)g.ntri * kBM * kGN + (gram_launches(ctx, g) + 1) / 2 + 1;
}
void gram_totals_init(rp_ctx *ctx, const std::string &name, GramArgs &g, cudaStream_t s) {
    const size_t n = (size_t)g.ntri * kBM * kGN, words = gram_totals_words(ctx, g);
    unsigned long long *t = ctx->buf_t<unsigned long long>(name, words);
    RP_CUDA(cudaMemsetAsync(t, 0, sizeof(unsigned long long) * words, s));
    g.out_hi = t;
    g.out_lo = t + n;
    g.next_unit = reinterpret_cast<int *>(t + 2 * n);
}

// One CTA per SM (the stages fill most of its shared memory), at most one per work unit;
// launches of at most gram_units_per_launch units, each with its own counter
void launch_gram(rp_ctx *ctx, const __half *const *X, int rows, long long cols, GramArgs g, cudaStream_t s) {
    smem_optin((const void *)gram_exact_kernel, kGramSmem);
    {
        // the SM's whole shared memory as such, so that CTAs of other kernels fit beside this one
        static std::atomic<unsigned long long> carved{0};
        const int dev = ctx->device;
        if (dev >= 0 && dev < 64 && !(carved.load() & (1ULL << dev))) {
            RP_CUDA(cudaFuncSetAttribute((const void *)gram_exact_kernel,
                                         cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared));
            carved.fetch_or(1ULL << dev);
        }
    }
    const int total = gram_units_total(g), per = gram_units_per_launch(ctx);
    CUtensorMap a[kGSlices], b[kGSlices];
    for (int q = 0; q < kGSlices; ++q) {
        a[q] = make_map(X[q], rows, cols, kBM);   // rows past `rows` read as zeros
        b[q] = make_map(X[q], rows, cols, kGN);
    }
    int *const counters = g.next_unit;
    for (int k = 0, u0 = 0; u0 < total; ++k, u0 += per) {
        g.unit0 = u0;
        g.nunits = std::min(per, total - u0);
        g.next_unit = counters + k;
        const int grid = std::min(g.nunits, ctx->sm_count > 0 ? ctx->sm_count : 1);
        gram_exact_kernel<<<grid, kGramThreads, kGramSmem, s>>>(a[0], a[1], a[2], a[3], b[0], b[1], b[2], b[3], g);
        RP_LAUNCH_CHECK();
    }
}


inline long long round_up(long long a, long long b) { return (a + b - 1) / b * b; }

}  // namespace

// Upper bound B_a on |Phi[a][m]| over the kept points, which sets the digit scale of the
// single-pass path (false: an exclusion radius below 0.5 Bohr makes the bound useless).
//   Real space: the filter keeps no point within rn_a (the scaled vdW radius) of an image
//   of atom a, and two images are a lattice vector apart, at least the smallest
//   interplanar spacing d, so at most one image is nearer than d/2; hence
//   sum <= erfc(s rn)/rn + (S - 1) erfc(s d/2)/(d/2), erfc(s x)/x decreasing.
//   Reciprocal space: |sum_k c_k cos(k.r)| <= sum_k |c_k|.
// Should a cell defeat the argument (an image outside the filter's 27 nearest to a
// point), the kernel counts the clamped values and the caller redoes the fit in two passes.
static bool phi_bounds(const rp_ewald *ew, int S, const double *rn, int N, double bound_scale,
                       std::vector<float> &scale) {
    const double *b = ew->box;
    double d = 1e300;
    for (int q = 0; q < 3; ++q) {
        const double *u = b + 3 * ((q + 1) % 3), *v = b + 3 * ((q + 2) % 3), *w = b + 3 * q;
        const double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
        const double area = std::sqrt(cx * cx + cy * cy + cz * cz);
        const double vol = std::fabs(w[0] * cx + w[1] * cy + w[2] * cz);
        if (area > 0.0) d = std::min(d, vol / area);
    }
    double rec = 0.0;
    for (double c : ew->kcoef) rec += std::fabs(c);
    const double sa = ew->sqrt_alpha, h = 0.5 * d;
    const double tail = (S > 1 && h > 0.0) ? (S - 1) * std::erfc(sa * h) / h : 0.0;
    scale.resize((size_t)N);
    for (int a = 0; a < N; ++a) {
        if (!(rn[a] >= 0.5)) return false;
        const double B = (std::erfc(sa * rn[a]) / rn[a] + tail + rec) * bound_scale;
        int e = 0;
        std::frexp(B, &e);  // B in [2^(e-1), 2^e): |x| = |Phi| 2^(-e-1) < 1/2
        scale[a] = std::ldexp(1.0f, -e - 1);
    }
    return true;
}

void gram_mixed(rp_ctx *ctx, const rp_ewald *ew, const double *atoms, int N, const int32_t *kept_idx_dev,
                const double *Vc_dev, int64_t M, double *A_dev, double *b_dev, double *sum_phi_dev,
                cudaStream_t stream, const double *vstats_dev, const std::string &slot, const double *rn,
                int *clamp_dev, const double *d_atoms_pre, const float2 *E_pre, TileConfig tiles) {
    RP_REQUIRE(N > 0 && M > 0, "rp_gram: need N > 0 and M > 0");
    std::vector<double> sh;
    int zero_idx = -1;
    prune_shifts(ew, atoms, N, sh, zero_idx);
    const int S = (int)(sh.size() / 3);
    RP_REQUIRE(S <= kMaxShifts, "rp_gram: more than 128 real-space shifts after pruning (cutoff too large for the cell)");
    const int nx = ew->grid.n_grid[0], ny = ew->grid.n_grid[1];
    const int n1c = ew->kmax;

    const double *d_atoms = d_atoms_pre;
    if (!d_atoms) {
        double *a = ctx->buf_t<double>("g_atoms" + slot, 3 * (size_t)N);
        RP_CUDA(cudaMemcpyAsync(a, atoms, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, stream));
        d_atoms = a;
    }
    double *d_shifts = ctx->buf_t<double>("g_shifts" + slot, sh.size());
    double *d_axis = ctx->buf_t<double>("g_axis" + slot, 9);
    RP_CUDA(cudaMemcpyAsync(d_shifts, sh.data(), sizeof(double) * sh.size(), cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_axis, ew->grid.axis, sizeof(double) * 9, cudaMemcpyHostToDevice, stream));
    int *d_status = ctx->status_words();  // cleared by the caller (rp_gram / the batch driver)

    // reciprocal rows of every atom (stages A and B; or the caller's, computed for a whole
    // pipeline group) and the double-float images, once per fit
    const float2 *E = E_pre;
    float4 *img = ctx->buf_t<float4>("m_img" + slot, 2 * (size_t)N * S);
    {
        StageTimer tt(ctx, "recip_rows", stream);
        if (!E) {
            float2 *e = ctx->buf_t<float2>("m_E" + slot, recip_rows_bytes(ew, N) / sizeof(float2));
            recip_rows(ctx, ew, d_atoms, nullptr, N, e, stream, slot);
            E = e;
        }
        images_df_kernel<<<ceil_div((long long)N * S, 128), 128, 0, stream>>>(d_atoms, N, d_shifts, S, img);
        RP_LAUNCH_CHECK();
    }

    // chunk the points so the per-chunk staging stays below ~6 GB
    const int Np = N + 1;                       // atoms + the ESP row
    const long long per_point = 8LL * N + 8LL * Np;  // Phi (double-float, two-pass) + four FP16 digits
    long long chunk = std::max<long long>(kBM, ((6LL << 30) / per_point) / kBM * kBM);
    if (ctx->chunk_cap > 0) chunk = std::max<long long>(kBM, std::min<long long>(chunk, ctx->chunk_cap / kBM * kBM));
    chunk = std::min<long long>(chunk, round_up(M, kBM));
    const long long chunk_pad = round_up(chunk, kKPad);

    // single pass: Phi goes straight to digits, scaled by the a-priori bounds, centre 0
    std::vector<float> hscale;
    const bool single = rn && clamp_dev && phi_bounds(ew, S, rn, N, ctx->bound_scale, hscale);
    float2 *phit = single ? nullptr : ctx->buf_t<float2>("m_phit" + slot, (size_t)N * chunk_pad);
    __half *X[kGSlices];  // one buffer: the Phi kernel addresses the slices by their distance
    X[0] = ctx->buf_t<__half>("m_X" + slot, (size_t)kGSlices * Np * chunk_pad);
    for (int q = 1; q < kGSlices; ++q) X[q] = X[0] + (size_t)q * Np * chunk_pad;
    int *d_clamped = ctx->status_words() + 1;  // second status word: fixed-point range overflows
    const int nblk = (int)ceil_div(chunk, kPhiPts);
    double *psum = single ? nullptr : ctx->buf_t<double>("m_psum" + slot, (size_t)N * nblk);
    float *pmax = single ? nullptr : ctx->buf_t<float>("m_pmax" + slot, (size_t)N * nblk);
    unsigned long long *rowsum = ctx->buf_t<unsigned long long>("m_rowsum" + slot, (size_t)Np);
    double *sums = ctx->buf_t<double>("m_sums" + slot, (size_t)Np);
    double *cvec = ctx->buf_t<double>("m_c" + slot, N);
    float2 *cdf = ctx->buf_t<float2>("m_cdf" + slot, N);
    float *scale = ctx->buf_t<float>("m_scale" + slot, N);
    double *G = ctx->buf_t<double>("m_G" + slot, (size_t)Np * Np);
    RP_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * Np * Np, stream));
    RP_CUDA(cudaMemsetAsync(rowsum, 0, sizeof(unsigned long long) * Np, stream));
    RP_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * Np, stream));

    // ESP row scale from max |Vc| (the filter's, or computed here)
    const double *vmax = vstats_dev ? vstats_dev + 1 : nullptr;
    if (!vstats_dev) {
        double *st = ctx->buf_t<double>("m_vmax" + slot, 1);
        absmax_kernel<<<1, 1024, 0, stream>>>(Vc_dev, M, st);
        RP_LAUNCH_CHECK();
        vmax = st;
    }

    if (single) {
        RP_CUDA(cudaMemcpyAsync(scale, hscale.data(), sizeof(float) * N, cudaMemcpyHostToDevice, stream));
        RP_CUDA(cudaMemsetAsync(cvec, 0, sizeof(double) * N, stream));
    }

    const int nt = (int)ceil_div(Np, kBM), ntj = (int)ceil_div(Np, kGN);
    int ntri = 0;  // 128 x 64 Gram tiles with columns at or right of the row block, up to the last row
    for (int ti = 0; ti < nt; ++ti) ntri += ntj - 2 * ti;
    // points per CTA: kGramSplit stages (1024 points, the int64 headroom, exact sums drained
    // once) or fewer, for more CTAs on cubes with few Gram tiles (the autotuner's choice)
    const int kb_split = kStagesPer64 * std::min(std::max(tiles.gram_split, 1), kGramSplit / kStagesPer64);

    for (long long m0 = 0; m0 < M; m0 += chunk) {
        const long long rows = std::min<long long>(chunk, M - m0);
        const long long rows_kpad = round_up(rows, kKPad);
        // 1. Phi of the chunk (real space + reciprocal stage C) and its column statistics
        const int nb = (int)ceil_div(rows, kPhiPts);
        if (single) {  // Phi of the chunk straight to the digits of X
            StageTimer tt(ctx, "phi", stream);
            // the digits' rows hold the chunk's padded length, as the Gram's tensor maps read them
            const PhiDigits dg{X[0], (long long)Np * chunk_pad, rows_kpad, scale, Vc_dev + m0, vmax,
                               rowsum, clamp_dev, N};
            launch_phi(kept_idx_dev, m0, rows, d_axis, ew->grid.axis, ew->box, nx, ny, d_atoms, N, d_shifts, S, zero_idx,
                       ew->cutoff, ew->sqrt_alpha, img, ew->d_exf, E, n1c, 3, nullptr, chunk_pad, nullptr, nullptr,
                       &dg, stream, tiles.phi_atoms, ctx->sm_count);
        } else {
            StageTimer tt(ctx, "phi", stream);
            launch_phi(kept_idx_dev, m0, rows, d_axis, ew->grid.axis, ew->box, nx, ny, d_atoms, N, d_shifts, S, zero_idx, ew->cutoff,
                       ew->sqrt_alpha, img, ew->d_exf, E, n1c, 3, phit, chunk_pad, psum, pmax, nullptr, stream,
                       tiles.phi_atoms, ctx->sm_count);
        }
        // 2. centre on the first chunk, a scale per chunk, fixed-point digits of X
        if (!single) {
            StageTimer tt(ctx, "center_slice", stream);
            if (m0 == 0) {
                colstats_finish_kernel<<<ceil_div(N, 4), 128, 0, stream>>>(psum, pmax, nb, N, rows, cvec, cdf, scale);
            } else {
                colstats_scale_kernel<<<ceil_div(N, 4), 128, 0, stream>>>(pmax, nb, N, cvec, scale);
            }
            RP_LAUNCH_CHECK();
            slice_rows_kernel<<<dim3(ceil_div(rows_kpad / 2, kSliceThreads), Np), kSliceThreads, 0, stream>>>(
                phit, chunk_pad, rows, rows_kpad, N, cdf, scale, Vc_dev, m0, vmax, X[0], X[1], X[2], X[3], d_clamped,
                rowsum);
            RP_LAUNCH_CHECK();
        }
        // 3. exact Gram tiles (work units over point splits add exactly into the tiles' 64-bit
        //    totals), then the totals rounded once into G
        {
            const int kb_total = (int)(rows_kpad / kBK);
            GramArgs g{};
            g.nt = nt;
            g.ntj = ntj;
            g.ntri = ntri;
            g.kb_total = kb_total;
            g.kb_per_split = kb_split;
            g.flush = kGramFlush;
            g.status = d_status;
            g.budget = ctx->wait_budget;
            gram_totals_init(ctx, "m_tsum" + slot, g, stream);
            const __half *Xq[kGSlices] = {X[0], X[1], X[2], X[3]};
            {
                StageTimer tt(ctx, "gram_exact", stream);
                launch_gram(ctx, Xq, Np, rows_kpad, g, stream);
            }
            StageTimer tr(ctx, "gram_totals", stream);
            gram_finish_tiles_kernel<<<dim3(ceil_div(kBM * kGN, 256), ntri), 256, 0, stream>>>(
                g.out_hi, g.out_lo, ntj, Np, scale, vmax, N, G);
            RP_LAUNCH_CHECK();
            rowsum_flush_kernel<<<ceil_div(Np, 128), 128, 0, stream>>>(rowsum, scale, vmax, N, sums);
            RP_LAUNCH_CHECK();
        }
    }
    finish_mixed_kernel<<<ceil_div(std::max<long long>((long long)N * N, N), 256), 256, 0, stream>>>(
        G, Np, sums, cvec, M, N, A_dev, b_dev, sum_phi_dev);
    RP_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- exact Gram of FP64 columns
// For the escalated (FP64) fit: the columns of a chunk of Phi (rows x N, row-major, ld N,
// centred) and the centred ESP are scaled by powers of two to |x| < 1/2 and cut into two
// 28-bit words, x = 2^-27 (I1 + 2^-27 I2) + O(2^-55); the 2(N+1) rows [I1 of every column;
// I2 of every column] go through the exact digit Gram (every digit product exact, tile
// totals exact, one FP64 rounding), and
//   G[a][b] += (G11 + 2^-27 (G12 + G21) + 2^-54 G22)[a][b] / (s_a s_b)
// with the ESP as column N (G[a][N] = (Phi^T V)[a]).  An FP64-accurate Gram from the
// tensor cores: 4x the work of the mixed path's Gram, instead of DSYRK at the FP64 rate.
// Where its digits (16 bytes per point and column) and tile totals (32 per pair of columns) have no
// room, the columns are taken two blocks at a time and the points block by block: the scales are of the
// whole columns and the totals exact integers, so every entry of G has the same bits.
namespace {

// The columns of a Gram: block I (i0 .. i0 + ni - 1) and then block J of the N + 1
struct WordCols {
    int i0, ni, j0, nj;
    int own_i, own_j;  // whether the products within I and within J are this Gram's to add
    __host__ __device__ int n() const { return ni + nj; }
    __device__ int global(int c) const { return c < ni ? i0 + c : j0 + c - ni; }
};

// max |x| of each column (N of Phi, then the ESP as column N), as order-preserving bits
__global__ void colmax_fp64_kernel(const double *__restrict__ P, long long rows, int N, const double *__restrict__ V,
                                   unsigned long long *__restrict__ mx) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c > N) return;
    const long long r0 = (long long)blockIdx.y * 256, r1 = min(rows, r0 + 256);
    double m = 0.0;
    for (long long r = r0; r < r1; ++r) m = fmax(m, fabs(c < N ? P[r * N + c] : V[r]));
    atomicMax(mx + c, (unsigned long long)__double_as_longlong(m));  // m >= 0: bits order like values
}

__device__ __forceinline__ double pow2_scale(unsigned long long mbits) {
    const double m = __longlong_as_double((long long)mbits);
    int e = 0;
    if (m > 0.0) frexp(m, &e);  // m in [2^(e-1), 2^e): m 2^(-e-1) < 1/2
    return ldexp(1.0, -e - 1);
}

// two 28-bit words of each value, as four 7-bit digits each: column c < n of the block (the ESP
// is column N) to rows c and c + n of the slices; a 32 x 32 tile per CTA through shared
// memory, so both the reads of Phi and the writes of the slices coalesce
__global__ void split_words_kernel(const double *__restrict__ P, long long rows, long long cols_pad, int N, WordCols wc,
                                   const double *__restrict__ V, const unsigned long long *__restrict__ mx,
                                   __half *__restrict__ X0, __half *__restrict__ X1, __half *__restrict__ X2,
                                   __half *__restrict__ X3) {
    __shared__ double t[32][33];
    const long long m0 = (long long)blockIdx.x * 32;
    const int c0 = blockIdx.y * 32, n = wc.n();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {  // t[point][column]
        const long long m = m0 + k;
        const int c = c0 + threadIdx.x, g = wc.global(c);
        double v = 0.0;
        if (m < rows && c < n) v = g < N ? P[m * N + g] : V[m];
        t[k][threadIdx.x] = v;
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {  // column c0 + k, point m0 + x
        const int c = c0 + k;
        const long long m = m0 + threadIdx.x;
        if (c >= n || m >= cols_pad) continue;
        const double x = t[threadIdx.x][k] * pow2_scale(mx[wc.global(c)]) * 134217728.0;  // |x| < 2^26
        const double i1 = rint(x);
        const double i2 = rint((x - i1) * 134217728.0);                          // |x - i1| <= 1/2
        digits4((int)i1, X0, X1, X2, X3, (long long)c * cols_pad + m);
        digits4((int)i2, X0, X1, X2, X3, (long long)(c + n) * cols_pad + m);
    }
}

// 2^-54 x the exact total of word rows (r, c), from the tile that holds (min, max)
__device__ __forceinline__ double tile_total(const unsigned long long *th, const unsigned long long *tl, int ntj,
                                             int r, int c) {
    if (r > c) {
        const int t = r;
        r = c;
        c = t;
    }
    const int ti = r / kBM, tj = c / kGN;
    const size_t k = (size_t)(ti * ntj - ti * (ti - 1) + tj - 2 * ti) * (kBM * kGN) + (c % kGN) * kBM + r % kBM;
    long long hi = (long long)th[k], lo = (long long)tl[k];
    hi += lo >> 32;
    lo &= 0xffffffffLL;
    return ldexp((double)hi * 4294967296.0 + (double)lo, -54);
}

// G[a][b] (N x N, either order: symmetric) and r[a] (b = N) += the combined words / (s_a s_b);
// rows a fastest, as the tiles store them
__global__ void combine_words_kernel(const unsigned long long *__restrict__ th,
                                     const unsigned long long *__restrict__ tl, int ntj, int N, WordCols wc,
                                     const unsigned long long *__restrict__ mx, double *__restrict__ G,
                                     double *__restrict__ r) {
    const int n = wc.n();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)n * n) return;
    const int lb = (int)(t / n), la = (int)(t - (long long)lb * n), a = wc.global(la), b = wc.global(lb);
    if (a >= N || (la < wc.ni && lb < wc.ni && !wc.own_i) || (la >= wc.ni && lb >= wc.ni && !wc.own_j)) return;
    const double g11 = tile_total(th, tl, ntj, la, lb), g12 = tile_total(th, tl, ntj, la, n + lb);
    const double g21 = tile_total(th, tl, ntj, lb, n + la), g22 = tile_total(th, tl, ntj, n + la, n + lb);
    const double v = (g11 + 7.450580596923828125e-9 * (g12 + g21) + 5.5511151231257827e-17 * g22) /
                     (pow2_scale(mx[a]) * pow2_scale(mx[b]));
    if (b < N) G[(size_t)b * N + a] += v;
    else r[a] += v;
}

// the Gram of the word rows of n columns over cols points
GramArgs words_args(rp_ctx *ctx, int n, long long cols) {
    GramArgs g{};
    g.nt = (int)ceil_div(2 * n, kBM);
    g.ntj = (int)ceil_div(2 * n, kGN);
    for (int ti = 0; ti < g.nt; ++ti) g.ntri += g.ntj - 2 * ti;
    g.kb_total = (int)(cols / kBK);
    g.kb_per_split = kGramSplit;
    g.flush = kGramFlush;
    g.status = ctx->status_words();  // cleared before and checked after by the caller
    g.budget = ctx->wait_budget;
    return g;
}
size_t words_totals_bytes(rp_ctx *ctx, int n, long long cols) {
    return sizeof(unsigned long long) * gram_totals_words(ctx, words_args(ctx, n, cols));
}
size_t words_digit_bytes(int n, long long cols) { return sizeof(__half) * kGSlices * 2 * (size_t)n * (size_t)cols; }

}  // namespace

size_t gram_words_bytes(rp_ctx *ctx, long long rows, int N) {
    const long long cols = round_up(rows, kKPad);
    return words_totals_bytes(ctx, N + 1, cols) + words_digit_bytes(N + 1, cols);
}

void gram_words_fp64(rp_ctx *ctx, const double *P, long long rows, int N, const double *V, double *G, double *r,
                     size_t scratch, cudaStream_t stream) {
    const int Np = N + 1;
    unsigned long long *mx = ctx->buf_t<unsigned long long>("w64_mx", (size_t)Np);
    RP_CUDA(cudaMemsetAsync(mx, 0, sizeof(unsigned long long) * Np, stream));
    colmax_fp64_kernel<<<dim3(ceil_div(Np, 256), ceil_div(rows, 256)), 256, 0, stream>>>(P, rows, N, V, mx);
    RP_LAUNCH_CHECK();
    // Blocks: the whole where it fits; else the largest blocks of columns whose totals leave room for the digits
    // of 4096 points (fewer, longer runs of the pipeline), down to 16 columns, and the points that then fit.
    long long cols = round_up(rows, kKPad);
    int block = Np, n = Np;
    if (words_totals_bytes(ctx, n, cols) + words_digit_bytes(n, cols) > scratch) {
        size_t totals = 0;
        for (int nb = 1;; ++nb) {
            block = (int)ceil_div(Np, nb);
            n = std::min(Np, nb == 1 ? block : 2 * block);
            totals = words_totals_bytes(ctx, n, cols);
            if (block <= 16 || totals + words_digit_bytes(n, std::min<long long>(cols, 4096)) <= scratch) break;
        }
        const size_t left = scratch > totals ? scratch - totals : 0;
        cols = std::min<long long>(cols, std::max<long long>(kKPad, (long long)(left / words_digit_bytes(n, kKPad)) * kKPad));
    }
    __half *X[kGSlices];
    for (int q = 0; q < kGSlices; ++q) X[q] = ctx->buf_t<__half>("w64_X" + std::to_string(q), 2 * (size_t)n * cols);
    const __half *Xq[kGSlices] = {X[0], X[1], X[2], X[3]};
    const int nb = (int)ceil_div(Np, block);
    auto gram = [&](const WordCols &wc) {
        GramArgs g = words_args(ctx, wc.n(), cols);
        gram_totals_init(ctx, "w64_tsum", g, stream);
        for (long long m0 = 0; m0 < rows; m0 += cols) {
            const long long part = std::min<long long>(cols, rows - m0), pad = round_up(part, kKPad);
            if (m0 > 0) {  // more points into the same totals, with fresh work counters
                g.kb_total = (int)(pad / kBK);
                RP_CUDA(cudaMemsetAsync(g.next_unit, 0, sizeof(int) * gram_launches(ctx, g), stream));
            }
            split_words_kernel<<<dim3(ceil_div(pad, 32), ceil_div(wc.n(), 32)), dim3(32, 8), 0, stream>>>(
                P + m0 * N, part, pad, N, wc, V + m0, mx, X[0], X[1], X[2], X[3]);
            RP_LAUNCH_CHECK();
            launch_gram(ctx, Xq, 2 * wc.n(), pad, g, stream);
        }
        combine_words_kernel<<<ceil_div((long long)wc.n() * wc.n(), 256), 256, 0, stream>>>(g.out_hi, g.out_lo, g.ntj, N,
                                                                                           wc, mx, G, r);
        RP_LAUNCH_CHECK();
    };
    auto first = [&](int b) { return b * block; };
    auto size = [&](int b) { return std::min(block, Np - b * block); };
    if (nb == 1) gram(WordCols{0, Np, 0, 0, 1, 0});
    for (int i = 0; i < nb; ++i)  // each pair once; a block's own products with its successor, the last's with its predecessor
        for (int j = i + 1; j < nb; ++j)
            gram(WordCols{first(i), size(i), first(j), size(j), j == i + 1, j == nb - 1 && j == i + 1});
}

}  // namespace rp

// Diagnostics (not part of the public ABI): a factor on the single-pass Phi bounds of
// the batched fit (1 = the analytic bounds).  A factor far below 1 makes every cube clamp
// and fall back to the two-pass fit, which a test compares with the normal path.
extern "C" int rp_debug_bound_scale(rp_ctx *ctx, double factor) {
    if (!ctx || !(factor > 0.0)) return RP_E_ARG;
    ctx->bound_scale = factor;
    return RP_OK;
}

// Diagnostics (not part of the public ABI): the clock budget of the Gram pipeline's waits
// (cycles < 0: the default, ~2 s; 0: every wait gives up at once, which exercises the
// timeout path: RP_E_TIMEOUT, the kernel unwinds, the ctx stays usable).
extern "C" int rp_debug_wait_budget(rp_ctx *ctx, long long cycles) {
    if (!ctx) return RP_E_ARG;
    ctx->wait_budget = cycles < 0 ? rp::tc::kWaitBudgetCycles : cycles;
    return RP_OK;
}

// Diagnostics (not part of the public ABI): an upper bound on the kept points per chunk of
// the staged mixed Gram (0 = the memory-based size), so tests can run many chunks on a
// small cube.
extern "C" int rp_debug_chunk_cap(rp_ctx *ctx, long long points) {
    if (!ctx || points < 0) return RP_E_ARG;
    ctx->chunk_cap = points;
    return RP_OK;
}

// Diagnostics: how many cubes of the last batched fit were redone in two passes.
extern "C" int rp_debug_last_fallbacks(const rp_ctx *ctx) { return ctx ? ctx->last_fallbacks : RP_E_ARG; }

namespace rp {
namespace {
__global__ void erfc_kernel(const float *__restrict__ x, long long n, float *__restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = erfc_nr2((float)kSqrtLog2e * x[t]);
}
}  // namespace
}  // namespace rp

// Diagnostics (not part of the public ABI): the real-space kernels' FP32 erfc at n
// arguments x (device arrays), for the test against FP64 erfc and CUDA's erfcf.
extern "C" int rp_debug_erfc(const float *x_dev, long long n, float *out_dev) {
    using namespace rp;
    if (!x_dev || !out_dev || n < 0) return RP_E_ARG;
    if (n == 0) return RP_OK;
    erfc_kernel<<<(unsigned)((n + 255) / 256), 256>>>(x_dev, n, out_dev);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return RP_E_CUDA;
    return RP_OK;
}

// Diagnostics (not part of the public ABI): the mixed path's Phi for the first
// `rows` kept points, atom-major [N][rows]; parts = 1 real space, 2 reciprocal,
// 3 both.  Used to check each part against FP64 separately.
extern "C" int rp_debug_mixed_phi(rp_ctx *ctx, const rp_ewald *ew, const double *atoms, int N,
                                  const int32_t *kept_idx_dev, int64_t rows, int parts, double *phi_dev) {
    using namespace rp;
    try {
        RP_CUDA(cudaSetDevice(ctx->device));
        RP_REQUIRE(N > 0 && rows > 0 && rows <= (1LL << 30) && parts >= 1 && parts <= 3, "bad arguments");
        std::vector<double> sh;
        int zero_idx = -1;
        prune_shifts(ew, atoms, N, sh, zero_idx);
        const int S = (int)(sh.size() / 3);
        double *d_atoms = ctx->buf_t<double>("g_atoms", 3 * (size_t)N);
        double *d_shifts = ctx->buf_t<double>("g_shifts", sh.size());
        double *d_axis = ctx->buf_t<double>("g_axis", 9);
        RP_CUDA(cudaMemcpy(d_atoms, atoms, sizeof(double) * 3 * N, cudaMemcpyHostToDevice));
        RP_CUDA(cudaMemcpy(d_shifts, sh.data(), sizeof(double) * sh.size(), cudaMemcpyHostToDevice));
        RP_CUDA(cudaMemcpy(d_axis, ew->grid.axis, sizeof(double) * 9, cudaMemcpyHostToDevice));
        float2 *E = ctx->buf_t<float2>("m_E", recip_rows_bytes(ew, N) / sizeof(float2));
        float4 *img = ctx->buf_t<float4>("m_img", 2 * (size_t)N * S);
        recip_rows(ctx, ew, d_atoms, nullptr, N, E, 0);
        images_df_kernel<<<ceil_div((long long)N * S, 128), 128>>>(d_atoms, N, d_shifts, S, img);
        RP_LAUNCH_CHECK();
        float2 *ph = ctx->buf_t<float2>("dbg_phi", (size_t)N * rows);
        launch_phi(kept_idx_dev, 0, rows, d_axis, ew->grid.axis, ew->box, ew->grid.n_grid[0], ew->grid.n_grid[1], d_atoms, N, d_shifts, S,
                   zero_idx, ew->cutoff, ew->sqrt_alpha, img, ew->d_exf, E, ew->kmax, parts, ph, rows, nullptr,
                   nullptr, nullptr, 0, kPhiAtoms, ctx->sm_count);
        df_to_double_kernel<<<ceil_div((long long)N * rows, 256), 256>>>(ph, (long long)N * rows, phi_dev);
        RP_LAUNCH_CHECK();
        RP_CUDA(cudaDeviceSynchronize());
        return RP_OK;
    } catch (const rp::Error &e) {
        ctx->last_error = e.msg;
        return e.code;
    }
}

// Diagnostics: the exact-Gram kernel on caller-provided FP16 slices X0 .. X3
// ([Np_pad][cols], cols a multiple of 64) -> 2^-54 * sum over points and all sixteen
// slice products of x_s y_u 2^(7(6-s-u)) (FP64, Np x Np).
extern "C" int rp_debug_gram_slices(rp_ctx *ctx, const void *X0, const void *X1, const void *X2, const void *X3,
                                    int Np, long long cols, int flush, int kb_split, double *I_dev) {
    using namespace rp;
    try {
        RP_CUDA(cudaSetDevice(ctx->device));
        const int nt = (int)ceil_div(Np, kBM), ntj = (int)ceil_div(Np, kGN);
        int ntri = 0;
        for (int ti = 0; ti < nt; ++ti) ntri += ntj - 2 * ti;
        const int kb_total = (int)(cols / kBK);
        // flush and kb_split count 64-point blocks (the padding unit): two stages each
        RP_REQUIRE(kb_split >= 1 && kb_split * kStagesPer64 <= kGramSplit, "kb_split must lie in [1, 16]");
        RP_CUDA(cudaMemset(ctx->d_status, 0, sizeof(int)));
        GramArgs g{};
        g.nt = nt; g.ntj = ntj; g.ntri = ntri; g.kb_total = kb_total; g.kb_per_split = kb_split * kStagesPer64;
        g.flush = kStagesPer64 * std::min(std::max(flush, 1), kGramFlush / kStagesPer64);
        g.status = ctx->d_status; g.budget = ctx->wait_budget;
        gram_totals_init(ctx, "dbg_tsum", g, 0);
        const __half *Xq[kGSlices] = {(const __half *)X0, (const __half *)X1, (const __half *)X2, (const __half *)X3};
        launch_gram(ctx, Xq, Np, cols, g, 0);
        float *ones = ctx->buf_t<float>("dbg_ones", Np);
        std::vector<float> h((size_t)Np, 1.0f);
        RP_CUDA(cudaMemcpy(ones, h.data(), sizeof(float) * Np, cudaMemcpyHostToDevice));
        RP_CUDA(cudaMemset(I_dev, 0, sizeof(double) * Np * Np));
        double *vmax = ctx->buf_t<double>("dbg_vmax", 1);  // unused: every row is an atom row (N = Np)
        RP_CUDA(cudaMemset(vmax, 0, sizeof(double)));
        gram_finish_tiles_kernel<<<dim3(ceil_div(kBM * kGN, 256), ntri), 256>>>(g.out_hi, g.out_lo, ntj, Np, ones,
                                                                               vmax, Np, I_dev);
        RP_LAUNCH_CHECK();
        RP_CUDA(cudaDeviceSynchronize());
        int st = 0;
        RP_CUDA(cudaMemcpy(&st, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost));
        if (st) fail(st, "gram kernel wait timed out");
        return RP_OK;
    } catch (const rp::Error &e) {
        ctx->last_error = e.msg;
        return e.code;
    }
}

