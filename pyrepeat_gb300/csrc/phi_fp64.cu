// FP64 Phi -> normal equations: the FP64 fit (--fp64) and the refit of an ill-conditioned mixed one.
//
// Per chunk of kept points (Phi is held for one chunk only):
//   Phi      = the separable reciprocal sum (the transform of recip_sep.cu): the plane stage once
//              per fit, the row stage for the grid rows that hold points of the chunk, the point
//              stage.  In FP64 throughout for the FP64 fit; with the plane and row stages in
//              double-float (~2^-46) for the refit.
//   Phi     += sum_s [r <= Rc] erfc(sqrt(alpha) r)/r (FP64, repeat.py:944-966)
//   Phi_c    = Phi - c  (c = column means of the first chunk: a per-column shift,
//              exactly corrected afterwards, so A needs no large cancellation)
//   G += Phi_c^T Phi_c, r += Phi_c^T Vc   (exact two-word Gram on the tensor cores, gram_words_fp64)
// Finally A = G - s s^T / M, b = r - s sum(Vc) / M with s = sum_m Phi_c[m,:]
// (= sum_phi - M c); this is repeat.py:2266-2276's mean correction written for
// the shifted columns.
// (The FP64 fit was a flat k-table DGEMM with an in-place real-space sum and a cuBLAS Gram: 108, 24
// and 16 ms on 36 M point-atom pairs at K = 754.)
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "df.cuh"
#include "erfc64.cuh"

namespace rp {
namespace {

// Real-space sum in FP64 (repeat.py:944-966) over tiles of kRsPts kept points x kRsAtoms
// atoms.  For each chunk of up to kRsShiftChunk shifts, the CTA first drops, per atom,
// every shift whose image lies farther than Rc + 1e-3 Bohr from the bounding box of its
// points (an FP32 test: FP32 rounding of the coordinates moves a distance by < 1e-4
// Bohr here, so no image within Rc is dropped).  Each thread then tests the remaining
// images of each atom against its point in FP32 with the same margin.  QUEUE false: the
// survivors are evaluated in place (the 1/r basis: one image per atom, reached by every point).
// QUEUE true (the periodic basis, whatever the order of the kept points): each thread queues its
// survivors (atom, image) in order, the CTA
// evaluates the queued pairs in FP64, every lane on one pair, so the FP64 pipe (a small
// fraction of the FP32 rate on this part, and as slow for one active lane as for 32)
// runs full warps instead of a warp per image that any of its points reaches, and each
// thread adds its pairs' terms in queue order (a rejected pair adds +0.0, which changes
// no sum).  Either way the FP64 expressions are the reference's.  Every image within Rc is therefore summed, in shift order, exactly as by a
// loop over all shifts.  The sums are accumulated in a shared-memory tile and added into
// phi[m][a] (row-major, ld N) with coalesced stores.
constexpr int kRsPts = 128;
constexpr int kRsAtoms = 16;
constexpr int kRsQueue = 16;  // queued pairs per point per round
// shifts per chunk: in place 128, queued 64 (its queue takes the rest of the shared memory)
template <bool QUEUE> __host__ __device__ constexpr int rs_chunk() { return QUEUE ? 64 : 128; }
size_t realspace_fp64_smem(bool queue) {
    return queue ? sizeof(float4) * kRsAtoms * rs_chunk<true>() + sizeof(double) * kRsQueue * kRsPts +
                       sizeof(unsigned short) * kRsQueue * kRsPts
                 : sizeof(float4) * kRsAtoms * rs_chunk<false>();
}
template <bool QUEUE>
__global__ void __launch_bounds__(kRsPts) realspace_fp64_kernel(
    const int32_t *__restrict__ kept, long long m0, long long rows, const double *__restrict__ axis, int nx, int ny,
    const double *__restrict__ atoms, int N, const double *__restrict__ shifts, int S, int zero_idx, double rc,
    double sa, double d2_in, double d2_self, ErfcTable tab, double *__restrict__ phi) {
    constexpr int kRsShiftChunk = rs_chunk<QUEUE>();
    extern __shared__ float4 rs_cand[];  // [kRsAtoms][kRsShiftChunk] image (x, y, z) in FP32, shift index
    double *qterm = reinterpret_cast<double *>(rs_cand + kRsAtoms * kRsShiftChunk);      // [kRsQueue][kRsPts]
    unsigned short *qitem = reinterpret_cast<unsigned short *>(qterm + kRsQueue * kRsPts);  // (atom << 7) | image
    __shared__ double tile[kRsAtoms][kRsPts + 1];
    __shared__ double gs[3][kRsPts];
    __shared__ int ncand[kRsAtoms];
    __shared__ int qoff[kRsPts + 1];
    __shared__ int wsum[kRsPts / 32];
    __shared__ int more;
    __shared__ float bb[2][3][kRsPts / 32];
    const long long mb = (long long)blockIdx.x * kRsPts;
    const int a0 = blockIdx.y * kRsAtoms, na = min(kRsAtoms, N - a0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long m = mb + threadIdx.x;
    const bool valid = m < rows;
    const int f = kept[m0 + (valid ? m : mb)];  // a lane past the end repeats the tile's first point
    const int layer = nx * ny;
    const int l = f / layer, rem = f - l * layer, j = rem / nx, i = rem - j * nx;
    double g[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        g[d] = ((double)i * axis[d] + (double)j * axis[3 + d]) + (double)l * axis[6 + d];
        gs[d][threadIdx.x] = g[d];
    }
    const float gf[3] = {(float)g[0], (float)g[1], (float)g[2]};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float mn = gf[d], mx = gf[d];
        for (int o = 16; o > 0; o >>= 1) {
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (lane == 0) {
            bb[0][d][warp] = mn;
            bb[1][d][warp] = mx;
        }
    }
    for (int a = 0; a < kRsAtoms; ++a) tile[a][threadIdx.x] = 0.0;
    __syncthreads();
    float bmin[3], bmax[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        bmin[d] = bb[0][d][0];
        bmax[d] = bb[1][d][0];
        for (int w = 1; w < kRsPts / 32; ++w) {
            bmin[d] = fminf(bmin[d], bb[0][d][w]);
            bmax[d] = fmaxf(bmax[d], bb[1][d][w]);
        }
    }
    const float reach = (float)rc + 1e-3f, reach2 = reach * reach;
    for (int s_lo = 0; s_lo < S; s_lo += kRsShiftChunk) {
        const int s_hi = min(S, s_lo + kRsShiftChunk);
        for (int a = warp; a < na; a += kRsPts / 32) {
            int base = 0;
            const double *pa = atoms + 3 * (size_t)(a0 + a);
            for (int s0 = s_lo; s0 < s_hi; s0 += 32) {
                const int s = s0 + lane;
                bool keep = false;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                if (s < s_hi) {
                    q = make_float4((float)(pa[0] + shifts[3 * s]), (float)(pa[1] + shifts[3 * s + 1]),
                                    (float)(pa[2] + shifts[3 * s + 2]), __int_as_float(s));
                    const float dx = fmaxf(fmaxf(bmin[0] - q.x, q.x - bmax[0]), 0.f);
                    const float dy = fmaxf(fmaxf(bmin[1] - q.y, q.y - bmax[1]), 0.f);
                    const float dz = fmaxf(fmaxf(bmin[2] - q.z, q.z - bmax[2]), 0.f);
                    keep = dx * dx + dy * dy + dz * dz <= reach2;
                }
                const unsigned bal = __ballot_sync(0xffffffffu, keep);
                if (keep) rs_cand[a * kRsShiftChunk + base + __popc(bal & ((1u << lane) - 1u))] = q;
                base += __popc(bal);
            }
            if (lane == 0) ncand[a] = base;
        }
        __syncthreads();
        // Evaluated where they are found (QUEUE false), the pairs cost a warp-wide FP64 pass
        // for every image that any lane of the warp reaches, which suits tiles whose points
        // lie close together; queued, they cost their number plus the queue's bookkeeping.
        {
            if (!QUEUE) {  // evaluate in place, in order
                for (int a = 0; a < na; ++a) {
                    const double *pa = atoms + 3 * (size_t)(a0 + a);
                    double acc = tile[a][threadIdx.x];
                    for (int c = 0; c < ncand[a]; ++c) {
                        const float4 h = rs_cand[a * kRsShiftChunk + c];
                        const float fx = gf[0] - h.x, fy = gf[1] - h.y, fz = gf[2] - h.z;
                        if (fx * fx + fy * fy + fz * fz > reach2) continue;
                        const int s = __float_as_int(h.w);
                        const double ex = g[0] - (pa[0] + shifts[3 * s]);
                        const double ey = g[1] - (pa[1] + shifts[3 * s + 1]);
                        const double ez = g[2] - (pa[2] + shifts[3 * s + 2]);
                        const double d2 = ex * ex + ey * ey + ez * ez;
                        if (!le_bits(d2, d2_in)) continue;
                        if (s == zero_idx && le_bits(d2, d2_self)) continue;
                        acc += erfc_term(d2, tab, sa);
                    }
                    tile[a][threadIdx.x] = acc;
                }
                __syncthreads();
                continue;
            }
        }
        // rounds: queue up to kRsQueue pairs per point (resuming where the last round stopped),
        // evaluate them with the whole CTA, add the terms in queue order
        int ra = 0, rcnd = 0;  // this thread's resume point (atom, image)
        for (;;) {
            int cnt = 0;
            while (ra < na && cnt < kRsQueue) {
                const int nc = ncand[ra];
                while (rcnd < nc && cnt < kRsQueue) {
                    const float4 h = rs_cand[ra * kRsShiftChunk + rcnd];
                    const float fx = gf[0] - h.x, fy = gf[1] - h.y, fz = gf[2] - h.z;
                    if (fx * fx + fy * fy + fz * fz <= reach2)
                        qitem[cnt++ * kRsPts + threadIdx.x] = (unsigned short)((ra << 7) | rcnd);
                    ++rcnd;
                }
                if (rcnd >= nc) {
                    ++ra;
                    rcnd = 0;
                }
            }
            // offsets of every thread's queue (block exclusive scan of cnt)
            int incl = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) wsum[warp] = incl;
            if (threadIdx.x == 0) more = 0;
            __syncthreads();
            int wbase = 0;
            for (int w = 0; w < warp; ++w) wbase += wsum[w];
            qoff[threadIdx.x] = wbase + incl - cnt;
            if (threadIdx.x == kRsPts - 1) qoff[kRsPts] = wbase + incl;
            if (ra < na) more = 1;
            __syncthreads();
            const int total = qoff[kRsPts];
            for (int idx = threadIdx.x; idx < total; idx += kRsPts) {
                int lo = 0, hi = kRsPts - 1;  // the owner: the last thread whose offset is <= idx
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (qoff[mid] <= idx) lo = mid;
                    else hi = mid - 1;
                }
                const int k = idx - qoff[lo];
                const unsigned short it = qitem[k * kRsPts + lo];
                const int a = it >> 7, c = it & 127;
                const int s = __float_as_int(rs_cand[a * kRsShiftChunk + c].w);
                const double *pa = atoms + 3 * (size_t)(a0 + a);
                const double ex = gs[0][lo] - (pa[0] + shifts[3 * s]);
                const double ey = gs[1][lo] - (pa[1] + shifts[3 * s + 1]);
                const double ez = gs[2][lo] - (pa[2] + shifts[3 * s + 2]);
                const double d2 = ex * ex + ey * ey + ez * ez;
                double term = 0.0;
                if (le_bits(d2, d2_in) && !(s == zero_idx && le_bits(d2, d2_self))) term = erfc_term(d2, tab, sa);
                qterm[k * kRsPts + lo] = term;
            }
            __syncthreads();
            for (int k = 0; k < cnt; ++k) tile[qitem[k * kRsPts + threadIdx.x] >> 7][threadIdx.x] += qterm[k * kRsPts + threadIdx.x];
            const int again = more;
            __syncthreads();  // the queue is refilled on the next pass
            if (!again) break;
        }
    }
    // tile[a][t] -> phi[(mb + t) * N + a0 + a]: kRsAtoms consecutive doubles per point
    for (int e = threadIdx.x; e < kRsPts * kRsAtoms; e += kRsPts) {
        const int t = e / kRsAtoms, a = e - t * kRsAtoms;
        if (mb + t < rows && a < na) phi[(mb + t) * N + a0 + a] += tile[a][t];
    }
}

// Column sums of a row-major rows x cols block (ld), FP64, deterministic:
// stage 1 sums fixed row slabs per column; stage 2 adds the slabs in order.
constexpr int kSlab = 256;
__global__ void colsum_stage1(const double *__restrict__ X, long long rows, int cols, int ld,
                              double *__restrict__ part) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    long long r0 = (long long)blockIdx.y * kSlab;
    if (c >= cols) return;
    long long r1 = min(r0 + kSlab, rows);
    double s = 0.0;
    for (long long r = r0; r < r1; ++r) s += X[r * ld + c];
    part[(size_t)blockIdx.y * cols + c] = s;
}
__global__ void colsum_stage2(const double *__restrict__ part, int nslab, int cols, double *__restrict__ out,
                              int accumulate) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    double s = 0.0;
    for (int k = 0; k < nslab; ++k) s += part[(size_t)k * cols + c];
    out[c] = accumulate ? out[c] + s : s;
}

__global__ void shift_columns_kernel(double *__restrict__ X, long long rows, int cols,
                                     const double *__restrict__ c) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= rows * cols) return;
    X[t] -= c[t % cols];
}

__global__ void set_mean_kernel(const double *__restrict__ sums, int n, double inv, double *__restrict__ c) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) c[t] = sums[t] * inv;
}

__global__ void finish_kernel(const double *__restrict__ G, const double *__restrict__ r,
                              const double *__restrict__ s, const double *__restrict__ sumV, long long M, int N,
                              double *__restrict__ A, double *__restrict__ b) {
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    double invM = 1.0 / (double)M;
    if (t < (long long)N * N) {
        int i = (int)(t / N), j = (int)(t - (long long)i * N);
        A[t] = G[t] - s[i] * s[j] * invM;
    }
    if (t < N) b[t] = r[t] - s[t] * (*sumV) * invM;
}

__global__ void shifted_sums_kernel(const double *__restrict__ sphi, const double *__restrict__ c, long long M,
                                    int N, double *__restrict__ s) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < N) s[t] = sphi[t] - (double)M * c[t];
}

// ---- FP64 separable reciprocal sum ----
// The transform of recip_sep.cu with the exact per-axis lattice phases ex, ey, ez of the grid
// (tables of the Ewald object) and W_a(n) = w_k e^{-i k.r_a},
//   F[l][n2][a][n1] = sum_n3 ez[n3][l] W[n2][n3][a][n1]      (every grid plane l)
//   E[r][a][n1]     = sum_n2 ey[n2][j_r] F[l_r][n2][a][n1]    (the rows r that hold kept points)
//   Phi[m][a]      += Re sum_n1 ex[n1][i_m] E[r_m][a][n1]     (every kept point)
// The FP64 fit (Num64) takes every stage in FP64; the refit (NumDf) the first two in double-float
// (~2^-46 relative, on the FP32 pipe, whose rate is many times the FP64 pipe's here), the
// weights and stage C in FP64.
// n1 in [0, P], n2, n3 in [-P, P], P = KMAX - 1 (stored with offset P; the FP64 tables
// carry offset KMAX).  On the 2000-atom triclinic cube this is ~35 GFLOP instead of the
// flat k-table's 158 (repeat.py:968-981 evaluated as one DGEMM).
struct RecBasis {
    double rb[9];
};

// U[a][d][n + P] = e^{-i n (b_d . r_a)}
__global__ void atom_phases64_kernel(const double *__restrict__ atoms, int N, RecBasis B, int P,
                                     double2 *__restrict__ U) {
    const int nw = 2 * P + 1;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * 3 * nw) return;
    const int n = t % nw - P, d = (t / nw) % 3, a = t / (3 * nw);
    const double *p = atoms + 3 * a;
    const double th = (p[0] * B.rb[3 * d] + p[1] * B.rb[3 * d + 1]) + p[2] * B.rb[3 * d + 2];
    double sn, cs;
    sincos((double)n * th, &sn, &cs);
    U[t] = make_double2(cs, -sn);
}

__device__ __forceinline__ double2 cmul64(double2 x, double2 y) {
    return make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
}

// The numbers of the plane and row stages: how they are stored, and a complex multiply-accumulate
struct Num64 {
    using T = double2;
    struct Acc {
        double x = 0.0, y = 0.0;
    };
    static __device__ __forceinline__ T store(double re, double im) { return make_double2(re, im); }
    static __device__ __forceinline__ void mac(Acc &a, T p, T q) {
        a.x = fma(p.x, q.x, a.x);
        a.x = fma(-p.y, q.y, a.x);
        a.y = fma(p.x, q.y, a.y);
        a.y = fma(p.y, q.x, a.y);
    }
    static __device__ __forceinline__ T pack(const Acc &a) { return make_double2(a.x, a.y); }
    static __device__ __forceinline__ double2 value(const Acc &a) { return make_double2(a.x, a.y); }
};
struct NumDf {
    using T = float4;
    struct Acc {
        dfa::acc re{0.f, 0.f}, im{0.f, 0.f};
    };
    static __device__ __forceinline__ T store(double re, double im) { return dfa::split(re, im); }
    static __device__ __forceinline__ void mac(Acc &a, const T &p, const T &q) { dfa::cmac(a.re, a.im, p, q); }
    static __device__ __forceinline__ T pack(const Acc &a) { return dfa::pack(a.re, a.im); }
    static __device__ __forceinline__ double2 value(const Acc &a) {
        return make_double2(dfa::to_double(a.re), dfa::to_double(a.im));
    }
};

// W[n2'][n3'][a][n1] = w_k e^{-i k.r_a} for the k-set (zero elsewhere: cleared before), from
// FP64 phase products
template <class Num>
__global__ void build_w64_kernel(const int *__restrict__ kidx, const double *__restrict__ kcoef, int K, int N,
                                 int P, const double2 *__restrict__ U, typename Num::T *__restrict__ W) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)N * K) return;
    const int a = (int)(t / K), k = (int)(t - (long long)a * K);
    const int nw = 2 * P + 1, n1c = P + 1;
    const int n1 = kidx[3 * k], n2 = kidx[3 * k + 1] + P, n3 = kidx[3 * k + 2] + P;
    const double2 *u = U + (size_t)a * 3 * nw;
    const double2 v = cmul64(cmul64(u[n1 + P], u[nw + n2]), u[2 * nw + n3]);
    const double w = kcoef[k];
    W[(((size_t)n2 * nw + n3) * N + a) * n1c + n1] = Num::store(w * v.x, w * v.y);
}

// stage A: one thread per (l, n2, a, n1), n1 fastest
template <class Num>
__global__ void stage_a64_kernel(const typename Num::T *__restrict__ W, const typename Num::T *__restrict__ ez, int nz,
                                 int N, int P, typename Num::T *__restrict__ F) {
    const int nw = 2 * P + 1, n1c = P + 1;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)nz * nw * N * n1c) return;
    const long long an = (long long)N * n1c;
    const int r = (int)(t % an);           // a n1c + n1
    const int n2 = (int)((t / an) % nw), l = (int)(t / (an * nw));
    typename Num::Acc acc;
    for (int n3 = 0; n3 < nw; ++n3) Num::mac(acc, ez[(size_t)n3 * nz + l], W[((size_t)n2 * nw + n3) * an + r]);
    F[t] = Num::pack(acc);
}

// stage B over the listed rows (row = j + l ny, *R of them, a count the host does not wait for): one
// thread per (a, n1), n1 fastest, the blocks along y striding over the rows; E is stored in FP64.
template <class Num>
__global__ void __launch_bounds__(128) stage_b64_kernel(const typename Num::T *__restrict__ F,
                                                        const typename Num::T *__restrict__ ey, int ny, int N, int P,
                                                        const int *__restrict__ rows, const int *__restrict__ R,
                                                        double2 *__restrict__ E) {
    const int nw = 2 * P + 1, n1c = P + 1, nr = *R;
    const long long an = (long long)N * n1c, r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= an) return;
    for (int ri = blockIdx.y; ri < nr; ri += gridDim.y) {
        const int row = rows[ri], l = row / ny, j = row - l * ny;
        typename Num::Acc acc;
        for (int n2 = 0; n2 < nw; ++n2) Num::mac(acc, ey[(size_t)n2 * ny + j], F[((size_t)l * nw + n2) * an + r]);
        E[ri * an + r] = Num::value(acc);
    }
}

// mark the grid rows that hold kept points m0 .. m0+rows-1
__global__ void mark_rows_kernel(const int32_t *__restrict__ kept, long long m0, long long rows, int nx,
                                 unsigned char *__restrict__ mark) {
    const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (m < rows) mark[kept[m0 + m] / nx] = 1;
}

// the marked rows numbered in order (one CTA): rowmap[row] their numbers, rowlist their rows, *R their
// count
__global__ void __launch_bounds__(1024) number_rows_kernel(const unsigned char *__restrict__ mark, int nrows,
                                                           int *__restrict__ rowmap, int *__restrict__ rowlist,
                                                           int *__restrict__ R) {
    __shared__ int part[1024];
    const int t = threadIdx.x, per = (nrows + 1023) / 1024, b0 = min(t * per, nrows), b1 = min(b0 + per, nrows);
    int c = 0;
    for (int b = b0; b < b1; ++b) c += mark[b];
    part[t] = c;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const int v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = t == 0 ? 0 : part[t - 1];
    for (int b = b0; b < b1; ++b)
        if (mark[b]) {
            rowmap[b] = run;
            rowlist[run++] = b;
        }
    if (t == 1023) *R = part[1023];
}

// stage C: phi[m][a] = Re sum_n1 ex[n1][i] E[rowmap[row]][a][n1], rows of phi ld apart  (one thread per
// (m, a), a fastest)
__global__ void stage_c64_kernel(const double2 *__restrict__ E, const double2 *__restrict__ ex, int nx, int N,
                                 int P, const int32_t *__restrict__ kept, long long m0, long long rows,
                                 const int *__restrict__ rowmap, double *__restrict__ phi, int ld) {
    const int n1c = P + 1;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= rows * N) return;
    const long long m = t / N;
    const int a = (int)(t - m * N);
    const int f = kept[m0 + m], row = f / nx, i = f - row * nx;
    const double2 *e = E + ((size_t)rowmap[row] * N + a) * n1c;
    double s = 0.0;
    for (int n1 = 0; n1 < n1c; ++n1) {
        const double2 x = ex[(size_t)n1 * nx + i], v = e[n1];
        s += x.x * v.x - x.y * v.y;
    }
    phi[m * ld + a] = s;
}

}  // namespace

void column_sums_fp64(const double *X, int64_t rows, int cols, int ld, double *out, bool accumulate, rp_ctx *ctx,
                      cudaStream_t s) {
    int nslab = (int)((rows + kSlab - 1) / kSlab);
    if (nslab == 0) {
        if (!accumulate) RP_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * cols, s));
        return;
    }
    double *part = ctx->buf_t<double>("colsum_part", (size_t)nslab * cols);
    dim3 g1(ceil_div(cols, 128), nslab);
    colsum_stage1<<<g1, 128, 0, s>>>(X, rows, cols, ld, part);
    RP_LAUNCH_CHECK();
    colsum_stage2<<<ceil_div(cols, 128), 128, 0, s>>>(part, nslab, cols, out, accumulate ? 1 : 0);
    RP_LAUNCH_CHECK();
}

void finish_normal_equations(const double *G, const double *r, const double *s_c, double *sumV_dev, int64_t M, int N,
                             double *A, double *b, cudaStream_t s) {
    long long n = std::max<long long>((long long)N * N, N);
    finish_kernel<<<ceil_div(n, 256), 256, 0, s>>>(G, r, s_c, sumV_dev, M, N, A, b);
    RP_LAUNCH_CHECK();
}

namespace {
// W and the plane stage; returns F
template <class Num>
typename Num::T *recip_planes64(rp_ctx *ctx, const rp_ewald *ew, const double *d_atoms, int N,
                                const typename Num::T *ez, cudaStream_t stream) {
    using T = typename Num::T;
    const int P = ew->kmax - 1, nw = 2 * P + 1, n1c = P + 1, nz = ew->grid.n_grid[2], K = ew->K;
    double2 *U = ctx->buf_t<double2>("g64_U", (size_t)N * 3 * nw);
    T *W = ctx->buf_t<T>("g64_W", (size_t)nw * nw * N * n1c);
    T *F = ctx->buf_t<T>("g64_F", (size_t)nz * nw * N * n1c);
    RP_CUDA(cudaMemsetAsync(W, 0, sizeof(T) * (size_t)nw * nw * N * n1c, stream));
    RecBasis rb;
    for (int q = 0; q < 9; ++q) rb.rb[q] = ew->rec[q];
    atom_phases64_kernel<<<ceil_div(N * 3 * nw, 128), 128, 0, stream>>>(d_atoms, N, rb, P, U);
    RP_LAUNCH_CHECK();
    build_w64_kernel<Num><<<ceil_div((long long)N * K, 128), 128, 0, stream>>>(ew->d_kidx, ew->d_kcoef, K, N, P, U, W);
    RP_LAUNCH_CHECK();
    stage_a64_kernel<Num><<<ceil_div((long long)nz * nw * N * n1c, 128), 128, 0, stream>>>(W, ez, nz, N, P, F);
    RP_LAUNCH_CHECK();
    return F;
}
}  // namespace

void gram_fp64(rp_ctx *ctx, const rp_ewald *ew, const double *atoms, int N, const int32_t *kept_idx_dev,
               const double *Vc_dev, int64_t M, double *A_dev, double *b_dev, double *sum_phi_dev,
               cudaStream_t stream, bool refit) {
    RP_REQUIRE(N > 0 && M > 0, "rp_gram: need N > 0 and M > 0");
    std::vector<double> sh;
    int zero_idx = -1;
    prune_shifts(ew, atoms, N, sh, zero_idx);
    const int S = (int)(sh.size() / 3);
    double *d_atoms = ctx->buf_t<double>("g_atoms", 3 * (size_t)N);
    double *d_shifts = ctx->buf_t<double>("g_shifts", sh.size());
    double *d_axis = ctx->buf_t<double>("g_axis", 9);
    RP_CUDA(cudaMemcpyAsync(d_atoms, atoms, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_shifts, sh.data(), sizeof(double) * sh.size(), cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_axis, ew->grid.axis, sizeof(double) * 9, cudaMemcpyHostToDevice, stream));

    // reciprocal part: the FP64 phase tables carry the offset KMAX on n2 and n3, the sum's range
    // starts at -(KMAX - 1)
    const int kp = ew->kmax - 1, n1c = kp + 1, nw = 2 * kp + 1;  // the separable sum's n range
    const int nx = ew->grid.n_grid[0], ny = ew->grid.n_grid[1], nz = ew->grid.n_grid[2], K = ew->K;
    const bool recip = K > 0 && kp >= 0;
    const size_t nrows = (size_t)ny * nz;

    // Points of a chunk, by the sizes alone (each chunk's Gram is rounded once, so what is left of the
    // scratch budget must not choose it): Phi and the reciprocal rows, at most one per point, within 4 GB;
    // without them Phi and the Gram's digits within 2 GB.
    const size_t point = sizeof(double) * (size_t)N, point_words = 16 * ((size_t)N + 1);
    const size_t per_point = recip ? point + sizeof(double2) * (size_t)N * n1c : point + point_words;
    int64_t chunk = std::max<int64_t>(256, (int64_t)(((size_t)(recip ? 4 : 2) << 30) / per_point));
    chunk = std::min<int64_t>(chunk, M);

    // Atoms of a block of the reciprocal sum, whose planes (W, F) and rows (E) are held at a time: all where
    // they fit, else fewer, with the planes formed again for every chunk.  Each atom's column is its own,
    // so the blocks do not change it.  The share is at least what an FP64 fit with a flat table of the
    // K wave vectors holds (the tables of a chunk of points and of the atoms), and for the refit the whole but
    // for the reciprocal rows that the points cannot need and a copy of the Gram's 2 (N + 1) columns.
    const size_t most_rows = std::min<size_t>(nrows, (size_t)chunk);
    auto recip_bytes = [&](size_t atoms_, size_t rows_) {
        return recip ? 16 * atoms_ * n1c * ((size_t)nw * nw + (size_t)nz * nw + rows_) + 48 * atoms_ * nw : 0;
    };
    const size_t words = gram_words_bytes(ctx, chunk, N), whole = recip_bytes(N, most_rows) + point * chunk + words;
    size_t need;
    if (refit) {
        need = recip_bytes(N, (size_t)ceil_div(chunk, nx)) + point * chunk + words + 32 * ((size_t)N + 1) * (N + 1);
    } else {
        const size_t flat = 16 * (size_t)K + point, flat_chunk = std::min<size_t>((size_t)M, std::max<size_t>(256, ((size_t)2 << 30) / flat));
        need = 16 * (size_t)K * N + flat * flat_chunk;
    }
    const size_t share = scratch_share(ctx, {"g64_U", "g64_W", "g64_F", "g64_E", "g64_P", "w64_X0", "w64_X1", "w64_X2", "w64_X3", "w64_tsum"}, need);
    int block = N;
    size_t words_share = words;
    if (whole > share) {
        const size_t rest = share > point * chunk ? share - point * chunk : 0;
        if (recip) block = (int)std::min<size_t>(N, std::max<size_t>(1, rest / 2 / recip_bytes(1, most_rows)));
        words_share = rest > recip_bytes(block, most_rows) ? rest - recip_bytes(block, most_rows) : 0;
        words_share = std::max<size_t>(words_share, 4 << 20);  // (64 columns and 3700 points at a time)
    }
    double2 *F64 = nullptr;
    float4 *Fdf = nullptr;
    auto planes = [&](int a0, int na) {
        if (refit) Fdf = recip_planes64<NumDf>(ctx, ew, d_atoms + 3 * (size_t)a0, na, ew->d_ezf, stream);
        else F64 = recip_planes64<Num64>(ctx, ew, d_atoms + 3 * (size_t)a0, na, ew->d_ez + nz, stream);
    };
    if (recip && block == N) {
        StageTimer tt(ctx, "fp64_recip_sep", stream);
        planes(0, N);
    }
    double *P = ctx->buf_t<double>("g64_P", (size_t)chunk * N);
    double *G = ctx->buf_t<double>("g64_G", (size_t)N * N);
    double *r = ctx->buf_t<double>("g64_r", (size_t)N);
    double *sphi = sum_phi_dev ? sum_phi_dev : ctx->buf_t<double>("g64_sphi", (size_t)N);
    double *csum = ctx->buf_t<double>("g64_csum", (size_t)N);
    double *c = ctx->buf_t<double>("g64_c", (size_t)N);
    double *s_c = ctx->buf_t<double>("g64_sc", (size_t)N);
    double *sumV = ctx->buf_t<double>("g64_sumV", 1);
    RP_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * N * N, stream));
    RP_CUDA(cudaMemsetAsync(r, 0, sizeof(double) * N, stream));
    RP_CUDA(cudaMemsetAsync(sphi, 0, sizeof(double) * N, stream));

    // the real-space term's table over the cutoff's range (the 1/r basis has alpha 0 and no cutoff)
    ErfcTable tab{nullptr, 0, 0};
    if (recip) tab = erfc_table(ctx, "g64_erfc", ew->sqrt_alpha, ew->cutoff, stream);
    const double d2_in = square_limit(ew->cutoff), d2_self = square_limit(1e-10);

    cublasHandle_t h = ctx->blas();
    RP_CUBLAS(cublasSetStream(h, stream));
    const double one = 1.0;
    for (int64_t m0 = 0; m0 < M; m0 += chunk) {
        const int64_t rows = std::min<int64_t>(chunk, M - m0);
        if (recip) {
            StageTimer tt(ctx, "fp64_recip_sep", stream);
            // the grid rows of this chunk's points, numbered on the device
            const int64_t most = std::min<int64_t>((int64_t)nrows, rows);
            unsigned char *mark = ctx->buf_t<unsigned char>("g64_mark", nrows);
            int *rowmap = ctx->buf_t<int>("g64_rowmap", nrows);
            int *rowlist = ctx->buf_t<int>("g64_rowlist", (size_t)most + 1);  // the count after the rows
            RP_CUDA(cudaMemsetAsync(mark, 0, nrows, stream));
            mark_rows_kernel<<<ceil_div(rows, 256), 256, 0, stream>>>(kept_idx_dev, m0, rows, nx, mark);
            RP_LAUNCH_CHECK();
            number_rows_kernel<<<1, 1024, 0, stream>>>(mark, (int)nrows, rowmap, rowlist, rowlist + most);
            RP_LAUNCH_CHECK();
            double2 *E64 = ctx->buf_t<double2>("g64_E", (size_t)most * block * n1c);
            for (int a0 = 0; a0 < N; a0 += block) {
                const int na = std::min(block, N - a0);
                if (block < N) planes(a0, na);
                // about 32 blocks per SM, or one per row
                const unsigned bx = ceil_div((long long)na * n1c, 128);
                const dim3 nb(bx, (unsigned)std::max<int64_t>(1, std::min<int64_t>(most, 32LL * std::max(1, ctx->sm_count) / bx)));
                if (refit)
                    stage_b64_kernel<NumDf><<<nb, 128, 0, stream>>>(Fdf, ew->d_eyf, ny, na, kp, rowlist, rowlist + most, E64);
                else
                    stage_b64_kernel<Num64><<<nb, 128, 0, stream>>>(F64, ew->d_ey + ny, ny, na, kp, rowlist, rowlist + most,
                                                                    E64);
                RP_LAUNCH_CHECK();
                stage_c64_kernel<<<ceil_div(rows * na, 128), 128, 0, stream>>>(E64, ew->d_ex, nx, na, kp, kept_idx_dev, m0,
                                                                               rows, rowmap, P + a0, N);
                RP_LAUNCH_CHECK();
            }
        } else {  // the non-periodic basis has no reciprocal part
            RP_CUDA(cudaMemsetAsync(P, 0, sizeof(double) * (size_t)rows * N, stream));
        }
        {
            StageTimer t_r(ctx, "fp64_realspace", stream);
            const size_t smem = realspace_fp64_smem(recip);  // candidates (and the pair queue): 32 or 36 KB
            auto kern = recip ? realspace_fp64_kernel<true> : realspace_fp64_kernel<false>;
            smem_optin((const void *)kern, smem);
            kern<<<dim3(ceil_div(rows, kRsPts), ceil_div(N, kRsAtoms)), kRsPts, smem, stream>>>(
                kept_idx_dev, m0, rows, d_axis, nx, ny, d_atoms, N, d_shifts, S, zero_idx, ew->cutoff, ew->sqrt_alpha,
                d2_in, d2_self, tab, P);
            RP_LAUNCH_CHECK();
        }
        column_sums_fp64(P, rows, N, N, csum, false, ctx, stream);
        // sphi += csum (accumulating stage-2 output keeps the order fixed)
        {
            const double *cs = csum;
            RP_CUBLAS(cublasDaxpy(h, N, &one, cs, 1, sphi, 1));
        }
        if (m0 == 0) {
            set_mean_kernel<<<ceil_div(N, 128), 128, 0, stream>>>(csum, N, 1.0 / (double)rows, c);
            RP_LAUNCH_CHECK();
        }
        shift_columns_kernel<<<ceil_div(rows * N, 256), 256, 0, stream>>>(P, rows, N, c);
        RP_LAUNCH_CHECK();
        // the exact two-word Gram on the tensor cores (G full, r included)
        StageTimer t_g(ctx, "fp64_gram_words", stream);
        gram_words_fp64(ctx, P, rows, N, Vc_dev + m0, G, r, words_share, stream);
    }
    column_sums_fp64(Vc_dev, M, 1, 1, sumV, false, ctx, stream);
    shifted_sums_kernel<<<ceil_div(N, 128), 128, 0, stream>>>(sphi, c, M, N, s_c);
    RP_LAUNCH_CHECK();
    finish_normal_equations(G, r, s_c, sumV, M, N, A_dev, b_dev, stream);
}

}  // namespace rp
