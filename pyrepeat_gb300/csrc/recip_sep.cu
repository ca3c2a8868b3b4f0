// Reciprocal-space Ewald sum by separable lattice phases (double-float, FP32 pipe).
//
// The k-sum of the reference (repeat.py:968-981; per point and atom
// sum_k w_k cos(k.(g - r_a)), w_k = kcoef) is evaluated for grid points, and a
// grid point g = i a0 + j a1 + l a2 of an n_x x n_y x n_z grid that spans the cell
// has k.g = 2 pi (n1 i/n_x + n2 j/n_y + n3 l/n_z) exactly for every reciprocal
// vector k = (n1, n2, n3).  With W_a(n) = w_k e^{-i k.r_a} (zero outside the k-set)
//
//   phi_recip(g, a) = Re sum_n1 ex[n1][i] sum_n2 ey[n2][j] sum_n3 ez[n3][l] W_a(n)
//
// is a three-stage separable transform, evaluated as
//   stage A   F[l][a][n2][n1] = sum_n3 ez[n3][l] W[a][n3][n2][n1]       (every grid plane l)
//   stage B   E[r][a][n1]     = sum_n2 ey[n2][j] F[l][a][n2][n1]         (every grid row r = j + l n_y)
//   stage C   phi_recip(m, a) = Re sum_n1 ex[n1][i_m] E[r_m][a][n1]      (per kept point, fused into
//                                                                        the real-space kernel)
// Stage C costs 2 KMAX real multiply-adds per point-atom instead of the 4 K of a dense
// point x k table contraction (K = 754 at KMAX 7): ~50x fewer operations, so the
// whole sum runs on the FP32 pipe instead of as a tensor-core GEMM.  The weights W
// are computed in double-float (~2^-44) and stored rounded to FP32; stages A, B and C
// use FP32 products (unbiased rounding, ~1e-7 relative like the FP32 real-space terms;
// measured 2.6-3.1e-7 of max|Phi| against FP64), with F and E stored as float2.
// Indices n1 in [0, P], n2, n3 in [-P, P] with P = KMAX - 1 (the k-set keeps
// n1^2 + n2^2 + n3^2 < KMAX^2); stored with offset P on n2 and n3.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "df.cuh"
#include "f32x2.cuh"

namespace rp {
namespace {

// One fit's reciprocal rows: its tables, scratch and output.  A launch carries up to
// kRecipJobs of them by value; every kernel below runs the blocks of all its jobs, job j
// owning blocks [blk[k][j], blk[k][j+1]) of kernel k, so a pipeline group of cubes costs one
// launch per stage instead of one per cube.
struct RecipJob {
    const double *atoms;   // [3N]
    const double *q;       // [N] charges (one weighted column) or nullptr (a column per atom)
    const int *kidx;       // [3K]
    const double *kcoef;   // [K]
    const float4 *EY, *EZ; // double-float phases of the grid rows / planes
    double2 *U;
    float4 *Udf;
    float2 *kdf;           // [K] the weights w_k as double-float (hi, lo), split once per fit
    float2 *W, *F, *E;
    double rb[9];          // reciprocal basis (rows)
    int N, ncols, K, P, ny, nz, ab;
    int ea, ra;            // stage A: (n2, n1) entries and planes of a CTA
    int ecols;             // columns of E's rows (recip_cols)
    const uint8_t *marks;  // [nz][ny / kJB, rounded up] whether stage B writes those rows, or null: all
};
constexpr int kRecipJobs = 64;
struct RecipLaunch {
    int n;
    int blk[kRecipJobs + 1];  // block offsets of the jobs in this kernel's grid
    RecipJob job[kRecipJobs];
};

// the job that owns block b (binary search over the offsets)
__device__ __forceinline__ int recip_job_of(const RecipLaunch &L, int b) {
    int lo = 0, hi = L.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (L.blk[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// U[a][d][n + P] = e^{-i n (b_d . r_a)} for n in [-P, P]: the per-axis atom phases, so that
// e^{-i k.r_a} = U[a][0][n1] U[a][1][n2] U[a][2][n3] needs 3 (2P+1) sincos per atom instead of K.
__global__ void atom_phases_kernel(const __grid_constant__ RecipLaunch L) {
    const int jb = recip_job_of(L, blockIdx.x);
    const RecipJob &J = L.job[jb];
    const int P = J.P, nw = 2 * P + 1;
    const int t = (blockIdx.x - L.blk[jb]) * blockDim.x + threadIdx.x;
    // the weights' double-float split for build_w_kernel, whose threads would otherwise each
    // run the FP64 conversions (the FP64 pipe is a small fraction of the FP32 rate here)
    const int nthreads = (L.blk[jb + 1] - L.blk[jb]) * blockDim.x;
    for (int k = t; k < J.K; k += nthreads) {
        const double w = J.kcoef[k];
        const float wh = (float)w;
        J.kdf[k] = make_float2(wh, (float)(w - (double)wh));
    }
    if (t >= J.N * 3 * nw) return;
    const int n = t % nw - P, d = (t / nw) % 3, a = t / (3 * nw);
    const double *p = J.atoms + 3 * a;
    const double th = (p[0] * J.rb[3 * d] + p[1] * J.rb[3 * d + 1]) + p[2] * J.rb[3 * d + 2];
    double s, c;
    sincos((double)n * th, &s, &c);
    J.U[t] = make_double2(c, -s);
    J.Udf[t] = dfa::split(c, -s);
}

__device__ __forceinline__ double2 cmul(double2 x, double2 y) {
    return make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
}

// W[col][n3'][n2'][n1] = w_k e^{-i k.r} (col = atom), or sum_a q_a w_k e^{-i k.r_a} (one
// charge-weighted column when q != nullptr), stored rounded to FP32.  Per atom the two
// phase products and the weight are double-float products on the FP32 pipe (~2^-44
// relative); the charge-weighted sum stays FP64.  (W is zero outside the k-set: the host
// clears it before this launch.)
__global__ void build_w_kernel(const __grid_constant__ RecipLaunch L) {
    const int jb = recip_job_of(L, blockIdx.x);
    const RecipJob &J = L.job[jb];
    long long t = (long long)(blockIdx.x - L.blk[jb]) * blockDim.x + threadIdx.x;
    const int K = J.K, P = J.P, lane = threadIdx.x & 31;
    if (J.q) t >>= 5;  // the charge-weighted column: a warp per k, its lanes over the atoms
    if (t >= (long long)J.ncols * K) return;
    const int col = (int)(t / K), k = (int)(t - (long long)col * K);
    const int n1c = P + 1, nw = 2 * P + 1;
    const int n1 = J.kidx[3 * k], n2 = J.kidx[3 * k + 1] + P, n3 = J.kidx[3 * k + 2] + P;
    float2 *out = J.W + (((long long)col * nw + n3) * nw + n2) * n1c + n1;
    if (J.q == nullptr) {
        const float4 *u = J.Udf + (size_t)col * 3 * nw;
        dfa::acc re{0.f, 0.f}, im{0.f, 0.f};
        dfa::cmac(re, im, u[n1 + P], u[nw + n2]);
        const float4 z12 = dfa::pack(re, im);
        re = im = dfa::acc{0.f, 0.f};
        dfa::cmac(re, im, z12, u[2 * nw + n3]);
        const float4 z3 = dfa::pack(re, im);
        const float2 wk = J.kdf[k];
        const float wh = wk.x, wl = wk.y;
        re = im = dfa::acc{0.f, 0.f};
        dfa::mac(re, wh, wl, z3.x, z3.y);
        dfa::mac(im, wh, wl, z3.z, z3.w);
        *out = make_float2(dfa::norm(re).x, dfa::norm(im).x);
        return;
    }
    double2 z = make_double2(0.0, 0.0);
    for (int a = lane; a < J.N; a += 32) {
        const double2 *u = J.U + (size_t)a * 3 * nw;
        const double2 v = cmul(cmul(u[n1 + P], u[nw + n2]), u[2 * nw + n3]);
        z.x += J.q[a] * v.x;
        z.y += J.q[a] * v.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        z.x += __shfl_xor_sync(0xffffffffu, z.x, o);
        z.y += __shfl_xor_sync(0xffffffffu, z.y, o);
    }
    const double w = J.kcoef[k];
    if (lane == 0) *out = make_float2((float)(w * z.x), (float)(w * z.y));
}

// Stages A and B are the same product, out[row][r] = sum_k t[k][row] f[k][r] (complex), with the planes
// and ez, or a plane's rows and ey, as rows.  f and the phases t, split into cosines and sines, sit
// in shared memory.  A thread owns kJB consecutive rows of two entries r: per k it reads two values
// of f and eight rows of phases (warp broadcasts) for 32 packed FMAs, two rows to an
// instruction, in the order of k and with the roundings of a scalar loop; a warp's stores of a row are
// consecutive in r.
// Bound by the FMA pipe, which a packed FMA holds for two cycles.  Measured per launch against one
// thread per eight n1 reading W through L1 (stage A) and one entry per thread with scalar FMAs
// (stage B, 60 instructions per k for 32 FMAs): 99 us from 291 and 359 from 587
// (424 atoms, 128^3, KMAX 12: 0.08 and 7.7 G multiply-adds, 667 MB of E; the FMA pipe is 66 % busy in stage
// B).  Several planes per stage B CTA, for one load of the phases, were slower (406 us).
constexpr int kJB = 8, kRecipT = 128;
__device__ __forceinline__ void rows_load_table(float *cs, float *sn, int np, const float4 *T, int nk, int rows, int r0, int n) {
    for (int q = threadIdx.x; q < nk * np; q += kRecipT) {
        const int k = q / np, j = q - k * np;
        const float4 y = j < n ? T[k * rows + r0 + j] : make_float4(0.f, 0.f, 0.f, 0.f);
        cs[q] = y.x;
        sn[q] = y.z;
    }
}
// entry r is at f[off(r) + k fk]; rows 0 .. n of out, of these the groups of kJB rows that group() lists,
// entries 0 .. an
template <class Off, class Group>
__device__ __forceinline__ void rows_product(const float2 *f, int fk, Off off, int ngroups, Group group, int an, const float *cs, const float *sn, int np,
                                             int nk, int n, float2 *out, long long stride) {
    const int half = (an + 1) >> 1, tasks = half * ngroups;
    for (int task = threadIdx.x; task < tasks; task += kRecipT) {
        const int t = task / half, r = task - t * half, jj = group(t);
        const bool two = r + half < an;
        const float2 *fa = f + off(r), *fb = f + off(two ? r + half : r);
        const float *c = cs + jj * kJB, *s = sn + jj * kJB;
        f2 re[2][kJB / 2], im[2][kJB / 2];
#pragma unroll
        for (int u = 0; u < kJB / 2; ++u) re[0][u] = re[1][u] = im[0][u] = im[1][u] = 0ull;
#pragma unroll 2
        for (int k = 0; k < nk; ++k) {
            const float2 v[2] = {*fa, *fb};
            const ulonglong2 c0 = *reinterpret_cast<const ulonglong2 *>(c), c1 = *reinterpret_cast<const ulonglong2 *>(c + 4);
            const ulonglong2 s0 = *reinterpret_cast<const ulonglong2 *>(s), s1 = *reinterpret_cast<const ulonglong2 *>(s + 4);
            const f2 cc[kJB / 2] = {c0.x, c0.y, c1.x, c1.y}, ss[kJB / 2] = {s0.x, s0.y, s1.x, s1.y};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const f2 x = dup2(v[e].x), y = dup2(v[e].y), ny = dup2(-v[e].y);
#pragma unroll
                for (int u = 0; u < kJB / 2; ++u) {
                    re[e][u] = fma2(cc[u], x, re[e][u]);
                    im[e][u] = fma2(cc[u], y, im[e][u]);
                }
#pragma unroll
                for (int u = 0; u < kJB / 2; ++u) {
                    re[e][u] = fma2(ss[u], ny, re[e][u]);
                    im[e][u] = fma2(ss[u], x, im[e][u]);
                }
            }
            fa += fk;
            fb += fk;
            c += np;
            s += np;
        }
        float2 *o = out + jj * kJB * stride + r;
#pragma unroll
        for (int u = 0; u < kJB / 2; ++u) {
            float2 a, b;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (e == 1 && !two) continue;
                unpack2(re[e][u], a.x, b.x);
                unpack2(im[e][u], a.y, b.y);
                if (jj * kJB + 2 * u < n) o[2 * u * stride + e * half] = a;
                if (jj * kJB + 2 * u + 1 < n) o[(2 * u + 1) * stride + e * half] = b;
            }
        }
    }
}

// Stage A, one CTA per (column, J.ea of its (n2, n1) entries, J.ra planes).
__global__ void __launch_bounds__(kRecipT) recip_stage_a_kernel(const __grid_constant__ RecipLaunch L) {
    extern __shared__ __align__(16) float smem_r[];
    const int jb = recip_job_of(L, blockIdx.x);
    const RecipJob &J = L.job[jb];
    const int n1c = J.P + 1, nw = 2 * J.P + 1, ne = nw * n1c, nc = (ne + J.ea - 1) / J.ea, nr = (J.nz + J.ra - 1) / J.ra;
    int b = blockIdx.x - L.blk[jb];
    const int l0 = (b % nr) * J.ra, n = min(J.ra, J.nz - l0);
    b /= nr;
    const int e0 = (b % nc) * J.ea, an = min(J.ea, ne - e0), a = b / nc;
    const int np = (n + kJB - 1) / kJB * kJB;
    float *cs = smem_r, *sn = cs + nw * np;  // np is a multiple of 8
    float2 *f = reinterpret_cast<float2 *>(sn + nw * np);
    const float2 *w = J.W + (long long)a * nw * ne + e0;
    for (int k = 0; k < nw; ++k)
        for (int r = threadIdx.x; r < an; r += kRecipT) f[k * an + r] = w[k * ne + r];
    rows_load_table(cs, sn, np, J.EZ, nw, J.nz, l0, n);
    __syncthreads();
    rows_product(f, an, [](int r) { return r; }, np / kJB, [](int t) { return t; }, an, cs, sn, np, nw, n,
                 J.F + ((long long)l0 * J.ncols + a) * ne + e0, (long long)J.ncols * ne);
}

// marks[l][j / kJB] = 1 for every kept point's row (j, l) (the host clears them)
__global__ void recip_mark_kernel(const int32_t *__restrict__ kept, const long long *__restrict__ count, int nx, int ny,
                                  uint8_t *__restrict__ marks) {
    const int ng = (ny + kJB - 1) / kJB;
    const long long M = *count;
    for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (long long)gridDim.x * blockDim.x) {
        const int row = kept[m] / nx, l = row / ny;
        marks[(long long)l * ng + (row - l * ny) / kJB] = 1;
    }
}

// Stage B, one CTA per (plane l, block of `ab` columns) of a job: the plane's F of those columns is one
// contiguous slab [a][n2][n1].
__global__ void __launch_bounds__(kRecipT, 6) recip_stage_b_kernel(const __grid_constant__ RecipLaunch L) {
    extern __shared__ __align__(16) float smem_r[];
    const int jb = recip_job_of(L, blockIdx.x);
    const RecipJob &J = L.job[jb];
    const int ncols = J.ncols, ny = J.ny, ab = J.ab;
    const int n1c = J.P + 1, nw = 2 * J.P + 1, ne = nw * n1c;
    const int nbx = (ncols + ab - 1) / ab, bloc = blockIdx.x - L.blk[jb];
    const int l = bloc / nbx, a0 = (bloc - l * nbx) * ab, na = min(ab, ncols - a0);
    const int np = (ny + kJB - 1) / kJB * kJB, ng = np / kJB;
    float *cs = smem_r, *sn = cs + nw * np;
    float2 *f = reinterpret_cast<float2 *>(sn + nw * np);
    int *live = reinterpret_cast<int *>(f + na * ne), nlive = ng;  // the groups to write
    if (J.marks) {
        nlive = 0;
        const uint8_t *m = J.marks + (long long)l * ng;
        for (int t0 = 0; t0 < ng; t0 += 32) {  // (every warp forms the same list)
            const int t = t0 + (threadIdx.x & 31);
            const unsigned on = __ballot_sync(0xffffffffu, t < ng && m[t]);
            if (on >> (threadIdx.x & 31) & 1) live[nlive + __popc(on & ((1u << (threadIdx.x & 31)) - 1))] = t;
            nlive += __popc(on);
        }
        if (nlive == 0) return;
    }
    const float2 *F = J.F + ((long long)l * ncols + a0) * ne;
#pragma unroll 4
    for (int t = threadIdx.x; t < na * ne; t += kRecipT) f[t] = F[t];
    rows_load_table(cs, sn, np, J.EY, nw, ny, 0, ny);
    __syncthreads();
    const bool all = J.marks == nullptr;
    rows_product(f, n1c, [=](int r) { return r / n1c * ne + r % n1c; }, nlive, [=](int t) { return all ? t : live[t]; },
                 na * n1c, cs, sn, np, nw, ny, J.E + ((long long)l * ny * J.ecols + a0) * n1c, (long long)J.ecols * n1c);
}

// stage B's columns per CTA: as many as fit 24 KB of shared memory (at most 16)
int stage_b_columns(int P) {
    const size_t col_bytes = sizeof(float2) * (size_t)(2 * P + 1) * (P + 1);
    return (int)std::max<size_t>(1, std::min<size_t>(16, (24u << 10) / col_bytes));
}
size_t table_bytes(int P, int rows) { return sizeof(float2) * (size_t)(2 * P + 1) * ((rows + kJB - 1) / kJB * kJB); }
size_t stage_b_smem(int P, int ny, int ab) {
    return table_bytes(P, ny) + sizeof(float2) * (size_t)(2 * P + 1) * ab * (P + 1) + sizeof(int) * ((ny + kJB - 1) / kJB);
}

}  // namespace

// E's rows hold an even number of atom columns, so that every second column of a KMAX 7 row
// starts on a 16-byte boundary for the Phi kernel's copies
static int recip_cols(int ncols) { return (ncols + 1) & ~1; }

size_t recip_rows_bytes(const rp_ewald *ew, int ncols) {
    const int P = ew->kmax - 1, n1c = P + 1;
    const long long nrows = (long long)ew->grid.n_grid[1] * ew->grid.n_grid[2];
    return sizeof(float2) * (size_t)nrows * recip_cols(ncols) * n1c;
}

void recip_rows_group(rp_ctx *ctx, const std::vector<RecipRowsJob> &jobs, cudaStream_t stream,
                      const std::string &tag, cudaEvent_t kept_ready) {
    if (jobs.empty()) return;
    // marks of the jobs that write only the rows near kept points
    std::vector<size_t> oM(jobs.size() + 1, 0);
    for (size_t j = 0; j < jobs.size(); ++j) {
        const int *g = jobs[j].ew->grid.n_grid;
        oM[j + 1] = oM[j] + (jobs[j].kept && jobs[j].ew->K > 0 ? (size_t)g[2] * ceil_div(g[1], kJB) : 0);
    }
    uint8_t *marks = oM.back() ? ctx->buf_t<uint8_t>("rs_marks" + tag, oM.back()) : nullptr;
    // scratch of every job in one arena per kind; the W arena is cleared with one memset
    std::vector<size_t> oW(jobs.size() + 1, 0), oF(jobs.size() + 1, 0), oU(jobs.size() + 1, 0),
        oK(jobs.size() + 1, 0);
    for (size_t j = 0; j < jobs.size(); ++j) {
        const rp_ewald *ew = jobs[j].ew;
        const int P = std::max(ew->kmax - 1, 0), n1c = P + 1, nw = 2 * P + 1;
        const int ncols = jobs[j].d_q ? 1 : jobs[j].N;
        const bool live = ew->K > 0;
        oW[j + 1] = oW[j] + (live ? (size_t)ncols * nw * nw * n1c : 0);
        oF[j + 1] = oF[j] + (live ? (size_t)ew->grid.n_grid[2] * nw * ncols * n1c : 0);
        oU[j + 1] = oU[j] + (live ? (size_t)jobs[j].N * 3 * nw : 0);
        oK[j + 1] = oK[j] + (live ? (size_t)ew->K : 0);
    }
    const size_t nj = jobs.size();
    float2 *W = ctx->buf_t<float2>("rs_W" + tag, std::max<size_t>(oW[nj], 1));
    float2 *F = ctx->buf_t<float2>("rs_F" + tag, std::max<size_t>(oF[nj], 1));
    double2 *U = ctx->buf_t<double2>("rs_U" + tag, std::max<size_t>(oU[nj], 1));
    float4 *Udf = ctx->buf_t<float4>("rs_Udf" + tag, std::max<size_t>(oU[nj], 1));
    float2 *kdf = ctx->buf_t<float2>("rs_kdf" + tag, std::max<size_t>(oK[nj], 1));
    if (oW[nj]) RP_CUDA(cudaMemsetAsync(W, 0, sizeof(float2) * oW[nj], stream));
    for (size_t j0 = 0; j0 < nj; j0 += kRecipJobs) {
        const size_t j1 = std::min(nj, j0 + kRecipJobs);
        RecipLaunch L{};
        int blk[4][kRecipJobs + 1] = {};
        // stage A's planes are split over CTAs where the columns alone would leave the GPU idle
        long long cols = 0;
        for (size_t j = j0; j < j1; ++j) cols += jobs[j].d_q ? 1 : jobs[j].N;
        const int splits = (int)std::min<long long>(4, ceil_div(456, std::max<long long>(cols, 1)));
        size_t smem_a = 0, smem_b = 0;
        L.n = 0;
        for (size_t j = j0; j < j1; ++j) {
            const RecipRowsJob &rj = jobs[j];
            const rp_ewald *ew = rj.ew;
            const int ncols = rj.d_q ? 1 : rj.N;
            if (ew->K == 0) {  // no k-vectors (the non-periodic basis): E is zero
                RP_CUDA(cudaMemsetAsync(rj.E, 0, recip_rows_bytes(ew, ncols), stream));
                continue;
            }
            const int P = ew->kmax - 1, n1c = P + 1, nw = 2 * P + 1;
            const int ny = ew->grid.n_grid[1], nz = ew->grid.n_grid[2];
            RecipJob &J = L.job[L.n];
            J.atoms = rj.d_atoms; J.q = rj.d_q; J.kidx = ew->d_kidx; J.kcoef = ew->d_kcoef;
            J.EY = ew->d_eyf; J.EZ = ew->d_ezf;
            J.U = U + oU[j]; J.Udf = Udf + oU[j]; J.kdf = kdf + oK[j]; J.W = W + oW[j]; J.F = F + oF[j];
            J.E = rj.E;
            J.marks = rj.kept ? marks + oM[j] : nullptr;
            for (int q = 0; q < 9; ++q) J.rb[q] = ew->rec[q];
            J.N = rj.N; J.ncols = ncols; J.K = ew->K; J.P = P; J.ny = ny; J.nz = nz; J.ab = stage_b_columns(P);
            J.ecols = rj.d_q ? 1 : recip_cols(ncols);
            // stage A's slab of W: up to 32 KB beside the phases (a column of KMAX 7 is 9.5 KB)
            const int ne = nw * n1c;
            RP_REQUIRE(sizeof(float2) * (size_t)nw * nz <= (200u << 10), "recip_rows: grid too large along z for KMAX");
            const size_t room = std::min<size_t>(32u << 10, (224u << 10) - table_bytes(P, nz));
            const int chunks = (int)ceil_div(ne, std::max<long long>(1, room / (sizeof(float2) * nw)));
            J.ea = (int)ceil_div(ne, chunks);
            J.ra = (int)ceil_div(ceil_div(nz, splits), kJB) * kJB;
            const int k = L.n;
            blk[0][k + 1] = blk[0][k] + (int)ceil_div((long long)rj.N * 3 * nw, 128);
            blk[1][k + 1] = blk[1][k] + (int)ceil_div((long long)ncols * ew->K, rj.d_q ? 4 : 128);
            blk[2][k + 1] = blk[2][k] + ncols * (int)ceil_div(ne, J.ea) * (int)ceil_div(nz, J.ra);
            blk[3][k + 1] = blk[3][k] + (int)ceil_div(ncols, J.ab) * nz;
            smem_a = std::max(smem_a, table_bytes(P, std::min(J.ra, nz)) + sizeof(float2) * (size_t)nw * J.ea);
            smem_b = std::max(smem_b, stage_b_smem(P, ny, J.ab));
            ++L.n;
        }
        if (L.n == 0) continue;
        RP_REQUIRE(smem_b <= (200u << 10), "recip_rows: KMAX too large");
        smem_optin((const void *)recip_stage_a_kernel, smem_a);
        smem_optin((const void *)recip_stage_b_kernel, smem_b);
        auto with = [&](int k) {
            std::copy(blk[k], blk[k] + L.n + 1, L.blk);
            return blk[k][L.n];
        };
        int g = with(0);
        atom_phases_kernel<<<g, 128, 0, stream>>>(L);
        RP_LAUNCH_CHECK();
        g = with(1);
        build_w_kernel<<<g, 128, 0, stream>>>(L);
        RP_LAUNCH_CHECK();
        g = with(2);
        recip_stage_a_kernel<<<g, kRecipT, smem_a, stream>>>(L);
        RP_LAUNCH_CHECK();
        if (oM[j1] > oM[j0]) {
            RP_CUDA(cudaStreamWaitEvent(stream, kept_ready, 0));
            RP_CUDA(cudaMemsetAsync(marks + oM[j0], 0, oM[j1] - oM[j0], stream));
            for (size_t j = j0; j < j1; ++j)
                if (oM[j + 1] > oM[j]) {
                    const int *n = jobs[j].ew->grid.n_grid;
                    recip_mark_kernel<<<152, 256, 0, stream>>>(jobs[j].kept, jobs[j].kept_count, n[0], n[1], marks + oM[j]);
                    RP_LAUNCH_CHECK();
                }
        }
        g = with(3);
        recip_stage_b_kernel<<<g, kRecipT, smem_b, stream>>>(L);
        RP_LAUNCH_CHECK();
    }
}

void recip_rows(rp_ctx *ctx, const rp_ewald *ew, const double *d_atoms, const double *d_q, int N, float2 *E,
                cudaStream_t stream, const std::string &slot) {
    recip_rows_group(ctx, {RecipRowsJob{ew, d_atoms, d_q, N, E}}, stream, slot);
}

}  // namespace rp
