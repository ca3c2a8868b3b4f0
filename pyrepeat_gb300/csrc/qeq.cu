// QEq charges (repeat.py:2539-2634, ChargeCalculator.compute_qeq_charges) on the device.
//
// J, the atoms' Coulomb matrix under the fit's Ewald object (repeat.py:2575-2595):
//   J_ii = j_self[i]  (the idempotential, 2 x hardness)
//   J_ij = sum over the FULL shift list (2 nmax + 1)^3 of erfc(sqrt(alpha) r) / r for every
//          image with r > 1e-10 (repeat.py:2615-2626: no cutoff, unlike the fit's
//          real-space sum)
//        + sum_k w_k cos(k . (r_i - r_j))                       (repeat.py:2628-2632)
// The k-sum is the Gram X^T X of the per-atom columns X = sqrt(w_k) [cos(k.r_a); sin(k.r_a)]
// (the w_k share one sign, the volume's), formed by the exact two-word Gram on the tensor cores (gram_words_fp64: each
// value to 2^-55 of its column's largest, the products summed exactly and rounded once).  A
// pair kernel adds the real-space sum of pair (i < j) and writes J_ij and J_ji, so J is
// exactly symmetric like the reference's.  With KMAX 0 (the non-periodic fit) alpha is 0, the
// shift list is the zero shift alone and there are no k-vectors, so J_ij = 1/r_ij (repeat.py:
// 2588-2595).
// (2000 atoms, K = 754: 0.84 ms against 6.2 for the k-sum as one triangle of an FP64 cuBLAS
// product, 0.18 against 2.6 for the pair kernel with FP64 distances of every image and FP64 erfc.)
//
// The charges: repeat.py:2597-2613 solves sum q = Q together with the rows
// (J q)_{i-1} - (J q)_i = chi_i - chi_{i-1}, i.e. (J q)_i + chi_i is the same for every
// atom.  That is the bordered system [J 1; 1^T 0] [q; mu] = [-chi; Q], the form of the fit's
// total-charge system, so it runs through the same solve (FP32 LU with FP64 refinement, FP64
// LU fallback).  Both systems have the same solution set in q.
#include <vector>

#include "common.cuh"
#include "erfc64.cuh"

namespace rp {
namespace {

// X[k][a] = sqrt(w_k) cos(k.r_a), X[K + k][a] = sqrt(w_k) sin(k.r_a)
__global__ void qeq_tables_kernel(const double *__restrict__ kvec, const double *__restrict__ kcoef, int K,
                                  const double *__restrict__ atoms, int N, double *__restrict__ X) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)N * K) return;
    const int k = (int)(t / N), a = (int)(t - (long long)k * N);
    const double kr =
        (atoms[3 * a] * kvec[3 * k] + atoms[3 * a + 1] * kvec[3 * k + 1]) + atoms[3 * a + 2] * kvec[3 * k + 2];
    double s, c;
    sincos(kr, &s, &c);
    const double w = sqrt(fabs(kcoef[k]));
    X[t] = w * c;
    X[(size_t)K * N + t] = w * s;
}

// 32 x 32 atom pairs (i, j), j block at or right of the i block, per CTA; the tile is transposed in
// shared memory so that both J_ij and J_ji are stored coalesced.  Images are tested in FP32, 32
// at a time, and each lane then runs the FP64 term for its own list (about one image in 27 of a
// 70 Bohr cell): an FP64 instruction holds its pipe for 16 cycles per warp, so a warp pays for
// its longest list instead of for every image that any of its pairs reaches.  On entry J_ij
// holds the Gram (sign: of the w_k; 0: no k-sum).
constexpr int kPairTile = 32;
__global__ void __launch_bounds__(256) qeq_pairs_kernel(const double *__restrict__ atoms, int N,
                                                        const double *__restrict__ shifts, int S, double sa,
                                                        ErfcTable tab, double d2_self, double sign,
                                                        const double *__restrict__ j_self, double *__restrict__ J) {
    __shared__ double tile[kPairTile][kPairTile + 1];
    __shared__ float sh[3][32];
    if (blockIdx.x < blockIdx.y) return;
    const int i0 = blockIdx.y * kPairTile, j0 = blockIdx.x * kPairTile;
    const int jj = threadIdx.x & 31, j = j0 + jj;
    // images with sqrt(alpha) r > 7 are skipped: each would add erfc(7)/r < 1e-24, against
    // entries of order 1e-2..1 whose ulp is above 1e-18 (KMAX 0: alpha 0, nothing is skipped)
    const float far2 = sa > 0.0 ? (float)((7.0 / sa) * (7.0 / sa)) : 3e38f;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // rows i0 + (threadIdx.x >> 5) + 8 u
    for (int s0 = 0; s0 < S; s0 += 32) {
        const int ns = min(32, S - s0);
        __syncthreads();
        if (threadIdx.x < 3 * 32 && (threadIdx.x & 31) < ns)
            sh[threadIdx.x >> 5][threadIdx.x & 31] = (float)shifts[3 * (s0 + (threadIdx.x & 31)) + (threadIdx.x >> 5)];
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + (threadIdx.x >> 5) + 8 * u;
            if (i >= N || j >= N || j <= i) continue;
            const double dx = atoms[3 * i] - atoms[3 * j], dy = atoms[3 * i + 1] - atoms[3 * j + 1],
                         dz = atoms[3 * i + 2] - atoms[3 * j + 2];
            const float fx = (float)dx, fy = (float)dy, fz = (float)dz;
            unsigned list = 0;
            for (int s = 0; s < ns; ++s) {
                const float x = fx + sh[0][s], y = fy + sh[1][s], z = fz + sh[2][s];
                if (!(x * x + y * y + z * z > far2)) list |= 1u << s;
            }
            while (list) {  // in shift order
                const int s = s0 + __ffs(list) - 1;
                list &= list - 1;
                const double x = dx + shifts[3 * s], y = dy + shifts[3 * s + 1], z = dz + shifts[3 * s + 2];
                const double d2 = x * x + y * y + z * z;
                if (!le_bits(d2, d2_self)) acc[u] += erfc_term(d2, tab, sa);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int ii = (threadIdx.x >> 5) + 8 * u, i = i0 + ii;
        double v = 0.0;
        if (i < N && j < N) {
            if (j > i) v = sign != 0.0 ? acc[u] + sign * J[(size_t)i * N + j] : acc[u];
            else if (j == i) v = j_self[i];
            if (j >= i) J[(size_t)i * N + j] = v;
        }
        tile[ii][jj] = v;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // row j0 + r of J: the tile's column r
        const int r = (threadIdx.x >> 5) + 8 * u, row = j0 + r, col = i0 + jj;
        if (row < N && col < N && row > col) J[(size_t)row * N + col] = tile[jj][r];
    }
}

}  // namespace

void qeq_run(rp_ctx *ctx, const rp_ewald *ew, const double *atoms, int N, const double *chi, const double *j_self,
             double qtot, double *q_out, double *J_out, double *info, cudaStream_t stream) {
    RP_REQUIRE(N > 0 && atoms && chi && j_self && q_out, "rp_qeq: need N > 0 and non-null atoms, chi, j_self, q");
    const int K = ew->K, K2 = 2 * ew->K;
    const int S = (int)(ew->shifts.size() / 3);
    RP_REQUIRE(S > 0, "rp_qeq: ewald object has no shifts");
    double *d_atoms = ctx->buf_t<double>("qeq_atoms", 3 * (size_t)N);
    double *d_sh = ctx->buf_t<double>("qeq_shifts", 3 * (size_t)S);
    double *d_js = ctx->buf_t<double>("qeq_jself", (size_t)N);
    double *d_b = ctx->buf_t<double>("qeq_b", (size_t)N);
    double *d_J = ctx->buf_t<double>("qeq_J", (size_t)N * N);
    double *d_q = ctx->buf_t<double>("qeq_q", (size_t)N);
    std::vector<double> nb((size_t)N);
    for (int i = 0; i < N; ++i) nb[i] = -chi[i];
    RP_CUDA(cudaMemcpyAsync(d_atoms, atoms, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_sh, ew->shifts.data(), sizeof(double) * 3 * S, cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_js, j_self, sizeof(double) * N, cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_b, nb.data(), sizeof(double) * N, cudaMemcpyHostToDevice, stream));

    double sign = 0.0;
    ErfcTable tab{nullptr, 0, 0};
    if (K > 0) {
        double *X = ctx->buf_t<double>("qeq_X", (size_t)K2 * N);
        double *zero = ctx->buf_t<double>("qeq_zero", (size_t)K2);  // the Gram's ESP column: none here
        double *rz = ctx->buf_t<double>("qeq_r", (size_t)N);
        {
            StageTimer tt(ctx, "qeq_tables", stream);
            const long long n = (long long)N * K;
            qeq_tables_kernel<<<ceil_div(n, 256), 256, 0, stream>>>(ew->d_kvec, ew->d_kcoef, K, d_atoms, N, X);
            RP_LAUNCH_CHECK();
        }
        sign = ew->kcoef[0] < 0.0 ? -1.0 : 1.0;
        StageTimer tt(ctx, "qeq_recip_gram", stream);
        RP_CUDA(cudaMemsetAsync(zero, 0, sizeof(double) * K2, stream));
        RP_CUDA(cudaMemsetAsync(d_J, 0, sizeof(double) * N * N, stream));
        RP_CUDA(cudaMemsetAsync(rz, 0, sizeof(double) * N, stream));
        status_clear(ctx, stream);
        // (at least what this stage's tables and matrix took as a cuBLAS product)
        const size_t need = (size_t)N * (16 * (size_t)K + 8 * (size_t)N);
        gram_words_fp64(ctx, X, K2, N, zero, d_J, rz,
                        scratch_share(ctx, {"w64_X0", "w64_X1", "w64_X2", "w64_X3", "w64_tsum"}, need), stream);
    }
    if (ew->sqrt_alpha > 0.0) tab = erfc_table(ctx, "qeq_erfc", ew->sqrt_alpha, 7.1 / ew->sqrt_alpha, stream);
    {
        StageTimer tt(ctx, "qeq_pairs", stream);
        const unsigned nb = ceil_div(N, kPairTile);
        qeq_pairs_kernel<<<dim3(nb, nb), 256, 0, stream>>>(d_atoms, N, d_sh, S, ew->sqrt_alpha, tab,
                                                           square_limit(1e-10), sign, d_js, d_J);
        RP_LAUNCH_CHECK();
    }
    if (K > 0) status_check(ctx, stream);
    {
        StageTimer tt(ctx, "qeq_solve", stream);
        static const int no_group[1] = {0};
        solve_run(ctx, d_J, d_b, N, 0, no_group, no_group, nullptr, nullptr, qtot, d_q, info, stream);
    }
    RP_CUDA(cudaMemcpyAsync(q_out, d_q, sizeof(double) * N, cudaMemcpyDeviceToHost, stream));
    if (J_out) RP_CUDA(cudaMemcpyAsync(J_out, d_J, sizeof(double) * N * N, cudaMemcpyDeviceToHost, stream));
    RP_CUDA(cudaStreamSynchronize(stream));
}

}  // namespace rp
