// Ewald potential of point charges at grid points: V(g) = sum_a q_a phi_a(g).
//
// Replaces the V_coul = Phi q evaluation of ChargeCalculator.compute_stats
// (repeat.py:2326-2441, used for --stats and --output) without forming Phi:
//   reciprocal  V_r(g) = Re sum_n1 ex[n1][i] E_q[r][n1]: the separable reciprocal
//               sum of recip_sep.cu applied to the structure factor
//               S(k) = sum_a q_a w_k e^{-i k.r_a} (one charge-weighted column)
//   real space  V_s(g) = sum_a q_a sum_s [|g-r_a-s| <= Rc] erfc(sqrt(alpha) r)/r
//               over a per-CTA candidate list of images near the CTA's points.
// Cost per point is O(KMAX + images within Rc) instead of O(N K).  The real-space
// terms are FP32 with double-float accumulation and the reciprocal part FP32
// (relative error ~1e-7), which is what an RMS of the fitted ESP or a synthetic
// ESP needs.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "df.cuh"

namespace rp {
namespace {

constexpr int kPotPts = 128;
constexpr int kPotWarps = kPotPts / 32;
constexpr int kPotCand = 384;  // images per warp and round

// one thread per point: V_r = Re sum_n1 ex[n1][i] E_q[r][n1]
__global__ void __launch_bounds__(kPotPts) potential_recip_kernel(const float4 *__restrict__ EX,
                                                                  const float2 *__restrict__ Eq, int n1c, int nx,
                                                                  const int32_t *__restrict__ idx, long long npts,
                                                                  double *__restrict__ out) {
    const long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= npts) return;
    const int f = idx ? idx[m] : (int)m;
    const int row = f / nx, i = f - row * nx;
    float rs = 0.f;
    for (int n = 0; n < n1c; ++n) {
        const float2 e = Eq[(long long)row * n1c + n];
        rs = dfa::cre32(rs, EX[(long long)n * nx + i], make_float4(e.x, 0.f, e.y, 0.f));
    }
    out[m] = (double)rs;
}

// Image positions atom + shift as double-float: (x, y, z) high parts and the charge, then the low parts
__global__ void potential_images_kernel(const double *__restrict__ atoms, const double *__restrict__ q, int N,
                                        const double *__restrict__ shifts, int S, float4 *__restrict__ img) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * S) return;
    const int a = t / S, s = t - a * S;
    const double x = atoms[3 * a] + shifts[3 * s], y = atoms[3 * a + 1] + shifts[3 * s + 1],
                 z = atoms[3 * a + 2] + shifts[3 * s + 2];
    const float hx = (float)x, hy = (float)y, hz = (float)z;
    img[2 * t] = make_float4(hx, hy, hz, (float)q[a]);
    img[2 * t + 1] = make_float4((float)(x - (double)hx), (float)(y - (double)hy), (float)(z - (double)hz), 0.f);
}

// (ah + al) - (bh + bl) rounded to FP32
__device__ __forceinline__ float df_diff(float ah, float al, float bh, float bl) {
    float s, e;
    dfa::two_sum(ah, -bh, s, e);
    return __fadd_rn(s, __fadd_rn(e, __fadd_rn(al, -bl)));
}

// One CTA per 128 points.  In rounds, each warp tests its share of the images against the points'
// bounding box in FP32 (a ballot per 32, so the order is fixed) and keeps the ones in reach
// relative to the CTA's first point; then every thread sums the terms of all of them.
// What bounds it: the instructions of the terms, 314 us for 270 atoms x 107k points in grid order.
// (With the images' positions formed in FP64 per CTA and culled by a sphere around the points,
// the whole call took 0.88 ms against 0.42: 12 FP64 instructions per image and CTA, each
// holding that pipe for 16 cycles per warp.)
__global__ void __launch_bounds__(kPotPts) potential_real_kernel(
    const double *__restrict__ axis, int nx, int ny, const int32_t *__restrict__ idx, long long npts,
    const float4 *__restrict__ img, int images, double rc, double sa, double *__restrict__ out) {
    __shared__ float4 cand[kPotWarps][kPotCand];  // image position relative to the tile origin, charge
    __shared__ int ncand[kPotWarps];
    __shared__ double origin[3];
    __shared__ float bb[2][3][kPotWarps];
    const long long mb = (long long)blockIdx.x * kPotPts;
    const long long m = mb + threadIdx.x;
    const int layer = nx * ny, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool valid = m < npts;
    double g[3];
    {
        const long long mm = valid ? m : mb;  // a lane past the end repeats the first point
        const int f = idx ? idx[mm] : (int)mm;
        const int l = f / layer, rem = f - l * layer, j = rem / nx, i = rem - j * nx;
        for (int d = 0; d < 3; ++d) g[d] = ((double)i * axis[d] + (double)j * axis[3 + d]) + (double)l * axis[6 + d];
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) origin[d] = g[d];
    __syncthreads();
    const float3 gl = make_float3((float)(g[0] - origin[0]), (float)(g[1] - origin[1]), (float)(g[2] - origin[2]));
    float oh[3], ol[3], lo[3], hi[3];
    {
        const float v[3] = {gl.x, gl.y, gl.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float mn = v[d], mx = v[d];
            for (int o = 16; o > 0; o >>= 1) {
                mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if (lane == 0) {
                bb[0][d][warp] = mn;
                bb[1][d][warp] = mx;
            }
            oh[d] = (float)origin[d];
            ol[d] = (float)(origin[d] - (double)oh[d]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float mn = bb[0][d][0], mx = bb[1][d][0];
        for (int w = 1; w < kPotWarps; ++w) {
            mn = fminf(mn, bb[0][d][w]);
            mx = fmaxf(mx, bb[1][d][w]);
        }
        lo[d] = mn + oh[d];
        hi[d] = mx + oh[d];
    }
    const float reach = (float)rc + 1e-3f;
    const float reach2 = reach * reach, rc2 = (float)(rc * rc), saf = (float)sa;
    dfa::acc acc{0.f, 0.f};  // double-float sum of FP32 terms (no FP64 per pair)
    for (int base = 0; base < images; base += kPotWarps * kPotCand) {
        const int t0 = base + warp * kPotCand, t1 = min(images, t0 + kPotCand);
        int n = 0;
        for (int t = t0 + lane; t - lane < t1; t += 32) {
            bool keep = false;
            float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t < t1) {
                h = img[2 * t];
                const float dx = fmaxf(fmaxf(lo[0] - h.x, h.x - hi[0]), 0.f);
                const float dy = fmaxf(fmaxf(lo[1] - h.y, h.y - hi[1]), 0.f);
                const float dz = fmaxf(fmaxf(lo[2] - h.z, h.z - hi[2]), 0.f);
                keep = !(dx * dx + dy * dy + dz * dz > reach2);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const float4 l = img[2 * t + 1];
                cand[warp][n + __popc(bal & ((1u << lane) - 1u))] =
                    make_float4(df_diff(h.x, l.x, oh[0], ol[0]), df_diff(h.y, l.y, oh[1], ol[1]),
                                df_diff(h.z, l.z, oh[2], ol[2]), h.w);
            }
            n += __popc(bal);
        }
        if (lane == 0) ncand[warp] = n;
        __syncthreads();
        for (int w = 0; w < kPotWarps; ++w) {
            const int nc = ncand[w];
            for (int c = 0; c < nc; ++c) {
                const float4 p = cand[w][c];
                const float dx = gl.x - p.x, dy = gl.y - p.y, dz = gl.z - p.z;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (r2 > rc2 || r2 <= 1e-20f) continue;
                const float rinv = rsqrtf(r2);
                float t, e;
                dfa::two_sum(acc.s, p.w * (erfcf(saf * (r2 * rinv)) * rinv), t, e);
                acc.s = t;
                acc.e = __fadd_rn(acc.e, e);
            }
        }
        __syncthreads();
    }
    if (valid) out[m] += dfa::to_double(acc);
}

}  // namespace

void potential_run(rp_ctx *ctx, const rp_ewald *ew, const double *atoms, const double *q, int N,
                   const int32_t *idx_dev, int64_t npts, double *out_dev, cudaStream_t stream) {
    RP_REQUIRE(atoms && q && out_dev && N > 0 && npts > 0, "rp_potential: bad arguments");
    std::vector<double> sh;
    int zero_idx = -1;
    prune_shifts(ew, atoms, N, sh, zero_idx);
    const int S = (int)(sh.size() / 3);
    RP_REQUIRE((long long)N * S < (1LL << 31), "rp_potential: too many images");
    double *d_atoms = ctx->buf_t<double>("p_atoms", 3 * (size_t)N);
    double *d_q = ctx->buf_t<double>("p_q", (size_t)N);
    double *d_shifts = ctx->buf_t<double>("p_shifts", sh.size());
    double *d_axis = ctx->buf_t<double>("p_axis", 9);
    RP_CUDA(cudaMemcpyAsync(d_atoms, atoms, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_q, q, sizeof(double) * N, cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_shifts, sh.data(), sizeof(double) * sh.size(), cudaMemcpyHostToDevice, stream));
    RP_CUDA(cudaMemcpyAsync(d_axis, ew->grid.axis, sizeof(double) * 9, cudaMemcpyHostToDevice, stream));
    const int nx = ew->grid.n_grid[0], ny = ew->grid.n_grid[1];
    float2 *Eq = ctx->buf_t<float2>("p_Eq", recip_rows_bytes(ew, 1) / sizeof(float2));
    recip_rows(ctx, ew, d_atoms, d_q, N, Eq, stream);
    potential_recip_kernel<<<ceil_div(npts, kPotPts), kPotPts, 0, stream>>>(ew->d_exf, Eq, ew->kmax, nx, idx_dev, npts,
                                                                           out_dev);
    RP_LAUNCH_CHECK();
    float4 *img = ctx->buf_t<float4>("p_img", 2 * (size_t)N * S);
    potential_images_kernel<<<ceil_div((long long)N * S, 128), 128, 0, stream>>>(d_atoms, d_q, N, d_shifts, S, img);
    RP_LAUNCH_CHECK();
    potential_real_kernel<<<ceil_div(npts, kPotPts), kPotPts, 0, stream>>>(d_axis, nx, ny, idx_dev, npts, img, N * S,
                                                                          ew->cutoff, ew->sqrt_alpha, out_dev);
    RP_LAUNCH_CHECK();
}

}  // namespace rp
