// The real-space Ewald term in FP64 from a table.
#pragma once

#include <cmath>

#include "common.cuh"

namespace rp {
namespace {

// erfc(s sqrt(u)) / sqrt(u), s = sqrt(alpha), as a Taylor polynomial of degree 9 about the centre of u's
// interval, 64 intervals per power of two: |u - centre| <= centre / 128, and over the cutoff's
// range (alpha u <= pi^2) the first term left out is below 2e-18 of the value (beyond it, up to
// alpha u = 49, below 1e-24 of 1 / sqrt(u)).  About 10 FP64
// instructions per term instead of ~75 for erfc, a square root and a division (an FP64
// instruction holds its pipe for 16 cycles per warp here).  The coefficients follow from the
// derivative d/du erfc(s sqrt(u)) = -s / sqrt(pi) e^(-s^2 u) u^(-1/2) by products of the series of
// e^(-s^2 u) and u^(-1/2).
constexpr int kErfcDeg = 9, kErfcPerOctave = 64;
constexpr int kErfcLow = -2;  // from u = 2^-2 (half a Bohr); nearer pairs take the functions themselves
struct ErfcTable {
    const double *c;  // [intervals][kErfcDeg + 1]; nullptr: the functions themselves (the 1/r basis)
    int base;         // high word >> 14 of the first interval
    int n;            // intervals
};
int erfc_intervals(double rc) {  // up to the power of two above Rc^2
    int e = 0;
    std::frexp(rc * rc, &e);
    return std::max(1, e - kErfcLow) * kErfcPerOctave;
}
__global__ void erfc_table_kernel(double sa, int n, int base, double *__restrict__ c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double u = __hiloint2double(((base + i) << 14) | 0x2000, 0);  // the interval's centre
    double h[kErfcDeg + 1], e[kErfcDeg + 1], g[kErfcDeg + 1];
    h[0] = 1.0 / sqrt(u);
    e[0] = exp(-sa * sa * u);
    for (int k = 1; k <= kErfcDeg; ++k) {
        h[k] = h[k - 1] * ((0.5 - k) / (k * u));
        e[k] = e[k - 1] * (-sa * sa / k);
    }
    g[0] = erfc(sa * sqrt(u));
    for (int k = 1; k <= kErfcDeg; ++k) {
        double t = 0.0;
        for (int q = 0; q < k; ++q) t += e[q] * h[k - 1 - q];
        g[k] = -sa * 0.56418958354775628694807945 * t / k;  // 1 / sqrt(pi)
    }
    for (int k = 0; k <= kErfcDeg; ++k) {
        double t = 0.0;
        for (int q = 0; q <= k; ++q) t += g[q] * h[k - q];
        c[(size_t)i * (kErfcDeg + 1) + k] = t;
    }
}
__device__ __noinline__ double erfc_term_direct(double d2, double sa) {
    const double r = sqrt(d2);
    return erfc(sa * r) / r;
}
__device__ __forceinline__ double erfc_term(double d2, const ErfcTable &tab, double sa) {
    const int hi = __double2hiint(d2), i = (hi >> 14) - tab.base;
    if (!tab.c || (unsigned)i >= (unsigned)tab.n) return erfc_term_direct(d2, sa);  // also infinities and NaN
    const double2 *c = reinterpret_cast<const double2 *>(tab.c + (size_t)i * (kErfcDeg + 1));
    const double t = d2 - __hiloint2double((hi & ~0x3fff) | 0x2000, 0);
    double2 q = c[kErfcDeg / 2];
    double v = fma(q.y, t, q.x);
#pragma unroll
    for (int k = kErfcDeg / 2 - 1; k >= 0; --k) {
        q = c[k];
        v = fma(fma(v, t, q.y), t, q.x);
    }
    return v;
}
// The largest double whose (correctly rounded) square root is at most r: r(d2) <= r and d2 <= this are
// the same decision, without the square root.
double square_limit(double r) {
    double t = r * r;
    while (std::sqrt(t) > r) t = std::nextafter(t, 0.0);
    for (double u = std::nextafter(t, 1e308); std::sqrt(u) <= r; u = std::nextafter(u, 1e308)) t = u;
    return t;
}
// a <= b for doubles that are not negative, off the FP64 pipe (their bits order like the values)
__device__ __forceinline__ bool le_bits(double a, double b) { return __double_as_longlong(a) <= __double_as_longlong(b); }

// The table for pairs up to distance r_max, in the ctx's scratch `name`, filled on the stream
ErfcTable erfc_table(rp_ctx *ctx, const std::string &name, double sa, double r_max, cudaStream_t stream) {
    const int n = erfc_intervals(r_max);
    double *t = ctx->buf_t<double>(name, (size_t)n * (kErfcDeg + 1));
    const int base = (1023 + kErfcLow) * kErfcPerOctave;  // exponent and six mantissa bits of 2^kErfcLow
    erfc_table_kernel<<<ceil_div(n, 64), 64, 0, stream>>>(sa, n, base, t);
    RP_LAUNCH_CHECK();
    return ErfcTable{t, base, n};
}

}  // namespace
}  // namespace rp
