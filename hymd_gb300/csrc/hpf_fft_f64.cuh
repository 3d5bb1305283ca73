// Register transforms on FP64 complex numbers for the energies: the lengths,
// splits and index maps of hpf_fft.cuh.
#pragma once

#include "hpf_fft.cuh"

namespace hpf_fft64 {

using hpf_fft::bitrev;
using hpf_fft::ilog2;
using hpf_fft::is_pow2;
using hpf_fft::split1;
using hpf_fft::Tw;

__device__ __forceinline__ double2 c_add(double2 a, double2 b) {
    return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 c_sub(double2 a, double2 b) {
    return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 c_mul(double2 a, double2 w) {
    return make_double2(fma(a.x, w.x, -(a.y * w.y)), fma(a.x, w.y, a.y * w.x));
}

// v * exp(-2 pi i m / 16), m = 0..7 (compile-time after unrolling)
__device__ __forceinline__ double2 rot16(double2 v, int m) {
    constexpr double c1 = 0.92387953251128675613, c2 = 0.70710678118654752440,
                     c3 = 0.38268343236508977173;
    switch (m) {
        case 0: return v;
        case 4: return make_double2(v.y, -v.x);
        case 2: return make_double2((v.x + v.y) * c2, (v.y - v.x) * c2);
        case 6: return make_double2((v.y - v.x) * c2, -(v.x + v.y) * c2);
        case 1: return c_mul(v, make_double2(c1, -c3));
        case 3: return c_mul(v, make_double2(c3, -c1));
        case 5: return c_mul(v, make_double2(-c3, -c1));
        default: return c_mul(v, make_double2(-c1, -c3));  // m == 7
    }
}

// v * exp(-2 pi i m / 12), m = 0..11
__device__ __forceinline__ double2 rot12(double2 v, int m) {
    constexpr double s = 0.86602540378443864676;
    switch (m) {
        case 0: return v;
        case 3: return make_double2(v.y, -v.x);
        case 6: return make_double2(-v.x, -v.y);
        case 9: return make_double2(-v.y, v.x);
        case 1: return c_mul(v, make_double2(s, -0.5));
        case 2: return c_mul(v, make_double2(0.5, -s));
        case 4: return c_mul(v, make_double2(-0.5, -s));
        case 5: return c_mul(v, make_double2(-s, -0.5));
        case 7: return c_mul(v, make_double2(-s, 0.5));
        case 8: return c_mul(v, make_double2(-0.5, s));
        case 10: return c_mul(v, make_double2(0.5, s));
        default: return c_mul(v, make_double2(s, 0.5));  // m == 11
    }
}

__device__ __forceinline__ void dft3(double2& b0, double2& b1, double2& b2) {
    constexpr double s3 = 0.86602540378443864676;
    const double2 s = c_add(b1, b2), d = c_sub(b1, b2);
    const double2 t = make_double2(fma(-0.5, s.x, b0.x), fma(-0.5, s.y, b0.y));
    const double2 m = make_double2(s3 * d.y, -s3 * d.x);  // -i (sqrt(3)/2) d
    b0 = c_add(b0, s);
    b1 = c_add(t, m);
    b2 = c_sub(t, m);
}

// forward transforms, natural order in and out (as hpf_fft::reg_fft)
template <int R>
__device__ __forceinline__ void reg_fft2(double2 (&a)[R]) {
    constexpr int bits = ilog2(R);
    double2 b[R];
#pragma unroll
    for (int i = 0; i < R; ++i) b[bitrev(i, bits)] = a[i];
#pragma unroll
    for (int h = 1; h < R; h <<= 1) {
#pragma unroll
        for (int i0 = 0; i0 < R; i0 += 2 * h) {
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const double2 u = b[i0 + j];
                const double2 v = rot16(b[i0 + j + h], j * (8 / h));
                b[i0 + j] = c_add(u, v);
                b[i0 + j + h] = c_sub(u, v);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = b[i];
}

template <int R>
__device__ __forceinline__ void reg_fft(double2 (&a)[R]) {
    if constexpr (R % 3 != 0) {
        reg_fft2<R>(a);
    } else {
        constexpr int P = R / 3;
        double2 y[3][P];
#pragma unroll
        for (int n2 = 0; n2 < P; ++n2) {
            double2 b0 = a[n2], b1 = a[P + n2], b2 = a[2 * P + n2];
            dft3(b0, b1, b2);
            y[0][n2] = b0;
            y[1][n2] = rot12(b1, (n2 * (12 / R)) % 12);
            y[2][n2] = rot12(b2, (2 * n2 * (12 / R)) % 12);
        }
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            reg_fft2<P>(y[k1]);
#pragma unroll
            for (int k2 = 0; k2 < P; ++k2) a[k1 + 3 * k2] = y[k1][k2];
        }
    }
}

// twiddle m of length N from the global tables
template <int N>
__device__ __forceinline__ double2 twiddle(const double2* __restrict__ tw, int m) {
    return __ldg(tw + Tw<N>::off + m * Tw<N>::stride);
}

}  // namespace hpf_fft64
