// Register transforms on double-float complex numbers (two FP32 words per
// part, about 48 significant bits) for the FP64 energies: the lengths,
// splits and index maps of hpf_fft.cuh, on GB300's FP32 pipe (its FP64 rate
// is 1/64 of it).
#pragma once

#include "hpf_fft.cuh"
#include "hpf_internal.cuh"

namespace hpf_fft_df {

using hpf_fft::bitrev;
using hpf_fft::ilog2;
using hpf_fft::is_pow2;
using hpf_fft::split1;
using hpf_fft::Tw;

// (re.hi, re.lo, im.hi, im.lo) as stored
struct CD {
    DF x, y;
};

__device__ __forceinline__ CD cd_load(float4 q) { return CD{DF{q.x, q.y}, DF{q.z, q.w}}; }
__device__ __forceinline__ float4 cd_store(CD a) {
    return make_float4(a.x.hi, a.x.lo, a.y.hi, a.y.lo);
}

__device__ __forceinline__ DF df_neg(DF a) { return DF{-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_sub(DF a, DF b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ DF df_mul(DF a, DF b) {
    const float p = __fmul_rn(a.hi, b.hi);  // (never contracted into the sum below)
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    const float hi = p + e;
    return DF{hi, e - (hi - p)};
}
// exact product with a power of two
__device__ __forceinline__ DF df_scale2(DF a, float s) { return DF{a.hi * s, a.lo * s}; }
// integer of up to 48 bits exactly; beyond that to 48 bits
__device__ __forceinline__ DF df_from_int(long long v) {
    const float hi = (float)v;
    return DF{hi, (float)(v - (long long)hi)};
}
__host__ __device__ __forceinline__ DF df_from_double(double v) {
    const float hi = (float)v;
    return DF{hi, (float)(v - (double)hi)};
}

__device__ __forceinline__ CD cd_add(CD a, CD b) { return CD{df_add(a.x, b.x), df_add(a.y, b.y)}; }
__device__ __forceinline__ CD cd_sub(CD a, CD b) { return CD{df_sub(a.x, b.x), df_sub(a.y, b.y)}; }
__device__ __forceinline__ CD cd_mul(CD a, CD w) {
    return CD{df_sub(df_mul(a.x, w.x), df_mul(a.y, w.y)),
              df_add(df_mul(a.x, w.y), df_mul(a.y, w.x))};
}

// double-float splits of cos(pi/8), cos(pi/4), cos(3 pi/8), sqrt(3)/2
__device__ __forceinline__ DF df_const(double v) { return df_from_double(v); }

// v * exp(-2 pi i m / 16), m = 0..7 (compile-time after unrolling)
__device__ __forceinline__ CD rot16(CD v, int m) {
    constexpr double c1 = 0.92387953251128675613, c2 = 0.70710678118654752440,
                     c3 = 0.38268343236508977173;
    switch (m) {
        case 0: return v;
        case 4: return CD{v.y, df_neg(v.x)};
        case 2: {
            const DF c = df_const(c2);
            return CD{df_mul(df_add(v.x, v.y), c), df_mul(df_sub(v.y, v.x), c)};
        }
        case 6: {
            const DF c = df_const(c2);
            return CD{df_mul(df_sub(v.y, v.x), c), df_neg(df_mul(df_add(v.x, v.y), c))};
        }
        case 1: return cd_mul(v, CD{df_const(c1), df_const(-c3)});
        case 3: return cd_mul(v, CD{df_const(c3), df_const(-c1)});
        case 5: return cd_mul(v, CD{df_const(-c3), df_const(-c1)});
        default: return cd_mul(v, CD{df_const(-c1), df_const(-c3)});  // m == 7
    }
}

// v * exp(-2 pi i m / 12), m = 0..11
__device__ __forceinline__ CD rot12(CD v, int m) {
    constexpr double s3 = 0.86602540378443864676;
    const DF s = df_const(s3), ms = df_const(-s3), h = DF{0.5f, 0.0f}, mh = DF{-0.5f, 0.0f};
    switch (m) {
        case 0: return v;
        case 3: return CD{v.y, df_neg(v.x)};
        case 6: return CD{df_neg(v.x), df_neg(v.y)};
        case 9: return CD{df_neg(v.y), v.x};
        case 1: return cd_mul(v, CD{s, mh});
        case 2: return cd_mul(v, CD{h, ms});
        case 4: return cd_mul(v, CD{mh, ms});
        case 5: return cd_mul(v, CD{ms, mh});
        case 7: return cd_mul(v, CD{ms, h});
        case 8: return cd_mul(v, CD{mh, s});
        case 10: return cd_mul(v, CD{h, s});
        default: return cd_mul(v, CD{s, h});  // m == 11
    }
}

__device__ __forceinline__ void dft3(CD& b0, CD& b1, CD& b2) {
    const DF s3 = df_const(0.86602540378443864676);
    const CD s = cd_add(b1, b2), d = cd_sub(b1, b2);
    const CD t = CD{df_sub(b0.x, df_scale2(s.x, 0.5f)), df_sub(b0.y, df_scale2(s.y, 0.5f))};
    const CD m = CD{df_mul(d.y, s3), df_neg(df_mul(d.x, s3))};  // -i (sqrt(3)/2) d
    b0 = cd_add(b0, s);
    b1 = cd_add(t, m);
    b2 = cd_sub(t, m);
}

// forward transforms, natural order in and out (as hpf_fft::reg_fft)
template <int R>
__device__ __forceinline__ void reg_fft2(CD (&a)[R]) {
    constexpr int bits = ilog2(R);
    CD b[R];
#pragma unroll
    for (int i = 0; i < R; ++i) b[bitrev(i, bits)] = a[i];
#pragma unroll
    for (int h = 1; h < R; h <<= 1) {
#pragma unroll
        for (int i0 = 0; i0 < R; i0 += 2 * h) {
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const CD u = b[i0 + j];
                const CD v = rot16(b[i0 + j + h], j * (8 / h));
                b[i0 + j] = cd_add(u, v);
                b[i0 + j + h] = cd_sub(u, v);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = b[i];
}

template <int R>
__device__ __forceinline__ void reg_fft(CD (&a)[R]) {
    if constexpr (R % 3 != 0) {
        reg_fft2<R>(a);
    } else {
        constexpr int P = R / 3;
        CD y[3][P];
#pragma unroll
        for (int n2 = 0; n2 < P; ++n2) {
            CD b0 = a[n2], b1 = a[P + n2], b2 = a[2 * P + n2];
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
__device__ __forceinline__ CD twiddle(const float4* __restrict__ tw, int m) {
    return cd_load(__ldg(tw + Tw<N>::off + m * Tw<N>::stride));
}

}  // namespace hpf_fft_df
