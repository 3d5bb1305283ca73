// FP64 field energies and pressure sums (hymd/field.py:619-703,
// hymd/pressure.py:9-179 by Parseval) on the meshes of the fused spectral
// passes: the paint's fixed-point accumulators -> half spectrum -> sums, in
// three kernels of double-float arithmetic.
//
// What bounds it is arithmetic: the transforms of T grids at 64-bit accuracy.
// GB300 issues 1/64 as many FP64 operations as FP32 ones, and a double-float
// addition (11 FP32 instructions) or product (7) is several times cheaper
// than an FP64 one.  Two FP32 words carry 48 bits, the accumulators (integers
// of at most 48 bits at up to 16 million beads a cell) enter exactly, and no
// scaling is applied before the sums: their error against 64-bit transforms
// is about 1e-15 (measured on energies and pressures of 300 to 1.3M beads, 8
// to 256 points an axis), that of the deposits' own 2^-24 quantisation 1e-11
// to 1e-8, as before.  Measured on GB300 against cuFFT D2Z and FP64 sums: a
// print step of a 162k-bead membrane at 64^3 (two evaluations) 908 -> 539 us,
// energy and gradients of 1.3M beads at 128^3 2812 -> 1414 us.  Meshes of
// other sizes take the D2Z path (hpf_field.cu).
#include <math.h>
#include <string.h>

#include "hpf_fft_df.cuh"

using namespace hpf_fft_df;
using hpf_fft::Idx;

namespace {

constexpr int kDfThreads = 128;
constexpr int kDfSums = 9;
constexpr int kDfMaxT = 8;

// ------------------------------------------------------------------- z ---
// R rows of a grid per block: accumulators (read, then cleared) -> length-h
// complex transform of the even/odd pairs -> half-spectrum rows.
constexpr int kDfRows = 16;

// Per axis, (k^2, H) of each index in double-float, H = exp(-sigma^2 k^2 / 2):
// n0 entries along x, n1 along y, nzc along z.  The filter is a product over
// the axes, so no mode needs an exponential of its own.
struct AxisTable {
    float4* e;
    int n0, n1, nzc;
};

__device__ __forceinline__ void fill_axis_table(const AxisTable& tab, const BoxState* bs,
                                                const Functional* fun) {
    const double s2h = fun->sigma2_half_d;
    const int n[3] = {tab.n0, tab.n1, tab.nzc};
    for (int i = threadIdx.x; i < tab.n0 + tab.n1 + tab.nzc; i += kDfThreads) {
        const int d = i < n[0] ? 0 : (i < n[0] + n[1] ? 1 : 2);
        const int j = d == 0 ? i : (d == 1 ? i - n[0] : i - n[0] - n[1]);
        const int m = d < 2 && j > n[d] / 2 ? j - n[d] : j;
        const double k = m * (2.0 * 3.14159265358979323846 / bs->L[d]);
        const DF k2 = df_from_double(k * k), H = df_from_double(exp(-s2h * k * k));
        tab.e[i] = make_float4(k2.hi, k2.lo, H.hi, H.lo);
    }
}

template <int H>
__global__ void __launch_bounds__(kDfThreads, 4)
k_df_z(unsigned long long* __restrict__ acc, float4* __restrict__ spec, int rows,
       const float4* __restrict__ tw, AxisTable tab, const BoxState* __restrict__ bs,
       const Functional* __restrict__ fun) {
    constexpr int N1 = split1(H), N2 = H / N1, R = kDfRows, Ls = (H + 1) | 1, Nzc = H + 1;
    extern __shared__ __align__(16) float4 smz[];
    float4* A = smz;
    float4* B = smz + R * Ls;
    const int64_t row0 = (int64_t)blockIdx.x * R + (int64_t)blockIdx.y * rows;
    const int nr = min(R, rows - (int)blockIdx.x * R);
    ulonglong2* a = reinterpret_cast<ulonglong2*>(acc) + row0 * H;
    // step 1: neighbouring lanes take neighbouring elements of a row
    for (int it = threadIdx.x; it < nr * N2; it += kDfThreads) {
        const int c = it / N2, n2 = it - c * N2;
        ulonglong2 raw[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) raw[i] = __ldcg(a + c * H + N2 * i + n2);
        CD v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i)
            v[i] = CD{df_from_int((long long)raw[i].x), df_from_int((long long)raw[i].y)};
        reg_fft<N1>(v);
        if (N2 > 1) {
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = cd_mul(v[k1], twiddle<H>(tw, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) (N2 > 1 ? A : B)[c * Ls + N2 * k1 + n2] = cd_store(v[k1]);
    }
    __syncthreads();
    // cleared for the next paint once the loads have returned
    for (int e = threadIdx.x; e < nr * H; e += kDfThreads) a[e] = make_ulonglong2(0ull, 0ull);
    if (N2 > 1) {
        // step 2: neighbouring lanes take neighbouring rows (odd row stride)
        for (int it = threadIdx.x; it < R * N1; it += kDfThreads) {
            const int k1 = it / R, c = it - k1 * R;
            if (c >= nr) continue;
            CD v[N2];
#pragma unroll
            for (int i = 0; i < N2; ++i) v[i] = cd_load(A[c * Ls + N2 * k1 + i]);
            reg_fft<N2>(v);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) B[c * Ls + k1 + N1 * k2] = cd_store(v[k2]);
        }
        __syncthreads();
    }
    // split: X[k] = E + w^k O, E = (Z[k] + conj Z[h-k]) / 2, O = -i (Z[k] -
    // conj Z[h-k]) / 2
    float4* out = spec + row0 * Nzc;
    for (int e = threadIdx.x; e < nr * Nzc; e += kDfThreads) {
        const int c = e / Nzc, k = e - c * Nzc;
        const CD zk = cd_load(B[c * Ls + (k == H ? 0 : k)]);
        const CD zp = cd_load(B[c * Ls + (k == 0 || k == H ? 0 : H - k)]);
        const CD E = CD{df_scale2(df_add(zk.x, zp.x), 0.5f), df_scale2(df_sub(zk.y, zp.y), 0.5f)};
        const CD O = CD{df_scale2(df_add(zk.y, zp.y), 0.5f), df_scale2(df_sub(zp.x, zk.x), 0.5f)};
        CD X;
        if (k == 0) X = cd_add(E, O);
        else if (k == H) X = cd_sub(E, O);
        else X = cd_add(E, cd_mul(O, twiddle<2 * H>(tw, k)));
        out[e] = cd_store(X);
    }
    // for the last pass, by one block
    if (blockIdx.x == 0 && blockIdx.y == 0) fill_axis_table(tab, bs, fun);
}

// ------------------------------------------------------------------- y ---
// W columns (x, kz) of a grid per block, transformed along y in place.
constexpr int kDfColsY = 16;

template <int N>
__global__ void __launch_bounds__(kDfThreads, 4)
k_df_y(float4* __restrict__ spec, int64_t Mc, int nzc, int cols, const float4* __restrict__ tw) {
    constexpr int N1 = split1(N), N2 = N / N1, W = kDfColsY;
    extern __shared__ __align__(16) float4 smy[];
    const int w = threadIdx.x % W, col = blockIdx.x * W + w;
    const bool on = col < cols;
    const int x = on ? col / nzc : 0, kz = on ? col - x * nzc : 0;
    float4* base = spec + (int64_t)blockIdx.y * Mc + (int64_t)x * N * nzc + kz;
    for (int n2 = threadIdx.x / W; n2 < N2; n2 += kDfThreads / W) {
        if (!on) continue;
        CD v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) v[i] = cd_load(__ldcg(base + (int64_t)(N2 * i + n2) * nzc));
        reg_fft<N1>(v);
        if (N2 > 1) {
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = cd_mul(v[k1], twiddle<N>(tw, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
            if (N2 > 1) smy[(N2 * k1 + n2) * W + w] = cd_store(v[k1]);
            else base[(int64_t)k1 * nzc] = cd_store(v[k1]);
        }
    }
    if (N2 == 1) return;
    __syncthreads();
    for (int k1 = threadIdx.x / W; k1 < N1; k1 += kDfThreads / W) {
        if (!on) continue;
        CD v[N2];
#pragma unroll
        for (int i = 0; i < N2; ++i) v[i] = cd_load(smy[(N2 * k1 + i) * W + w]);
        reg_fft<N2>(v);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) base[(int64_t)(k1 + N1 * k2) * nzc] = cd_store(v[k2]);
    }
}

// -------------------------------------------------------------- x, sums ---
struct DfGeom {
    int n0, n1, nzc, T, G;  // G: grids (T, or T + 1 with the charges)
    int W, ws, ts;          // columns per tile, log2 W, stride of a grid's block
    int64_t Mc;
    double scale[kDfMaxT + 1];  // paint mass (charges: 1) x 2^-24 / M
    double qt[kDfMaxT];
    double four_pi_fac;
};

// One block per tile of W (y, kz) columns of all grids: transform along x,
// then per mode the Parseval terms (as k_energy_f64), reduced in double-float.
template <int N>
__global__ void __launch_bounds__(kDfThreads, 4)
k_df_x(const float4* __restrict__ spec, DfGeom g, const BoxState* __restrict__ bs,
       const Functional* __restrict__ fun, double* out, float2* __restrict__ partials,
       unsigned int* ticket, const float4* __restrict__ tw, AxisTable tab) {
    constexpr int N1 = split1(N), N2 = N / N1;
    extern __shared__ __align__(16) float4 smx[];
    __shared__ float4 ax[N];  // (kx^2, H)
    __shared__ float2 hyz[8], ky2[8], kz2[8];  // per column: H of y and z, k^2
    __shared__ float wk[8];
    __shared__ float2 Q[kDfMaxT * kDfMaxT], tq[kDfMaxT];
    __shared__ float2 red[kDfSums * (kDfThreads / 32)];
    __shared__ bool is_last;
    const int W = g.W, ws = g.ws, TS = g.ts, T = g.T;
    const int64_t plane = (int64_t)g.n1 * g.nzc;
    const int j0 = blockIdx.x * W;
    const int cols = g.G * W;
    const double inv_dV = 1.0 / bs->dV;
    auto put = [](double v) {
        const DF d = df_from_double(v);
        return make_float2(d.hi, d.lo);
    };
    auto get = [](float2 v) { return DF{v.x, v.y}; };
    for (int i = threadIdx.x; i < N; i += kDfThreads) ax[i] = tab.e[i];
    for (int w = threadIdx.x; w < W; w += kDfThreads) {
        const int j = j0 + w, iy = j / g.nzc, iz = j - iy * g.nzc;
        const float4 ay = tab.e[g.n0 + iy], az = tab.e[g.n0 + g.n1 + iz];
        ky2[w] = make_float2(ay.x, ay.y);
        kz2[w] = make_float2(az.x, az.y);
        const DF H = df_mul(DF{ay.z, ay.w}, DF{az.z, az.w});
        hyz[w] = make_float2(H.hi, H.lo);
        wk[w] = (iz == 0 || iz == g.nzc - 1) ? 1.0f : 2.0f;
    }
    // Q with the grids' scales folded in, off-diagonal pairs counted once
    for (int e = threadIdx.x; e < T * T; e += kDfThreads) {
        const int t = e / T, j = e - t * T;
        Q[e] = put((t == j ? 1.0 : 2.0) * fun->Qd[e] * (g.scale[t] * inv_dV) *
                   (g.scale[j] * inv_dV));
    }
    for (int t = threadIdx.x; t < T; t += kDfThreads) tq[t] = put(g.qt[t] * g.scale[t] * inv_dV);
    const bool has_q = g.G > T;
    const double sq = has_q ? g.scale[T] * inv_dV : 0.0;
    const DF fq = df_from_double(g.four_pi_fac * sq);
    const DF fqq = df_from_double(g.four_pi_fac * sq * sq);
    // transform along x
    for (int it = threadIdx.x; it < cols * N2; it += kDfThreads) {
        const int n2 = it / cols, c = it - n2 * cols, t = c >> ws, w = c & (W - 1);
        const float4* src = spec + (int64_t)t * g.Mc + j0 + w;
        CD v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) v[i] = cd_load(__ldg(src + (N2 * i + n2) * plane));
        reg_fft<N1>(v);
        if (N2 > 1) {
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = cd_mul(v[k1], twiddle<N>(tw, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) smx[t * TS + (N2 * k1 + n2) * W + w] = cd_store(v[k1]);
    }
    __syncthreads();
    if (N2 > 1) {
        for (int it = threadIdx.x; it < cols * N1; it += kDfThreads) {
            const int k1 = it / cols, c = it - k1 * cols, t = c >> ws, w = c & (W - 1);
            float4* p = smx + t * TS + N2 * k1 * W + w;
            CD v[N2];
#pragma unroll
            for (int i = 0; i < N2; ++i) v[i] = cd_load(p[i * W]);
            reg_fft<N2>(v);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) p[k2 * W] = cd_store(v[k2]);
        }
        __syncthreads();
    }
    // modes
    DF acc[kDfSums];
#pragma unroll
    for (int k = 0; k < kDfSums; ++k) acc[k] = DF{0.0f, 0.0f};
    for (int e = threadIdx.x; e < N * W; e += kDfThreads) {
        const int p = e >> ws, w = e & (W - 1);
        const int ix = Idx<N>::freq(p);
        const bool origin = ix == 0 && j0 + w == 0;
        const float4 axe = ax[ix];
        const DF kk[3] = {DF{axe.x, axe.y}, get(ky2[w]), get(kz2[w])};
        const DF H = df_mul(DF{axe.z, axe.w}, get(hyz[w]));
        const DF H2 = df_scale2(df_mul(H, H), wk[w]);  // w_k H^2
        const float4* col = smx + p * W + w;
        DF q = DF{0.0f, 0.0f};
        for (int t = 0; t < T; ++t) {
            const CD a = cd_load(col[t * TS]);
            if (origin) out[16 + t] = ((double)a.x.hi + (double)a.x.lo) * (g.scale[t] * inv_dV);
            for (int j = t; j < T; ++j) {
                const CD b = cd_load(col[j * TS]);
                const DF d = df_add(df_mul(a.x, b.x), df_mul(a.y, b.y));
                q = df_add(q, df_mul(get(Q[t * T + j]), d));
            }
        }
        if (!origin) {
            q = df_mul(q, H2);
            acc[0] = df_add(acc[0], q);
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[1 + d] = df_add(acc[1 + d], df_mul(q, kk[d]));
        }
        if (has_q) {
            // psi = 4 pi f H rho / k^2 (k^2 = 1 at k = 0); 1 / k^2 by one
            // Newton step in double-float
            const DF k2 = origin ? DF{1.0f, 0.0f} : df_add(kk[0], df_add(kk[1], kk[2]));
            const float r0 = 1.0f / k2.hi;
            const DF e1 = df_sub(DF{1.0f, 0.0f}, df_mul(k2, DF{r0, 0.0f}));
            const DF ik = df_add(DF{r0, 0.0f}, df_mul(DF{r0, 0.0f}, df_add(e1, df_mul(e1, e1))));
            const CD rho = cd_load(col[T * TS]);
            const DF rr = df_add(df_mul(rho.x, rho.x), df_mul(rho.y, rho.y));
            acc[4] = df_add(acc[4], df_scale2(df_mul(df_mul(fqq, df_mul(H, ik)), rr), wk[w]));
            DF cr = DF{0.0f, 0.0f};
            for (int t = 0; t < T; ++t) {
                const CD a = cd_load(col[t * TS]);
                cr = df_add(cr, df_mul(get(tq[t]),
                                       df_add(df_mul(rho.x, a.x), df_mul(rho.y, a.y))));
            }
            cr = df_mul(df_mul(fq, df_mul(H2, ik)), cr);
            acc[5] = df_add(acc[5], cr);
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[6 + d] = df_add(acc[6 + d], df_mul(cr, kk[d]));
        }
    }
    // block partials, then the last block's sum over them in a fixed order
    warp_df_reduce<kDfSums>(acc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = kDfThreads / 32;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < kDfSums; ++k) red[k * NW + warp] = make_float2(acc[k].hi, acc[k].lo);
    }
    __syncthreads();
    if (threadIdx.x < kDfSums) {
        DF s = get(red[threadIdx.x * NW]);
        for (int i = 1; i < NW; ++i) s = df_add(s, get(red[threadIdx.x * NW + i]));
        partials[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = make_float2(s.hi, s.lo);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int k = warp; k < kDfSums; k += NW) {
        DF s[1] = {DF{0.0f, 0.0f}};
        for (unsigned int b = lane; b < gridDim.x; b += 32)
            s[0] = df_add(s[0], get(__ldcg(partials + (size_t)k * gridDim.x + b)));
        warp_df_reduce<1>(s);
        if (lane == 0) out[k] = (double)s[0].hi + (double)s[0].lo;
    }
    if (threadIdx.x == 0) *ticket = 0u;
}

template <class F>
int with_df_x(int n, F f) {
    switch (n) {
        case 8: return f(k_df_x<8>);
        case 16: return f(k_df_x<16>);
        case 32: return f(k_df_x<32>);
        case 64: return f(k_df_x<64>);
        case 128: return f(k_df_x<128>);
        case 256: return f(k_df_x<256>);
        case 24: return f(k_df_x<24>);
        case 48: return f(k_df_x<48>);
        case 96: return f(k_df_x<96>);
        case 192: return f(k_df_x<192>);
        default: return HPF_ERR_ARG;
    }
}

template <class F>
int with_df_y(int n, F f) {
    switch (n) {
        case 16: return f(k_df_y<16>);
        case 32: return f(k_df_y<32>);
        case 64: return f(k_df_y<64>);
        case 128: return f(k_df_y<128>);
        case 24: return f(k_df_y<24>);
        case 48: return f(k_df_y<48>);
        case 96: return f(k_df_y<96>);
        default: return HPF_ERR_ARG;
    }
}

template <class F>
int with_df_z(int h, F f) {
    switch (h) {
        case 8: return f(k_df_z<8>);
        case 16: return f(k_df_z<16>);
        case 32: return f(k_df_z<32>);
        case 64: return f(k_df_z<64>);
        case 12: return f(k_df_z<12>);
        case 24: return f(k_df_z<24>);
        case 48: return f(k_df_z<48>);
        default: return HPF_ERR_ARG;
    }
}

constexpr size_t kDfMaxSmem = 100 * 1024;

size_t x_smem(int n0, int G, int W, int* ts) {
    // blocks of W < 8 columns are set off by half a bank row each
    const int s = n0 * W + (W < 8 ? W : 0);
    if (ts) *ts = s;
    return sizeof(float4) * (size_t)G * s;
}

}  // namespace

// Twiddles (double-float) and the reduction scratch, on first use, filled in
// the stream of the call that needs them (never under capture).
int energy_df_setup(hpf_ctx* c, cudaStream_t st) {
    if (c->df_tw) return HPF_OK;
    using hpf_fft::kTable2;
    using hpf_fft::kTable3;
    float4 h[kTable2 + kTable3];
    for (int m = 0; m < kTable2 + kTable3; ++m) {
        const double n = m < kTable2 ? kTable2 : kTable3, i = m < kTable2 ? m : m - kTable2;
        const double a = -2.0 * 3.14159265358979323846 * i / n;
        const DF cs = df_from_double(cos(a)), sn = df_from_double(sin(a));
        h[m] = make_float4(cs.hi, cs.lo, sn.hi, sn.lo);
    }
    const size_t tiles = (size_t)c->n1 * (c->n2 / 2 + 1) / 4;
    const size_t bytes = sizeof(float2) * (kDfSums * tiles + 1 + (kDfSums * tiles + 1) % 2) +
                         sizeof(float4) * (size_t)(c->n0 + c->n1 + c->n2 / 2 + 1);
    float4* tw = nullptr;
    HPF_CUDA_TRY(cudaMalloc(&tw, sizeof(h) + bytes));
    // (h is pageable: copied from before the call returns)
    if (cudaMemcpyAsync(tw, h, sizeof(h), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(reinterpret_cast<char*>(tw) + sizeof(h), 0, bytes, st) != cudaSuccess) {
        cudaFree(tw);
        return HPF_ERR_CUDA;
    }
    c->df_tw = tw;
    return HPF_OK;
}

// The accumulators' G grids (T densities, and the charges after them when
// G = T + 1), painted -> out as hpf_energy_fp64; the accumulators are cleared.
// spec: double-float half spectra, float4[G][Mc].
int energy_df(hpf_ctx* c, int G, const double* type_mass, const double* type_charges,
              double four_pi_fac, float4* spec, double* out, cudaStream_t st) {
    const int T = c->T, rows = c->n0 * c->n1, nzc = c->n2 / 2 + 1, h = c->n2 / 2;
    DfGeom g;
    memset(&g, 0, sizeof(g));
    g.n0 = c->n0;
    g.n1 = c->n1;
    g.nzc = nzc;
    g.T = T;
    g.G = G;
    g.Mc = c->Mc;
    g.four_pi_fac = four_pi_fac;
    const double unit = (double)kFixInv / (double)c->M;
    for (int t = 0; t < T; ++t) {
        g.scale[t] = type_mass[t] * unit;
        g.qt[t] = type_charges ? type_charges[t] : 0.0;
    }
    g.scale[T] = unit;
    // the widest tile that fits, still two tiles for every SM
    g.W = 8;
    const int64_t cols = (int64_t)c->n1 * nzc;
    while (g.W > 4 && (x_smem(c->n0, G, g.W, nullptr) > kDfMaxSmem / 2 || cols / g.W < 304)) g.W >>= 1;
    g.ws = g.W == 8 ? 3 : 2;
    const size_t xs = x_smem(c->n0, G, g.W, &g.ts);
    const float4* tw = c->df_tw;
    float2* part = reinterpret_cast<float2*>(c->df_tw + hpf_fft::kTable2 + hpf_fft::kTable3);
    const int tiles = (int)(cols / g.W);
    unsigned int* ticket = reinterpret_cast<unsigned int*>(
        part + (size_t)kDfSums * ((size_t)c->n1 * nzc / 4));
    const size_t words = (size_t)kDfSums * ((size_t)c->n1 * nzc / 4) + 1;
    const AxisTable tab{reinterpret_cast<float4*>(part + words + words % 2), c->n0, c->n1, nzc};
    int r = with_df_z(h, [&](auto k) {
        const size_t zs = sizeof(float4) * 2 * kDfRows * (size_t)((h + 1) | 1);
        k<<<dim3((rows + kDfRows - 1) / kDfRows, G), kDfThreads, zs, st>>>(c->d_acc, spec, rows, tw, tab,
                                                                            c->d_box, c->d_fun);
        return cudaGetLastError() == cudaSuccess ? HPF_OK : HPF_ERR_CUDA;
    });
    if (r != HPF_OK) return r;
    r = with_df_y(c->n1, [&](auto k) {
        const int n = c->n0 * nzc;
        const size_t ys = sizeof(float4) * kDfColsY * (size_t)c->n1;
        k<<<dim3((n + kDfColsY - 1) / kDfColsY, G), kDfThreads, ys, st>>>(spec, c->Mc, nzc, n, tw);
        return cudaGetLastError() == cudaSuccess ? HPF_OK : HPF_ERR_CUDA;
    });
    if (r != HPF_OK) return r;
    return with_df_x(c->n0, [&](auto k) {
        if (xs > 48 * 1024 &&
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kDfMaxSmem) != cudaSuccess)
            return (int)HPF_ERR_CUDA;
        k<<<tiles, kDfThreads, xs, st>>>(spec, g, c->d_box, c->d_fun, out, part, ticket, tw, tab);
        return cudaGetLastError() == cudaSuccess ? (int)HPF_OK : (int)HPF_ERR_CUDA;
    });
}

// Whether the mesh, type count and functional sums above apply.
bool energy_df_ok(const hpf_ctx* c) {
    return c->spec_ok && c->spec_fused && c->T <= kDfMaxT &&
           x_smem(c->n0, c->T + 1, 4, nullptr) <= kDfMaxSmem;
}
