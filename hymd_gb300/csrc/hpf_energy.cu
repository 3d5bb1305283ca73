// FP64 field energies and pressure sums (hymd/field.py:619-703,
// hymd/pressure.py:9-179 by Parseval) on the meshes of the fused spectral
// passes: the paint's fixed-point accumulators -> half spectrum -> sums, in
// three kernels of FP64 arithmetic.
//
// What bounds it is the FP64 pipe, which issues 1/64 as many operations as
// the FP32 one: at 128^3 with five types the transforms are some 0.35 G of
// them and the sums 0.07 G, 0.67 ms at the 0.62 T a second that 152 SMs
// issue.  So the kernels do no more of them than the sums need: T grids and
// not always T + 1, no scaling pass (the integers enter as they are, exact up
// to 2^53; masses, 2^-24, 1 / dV and the split's factor 1/2 are folded into
// Q), one product of tabulated per-axis factors in place of an exponential a
// mode, both halves of a real row's split from one twiddle product.  Measured
// on GB300 against cuFFT D2Z and k_energy_f64, whole call without charges,
// five types: 162k beads at 64^3 137 us (231), 1.3M beads at 128^3 915 us
// (1568; z 250, y 211, x with the sums 354).
//
// Accuracy: as the D2Z path's.  On deposits that are exact (beads on mesh
// points) both are within 2 x 2^-53 of the sum of the terms' absolute values
// of a transform in extended precision.  Two FP32 words a number would be
// faster (369 against 502 us for a print step of 162k beads, 1353 against 1920
// for energy and gradients of 1.3M), but hold 48 bits: 2 to 30 x 2^-53 on the
// same deposits, a cancelling quadratic form to 2e-12 instead of 3e-15, and
// nothing at all in units whose sums lie outside FP32's exponents.  Meshes of
// other sizes take the D2Z path (hpf_field.cu).
#include <math.h>
#include <string.h>

#include "hpf_fft_f64.cuh"
#include "hpf_internal.cuh"

using namespace hpf_fft64;
using hpf_fft::Idx;

namespace {

constexpr int kE64Threads = 128;
constexpr int kE64Sums = 9;
constexpr int kE64MaxT = 8;

// ------------------------------------------------------------------- z ---
// R rows of a grid per block: accumulators (read, then cleared) -> length-h
// complex transform of the even/odd pairs -> half-spectrum rows.
constexpr int kE64Rows = 16;

// Per axis, (k^2, H) of each index, H = exp(-sigma^2 k^2 / 2): n0 entries along
// x, n1 along y, nzc along z.  The filter is a product over the axes, so no
// mode needs an exponential of its own.
struct AxisTable {
    double2* e;
    int n0, n1, nzc;
};

__device__ __forceinline__ void fill_axis_table(const AxisTable& tab, const BoxState* bs,
                                                const Functional* fun) {
    const double s2h = fun->sigma2_half_d;
    const int n[3] = {tab.n0, tab.n1, tab.nzc};
    for (int i = threadIdx.x; i < tab.n0 + tab.n1 + tab.nzc; i += kE64Threads) {
        const int d = i < n[0] ? 0 : (i < n[0] + n[1] ? 1 : 2);
        const int j = d == 0 ? i : (d == 1 ? i - n[0] : i - n[0] - n[1]);
        const int m = d < 2 && j > n[d] / 2 ? j - n[d] : j;
        const double k = m * (2.0 * 3.14159265358979323846 / bs->L[d]);
        tab.e[i] = make_double2(k * k, exp(-s2h * k * k));
    }
}

template <int H>
__global__ void __launch_bounds__(kE64Threads, 4)
k_e64_z(unsigned long long* __restrict__ acc, double2* __restrict__ spec, int rows,
        const double2* __restrict__ tw, AxisTable tab, const BoxState* __restrict__ bs,
        const Functional* __restrict__ fun) {
    constexpr int N1 = split1(H), N2 = H / N1, R = kE64Rows, Ls = (H + 1) | 1, Nzc = H + 1;
    extern __shared__ __align__(16) double2 smz[];
    double2* A = smz;
    double2* B = smz + R * Ls;
    const int64_t row0 = (int64_t)blockIdx.x * R + (int64_t)blockIdx.y * rows;
    const int nr = min(R, rows - (int)blockIdx.x * R);
    ulonglong2* a = reinterpret_cast<ulonglong2*>(acc) + row0 * H;
    // step 1: neighbouring lanes take neighbouring elements of a row
    for (int it = threadIdx.x; it < nr * N2; it += kE64Threads) {
        const int c = it / N2, n2 = it - c * N2;
        ulonglong2 raw[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) raw[i] = __ldcg(a + c * H + N2 * i + n2);
        double2 v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i)
            v[i] = make_double2((double)(long long)raw[i].x, (double)(long long)raw[i].y);
        reg_fft<N1>(v);
        if (N2 > 1) {
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = c_mul(v[k1], twiddle<H>(tw, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) (N2 > 1 ? A : B)[c * Ls + N2 * k1 + n2] = v[k1];
    }
    __syncthreads();
    // cleared for the next paint once the loads have returned
    for (int e = threadIdx.x; e < nr * H; e += kE64Threads) a[e] = make_ulonglong2(0ull, 0ull);
    if (N2 > 1) {
        // step 2: neighbouring lanes take neighbouring rows (odd row stride)
        for (int it = threadIdx.x; it < R * N1; it += kE64Threads) {
            const int k1 = it / R, c = it - k1 * R;
            if (c >= nr) continue;
            double2 v[N2];
#pragma unroll
            for (int i = 0; i < N2; ++i) v[i] = A[c * Ls + N2 * k1 + i];
            reg_fft<N2>(v);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) B[c * Ls + k1 + N1 * k2] = v[k2];
        }
        __syncthreads();
    }
    // split, with X doubled (the sums' unit takes the factor): 2 E = Z[k] +
    // conj Z[h-k], 2 O = -i (Z[k] - conj Z[h-k]), X[k] = E + w^k O and
    // X[h-k] = conj(E - w^k O)
    constexpr int Half = H / 2 + 1;
    double2* out = spec + row0 * Nzc;
    for (int e = threadIdx.x; e < nr * Half; e += kE64Threads) {
        const int c = e / Half, k = e - c * Half;
        const double2 zk = B[c * Ls + k], zp = B[c * Ls + (k == 0 ? 0 : H - k)];
        const double2 E = make_double2(zk.x + zp.x, zk.y - zp.y);
        const double2 O = make_double2(zk.y + zp.y, zp.x - zk.x);
        const double2 P = k == 0 ? O : c_mul(O, twiddle<2 * H>(tw, k));
        out[c * Nzc + k] = c_add(E, P);
        if (2 * k != H) out[c * Nzc + H - k] = make_double2(E.x - P.x, P.y - E.y);
    }
    // for the last pass, by one block
    if (blockIdx.x == 0 && blockIdx.y == 0) fill_axis_table(tab, bs, fun);
}

// ------------------------------------------------------------------- y ---
// W columns (x, kz) of a grid per block, transformed along y in place.
constexpr int kE64Cols = 16;

template <int N>
__global__ void __launch_bounds__(kE64Threads, 4)
k_e64_y(double2* __restrict__ spec, int64_t Mc, int nzc, int cols,
        const double2* __restrict__ tw) {
    constexpr int N1 = split1(N), N2 = N / N1, W = kE64Cols;
    extern __shared__ __align__(16) double2 smy[];
    const int w = threadIdx.x % W, col = blockIdx.x * W + w;
    const bool on = col < cols;
    const int x = on ? col / nzc : 0, kz = on ? col - x * nzc : 0;
    double2* base = spec + (int64_t)blockIdx.y * Mc + (int64_t)x * N * nzc + kz;
    for (int n2 = threadIdx.x / W; n2 < N2; n2 += kE64Threads / W) {
        if (!on) continue;
        double2 v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) v[i] = __ldcg(base + (int64_t)(N2 * i + n2) * nzc);
        reg_fft<N1>(v);
        if (N2 > 1) {
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = c_mul(v[k1], twiddle<N>(tw, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
            if (N2 > 1) smy[(N2 * k1 + n2) * W + w] = v[k1];
            else base[(int64_t)k1 * nzc] = v[k1];
        }
    }
    if (N2 == 1) return;
    __syncthreads();
    for (int k1 = threadIdx.x / W; k1 < N1; k1 += kE64Threads / W) {
        if (!on) continue;
        double2 v[N2];
#pragma unroll
        for (int i = 0; i < N2; ++i) v[i] = smy[(N2 * k1 + i) * W + w];
        reg_fft<N2>(v);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) base[(int64_t)(k1 + N1 * k2) * nzc] = v[k2];
    }
}

// -------------------------------------------------------------- x, sums ---
struct E64Geom {
    int n0, n1, nzc, T, G;  // G: grids (T, or T + 1 with the charges)
    int W, ws, ts;          // columns per tile, log2 W, stride of a grid's block
    int64_t Mc;
    double scale[kE64MaxT + 1];  // paint mass (charges: 1) x 2^-24 / 2 M
    double qt[kE64MaxT];
    double four_pi_fac;
};

// One block per tile of W (y, kz) columns of all grids: transform along x,
// then per mode the Parseval terms (as k_energy_f64), reduced in FP64.
template <int N>
__global__ void __launch_bounds__(kE64Threads, 4)
k_e64_x(const double2* __restrict__ spec, E64Geom g, const BoxState* __restrict__ bs,
        const Functional* __restrict__ fun, double* out, double* partials, unsigned int* ticket,
        const double2* __restrict__ tw, AxisTable tab) {
    constexpr int N1 = split1(N), N2 = N / N1;
    extern __shared__ __align__(16) double2 smx[];
    __shared__ double2 ax[N];  // (kx^2, H)
    __shared__ double hyz[8], ky2[8], kz2[8], wk[8];  // per column: H of y and z, k^2, weight
    __shared__ double Q[kE64MaxT * kE64MaxT], tq[kE64MaxT];
    const int W = g.W, ws = g.ws, TS = g.ts, T = g.T;
    const int64_t plane = (int64_t)g.n1 * g.nzc;
    const int j0 = blockIdx.x * W;
    const int cols = g.G * W;
    const double inv_dV = 1.0 / bs->dV;
    for (int i = threadIdx.x; i < N; i += kE64Threads) ax[i] = tab.e[i];
    for (int w = threadIdx.x; w < W; w += kE64Threads) {
        const int j = j0 + w, iy = j / g.nzc, iz = j - iy * g.nzc;
        const double2 ay = tab.e[g.n0 + iy], az = tab.e[g.n0 + g.n1 + iz];
        ky2[w] = ay.x;
        kz2[w] = az.x;
        hyz[w] = ay.y * az.y;
        wk[w] = (iz == 0 || iz == g.nzc - 1) ? 1.0 : 2.0;
    }
    // Q with the grids' scales folded in, off-diagonal pairs counted once
    for (int e = threadIdx.x; e < T * T; e += kE64Threads) {
        const int t = e / T, j = e - t * T;
        Q[e] = (t == j ? 1.0 : 2.0) * fun->Qd[e] * (g.scale[t] * inv_dV) * (g.scale[j] * inv_dV);
    }
    for (int t = threadIdx.x; t < T; t += kE64Threads) tq[t] = g.qt[t] * g.scale[t] * inv_dV;
    const bool has_q = g.G > T;
    const double sq = has_q ? g.scale[T] * inv_dV : 0.0;
    const double fq = g.four_pi_fac * sq, fqq = fq * sq;
    // transform along x
    for (int it = threadIdx.x; it < cols * N2; it += kE64Threads) {
        const int n2 = it / cols, c = it - n2 * cols, t = c >> ws, w = c & (W - 1);
        const double2* src = spec + (int64_t)t * g.Mc + j0 + w;
        double2 v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) v[i] = __ldg(src + (N2 * i + n2) * plane);
        reg_fft<N1>(v);
        if (N2 > 1) {
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) v[k1] = c_mul(v[k1], twiddle<N>(tw, n2 * k1));
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) smx[t * TS + (N2 * k1 + n2) * W + w] = v[k1];
    }
    __syncthreads();
    if (N2 > 1) {
        for (int it = threadIdx.x; it < cols * N1; it += kE64Threads) {
            const int k1 = it / cols, c = it - k1 * cols, t = c >> ws, w = c & (W - 1);
            double2* p = smx + t * TS + N2 * k1 * W + w;
            double2 v[N2];
#pragma unroll
            for (int i = 0; i < N2; ++i) v[i] = p[i * W];
            reg_fft<N2>(v);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) p[k2 * W] = v[k2];
        }
        __syncthreads();
    }
    // modes
    double acc[kE64Sums];
#pragma unroll
    for (int k = 0; k < kE64Sums; ++k) acc[k] = 0.0;
    for (int e = threadIdx.x; e < N * W; e += kE64Threads) {
        const int p = e >> ws, w = e & (W - 1);
        const int ix = Idx<N>::freq(p);
        const bool origin = ix == 0 && j0 + w == 0;
        const double2 axe = ax[ix];
        const double kk[3] = {axe.x, ky2[w], kz2[w]};
        const double H = axe.y * hyz[w];
        const double H2 = H * H * wk[w];  // w_k H^2
        const double2* col = smx + p * W + w;
        double q = 0.0;
        for (int t = 0; t < T; ++t) {
            const double2 a = col[t * TS];
            if (origin) out[16 + t] = a.x * (g.scale[t] * inv_dV);
            for (int j = t; j < T; ++j) {
                const double2 b = col[j * TS];
                q = fma(Q[t * T + j], fma(a.x, b.x, a.y * b.y), q);
            }
        }
        if (!origin) {
            q *= H2;
            acc[0] += q;
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[1 + d] = fma(q, kk[d], acc[1 + d]);
        }
        if (has_q) {
            // psi = 4 pi f H rho / k^2 (k^2 = 1 at k = 0)
            const double ik = origin ? 1.0 : 1.0 / (kk[0] + kk[1] + kk[2]);
            const double2 rho = col[T * TS];
            acc[4] = fma(fqq * H * ik * wk[w], fma(rho.x, rho.x, rho.y * rho.y), acc[4]);
            double cr = 0.0;
            for (int t = 0; t < T; ++t) {
                const double2 a = col[t * TS];
                cr = fma(tq[t], fma(rho.x, a.x, rho.y * a.y), cr);
            }
            cr *= fq * H2 * ik;
            acc[5] += cr;
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[6 + d] = fma(cr, kk[d], acc[6 + d]);
        }
    }
    if (has_q) {
        grid_reduce_store<kE64Sums>(acc, partials, ticket, out, false);
        return;
    }
    if (blockIdx.x == 0 && threadIdx.x < kE64Sums - 4) out[4 + threadIdx.x] = 0.0;
    double first[4] = {acc[0], acc[1], acc[2], acc[3]};
    grid_reduce_store<4>(first, partials, ticket, out, false);
}

template <class F>
int with_e64_x(int n, F f) {
    switch (n) {
        case 8: return f(k_e64_x<8>);
        case 16: return f(k_e64_x<16>);
        case 32: return f(k_e64_x<32>);
        case 64: return f(k_e64_x<64>);
        case 128: return f(k_e64_x<128>);
        case 256: return f(k_e64_x<256>);
        case 24: return f(k_e64_x<24>);
        case 48: return f(k_e64_x<48>);
        case 96: return f(k_e64_x<96>);
        case 192: return f(k_e64_x<192>);
        default: return HPF_ERR_ARG;
    }
}

template <class F>
int with_e64_y(int n, F f) {
    switch (n) {
        case 16: return f(k_e64_y<16>);
        case 32: return f(k_e64_y<32>);
        case 64: return f(k_e64_y<64>);
        case 128: return f(k_e64_y<128>);
        case 24: return f(k_e64_y<24>);
        case 48: return f(k_e64_y<48>);
        case 96: return f(k_e64_y<96>);
        default: return HPF_ERR_ARG;
    }
}

template <class F>
int with_e64_z(int h, F f) {
    switch (h) {
        case 8: return f(k_e64_z<8>);
        case 16: return f(k_e64_z<16>);
        case 32: return f(k_e64_z<32>);
        case 64: return f(k_e64_z<64>);
        case 12: return f(k_e64_z<12>);
        case 24: return f(k_e64_z<24>);
        case 48: return f(k_e64_z<48>);
        default: return HPF_ERR_ARG;
    }
}

constexpr size_t kE64MaxSmem = 100 * 1024;

size_t x_smem(int n0, int G, int W, int* ts) {
    // blocks of W < 8 columns are set off by half a bank row each
    const int s = n0 * W + (W < 8 ? W : 0);
    if (ts) *ts = s;
    return sizeof(double2) * (size_t)G * s;
}

}  // namespace

// Doubles of scratch behind the twiddles: the partial sums of the narrowest
// tiles, the ticket, then (16-byte aligned) the axis table.
static size_t e64_words(const hpf_ctx* c) {
    const size_t w = (size_t)kE64Sums * ((size_t)c->n1 * (c->n2 / 2 + 1) / 4) + 1;
    return w + w % 2;
}

// exp(-2 pi i m / n), n a multiple of 8: from an angle of at most pi / 4, so
// that its rounding does not show in the table.
static double2 unit_root(int m, int n) {
    const int oct = 8 * m / n, r = m - oct * (n / 8);
    const double a = 2.0 * 3.14159265358979323846 * (oct & 1 ? n / 8 - r : r) / n;
    const double c = cos(a), s = sin(a);
    const bool swap = oct == 1 || oct == 2 || oct == 5 || oct == 6;
    const double x = swap ? s : c, y = swap ? c : s;
    return make_double2(oct >= 2 && oct <= 5 ? -x : x, oct >= 4 ? y : -y);
}

// Twiddles and the reduction scratch, on first use, filled in the stream of
// the call that needs them (never under capture).
int energy_fused_setup(hpf_ctx* c, cudaStream_t st) {
    if (c->e64_tw) return HPF_OK;
    using hpf_fft::kTable2;
    using hpf_fft::kTable3;
    double2 h[kTable2 + kTable3];
    for (int m = 0; m < kTable2; ++m) h[m] = unit_root(m, kTable2);
    for (int m = 0; m < kTable3; ++m) h[kTable2 + m] = unit_root(m, kTable3);
    const size_t bytes = sizeof(double) * e64_words(c) +
                         sizeof(double2) * (size_t)(c->n0 + c->n1 + c->n2 / 2 + 1);
    double2* tw = nullptr;
    HPF_CUDA_TRY(cudaMalloc(&tw, sizeof(h) + bytes));
    // (h is pageable: copied from before the call returns)
    if (cudaMemcpyAsync(tw, h, sizeof(h), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(reinterpret_cast<char*>(tw) + sizeof(h), 0, bytes, st) != cudaSuccess) {
        cudaFree(tw);
        return HPF_ERR_CUDA;
    }
    c->e64_tw = tw;
    return HPF_OK;
}

// The accumulators' G grids (T densities, and the charges after them when
// G = T + 1), painted -> out as hpf_energy_fp64; the accumulators are cleared.
// spec: half spectra, double2[G][Mc].
int energy_fused(hpf_ctx* c, int G, const double* type_mass, const double* type_charges,
                 double four_pi_fac, double2* spec, double* out, cudaStream_t st) {
    const int T = c->T, rows = c->n0 * c->n1, nzc = c->n2 / 2 + 1, h = c->n2 / 2;
    E64Geom g;
    memset(&g, 0, sizeof(g));
    g.n0 = c->n0;
    g.n1 = c->n1;
    g.nzc = nzc;
    g.T = T;
    g.G = G;
    g.Mc = c->Mc;
    g.four_pi_fac = four_pi_fac;
    const double unit = 0.5 * (double)kFixInv / (double)c->M;
    for (int t = 0; t < T; ++t) {
        g.scale[t] = type_mass[t] * unit;
        g.qt[t] = type_charges ? type_charges[t] : 0.0;
    }
    g.scale[T] = unit;
    // the widest tile that fits, still two tiles for every SM
    g.W = 8;
    const int64_t cols = (int64_t)c->n1 * nzc;
    while (g.W > 4 && (x_smem(c->n0, G, g.W, nullptr) > kE64MaxSmem / 2 || cols / g.W < 304)) g.W >>= 1;
    g.ws = g.W == 8 ? 3 : 2;
    const size_t xs = x_smem(c->n0, G, g.W, &g.ts);
    const double2* tw = c->e64_tw;
    double* part = reinterpret_cast<double*>(c->e64_tw + hpf_fft::kTable2 + hpf_fft::kTable3);
    const int tiles = (int)(cols / g.W);
    unsigned int* ticket = reinterpret_cast<unsigned int*>(
        part + (size_t)kE64Sums * ((size_t)c->n1 * nzc / 4));
    const AxisTable tab{reinterpret_cast<double2*>(part + e64_words(c)), c->n0, c->n1, nzc};
    int r = with_e64_z(h, [&](auto k) {
        const size_t zs = sizeof(double2) * 2 * kE64Rows * (size_t)((h + 1) | 1);
        k<<<dim3((rows + kE64Rows - 1) / kE64Rows, G), kE64Threads, zs, st>>>(c->d_acc, spec, rows, tw, tab,
                                                                            c->d_box, c->d_fun);
        return cudaGetLastError() == cudaSuccess ? HPF_OK : HPF_ERR_CUDA;
    });
    if (r != HPF_OK) return r;
    r = with_e64_y(c->n1, [&](auto k) {
        const int n = c->n0 * nzc;
        const size_t ys = sizeof(double2) * kE64Cols * (size_t)c->n1;
        k<<<dim3((n + kE64Cols - 1) / kE64Cols, G), kE64Threads, ys, st>>>(spec, c->Mc, nzc, n, tw);
        return cudaGetLastError() == cudaSuccess ? HPF_OK : HPF_ERR_CUDA;
    });
    if (r != HPF_OK) return r;
    return with_e64_x(c->n0, [&](auto k) {
        if (xs > 48 * 1024 &&
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kE64MaxSmem) != cudaSuccess)
            return (int)HPF_ERR_CUDA;
        k<<<tiles, kE64Threads, xs, st>>>(spec, g, c->d_box, c->d_fun, out, part, ticket, tw, tab);
        return cudaGetLastError() == cudaSuccess ? (int)HPF_OK : (int)HPF_ERR_CUDA;
    });
}

// Whether the mesh, type count and functional sums above apply.
bool energy_fused_ok(const hpf_ctx* c) {
    return c->spec_ok && c->spec_fused && c->T <= kE64MaxT &&
           x_smem(c->n0, c->T + 1, 4, nullptr) <= kE64MaxSmem;
}
