// Gaussian convolution of the plain form (src/box.cpp:622-695): the 2-D
// transforms evaluated as separable direct DFTs in a fixed summation order,
// without FMA, so that the result is the oracle's bit for bit.
//
//   rows      T[r][f] = sum_c x[r][c] w^(f c)            f < half = n/2 + 1
//   columns   Y[q][f] = G(f, min(q, n-q)) sum_r T[r][f] w^(q r)
//   inverse   T[r][f] = sum_q Y[q][f] conj(w)^(q r)
//   rows      x[r][c] = T[r][0] + 2 sum_f Re(T[r][f] conj(w)^(f c)) (+ Nyquist)
//
// About 12 n^3 FP64 additions and multiplications per box, which the FP64 pipe
// bounds (64 lanes per SM and cycle: 0.4 ms for 5,000 boxes of mean edge 48),
// provided that shared memory keeps up: a value and a twiddle factor are 16
// bytes each, and shared memory delivers 128 per cycle.  So each thread sums a
// tile of outputs (2 rows x 4 frequencies, 4 x 2 complex values in the columns,
// 2 rows x 8 columns), in which every loaded value serves two to eight products:
// 8 to 12 of the 16 cycles that a tile's products take per quarter SM are
// loads.  The spectrum T and its transform Y stay in shared memory.  Twiddle
// factors come from the table of w^k by an index advanced modulo n; lanes run
// along the index that does not enter it, so a warp's lookup is a broadcast
// from two or three addresses.
//
// Measured (B200, stage time; before: one output per thread, both spectra and
// the table in device memory): 5,000 boxes 2.52 -> 0.95 ms, 1,000 boxes of mean
// edge 44 742 -> 220 us.  The FP64 pipe is then busy half of the time; the rest
// is the loop's own latency and the barriers between the transforms (2, 3 or 4
// CTAs per SM make no difference).
#pragma once

#include "gg_device.cuh"
#include "gg_kernels.cuh"

namespace gg {
namespace {  // internal linkage: each form's translation unit has its own copy

// Row stride (complex values) of the spectrum: odd, so that lanes that walk
// rows side by side meet distinct banks.
__host__ __device__ constexpr int dft_stride(int n) { return (n / 2 + 1) | 1; }

// T, Y (also the staged input and output rows) and the twiddle table.
__host__ __device__ constexpr size_t dft_smem(int n) { return 16 * (size_t)n * (2 * dft_stride(n) + 1); }

// k + step modulo n, all in bytes of the twiddle table (k, step < 16 n).
__device__ __forceinline__ unsigned dft_next(unsigned k, unsigned step, unsigned n16) {
    k += step;
    return min(k, k - n16);  // k - n16 wraps above k when k < n16
}

__device__ __forceinline__ double2 dft_twiddle(const double2* w, unsigned k) {
    return *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(w) + k);
}

// One box by the whole CTA: in -> out, both n x n in device memory; tw its
// twiddles, G its multipliers (half x half).
__device__ __forceinline__ void conv_dft_staged(const double* __restrict__ in, double* __restrict__ out, int n,
                                                const double2* __restrict__ tw, const double* __restrict__ G,
                                                unsigned char* smem) {
    const int half = n / 2 + 1, hs = dft_stride(n), xs = n | 1;
    double2* const T = reinterpret_cast<double2*>(smem);
    double2* const Y = T + n * hs;
    double2* const w = Y + n * hs;
    double* const X = reinterpret_cast<double*>(Y);  // n rows of xs <= 2 hs values
    const unsigned n16 = 16u * (unsigned)n;
    for (int k = threadIdx.x; k < n; k += blockDim.x) w[k] = tw[k];
    for (int p = threadIdx.x; p < n * n; p += blockDim.x) {
        const int r = p / n;
        X[r * xs + p - r * n] = in[p];
    }
    __syncthreads();
    const int pairs = (n + 1) >> 1;  // a thread takes rows r and r + pairs
    // rows, real to complex
    for (int t = threadIdx.x; t < ((half + 3) >> 2) * pairs; t += blockDim.x) {
        const int g = t / pairs, r = t - g * pairs, f0 = 4 * g;
        const double* const xa = X + r * xs;
        const double* const xb = X + min(r + pairs, n - 1) * xs;
        unsigned k[4], step[4];
        double re[2][4], im[2][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            step[u] = 16u * (unsigned)min(f0 + u, half - 1);
            k[u] = 0;
            re[0][u] = im[0][u] = re[1][u] = im[1][u] = 0;
        }
#pragma unroll 2
        for (int c = 0; c < n; ++c) {
            const double va = xa[c], vb = xb[c];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double2 e = dft_twiddle(w, k[u]);
                re[0][u] = re[0][u] + va * e.x;
                im[0][u] = im[0][u] + va * e.y;
                re[1][u] = re[1][u] + vb * e.x;
                im[1][u] = im[1][u] + vb * e.y;
                k[u] = dft_next(k[u], step[u], n16);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (f0 + u < half) {
                T[r * hs + f0 + u] = make_double2(re[0][u], im[0][u]);
                if (r + pairs < n) T[(r + pairs) * hs + f0 + u] = make_double2(re[1][u], im[1][u]);
            }
    }
    __syncthreads();
    // columns f and f + fp, forward then back, four outputs of each per thread
    const int fp = (half + 1) >> 1, citems = ((n + 3) >> 2) * fp;
    const int hmax = (n - 1) / 2;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const bool back = pass == 1;
        const double2* const from = back ? Y : T;
        double2* const to = back ? T : Y;
        for (int t = threadIdx.x; t < citems; t += blockDim.x) {
            const int g = t / fp, fa = t - g * fp, q0 = 4 * g;
            const int fb = min(fa + fp, half - 1);
            const double2 *a = from + fa, *b = from + fb;
            unsigned k[4], step[4];
            double re[2][4], im[2][4];
            double2 na = *a, nb = *b, ne[4];  // loaded one step ahead
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                step[u] = 16u * (unsigned)min(q0 + u, n - 1);
                k[u] = 0;
                ne[u] = w[0];
                re[0][u] = im[0][u] = re[1][u] = im[1][u] = 0;
            }
#pragma unroll 1
            for (int r = 0; r < n; ++r) {
                const double2 va = na, vb = nb;
                double2 w4[4];
                a += hs;  // after the last row: read (within the CTA's shared memory) and not used
                b += hs;
                na = *a;
                nb = *b;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    w4[u] = ne[u];
                    k[u] = dft_next(k[u], step[u], n16);
                    ne[u] = dft_twiddle(w, k[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    double2 e = w4[u];
                    if (back) e.y = -e.y;  // conjugate
                    re[0][u] = re[0][u] + (va.x * e.x - va.y * e.y);
                    im[0][u] = im[0][u] + (va.x * e.y + va.y * e.x);
                    re[1][u] = re[1][u] + (vb.x * e.x - vb.y * e.y);
                    im[1][u] = im[1][u] + (vb.x * e.y + vb.y * e.x);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int q = q0 + u;
                if (q >= n) continue;
                // forward: the multiplier; back: the last transform's factor 2 (exact)
                const int j2 = min(q, n - q);
                const double ga = back ? (fa >= 1 && fa <= hmax ? 2.0 : 1.0) : G[fa * half + j2];
                to[q * hs + fa] = make_double2(re[0][u] * ga, im[0][u] * ga);
                if (fa + fp < half) {
                    const double gb = back ? (fb <= hmax ? 2.0 : 1.0) : G[fb * half + j2];
                    to[q * hs + fb] = make_double2(re[1][u] * gb, im[1][u] * gb);
                }
            }
        }
        __syncthreads();
    }
    // rows, complex to real: eight columns of two rows
    for (int t = threadIdx.x; t < ((n + 7) >> 3) * pairs; t += blockDim.x) {
        const int g = t / pairs, r = t - g * pairs, c0 = 8 * g;
        const double2* const a = T + r * hs;
        const double2* const b = T + min(r + pairs, n - 1) * hs;
        unsigned k[8], step[8];
        double acc[2][8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            step[u] = 16u * (unsigned)min(c0 + u, n - 1);
            k[u] = 0;
            acc[0][u] = a[0].x;
            acc[1][u] = b[0].x;
        }
#pragma unroll 1
        for (int f = 1; f <= hmax; ++f) {
            const double2 va = a[f], vb = b[f];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                k[u] = dft_next(k[u], step[u], n16);
                const double2 e = dft_twiddle(w, k[u]);
                acc[0][u] = acc[0][u] + (va.x * e.x + va.y * e.y);
                acc[1][u] = acc[1][u] + (vb.x * e.x + vb.y * e.y);
            }
        }
        if ((n & 1) == 0) {
            const double na = a[n / 2].x, nb = b[n / 2].x;
#pragma unroll
            for (int u = 0; u < 8; ++u) {  // c0 is even: the column's parity is u's
                acc[0][u] = acc[0][u] + ((u & 1) ? -na : na);
                acc[1][u] = acc[1][u] + ((u & 1) ? -nb : nb);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c0 + u < n) {
                X[r * xs + c0 + u] = acc[0][u];
                if (r + pairs < n) X[(r + pairs) * xs + c0 + u] = acc[1][u];
            }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n * n; p += blockDim.x) {
        const int r = p / n;
        out[p] = X[r * xs + p - r * n];
    }
}

// Launches by box edge, side by side on three streams: each box takes little
// more shared memory than it needs and one round of its threads per transform
// (n = 52: 182 tiles each).  Larger boxes go to k_conv_dft.
template <int kBin>
struct DftBin {
    static constexpr int kLow = kBin == 0 ? 0 : kBin == 1 ? 52 : 64;
    static constexpr int kHigh = kBin == 0 ? 52 : kBin == 1 ? 64 : 116;
    static constexpr int kThreads = kBin == 0 ? 192 : kBin == 1 ? 320 : 512;
    static constexpr int kPerSm = kBin == 0 ? 3 : kBin == 1 ? 2 : 1;
    static_assert((dft_smem(kHigh) + 1024) * kPerSm <= 227 * 1024);
};
constexpr int kDftEdge = DftBin<2>::kHigh;

// CTA per grain and, in tangent mode, per field: blockIdx.y - 1 is the
// tangent field (-1: the distance field itself).
template <int kBin>
__global__ void __launch_bounds__(DftBin<kBin>::kThreads, DftBin<kBin>::kPerSm) k_conv_dft_s(NetConst C, NetState* S) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int g = blockIdx.x + 1, tk = (int)blockIdx.y - 1;
    if (g > C.N || C.state[g] != G_EXISTS || halted(S)) return;
    const Box bx = S->box_cur[g];
    const int n = box_w(bx);
    if (n != box_h(bx) || n > C.tmax) return;  // k_conv_dft reports these
    if (n <= DftBin<kBin>::kLow || n > DftBin<kBin>::kHigh) return;
    const double* in = tk < 0 ? phiA_of<double>(S) : reinterpret_cast<double*>(S->dphiA) + tk * S->phi_cap;
    double* out = tk < 0 ? phiB_of<double>(S) : reinterpret_cast<double*>(S->dphiB) + tk * S->phi_cap;
    conv_dft_staged(in + S->off_cur[g], out + S->off_cur[g], n,
                    reinterpret_cast<const double2*>(C.tw) + C.tw_off[n], C.gk + C.gk_off[n], s_raw);
}

// Boxes above kDftEdge, one output per thread, the spectra in the grain's
// scratch in device memory (so the distance field and the `tangents` tangent
// fields one after the other); also reports a box that has no tables.
__device__ void conv_dft_box(const NetConst& C, const double* in, double* out, double* s1, int n);

__global__ void __launch_bounds__(256) k_conv_dft(NetConst C, NetState* S, int tangents) {
    const int g = blockIdx.x + 1;
    if (g > C.N || C.state[g] != G_EXISTS || halted(S)) return;
    const Box bx = S->box_cur[g];
    const int n = box_w(bx);
    if (n <= 0) return;
    if (n != box_h(bx) || n > C.tmax) {
        if (threadIdx.x == 0) set_status(S, n > C.tmax ? S_TABLE_RANGE : S_INDEX);
        return;
    }
    if (n <= kDftEdge) return;
    double* s1 = reinterpret_cast<double*>(S->spec) + S->soff_cur[g];  // 2 x n x half complex
    conv_dft_box(C, phiA_of<double>(S) + S->off_cur[g], phiB_of<double>(S) + S->off_cur[g], s1, n);
    for (int tk = 0; tk < tangents; ++tk) {
        __syncthreads();
        conv_dft_box(C, reinterpret_cast<double*>(S->dphiA) + tk * S->phi_cap + S->off_cur[g],
                     reinterpret_cast<double*>(S->dphiB) + tk * S->phi_cap + S->off_cur[g], s1, n);
    }
}

__device__ void conv_dft_box(const NetConst& C, const double* in, double* out, double* s1, int n) {
    const int half = n / 2 + 1;
    double* s2 = s1 + 2 * (int64_t)n * half;
    const double* w = C.tw + 2 * C.tw_off[n];
    const double* G = C.gk + C.gk_off[n];
    const int tot = n * half;
    for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
        const int r = idx / half, f = idx - r * half;
        double re = 0, im = 0;
        const double* xr = in + r * n;
        int k = 0;
        for (int c = 0; c < n; ++c) {
            const double v = xr[c];
            re = re + v * w[2 * k];
            im = im + v * w[2 * k + 1];
            k += f;
            if (k >= n) k -= n;
        }
        s1[2 * idx] = re;
        s1[2 * idx + 1] = im;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
        const int q = idx / half, f = idx - q * half;
        double re = 0, im = 0;
        int k = 0;
        for (int r = 0; r < n; ++r) {
            const double a = s1[2 * (r * half + f)], b = s1[2 * (r * half + f) + 1];
            const double wc = w[2 * k], ws = w[2 * k + 1];
            re = re + (a * wc - b * ws);
            im = im + (a * ws + b * wc);
            k += q;
            if (k >= n) k -= n;
        }
        const double gv = G[f * half + min(q, n - q)];
        s2[2 * idx] = re * gv;
        s2[2 * idx + 1] = im * gv;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
        const int r = idx / half, f = idx - r * half;
        double re = 0, im = 0;
        int k = 0;
        for (int q = 0; q < n; ++q) {
            const double a = s2[2 * (q * half + f)], b = s2[2 * (q * half + f) + 1];
            const double wc = w[2 * k], ws = -w[2 * k + 1];
            re = re + (a * wc - b * ws);
            im = im + (a * ws + b * wc);
            k += r;
            if (k >= n) k -= n;
        }
        s1[2 * idx] = re;
        s1[2 * idx + 1] = im;
    }
    __syncthreads();
    const int hmax = (n - 1) / 2;
    for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
        const int r = idx / n, c = idx - r * n;
        const double* t = s1 + 2 * (int64_t)r * half;
        double acc = t[0];
        int k = 0;
        for (int f = 1; f <= hmax; ++f) {
            k += c;
            if (k >= n) k -= n;
            acc = acc + 2.0 * (t[2 * f] * w[2 * k] + t[2 * f + 1] * w[2 * k + 1]);
        }
        if ((n & 1) == 0) {
            const double nyq = t[2 * (n / 2)];
            acc = acc + ((c & 1) ? -nyq : nyq);
        }
        out[idx] = acc;
    }
}

}  // namespace
}  // namespace gg
