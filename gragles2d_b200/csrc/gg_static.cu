// Allocation-free box convolution (gg_convolve_box_static in gg_step.h).
//
// Some callers cannot allocate device memory: an application that hands this
// library device buffers from its own memory pool and does not let plug-ins
// allocate (to keep its pool the only owner of device memory and avoid
// fragmentation or out-of-memory failures in the middle of a run).  For them
// this file convolves one n x n distance-field box with the Gaussian kernel
// of the convolution stage, using only device memory compiled into the
// library: a file-scope scratch array of fixed size, which every GPU that
// loads the library holds until the process exits.  The caller passes the
// input and output boxes; nothing here calls cudaMalloc, cudaFree or any
// allocating library routine.
//
// The arithmetic is the plain form's (separable direct DFTs in a fixed order,
// host-computed twiddles and Gaussian multipliers, no FMA contraction), so
// the result is bit-identical to the convolution stage of a plain context.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>

#include "../../include/gg_step.h"

namespace {

constexpr int kMaxN = GG_STATIC_CONV_MAX_N;
constexpr int kMaxHalf = kMaxN / 2 + 1;
// Layout of the scratch (doubles): two spectra of n x (n/2+1) complex values.
constexpr size_t kSpecDoubles = 2 * (size_t)kMaxN * kMaxHalf;
constexpr size_t kScratchDoubles = 2 * kSpecDoubles;

// The tables of one call travel as kernel parameters (19 KB at most, of the
// 32 KB a kernel takes): no copy to the device, and nothing of the caller's
// frame to wait for.
template <int kN>  // for n <= kN
struct Twiddles {
    double2 w[kN];  // exp(-2 pi i k / n)
};
template <int kN>
struct Multipliers {
    double g[(kN / 2 + 1) * (kN / 2 + 2) / 2];  // G(i, j) = G(j, i) at j (j + 1) / 2 + i, i <= j
};
static_assert(sizeof(Twiddles<kMaxN>) + sizeof(Multipliers<kMaxN>) < 32000);

// The fixed device scratch.  In host code this name is only a host-side
// stand-in for the symbol, not a device address: the address used by kernels
// comes from cudaGetSymbolAddress on each device (see scratch_on_device).
static __device__ __align__(256) double g_conv_scratch[kScratchDoubles];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
double* g_scratch_ptr[kMaxDevices] = {};

constexpr double kPiS = 3.14159265358979323846;

// A failed runtime call: consume the runtime's last error as well, so that
// this failure is not reported again by a later, unrelated call.
int cuda_error() {
    (void)cudaGetLastError();
    return GG_E_CUDA;
}

// Same expressions as the context's table builder, so the tables match bit
// for bit.
void twiddle(int n, int k, double* re, double* im) {
    double ang = (2.0 * kPiS * (double)k) / (double)n;
    *re = cos(ang);
    *im = -sin(ang);
}

double gaussian_multiplier(int n, int i2, int j2, double dt, int nn) {
    double nsq = nn * nn;
    double n_nsq = n * n;
    return exp(-sqrt(2 / kPiS) * (i2 * i2 + j2 * j2) * 4.0 * dt * nsq / n_nsq * kPiS * kPiS) / n_nsq;
}

// Device address of the scratch on the current device, looked up once per
// device (the first call on a device does this set-up).
int scratch_on_device(double** out) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return cuda_error();
    if (dev < 0 || dev >= kMaxDevices) return GG_E_CUDA;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_conv_scratch);
        if (e != cudaSuccess) return cuda_error();
        if (!p) return GG_E_CUDA;
        g_scratch_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_ptr[dev];
    return GG_OK;
}

// The same sums in the same order as the plain convolution stage, one output
// per thread, spread over the device: a CTA per row, per column (forward,
// multiplier and back), per row.  Each sum is a chain of up to 128 additions
// (8 cycles each), so a transform takes 2 to 3 us whatever its parallelism; one
// CTA for the whole box took 1.3 ms at n = 128.  A whole call: 1374 -> 54 us at
// n = 128 (half of it the host's multipliers), 76 -> 30 us at n = 45.
constexpr int kThreads = kMaxN;

template <int kN>
__device__ __forceinline__ void stage_twiddles(const Twiddles<kN>& t, double2* w, int n) {
    for (int k = threadIdx.x; k < n; k += blockDim.x) w[k] = t.w[k];
}

// Forward transform of a real row x at frequency f.
__device__ __forceinline__ double2 row_sum(const double* x, const double2* w, int n, int f) {
    double re = 0, im = 0;
    int k = 0;
#pragma unroll 4
    for (int c = 0; c < n; ++c) {
        const double2 e = w[k];
        re = re + x[c] * e.x;
        im = im + x[c] * e.y;
        k += f;
        if (k >= n) k -= n;
    }
    return make_double2(re, im);
}

// Forward transform of the column a[0], a[stride], ... at frequency q, times
// the multiplier at (f, q).
template <int kN>
__device__ __forceinline__ double2 column_sum(const double2* a, int stride, const double2* w, int n, int f, int q,
                                              const Multipliers<kN>& G) {
    double re = 0, im = 0;
    int k = 0;
#pragma unroll 4
    for (int r = 0; r < n; ++r) {
        const double2 v = a[r * stride], e = w[k];
        re = re + (v.x * e.x - v.y * e.y);
        im = im + (v.x * e.y + v.y * e.x);
        k += q;
        if (k >= n) k -= n;
    }
    const int j2 = q < n - q ? q : n - q, lo = f < j2 ? f : j2, hi = f < j2 ? j2 : f;
    const double gv = G.g[hi * (hi + 1) / 2 + lo];
    return make_double2(re * gv, im * gv);
}

// Inverse transform of the column y[0], y[stride], ... at row r.
__device__ __forceinline__ double2 column_back(const double2* y, int stride, const double2* w, int n, int r) {
    double re = 0, im = 0;
    int k = 0;
#pragma unroll 4
    for (int p = 0; p < n; ++p) {
        const double2 v = y[p * stride], e = w[k];
        const double ws = -e.y;
        re = re + (v.x * e.x - v.y * ws);
        im = im + (v.x * ws + v.y * e.x);
        k += r;
        if (k >= n) k -= n;
    }
    return make_double2(re, im);
}

// Inverse transform of the half spectrum t of a row at column c.
__device__ __forceinline__ double row_back(const double2* t, const double2* w, int n, int c) {
    const int hmax = (n - 1) / 2;
    double acc = t[0].x;
    int k = 0;
#pragma unroll 4
    for (int f = 1; f <= hmax; ++f) {
        k += c;
        if (k >= n) k -= n;
        const double2 e = w[k];
        acc = acc + 2.0 * (t[f].x * e.x + t[f].y * e.y);
    }
    if ((n & 1) == 0) {
        const double nyq = t[n / 2].x;
        acc = acc + ((c & 1) ? -nyq : nyq);
    }
    return acc;
}

__global__ void __launch_bounds__(kThreads) k_box_rows(const double* __restrict__ in, int n, double2* __restrict__ T,
                                                       const __grid_constant__ Twiddles<kMaxN> tw) {
    __shared__ double2 w[kMaxN];
    __shared__ double x[kMaxN];
    const int half = n / 2 + 1, r = blockIdx.x, f = threadIdx.x;
    stage_twiddles(tw, w, n);
    if (f < n) x[f] = in[(size_t)r * n + f];
    __syncthreads();
    if (f < half) T[(size_t)r * half + f] = row_sum(x, w, n, f);
}

__global__ void __launch_bounds__(kThreads) k_box_columns(const double2* __restrict__ T, int n,
                                                          double2* __restrict__ out,
                                                          const __grid_constant__ Twiddles<kMaxN> tw,
                                                          const __grid_constant__ Multipliers<kMaxN> G) {
    __shared__ double2 w[kMaxN], a[kMaxN], y[kMaxN];
    const int half = n / 2 + 1, f = blockIdx.x, q = threadIdx.x;
    stage_twiddles(tw, w, n);
    if (q < n) a[q] = T[(size_t)q * half + f];
    __syncthreads();
    if (q < n) y[q] = column_sum(a, 1, w, n, f, q, G);
    __syncthreads();
    if (q < n) out[(size_t)q * half + f] = column_back(y, 1, w, n, q);  // thread q is row q now
}

__global__ void __launch_bounds__(kThreads) k_box_back(const double2* __restrict__ T, int n, double* __restrict__ out,
                                                       const __grid_constant__ Twiddles<kMaxN> tw) {
    __shared__ double2 w[kMaxN], t[kMaxHalf];
    const int half = n / 2 + 1, r = blockIdx.x, c = threadIdx.x;
    stage_twiddles(tw, w, n);
    if (c < half) t[c] = T[(size_t)r * half + c];
    __syncthreads();
    if (c < n) out[(size_t)r * n + c] = row_back(t, w, n, c);
}

// Boxes up to kSmallN in one CTA and one launch: three launches and the larger
// tables cost some 8 us more than such a box's sums (a whole call at n = 8: 23 us
// here, 32 there; at 32: 36 and 37; at 40, with 1024 threads, 46 and 37).
constexpr int kSmallN = 32;
constexpr int kSmallHalf = kSmallN / 2 + 1;
constexpr int kSmallThreads = 544;  // an output of a half spectrum each

__global__ void __launch_bounds__(kSmallThreads) k_box_small(const double* __restrict__ in, int n,
                                                             double* __restrict__ out,
                                                             const __grid_constant__ Twiddles<kSmallN> tw,
                                                             const __grid_constant__ Multipliers<kSmallN> G) {
    static_assert(kSmallThreads >= kSmallN * kSmallHalf);
    __shared__ double2 w[kSmallN], a[kSmallN * kSmallHalf], y[kSmallN * kSmallHalf];
    __shared__ double x[kSmallN * kSmallN];
    const int half = n / 2 + 1, t = threadIdx.x, r = t / half, f = t - r * half;
    stage_twiddles(tw, w, n);
    for (int q = t; q < n * n; q += kSmallThreads) x[q] = in[q];
    __syncthreads();
    if (r < n) a[t] = row_sum(x + r * n, w, n, f);
    __syncthreads();
    if (r < n) y[t] = column_sum(a + f, half, w, n, f, r, G);
    __syncthreads();
    if (r < n) a[t] = column_back(y + f, half, w, n, r);
    __syncthreads();
    for (int q = t; q < n * n; q += kSmallThreads) {
        const int row = q / n;
        out[q] = row_back(a + row * half, w, n, q - row * n);
    }
}

// The tables of an n x n box, built on the host stack (no heap allocation);
// every value the kernels read is written here.
template <int kN>
void box_tables(int n, double dt, int nn, Twiddles<kN>& tw, Multipliers<kN>& G) {
    for (int k = 0; k < n; ++k) twiddle(n, k, &tw.w[k].x, &tw.w[k].y);
    for (int j2 = 0; j2 < n / 2 + 1; ++j2)  // the argument is i2^2 + j2^2: symmetric
        for (int i2 = 0; i2 <= j2; ++i2) G.g[j2 * (j2 + 1) / 2 + i2] = gaussian_multiplier(n, i2, j2, dt, nn);
}

}  // namespace

extern "C" int gg_convolve_box_static(const double* d_in, double* d_out, int32_t n, double dt,
                                      int32_t real_domain_size, void* stream) {
    if (n < 1 || n > kMaxN) return GG_E_INVALID;
    if (!d_in || !d_out || real_domain_size < 1 || !(dt > 0)) return GG_E_INVALID;
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    // A call waits for the stream, which a stream capture does not admit: a
    // capturing stream is refused before anything is issued on it, so the
    // capture stays valid.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) return cuda_error();
    if (cap != cudaStreamCaptureStatusNone) return GG_E_INVALID;
    double* scratch = nullptr;
    const int rc = scratch_on_device(&scratch);
    if (rc != GG_OK) return rc;
    if (n <= kSmallN) {
        Twiddles<kSmallN> tw;
        Multipliers<kSmallN> G;
        box_tables(n, dt, real_domain_size, tw, G);
        k_box_small<<<1, kSmallThreads, 0, s>>>(d_in, n, d_out, tw, G);
    } else {
        Twiddles<kMaxN> tw;
        Multipliers<kMaxN> G;
        box_tables(n, dt, real_domain_size, tw, G);
        double2* const s1 = reinterpret_cast<double2*>(scratch);
        double2* const s2 = s1 + kSpecDoubles / 2;
        k_box_rows<<<n, kThreads, 0, s>>>(d_in, n, s1, tw);
        k_box_columns<<<n / 2 + 1, kThreads, 0, s>>>(s1, n, s2, tw, G);
        k_box_back<<<n, kThreads, 0, s>>>(s2, n, d_out, tw);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_error();
    e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? GG_OK : cuda_error();
}
