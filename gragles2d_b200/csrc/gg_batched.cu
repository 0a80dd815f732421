// Batched form: FP32 distance fields and convolution (FP64 contour areas,
// energies and lengths), every stage over all grains, captured per step as
// one CUDA graph by the host.
#include "gg_corrector.cuh"
#include "gg_kernels.cuh"
#include "gg_launch.cuh"
#include "gg_redist.cuh"
#include "gg_warp.cuh"

namespace gg {

constexpr int kConvSmemEdgeMax = 128;  // largest tunable edge with the intermediate in shared memory
constexpr int kSepStrip = 4;       // outputs per thread along the convolution axis

// Gaussian convolution as a separable circular convolution in real space:
// out = K X K^T with K[r][r'] = k_n[(r - r') mod n], where k_n is the real
// kernel whose DFT is the reference's Gaussian multiplier
// (src/box.cpp:674-687, G(i2, j2) = g(i2) g(j2) / n^2).  One CTA per grain.
// The kernel is laid out once as kx[j] = k_n[(j - (n-1)) mod n], j < 2n-1
// (zero-padded), so output c of a row is sum_c' X[c'] kx[c - c' + n - 1]:
// each thread accumulates strips of 4 consecutive outputs of two rows (or
// columns) while a 4-entry register window slides down kx (one shared-memory
// load of the kernel per 8 FMAs).  Taps farther than R (circularly) from the
// strip are left out: the host sets R so that every dropped k_n entry is
// below 2^-26 k_n[0].

// The (at most two) index ranges of c' within circular distance R of the
// strip [c0, c0 + 4), as [s0, e0) and [s1, e1).
__device__ __forceinline__ void band_ranges(int c0, int n, int R, int* s0, int* e0, int* s1, int* e1) {
    *s1 = 0;
    *e1 = 0;
    if (2 * R + kSepStrip >= n) {
        *s0 = 0;
        *e0 = n;
        return;
    }
    const int lo = c0 - R, hi = c0 + kSepStrip + R;
    if (lo < 0) {
        *s0 = lo + n;
        *e0 = n;
        *e1 = hi;
    } else if (hi > n) {
        *s0 = lo;
        *e0 = n;
        *e1 = hi - n;
    } else {
        *s0 = lo;
        *e0 = hi;
    }
}

// The taps of band_ranges as one walk of the same length for every strip of
// a box, so that the lanes of a warp run one loop together (the row pass,
// whose strips differ within a warp): the walk starts at c' = *first and
// wraps from n - 1 to 0, *taps steps, with the kernel window starting at kx
// index *base.  In a banded box every strip starts at R + n - 1, one period
// of k_n above the first range's index when that range wraps; kx holds k_n
// periodically below index 2n - 1, so every stored output meets the same
// kernel values in the same order as over the two ranges (the window's
// extra entries past the row end feed only the unstored outputs of a last,
// partial strip).
__device__ __forceinline__ void band_walk(int c0, int n, int R, int* first, int* taps, int* base) {
    if (2 * R + kSepStrip >= n) {
        *first = 0;
        *taps = n;
        *base = c0 + n - 1;
        return;
    }
    const int lo = c0 - R;
    *first = lo < 0 ? lo + n : lo;
    *taps = 2 * R + kSepStrip;
    *base = R + n - 1;
}

// rows: two rows per thread share each kernel window load
__device__ __forceinline__ void sep_pass_rows(const float* __restrict__ X, float* __restrict__ T,
                                              const float* __restrict__ kx, int n, int R) {
    const int nb = (n + kSepStrip - 1) / kSepStrip;
    const int npair = (n + 1) >> 1;
    for (int t = threadIdx.x; t < npair * nb; t += blockDim.x) {
        const int rp = t / nb, c0 = (t - rp * nb) * kSepStrip;
        const int r = 2 * rp;
        const bool two = r + 1 < n;
        const float* xa = X + r * n;
        const float* xb = two ? xa + n : xa;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
        int cp, taps, base;
        band_walk(c0, n, R, &cp, &taps, &base);
        float w0 = kx[base], w1 = kx[base + 1], w2 = kx[base + 2], w3 = kx[base + 3];
#pragma unroll 4
        for (int k = 0; k < taps; ++k) {
            const float x = xa[cp], y = xb[cp];
            a0 = fmaf(x, w0, a0);
            a1 = fmaf(x, w1, a1);
            a2 = fmaf(x, w2, a2);
            a3 = fmaf(x, w3, a3);
            b0 = fmaf(y, w0, b0);
            b1 = fmaf(y, w1, b1);
            b2 = fmaf(y, w2, b2);
            b3 = fmaf(y, w3, b3);
            cp = cp + 1 == n ? 0 : cp + 1;
            --base;
            w3 = w2;
            w2 = w1;
            w1 = w0;
            w0 = kx[base];
        }
        float* ta = T + r * n + c0;
        ta[0] = a0;
        if (c0 + 1 < n) ta[1] = a1;
        if (c0 + 2 < n) ta[2] = a2;
        if (c0 + 3 < n) ta[3] = a3;
        if (two) {
            float* tb = ta + n;
            tb[0] = b0;
            if (c0 + 1 < n) tb[1] = b1;
            if (c0 + 2 < n) tb[2] = b2;
            if (c0 + 3 < n) tb[3] = b3;
        }
    }
}

// columns: columns c and c + ceil(n/2) per thread share each kernel window load
__device__ __forceinline__ void sep_pass_cols(const float* __restrict__ T, float* __restrict__ out,
                                              const float* __restrict__ kx, int n, int R) {
    const int nb = (n + kSepStrip - 1) / kSepStrip;
    const int half = (n + 1) >> 1;
    for (int t = threadIdx.x; t < half * nb; t += blockDim.x) {
        const int rb = t / half, c = t - rb * half, r0 = rb * kSepStrip;
        const bool two = c + half < n;
        const int c2 = two ? c + half : c;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
        int rs[2], re[2];
        band_ranges(r0, n, R, &rs[0], &re[0], &rs[1], &re[1]);
        for (int q = 0; q < 2; ++q) {
            int base = r0 + n - 1 - rs[q];
            float w0 = kx[base], w1 = kx[base + 1], w2 = kx[base + 2], w3 = kx[base + 3];
#pragma unroll 4
            for (int rp = rs[q]; rp < re[q]; ++rp) {
                const float x = T[rp * n + c], y = T[rp * n + c2];
                a0 = fmaf(w0, x, a0);
                a1 = fmaf(w1, x, a1);
                a2 = fmaf(w2, x, a2);
                a3 = fmaf(w3, x, a3);
                b0 = fmaf(w0, y, b0);
                b1 = fmaf(w1, y, b1);
                b2 = fmaf(w2, y, b2);
                b3 = fmaf(w3, y, b3);
                --base;
                w3 = w2;
                w2 = w1;
                w1 = w0;
                w0 = kx[base];
            }
        }
        out[r0 * n + c] = a0;
        if (r0 + 1 < n) out[(r0 + 1) * n + c] = a1;
        if (r0 + 2 < n) out[(r0 + 2) * n + c] = a2;
        if (r0 + 3 < n) out[(r0 + 3) * n + c] = a3;
        if (two) {
            out[r0 * n + c2] = b0;
            if (r0 + 1 < n) out[(r0 + 1) * n + c2] = b1;
            if (r0 + 2 < n) out[(r0 + 2) * n + c2] = b2;
            if (r0 + 3 < n) out[(r0 + 3) * n + c2] = b3;
        }
    }
}

// Extended kernel length: 2n-1 entries plus the window's look-ahead, and one
// guard entry below index 0 (the window reads kx[-1] after its last step).
__device__ __forceinline__ int kx_len(int n) { return 2 * n + kSepStrip + 1; }

__global__ void __launch_bounds__(128) k_conv_sep(NetConst C, NetState* S) {
    extern __shared__ float sm[];
    const int g = grain_at(S, blockIdx.x);
    if (g > C.N || C.state[g] != G_EXISTS || halted(S)) return;
    const Box bx = S->box_cur[g];
    const int n = box_w(bx);
    if (n <= 0) return;
    if (n != box_h(bx) || n > C.tmax) {
        if (threadIdx.x == 0) set_status(S, n > C.tmax ? S_TABLE_RANGE : S_INDEX);
        return;
    }
    const float* in = reinterpret_cast<const float*>(S->phiA) + S->off_cur[g];
    float* out = reinterpret_cast<float*>(S->phiB) + S->off_cur[g];
    const float* kg = C.ck + C.ck_off[n];
    const bool fits = n <= C.conv_smem_edge;
    float* kx = sm + 1;  // sm[0] is the guard entry kx[-1]
    const int kl = kx_len(n);
    float* T = fits ? sm + 1 + kl : reinterpret_cast<float*>(S->spec) + S->soff_cur[g];
    for (int j = threadIdx.x; j < kl; j += blockDim.x) {
        int m = j - (n - 1);
        m %= n;
        if (m < 0) m += n;
        kx[j] = j < 2 * n - 1 ? kg[m] : 0.f;
    }
    if (threadIdx.x == 0) sm[0] = 0.f;
    __syncthreads();
    const int R = (int)kg[n];  // band radius stored after the n kernel entries
    sep_pass_rows(in, T, kx, n, R);
    __syncthreads();
    sep_pass_cols(T, out, kx, n, R);
}

size_t conv_sep_smem(int tmax, int edge) {
    // the row-pass intermediate of a box (edge up to `edge`) with its
    // extended kernel, or the extended kernel alone of the largest box (whose
    // intermediate goes to the grain's scratch in device memory)
    const int n = tmax < edge ? tmax : edge;
    const size_t staged = (size_t)n * n + 2 * (size_t)n + kSepStrip + 2;
    const size_t kernel_only = 2 * (size_t)tmax + kSepStrip + 2;
    return sizeof(float) * (staged > kernel_only ? staged : kernel_only);
}

// Batched-form corrector: same sectors as k_corrector (from k_sectors), with
// the previous contour staged in shared memory (FP32 box-local
// coordinates) and the per-pixel work in FP32, except the discrete decisions
// of the projection, which follow the reference's FP64 arithmetic.  Each
// warp scans the box in tiles and collects the pixels near the boundary, about a
// fifth, in a queue that full warps correct, each lane searching its own cell
// window.  The main kernel stages contours up to kCorrStagedPts points; the
// large-contour kernel, persistent over NetState::big_list, up to kCorrBigPts;
// longer ones are read from device memory in FP64.
//
// 20,000 Read-Shockley grains: 973 us with a warp correcting the pixels of its
// 8 x 4 tile in place (a third of the lanes busy, one pixel's loads in flight
// per lane), 605 us with the queue, of which the set-up takes 120 (a chain of
// dependent loads and five barriers), the scan 160 and the corrections 300;
// their floor, two fields read and a little written, is 60.  What bounds it is
// latency at 7 CTAs of 72 registers per SM (6: 676, 8 with spills: 676).
constexpr int kCorrBigPts = 1024;

// Nearest contour vertex of projectToGrainBondary (src/grainBoundary.cpp:
// 365-381) through a uniform grid of cells over the previous box: the
// vertices are bucketed by cell (counting sort in shared memory), and a pixel
// measures the vertices of the 3 x 3 cells around its own (in FP32, near-ties
// again in FP64 from the contour itself: see nearest_vertex).  Every vertex within `cell` of the pixel lies in that
// window, so when the smallest distance found is at most (cell - 1e-3)^2 (the
// margin covers the cell index of a vertex on a cell edge) it is the smallest
// over the whole contour; ties go to the lowest index, as the reference's
// strict < over ascending k.  Otherwise the pixel scans every vertex.
constexpr int kCellMax = 24;          // cells per side
template <int kPts>  // vertices bucketed (the staged contours)
struct VertexBuckets {
    int ncx, ncy, cell;
    float inv;  // 1 / cell
    int end[kCellMax * kCellMax + 1];  // after the fill: end[c + 1] = first vertex of cell c
    short list[kPts];
};

template <int kPts>
__device__ __forceinline__ int bucket_of(const VertexBuckets<kPts>& B, float2 v) {
    const int cx = min(max((int)floorf(v.x * B.inv), 0), B.ncx - 1);
    const int cy = min(max((int)floorf(v.y * B.inv), 0), B.ncy - 1);
    return cy * B.ncx + cx;
}

// All threads: buckets of the vertices 0 .. npts-1 from their staged FP32
// box-local coordinates P32 (each within 2^-24 L of the exact one; the cell from
// the product with 1 / cell adds 2^-23 L, all far inside the search's 1e-3
// margin for the boxes of at most kPts vertices).  Ends with a barrier.
template <int kPts>
__device__ void build_buckets(VertexBuckets<kPts>& B, const float2* P32, int npts, int wi, int hi) {
    const int cs = max(4, (max(wi, hi) + kCellMax - 1) / kCellMax);
    const int ncx = (wi + cs - 1) / cs, ncy = (hi + cs - 1) / cs, nc = ncx * ncy;
    if (threadIdx.x == 0) {
        B.ncx = ncx;
        B.ncy = ncy;
        B.cell = cs;
        B.inv = 1.f / (float)cs;
    }
    for (int c = threadIdx.x; c <= nc; c += blockDim.x) B.end[c] = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < npts; k += blockDim.x)
        atomicAdd(&B.end[bucket_of(B, P32[k]) + 1], 1);
    __syncthreads();
    if (threadIdx.x < 32) {  // inclusive scan of the counts by one warp
        int carry = 0;
        for (int c0 = 1; c0 <= nc; c0 += 32) {
            const int c = c0 + (int)threadIdx.x;
            int v = c <= nc ? B.end[c] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if ((int)threadIdx.x >= o) v += u;
            }
            if (c <= nc) B.end[c] = v + carry;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < npts; k += blockDim.x) {
        const int pos = atomicSub(&B.end[bucket_of(B, P32[k]) + 1], 1) - 1;
        B.list[pos] = (short)k;
    }
    __syncthreads();
}

constexpr unsigned kKeyIndexBits = 10;
constexpr unsigned kKeyIndexMask = (1u << kKeyIndexBits) - 1u;
static_assert(kCorrStagedPts <= kCorrBigPts && kCorrBigPts <= (1 << kKeyIndexBits), "vertex index must fit the key");

// The reference's nearest vertex of the pixel (px, py) (grid coordinates), by
// one lane.  It scans the vertices of its 3 x 3 cell window in FP32 on the
// staged box-local contour P32 (each coordinate within 2^-24 L of the exact
// local value, L the box edge, so a squared distance d within 3 sqrt(d) 2^-24 L
// + 3e-7 d of the exact one): each candidate is one 32-bit key, the distance's
// bits with the low 10 replaced by the vertex index, and the lane keeps its
// smallest key k1 and the second smallest k2.  The window's three cell rows are
// three ranges of the list, walked as one so that the warp's trip count is the
// longest window and not the sum of the longest rows.  A lane whose two best lie
// within twice the rounding bound (tie_margin with eps_c = 8 2^-24 L; the keys'
// truncation taken on both sides) measures the candidates within that margin
// again in FP64 from the contour itself, lowest index first at equal distance.
// A lane whose best distance exceeds (cell - 1e-3)^2 scans every vertex in FP64
// (a vertex within `cell` of the pixel lies in its window).
template <int kPts>
__device__ __forceinline__ int nearest_vertex(const VertexBuckets<kPts>& B, const float2* P32, const CPoint* P,
                                              int npts, int px, int py, int ox, int oy, float eps_c) {
    const int cs = B.cell;
    const int lx = px - ox, ly = py - oy;
    const float fx = (float)lx, fy = (float)ly;
    // the pixel's cell (half a pixel in, the rounding of 1 / cell is no matter)
    const int cx = min(max((int)floorf((fx + 0.5f) * B.inv), 0), B.ncx - 1);
    const int cy = min(max((int)floorf((fy + 0.5f) * B.inv), 0), B.ncy - 1);
    const int ncell = B.ncx * B.ncy;
    int start[3], upto[3], total = 0;
    for (int r = 0; r < 3; ++r) {
        const int yy = cy - 1 + r;
        int q0 = 0, q1 = 0;
        if (yy >= 0 && yy < B.ncy) {
            // the cells of a row are consecutive in the list
            q0 = B.end[yy * B.ncx + max(cx - 1, 0) + 1];
            const int cl = yy * B.ncx + min(cx + 1, B.ncx - 1);
            q1 = cl + 1 < ncell ? B.end[cl + 2] : npts;
        }
        start[r] = q0 - total;
        total += q1 - q0;
        upto[r] = total;
    }
    unsigned k1 = 0xffffffffu, k2 = 0xffffffffu;
#pragma unroll 2
    for (int q = 0; q < total; ++q) {
        const int k = B.list[q + (q < upto[0] ? start[0] : q < upto[1] ? start[1] : start[2])];
        const float2 v = P32[k];
        const float dx = fx - v.x, dy = fy - v.y;
        const float d = fmaf(dy, dy, dx * dx);
        const unsigned key = (__float_as_uint(d) & ~kKeyIndexMask) | (unsigned)k;
        k2 = min(k2, max(k1, key));
        k1 = min(k1, key);
    }
    const float d1 = __uint_as_float(min(k1 | kKeyIndexMask, 0x7f7fffffu));
    const float r = (float)cs - 1e-3f;
    const bool covered = k1 != 0xffffffffu && d1 <= r * r;
    const float thr = d1 + tie_margin(d1, eps_c);
    const bool tie = covered && k2 != 0xffffffffu && __uint_as_float(k2 & ~kKeyIndexMask) <= thr;
    int nearest = (int)(k1 & kKeyIndexMask);
    if (!covered) {
        const double dpx = (double)px, dpy = (double)py;
        double best = 1000000.0;  // the reference's initial minDist
        nearest = -1;
        for (int k = 0; k < npts; ++k) {
            const double d = dist2_rn(dpx, dpy, P[k]);
            if (d < best) {
                best = d;
                nearest = k;
            }
        }
    } else if (tie) {
        const double dpx = (double)px, dpy = (double)py;
        double best = 1000000.0;
        nearest = -1;
        for (int q = 0; q < total; ++q) {
            const int k = B.list[q + (q < upto[0] ? start[0] : q < upto[1] ? start[1] : start[2])];
            const float dx = fx - P32[k].x, dy = fy - P32[k].y;
            if (fmaf(dy, dy, dx * dx) > thr) continue;
            const double d = dist2_rn(dpx, dpy, P[k]);
            if (d < best || (d == best && k < nearest)) {
                best = d;
                nearest = k;
            }
        }
    }
    return nearest;
}

// Distance from (fx, fy) to segment a -> b (the reference's three cases);
// *lam receives the unclamped projection parameter.
__device__ __forceinline__ float seg_dist32(float2 a, float2 b, float fx, float fy, float* lam) {
    const float ux = b.x - a.x, uy = b.y - a.y;
    const float l = ((fx - a.x) * ux + (fy - a.y) * uy) / (ux * ux + uy * uy);
    float dx, dy;
    if (l < 0) {
        dx = fx - a.x;
        dy = fy - a.y;
    } else if (l > 1) {
        dx = b.x - fx;
        dy = b.y - fy;
    } else {
        dx = fx - (a.x + ux * l);
        dy = fy - (a.y + uy * l);
    }
    *lam = l;
    return dx * dx + dy * dy;
}

// The segment step of projectToGrainBondary (src/grainBoundary.cpp:383-420)
// on the FP32 local contour P32: the segment after the vertex first, the one
// before it wins only if strictly closer.  When both projections fall beyond
// the vertex, both distances are the vertex's (equal in FP64 too) and the
// segment after it wins with lambda 0; when the two distances lie within the
// FP32 rounding margin (eps_c = 8 2^-24 L, L bounding the local coordinates)
// the step is taken again in FP64 from the contour itself.
__device__ __forceinline__ int segment_step(const float2* P32, const CPoint* P, int asize, int px, int py, int ox,
                                           int oy, float eps_c, int nearest, float* out_lambda) {
    const float fx = (float)(px - ox), fy = (float)(py - oy);
    float la, lb;
    const float da = seg_dist32(P32[nearest], P32[nearest + 1], fx, fy, &la);
    const int nv = nearest == 0 ? asize - 1 : nearest;
    const float db = seg_dist32(P32[nv - 1], P32[nv], fx, fy, &lb);
    if (la <= 0.f && lb >= 1.f) {
        *out_lambda = 0.f;
        return nearest;
    }
    if (fabsf(da - db) <= 4.f * tie_margin(fminf(da, db), eps_c)) {
        double dl = 0;
        const int seg = segment_of_vertex(P, asize, (double)px, (double)py, nearest, &dl);
        *out_lambda = (float)dl;
        return seg;
    }
    const bool before = db < da;
    const float lam = before ? lb : la;
    *out_lambda = fminf(fmaxf(lam, 0.f), 1.f);
    return before ? nv - 1 : nearest;
}

// An interpolating sector as the per-pixel weights use it.
struct SectorWeights {
    float length, left_w, right_w, boundary_w;
    int32_t both;  // boundary sectors on both sides
};

// Shared memory of one CTA of the batched corrector.
template <int kPts>
struct CorrectorSmem {
    float2 sp[kPts];  // the contour, FP32 box-local
    NbTable nbt;
    VertexBuckets<kPts> vb;
    float cw[kMaxConstSectors];
    SectorWeights is[kMaxInterpSectors];
    int16_t sid[kPts];  // per-segment sector table
    float acc[kPts];
    unsigned queue[4][160];  // per warp: pixels to correct, y << 16 | x
};

// The correction of grain g, if it is corrected at all this step, by the whole
// CTA (all threads call it; every early return is uniform over the CTA).
template <bool kForces, int kPts>
__device__ __forceinline__ void correct_grain(const NetConst& C, NetState* S, int g, CorrectorSmem<kPts>& sm) {
    float2* sp = sm.sp;
    NbTable& nbt = sm.nbt;
    VertexBuckets<kPts>& vb = sm.vb;
    int16_t* s_sid = sm.sid;
    float* s_acc = sm.acc;
    // everything that hangs on g alone is loaded before the first decision
    const bool live = C.state[g] == G_EXISTS & C.regular[g] != 0 & S->loop != 0 & !halted(S);
    const int64_t coff = S->coff_prev[g];
    const int size = S->cn_prev[g];
    const Box ib = S->box_prev[g], bo = S->box_cur[g];
    const int64_t off_prev = S->off_prev[g], off_cur = S->off_cur[g];
    if (!live || size < 2) return;
    const CPoint* P = S->contPrev + coff;
    const uint32_t* idl = S->idPrev + off_prev;
    const bool staged = size <= kPts;
    // the contour in FP32 coordinates local to the previous box (its points
    // lie inside it), so the search's rounding is relative to the box edge
    const int ox = ib.x0, oy = ib.y0;
    if (staged)
        for (int k = threadIdx.x; k < size; k += blockDim.x)
            sp[k] = make_float2((float)(P[k].x - ox), (float)(P[k].y - oy));
    // the sectors, built one step ahead (k_sectors), and the per-segment table
    const SectorPack* pk = reinterpret_cast<const SectorPack*>(C.secpack) + g;
    const int nconst = pk->nconst, ninterp = pk->ninterp;
    for (int c = threadIdx.x; c < nconst; c += blockDim.x) sm.cw[c] = (float)pk->cw[c];
    for (int c = threadIdx.x; c < ninterp; c += blockDim.x) {
        const InterpSector& from = pk->is[c];
        sm.is[c] = SectorWeights{(float)from.length, (float)from.left_w, (float)from.right_w, (float)from.boundary_w,
                                 from.lb >= 0 && from.rb >= 0};
    }
    const int16_t* tsid = C.segsec + coff;
    const float* tacc = C.segacc + coff;
    if (staged) {
        for (int q = threadIdx.x; q < size - 1; q += blockDim.x) {
            s_sid[q] = tsid[q];
            s_acc[q] = tacc[q];
        }
    }
    build_nb_table(C, g, nbt);
    if (staged) build_buckets(vb, sp, size - 1, box_w(ib), box_h(ib));  // ends with a barrier
    __syncthreads();
    const int x0 = ib.x0 < bo.x0 ? bo.x0 : ib.x0;
    const int y0 = ib.y0 < bo.y0 ? bo.y0 : ib.y0;
    const int x1 = ib.x1 > bo.x1 ? bo.x1 : ib.x1;
    const int y1 = ib.y1 > bo.y1 ? bo.y1 : ib.y1;
    if (x1 <= x0 || y1 <= y0) return;
    const int w = x1 - x0, hgt = y1 - y0;
    const float* in = reinterpret_cast<const float*>(S->phiA) + off_cur;
    float* out = reinterpret_cast<float*>(S->phiB) + off_cur;
    const int wo = box_w(bo), wi = box_w(ib);
    const float delta = (float)C.delta;
    const int real = size - 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int ntx = (w + 15) >> 4;
    const bool far_ok = C.gamma_hagb <= 1.0 && C.m_hagb <= 1.0;
    // driving-force terms (src/box.cpp:511-527) of a pixel owned by `id`
    const auto force = [&](uint32_t id) {
        double f = 0;
        if (C.stored) f += nb_stored_force(nbt, (int)id) * C.dt / C.time_slope;
        if (C.magnetic) f += nb_magnetic_force(nbt, (int)id) * C.dt / C.time_slope;
        return (float)f;
    };
    // rounding margin of the FP32 segment step: 8 2^-24 L, L bounding every
    // local coordinate of the contour and the pixels
    const float eps_c = 8.f * 5.9604645e-8f * (float)(max(wi, box_h(ib)) + 2);
    // Each warp scans 16 x 8 tiles, four pixels per lane with their loads in
    // flight together: pixels at or below -delta are set to -delta, far ones
    // keep their convolved value, and the others, about a fifth, join the warp's
    // queue, which is corrected by full warps.
    //
    // The corrected value val + (conv - val) w lies between val and
    // 2 conv - val for every weight w in [0, 2]; with the relative
    // high-angle energy and mobility at most 1 the weights (energy x
    // mobility products, junction sums of three energies, their blends)
    // stay below 2 (far_ok).  When val, conv and
    // 2 conv - val all lie on the same side beyond 0.3 delta (2.1 cells),
    // the pixel keeps that side whatever its weight, and it is not next to
    // a sign change of these near-distance fields; only signs and the
    // values next to sign changes reach the comparison's zero crossings
    // and the redistancing that replaces the field.  Such a pixel takes
    // weight 1 (the convolved value) without the projection.  (On the
    // 20,000-grain workload the areas stay bit-identical for 10 steps and
    // within 1.3e-7 relative, in 18 grains, after 40.)
    const float far_level = 0.3f * delta;
    unsigned* queue = sm.queue[warp];
    const int nty = (hgt + 7) >> 3;
    int tx = warp % ntx, ty = warp / ntx, queued = 0;
    for (bool more = true; more;) {
        more = ty < nty;
        if (more) {
            const int x = tx * 16 + (lane & 15), yt = ty * 8 + (lane >> 4);
            for (tx += nwarps; tx >= ntx; tx -= ntx) ++ty;
            const int j = x0 + x;
            float val[4], conv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int y = yt + 2 * u;
                const int k = (y0 + y - bo.y0) * wo + (j - bo.x0);
                val[u] = conv[u] = 0.f;
                if (x < w && y < hgt) {
                    val[u] = __ldg(in + k);
                    conv[u] = out[k];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int y = yt + 2 * u, i = y0 + y;
                const bool inside = x < w && y < hgt;
                const bool valid = inside && val[u] > -delta;
                const float stretched = 2.f * conv[u] - val[u];
                const bool far = far_ok && valid &&
                                 ((val[u] >= far_level && conv[u] >= far_level && stretched >= far_level) ||
                                  (val[u] <= -far_level && conv[u] <= -far_level && stretched <= -far_level));
                const bool need = valid && !far;
                if (inside && (kForces ? !need : !valid)) {
                    float se = 0.f;
                    if (kForces) se = force(idl[(i - ib.y0) * wi + (j - ib.x0)]);
                    out[(i - bo.y0) * wo + (j - bo.x0)] = (far ? conv[u] : -delta) - se;
                }
                const unsigned needs = __ballot_sync(0xffffffffu, need);
                if (need) queue[queued + __popc(needs & ((1u << lane) - 1u))] = (unsigned)y << 16 | (unsigned)x;
                queued += __popc(needs);
            }
            __syncwarp();
        }
        while (queued >= 32 || (!more && queued > 0)) {
            const bool busy = lane < queued;
            queued = queued > 32 ? queued - 32 : 0;  // from the end
            const unsigned item = busy ? queue[queued + lane] : 0u;
            __syncwarp();
            if (!busy) break;
            const int i = y0 + (int)(item >> 16), j = x0 + (int)(item & 0xffffu);
            const int k = (i - bo.y0) * wo + (j - bo.x0);
            const int at_id = (i - ib.y0) * wi + (j - ib.x0);
            const float val = __ldg(in + k), conv = out[k];
            float lambda = 0.f;
            int segment = 0;
            if (staged) {
                const int nv = nearest_vertex(vb, sp, P, size - 1, j, i, ox, oy, eps_c);
                if (nv >= 0) segment = segment_step(sp, P, size, j, i, ox, oy, eps_c, nv, &lambda);
            } else {
                double dl = 0;
                segment = project_to_boundary(P, size, (double)j, (double)i, &dl);
                lambda = (float)dl;
            }
            const int sid = staged ? s_sid[segment] : tsid[segment];
            float interpolator = sid > -2 ? 0.f : staged ? s_acc[segment] : tacc[segment];
            float weight;
            if (sid >= 0) {
                weight = sm.cw[sid];
            } else if (sid == -1) {
                // getGBEnergyTimesGBMobility(i, j) through the neighbour table
                const int id = (int)idl[at_id];
                weight = 1.f;
                for (int e = 0; e < nbt.n; ++e)
                    if (nbt.id[e] == id) {
                        weight = (float)nbt.w[e];
                        break;
                    }
            } else {
                const SectorWeights& s = sm.is[-2 - sid];
                const int kn = wrap_next(segment, real);
                float ax, ay;
                if (staged) {
                    ax = (sp[kn].x - sp[segment].x) * lambda;
                    ay = (sp[kn].y - sp[segment].y) * lambda;
                } else {
                    ax = (float)((P[kn].x - P[segment].x) * lambda);
                    ay = (float)((P[kn].y - P[segment].y) * lambda);
                }
                interpolator += sqrtf(ax * ax + ay * ay);
                interpolator /= s.length;
                interpolator = fminf(fmaxf(interpolator, 0.f), 1.f);
                const float lw = s.left_w, rw = s.right_w;
                if (s.both) {
                    const float isr = (float)C.isr, len = s.length;
                    const float quot = (len > 2 * isr ? 2 * isr : len);
                    const float amplitude = (s.boundary_w - (lw + rw) / 2) / (2 * isr) * quot + (lw + rw) / 2;
                    const float a0 = 2 * rw, a1 = -4 * amplitude, a2 = 2 * lw;
                    const float A = a0 + a1 + a2, B = -(a0 * 1.5f + a1 + a2 * 0.5f), Cc = a0 * 0.5f;
                    weight = A * interpolator * interpolator + B * interpolator + Cc;
                } else {
                    weight = interpolator * lw + (1 - interpolator) * rw;
                }
            }
            float se = 0.f;
            if (kForces) se = force(idl[at_id]);
            out[k] = val + (conv - val) * weight - se;
        }
    }
}

// CTA per grain from the work queue, contours staged up to kCorrStagedPts;
// grains flagged for the large-contour kernel are left to it.
template <bool kForces>
__global__ void __launch_bounds__(128, 7) k_corrector_f(NetConst C, NetState* S) {
    __shared__ __align__(16) CorrectorSmem<kCorrStagedPts> sm;
    const int g = grain_at(S, blockIdx.x);
    if (S->big_flag[g]) return;
    correct_grain<kForces, kCorrStagedPts>(C, S, g, sm);
}

// Persistent over NetState::big_list: the grains whose contour is longer than
// the main kernel stages, up to kCorrBigPts staged; CTA b takes entries b,
// b + G, ... (G CTAs).  The grid (kCorrBigPerSm CTAs per SM) usually covers
// the whole list, so every such grain starts at once, and the launch has the
// device's highest priority, so that these CTAs are placed before the
// pending ones of the main corrector beside them.
template <bool kForces>
__global__ void __launch_bounds__(128) k_corrector_big(NetConst C, NetState* S) {
    __shared__ __align__(16) CorrectorSmem<kCorrBigPts> sm;
    const int n = S->n_big;
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const int g = S->big_list[q];
        correct_grain<kForces, kCorrBigPts>(C, S, g, sm);
        __syncthreads();  // the next grain overwrites the shared memory
    }
}

// SMs of the device, the unit of the persistent grids
int g_big_grid = 148;
// highest stream priority of the device (numerically lowest)
int g_high_priority = 0;
constexpr int kCorrBigPerSm = 4;

void launch_corrector_main(const NetConst& C, NetState* dS, cudaStream_t s) {
    if (C.stored || C.magnetic)
        k_corrector_f<true><<<C.N, 128, 0, s>>>(C, dS);
    else
        k_corrector_f<false><<<C.N, 128, 0, s>>>(C, dS);
}

void launch_corrector_big(const NetConst& C, NetState* dS, cudaStream_t s) {
    const int grid = C.N < kCorrBigPerSm * g_big_grid ? C.N : kCorrBigPerSm * g_big_grid;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = g_high_priority;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (C.stored || C.magnetic)
        cudaLaunchKernelEx(&cfg, k_corrector_big<true>, C, dS);
    else
        cudaLaunchKernelEx(&cfg, k_corrector_big<false>, C, dS);
}

// Both correctors on one stream (the graph runs them on two).
void launch_corrector_f(const NetConst& C, NetState* dS, cudaStream_t s) {
    launch_corrector_big(C, dS, s);
    launch_corrector_main(C, dS, s);
}

cudaError_t batched_resample(const NetConst& C, NetState* dS, double h_old, double hn, double delta_old,
                             cudaStream_t s) {
    if (C.N > 0) k_resample<float><<<C.N, 256, 0, s>>>(C, dS, h_old, hn, delta_old);
    return cudaGetLastError();
}

// The large-box bin: a persistent grid walks the work queue (largest boxes
// first) and stops at the first existing grain at or below C.big_edge, where
// k_redistance's begin.
__global__ void __launch_bounds__(RedistLarge<float>::kThreads, RedistLarge<float>::kPerSm)
    k_redistance_big(NetConst C, NetState* S) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    if (!S->order) return;
    for (int slot = blockIdx.x; slot < C.N; slot += gridDim.x) {
        const int g = S->order[slot];
        // a grain that vanished in this step's level set keeps its place in
        // the queue; existing grains are in descending box edge
        if (C.state[g] != G_EXISTS || halted(S)) continue;
        if (box_w(S->box_cur[g]) <= C.big_edge) return;
        redistance_grain<float, true>(C, S, g, s_raw);
        __syncthreads();  // the next grain reuses the shared buffers
    }
}

cudaError_t batched_prepare(int tmax) {
    cudaError_t e = cudaFuncSetAttribute(k_conv_sep, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)conv_sep_smem(tmax, kConvSmemEdgeMax));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_redistance_big, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)redist_smem<float, true>());
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    g_big_grid = sms > 0 ? sms : 148;
    int least = 0, greatest = 0;
    if ((e = cudaDeviceGetStreamPriorityRange(&least, &greatest)) != cudaSuccess) return e;
    g_high_priority = greatest;
    return cudaSuccess;
}

// Launch with the device's highest priority: beside another kernel its CTAs
// are placed first.
template <class K>
void launch_first(K kernel, int grid, int threads, size_t smem, cudaStream_t s, const NetConst& C, NetState* dS) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = g_high_priority;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, C, dS);
}

// The largest boxes' level set (8 one-warp CTAs per SM) and the others'.
void launch_levelset_big(const NetConst& C, NetState* dS, cudaStream_t s) {
    launch_first(k_levelset_big<float>, C.N < 8 * g_big_grid ? C.N : 8 * g_big_grid, 32, 0, s, C, dS);
}

void launch_levelset_main(const NetConst& C, NetState* dS, cudaStream_t s) {
    k_levelset_w<float><<<(C.N + kGrainsPerBlock - 1) / kGrainsPerBlock, 32 * kGrainsPerBlock, 0, s>>>(C, dS);
}

// Both on one stream (the graph runs them on two).
void launch_levelset(const NetConst& C, NetState* dS, cudaStream_t s) {
    launch_levelset_big(C, dS, s);
    launch_levelset_main(C, dS, s);
}

// The large-box bin of the redistancing.
void launch_redistance_big(const NetConst& C, NetState* dS, cudaStream_t s) {
    using L = RedistLarge<float>;
    const int most = L::kPerSm * g_big_grid;
    launch_first(k_redistance_big, C.N < most ? C.N : most, L::kThreads, redist_smem<float, true>(), s, C, dS);
}

void launch_redistance_main(const NetConst& C, NetState* dS, cudaStream_t s) {
    k_redistance<float, false><<<C.N, kRedistThreads, redist_smem<float, false>(), s>>>(C, dS);
}

// Both on one stream (the graph runs them on two).
void launch_redistance(const NetConst& C, NetState* dS, cudaStream_t s) {
    launch_redistance_big(C, dS, s);
    launch_redistance_main(C, dS, s);
}

cudaError_t batched_init(const NetConst& C, NetState* dS, const int32_t* d_ids, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_init_phi<float><<<C.N, 256, 0, s>>>(C, dS, d_ids);
    // the step's redistancing kernels take grains from the work queue, so it
    // is built from the initial boxes first
    k_order<<<1, 1024, 0, s>>>(C, dS);
    launch_redistance(C, dS, s);
    cudaError_t e = swap_phi(dS, s);
    if (e != cudaSuccess) return e;
    k_init_contour_big<float><<<C.N, 32, 0, s>>>(C, dS);
    k_init_contour_w<float><<<(C.N + kGrainsPerBlock - 1) / kGrainsPerBlock, 32 * kGrainsPerBlock, 0, s>>>(C, dS);
    return cudaGetLastError();
}

size_t batched_sector_pack_bytes() { return sizeof(SectorPack); }

cudaError_t batched_sectors(const NetConst& C, NetState* dS, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_sectors<false, float><<<C.N, 32, 0, s>>>(C, dS);
    return cudaGetLastError();
}

cudaError_t batched_order(const NetConst& C, NetState* dS, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_order<<<1, 1024, 0, s>>>(C, dS);
    return cudaGetLastError();
}

cudaError_t batched_init_polygon(const NetConst& C, NetState* dS, cudaStream_t s) {
    if (C.N <= 0) return cudaSuccess;
    k_polygon_phi<float><<<C.N, 256, 0, s>>>(C, dS);
    return cudaGetLastError();
}

cudaError_t batched_stage_kernel(const NetConst& C, NetState* dS, int which, cudaStream_t s, const LaunchCfg& cfg) {
    const int wblocks = (C.N + kGrainsPerBlock - 1) / kGrainsPerBlock;
    switch (which) {
        case 0: k_conv_sep<<<C.N, 128, conv_sep_smem(C.tmax, C.conv_smem_edge), s>>>(C, dS); break;
        case 1: if (!C.isotropic) launch_corrector_f(C, dS, s); break;
        case 2: k_second_order_w<<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS); break;
        case 3: k_compare<float><<<C.N, cfg.compare_threads, 0, s>>>(C, dS); break;
        case 4: launch_levelset(C, dS, s); break;
        case 5: k_alloc<<<1, 1024, 0, s>>>(C, dS, 1); break;
        case 6:
            k_neighbours_w<float><<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS, reinterpret_cast<PointInfo*>(C.ptinfo));
            k_sectors<true, float><<<C.N, 32, 0, s>>>(C, dS);
            break;
        case 7: launch_redistance(C, dS, s); break;
        default:
            k_finalize<<<1, 1024, 0, s>>>(C, dS, 1);
            k_order<<<1, 1024, 0, s>>>(C, dS);
            break;
    }
    return cudaGetLastError();
}

cudaError_t batched_stages(const NetConst& C, NetState* dS, int stages, cudaStream_t s, const LaunchCfg& cfg) {
    if (C.N <= 0) return cudaSuccess;
    const int wblocks = (C.N + kGrainsPerBlock - 1) / kGrainsPerBlock;
    if (stages & ST_CONV) {
        k_conv_sep<<<C.N, 128, conv_sep_smem(C.tmax, C.conv_smem_edge), s>>>(C, dS);
        if (!C.isotropic) launch_corrector_f(C, dS, s);
    }
    if (stages & ST_SECOND) k_second_order_w<<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS);
    if (stages & ST_COMPARE) k_compare<float><<<C.N, cfg.compare_threads, 0, s>>>(C, dS);
    if (stages & ST_LEVELSET) launch_levelset(C, dS, s);
    if (stages & ST_REDIST) {
        k_alloc<<<1, 1024, 0, s>>>(C, dS, 1);
        k_neighbours_w<float><<<wblocks, 32 * kGrainsPerBlock, 0, s>>>(C, dS, reinterpret_cast<PointInfo*>(C.ptinfo));
        k_sectors<true, float><<<C.N, 32, 0, s>>>(C, dS);
        launch_redistance(C, dS, s);
        k_finalize<<<1, 1024, 0, s>>>(C, dS, 1);
        k_order<<<1, 1024, 0, s>>>(C, dS);
    }
    return cudaGetLastError();
}

cudaError_t batched_step_graph(const NetConst& C, NetState* dS, cudaStream_t s, const LaunchCfg& cfg) {
    if (C.N <= 0) return cudaSuccess;
    const cudaStream_t s2 = cfg.side[0], s3 = cfg.side[1];
    cudaEvent_t* const ev = cfg.ev;
    const int wblocks = (C.N + kGrainsPerBlock - 1) / kGrainsPerBlock;
    cudaError_t e;
    // second-order lists (lists and boxes only) beside convolution + corrector (fields)
    if ((e = cudaEventRecord(ev[0], s)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(s2, ev[0], 0)) != cudaSuccess) return e;
    k_second_order_w<<<wblocks, 32 * kGrainsPerBlock, 0, s2>>>(C, dS);
    k_conv_sep<<<C.N, 128, conv_sep_smem(C.tmax, C.conv_smem_edge), s>>>(C, dS);
    if (!C.isotropic) {
        // the large-contour corrector beside the main one
        if ((e = cudaEventRecord(ev[4], s)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(s2, ev[4], 0)) != cudaSuccess) return e;
        launch_corrector_big(C, dS, s2);
        launch_corrector_main(C, dS, s);
    }
    if ((e = cudaEventRecord(ev[1], s2)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(s, ev[1], 0)) != cudaSuccess) return e;
    k_compare<float><<<C.N, cfg.compare_threads, 0, s>>>(C, dS);
    // the largest boxes' contours beside the others
    if ((e = cudaEventRecord(ev[0], s)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(s3, ev[0], 0)) != cudaSuccess) return e;
    launch_levelset_big(C, dS, s3);
    if ((e = cudaEventRecord(ev[5], s3)) != cudaSuccess) return e;
    launch_levelset_main(C, dS, s);
    if ((e = cudaStreamWaitEvent(s, ev[5], 0)) != cudaSuccess) return e;
    k_alloc<<<1, 1024, 0, s>>>(C, dS, 1);
    // volume / energy / neighbours (contours, lists) and the next step's
    // sectors beside redistancing (fields)
    if ((e = cudaEventRecord(ev[2], s)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(s3, ev[2], 0)) != cudaSuccess) return e;
    launch_redistance_big(C, dS, s3);
    if ((e = cudaEventRecord(ev[5], s3)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(s2, ev[2], 0)) != cudaSuccess) return e;
    k_neighbours_w<float><<<wblocks, 32 * kGrainsPerBlock, 0, s2>>>(C, dS, reinterpret_cast<PointInfo*>(C.ptinfo));
    k_sectors<true, float><<<C.N, 32, 0, s2>>>(C, dS);  // the next step's sectors
    if ((e = cudaEventRecord(ev[3], s2)) != cudaSuccess) return e;
    launch_redistance_main(C, dS, s);
    if ((e = cudaStreamWaitEvent(s, ev[3], 0)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(s, ev[5], 0)) != cudaSuccess) return e;
    k_finalize<<<1, 1024, 0, s>>>(C, dS, 1);
    k_order<<<1, 1024, 0, s>>>(C, dS);  // the next step's work queue, from its boxes
    return cudaGetLastError();
}

}  // namespace gg
