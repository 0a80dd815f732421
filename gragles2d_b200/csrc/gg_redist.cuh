// Redistancing (LSbox::executeRedistancing, src/box.cpp:1259-1399): the
// compared field (arena A, box_cur) -> phi_{t+1} (arena B, box_new), clamped
// to +-delta.  Four directional sweeps over the new box: y forward and back
// with one thread per column, then x forward and back with one thread per row.
//
// Each sweep is a recurrence along the box's edge, so it costs the length of
// one step's dependent chain times the steps, hidden only by other boxes'
// warps on the same SM.  The form below leaves one addition, one comparison
// and one select in a step, keeps little shared memory per box, and gives the
// values of the reference's loop exactly:
//
//  - the zero-crossing values (two divisions each) do not depend on the
//    recurrence.  The pixel pairs with a sign change (about two per boundary
//    row and column, 5% of a 44^2 box) are listed first, and the listed ones
//    evaluated across the lanes;
//  - the output starts at -1, so a y crossing value z (|z| < 1) is put in its
//    pixel before the y forward sweep, and an x crossing value with |z| below
//    the y sweeps' result in its pixel before the x forward sweep.  Every
//    sweep is then the same step: cand = cur +- h replaces the pixel's value
//    o if |cand| < |o|, or if |cand| = |o| and o is a crossing value just put
//    there (which the reference tests after the candidate);
//  - that case of equality only matters when cand = -z, for which the previous
//    pixel must hold a value of the wrong sign and of magnitude above h.  Wrong
//    signs come only from the -1 start values, 1 - k h after k steps, so not in
//    a box that is a few cells smaller than the domain (kFlags off; the plain
//    form keeps the test in every box);
//  - the input itself is not kept: the first pass turns it into bit masks of
//    its signs, one ballot per 32 pixels, and the pairs with a sign change are
//    exclusive ors of mask words.  That needs values whose sign is +-1 and
//    whose products with each other do not underflow; a box with a zero, a NaN
//    or a magnitude below 1e-20 (1e-150 in FP64) takes redistance_strips.
//
// Measured (B200, the stage's device time, before: input and output staged as
// fields, the crossing divisions inside the sweeps): 20,000 grains (FP32, mean
// edge 48) 564 -> 341 us; 100,000 clustered grains (edges up to 260) 8.28 ->
// 2.52 ms; 5,000 grains in FP64 576 -> 253 us; one box of a small network 60
// -> 10 us.  It is bound by instruction issue where many boxes run (62% of the
// slots, about 10,700 warp instructions per box) and by the sweeps' chain (35
// cycles per step) where few do.
#pragma once

#include "gg_grain.cuh"
#include "gg_kernels.cuh"

namespace gg {
namespace {  // internal linkage: each form's translation unit has its own copy

// The largest value below v > 0 (NaN for 0, below which there is none).
__device__ __forceinline__ float value_below(float v) { return __int_as_float(__float_as_int(v) - 1); }
__device__ __forceinline__ double value_below(double v) { return __longlong_as_double(__double_as_longlong(v) - 1); }

// h with its sign set by the top bit of w.
__device__ __forceinline__ float signed_by(float h, unsigned w) {
    return __uint_as_float(__float_as_uint(h) | (w & 0x80000000u));
}
__device__ __forceinline__ double signed_by(double h, unsigned w) {
    return __hiloint2double((int)((unsigned)__double2hiint(h) | (w & 0x80000000u)), __double2loint(h));
}

// The zero-crossing value of the pair (a, c), a * c <= 0 (src/box.cpp:1293-1297);
// NaN where the slope is zero, which no test selects.
template <typename R>
__device__ __forceinline__ R crossing_value(R a, R c, R h) {
    const R slope = (c - a) / h;
    const R dz = -a / slope;
    return -dz * (R)sgn(slope);
}

// One step: cand against the pixel's value o; with `tie`, cand also wins at
// equal magnitude.
template <typename R>
__device__ __forceinline__ bool takes(R cand, R o, bool tie) {
    return fabs(cand) <= (tie ? fabs(o) : value_below(fabs(o)));
}

// Whether v may take the staged form (see the head of the file).
__device__ __forceinline__ bool ordinary(float v) { return fabsf(v) >= 1e-20f; }
__device__ __forceinline__ bool ordinary(double v) { return fabs(v) >= 1e-150; }

// Shared memory of a staged box with an edge of up to kCap: the output, the
// sources with kSource, and per row the bit masks of the input's sign (1:
// negative) and, with kFlags, of the x crossing values in place.  The box has
// a border of kPad cells (its values are never used): sweeps run in groups of
// kPad steps and may end inside it, and the row stride is a constant, odd (rows
// walked side by side meet distinct banks).  Bit kPad + c of a row's mask is
// column c of the box.
constexpr int kPad = 4;
constexpr int kCrossList = 256;  // crossing pairs a warp lists; a box with more goes the way of a large one

template <typename R, int kCap, int kThreads, bool kSource>
struct RedistSmem {
    static constexpr int kStride = (kCap + 2 * kPad) | 1;
    static constexpr int kRows = kCap + 2 * kPad;
    static constexpr int kWords = (kCap + 2 * kPad + 31) / 32 + 1;  // one past the last is readable
    static constexpr int kLists = (kCap + 35) / 36;                  // warps that list pairs, 32 rows at a time
    static_assert(kLists <= kThreads / 32);
    R cell[kRows * kStride];
    R z[kLists][kCrossList];  // crossing values of the listed pairs
    unsigned list[kLists][kCrossList];  // row << 16 | column of the intersection, top bit for an x pair
    unsigned neg[kRows * kWords], flag[kRows * kWords];
    int src[kSource ? kRows * kStride : 1];
    int refused;
    static __device__ __forceinline__ int at(int r, int c) { return (r + kPad) * kStride + c + kPad; }
    static __device__ __forceinline__ int word(int r, int c) { return (r + kPad) * kWords + ((c + kPad) >> 5); }
};

// Steps of one sweep in groups of kPad: targets p[0], p[S], ...; load(g)
// fetches group g's mask bits, sign(bits, u) sets step u's sign bit and
// tie(bits, u, o) says whether a candidate of the same magnitude wins.  The
// next group is loaded before the current one is computed.
template <typename R, int S, bool kTies, bool kSource, class Load, class Sign, class Tie>
__device__ __forceinline__ void sweep_line(R* p, int* ps, int cnt, R cur, R h, Load load, Sign sign, Tie tie) {
    int groups = (cnt + kPad - 1) / kPad, g = 0;
    if (groups <= 0) return;
    int src = kSource ? ps[-S] : 0;
    auto fetch = [&](R (&o)[kPad], int at) {
#pragma unroll
        for (int u = 0; u < kPad; ++u) o[u] = p[(at + u) * S];
    };
    auto run = [&](const R (&o)[kPad], const auto& bits) {
#pragma unroll
        for (int u = 0; u < kPad; ++u) {
            const R cand = cur + signed_by(h, sign(bits, u));
            const bool in = kTies ? takes(cand, o[u], tie(bits, u, o[u])) : fabs(cand) < fabs(o[u]);
            cur = in ? cand : o[u];
            p[u * S] = cur;
            if constexpr (kSource) {
                if (!in) src = ps[u * S];
                ps[u * S] = src;
            }
        }
        p += kPad * S;
        ps += kPad * S;
    };
    R a[kPad], b[kPad];
    fetch(a, 0);
    auto wa = load(0), wb = wa;
    while (true) {
        if (g + 1 < groups) {
            fetch(b, kPad);
            wb = load(g + 1);
        }
        run(a, wa);
        if (++g == groups) break;
        if (g + 1 < groups) {
            fetch(a, kPad);
            wa = load(g + 1);
        }
        run(b, wb);
        if (++g == groups) break;
    }
}

struct MaskRows {  // mask words of kPad rows of one column
    unsigned w[kPad];
};
struct MaskBits {  // mask bits of kPad columns of one row, with their flags
    unsigned w, f;
};

// y sweep of column c from row r, whose cell p is: forward or backward to the
// box's end.
template <typename R, class M, bool kForward, bool kFlags, bool kSource>
__device__ __forceinline__ void y_sweep(M& m, int r, int c, int cnt, R h) {
    constexpr int kDir = kForward ? 1 : -1, S = kDir * M::kStride;
    const int i = M::at(r, c), sft = 31 - ((c + kPad) & 31);
    const unsigned* const n = m.neg + M::word(r + kDir, c);
    sweep_line<R, S, kForward && kFlags, kSource>(
        m.cell + i + S, m.src + (kSource ? i + S : 0), cnt, m.cell[i], h,
        [&](int g) {
            MaskRows w;
#pragma unroll
            for (int u = 0; u < kPad; ++u) w.w[u] = n[(g * kPad + u) * kDir * M::kWords];
            return w;
        },
        [&](const MaskRows& w, int u) { return w.w[u] << sft; },
        // a value other than -1 here is a crossing value
        [](const MaskRows&, int, R o) { return o != (R)-1; });
}

// x sweep of row r from column c.
template <typename R, class M, bool kForward, bool kFlags, bool kSource>
__device__ __forceinline__ void x_sweep(M& m, int r, int c, int cnt, R h) {
    constexpr int S = kForward ? 1 : -1;
    const int i = M::at(r, c), row = (r + kPad) * M::kWords;
    // mask position of a group's lowest column
    const int low = kForward ? c + 1 + kPad : c;
    auto bits = [&](const unsigned* v, int b) {
        return __funnelshift_r(v[row + (b >> 5)], v[row + (b >> 5) + 1], b & 31);
    };
    sweep_line<R, S, kForward && kFlags, kSource>(
        m.cell + i + S, m.src + (kSource ? i + S : 0), cnt, m.cell[i], h,
        [&](int g) {
            const int b = low + g * kPad * S;
            MaskBits w{bits(m.neg, b), 0u};
            if (kForward && kFlags) w.f = bits(m.flag, b);
            return w;
        },
        [](const MaskBits& w, int u) { return w.w << (31 - (kForward ? u : kPad - 1 - u)); },
        [](const MaskBits& w, int u, R) { return (w.f >> u & 1u) != 0u; });
}

// x sweep of a row without input: the sign is the target's own.
template <typename R, class M, int kDir, bool kSource>
__device__ __forceinline__ void x_sweep_free(M& m, int r, int c, int cnt, R h) {
    R* p = m.cell + M::at(r, c);
    int* ps = m.src + (kSource ? M::at(r, c) : 0);
    R cur = *p;
    int src = kSource ? *ps : 0;
    for (int t = 0; t < cnt; ++t) {
        p += kDir;
        ps += kDir;
        const R o = *p;
        const R cand = cur + (o > (R)0 ? h : (o < (R)0 ? -h : (R)0));
        const bool in = fabs(cand) < fabs(o);
        cur = in ? cand : o;
        *p = cur;
        if constexpr (kSource) {
            if (!in) src = *ps;
            *ps = src;
        }
    }
}

// A grain's input and output of the redistancing.
template <typename R>
struct RedistGrain {
    const R* in;  // compared field, row-major over bi
    Box bi;
    R* out;  // row-major over bo
    Box bo;
    R h, delta;
    // the intersection of the two boxes, the only part of the input that is read
    int ixmin, iymin, ixmax, iymax;
    __device__ R at(int i, int j) const { return in[(int64_t)(i - bi.y0) * (bi.x1 - bi.x0) + (j - bi.x0)]; }
};

template <typename R>
__device__ RedistGrain<R> redist_grain(const NetConst& C, NetState* S, int g) {
    RedistGrain<R> G;
    G.in = phiA_of<R>(S) + S->off_cur[g];
    G.out = phiB_of<R>(S) + S->off_new[g];
    G.bi = S->box_cur[g];
    G.bo = S->box_new[g];
    G.h = (R)C.h;
    G.delta = (R)C.delta;
    G.ixmin = max(G.bi.x0, G.bo.x0);
    G.iymin = max(G.bi.y0, G.bo.y0);
    G.ixmax = min(G.bi.x1, G.bo.x1);
    G.iymax = min(G.bi.y1, G.bo.y1);
    return G;
}

template <typename R>
__device__ __forceinline__ R clamp_delta(R v, R delta) {
    return v < -delta ? -delta : (v > delta ? delta : v);
}


// The sweeps of a staged box whose crossing lists are evaluated.  The warps
// but the last take the columns and the rows with input, the last warp the
// rows below the input.
template <typename R, class M, bool kFlags, bool kSource>
__device__ __forceinline__ void staged_sweeps(const RedistGrain<R>& G, M& m, int listed) {
    const int wo = box_w(G.bo), ho = box_h(G.bo);
    const int cx = G.ixmin - G.bo.x0, cy = G.iymin - G.bo.y0, ey = G.iymax - G.bo.y0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nline = (blockDim.x >> 5) - 1;
    const R h = G.h;
    if (warp < nline)
        for (int c = cx + warp * 32 + lane; c < wo; c += 32 * nline) {
            if (cy < ho - 1) y_sweep<R, M, true, kFlags, kSource>(m, cy, c, ho - 1 - cy, h);
            if (ey - 1 > 0) y_sweep<R, M, false, kFlags, kSource>(m, ey - 1, c, ey - 1, h);
        }
    __syncthreads();
    // x crossing values into their pixels
    for (int q = lane; q < listed; q += 32) {
        const unsigned e = m.list[warp][q];
        if (!(e >> 31)) continue;
        const int r = cy + (int)((e >> 16) & 0x7fff), c = cx + (int)(e & 0xffff), p = M::at(r, c);
        const R z = m.z[warp][q];
        if (fabs(m.cell[p]) > fabs(z)) {
            m.cell[p] = z;
            if constexpr (kSource) m.src[p] = 2 * p + 1;
            if constexpr (kFlags) atomicOr(&m.flag[M::word(r, c)], 1u << ((c + kPad) & 31));
        }
    }
    __syncthreads();
    const int last = G.ixmax - 1 - G.bo.x0;
    if (warp < nline) {
        for (int r = cy + warp * 32 + lane; r < min(ey, ho); r += 32 * nline) {
            if (cx < wo - 1) x_sweep<R, M, true, kFlags, kSource>(m, r, cx, wo - 1 - cx, h);
            if (last > 0) x_sweep<R, M, false, kFlags, kSource>(m, r, last, last, h);
        }
    } else {
        for (int r = max(ey, cy) + lane; r < ho; r += 32) {
            if (cx < wo - 1) x_sweep_free<R, M, 1, kSource>(m, r, cx, wo - 1 - cx, h);
            if (last > 0) x_sweep_free<R, M, -1, kSource>(m, r, last, last, h);
        }
    }
    __syncthreads();
}

// The whole box in shared memory; all threads of the CTA call it (at least
// two warps).  Returns false, with nothing written to G.out, for a box that
// is not of the staged form (see the head of the file) or whose crossing pairs
// do not fit the lists.  With kSource the unclamped output and the sources
// stay in m for the caller (2 p for the y crossing, 2 p + 1 for the x crossing
// of the pixel at cell p, -1 for the start value); without it the clamped
// output is written to G.out.
template <typename R, class M, bool kSource>
__device__ __forceinline__ bool redistance_staged(const RedistGrain<R>& G, int nn, M& m) {
    const int wo = box_w(G.bo), ho = box_h(G.bo), wi = box_w(G.bi);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const R h = G.h;
    const int wI = max(G.ixmax - G.ixmin, 0), hI = max(G.iymax - G.iymin, 0);
    const int cx = G.ixmin - G.bo.x0, cy = G.iymin - G.bo.y0;  // the intersection's corner in the output box
    const int words = (wo + kPad + 31) >> 5;                   // mask words with columns of the box
    const bool flags = sizeof(R) == 8 || max(wo, ho) + 4 > nn;  // (see the head of the file; 4 cells of margin)
    if (threadIdx.x == 0) m.refused = 0;
    // the input's signs: two words of a row per pair of ballots, 2 kU loads in
    // flight; outside the intersection the sign is that of the start value -1,
    // which the reference takes there
    constexpr int kU = sizeof(R) == 4 ? 8 : 6;
    const R* const in = G.in + (int64_t)(G.iymin - G.bi.y0) * wi + (G.ixmin - G.bi.x0);
    bool fine = true;
    for (int w = 0; w < words; w += 2) {
        const int c = 32 * w + lane - kPad - cx;  // column of the intersection
        const bool ca = c >= 0 && c < wI, cb = c + 32 >= 0 && c + 32 < wI;
        const R* p = in + warp * wi + c;
        for (int r0 = warp; r0 < hI; r0 += kU * nwarps) {
            R a[kU], b[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const bool row = r0 + u * nwarps < hI;
                a[u] = ca && row ? p[0] : (R)-1;
                b[u] = cb && row ? p[32] : (R)-1;
                p += nwarps * wi;
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const unsigned na = __ballot_sync(0xffffffffu, a[u] < (R)0);
                const unsigned nb = __ballot_sync(0xffffffffu, b[u] < (R)0);
                fine = fine && ordinary(a[u]) && ordinary(b[u]);
                const int r = r0 + u * nwarps;
                if (lane < 2 && r < hI) m.neg[(cy + r + kPad) * M::kWords + w + lane] = lane ? nb : na;
            }
        }
    }
    for (int r = threadIdx.x; r < ho; r += blockDim.x) {
        if (r < cy || r >= cy + hI)
            for (int w = 0; w < words; ++w) m.neg[(r + kPad) * M::kWords + w] = ~0u;
        if (flags)
            for (int w = 0; w < words; ++w) m.flag[(r + kPad) * M::kWords + w] = 0u;
    }
    // start values, 16 bytes at a time
    {
        const R v[16 / sizeof(R)] = {(R)-1, (R)-1};
        uint4 four = *reinterpret_cast<const uint4*>(v);
        if (sizeof(R) == 4) four.z = four.w = four.x;
        uint4* const to = reinterpret_cast<uint4*>(m.cell);
        const int n = ((ho + 2 * kPad) * M::kStride * (int)sizeof(R)) / 16;
        for (int q = threadIdx.x; q < n; q += blockDim.x) to[q] = four;
        if constexpr (kSource)
            for (int q = threadIdx.x; q < (ho + 2 * kPad) * M::kStride; q += blockDim.x) m.src[q] = -1;
    }
    __syncthreads();
    if (!__all_sync(0xffffffffu, fine) && lane == 0) m.refused = 1;
    // the pairs with a sign change, one row per lane: y pairs with the row
    // below, x pairs with the next column
    int listed = 0;
    for (int rb = warp < M::kLists ? 32 * warp : hI; rb < hI; rb += 32 * M::kLists) {
        const int r = rb + lane;
        const unsigned* const n = m.neg + (cy + min(r, hI - 1) + kPad) * M::kWords;
        // word w's columns [0, last] of the intersection
        auto within = [&](int w, int last) {
            const int lo = cx + kPad - 32 * w, hi = cx + last + kPad - 32 * w;
            return hi < 0 || lo > 31 ? 0u : (~0u << max(lo, 0)) & (~0u >> (31 - min(hi, 31)));
        };
        constexpr int kMost = M::kWords - 1;
        unsigned y[kMost], x[kMost];
        int cnt = 0;
#pragma unroll
        for (int w = 0; w < kMost; ++w) {
            y[w] = x[w] = 0u;
            if (w < words && r < hI) {
                const unsigned v = n[w];
                if (r + 1 < hI) y[w] = (v ^ n[M::kWords + w]) & within(w, wI - 1);
                x[w] = (v ^ __funnelshift_r(v, n[w + 1], 1)) & within(w, wI - 2);
                cnt += __popc(y[w]) + __popc(x[w]);
            }
        }
        int pos = cnt;
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pos, d);
            if (lane >= d) pos += v;
        }
        const int total = __shfl_sync(0xffffffffu, pos, 31);
        pos += listed - cnt;
        listed += total;
        if (listed <= kCrossList) {
#pragma unroll
            for (int w = 0; w < kMost; ++w) {
                const unsigned at = (unsigned)(r << 16 | 32 * w) - (unsigned)(kPad + cx);
                for (; y[w]; y[w] &= y[w] - 1) m.list[warp][pos++] = at + (unsigned)(__ffs(y[w]) - 1);
                for (; x[w]; x[w] &= x[w] - 1) m.list[warp][pos++] = 0x80000000u | (at + (unsigned)(__ffs(x[w]) - 1));
            }
        }
    }
    if (listed > kCrossList) {
        if (lane == 0) m.refused = 1;
        listed = 0;
    }
    __syncwarp();
    for (int q0 = 0; q0 < listed; q0 += 64) {
        unsigned e[2];
        R a[2], c[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 32 * u + lane;
            e[u] = q < listed ? m.list[warp][q] : 0u;
            const int r = (int)((e[u] >> 16) & 0x7fff), k = r * wi + (int)(e[u] & 0xffff);
            a[u] = c[u] = (R)-1;
            if (q < listed) {
                a[u] = in[k];
                c[u] = in[e[u] >> 31 ? k + 1 : k + wi];
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 32 * u + lane;
            if (q >= listed) break;
            const R z = crossing_value(a[u], c[u], h);
            if (e[u] >> 31) {
                m.z[warp][q] = z;
            } else if (fabs(z) < (R)1) {
                const int p = M::at(cy + (int)((e[u] >> 16) & 0x7fff), cx + (int)(e[u] & 0xffff));
                m.cell[p] = z;
                if constexpr (kSource) m.src[p] = 2 * p;
            }
        }
    }
    __syncthreads();
    if (m.refused) return false;
    if (sizeof(R) == 4 && !flags)
        staged_sweeps<R, M, false, kSource>(G, m, listed);
    else
        staged_sweeps<R, M, true, kSource>(G, m, listed);
    if constexpr (!kSource)
        for (int r0 = warp; r0 < ho; r0 += 4 * nwarps)  // four rows' loads in flight
            for (int c = lane; c < wo; c += 32) {
                R v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = m.cell[M::at(min(r0 + u * nwarps, ho - 1), c)];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (r0 + u * nwarps < ho) G.out[(r0 + u * nwarps) * wo + c] = clamp_delta(v[u], G.delta);
            }
    return true;
}

// Shared memory of redistance_strips: a 32 x 33 tile and its masks per warp.
template <typename R>
__host__ __device__ constexpr size_t redist_strip_bytes(int threads) {
    return (size_t)(threads / 32) * (32 * 33 * sizeof(R) + 96 * 4);
}

// A box that does not fit shared memory: the output stays in device memory.
// The y sweeps stream the columns (coalesced, eight rows ahead); the x sweeps
// take 32 rows per warp through 32 x 32 tiles in shared memory.
template <typename R>
__device__ __noinline__ void redistance_strips(const RedistGrain<R>& G, unsigned char* smem) {
    const int wo = box_w(G.bo), ho = box_h(G.bo), wi = box_w(G.bi);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const R h = G.h, delta = G.delta;
    const int cx = G.ixmin - G.bo.x0, cy = G.iymin - G.bo.y0;
    const int ex = G.ixmax - G.bo.x0, ey = G.iymax - G.bo.y0;  // one past the intersection, in the output box
    const R* const in = G.in + (int64_t)(G.bo.y0 - G.bi.y0) * wi + (G.bo.x0 - G.bi.x0);  // at the output box's corner
    constexpr int kU = 8;
    for (int c = threadIdx.x; c < wo; c += blockDim.x) {
        R* const col = G.out + c;
        if (c < cx) {  // no y sweep there
            for (int r = 0; r < ho; ++r) col[(int64_t)r * wo] = r < cy ? clamp_delta((R)-1, delta) : (R)-1;
            continue;
        }
        const bool given = c < ex;
        const R* const ic = in + c;
        auto load = [&](int r) { return given && r >= cy && r < ey ? ic[(int64_t)r * wi] : (R)-1; };
        if (cy < ho) {
            // v0: input of the target row, then the row after it
            R v[kU + 1], vn[kU];
#pragma unroll
            for (int u = 0; u <= kU; ++u) v[u] = load(cy + u);
            R cur = (R)0;
            for (int r0 = cy; r0 < ho; r0 += kU) {
#pragma unroll
                for (int u = 0; u < kU; ++u) vn[u] = load(r0 + kU + 1 + u);
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int r = r0 + u;
                    if (r >= ho) break;
                    R V = (R)-1;
                    if (given && r < ey - 1 && v[u] * v[u + 1] <= (R)0) {
                        const R z = crossing_value(v[u], v[u + 1], h);
                        if (fabs(z) < (R)1) V = z;
                    }
                    if (r == cy) {
                        cur = V;
                    } else {
                        const R cand = cur + (R)sgn(v[u]) * h;
                        if (takes(cand, V, V != (R)-1)) cur = cand;
                        else cur = V;
                    }
                    col[(int64_t)r * wo] = cur;
                }
                v[0] = v[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) v[u + 1] = vn[u];
            }
        }
        // backward; rows above the intersection are final after it
        if (ey - 1 > 0) {
            auto out_at = [&](int r) { return r >= cy && r < ho ? col[(int64_t)r * wo] : (R)-1; };
            R cur = out_at(ey - 1);
            R o[kU], v[kU], on[kU], vn[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                o[u] = ey - 2 - u >= 0 ? out_at(ey - 2 - u) : (R)0;
                v[u] = load(ey - 2 - u);
            }
            for (int r0 = ey - 2; r0 >= 0; r0 -= kU) {
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    on[u] = r0 - kU - u >= 0 ? out_at(r0 - kU - u) : (R)0;
                    vn[u] = load(r0 - kU - u);
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int r = r0 - u;
                    if (r < 0) break;
                    const R cand = cur + (R)sgn(v[u]) * h;
                    cur = fabs(cand) < fabs(o[u]) ? cand : o[u];
                    col[(int64_t)r * wo] = r < cy ? clamp_delta(cur, delta) : cur;
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    o[u] = on[u];
                    v[u] = vn[u];
                }
            }
        }
        // rows above the intersection that the sweep did not reach
        for (int r = max(ey - 1, 0); r < min(cy, ho); ++r) col[(int64_t)r * wo] = clamp_delta((R)-1, delta);
    }
    __syncthreads();
    R* const to = reinterpret_cast<R*>(smem) + warp * 32 * 33;  // output tile [row][column]
    unsigned* const masks = reinterpret_cast<unsigned*>(reinterpret_cast<R*>(smem) + nwarps * 32 * 33) + warp * 96;
    // rows r0 .. r0 + 31, columns c0 .. c0 + cnt - 1 into the tile, with their
    // masks; the x crossing values go in only for the forward sweep
    auto fill = [&](int r0, int c0, int cnt, bool forward) {
        const int c = c0 + lane;
        for (int u0 = 0; u0 < 32; u0 += kU) {
            R o[kU], a[kU], b[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int r = r0 + u0 + u;
                const bool ok = r < ho && lane < cnt, given = ok && r < ey && c >= cx && c < ex;
                o[u] = ok ? G.out[(int64_t)r * wo + c] : (R)0;
                a[u] = given ? in[(int64_t)r * wi + c] : (R)-1;
                b[u] = forward && given && c + 1 < ex ? in[(int64_t)r * wi + c + 1] : (R)-1;
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int r = r0 + u0 + u;
                bool flag = false;
                if (forward && r < ey && c >= cx && c + 1 < ex && a[u] * b[u] <= (R)0) {
                    const R z = crossing_value(a[u], b[u], h);
                    flag = fabs(o[u]) > fabs(z);
                    if (flag) o[u] = z;
                }
                to[(u0 + u) * 33 + lane] = o[u];
                const unsigned nb = __ballot_sync(0xffffffffu, a[u] < (R)0);
                const unsigned zb = __ballot_sync(0xffffffffu, !(a[u] < (R)0) && !(a[u] > (R)0));
                const unsigned fb = __ballot_sync(0xffffffffu, flag);
                if (lane == 0) {
                    masks[u0 + u] = nb;
                    masks[32 + u0 + u] = zb;
                    masks[64 + u0 + u] = fb;
                }
            }
        }
        __syncwarp();
    };
    for (int r0 = cy + 32 * warp; r0 < ho; r0 += 32 * nwarps) {
        const int rows = min(32, ho - r0);
        const bool free = r0 + lane >= ey;  // a row without input takes the target's own sign
        R* const mo = to + lane * 33;
        auto step_of = [&](int k, R o) {
            if (free) return (R)sgn(o) * h;
            return masks[32 + lane] >> k & 1u ? (R)0 : signed_by(h, masks[lane] << (31 - k));
        };
        R cur = (R)0;
        if (cx < wo - 1) {
            for (int c0 = cx; c0 < wo; c0 += 32) {
                const int cnt = min(32, wo - c0);
                fill(r0, c0, cnt, true);
                if (lane < rows)
                    for (int k = 0; k < cnt; ++k) {
                        const R o = mo[k];
                        const R cand = cur + step_of(k, o);
                        cur = c0 + k > cx && takes(cand, o, masks[64 + lane] >> k & 1u) ? cand : o;
                        mo[k] = cur;
                    }
                __syncwarp();
                for (int u = 0; u < rows; ++u)
                    if (lane < cnt) G.out[(int64_t)(r0 + u) * wo + c0 + lane] = to[u * 33 + lane];
                __syncwarp();
            }
        }
        for (int c1 = wo; c1 > 0; c1 -= 32) {
            const int c0 = max(0, c1 - 32), cnt = c1 - c0;
            fill(r0, c0, cnt, false);
            if (lane < rows && ex - 1 > 0)
                for (int k = min(cnt, ex - c0) - 1; k >= 0; --k) {
                    const R o = mo[k];
                    const R cand = cur + step_of(k, o);
                    cur = c0 + k < ex - 1 && fabs(cand) < fabs(o) ? cand : o;
                    mo[k] = cur;
                }
            __syncwarp();
            for (int u = 0; u < rows; ++u)
                if (lane < cnt) G.out[(int64_t)(r0 + u) * wo + c0 + lane] = clamp_delta(to[u * 33 + lane], delta);
            __syncwarp();
        }
    }
}

// Launches.  Boxes of ordinary size take three warps (two for the lines, one
// for the rows below the input) and just the shared memory they need, so that
// many share an SM; the larger ones take more of both.
constexpr int kRedistEdge = 64;  // largest box edge of the first kind
constexpr int kRedistThreads = 96;
template <typename R>
struct RedistLarge;
template <>
struct RedistLarge<float> {
    static constexpr int kEdge = 144, kThreads = 192, kPerSm = 2;
};
template <>
struct RedistLarge<double> {
    static constexpr int kEdge = 150, kThreads = 192, kPerSm = 1;
};
template <typename R, bool kLarge>
__host__ __device__ constexpr int redist_edge() { return kLarge ? RedistLarge<R>::kEdge : kRedistEdge; }
template <typename R, bool kLarge>
__host__ __device__ constexpr int redist_threads() { return kLarge ? RedistLarge<R>::kThreads : kRedistThreads; }
template <typename R, bool kLarge>
using RedistCta = RedistSmem<R, redist_edge<R, kLarge>(), redist_threads<R, kLarge>(), false>;
template <typename R, bool kLarge>
constexpr size_t redist_smem() {
    const size_t a = sizeof(RedistCta<R, kLarge>), b = redist_strip_bytes<R>(redist_threads<R, kLarge>());
    return a > b ? a : b;
}
static_assert(redist_smem<float, false>() <= 28 * 1024);   // 8 CTAs per SM
static_assert(redist_smem<double, false>() <= 56 * 1024);  // 4
static_assert(redist_smem<float, true>() <= 113 * 1024);   // 2
static_assert(redist_smem<double, true>() <= 226 * 1024);  // 1

// Grain g by the whole CTA.
template <typename R, bool kLarge>
__device__ __forceinline__ void redistance_grain(const NetConst& C, NetState* S, int g, unsigned char* smem) {
    const RedistGrain<R> G = redist_grain<R>(C, S, g);
    using M = RedistCta<R, kLarge>;
    if (max(box_w(G.bo), box_h(G.bo)) > redist_edge<R, kLarge>() ||
        !redistance_staged<R, M, false>(G, C.nn, *reinterpret_cast<M*>(smem)))
        redistance_strips<R>(G, smem);
}

// CTA per grain.  With a work queue (batched form) k_redistance<R, false> takes
// the boxes up to C.big_edge; without (plain form) the two launches split at
// kRedistEdge.
template <typename R, bool kLarge>
__global__ void __launch_bounds__(redist_threads<R, kLarge>(), kLarge ? 1 : (sizeof(R) == 4 ? 8 : 4))
    k_redistance(NetConst C, NetState* S) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int g = grain_at(S, blockIdx.x);
    if (g > C.N || C.state[g] != G_EXISTS || halted(S)) return;
    if (S->order) {
        if (box_w(S->box_cur[g]) > C.big_edge) return;  // the large-box bin
    } else {
        const Box bo = S->box_new[g];
        if ((max(box_w(bo), box_h(bo)) > kRedistEdge) != kLarge) return;
    }
    redistance_grain<R, kLarge>(C, S, g, s_raw);
}

}  // namespace
}  // namespace gg
