// Warp-per-grain versions of the per-grain sequential stages (level set,
// volume/energy/neighbours, second-order lists).  The parts of each
// reference routine that are independent per pixel, per contour point or per
// list entry run across the 32 lanes; every order-dependent part keeps the
// reference's order, so the FP64 form stays bit-identical: the marching-squares
// walk is put together from pieces, and sums add their terms one by one (the
// batched form's by trees).
#pragma once

#include "gg_grain.cuh"
#include "gg_kernels.cuh"

namespace gg {
namespace {  // internal linkage: each form's translation unit has its own copy

constexpr int kGrainsPerBlock = 4;  // warps (grains) per CTA of the warp kernels

__device__ __forceinline__ int warp_min_i(int v) {
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// First pixel of the box (row-major) with phi >= 0, as the scan of
// generateContour (src/marchingSquares.cpp:32-42); -1 if none.
template <typename R>
__device__ int first_inside_warp(const Field<R>& f, int lane) {
    const int w = box_w(f.b), h = box_h(f.b);
    for (int r = 0; r < h; ++r) {
        int best = 0x7fffffff;
        for (int c = lane; c < w; c += 32)
            if ((double)f.v[r * w + c] >= 0) {
                best = c;
                break;
            }
        best = warp_min_i(best);
        if (best != 0x7fffffff) return r * w + best;
    }
    return -1;
}

// Marching-squares walk from a known start pixel (src/marchingSquares.cpp:44-187).
// The four corner values of the current square are kept in registers and
// only the two corners a move uncovers are loaded; the last emitted point
// is kept in registers for insertPoint's duplicate test; junction corners
// are only read where a junction is possible (at most two inside corners).
template <typename R>
__device__ void ms_walk(const Field<R>& f, const uint32_t* idl, uint32_t own, int startX, int startY,
                        ContourOut& o, double2* xy) {
    o.n = 0;
    o.jn = 0;
    const Box b = f.b;
    const int w = b.x1 - b.x0;
    auto val = [&](int row, int col, double* v) -> bool {  // value and isInside
        if (row < b.y0 || row >= b.y1 || col < b.x0 || col >= b.x1) {
            *v = -1.0;
            return false;
        }
        *v = (double)f.v[(row - b.y0) * w + (col - b.x0)];
        return *v >= 0;
    };
    int left = startX - 1, right = startX, top = startY - 1, bottom = startY;
    double vTL, vTR, vBL, vBR;
    bool iTL = val(top, left, &vTL), iTR = val(top, right, &vTR);
    bool iBL = val(bottom, left, &vBL), iBR = val(bottom, right, &vBR);
    int next = MS_NONE, prev = MS_NONE;
    double lastx = 0, lasty = 0, firstx = 0, firsty = 0;
    const long limit = 4L * (w + 2) * (box_h(b) + 2) + 16;
    long it = 0;
    do {
        int mask = 0;
        if (iTL) mask |= C_TL;
        if (iTR) mask |= C_TR;
        if (iBL) mask |= C_BL;
        if (iBR) mask |= C_BR;
        bool emit = true;
        switch (mask) {
            case C_TL: next = MS_UP; break;
            case C_TR: next = MS_RIGHT; break;
            case C_TL | C_TR: next = MS_RIGHT; break;
            case C_BL: next = MS_LEFT; break;
            case C_BL | C_TL: next = MS_UP; break;
            case C_BL | C_TR:
                next = (prev == MS_UP) ? MS_RIGHT : MS_LEFT;
                emit = false;
                break;
            case C_BL | C_TR | C_TL: next = MS_RIGHT; break;
            case C_BR: next = MS_DOWN; break;
            case C_BR | C_TL:
                next = (prev == MS_RIGHT) ? MS_DOWN : MS_UP;
                emit = false;
                break;
            case C_BR | C_TR: next = MS_DOWN; break;
            case C_BR | C_TR | C_TL: next = MS_DOWN; break;
            case C_BR | C_BL: next = MS_LEFT; break;
            case C_BR | C_BL | C_TL: next = MS_UP; break;
            case C_BR | C_BL | C_TR: next = MS_LEFT; break;
            default: emit = false; break;
        }
        if (emit) {  // generatePoint (src/marchingSquares.cpp:204-265) on the cached corners
            double px, py, delta, position;
            switch (next) {
                case MS_LEFT:
                    px = left;
                    if (top < b.y0) {
                        py = bottom;
                    } else {
                        delta = vBL - vTL;
                        position = bottom - vBL / delta;
                        py = position;
                    }
                    break;
                case MS_RIGHT:
                    px = right;
                    if (bottom >= b.y1) {
                        py = top;
                    } else {
                        delta = vTR - vBR;
                        position = top + vTR / delta;
                        py = position;
                    }
                    break;
                case MS_UP:
                    py = top;
                    if (right >= b.x1) {
                        px = left;
                    } else {
                        delta = vTL - vTR;
                        position = left + vTL / delta;
                        px = position;
                    }
                    break;
                default:
                    py = bottom;
                    if (left < b.x0) {
                        px = right;
                    } else {
                        delta = vBR - vBL;
                        position = right - vBR / delta;
                        px = position;
                    }
                    break;
            }
            if (o.n == 0 || px != lastx || py != lasty) {  // insertPoint
                if (o.n >= o.cap) {
                    o.status |= S_CONTOUR_OVERFLOW;
                } else {
                    if (xy) {
                        xy[o.n] = make_double2(px, py);
                    } else {
                        CPoint& q = o.pts[o.n];
                        q.x = px;
                        q.y = py;
                        q.energy = -1.0;
                        q.mob = -1.0;
                    }
                    if (o.n == 0) {
                        firstx = px;
                        firsty = py;
                    }
                    o.n++;
                    lastx = px;
                    lasty = py;
                }
            }
        }
        if (__popc(mask) < 3) ms_junction(f, idl, own, mask, top, bottom, left, right, o);
        switch (next) {
            case MS_UP:
                top--;
                bottom--;
                vBL = vTL;
                vBR = vTR;
                iBL = iTL;
                iBR = iTR;
                iTL = val(top, left, &vTL);
                iTR = val(top, right, &vTR);
                break;
            case MS_DOWN:
                top++;
                bottom++;
                vTL = vBL;
                vTR = vBR;
                iTL = iBL;
                iTR = iBR;
                iBL = val(bottom, left, &vBL);
                iBR = val(bottom, right, &vBR);
                break;
            case MS_LEFT:
                left--;
                right--;
                vTR = vTL;
                vBR = vBL;
                iTR = iTL;
                iBR = iBL;
                iTL = val(top, left, &vTL);
                iBL = val(bottom, left, &vBL);
                break;
            case MS_RIGHT:
                left++;
                right++;
                vTL = vTR;
                vBL = vBR;
                iTL = iTR;
                iBL = iBR;
                iTR = val(top, right, &vTR);
                iBR = val(bottom, right, &vBR);
                break;
            default: break;
        }
        prev = next;
        if (++it > limit) {
            o.status |= S_WALK_LIMIT;
            break;
        }
    } while (left != startX - 1 || bottom != startY);
    if (o.n > 0 && (firstx != lastx || firsty != lasty)) {
        if (o.n >= o.cap) {
            o.status |= S_CONTOUR_OVERFLOW;
        } else {
            if (xy)
                xy[o.n] = make_double2(firstx, firsty);
            else
                o.pts[o.n] = o.pts[0];
            o.n++;
        }
    }
}

// Contour routines over a shared-memory (x, y) buffer: the same operations
// as project_to_boundary, contour_volume, contour_perimeter and
// clear_contour_area on CPoint arrays (src/grainBoundary.cpp:201-231, 365-447,
// src/box.cpp:1888-1906).  The projection starts from the nearest vertex
// (nearest_xy; -1 if none lies within the reference's initial distance).
__device__ int project_xy(const double2* P, int asize, double px, double py, int nearest, double* out_lambda) {
    double lam_out = *out_lambda;
    if (nearest < 0) return 0;
    int minimal_segment = nearest;
    double dist = 0, minDist = 1000000.0;
    int next = nearest + 1;
    double ux = P[next].x - P[nearest].x, uy = P[next].y - P[nearest].y;
    double lambda = (px - P[nearest].x) * ux + (py - P[nearest].y) * uy;
    lambda /= (ux * ux + uy * uy);
    if (lambda < 0)
        dist = len_sqr(px - P[nearest].x, py - P[nearest].y);
    else if (lambda > 1)
        dist = len_sqr(P[next].x - px, P[next].y - py);
    else
        dist = len_sqr(px - (P[nearest].x + ux * lambda), py - (P[nearest].y + uy * lambda));
    if (dist < minDist) {
        minimal_segment = nearest;
        minDist = dist;
        lam_out = lambda;
    }
    if (nearest == 0) nearest = asize - 1;
    int previous = nearest - 1;
    ux = P[nearest].x - P[previous].x;
    uy = P[nearest].y - P[previous].y;
    lambda = (px - P[previous].x) * ux + (py - P[previous].y) * uy;
    lambda /= (ux * ux + uy * uy);
    if (lambda < 0)
        dist = len_sqr(px - P[previous].x, py - P[previous].y);
    else if (lambda > 1)
        dist = len_sqr(P[nearest].x - px, P[nearest].y - py);
    else
        dist = len_sqr(px - (P[previous].x + ux * lambda), py - (P[previous].y + uy * lambda));
    if (dist < minDist) {
        minimal_segment = previous;
        minDist = dist;
        lam_out = lambda;
    }
    if (lam_out > 1) lam_out = 1;
    if (lam_out < 0) lam_out = 0;
    *out_lambda = lam_out;
    return minimal_segment;
}

// The nearest of the vertices 0 .. asize-2 to (px, py), the first one at equal
// distance (the reference's strict < over ascending k), by groups of four
// lanes: every lane of a group returns it.  All 32 lanes call it.
__device__ __forceinline__ int nearest_xy(const double2* P, int asize, double px, double py) {
    const int lane = threadIdx.x & 31;
    double best = 1000000.0;
    int nearest = INT_MAX;
    for (int k = lane & 3; k < asize - 1; k += 4) {
        const double dist = len_sqr(px - P[k].x, py - P[k].y);
        if (dist < best) {
            best = dist;
            nearest = k;
        }
    }
    for (int o = 1; o < 4; o <<= 1) {
        const double d = __shfl_xor_sync(0xffffffffu, best, o);
        const int k = __shfl_xor_sync(0xffffffffu, nearest, o);
        if (d < best || (d == best && k < nearest)) {
            best = d;
            nearest = k;
        }
    }
    return nearest == INT_MAX ? -1 : nearest;
}

// The junctions projected onto the contour (extractBoundaryAndJunctions,
// src/grainBoundary.cpp:51-61), eight at a time.
__device__ __forceinline__ void project_junctions(const double2* xy, const ContourOut& o, int lane) {
    for (int j0 = 0; j0 < o.jn; j0 += 8) {
        const int j = j0 + (lane >> 2);
        const bool busy = j < o.jn;
        const double jx = busy ? o.js[j].x : 0, jy = busy ? o.js[j].y : 0;
        const int nearest = nearest_xy(xy, o.n, jx, jy);
        if (!busy || (lane & 3) != 0) continue;
        double lambda = 0.0;
        const int seg = project_xy(xy, o.n, jx, jy, nearest, &lambda);
        const int nx = periodic(seg + 1, o.n);
        o.js[j].x = xy[seg].x + (xy[nx].x - xy[seg].x) * lambda;
        o.js[j].y = xy[seg].y + (xy[nx].y - xy[seg].y) * lambda;
        o.js[j].segment = seg;
        o.js[j].lambda = lambda;
    }
}

// ExplicitGrainBoundary::computeVolume / computePerimeter
// (src/grainBoundary.cpp:201-213, 224-231) by the whole warp: lanes evaluate
// the per-segment terms side by side, then the terms are added one after the
// other in contour order (every lane holds the same sum, rounded exactly as
// the reference's loop).
__device__ __forceinline__ double volume_xy(const double2* P, int n, double h) {
    const int lane = threadIdx.x & 31;
    double v = 0;
    for (int i0 = 0; i0 < n - 1; i0 += 32) {
        const int i = i0 + lane;
        double t = 0;
        if (i < n - 1) t = (P[i].y + P[i + 1].y) * (P[i].x - P[i + 1].x);
        const int m = n - 1 - i0 < 32 ? n - 1 - i0 : 32;
        for (int q = 0; q < m; ++q) v += __shfl_sync(0xffffffffu, t, q);
    }
    return fabs(v) * h * h * 0.5;
}

__device__ __forceinline__ double perimeter_xy(const double2* P, int n, double h) {
    const int lane = threadIdx.x & 31;
    double p = 0;
    for (int i0 = 0; i0 < n - 1; i0 += 32) {
        const int i = i0 + lane;
        double t = 0;
        if (i < n - 1) {
            const double dx = P[i].x - P[i + 1].x, dy = P[i].y - P[i + 1].y;
            t = sqrt(dx * dx + dy * dy) * h;
        }
        const int m = n - 1 - i0 < 32 ? n - 1 - i0 : 32;
        for (int q = 0; q < m; ++q) p += __shfl_sync(0xffffffffu, t, q);
    }
    return p;
}

// The same two sums for the batched form, whose areas and perimeters need
// not round as the reference's loop does: each lane adds its own terms, then
// a tree to lane 0, broadcast (every lane holds the same bits).
__device__ __forceinline__ double warp_sum_to_all(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);
}

__device__ __forceinline__ double volume_xy_tree(const double2* P, int n, double h) {
    double v = 0;
    for (int i = threadIdx.x & 31; i < n - 1; i += 32) v += (P[i].y + P[i + 1].y) * (P[i].x - P[i + 1].x);
    return fabs(warp_sum_to_all(v)) * h * h * 0.5;
}

__device__ __forceinline__ double perimeter_xy_tree(const double2* P, int n, double h) {
    double p = 0;
    for (int i = threadIdx.x & 31; i < n - 1; i += 32) {
        const double dx = P[i].x - P[i + 1].x, dy = P[i].y - P[i + 1].y;
        p += sqrt(dx * dx + dy * dy) * h;
    }
    return warp_sum_to_all(p);
}

// The level set's sums in the form's rounding: the reference's order in
// FP64 (plain), the tree in the batched form.
template <typename R>
__device__ __forceinline__ double form_volume(const double2* P, int n, double h) {
    if constexpr (sizeof(R) == 4) return volume_xy_tree(P, n, h);
    else return volume_xy(P, n, h);
}
template <typename R>
__device__ __forceinline__ double form_perimeter(const double2* P, int n, double h) {
    if constexpr (sizeof(R) == 4) return perimeter_xy_tree(P, n, h);
    else return perimeter_xy(P, n, h);
}

// LSbox::clearContourGrainArea (src/box.cpp:1888-1906) by the whole warp (every
// pixel's test and write are its own).
template <typename R>
__device__ bool clear_area_xy(R* phi, const Box& b, const double2* P, int n, double h) {
    if (n == 0) return true;
    const int lane = threadIdx.x & 31;
    double minx = P[0].x, maxx = P[0].x, miny = P[0].y, maxy = P[0].y;
    for (int i = lane; i < n; i += 32) {
        minx = fmin(minx, P[i].x);
        maxx = fmax(maxx, P[i].x);
        miny = fmin(miny, P[i].y);
        maxy = fmax(maxy, P[i].y);
    }
    for (int o = 16; o > 0; o >>= 1) {
        minx = fmin(minx, __shfl_xor_sync(0xffffffffu, minx, o));
        maxx = fmax(maxx, __shfl_xor_sync(0xffffffffu, maxx, o));
        miny = fmin(miny, __shfl_xor_sync(0xffffffffu, miny, o));
        maxy = fmax(maxy, __shfl_xor_sync(0xffffffffu, maxy, o));
    }
    bool ok = true;
    for (int i = (int)(miny - 1); i < maxy + 1; i++)
        for (int j = (int)(minx - 1) + lane; j < maxx + 1; j += 32) {
            uint32_t k;
            if (!buf_index(b, i, j, &k)) {
                ok = false;
                continue;
            }
            if ((double)phi[k] >= 0) phi[k] = (R)(-h);
        }
    return __all_sync(0xffffffffu, ok);
}

// Shared buffers of one warp's contour extraction: the padded bitmap of the
// box, the recorded walk steps, the contour points (before them, the starts and
// pieces of walk_parallel).  Boxes up to 97 cells take the small ones, four
// warps to a CTA; larger ones (to 222 cells) a CTA of one warp with the large
// ones, beside them.  What fits neither is walked by one lane in device memory,
// which takes some 250 us for a box of 100 cells.  (Smaller buffers at seven CTAs
// per SM instead of five take 20,000 grains in 253 us instead of 276, but their 72
// registers spill, and 1,000 grains take 85 us instead of 63.)
template <int kBitmapWords, int kSteps, int kPoints>
struct WalkBuffers {
    static constexpr int kBitmap = kBitmapWords, kTrace = kSteps, kPts = kPoints;
    double2 xy[kPoints];
    uint32_t bm[kBitmapWords];
    uint16_t trace[kSteps];
};
using SmallWalk = WalkBuffers<400, 768, 448>;
using LargeWalk = WalkBuffers<1570, 2048, 1024>;

// Whether a box's padded bitmap fits.
template <class W>
__device__ __forceinline__ bool walk_fits(const Box& b) {
    const int w = box_w(b), hgt = box_h(b), wpr = (w + 2 + 31) >> 5;
    return w + 2 <= 1024 && (hgt + 2) * wpr + 1 <= W::kBitmap && (hgt + 1) * (w + 1) <= 65535;
}

template <class W, typename R>
__device__ int extract_bitmap_warp(const Field<R>& f, const uint32_t* idl, uint32_t own, ContourOut& o, int lane, W& ws);

// Contour + junctions of one grain by one warp; returns false if no pixel
// has phi >= 0.  The walk writes into the warp's shared buffer xy (or, for a
// contour longer than the buffer, directly into the global contour);
// junctions are projected by four lanes each (one where the points are not in
// shared memory).  On return *in_shared says where the points are.
template <class W, typename R>
__device__ bool extract_warp(const Field<R>& f, const uint32_t* idl, uint32_t own, ContourOut& o, int lane, W& ws,
                             bool* in_shared) {
    double2* const xy = ws.xy;
    {
        const uint32_t st0 = o.status;
        const int r = extract_bitmap_warp(f, idl, own, o, lane, ws);
        if (r >= 0) {
            *in_shared = true;
            return r == 1;
        }
        o.status = st0;  // does not fit the shared buffers: walk in global memory
        o.jn = 0;
    }
    const int start = first_inside_warp(f, lane);
    if (start < 0) {
        o.n = 0;
        o.jn = 0;
        return false;
    }
    const int w = box_w(f.b);
    const int gcap = o.cap;
    bool shared = true;
    if (lane == 0) {
        o.cap = gcap < W::kPts ? gcap : W::kPts;
        ms_walk(f, idl, own, f.b.x0 + start % w, f.b.y0 + start / w, o, xy);
        if ((o.status & S_CONTOUR_OVERFLOW) && gcap > W::kPts) {  // long contour: walk again into global memory
            o.status &= ~S_CONTOUR_OVERFLOW;
            o.cap = gcap;
            ms_walk(f, idl, own, f.b.x0 + start % w, f.b.y0 + start / w, o, (double2*)nullptr);
            shared = false;
        }
        o.cap = gcap;
    }
    shared = __shfl_sync(0xffffffffu, shared, 0);
    o.n = __shfl_sync(0xffffffffu, o.n, 0);
    o.jn = __shfl_sync(0xffffffffu, o.jn, 0);
    o.status = __shfl_sync(0xffffffffu, o.status, 0);
    __syncwarp();
    if (o.n >= 2 && shared) project_junctions(xy, o, lane);
    if (o.n >= 2 && !shared) {
        for (int j = lane; j < o.jn; j += 32) {
            double lambda = 0.0;
            const int seg = project_to_boundary(o.pts, o.n, o.js[j].x, o.js[j].y, &lambda);
            const int nx = periodic(seg + 1, o.n);
            o.js[j].x = o.pts[seg].x + (o.pts[nx].x - o.pts[seg].x) * lambda;
            o.js[j].y = o.pts[seg].y + (o.pts[nx].y - o.pts[seg].y) * lambda;
            o.js[j].segment = seg;
            o.js[j].lambda = lambda;
        }
    }
    __syncwarp();
    *in_shared = shared;
    return true;
}

// Corner mask of the marching-squares cell whose top-left pixel is at padded
// row tr, padded column lc (C_TL | C_TR from row tr, C_BL | C_BR from tr + 1).
__device__ __forceinline__ int cell_mask(const uint32_t* bm, int wpr, int tr, int lc) {
    const uint32_t* rt = bm + tr * wpr + (lc >> 5);
    const int sh = lc & 31;
    const uint32_t top2 = __funnelshift_r(rt[0], rt[1], sh);
    const uint32_t bot2 = __funnelshift_r(rt[wpr], rt[wpr + 1], sh);
    return (int)((top2 & 3u) | ((bot2 & 3u) << 2));
}

// Next direction of generateContour's switch for each corner mask
// (src/marchingSquares.cpp:64-154), two bits per mask; the saddles 6 and 9
// and the empty / full masks 0 and 15 are decided separately.
constexpr uint32_t ms_next_bits() {
    const int dir[16] = {0, MS_UP, MS_RIGHT, MS_RIGHT, MS_LEFT, MS_UP, 0, MS_RIGHT,
                         MS_DOWN, 0, MS_DOWN, MS_DOWN, MS_LEFT, MS_UP, MS_LEFT, 0};
    uint32_t t = 0;
    for (int m = 0; m < 16; ++m) t |= (uint32_t)dir[m] << (2 * m);
    return t;
}
constexpr uint32_t kMsNext = ms_next_bits();
// masks whose case generates a point (all but 0, 6, 9, 15)
constexpr uint32_t kMsEmit = 0xFFFFu & ~((1u << 0) | (1u << 6) | (1u << 9) | (1u << 15));

// One step of generateContour's walk (src/marchingSquares.cpp:44-187) on the
// bitmap, in padded coordinates lc = left - x0 + 1, tr = top - y0 + 1; `dir` is
// the last step's direction.  The switch of the reference is evaluated as
// selects, so a step has no branch.
__device__ __forceinline__ int walk_dir(int mask, int dir) {
    const int tab = (int)((kMsNext >> (2 * mask)) & 3u);
    const int s6 = dir == MS_UP ? MS_RIGHT : MS_LEFT;
    const int s9 = dir == MS_RIGHT ? MS_DOWN : MS_UP;
    return mask == (C_BL | C_TR) ? s6 : mask == (C_BR | C_TL) ? s9 : (mask == 0 || mask == 15) ? dir : tab;
}

// The whole walk from cell (tr0, lc0) by one lane: records the cell index
// tr * cw + lc of every step (the step's direction is recovered later from the
// next recorded cell).  Returns the steps, -1 if they exceed the trace buffer.
template <class W>
__device__ int walk_serial(W& ws, int wpr, int cw, int hgt, int tr0, int lc0, uint32_t* status) {
    const int limit = 4 * (cw + 1) * (hgt + 2) + 16;
    int lc = lc0, tr = tr0, dir = MS_NONE, nsteps = 0;
    do {
        dir = walk_dir(cell_mask(ws.bm, wpr, tr, lc), dir);
        ws.trace[nsteps] = (uint16_t)(tr * cw + lc);
        ++nsteps;
        lc += (dir == MS_RIGHT) - (dir == MS_LEFT);
        tr += (dir == MS_DOWN) - (dir == MS_UP);
        if (nsteps >= W::kTrace || nsteps > limit) break;
    } while (lc != lc0 || tr != tr0);
    if (lc != lc0 || tr != tr0) {
        if (nsteps >= W::kTrace) return -1;
        *status |= S_WALK_LIMIT;
    }
    return nsteps;
}

// The same walk by the warp.  Away from the saddles a cell's step does not
// depend on how it was reached, so the walk from any such cell on the contour is
// a piece of the whole one: lane 0 starts at (tr0, lc0), the others at the first
// and the last boundary cell of 16 rows spread over the grain, each walks until
// it meets a start, and the pieces are strung together from lane 0's until one
// ends at (tr0, lc0).  Pieces of other contours in the box are left out.  A step
// is a chain of some 110 cycles and 40 instructions, so 130 steps of one lane
// were two fifths of the level set's instructions; the longest piece has about
// 15.  The starts' bitmap and the pieces lie in the points' buffer, which is
// still unused.  Returns the steps, now in ws.trace, -1 if they exceed it, and
// 0 if a piece does not fit its buffer or the pieces do not close (the caller
// then walks with one lane).
template <class W>
__device__ __forceinline__ int walk_parallel(W& ws, int wpr, int cw, int hgt, int tr0, int lc0, int row_first,
                                             int row_last, int lane) {
    const unsigned FULL = 0xffffffffu;
    constexpr int kPiece = (int)((sizeof(ws.xy) - 4 * W::kBitmap) / (2 * 32));
    static_assert(kPiece >= 64, "room for a piece of the walk per lane");
    uint32_t* const starts = reinterpret_cast<uint32_t*>(ws.xy);
    uint16_t* const piece = reinterpret_cast<uint16_t*>(starts + W::kBitmap) + lane * kPiece;
    for (int q = lane; q < (hgt + 2) * wpr + 1; q += 32) starts[q] = 0u;
    int tr = tr0, lc = lc0;
    bool active = true;
    if (lane != 0) {
        tr = 1 + row_first + (row_last - row_first) * (lane >> 1) / 15;  // the row of the cell's upper corners
        const uint32_t* row = ws.bm + tr * wpr;
        lc = -1;
        for (int q = 0; q < wpr; ++q) {
            const uint32_t word = row[q];
            if (word == 0u) continue;
            if (lane & 1)
                lc = 32 * q + 31 - __clz(word);  // the last inside pixel is its upper left corner
            else if (lc < 0)
                lc = 32 * q + __ffs(word) - 2;  // the first inside pixel is its upper right corner
        }
        active = lc >= 0;
        if (active) {
            const int mask = cell_mask(ws.bm, wpr, tr, lc);
            active = mask != (C_BL | C_TR) && mask != (C_BR | C_TL);
        }
    }
    __syncwarp();
    if (active) atomicOr(&starts[tr * wpr + (lc >> 5)], 1u << (lc & 31));
    __syncwarp();
    const int first = active ? tr * cw + lc : -1;
    int at = first, len = 0, dir = MS_NONE, row = tr * wpr;
    bool closed = false;
    while (active) {
        const uint32_t* rt = ws.bm + row + (lc >> 5);
        const int sh = lc & 31;
        closed = len > 0 && ((starts[row + (lc >> 5)] >> sh) & 1u);
        if (closed || len == kPiece) break;
        const uint32_t top2 = __funnelshift_r(rt[0], rt[1], sh), bot2 = __funnelshift_r(rt[wpr], rt[wpr + 1], sh);
        dir = walk_dir((int)((top2 & 3u) | ((bot2 & 3u) << 2)), dir);
        piece[len++] = (uint16_t)at;
        const int dx = (dir == MS_RIGHT) - (dir == MS_LEFT), dy = (dir == MS_DOWN) - (dir == MS_UP);
        lc += dx;
        row += dy * wpr;
        at += dx + dy * cw;
    }
    __syncwarp();
    // string the pieces together
    const int origin = tr0 * cw + lc0;
    int total = 0, mine = -1, cur = 0;
    bool whole = false;
    for (int k = 0; k < 32; ++k) {
        const int end = __shfl_sync(FULL, closed ? at : -1, cur);
        if (end < 0) break;
        if (lane == cur) mine = total;
        total += __shfl_sync(FULL, len, cur);
        whole = end == origin;
        if (whole) break;
        cur = __ffs(__ballot_sync(FULL, first == end)) - 1;
    }
    if (!whole) return 0;
    if (total > W::kTrace) return -1;
    if (mine >= 0)
        for (int i = 0; i < len; ++i) ws.trace[mine + i] = piece[i];
    return total;
}

// Marching squares with the inside/outside decisions taken from a bitmap of
// the box in shared memory (built with one ballot per 32 pixels, with a
// zero border of one pixel all round so the walk needs no bounds tests), the
// walk recorded as a trace of cells (walk_parallel), and the points, junctions and duplicate removal evaluated
// across the lanes in walk order.  Returns 0 if no pixel is inside, 1 on
// success, -1 if the box or the walk does not fit the shared buffers (the
// caller then walks in global memory).
template <class W, typename R>
__device__ int extract_bitmap_warp(const Field<R>& f, const uint32_t* idl, uint32_t own, ContourOut& o, int lane,
                                   W& ws) {
    double2* const xy = ws.xy;
    const Box b = f.b;
    const int w = box_w(b), hgt = box_h(b);
    // padded bitmap: row r + 1, bit c + 1 hold pixel (r, c) of the box
    const int wpr = (w + 2 + 31) >> 5;
    if (!walk_fits<W>(b)) return -1;
    bool nonfinite = false;  // a NaN or infinity anywhere in the field
    for (int r0 = 0; r0 < hgt + 2; r0 += 8)  // eight rows of two words: 16 loads in flight
        for (int q0 = 0; q0 < wpr; q0 += 2) {
            bool in[2][8];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int c = (q0 + k) * 32 + lane - 1;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int r = r0 + u - 1;
                    const bool pix = q0 + k < wpr && r >= 0 && r < hgt && c >= 0 && c < w;
                    const R v = pix ? f.v[r * w + c] : (R)0;  // tested in the field's own type
                    nonfinite |= !isfinite(v);
                    in[k][u] = pix && v >= (R)0;
                }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t word = __ballot_sync(0xffffffffu, in[k][u]);
                    if (lane == 0 && r0 + u < hgt + 2 && q0 + k < wpr) ws.bm[(r0 + u) * wpr + q0 + k] = word;
                }
        }
    if (lane == 0) ws.bm[(hgt + 2) * wpr] = 0u;
    if (__any_sync(0xffffffffu, nonfinite) && lane == 0) o.status |= S_NAN;
    __syncwarp();
    // first and last inside words in row-major order
    int q_first = INT_MAX, q_last = -1;
    for (int q = lane; q < hgt * wpr; q += 32)
        if (ws.bm[wpr + q]) {
            q_first = min(q_first, q);
            q_last = q;
        }
    q_first = __reduce_min_sync(0xffffffffu, q_first);
    q_last = __reduce_max_sync(0xffffffffu, q_last);
    if (q_last < 0) {
        o.n = 0;
        o.jn = 0;
        return 0;
    }
    const int row_first = q_first / wpr, row_last = q_last / wpr;
    // the walk's first cell: the first inside pixel at its lower right corner
    const int cw = w + 1;
    const int tr0 = row_first, lc0 = (q_first - row_first * wpr) * 32 + (__ffs(ws.bm[wpr + q_first]) - 1) - 1;
    uint32_t st = 0;
    int nsteps = walk_parallel(ws, wpr, cw, hgt, tr0, lc0, row_first, row_last, lane);
    if (nsteps == 0) {
        if (lane == 0) nsteps = walk_serial(ws, wpr, cw, hgt, tr0, lc0, &st);
        nsteps = __shfl_sync(0xffffffffu, nsteps, 0);
        st = __shfl_sync(0xffffffffu, st, 0);
    }
    if (nsteps < 0) return -1;  // longer than the trace buffer: walk again in global memory
    o.status |= st;
    __syncwarp();
    // points and junctions of every step, in walk order.  Two 32-step
    // chunks per pass: each lane first issues the field and IDLocal loads of
    // both its steps (generatePoint's two values, generateJunction's corners),
    // then evaluates the steps in order.
    const unsigned lt = (1u << lane) - 1u;
    int ne = 0;
    int jn = 0;
    bool point_overflow = false;
    for (int t0 = 0; t0 < nsteps; t0 += 64) {
        int mask[2], next[2], left[2], top[2];
        bool emit[2], pv[2], jv[2];
        R va[2], vc[2];
        uint32_t id4[2][4];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int t = t0 + 32 * k + lane;
            mask[k] = 0;
            next[k] = MS_UP;
            left[k] = 0;
            top[k] = 0;
            emit[k] = pv[k] = jv[k] = false;
            va[k] = vc[k] = (R)0;
            id4[k][0] = id4[k][1] = id4[k][2] = id4[k][3] = own;
            if (t < nsteps) {
                // the step's direction is the move to the next recorded cell
                const int c = ws.trace[t], cn = ws.trace[t + 1 < nsteps ? t + 1 : 0];
                const int tr = c / cw, lc = c - tr * cw;
                left[k] = lc - 1 + b.x0;
                top[k] = tr - 1 + b.y0;
                const int m = cell_mask(ws.bm, wpr, tr, lc);
                mask[k] = m;
                const int dcell = cn - c;
                const int nx = dcell == -cw ? MS_UP : dcell == cw ? MS_DOWN : dcell == -1 ? MS_LEFT : MS_RIGHT;
                next[k] = nx;
                emit[k] = (kMsEmit >> m) & 1u;
                const int lf = left[k], tp = top[k], right = lf + 1, bottom = tp + 1;
                // generatePoint's values: a then c, delta = a - c (src/marchingSquares.cpp:204-265)
                const int ra = nx == MS_RIGHT || nx == MS_UP ? tp : bottom;
                const int ca = nx == MS_LEFT || nx == MS_UP ? lf : right;
                const int rc = nx == MS_LEFT ? tp : nx == MS_RIGHT ? bottom : ra;
                const int cc = nx == MS_UP ? right : nx == MS_DOWN ? lf : ca;
                pv[k] = nx == MS_LEFT ? tp >= b.y0 : nx == MS_RIGHT ? bottom < b.y1 : nx == MS_UP ? right < b.x1 : lf >= b.x0;
                if (emit[k] && pv[k]) {
                    va[k] = f.v[(ra - b.y0) * w + (ca - b.x0)];
                    vc[k] = f.v[(rc - b.y0) * w + (cc - b.x0)];
                }
                jv[k] = __popc(m) < 3 && bottom >= b.y0 && bottom < b.y1 && tp >= b.y0 && tp < b.y1 && lf >= b.x0 &&
                        lf < b.x1 && right >= b.x0 && right < b.x1;
                if (jv[k]) {  // generateJunction's corners, in its order
                    if (!(m & C_BL)) id4[k][0] = idl[(bottom - b.y0) * w + (lf - b.x0)];
                    if (!(m & C_TL)) id4[k][1] = idl[(tp - b.y0) * w + (lf - b.x0)];
                    if (!(m & C_BR)) id4[k][2] = idl[(bottom - b.y0) * w + (right - b.x0)];
                    if (!(m & C_TR)) id4[k][3] = idl[(tp - b.y0) * w + (right - b.x0)];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int lf = left[k], tp = top[k], right = lf + 1, bottom = tp + 1;
            double px = 0, py = 0;
            if (emit[k]) {  // generatePoint on the loaded values
                const int nx = next[k];
                const bool across = nx == MS_LEFT || nx == MS_RIGHT;
                // from the first value's corner to the second one's
                const double q = pv[k] ? (double)va[k] / ((double)va[k] - (double)vc[k]) : 0.0;
                const int from = nx == MS_LEFT ? bottom : nx == MS_RIGHT ? tp : nx == MS_UP ? lf : right;
                const double cut = nx == MS_LEFT || nx == MS_DOWN ? from - q : from + q;
                px = across ? (nx == MS_LEFT ? lf : right) : cut;
                py = across ? cut : (nx == MS_UP ? tp : bottom);
            }
            uint32_t boxes[4] = {0xFFFFFFu, 0xFFFFFFu, 0xFFFFFFu, 0xFFFFFFu};
            int order = 0;
            bool junc = false;
            if (jv[k]) {
                insert_distinct(id4[k][0], boxes, order);
                insert_distinct(id4[k][1], boxes, order);
                insert_distinct(id4[k][2], boxes, order);
                insert_distinct(id4[k][3], boxes, order);
                junc = order > 2;
            }
            const uint32_t eb = __ballot_sync(0xffffffffu, emit[k]);
            if (emit[k]) {
                const int pos = ne + __popc(eb & lt);
                if (pos < W::kPts)
                    xy[pos] = make_double2(px, py);
                else
                    point_overflow = true;
            }
            ne += __popc(eb);
            const uint32_t jb = __ballot_sync(0xffffffffu, junc);
            if (junc) {
                const int pos = jn + __popc(jb & lt);
                if (pos < o.jcap) {
                    Junction& j = o.js[pos];
                    j.type = order;
                    for (int q = 0; q < 4; ++q) j.grains[q] = q < order ? boxes[q] : 0xFFFFFFFFu;
                    j.segment = -1;
                    j.lambda = 0;
                    j.x = lf + 0.5;
                    j.y = tp + 0.5;
                }
            }
            jn += __popc(jb);
        }
    }
    if (__any_sync(0xffffffffu, point_overflow)) return -1;
    if (jn > o.jcap) o.status |= S_JUNCTION_OVERFLOW;  // on every lane: the caller reads the first one's
    o.jn = jn < o.jcap ? jn : o.jcap;
    __syncwarp();
    // insertPoint's duplicate test: a candidate equal to its predecessor is dropped
    int n = 0;
    for (int i0 = 0; i0 < ne; i0 += 32) {
        const int i = i0 + lane;
        double2 pnt = make_double2(0, 0);
        bool keep = false;
        if (i < ne) {
            pnt = xy[i];
            keep = i == 0 || pnt.x != xy[i - 1].x || pnt.y != xy[i - 1].y;
        }
        __syncwarp();
        const uint32_t kb = __ballot_sync(0xffffffffu, keep);
        if (keep) xy[n + __popc(kb & lt)] = pnt;
        n += __popc(kb);
        __syncwarp();
    }
    const int cap = o.cap < W::kPts ? o.cap : W::kPts;
    if (n > 0 && (xy[0].x != xy[n - 1].x || xy[0].y != xy[n - 1].y)) {  // close the loop
        if (lane == 0 && n < W::kPts) xy[n] = xy[0];
        n++;
    }
    if (n > cap) {
        o.status |= S_CONTOUR_OVERFLOW;
        n = cap;
    }
    o.n = n;
    __syncwarp();
    if (n >= 2) project_junctions(xy, o, lane);
    __syncwarp();
    return 1;
}

// grainhdl::level_set -> LSbox::extractContour (src/grainhdl.cpp:830-848,
// src/box.cpp:1089-1153), one warp per grain.  20,000 grains: 385 us with the
// walk on one lane and a junction's projection on another, 276 with both spread
// over the warp (1,000 grains 82 and 63); their floor, a field and a few values
// of IDLocal read and the contour written, is 35.  Instructions (bitmap, points)
// at 20 warps per SM bound it now, in small networks the latency of one box.
template <typename R, class W>
__device__ __forceinline__ void levelset_grain(const NetConst& C, NetState* S, int g, W& walk) {
    const int lane = threadIdx.x & 31;
    const int st = C.state[g];
    const Box bc = S->box_cur[g];
    if (st != G_EXISTS) {
        if (lane == 0) {
            if (st == G_VANISHED) {
                C.state[g] = G_GONE;
                C.gone_loop[g] = S->loop;
            }
            S->box_new[g] = bc;
            S->cn_cur[g] = 0;
            S->jn_cur[g] = 0;
        }
        return;
    }
    double2* const xy = walk.xy;
    const int old_len = S->cn_prev[g];
    R* phi = phiA_of<R>(S) + S->off_cur[g];
    Field<R> f{phi, bc};
    const uint32_t* idl = S->idCur + S->off_cur[g];
    ContourOut o{S->contCur + S->coff_cur[g], S->ccap_cur[g], 0, S->jCur + (int64_t)g * C.jmax, C.jmax, 0, 0};
    bool shared = true;
    bool ok = extract_warp(f, idl, (uint32_t)g, o, lane, walk, &shared);
    int irregular = 0;
    if (ok) {
        double newVolume = 0;
        bool regular_motion = true;
        if (shared) newVolume = form_volume<R>(xy, o.n, C.h);
        if (lane == 0) {
            if (!shared) newVolume = contour_volume(o.pts, o.n, C.h);
            regular_motion = motion_regular(old_len, o.n, C.volume[g], newVolume, C.dt, &irregular);
        }
        regular_motion = __shfl_sync(0xffffffffu, regular_motion, 0);
        int tries = 0;
        while (!regular_motion) {  // clear the grain area and extract again (src/box.cpp:1099-1114)
            bool in_range = true;
            if (shared)
                in_range = clear_area_xy(phi, bc, xy, o.n, C.h);
            else if (lane == 0)
                in_range = clear_contour_area(phi, bc, o.pts, o.n, C.h);
            if (!in_range) o.status |= S_INDEX;
            __syncwarp();
            ok = extract_warp(f, idl, (uint32_t)g, o, lane, walk, &shared);
            if (!ok) break;
            if (shared) newVolume = form_volume<R>(xy, o.n, C.h);
            if (lane == 0) {
                if (!shared) newVolume = contour_volume(o.pts, o.n, C.h);
                regular_motion = motion_regular(old_len, o.n, C.volume[g], newVolume, C.dt, &irregular);
                if (++tries > 64) {
                    o.status |= S_RETRY_LIMIT;
                    regular_motion = true;
                }
            }
            regular_motion = __shfl_sync(0xffffffffu, regular_motion, 0);
        }
        if (lane == 0 && ok && !isfinite(newVolume)) o.status |= S_NAN;
    }
    if (ok && shared) {  // publish the contour (energy and mobility still unset, as generatePoint leaves them)
        for (int i = lane; i < o.n; i += 32) {
            CPoint q;
            q.x = xy[i].x;
            q.y = xy[i].y;
            q.energy = -1.0;
            q.mob = -1.0;
            o.pts[i] = q;
        }
    }
    double perim = 0;
    if (ok && shared) perim = form_perimeter<R>(xy, o.n, C.h);
    if (ok && !shared && lane == 0) perim = contour_perimeter(o.pts, o.n, C.h);
    if (lane != 0) return;
    if (o.status) set_status(S, o.status);
    C.regular[g] = 1;
    if (!ok) {
        C.state[g] = G_VANISHED;
        S->box_new[g] = bc;
        S->cn_cur[g] = 0;
        S->jn_cur[g] = 0;
        return;
    }
    if (irregular) C.regular[g] = 0;
    int* nb = C.newbb + 4 * (int64_t)g;
    Box nbx = bc;
    if (!C.decouple) {
        if (nb[0] < 0) nb[0] = 0;
        if (nb[2] < 0) nb[2] = 0;
        if (nb[1] > C.m) nb[1] = C.m;
        if (nb[3] > C.m) nb[3] = C.m;
        nbx = resize_to_square(Box{nb[0], nb[1], nb[2], nb[3]}, C.m);
    }
    S->box_new[g] = nbx;
    C.perimeter[g] = perim;
    S->cn_cur[g] = o.n;
    S->jn_cur[g] = o.jn;
}

template <typename R>
__global__ void __launch_bounds__(32 * kGrainsPerBlock, 5) k_levelset_w(NetConst C, NetState* S) {
    __shared__ SmallWalk s_walk[kGrainsPerBlock];
    const int wid = threadIdx.x >> 5;
    const int slot = blockIdx.x * kGrainsPerBlock + wid;
    const int g = slot < C.N ? grain_at(S, slot) : C.N + 1;
    if (g > C.N || halted(S)) return;
    if (!walk_fits<SmallWalk>(S->box_cur[g])) return;  // k_levelset_big's
    levelset_grain<R>(C, S, g, s_walk[wid]);
}

// The grains whose boxes do not fit the small buffers, whatever their state:
// the two kernels run side by side or one after the other and both write the
// state (a vanished grain is deleted in the next step, not in the one it
// vanished in), so a grain belongs to one of them by its box alone, which
// neither changes.  One-warp CTAs over all slots, a lane per slot; the slots of
// one CTA are a grid apart, so that the largest boxes, which come first in the
// work queue, go to different ones.
template <typename R>
__global__ void __launch_bounds__(32) k_levelset_big(NetConst C, NetState* S) {
    __shared__ LargeWalk s_walk;
    if (halted(S)) return;
    for (int s0 = blockIdx.x; s0 < C.N; s0 += 32 * gridDim.x) {
        const int slot = s0 + (int)(threadIdx.x * gridDim.x);
        const int g = slot < C.N ? grain_at(S, slot) : 0;
        unsigned mine = __ballot_sync(0xffffffffu, g > 0 && !walk_fits<SmallWalk>(S->box_cur[g]));
        for (; mine; mine &= mine - 1) {
            levelset_grain<R>(C, S, __shfl_sync(0xffffffffu, g, __ffs(mine) - 1), s_walk);
            __syncwarp();
        }
    }
}

// Initial contours of a voxelized network (distanceInitialisation ->
// LSbox::extractContour on the initial distance field): one warp per grain
// with the level set's warp-parallel extraction (bitmap walk, points, junctions
// and their projection across the lanes), into the previous-step roles the
// first corrector reads.
template <typename R, class W>
__device__ __forceinline__ void init_contour_grain(const NetConst& C, NetState* S, int g, W& walk) {
    const int lane = threadIdx.x & 31;
    double2* const xy = walk.xy;
    Field<R> f{phiA_of<R>(S) + S->off_cur[g], S->box_cur[g]};
    const uint32_t* idl = S->idPrev + S->off_prev[g];
    ContourOut o{S->contPrev + S->coff_prev[g], S->ccap_prev[g], 0, S->jPrev + (int64_t)g * C.jmax, C.jmax, 0, 0};
    bool shared = true;
    const bool ok = extract_warp(f, idl, (uint32_t)g, o, lane, walk, &shared);
    double vol = 0;
    if (ok && shared) {
        for (int i = lane; i < o.n; i += 32) {
            CPoint q;
            q.x = xy[i].x;
            q.y = xy[i].y;
            q.energy = -1.0;
            q.mob = -1.0;
            o.pts[i] = q;
        }
        vol = form_volume<R>(xy, o.n, C.h);
    }
    if (lane != 0) return;
    if (o.status) set_status(S, o.status);
    if (!ok) {
        C.state[g] = G_VANISHED;
        S->cn_prev[g] = 0;
        S->jn_prev[g] = 0;
        C.volume[g] = 0;
        return;
    }
    if (!shared) vol = contour_volume(o.pts, o.n, C.h);
    S->cn_prev[g] = o.n;
    S->jn_prev[g] = o.jn;
    C.volume[g] = vol;
}

template <typename R>
__global__ void __launch_bounds__(32 * kGrainsPerBlock, 5) k_init_contour_w(NetConst C, NetState* S) {
    __shared__ SmallWalk s_walk[kGrainsPerBlock];
    const int wid = threadIdx.x >> 5;
    const int g = blockIdx.x * kGrainsPerBlock + wid + 1;
    if (g > C.N || C.state[g] != G_EXISTS || halted(S) || !walk_fits<SmallWalk>(S->box_cur[g])) return;
    init_contour_grain<R>(C, S, g, s_walk[wid]);
}

template <typename R>
__global__ void __launch_bounds__(32) k_init_contour_big(NetConst C, NetState* S) {
    __shared__ LargeWalk s_walk;
    const int g = blockIdx.x + 1;
    if (g > C.N || C.state[g] != G_EXISTS || halted(S) || walk_fits<SmallWalk>(S->box_cur[g])) return;
    init_contour_grain<R>(C, S, g, s_walk);
}

// Per contour point result of the neighbour probe of buildDirectNeighbours.
struct PointInfo {
    int32_t cid;
    int32_t pad;
    double theta;
    double len;
};

constexpr int kNbPts = 256;  // per-warp shared buffers of the neighbour build

// LSbox::computeVolumeAndEnergy + ExplicitGrainBoundary::buildDirectNeighbours
// (src/box.cpp:1201-1228, src/grainBoundary.cpp:85-199), one warp per grain:
// lanes probe contour points, evaluate the per-pair physics and the terms of
// the area and energy sums into shared memory; lane 0 builds the neighbour
// list and adds the terms in contour order (the reference's order; the
// batched form sums by trees instead).  Latency bounds it (a chain of five
// dependent loads per point, then the FP64 physics of a few neighbours):
// 20,000 grains 176 us with a point's chain at a time per lane in three passes
// over the contour, 136 us in one pass with two points' chains side by side (one:
// 139, four: 144 at 72 registers) and room for 256 points per warp in shared
// memory, which 99% of a network's contours need at most.
template <typename R>
__global__ void __launch_bounds__(32 * kGrainsPerBlock) k_neighbours_w(NetConst C, NetState* S, PointInfo* scratch) {
    __shared__ int s_cid[kGrainsPerBlock][kNbPts];
    __shared__ double s_len[kGrainsPerBlock][kNbPts];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int slot = blockIdx.x * kGrainsPerBlock + wid;
    const int g = slot < C.N ? grain_at(S, slot) : C.N + 1;
    if (g > C.N || C.state[g] != G_EXISTS || C.regular[g] == 0 || halted(S)) return;
    const int loop = S->loop;
    CPoint* P = S->contCur + S->coff_cur[g];
    PointInfo* info = scratch + S->coff_cur[g];
    const int n = S->cn_cur[g];
    const double h = C.h;
    const Box bc = S->box_cur[g];
    const R* phi = phiA_of<R>(S) + S->off_cur[g];
    const uint32_t* idl = S->idCur + S->off_cur[g];
    const double* qg = C.quat + 4 * (int64_t)g;
    const bool sh = n - 1 <= kNbPts;
    auto CID = [&](int q) -> int& { return sh ? s_cid[wid][q] : info[q].cid; };
    auto LEN = [&](int q) -> double& { return sh ? s_len[wid][q] : info[q].len; };
    // One pass over the points, kU per lane with each level of their loads in
    // flight together: the area's terms (computeVolume, src/grainBoundary.cpp:
    // 201-213; added in contour order in the plain form, by a tree in the
    // batched one, as the sums below), the segments' lengths, and the probes,
    // the first failing one of which ends the reference's loop.
    constexpr bool kTree = sizeof(R) == sizeof(float);
    constexpr int kU = 2;
    double v = 0;
    int first_bad = 0x7fffffff;
    for (int i0 = 0; i0 < n - 1; i0 += 32 * kU) {
        double px[kU], py[kU], area[kU], len[kU];
        uint32_t k[kU], cid[kU];
        bool bad[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = i0 + 32 * u + lane;
            px[u] = py[u] = area[u] = len[u] = 0;
            if (i < n - 1) {
                px[u] = P[i].x;
                py[u] = P[i].y;
                const double qx = P[i + 1].x, qy = P[i + 1].y;
                if constexpr (kTree)
                    v += (py[u] + qy) * (px[u] - qx);
                else
                    area[u] = (py[u] + qy) * (px[u] - qx);
                const double dx = px[u] - qx, dy = py[u] - qy;
                len[u] = sqrt(dx * dx + dy * dy);
            }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            // the corners in the reference's order; the first whose field is
            // not positive is the probe, else the fourth, and a corner outside
            // the box before that is a failure
            const int gx = (int)px[u], gy = (int)py[u];
            const int gx1 = (int)(px[u] + 1), gy1 = (int)(py[u] + 1);
            uint32_t k0 = 0, k1 = 0, k2 = 0;
            const bool in0 = buf_index(bc, gy, gx, &k0), in1 = buf_index(bc, gy, gx1, &k1);
            const bool in2 = buf_index(bc, gy1, gx1, &k2);
            const bool live = i0 + 32 * u + lane < n - 1;
            const double f0 = live && in0 ? (double)phi[k0] : 0, f1 = live && in1 ? (double)phi[k1] : 0;
            const double f2 = live && in2 ? (double)phi[k2] : 0;
            const bool past0 = in0 && f0 > 0, past1 = past0 && in1 && f1 > 0, past2 = past1 && in2 && f2 > 0;
            const int x = past0 && !past2 ? gx1 : gx, y = past1 ? gy1 : gy;
            bad[u] = !in0 || (past0 && !in1) || (past1 && !in2) || y < 0 || y >= bc.y1 || x < 0 || x >= bc.x1;
            bad[u] = !buf_index(bc, y, x, &k[u]) || bad[u];
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) cid[u] = !bad[u] && i0 + 32 * u + lane < n - 1 ? idl[k[u]] : 0u;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            if (cid[u] > (uint32_t)C.N)
                bad[u] = true;
            else if (cid[u] != 0 && C.state[cid[u]] == G_GONE)
                bad[u] = true;
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = i0 + 32 * u + lane;
            if (i < n - 1) {
                CID(i) = bad[u] ? -1 : (int)cid[u];
                LEN(i) = len[u];
                if (bad[u]) first_bad = min(first_bad, i);
            }
            if constexpr (!kTree) {
                const int m = min(n - 1 - (i0 + 32 * u), 32);
                for (int q = 0; q < m; ++q) v += __shfl_sync(FULL, area[u], q);
            }
        }
    }
    if constexpr (kTree) v = warp_sum_to_all(v);
    const double newVolume = fabs(fabs(v) * h * h * 0.5);
    first_bad = warp_min_i(first_bad);
    const int upto = first_bad < n - 1 ? first_bad : n - 1;
    __syncwarp();
    // neighbour list in first-occurrence order (one entry per distinct
    // neighbour, at most `cap`; later new neighbours are dropped), then each
    // entry's length summed over its points in contour order
    __shared__ int s_nid[kGrainsPerBlock][48];
    const int cap = C.nbmax < 48 ? C.nbmax : 48;
    int nn = 0;
    bool overflow = false;
    const unsigned lt = (1u << lane) - 1u;
    for (int i0 = 0; i0 < upto; i0 += 32) {
        const int i = i0 + lane;
        const int cid = i < upto ? CID(i) : -2;
        bool fresh = i < upto;
        for (int e = 0; e < nn && fresh; ++e)
            if (s_nid[wid][e] == cid) fresh = false;
        const unsigned same = __match_any_sync(FULL, cid);
        fresh = fresh && (__ffs(same) - 1) == lane;
        const unsigned fb = __ballot_sync(FULL, fresh);
        if (fresh) {
            const int pos = nn + __popc(fb & lt);
            if (pos < cap) s_nid[wid][pos] = cid;
        }
        if (nn + __popc(fb) > cap) overflow = true;
        nn = min(nn + __popc(fb), cap);
        __syncwarp();
    }
    // each listed neighbour's misorientation, energy and mobility, once
    __shared__ double s_nth[kGrainsPerBlock][48], s_nen[kGrainsPerBlock][48], s_nmob[kGrainsPerBlock][48];
    for (int e = lane; e < nn; e += 32) {
        const double theta = grain_misorientation(qg, C.quat + 4 * (int64_t)s_nid[wid][e]);
        s_nth[wid][e] = theta;
        s_nen[wid][e] = read_shockley(theta, C);
        s_nmob[wid][e] = mobility_model(theta, C);
    }
    __syncwarp();
    // physics of the points before the first failure; energy terms of all
    // points, added in contour order (computeEnergy, src/grainBoundary.cpp:215-222)
    double energy_sum = 0;
    for (int i0 = 0; i0 < n - 1; i0 += 32) {
        const int i = i0 + lane;
        double term = 0;
        if (i < n - 1) {
            const double len = LEN(i);
            double energy = -1.0;  // generatePoint's value, kept where the loop never reached
            if (i < upto) {
                // the neighbour's physics, evaluated once per neighbour above
                // (the same calls on the same orientations)
                const int cid = CID(i);
                int e = 0;
                while (e < nn && s_nid[wid][e] != cid) ++e;
                double mob;
                if (e < nn) {
                    mob = s_nmob[wid][e];
                    energy = s_nen[wid][e];
                } else {  // beyond the list's capacity
                    const double theta = grain_misorientation(qg, C.quat + 4 * (int64_t)cid);
                    mob = mobility_model(theta, C);
                    energy = read_shockley(theta, C);
                }
                P[i].mob = mob;
                P[i].energy = energy;
            }
            term = len * energy * h;
        }
        if constexpr (kTree) {
            energy_sum += term;
        } else {
            const int m = n - 1 - i0 < 32 ? n - 1 - i0 : 32;
            for (int q = 0; q < m; ++q) energy_sum += __shfl_sync(FULL, term, q);
        }
    }
    if constexpr (kTree) energy_sum = warp_sum_to_all(energy_sum);
    __syncwarp();
    Neighbour* nb = C.nb + (int64_t)g * C.nbmax;
    __shared__ double s_nlen[kGrainsPerBlock][48];
    if constexpr (kTree) {  // each neighbour's length by the whole warp
        for (int e = 0; e < nn; ++e) {
            const int cid = s_nid[wid][e];
            double len = 0;
            for (int i = lane; i < upto; i += 32)
                if (CID(i) == cid) len += LEN(i) * h;
            len = warp_sum_to_all(len);
            if (lane == 0) s_nlen[wid][e] = len;
        }
        __syncwarp();
    }
    for (int e = lane; e < nn; e += 32) {
        const int cid = s_nid[wid][e];
        double len = 0;
        if constexpr (kTree) {
            len = s_nlen[wid][e];
        } else {
            for (int i = 0; i < upto; ++i)
                if (CID(i) == cid) len += LEN(i) * h;
        }
        nb[e].id = cid;
        nb[e].length = len;
        nb[e].energy = s_nen[wid][e];
        nb[e].misori = s_nth[wid][e];
        nb[e].mobility = s_nmob[wid][e];
    }
    if (lane != 0) return;
    C.nb_n[g] = nn;
    if (overflow) set_status(S, S_NEIGHBOUR_OVERFLOW);
    if (first_bad < n - 1) {
        C.regular[g] = 0;  // markAsInvalidMotion (src/box.cpp:1939-1945)
    } else if (n > 0) {
        P[n - 1].energy = P[0].energy;
        P[n - 1].mob = P[0].mob;
    }
    C.energy[g] = energy_sum;
    double dA = newVolume - C.volume[g];
    dA = dA / C.dt;
    dA = dA * (3 / kPi);
    const unsigned int lp = (unsigned int)loop;
    if ((unsigned long)(lp - 1u) % (unsigned long)C.analysis_timestep == 0 || lp == 0) C.meanda[g] = 0;
    C.meanda[g] += dA;
    C.volume[g] = newVolume;
}

// LSbox::computeSecondOrderNeighbours (src/box.cpp:1027-1068), one warp per
// grain: candidates of each member's list are tested across lanes and the
// accepted ones appended in list order.
__global__ void __launch_bounds__(32 * kGrainsPerBlock) k_second_order_w(NetConst C, NetState* S) {
    constexpr int kL = 128;
    __shared__ int s_list[kGrainsPerBlock][kL];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int slot = blockIdx.x * kGrainsPerBlock + wid;
    const int g = slot < C.N ? grain_at(S, slot) : C.N + 1;
    if (g > C.N || C.state[g] != G_EXISTS) return;
    const int K = C.kmax < kL ? C.kmax : kL;
    const int* sec = C.sec_ids + (int64_t)g * C.kmax;
    const int ns = C.sec_n[g];
    int* list = s_list[wid];
    const unsigned lt = (1u << lane) - 1u;
    int nc = 0;
    bool overflow = false;
    for (int a0 = 0; a0 < ns; a0 += 32) {  // existing members, in order
        const int a = a0 + lane;
        const bool take = a < ns && C.state[sec[a]] == G_EXISTS;
        const unsigned bal = __ballot_sync(0xffffffffu, take);
        if (take) {
            const int pos = nc + __popc(bal & lt);
            if (pos < K) list[pos] = sec[a]; else overflow = true;
        }
        nc += __popc(bal);
        if (nc > K) nc = K;
    }
    __syncwarp();
    const Box mine = S->box_cur[g];
    for (int a = 0; a < ns; ++a) {
        const int id = sec[a];
        const int* s2 = C.sec_ids + (int64_t)id * C.kmax;
        const int n2 = C.sec_n[id];
        for (int q0 = 0; q0 < n2; q0 += 32) {
            const int q = q0 + lane;
            bool take = false;
            int c = 0;
            if (q < n2) {
                c = s2[q];
                take = C.state[c] == G_EXISTS && c != g && c != 0 && boxes_intersect(mine, S->box_cur[c]);
                if (take)
                    for (int e = 0; e < nc; ++e)
                        if (list[e] == c) {
                            take = false;
                            break;
                        }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int pos = nc + __popc(bal & lt);
                if (pos < K) list[pos] = c; else overflow = true;
            }
            nc += __popc(bal);
            if (nc > K) nc = K;
            __syncwarp();
        }
    }
    int* cmp = C.cmp_ids + (int64_t)g * C.kmax;
    for (int e = lane; e < nc; e += 32) cmp[e] = list[e];
    if (lane == 0) {
        C.cmp_n[g] = nc;
        if (overflow || C.kmax > kL) set_status(S, overflow ? S_LIST_OVERFLOW : 0u);
    }
}

}  // namespace
}  // namespace gg
