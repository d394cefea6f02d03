// ft_slots.cuh — the leaves of a curve's subdivision by address.
//
// footile flattens curves by recursive De Casteljau subdivision (plotter.rs:248-265, 311-332).
// Walked depth first by one thread that is a chain of dependent nodes with a stack in local
// memory, twice over when the leaves have to be counted before they are placed.  Here a leaf is
// addressed instead: with D the depth at which the whole curve is flat, slot i of 2^D takes the
// path of the bits of i from the root (0 left, 1 right, most significant first), D levels of
// midpoints and no stack — the same arithmetic on the same operands, so the same points.  A
// node that is flat above D is a leaf owned by the first slot of its range; the other slots of
// the range own nothing.
#pragma once

#include "ft_device.cuh"

namespace ftk {

constexpr int SLOT_DEPTH = 12;  // deepest D of a slot walk; deeper curves are walked depth first

// Depth D at which every node of the curve's subdivision is flat (more than SLOT_DEPTH: not
// known to be), and the depth `safe` above which no node is flat.  Both hold for the rounded
// arithmetic of the walk, so that nodes at D and above `safe` need no check.
//
// At depth k a node centred at t has the flatness vector 4^-k p''(t) / 8 (quads: p'' constant;
// cubics: linear, so the outermost two nodes of a level have the longest, and the point of the
// curve where p'' is shortest bounds all of them from below).  In the walk a level of midpoints
// adds at most three roundings of half an ulp of the largest coordinate m (2^-24 m) to each
// coordinate of a node; the flatness test compares two such points, and the estimate itself
// rounds ten times at most: (9 k + 24) 2^-24 m covers both coordinates of the difference.
__device__ __forceinline__ int curve_depth(P2 a, P2 b, P2 c, P2 d, bool cubic, float tol, int& safe) {
    const float m = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))),
                          fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(d.x), fabsf(d.y)))) *
                    5.9604645e-8f;
    float lo = tol * 0.99998f - 24.0f * m, hi = tol * 1.00002f + 24.0f * m;
    safe = 0;
    int k = 0;
    if (!cubic) {
        const float x = a.x - 2.0f * b.x + c.x, y = a.y - 2.0f * b.y + c.y;
        float f = (x * x + y * y) * 0.0625f;
        for (; k <= SLOT_DEPTH; k++) {
            if (lo > 0.0f && f <= lo * lo) break;
            if (f > hi * hi) safe = k + 1;
            f *= 0.0625f;
            lo -= 9.0f * m;
            hi += 9.0f * m;
        }
        return k;
    }
    const float x0 = 0.75f * (a.x - 2.0f * b.x + c.x), y0 = 0.75f * (a.y - 2.0f * b.y + c.y);
    const float x1 = 0.75f * (b.x - 2.0f * c.x + d.x) - x0, y1 = 0.75f * (b.y - 2.0f * c.y + d.y) - y0;
    const float n2 = x1 * x1 + y1 * y1;
    const float t = n2 > 0.0f ? fminf(fmaxf(-(x0 * x1 + y0 * y1) / n2, 0.0f), 1.0f) : 0.0f;
    const float wx = x0 + t * x1, wy = y0 + t * y1, w2 = (wx * wx + wy * wy) * 0.999f;
    float h = 0.5f, s = 1.0f;
    for (; k <= SLOT_DEPTH; k++) {
        const float ux = x0 + h * x1, uy = y0 + h * y1, vx = x0 + (1.0f - h) * x1, vy = y0 + (1.0f - h) * y1;
        if (lo > 0.0f && fmaxf(ux * ux + uy * uy, vx * vx + vy * vy) * s <= lo * lo) break;
        if (w2 * s > hi * hi) safe = k + 1;
        h *= 0.5f;
        s *= 0.0625f;
        lo -= 9.0f * m;
        hi += 9.0f * m;
    }
    return k;
}

// The leaf at slot `idx` of a quad (plotter.rs:248-265): its end points in a and c, with W the
// widths there in wa and wc (wb: the control point's).  Returns the leaf's depth, or -1 when the
// slot owns no leaf.
template <bool W = false>
__device__ __forceinline__ int quad_slot(P2& a, P2 b, P2& c, float& wa, float wb, float& wc, int idx, int D, int safe,
                                         float tol_sq) {
    for (int k = 0; k < D; k++) {
        const P2 ab = pmid(a, b), bc = pmid(b, c), m = pmid(ab, bc);
        if (k >= safe && pdist_sq(m, pmid(a, c)) <= tol_sq) return (idx & ((1 << (D - k)) - 1)) ? -1 : k;
        float wab = 0.f, wbc = 0.f, wm = 0.f;
        if (W) {
            wab = fmid(wa, wb);
            wbc = fmid(wb, wc);
            wm = fmid(wab, wbc);
        }
        if ((idx >> (D - 1 - k)) & 1) {
            a = m;
            b = bc;
            if (W) {
                wa = wm;
                wb = wbc;
            }
        } else {
            b = ab;
            c = m;
            if (W) {
                wb = wab;
                wc = wm;
            }
        }
    }
    return D;
}
// The same for a cubic (plotter.rs:311-332): end points in a and e.
template <bool W = false>
__device__ __forceinline__ int cubic_slot(P2& a, P2 b, P2 c, P2& e, float& wa, float wb, float wc, float& we, int idx,
                                          int D, int safe, float tol_sq) {
    for (int k = 0; k < D; k++) {
        const P2 ab = pmid(a, b), bc = pmid(b, c), cd = pmid(c, e);
        const P2 abbc = pmid(ab, bc), bccd = pmid(bc, cd), m = pmid(abbc, bccd);
        if (k >= safe && pdist_sq(m, pmid(a, e)) <= tol_sq) return (idx & ((1 << (D - k)) - 1)) ? -1 : k;
        float wab = 0.f, wcd = 0.f, wabbc = 0.f, wbccd = 0.f, wm = 0.f;
        if (W) {
            const float wbc = fmid(wb, wc);
            wab = fmid(wa, wb);
            wcd = fmid(wc, we);
            wabbc = fmid(wab, wbc);
            wbccd = fmid(wbc, wcd);
            wm = fmid(wabbc, wbccd);
        }
        if ((idx >> (D - 1 - k)) & 1) {
            a = m;
            b = bccd;
            c = cd;
            if (W) {
                wa = wm;
                wb = wbccd;
                wc = wcd;
            }
        } else {
            b = ab;
            c = abbc;
            e = m;
            if (W) {
                wb = wab;
                wc = wabbc;
                we = wm;
            }
        }
    }
    return D;
}

// The op of each slot of a warp's window: `off` lists the first slots of the ops that have any
// (ascending, 32 times INT_MAX after the last), s0 is the window's first slot, j0 an op at or
// before it (moved up to the op of s0).  Returns the op of slot s0 + lane.
__device__ __forceinline__ int slot_op(const int* off, int s0, int& j0) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        const unsigned m = __ballot_sync(0xFFFFFFFFu, off[j0 + 1 + lane] <= s0);
        j0 += __popc(m);
        if (m != 0xFFFFFFFFu) break;
    }
    const int rel = off[j0 + 1 + lane] - s0;
    const unsigned starts = __reduce_or_sync(0xFFFFFFFFu, rel < 32 ? 1u << rel : 0u);
    return j0 + __popc(starts & (0xFFFFFFFFu >> (31 - lane)));
}

}  // namespace ftk
