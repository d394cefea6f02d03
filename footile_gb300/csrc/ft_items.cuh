// ft_items.cuh — cell areas of (segment, row) items spread over a warp, and the resolve of rows
// of cells, eight pixels a lane (tile rasteriser, single-call band compositor).
#pragma once

#include "ft_device.cuh"
#include "ft_kernels.cuh"

namespace ftk {

constexpr unsigned ALL = 0xFFFFFFFFu;

// ---------------------------------------------------------------- arithmetic
// Low 32 bits of n * 65536 / d (truncated), d != 0: Fixed division (fixed.rs:49-56) of
// magnitudes without the 64-bit divide.  The quotient is estimated in float (relative error
// below 2^-21), the remainder corrects it: a second estimate of what is missing leaves less
// than one unit, which the last comparisons settle.  With n and d below 2^28 (4,096 pixels)
// the remainder stays below 2^23 + d, so 32-bit wrapping arithmetic holds it.  Larger
// operands and quotients of 2^31 and above (slopes of 32,768 and more) take the 64-bit divide.
__device__ __forceinline__ unsigned fx_quot(unsigned n, unsigned d) {
    float f;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)d));
    const float est = (float)n * f * 65536.0f;
    if (((n | d) >> 28) || est >= 2147483000.0f) return (unsigned)(((unsigned long long)n << 16) / d);
    unsigned q = (unsigned)est;
    int r = (int)((n << 16) - q * d);
    const int q2 = __float2int_rn((float)r * f);
    r = (int)((unsigned)r - (unsigned)q2 * d);
    return q + (unsigned)q2 - (r < 0 ? 1u : 0u) + (r >= (int)d ? 1u : 0u);
}
__device__ __forceinline__ unsigned uabs(int v) { return v < 0 ? 0u - (unsigned)v : (unsigned)v; }
// fxdiv for any operands (b != 0)
__device__ __forceinline__ int fx_div(int a, int b) {
    const unsigned q = fx_quot(uabs(a), uabs(b));
    return (a ^ b) < 0 ? (int)(0u - q) : (int)q;
}

// Fixed::from(f32) (fixed.rs:88-93): the conversion instruction saturates and takes NaN to 0
__device__ __forceinline__ int to_fx(float f) { return __float2int_rz(__fmul_rn(f, 65536.0f)); }

// A segment ready for run_items: for lane's segment, `n_items` items, rows counted from `row0`,
// the area row of its first row.  ra: x leaving its first row, the inverse slope, x entering
// the row the segment starts in, and the way back from the bottom of its last row to its end.
struct SegRec {
    int n_items;
    int4 ra, rb;
};
// Items of a segment that reaches rows [yb0, yb1): its rows there, each as 2^ls lanes of CELLS
// cells (item_shift; the raster is W pixels wide).  (ux, fu): where it starts and the y fraction there, fl: the fraction where it ends.
__device__ __forceinline__ SegRec seg_items(int ux, int fu, int fl, int start, int end, int inv, int step, bool neg,
                                            int yb0, int yb1, int pitch, int W) {
    SegRec s;
    const int pu = (fu + 128) >> 8, pl = (fl + 128) >> 8;  // pixel_cov of the fractions
    const int ya = max(start, yb0), yl = min(fl ? end : end - 1, yb1 - 1);
    const int nrow = yl - ya + 1;
    // the longest walk of its rows: cov * 256 / step cells and one, rounded up
    const int most = start == end ? pl - pu : (end - start > 1 ? 256 : max(256 - pu, pl));
    const int cells = (int)__fdividef((float)max(most, 0) * 256.0256f, (float)step) + 2;
    const int ls = item_shift(cells, W);
    s.n_items = nrow > 0 ? nrow << ls : 0;
    s.ra.x = wadd(wadd(ux, fxmul(inv, FX_ONE - fu)), wmul(ya - start, inv));
    s.ra.y = inv;
    s.ra.z = ux;
    s.ra.w = fl ? fxmul(inv, FX_ONE - fl) : 0;
    s.rb.x = 0;
    s.rb.y = step | (ls << 20);
    s.rb.z = (ya - yb0) * pitch;
    s.rb.w = pl | (pu << 9) | ((ya == start ? 1 : 0) << 18) | ((fl && yl == end ? 1 : 0) << 19) | ((neg ? 1 : 0) << 20) |
             (int)((unsigned)nrow << 21);
    return s;
}

// Cell areas of the lanes' segments into `area` (rows of `pitch` cells, the raster W pixels
// wide), scaled by 2^16: the i16 sums of footile wrap in the upper halves.
//
// One lane works out a segment; the (segment, row) items are then spread over the lanes, an
// item that walks many cells as several lanes of CELLS cells each, so that a window of 32
// costs the same whatever the slopes in it: the walk is closed (x_cov after j cells is
// first + j * step), so any lane can start in the middle of it.  rec: 64 records of the warp;
// cells: those that `area` holds.
__device__ __forceinline__ void run_items(int4* rec, SegRec s, int* area, int cells, int pitch, int W) {
    const int lane = threadIdx.x & 31;
    int inc = s.n_items;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(ALL, inc, o);
        if (lane >= o) inc += t;
    }
    const int off = inc - s.n_items, tot = __shfl_sync(ALL, inc, 31);
    // segments with items, in order
    const bool on = s.n_items > 0;
    const unsigned has = __ballot_sync(ALL, on);
    if (on) {
        const int at = __popc(has & ((1u << lane) - 1u));
        s.rb.x = off;
        rec[2 * at] = s.ra;
        rec[2 * at + 1] = s.rb;
    }
    __syncwarp();
    for (int w0 = 0; w0 < tot; w0 += 32) {
        // the segment of item w0 + lane: segments that start at or before it (each has an item)
        const int rel = off - w0;
        const unsigned at = __reduce_or_sync(ALL, (on && rel >= 0 && rel < 32) ? 1u << rel : 0u);
        const int before = __popc(__ballot_sync(ALL, on && rel < 0));
        const int item = w0 + lane;
        if (item >= tot) continue;
        const int j = before + __popc(at & (ALL >> (31 - lane))) - 1;
        if (!ck(j >= 0 && j < 32, 19)) continue;
        const int4 A = rec[2 * j], C = rec[2 * j + 1];
        const int ls = C.y >> 20, step = C.y & 0xFFFFF;
        const int k = (item - C.x) >> ls, c0 = ((item - C.x) & ((1 << ls) - 1)) * CELLS;
        const bool st = ((C.w >> 18) & 1) && k == 0, en = ((C.w >> 19) & 1) && k == (int)((unsigned)C.w >> 21) - 1;
        const int cov = (en ? C.w & 511 : 256) - (st ? (C.w >> 9) & 511 : 0);
        const int xb = wadd(A.x, wmul(k, A.y));
        const int x0 = st ? A.z : wsub(xb, A.y), x1 = en ? wsub(xb, A.w) : xb;
        const int mnx = min(x0, x1), mxx = max(x0, x1);
        const int minp = mnx >> 16, maxp = mxx >> 16;
        if (cov <= 0 || minp >= W) continue;
        // fig.rs:285-321: x_cov runs first, first + step, ...; each cell gets the growth of
        // min(pixel_cov(x_cov), cov).  pixel_cov(x) is (x + 128) >> 8 for x in [0, ONE], and
        // cov <= 256 stands in for the cap at ONE.
        const unsigned r = minp == maxp ? ((unsigned)(FX_ONE - fxfract(fxavg(mxx, mnx))) * (unsigned)cov) >> 8
                                        : (unsigned)(FX_ONE - fxfract(mnx)) >> 1;
        unsigned xc = (unsigned)(((unsigned long long)r * (unsigned)step) >> 16) + 128u;
        int* cell = area + C.z + k * pitch + c0;
        int left = W - c0;  // cells to the raster's end; the row has CELLS - 1 spare ones after it
        if (minp < 0) {
            // cells left of the raster all land in cell 0 (fig.rs:295): their sum telescopes
            const unsigned long long v = (unsigned long long)xc + (unsigned long long)(unsigned)-minp * (unsigned)step;
            xc = v > FX_ONE + 128 ? FX_ONE + 128 : (unsigned)v;
        } else {
            cell += minp;
            left -= minp;
        }
        if (left <= 0) continue;
        xc += (unsigned)c0 * (unsigned)step;
        int prev = c0 ? min((int)((xc - (unsigned)step) >> 8), cov) : 0;
        const int sgn = (C.w >> 20) & 1 ? -FX_ONE : FX_ONE;
#pragma unroll
        for (int u = 0; u < CELLS; u++) {
            const int v = min((int)(xc >> 8), cov);
            if (v != prev && ck((unsigned)(cell + u - area) < (unsigned)cells, 18)) atomicAdd(cell + u, (v - prev) * sgn);
            prev = v;
            xc += (unsigned)step;
        }
    }
    __syncwarp();
}

// Fill rule on four running sums (i16, in the upper halves; imgbuf.rs:54-61, 157-167),
// packed into bytes
template <int RULE>
__device__ __forceinline__ unsigned resolve4(int a, int b, int c, int d) {
    if (RULE == FT_NONZERO) {  // clamp to 0 .. 255
        a = __vimin_s32_relu(a, 0x00FFFFFF);
        b = __vimin_s32_relu(b, 0x00FFFFFF);
        c = __vimin_s32_relu(c, 0x00FFFFFF);
        d = __vimin_s32_relu(d, 0x00FFFFFF);
    } else {  // |v - odd|: t or 512 - t of the low nine bits t, at most 255
        a &= 0x01FF0000;
        b &= 0x01FF0000;
        c &= 0x01FF0000;
        d &= 0x01FF0000;
        a = __vimin3_s32(a, 0x02000000 - a, 0x00FF0000);
        b = __vimin3_s32(b, 0x02000000 - b, 0x00FF0000);
        c = __vimin3_s32(c, 0x02000000 - c, 0x00FF0000);
        d = __vimin3_s32(d, 0x02000000 - d, 0x00FF0000);
    }
    return __byte_perm(__byte_perm(a, b, 0x0062), __byte_perm(c, d, 0x0062), 0x5410);
}
// The last n (one to three) bytes of a row, from w, to a 4-byte aligned address
__device__ __forceinline__ void store_tail(uint8_t* dp, unsigned w, int n) {
    if (n & 2) *reinterpret_cast<unsigned short*>(dp) = (unsigned short)w;
    if (n & 1) dp[n & 2] = (uint8_t)(w >> (8 * (n & 2)));
}

// A row's eight cells of one lane, cleared, and their running sum in s[0 .. 7]; `inc` gets the
// inclusive sum over the row's lanes (l: the lane in its row).
__device__ __forceinline__ void take8(int* ap, bool in, int l, unsigned* s, unsigned& inc) {
    int4 a = make_int4(0, 0, 0, 0), b = a;
    if (in) {
        a = reinterpret_cast<const int4*>(ap)[0];
        b = reinterpret_cast<const int4*>(ap)[1];
        reinterpret_cast<int4*>(ap)[0] = make_int4(0, 0, 0, 0);
        reinterpret_cast<int4*>(ap)[1] = make_int4(0, 0, 0, 0);
    }
    s[0] = a.x;
    s[1] = s[0] + a.y;
    s[2] = s[1] + a.z;
    s[3] = s[2] + a.w;
    s[4] = s[3] + b.x;
    s[5] = s[4] + b.y;
    s[6] = s[5] + b.z;
    s[7] = s[6] + b.w;
    inc = s[7];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {  // lane l of a row takes from lane l - o of the same row
        const unsigned t = __shfl_up_sync(ALL, inc, o);
        if (l >= o) inc += t;
    }
}
// The eight pixels of sums s + ex, the figure's direction (sg: 1 or -1) flipping every sum
template <int RULE>
__device__ __forceinline__ uint2 pixels8(const unsigned* s, unsigned ex, int sg) {
    int u[8];
    const unsigned exs = ex * (unsigned)sg;
#pragma unroll
    for (int k = 0; k < 8; k++) u[k] = (int)(s[k] * (unsigned)sg + exs);
    return make_uint2(resolve4<RULE>(u[0], u[1], u[2], u[3]), resolve4<RULE>(u[4], u[5], u[6], u[7]));
}

}  // namespace ftk
