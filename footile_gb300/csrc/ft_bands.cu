// ft_bands.cu — a single call's rows (ft_fill / ft_stroke on a large canvas, an
// ft_composite_batch of one path): its edges are binned by bands of P.band_rows rows.
//
// One CTA per band holds the band's cells in shared memory (131 KB for eight rows of 4,096),
// so one CTA is resident per SM and its warps alone hide the latencies: 32 of them.  Each warp
// takes 32 edges of the band at a time and spreads their (edge, row) items over its lanes, with
// no barrier until the cells are done; then several warps share a row, each summing its part
// before the parts are resolved with what lies left of them.  (Eight warps with block scans per
// 256 edges: 73 us for the 4096 x 4096 scene's 512 bands.)
#include <algorithm>

#include "ft_items.cuh"

namespace ftk {
namespace {

// Shared memory: the warps' records, the cells, the row parts' sums.
__host__ __device__ constexpr int band_smem(int threads, int rows, int width) {
    return threads / 32 * 64 * (int)sizeof(int4) + rows * tile_pitch(width) * 4 + threads / 32 * 4;
}

// Eight pixels to dp, nb of them inside the row; al: the rows' alignment (8, 4 or 1 bytes).
__device__ __forceinline__ void store8(uint8_t* dp, uint2 px, int nb, int al) {
    if (al == 8 && nb >= 8) {
        *reinterpret_cast<uint2*>(dp) = px;
    } else if (al >= 4) {
        if (nb >= 4) *reinterpret_cast<unsigned*>(dp) = px.x;
        if (nb >= 8)
            *reinterpret_cast<unsigned*>(dp + 4) = px.y;
        else if (nb & 3)
            store_tail(dp + (nb & 4), nb < 4 ? px.x : px.y, nb & 3);
    } else {
        for (int k = 0; k < min(nb, 8); k++) dp[k] = (uint8_t)((k < 4 ? px.x : px.y) >> (8 * (k & 3)));
    }
}

template <int RULE>
__device__ __forceinline__ void band_part(int* row, uint8_t* drow, int x0, int x1, int W, unsigned carry, int al) {
    const int lane = threadIdx.x & 31;
    for (int x = x0; x < x1; x += 256) {
        const int at = x + 8 * lane, nb = W - at;
        unsigned s[8], inc;
        take8(row + at, nb > 0, lane, s, inc);
        const uint2 px = pixels8<RULE>(s, inc - s[7] + carry, 1);
        carry += __shfl_sync(ALL, inc, 31);
        if (nb > 0) store8(drow + at, px, nb, al);
    }
}

template <int NT>
__global__ void __launch_bounds__(NT, 1) k_band_single(KParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = (int)P.canvas_w, H = (int)P.canvas_h, R = P.band_rows, b = blockIdx.x;
    const int pitch = tile_pitch(W);
    int4* rec = reinterpret_cast<int4*>(smem) + warp * 64;
    int* area = reinterpret_cast<int*>(smem + NW * 64 * sizeof(int4));
    int* part = area + R * pitch;
    const int4 cr = P.crec[0];
    const int r0 = max(b * R, cr.x), r1 = min(b * R + R, H);  // rows the call draws here
    if (r0 >= r1) return;
    const int nr = r1 - r0;
    for (int x = tid * 4; x < nr * pitch; x += NT * 4) *reinterpret_cast<int4*>(area + x) = make_int4(0, 0, 0, 0);
    const int o0 = P.bandoff[b], ne = P.bandoff[b + 1] - o0;
    const int4* edges = reinterpret_cast<const int4*>(
        P.pool + ((unsigned long long)(unsigned)cr.z | ((unsigned long long)(unsigned)cr.w << 32)) + o0);
    const int yb0 = r0 + cr.y, yb1 = r1 + cr.y;  // scan rows
    __syncthreads();
    // few edges: fewer per warp, so that every warp has some
    const int per_warp = min(32, max(4, (ne + NW - 1) / NW));
    for (int g = warp * per_warp; g < ne; g += NW * per_warp) {
        SegRec s;
        s.n_items = 0;
        s.ra = s.rb = make_int4(0, 0, 0, 0);
        if (lane < per_warp && g + lane < ne &&
            ck((unsigned long long)(reinterpret_cast<const EdgeRec*>(edges) - P.pool) + g + lane < P.pool_cap, 27)) {
            const int4 a = edges[2 * (g + lane)], c = edges[2 * (g + lane) + 1];
            const EdgeRec E{a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
            const int fu = fxfract(E.y_upper);
            // x_bot0 is the x it starts at, moved to the bottom of its first row (fig.rs:187-199)
            if (E.ed)
                s = seg_items(wsub(E.x_bot0, fxmul(E.inv_slope, FX_ONE - fu)), fu, fxfract(E.y_lower), E.start_row,
                              E.end_row, E.inv_slope, E.step_pix > 0 ? E.step_pix : FX_ONE, E.ed < 0, yb0, yb1, pitch, W);
        }
        run_items(rec, s, area, R * pitch, pitch, W);
    }
    __syncthreads();
    const int parts = NW / R;  // warps per row (R <= 8 <= NW)
    const int steps = (W + 255) >> 8, per = (steps + parts - 1) / parts;
    const int q = warp / parts, p = warp % parts;  // this warp's row and its part of it
    const int x0 = min(p * per * 256, W), x1 = min(x0 + per * 256, W);
    if (q < nr && p + 1 < parts) {
        unsigned sum = 0;
        for (int x = x0 + 8 * lane; x < x1; x += 256) {
            const int4 u = *reinterpret_cast<const int4*>(area + q * pitch + x);
            const int4 v = *reinterpret_cast<const int4*>(area + q * pitch + x + 4);
            sum += (unsigned)u.x + (unsigned)u.y + (unsigned)u.z + (unsigned)u.w + (unsigned)v.x + (unsigned)v.y +
                   (unsigned)v.z + (unsigned)v.w;
        }
        sum = __reduce_add_sync(ALL, sum);
        if (lane == 0 && ck(q * pitch + x1 <= R * pitch, 26)) part[warp] = (int)sum;
    }
    __syncthreads();
    if (q >= nr || !ck(q * pitch + min((x1 + 7) & ~7, pitch) <= R * pitch && r0 + q < H, 26)) return;
    const int al = ((reinterpret_cast<uintptr_t>(P.rasters) | P.canvas_stride) & 7) == 0
                       ? 8
                       : ((reinterpret_cast<uintptr_t>(P.rasters) | P.canvas_stride) & 3) == 0 ? 4 : 1;
    unsigned carry = 0;
    for (int k = 0; k < p; k++) carry += (unsigned)part[warp - p + k];
    uint8_t* drow = P.rasters + (size_t)(r0 + q) * P.canvas_stride;
    if (P.rule == FT_NONZERO)
        band_part<FT_NONZERO>(area + q * pitch, drow, x0, x1, W, carry, al);
    else
        band_part<FT_EVENODD>(area + q * pitch, drow, x0, x1, W, carry, al);
}

// SrcOver of one call's colour from its mask onto a canvas that no tensor map fits (rows not on
// 16-byte boundaries): 1,024 pixels of a row per CTA, four loads in flight per thread.
constexpr int SR_PX = 4;
__global__ void __launch_bounds__(256) k_srcover_rows(uint8_t* canvas, unsigned stride, const uint8_t* mask,
                                                      unsigned mstride, int W, int r0, int nseg, unsigned clr) {
    const int r = r0 + (int)(blockIdx.x / nseg), x0 = (int)(blockIdx.x % nseg) * (256 * SR_PX) + threadIdx.x;
    unsigned* row = reinterpret_cast<unsigned*>(canvas + (size_t)r * stride);
    const uint8_t* m = mask + (size_t)r * mstride;
    unsigned d[SR_PX], a[SR_PX];
#pragma unroll
    for (int k = 0; k < SR_PX; k++) {
        const int x = x0 + 256 * k;
        d[k] = x < W ? row[x] : 0u;
        a[k] = x < W ? m[x] : 0u;
    }
#pragma unroll
    for (int k = 0; k < SR_PX; k++) {
        const int x = x0 + 256 * k;
        if (x < W && (a[k] || low_channels(d[k]))) row[x] = srcover_rgba(d[k], clr, a[k]);
    }
}

template <int NT>
cudaError_t launch_band(const KParams& p, cudaStream_t s) {
    const int smem = band_smem(NT, p.band_rows, (int)p.canvas_w);
    k_band_single<NT><<<p.n_bands, NT, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace

// As many warps as shared memory holds records for beside the band's cells.
cudaError_t launch_band_single(const KParams& p, int max_smem, cudaStream_t s) {
    if (band_smem(1024, p.band_rows, (int)p.canvas_w) <= max_smem) return launch_band<1024>(p, s);
    if (band_smem(512, p.band_rows, (int)p.canvas_w) <= max_smem) return launch_band<512>(p, s);
    return launch_band<256>(p, s);
}

cudaError_t launch_srcover_rows(uint8_t* canvas, uint32_t stride, const uint8_t* mask, uint32_t mstride, int W, int H,
                                int r0, unsigned clr, cudaStream_t s) {
    if (r0 >= H || W <= 0) return cudaSuccess;
    const int nseg = (W + 256 * SR_PX - 1) / (256 * SR_PX);
    k_srcover_rows<<<(H - r0) * nseg, 256, 0, s>>>(canvas, stride, mask, mstride, W, r0, nseg, clr);
    return cudaGetLastError();
}

cudaError_t take_check_bands(CheckState* s, bool reached) { return take_check(s, reached); }

cudaError_t setup_bands() {
    cudaError_t e = allow_smem((const void*)k_band_single<256>);
    if (e == cudaSuccess) e = allow_smem((const void*)k_band_single<512>);
    return e == cudaSuccess ? allow_smem((const void*)k_band_single<1024>) : e;
}

int band_single_smem(int band_rows, int width) { return band_smem(256, band_rows, width); }

}  // namespace ftk
