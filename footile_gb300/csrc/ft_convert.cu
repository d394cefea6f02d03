// ft_convert.cu — Rgba8p -> SRgba8 and Matte8 -> SGray8 on the device, and the float
// ordered SrcOver of coverage layers with its adjoint.
//
// footile plots in linear premultiplied Rgba8p / Matte8; its examples then convert with
// pix (`Raster::<SRgba8>::with_raster`, examples/fishy.rs:33; `Raster::<SGray8>`,
// examples/drop.rs:22): straight alpha (channel / alpha) and the sRGB transfer
// function.  The conversion of one channel depends only on (alpha, channel), so it is a
// 256 x 256 byte table the host builds once (correctly rounded sRGB encoding of
// channel / alpha, IEC 61966-2-1) and every thread reads from shared memory.
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/footile_gpu.h"

namespace ftc {

// A memory stream (8192 x 8192 Rgba8p: 537 MB, 79 us at the copy rate) held back by its lookups,
// three bytes from random words per pixel (3.4 accesses of the 32 banks each): what helps is
// warps, 64 per SM on two tables.  Matte8 reads only the row of alpha 255, which is held with a
// column of words per lane, so that lanes never meet.  Rasters without padding between the rows
// are one row.  24 warps per SM, three tables and a 64-bit divide per 16 bytes: 110.8 us; this way
// 90.6 us (two loads of a thread in flight 99 us; the alpha 255 row in columns for Rgba8p too,
// beside the table, 120 us).  Matte8 45 / 35 us.  1531 x 1117, whose rows start at any word, byte
// by byte 53 us, as one row 18 us.
constexpr int CBLOCK = 1024;
constexpr int FULL_ROW = 64 * 32 * 4;  // the columns
__host__ __device__ constexpr int convert_smem(bool rgba) { return rgba ? 256 * 256 : FULL_ROW; }

__device__ __forceinline__ unsigned byte_at(unsigned addr) {  // of shared memory
    unsigned v;
    asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// lut: the table (a * 256 + c), for Matte8 the lane's column, as a shared address
template <bool RGBA>
__device__ __forceinline__ unsigned convert_e(unsigned p, unsigned lut) {
    const unsigned c0 = p & 0xFFu, c1 = (p >> 8) & 0xFFu, c2 = (p >> 16) & 0xFFu, c3 = p >> 24;
    if (RGBA) {
        const unsigned row = lut + (c3 << 8);
        return byte_at(row + c0) | (byte_at(row + c1) << 8) | (byte_at(row + c2) << 16) | (p & 0xFF000000u);
    }
    auto at = [&](unsigned c) { return byte_at(lut + (((c & 0xFCu) << 5) | (c & 3u))); };
    return at(c0) | (at(c1) << 8) | (at(c2) << 16) | (at(c3) << 24);
}
template <bool RGBA>
__device__ __forceinline__ uint4 convert_e(uint4 v, unsigned lut) {
    return make_uint4(convert_e<RGBA>(v.x, lut), convert_e<RGBA>(v.y, lut), convert_e<RGBA>(v.z, lut),
                      convert_e<RGBA>(v.w, lut));
}

// `n` elements of T per row, from byte `off` of each
template <bool RGBA, class T>
__device__ __forceinline__ void convert_rows(const uint8_t* src, uint64_t src_stride, uint8_t* dst, uint64_t dst_stride,
                                             uint64_t off, uint64_t n, uint32_t h, unsigned lut) {
    const uint64_t total = n * h;
    for (uint64_t i = (uint64_t)blockIdx.x * CBLOCK + threadIdx.x; i < total; i += (uint64_t)gridDim.x * CBLOCK) {
        uint64_t y = 0;
        if (h > 1) y = total >> 32 ? i / n : (uint32_t)i / (uint32_t)n;
        const uint64_t at = off + (i - y * n) * sizeof(T);
        *reinterpret_cast<T*>(dst + y * dst_stride + at) =
            convert_e<RGBA>(*reinterpret_cast<const T*>(src + y * src_stride + at), lut);
    }
}

template <bool RGBA>
__global__ void __launch_bounds__(CBLOCK, 2) k_convert(const uint8_t* src, uint32_t src_stride, uint8_t* dst,
                                                       uint32_t dst_stride, uint32_t w, uint32_t h,
                                                       const uint8_t* __restrict__ lut_g) {
    extern __shared__ __align__(16) uint8_t smem[];
    if (RGBA) {
        for (int i = threadIdx.x; i < 256 * 256 / 16; i += CBLOCK)
            reinterpret_cast<uint4*>(smem)[i] = reinterpret_cast<const uint4*>(lut_g)[i];
    } else {
        for (int i = threadIdx.x; i < FULL_ROW / 4; i += CBLOCK)
            reinterpret_cast<unsigned*>(smem)[i] = reinterpret_cast<const unsigned*>(lut_g + 0xFF00)[i >> 5];
    }
    __syncthreads();
    const unsigned lut = (unsigned)__cvta_generic_to_shared(smem) + (RGBA ? 0 : 4 * (threadIdx.x & 31));
    uint64_t row_bytes = RGBA ? 4ull * w : w;
    if (src_stride == row_bytes && dst_stride == row_bytes) {
        row_bytes *= h;
        h = 1;
    }
    const uintptr_t align = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst) |
                            (h > 1 ? (uintptr_t)(src_stride | dst_stride) : 0);
    const uint64_t vec = align & 15 ? 0 : row_bytes / 16, words = align & 3 ? 0 : (row_bytes - vec * 16) / 4;
    if (vec) convert_rows<RGBA, uint4>(src, src_stride, dst, dst_stride, 0, vec, h, lut);
    if (words) convert_rows<RGBA, unsigned>(src, src_stride, dst, dst_stride, vec * 16, words, h, lut);
    // the last bytes of Matte8 rows; all of rows that start at any byte
    const uint64_t done = vec * 16 + words * 4, tail = row_bytes - done, n_tail = tail * h;
    for (uint64_t t = (uint64_t)blockIdx.x * CBLOCK + threadIdx.x; t < n_tail; t += (uint64_t)gridDim.x * CBLOCK) {
        const uint64_t y = t / tail, b = done + (t - y * tail);
        const uint8_t* s = src + y * src_stride;
        uint8_t* d = dst + y * dst_stride;
        if (!RGBA) {
            d[b] = lut_g[0xFF00 | s[b]];
        } else {
            const unsigned a = s[b | 3];
            d[b] = (b & 3) == 3 ? (uint8_t)a : smem[(a << 8) | s[b]];
        }
    }
}

cudaError_t setup_convert() {
    return cudaFuncSetAttribute(k_convert<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, convert_smem(true));
}
int convert_block() { return CBLOCK; }
int convert_blocks_per_sm(int src_fmt) {
    const bool rgba = src_fmt == FT_RGBA8P;
    auto kern = rgba ? k_convert<true> : k_convert<false>;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, CBLOCK, convert_smem(rgba)) != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

cudaError_t launch_convert(int src_fmt, const uint8_t* src, uint32_t src_stride, uint8_t* dst, uint32_t dst_stride,
                           uint32_t w, uint32_t h, const uint8_t* lut, int grid, cudaStream_t s) {
    const bool rgba = src_fmt == FT_RGBA8P;
    auto kern = rgba ? k_convert<true> : k_convert<false>;
    kern<<<grid, CBLOCK, convert_smem(rgba), s>>>(src, src_stride, dst, dst_stride, w, h, lut);
    return cudaGetLastError();
}


// ------------------------------------------------------ ordered SrcOver adjoint
// The composite of an ordered batch in float: layer n (coverage cov_n, premultiplied
// colour c_n with alpha a_n, as footile's pix SrcOver, fig.rs:637-643) gives
//   C_n = c_n * cov_n + C_{n-1} * (1 - a_n * cov_n).
// With G = dLoss/dC_N, the factor (1 - a_n cov_n) is one scalar for all four channels,
// so dLoss/dcov_n = P_n * (G . c_n - a_n * E_{n-1}) with P_n the product of the later
// factors and E_n = G . C_n following the same recurrence as C (scalar).  Backward:
// one pass forward for E (recomputed, nothing kept from the forward call), written
// into the gradient planes, then one pass backward for P.  No division, so opaque
// layers (factor 0) are exact.  One thread per pixel; planes are n_layers x n_px floats.
// Bound by the planes' stream from memory, and below some 300,000 pixels by the latency of a pixel's
// chain: the recurrence goes SB layers at a time, the loads of the next SB in flight meanwhile.  A
// thread takes one pixel, a CTA SO_BLOCK of them; how many fit a round of resident CTAs chooses the
// shape (launch_srcover).  400 layers of mostly empty coverage, forward / backward of some / of all:
// 100,000 pixels 53 / 131 / 147 us, 180,000 67 / 196 / 300, 260,000 96 / 266 / 375, 1,000,000
// 289 / 893 / 1,370; loads and recurrence in turn 111 / 131 / 153, 112 / 225 / 313, 120 / 273 / 385,
// 447 / 944 / 1,415.
constexpr int SB = 8;
constexpr int SO_BLOCK = 128;

// `step(k, v)` for k = 0 .. n - 1 in turn, v[u] = the SB coverages from layer(k) on (layer(k) +
// dir * u), loaded a step ahead
template <int SB, class Step>
__device__ __forceinline__ void stream_layers(const float* cov, uint64_t plane, uint32_t n, uint32_t first, int dir,
                                              Step step) {
    const float* at = cov + (uint64_t)first * plane;
    const int64_t inc = dir < 0 ? -(int64_t)plane : (int64_t)plane;
    float nx[SB];
    if (n) {
#pragma unroll
        for (int u = 0; u < SB; u++) nx[u] = __ldcs(at + u * inc);
    }
    for (uint32_t k = 0; k < n; k++) {
        float v[SB];
#pragma unroll
        for (int u = 0; u < SB; u++) v[u] = nx[u];
        at += SB * inc;
        if (k + 1 < n) {
#pragma unroll
            for (int u = 0; u < SB; u++) nx[u] = __ldcs(at + u * inc);
        }
        step(k, v);
    }
}

// A step of SB layers: 8 take 40 registers, 12 CTAs per SM; 4 take 32 and 16.
template <int SB>
__global__ void k_srcover_fwd(const float* __restrict__ cov, uint32_t n_layers, uint64_t plane,
                              const float4* __restrict__ clr, const float4* __restrict__ init,
                              float4* __restrict__ out, uint32_t n_px) {
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_px;
         p += (uint64_t)gridDim.x * blockDim.x) {
        float4 c = init ? init[p] : make_float4(0.f, 0.f, 0.f, 0.f);
        auto layer = [&](uint32_t n, float v) {
            if (v == 0.0f) return;
            const float4 k = clr[n];
            const float f = 1.0f - k.w * v;
            c = make_float4(k.x * v + c.x * f, k.y * v + c.y * f, k.z * v + c.z * f, k.w * v + c.w * f);
        };
        stream_layers<SB>(cov + p, plane, n_layers / SB, 0, 1, [&](uint32_t k, const float* v) {
#pragma unroll
            for (int u = 0; u < SB; u++) layer(k * SB + u, v[u]);
        });
        for (uint32_t n = n_layers / SB * SB; n < n_layers; n++) layer(n, __ldcs(cov + (uint64_t)n * plane + p));
        out[p] = c;
    }
}

// PARTIAL: dLoss/dcov only where 0 < cov < 1 (elsewhere the plane is neither read nor
// written) — all a NonZero coverage adjoint needs, since dcov/dS is 0 at cov 0 and 1.
template <bool PARTIAL, int PER_SM>
__global__ void __launch_bounds__(SO_BLOCK, PER_SM) k_srcover_bwd(const float* __restrict__ cov, uint32_t n_layers, uint64_t plane,
                              const float4* __restrict__ clr, const float4* __restrict__ init,
                              const float4* __restrict__ grad_out, float* __restrict__ grad_cov,
                              float4* __restrict__ grad_init, uint32_t n_px) {
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_px;
         p += (uint64_t)gridDim.x * blockDim.x) {
        const float4 g = grad_out[p];
        const float4 c0 = init ? init[p] : make_float4(0.f, 0.f, 0.f, 0.f);
        float e = g.x * c0.x + g.y * c0.y + g.z * c0.z + g.w * c0.w;
        auto keep = [](float v) { return !PARTIAL || (v > 0.0f && v < 1.0f); };
        // E_{n-1} = g . C_{n-1} into the gradient plane
        auto up = [&](uint32_t n, float v) {
            if (keep(v)) grad_cov[(uint64_t)n * plane + p] = e;
            if (v == 0.0f) return;
            const float4 k = clr[n];
            e = (g.x * k.x + g.y * k.y + g.z * k.z + g.w * k.w) * v + e * (1.0f - k.w * v);
        };
        stream_layers<SB>(cov + p, plane, n_layers / SB, 0, 1, [&](uint32_t k, const float* v) {
#pragma unroll
            for (int u = 0; u < SB; u++) up(k * SB + u, v[u]);
        });
        for (uint32_t n = n_layers / SB * SB; n < n_layers; n++) up(n, __ldcs(cov + (uint64_t)n * plane + p));
        // then the suffix products P, last layer first
        float P = 1.0f;
        auto down = [&](uint32_t n, float v, float en) {
            const float4 k = clr[n];
            if (keep(v)) grad_cov[(uint64_t)n * plane + p] = P * ((g.x * k.x + g.y * k.y + g.z * k.z + g.w * k.w) - k.w * en);
            P *= 1.0f - k.w * v;
        };
        stream_layers<SB>(cov + p, plane, n_layers / SB, n_layers - 1, -1, [&](uint32_t k, const float* v) {
            const uint32_t m = n_layers - k * SB;
            float en[SB];
#pragma unroll
            for (int u = 0; u < SB; u++) en[u] = keep(v[u]) ? grad_cov[(uint64_t)(m - 1 - u) * plane + p] : 0.0f;
#pragma unroll
            for (int u = 0; u < SB; u++) down(m - 1 - u, v[u], en[u]);
        });
        for (uint32_t m = n_layers % SB; m > 0; m--) {
            const float v = __ldcs(cov + (uint64_t)(m - 1) * plane + p);
            down(m - 1, v, keep(v) ? grad_cov[(uint64_t)(m - 1) * plane + p] : 0.0f);
        }
        if (grad_init) grad_init[p] = make_float4(g.x * P, g.y * P, g.z * P, g.w * P);
    }
}

cudaError_t launch_srcover(bool backward, const float* cov, uint32_t n_layers, uint64_t plane, const float4* clr,
                           const float4* init, float4* out, const float4* grad_out, float* grad_cov,
                           float4* grad_init, uint32_t n_px, int sm_count, cudaStream_t s, bool partial) {
    // CTAs that a canvas needs, and that a round takes with `per_sm` on an SM
    const unsigned ctas = (unsigned)(((uint64_t)n_px + SO_BLOCK - 1) / SO_BLOCK);
    auto round = [&](unsigned per_sm) { return per_sm * (unsigned)sm_count; };
    // under few layers a pixel costs less than a CTA's launch: some take several
    const unsigned grid = n_layers < SB && ctas > round(32) ? round(32) : ctas;
    if (backward) {
        // 8 per SM with 64 registers; 9 with 56, spilled, where the ninth completes the one round.  172,800
        // pixels, 9 / 8 on 152 SMs: coverage of some 191 / 196 us, of all 239 / 295; elsewhere 8 are
        // faster (100,000 158 / 147, 220,000 352 / 330, 180,000 of some 213 / 196)
        const bool nine = ctas > round(8) && ctas <= round(9);
        auto kern = partial ? (nine ? k_srcover_bwd<true, 9> : k_srcover_bwd<true, 8>)
                            : (nine ? k_srcover_bwd<false, 9> : k_srcover_bwd<false, 8>);
        kern<<<grid, SO_BLOCK, 0, s>>>(cov, n_layers, plane, clr, init, grad_out, grad_cov, grad_init, n_px);
    } else {
        // steps of 4 layers with 16 CTAs per SM where that is one round and 12 are not (260,000 pixels, 4 / 8
        // layers a step 96 / 108 us; 220,000, one round either way, 83 / 81; 1,000,000, the rest among
        // several rounds, 309 / 289), and under fewer layers than a step of 8
        const bool four = n_layers < SB || (ctas > round(12) && ctas <= round(16));
        auto kern = four ? k_srcover_fwd<4> : k_srcover_fwd<SB>;
        kern<<<grid, SO_BLOCK, 0, s>>>(cov, n_layers, plane, clr, init, out, n_px);
    }
    return cudaGetLastError();
}

}  // namespace ftc
