// ft_kernels.cuh — launch interface between the C ABI (ft_capi.cu) and the kernels.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/footile_gpu.h"

namespace ftk {

constexpr int BLOCK = 256;                 // threads per CTA
constexpr int NWARP = BLOCK / 32;
constexpr int RAW_CAP = 2048;              // raw (pre-dedupe) vertices per compaction window
constexpr int PT_CAP = FT_MAX_POINTS;      // vertices kept per figure (u16 vertex ids)
constexpr int OUT_CAP = 2 * RAW_CAP;       // stroke outline points staged per window

// One unit of the device work queue: rows [row_begin, row_end) of one path's
// raster, rasterised `band_rows` rows at a time.
struct WorkItem {
    uint32_t path;
    uint32_t row_begin;
    uint32_t row_end;
    uint32_t band_rows;
};

// One non-horizontal edge of a figure (footile fig.rs:47-66), 32 bytes.  `ed` is
// +1 when the edge direction equals the figure direction, -1 otherwise, 0 for
// "no edge" (horizontal or degenerate segment).
struct __align__(16) EdgeRec {
    int y_upper, y_lower, x_bot0, inv_slope;
    int step_pix, ed, start_row, end_row;
};

// One stroke sub-path (stroker.rs:31-40).
struct SubRec {
    int start;     // first stroke point
    int n;         // points
    int joined;    // joined ends
    int len;       // SubStroke::len() (u16 arithmetic)
    int item_off;  // first outline item of this sub-stroke
    int pad[3];
};

// Per-CTA scratch in global memory, private to one resident CTA and reused for
// every work item it takes (stays L2-resident for small figures).  Every array
// starts on a 256-byte boundary.
constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t SCR_PTS = 0;                                                   // int2[PT_CAP] vertices
constexpr size_t SCR_SS = align256(SCR_PTS + (size_t)PT_CAP * sizeof(int2));    // int[PT_CAP] sub-figure starts
constexpr size_t SCR_EDGES = align256(SCR_SS + (size_t)PT_CAP * sizeof(int));   // EdgeRec[PT_CAP]
constexpr size_t SCR_SPTS = align256(SCR_EDGES + (size_t)PT_CAP * sizeof(EdgeRec));  // float4[PT_CAP] stroke points
constexpr size_t SCR_SUBS = align256(SCR_SPTS + (size_t)PT_CAP * sizeof(float4));    // SubRec[PT_CAP] sub-strokes
constexpr size_t SCR_SOFF = align256(SCR_SUBS + (size_t)PT_CAP * sizeof(SubRec));    // int[2*PT_CAP+8] offsets
// Raw (pre-dedupe) vertices of one chunk of ops, emitted once by all threads and
// compacted window by window (CTA figure builds): positions as int2 (fills) or float4
// with the width (strokes), sub-figure start flags, stroke join flags, source ops.
constexpr int RAWG = 32768;
constexpr size_t SCR_RAWG = align256(SCR_SOFF + (size_t)(2 * PT_CAP + 8) * sizeof(int));  // float4[RAWG]
constexpr size_t SCR_RSG = align256(SCR_RAWG + (size_t)RAWG * 16);                         // u8[RAWG]
constexpr size_t SCR_JPG = align256(SCR_RSG + (size_t)RAWG);                               // u8[RAWG]
constexpr size_t SCR_OPIG = align256(SCR_JPG + (size_t)RAWG);                              // int[RAWG]
constexpr size_t SCRATCH_BYTES_PER_CTA = align256(SCR_OPIG + (size_t)RAWG * sizeof(int));

// Scratch layout of one CTA figure build for figures of up to `cap` vertices: the
// SCR_* layout above for footile's cap, larger for the un-capped extension (fills).
struct ScrLayout {
    size_t pts, ss, edges, spts, subs, soff, rawg, rsg, jpg, opig, bytes;
};
constexpr ScrLayout scr_layout(size_t cap) {
    ScrLayout L{};
    L.pts = 0;
    L.ss = align256(L.pts + cap * sizeof(int2));
    L.edges = align256(L.ss + cap * sizeof(int));
    L.spts = align256(L.edges + cap * sizeof(EdgeRec));
    L.subs = align256(L.spts + (size_t)PT_CAP * sizeof(float4));
    L.soff = align256(L.subs + (size_t)PT_CAP * sizeof(SubRec));
    L.rawg = align256(L.soff + (size_t)(2 * PT_CAP + 8) * sizeof(int));
    L.rsg = align256(L.rawg + (size_t)RAWG * 16);
    L.jpg = align256(L.rsg + (size_t)RAWG);
    L.opig = align256(L.jpg + (size_t)RAWG);
    L.bytes = align256(L.opig + (size_t)RAWG * sizeof(int));
    return L;
}
static_assert(scr_layout(PT_CAP).bytes == SCRATCH_BYTES_PER_CTA && scr_layout(PT_CAP).rawg == SCR_RAWG &&
                  scr_layout(PT_CAP).edges == SCR_EDGES && scr_layout(PT_CAP).subs == SCR_SUBS,
              "scratch layouts agree");
// Largest figure of the un-capped extension (ft_set_figure_cap).
constexpr uint32_t FIG_CAP_MAX = 1u << 26;

// Grid-wide figure build of one fill path (launch_grid_build): per-op and per-raw-vertex
// arrays in one device buffer laid out by gb_layout.
constexpr int GB_PER = 4;                      // raw vertices per thread of the tile kernels
constexpr int GB_TILE = GB_PER * BLOCK;        // raw vertices per tile
constexpr int GB_TOP_BLOCKS = 512;             // CTAs of the top-vertex search
// An op's curve walk is split at depth d0 over 2^d0 threads: 8, or a warp while the ops are few
// enough for all warps to be resident (GB_WIDE_OPS).  8 / 16 / 32 threads on the 2,048 ops that
// complete a capped figure: 4096 x 4096 scene 188 / 178 / 168 us, its stroke 288 / 280 / 268;
// on 3,780 ops, poster of 1531 x 1117 119 / 116 / 116 us.
constexpr int GB_WIDE_OPS = 8192;
constexpr __host__ __device__ int gb_d0(size_t n_ops) { return n_ops <= (size_t)GB_WIDE_OPS ? 5 : 3; }
constexpr __host__ __device__ int gb_ctas(size_t n_ops) { return (int)(((n_ops << gb_d0(n_ops)) + BLOCK - 1) / BLOCK); }
constexpr int GB_STATE = 512;                  // bytes of counters at the front (gb_layout)
constexpr long long GB_RAW_MAX = 1ll << 29;    // raw vertices the grid build takes at most
struct GridBuildBufs {
    const ft_op* ops;   // the path's ops
    int n_ops;
    const float* s_width;  // pen width before the path (device)
    int raw_cap;        // raw vertices the arrays hold (a multiple of GB_TILE)
    unsigned* done;     // [8] tickets: the last CTA of a kernel to finish runs its scan
    long long* n_raw;   // raw vertices of the path
    int* count;         // vertices kept
    int4* opa;          // per 256 ops: last Move/Line/Quad/Cubic/Close op, last PenWidth op, last Close/Move op
    int* opw;           // per op: last PenWidth op at or before it in its 256 (strokes)
    int d0;             // gb_d0(n_ops)
    long long* opn;     // per block of the walks: raw vertices
    int2* opi;          // per op: last Move/Line/Quad/Cubic/Close op before it in its 256, raw offset in its block
    int* opl;           // per op and lane: the lane's raw offset in the op
    int2* raw;          // raw vertices, 16.16
    unsigned char* fl;  // per raw vertex: 1 = starts a sub-figure
    unsigned char* kp;  // per raw vertex: 1 = kept, 2 = pops its sub-figure's first vertex
    int* rk;            // per raw vertex: the first raw vertex of its sub-figure
    int* tr_all;        // the tile starts of both builds, n_tr of them: k_gb_ops resets them
    int n_tr;
    int* tr;            // per tile: last sub-figure start
    int4* tp;           // per tile: position aggregate (kept - popped, runs, max prefix)
    int4* top;          // per CTA of the top-vertex search: min (y, x, id)
    int* final_flag;    // nullable: set when the cap is reached (the figure is complete)
    const int* skip;    // nullable: the kernels after k_gb_ops do nothing when *skip is set
};
// Grid-wide build of one stroke path (the stroker's points, sub-strokes and outline, then
// the outline's figure through the fill build's k_gb_keep / k_gb_write / k_gb_top).
constexpr int GS_ITEMS_CAP = 6 * PT_CAP + 256;  // outline items of 65,535 stroke points at most
struct GridStrokeBufs {
    int sraw_cap;        // raw stroke points the arrays hold (a multiple of GB_TILE)
    long long* n_sraw;   // raw stroke points of the path
    int* st;             // [0] points kept, [1] sub-strokes, [2] op of the last kept point, [3] last
                         // Move/Line/Quad/Cubic/Close op, [4] last Close/Move op, [5] outline items,
                         // [6] the 65,535-point cap was reached
    unsigned* done;      // [8] tickets
    float4* raw4;        // raw stroke points: x, y, width
    unsigned char* sfl;  // per raw point: 1 starts a sub-stroke, 2 its op is not a Move
    int* sopi;           // per raw point: its op
    int2* stile;         // per tile of raw points: kept, sub-stroke starts
    int* subt;           // per 256 sub-strokes: outline items
    int2* itoff;         // per outline item: raw offset in its 256; raw vertices, the top bit when it starts a run
    float4* itp;         // per outline item: its first two points
    int* itc;            // per 256 outline items: raw vertices
    int* final_flag;     // nullable: set when the 65,535-point cap is reached (the points are complete)
    const int* skip;     // nullable: the stroke point kernels do nothing when *skip is set
};
struct GbLayout {
    size_t state, opa, opw, opn, opi, opl, raw, fl, kp, rk, tr, tr2, tp, top;
    size_t raw4, sfl, sopi, stile, subt, itoff, itc, itp, bytes;
};
constexpr GbLayout gb_layout(size_t n_ops, size_t raw_cap, size_t sraw_cap = 0) {
    GbLayout g{};
    const size_t nbo = (n_ops + BLOCK - 1) / BLOCK, nbw = (size_t)gb_ctas(n_ops),
                 ntiles = raw_cap / GB_TILE;
    // two builds' done[8] at 0 / 128, n_raw at 32 / 160, count at 40 / 168, final at 44 / 172;
    // a stroke build's st[] at 128, n_sraw at 160, done[] at 192, its probe's n_sraw at 256,
    // done[] at 288, final at 320
    g.state = 0;
    g.opa = GB_STATE;
    g.opw = align256(g.opa + nbo * 16);
    g.opn = align256(g.opw + n_ops * 4);
    g.opi = align256(g.opn + nbw * 8);
    g.opl = align256(g.opi + n_ops * 8);
    g.raw = align256(g.opl + (n_ops << gb_d0(n_ops)) * 4);
    g.fl = align256(g.raw + raw_cap * 8);
    g.kp = align256(g.fl + raw_cap);
    g.rk = align256(g.kp + raw_cap);
    g.tr = align256(g.rk + raw_cap * 4);
    g.tr2 = align256(g.tr + ntiles * 4);
    g.tp = align256(g.tr2 + ntiles * 4);
    g.top = align256(g.tp + ntiles * 16);
    g.raw4 = align256(g.top + (size_t)GB_TOP_BLOCKS * 16);
    g.sfl = align256(g.raw4 + sraw_cap * 16);
    g.sopi = align256(g.sfl + sraw_cap);
    g.stile = align256(g.sopi + sraw_cap * 4);
    g.subt = align256(g.stile + sraw_cap / GB_TILE * 8);
    g.itoff = align256(g.subt + (sraw_cap ? (size_t)(PT_CAP / BLOCK + 1) * 4 : 0));
    g.itc = align256(g.itoff + (sraw_cap ? (size_t)GS_ITEMS_CAP * 8 : 0));
    g.itp = align256(g.itc + (sraw_cap ? (size_t)(GS_ITEMS_CAP / BLOCK + 1) * 4 : 0));
    g.bytes = align256(g.itp + (sraw_cap ? (size_t)GS_ITEMS_CAP * 16 : 0));
    return g;
}

struct KParams {
    const ft_op* ops;
    const ft_path_desc* paths;
    const WorkItem* items;   // CTA work items (large paths, row ranges)
    uint32_t n_items;
    const WorkItem* items_w; // tile rasteriser's work items
    uint32_t n_items_w;
    uint32_t* overflow;      // tile items handed over to the CTA kernel (single: a flag per CTA)
    uint32_t* queue;         // [0]: next CTA item, [1]: next tile item, [2]: overflow count
    uint8_t* rasters;
    int32_t* status;         // per path, atomicMax of FT_ERR_* codes
    float* sw_out;           // per path pen width after the call (nullable)
    int host_rasters;        // rasters are mapped host memory: Matte8 rows go out as aligned words
    int single, rows_per;    // one path, `d`, CTA b drawing rows b * rows_per .. (as TileParams)
    ft_path_desc d;
    const float* sw_chain;   // nullable: initial pen width of every path
    unsigned char* scratch;  // gridDim.x * SCRATCH_BYTES_PER_CTA bytes
    float xf[6];
    float tol, tol_sq;
    int join;
    float miter_limit;
    float miter_g;           // ft_miter_angle(miter_limit): the miter decision's threshold on |th/2|
    int rule;
    int fmt;
    int stroke;
    int smem_bytes;
    // ordered composite of all paths onto one raster (ft_composite_batch)
    uint32_t canvas_w, canvas_h, canvas_stride;
    int band_rows;               // rows per band
    int n_bands;
    EdgeRec* pool;               // binned edges of all paths
    unsigned long long* pool_used;  // bump counter (edges)
    unsigned long long pool_cap;    // edges
    int* bandoff;                // per path: n_bands + 1 offsets into its pool run
    int4* crec;                  // per path: rowbegin, tmin, pool offset lo, pool offset hi
    // figure builds of the ordered compositor (k_cbuild): vertex cap and scratch layout
    int pt_cap;                  // PT_CAP, or more for un-capped fills
    ScrLayout L;                 // scr_layout(pt_cap); gridDim.x * L.bytes of scratch
    // one path (split_bin): k_cbuild stops after the figure and its direction, the
    // grid-wide kernels below build and bin its edges
    int split_bin;
    int4* fig_state;             // count, direction, top row, edges fit the pool
    int* bin_hist;               // n_bands counts, then n_bands fill cursors
    // Rgba8p tile compositor (k_ctile): segment width in pixels (128 or a multiple of
    // 256, at most 1,024) and whether the canvas is staged by TMA through the tensor map passed
    // beside these
    int seg_w;
    int use_tma;
    int bin_segs;         // segments of seg_w pixels that a band's edges are binned by (1: not)
    int tile_batches;     // batches the calls are cut into (k_ctile)
    unsigned* tile_done;  // per tile: batches done, then per tile: rounds of 32 calls that warps are through with
    unsigned char* summary;  // a single call's page-locked read-back: edges binned, crec[0] at 16, the
                             // grid build's counters at GB_STATE
    // one fill path built over the whole GPU (launch_grid_build) instead of by k_cbuild
    GridBuildBufs gb;
    GridStrokeBufs gs;  // and the stroker's part of one stroke path (launch_grid_stroke)
};

// The tile rasteriser (ft_tile.cu): fills of small canvases, one CTA of TILE_THREADS per
// path, of TILE_THREADS_TINY where all of a batch's are tiny, or of TILE_THREADS_FEW per row range
// of a path when there are few paths.
constexpr int TILE_THREADS = 128, TILE_THREADS_TINY = 32, TILE_THREADS_FEW = 512;
// Tiny: TILE_TINY_PATHS canvases per SM and more, up to TILE_TINY_SIDE a side under TILE_TINY_OPS ops
// at most, where four warps wait for one another more than they share.  Four warps / one a path,
// 65,536 canvases of 8 x 8 under 3 lines 389 / 144 us, of 24 x 24 under 14 curves 700 / 434, zoomed in
// 1,000 times 5,764 / 5,560.  Of fewer canvases each path's chain sets the time, longer by one warp:
// 20,000 of the same 223 / 146, zoomed in 1,807 / 1,847, 8,000 98 / 68, 763 / 841, 1,200 25 / 29, 156 / 262;
// of more ops the scratch of so many CTAs holds too little: 65,536 under 30 curves 956 / 742,
// zoomed in 12,031 / 70,407 (handed over).
constexpr int TILE_TINY_SIDE = 24, TILE_TINY_OPS = 16, TILE_TINY_PATHS = 128;
constexpr int TILE_MAX_SIDE = 512;                      // canvases up to this width and height (batches)
constexpr int TILE_CAP = 32768, TILE_CAP_TINY = 8192, TILE_CAP_FEW = 65504;  // segment slots per CTA (at most the vertex cap)
static_assert(TILE_CAP % 32 == 0 && TILE_CAP_TINY % 32 == 0 && TILE_CAP_FEW % 32 == 0 && TILE_CAP_FEW <= PT_CAP, "a tile figure never reaches the cap");
// Rows of a single call's ranges, a CTA each: 8, and no more ranges than SMs.  Two builds on one SM
// take longer than one with twice the rows to draw: 30,000 curves on 500 x 2000 in 250 / 143 ranges
// on 152 SMs 2,533 / 1,814 us, 500 curves on 64 x 16000 in 302 / 151 2,034 / 1,413 us.
inline __host__ __device__ int single_rows(int h, int sms) {
    const int even = (h + (sms > 1 ? sms : 1) - 1) / (sms > 1 ? sms : 1);
    return even > 8 ? even : 8;
}
// Cells from one row of a band to the next: three spare cells (a walk of four cells may run
// past the raster's last), a multiple of eight.
__host__ __device__ constexpr int tile_pitch(int w) { return (w + 3 + 7) & ~7; }
constexpr size_t tile_scratch(int cap) { return align256((size_t)cap * 16 + (size_t)cap / 8); }
struct TileParams {
    const ft_op* ops;
    const ft_path_desc* paths;
    const WorkItem* items;
    uint32_t n_items;
    uint32_t* overflow;      // items handed to k_raster (single: per CTA, whether its rows are)
    uint32_t* queue;         // [1]: next item, [2]: overflow count
    // one path (ft_fill): CTA b draws rows b * rows_per .. of it; the descriptor is `d`, nothing is
    // uploaded or reset before the launch
    int single, rows_per;
    ft_path_desc d;
    uint8_t* rasters;
    int32_t* status;         // per path, atomicMax of FT_ERR_* codes
    float* sw_out;           // per path pen width after the call (nullable)
    const float* sw_chain;   // nullable: initial pen width of every path
    unsigned char* scratch;  // gridDim.x * tile_scratch(cap) bytes
    int cap;                 // segment slots per CTA
    int area_ints;           // cells of a band (a multiple of 8, at least one row of every item)
    int host_rasters;        // rasters are mapped host memory
    int rule, fmt;
    float xf[6];
    float tol, tol_sq;
};
// A row of a segment goes to 2^item_shift lanes of CELLS cells each.  `cells`: the row's longest
// walk; of a raster W pixels wide it needs no more than W (cells right of the raster are dropped,
// those left of it are one): 3,000 canvases of 64 x 64 under flat segments of 32,000 pixels 3,440 us
// by the walk alone, 255 us this way, 270 us with one lane a row.
constexpr int CELLS = 4;
inline __host__ __device__ int item_shift(int cells, int W) {
    const int more = ((cells < W ? cells : W) - 1) / CELLS;
#ifdef __CUDA_ARCH__
    return 32 - __clz(more);
#else
    int s = 0;
    while (more >> s) s++;
    return s;
#endif
}
int tile_smem(int threads, int area_ints, bool staged);
// What one launch of the tile rasteriser runs with.
struct TilePlan {
    int threads = TILE_THREADS, cap = TILE_CAP;
    int few_area = 8;    // with TILE_THREADS_FEW: the largest item's cells, up to 96 KB
    int few_staged = 8;  // the same where rows are staged
    // Rgba8p and host rows are staged as bytes
    static bool staged(int fmt, bool host) { return host || fmt == FT_RGBA8P; }
    // Batches: the cells that leave room for eight CTAs per SM.  65,536 glyphs with 2,560 /
    // 3,328 / 4,096 / 4,992 cells (the last seven CTAs): 4.75 / 4.46 / 4.29 / 4.34 ms.
    // Tiny: 32 CTAs per SM.
    int area(int fmt, bool host) const {
        if (threads == TILE_THREADS_TINY) return staged(fmt, host) ? 768 : 1000;
        if (threads == TILE_THREADS_FEW) return staged(fmt, host) ? few_staged : few_area;
        return staged(fmt, host) ? 3712 : 4736;
    }
    int smem(int fmt, bool host) const { return tile_smem(threads, area(fmt, host), staged(fmt, host)); }
};
int tile_blocks_per_sm(int threads, int smem);
cudaError_t launch_tile(const TileParams& p, int threads, int grid, int smem, cudaStream_t s);

// Ordered composite: per-path figure build and edge binning, then one CTA per band.
// `few_ctas`: at most one CTA per SM — prefer L1 over shared memory (the curve walks'
// stacks are in local memory).
cudaError_t launch_composite_build(const KParams& p, int grid, int smem_bytes, cudaStream_t s, bool few_ctas);
cudaError_t launch_composite_bands(const KParams& p, int smem_bytes, cudaStream_t s);
// Rgba8p: tiles of band_rows x seg_w pixels, canvas staged through `tmap` when use_tma.
// p.tile_done: 2 * composite_tiles(p) words, p.queue[3] zero.
cudaError_t launch_composite_tiles(KParams p, const CUtensorMap& tmap, int sm_count, cudaStream_t s);
int composite_tiles(const KParams& p);
// Waits of the tile compositor end after this many polls in which the work waited for has not moved
// (64 s and more of polling).  Polls and not the clock: neither calls that take long nor a GPU
// given to others meanwhile may fail a composite.
constexpr unsigned CT_POLLS_TILE = 1u << 27;  // of half a microsecond and more
constexpr unsigned CT_POLLS_SMEM = 1u << 31;  // of some 60 cycles
struct Patience {
    unsigned seen = 0, polls = 0;
    // after a poll that found `moved`, any word that the work waited for changes as it goes on
    __host__ __device__ bool ends(unsigned moved, unsigned limit) {
        if (moved != seen) {
            seen = moved;
            polls = 0;
        }
        return ++polls > limit;
    }
};
constexpr int CT_MAX_SEGS = 4;  // segments of a row in one tile
// Edges of a run of `n` that a warp asks L1 for ahead, one a lane.  A call may have none in a
// warp's bin, and the last run of the pool ends where the pool may end: never past the run.
constexpr __host__ __device__ int ct_ahead(int n) { return n < 32 ? n : 32; }
int composite_tile_smem(int band_rows, int bin_segs, int seg_w, bool staged);
int composite_tile_rows(int band_rows, int bin_segs);  // rows of a tile (and of its tensor-map boxes)
// SrcOver of one call's colour onto the canvas rows r0.. from its Matte8 coverage `mask`
// (both as 2-D tensor maps with boxes of SO_COLS x SO_ROWS elements: the kernel's stage
// size and its expected transaction bytes derive from the same two constants), streamed
// by TMA.
constexpr int SO_ROWS = 8, SO_COLS = 256;
cudaError_t launch_srcover_mask(const CUtensorMap& canvas, const CUtensorMap& mask, int W, int H, int r0,
                                unsigned clr, int32_t* status, int sm_count, cudaStream_t s);
// Edges and band bins of a single path's figure (after k_cbuild with split_bin), over
// the whole GPU: edge records and band counts, a scan and pool allocation, the fill.
cudaError_t launch_figure_bins(const KParams& p, int grid, cudaStream_t s);
// The figure of one fill path (p.gb's ops) over the whole GPU, in place of k_cbuild with
// split_bin: vertices and sub-figure starts into CTA 0's scratch, fig_state[0], the pen
// width after the path and the path's status.  p.gb's state (done, n_raw, count) must be
// zero before the launch; k_gb_ops resets tr, the queue, the path's status, the pool
// counter and the bins.  When the path has more raw vertices than p.gb.raw_cap, *n_raw
// says how many and nothing else is written but a figure of no vertices; the caller grows
// the arrays and builds again.  `probe`
// (nullable): the same build over a prefix of the ops first (its own state and tr, its
// final_flag the full build's skip): when the cap is reached within the prefix the figure
// is complete and the full build does nothing.
cudaError_t launch_grid_build(const KParams& p, int sm_count, cudaStream_t s, const KParams* probe = nullptr);
// The same for one stroke path (p.gb and p.gs): stroke points, sub-strokes and outline over
// the whole GPU, then the outline's figure as launch_grid_build builds a fill's.  p.gs's
// state (st, n_sraw, done) must be zero before the launch, as p.gb's.  When the path has
// more raw stroke points than p.gs.sraw_cap, or its outline more raw vertices than
// p.gb.raw_cap, *n_sraw / *n_raw say how many and the figure is empty.
// `probe` (nullable): the stroke points first over a prefix of the ops (its own n_sraw,
// done and final_flag, the full build's skip): when the point cap is reached there the
// points are complete and the full build's point kernels do nothing.
cudaError_t launch_grid_stroke(const KParams& p, int sm_count, cudaStream_t s, const KParams* probe = nullptr);
// Shared memory either band compositor needs for rows of `width` pixels.
int composite_bands_smem(int band_rows, int width);
// A single call's rows from its binned edges (Matte8, or the coverage mask of an Rgba8p call).
cudaError_t launch_band_single(const KParams& p, int max_smem, cudaStream_t s);
int band_single_smem(int band_rows, int width);
// SrcOver of one call's colour from its mask, for canvases that no tensor map fits.
cudaError_t launch_srcover_rows(uint8_t* canvas, uint32_t stride, const uint8_t* mask, uint32_t mstride, int W, int H,
                                int r0, unsigned clr, cudaStream_t s);
int composite_build_blocks_per_sm(int smem_bytes, bool stroke);

// Static shared memory of the kernel besides the dynamic area buffer.
constexpr int RASTER_FIXED_SMEM = BLOCK * (int)sizeof(EdgeRec) + 3 * BLOCK * 4 + 256 + 4096;

// Launch the persistent rasteriser.  Returns the CUDA error of the launch.
// `chained`: right behind the tile rasteriser of the same path.
cudaError_t launch_raster(const KParams& p, int grid, int smem_bytes, cudaStream_t s, bool few_ctas,
                          bool chained = false);
// Resident CTAs per SM for `smem_bytes` of dynamic shared memory.
int raster_blocks_per_sm(int smem_bytes, bool stroke);

// Maximum dynamic shared memory the kernel may be configured for.
int raster_max_smem();

// Let the kernels take as much dynamic shared memory as the current device has.  The limit belongs
// to a kernel and device, not to a context: it is set to the same value whenever a context is
// created and by no launch (a launch that set it to its own size took it away from another
// context's thread between that one's setting and launch).
cudaError_t allow_smem(const void* kern);
cudaError_t setup_kernels();
cudaError_t setup_tile();
cudaError_t setup_bands();
// The check build's state of the other source files (ft_device.cuh, take_check).
struct CheckState;
cudaError_t take_check_tile(CheckState* s, bool reached);
cudaError_t take_check_bands(CheckState* s, bool reached);

}  // namespace ftk
