// ft_kernels.cu — the GB300 fill/stroke rasteriser (sm_103a).
//
// One persistent kernel drains a device queue of work items (a path and a range
// of its raster rows).  For each item one CTA of 256 threads:
//
//  1. walks the path ops in chunks of 256 (footile plotter.rs:175-224): two block
//     max-scans give every op its pen, pen width and "starts a new sub-figure"
//     flag, so each thread then flattens its own op independently;
//  2. flattens quads / cubics by recursive De Casteljau subdivision
//     (plotter.rs:248-265, 311-332) with an explicit per-thread stack, IEEE f32
//     without contraction, in the reference's depth-first leaf order: a count
//     pass, a block scan, then an emit pass into a shared-memory window;
//  3. builds the figure (fig.rs:428-461): warp 0 drops coincident vertices, pops
//     a closing vertex equal to the sub-figure start and applies the 65,535-vertex
//     cap, with ballots over 32 vertices at a time;
//  4. finds the top vertex (min (y, x, id), the head of footile's stable (Y,X)
//     sort, fig.rs:493-496) and the figure direction (fig.rs:402-411), and turns
//     every non-horizontal segment into an edge (fig.rs:179-201) — each segment
//     yields exactly the edge the active-edge sweep would add;
//  5. rasterises bands of rows: every (edge, row) pair is independent (x at the
//     bottom of row k is x_bot0 + k*inv_slope, wrapping), and its per-cell
//     coverage (fig.rs:285-321) has a closed form, so threads take (edge, row)
//     items and add signed cell areas into a shared-memory i32 band buffer with
//     atomics.  i16 wrapping sums commute, so the i32 sums truncated to i16 equal
//     footile's;
//  6. resolves each band row with a warp scan (__shfl_up_sync) and the NonZero /
//     EvenOdd rule (imgbuf.rs:38-199), then overwrites Matte8 rows or composites
//     premultiplied RGBA with pix SrcOver (fig.rs:629-665).
//
// Rows footile writes: from max(top_row, 0) to the bottom of the raster, raster
// row r receiving scan row r + min(top_row, 0) (fig.rs:496-499, 536-553).
#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstring>

#include <cuda.h>

#include "ft_adjoint.cuh"
#include "ft_device.cuh"
#include "ft_items.cuh"
#include "ft_kernels.cuh"
#include "ft_slots.cuh"

namespace ftk {

constexpr unsigned FULL = 0xFFFFFFFFu;

// Curve leaves of an op kept (in local memory) from the count pass for the emit pass;
// ops with more leaves are walked again.
constexpr int LEAF_CACHE_CTA = 256;
constexpr int SRAW = 1024;            // stroke points per window (float4 in the raw window's bytes)

// Kernels launched one after another on small data (the grid-wide builds): each waits for the
// one before (programmatic dependent launch) and lets the next be set up meanwhile, so that
// a launch's latency is spent while its predecessor still runs.
__device__ __forceinline__ void chain_link() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... A>
cudaError_t launch_chain(void (*kern)(A...), int grid, int threads, int smem, cudaStream_t s, const A&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// ------------------------------------------------------------ block scans
__device__ __forceinline__ int warp_incl_sum(int v) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
__device__ __forceinline__ unsigned warp_incl_sum_u(unsigned v) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned t = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += t;
    }
    return v;
}
__device__ __forceinline__ int warp_incl_max(int v) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v = max(v, t);
    }
    return v;
}
// Exclusive block sum; `total` receives the block total.  tmp: NWARP ints.
__device__ int block_excl_sum(int v, int* tmp, int& total) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = warp_incl_sum(v);
    if (lane == 31) tmp[w] = inc;
    __syncthreads();
    if (w == 0) {
        int t = lane < NWARP ? tmp[lane] : 0;
        t = warp_incl_sum(t);
        if (lane < NWARP) tmp[lane] = t;
    }
    __syncthreads();
    int base = w > 0 ? tmp[w - 1] : 0;
    total = tmp[NWARP - 1];
    __syncthreads();
    return base + inc - v;
}
// Inclusive block max.
__device__ int block_incl_max(int v, int* tmp) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = warp_incl_max(v);
    if (lane == 31) tmp[w] = inc;
    __syncthreads();
    if (w == 0) {
        int t = lane < NWARP ? tmp[lane] : -1;
        t = warp_incl_max(t);
        if (lane < NWARP) tmp[lane] = t;
    }
    __syncthreads();
    int r = w > 0 ? max(inc, tmp[w - 1]) : inc;
    __syncthreads();
    return r;
}
// Inclusive and exclusive block max (identity -1) in one pass.
__device__ void block_max_scan(int v, int* tmp, int& incl, int& excl) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = warp_incl_max(v);
    int wex = __shfl_up_sync(FULL, inc, 1);
    if (lane == 0) wex = -1;
    if (lane == 31) tmp[w] = inc;
    __syncthreads();
    if (w == 0) {
        int t = lane < NWARP ? tmp[lane] : -1;
        t = warp_incl_max(t);
        if (lane < NWARP) tmp[lane] = t;
    }
    __syncthreads();
    int carry = w > 0 ? tmp[w - 1] : -1;
    incl = max(inc, carry);
    excl = max(wex, carry);
    __syncthreads();
}

// The thread group of the figure builder: a whole CTA.
struct BlockG {
    static constexpr int N = BLOCK;
    static constexpr int RAW = RAW_CAP;
    __device__ static int rank() { return threadIdx.x; }
    __device__ static void sync() { __syncthreads(); }
    __device__ static int excl_sum(int v, int* tmp, int& total) { return block_excl_sum(v, tmp, total); }
    __device__ static int incl_max(int v, int* tmp) { return block_incl_max(v, tmp); }
    __device__ static void max_scan(int v, int* tmp, int& incl, int& excl) { block_max_scan(v, tmp, incl, excl); }
};
// ------------------------------------------------- De Casteljau flattening
// Stack frames of the walks: the right half of a subdivided curve.  A frame keeps no
// start point: the right half starts where the last leaf of the left half ends (that
// leaf's end point is the same value, carried down unchanged).  Fills carry no widths.
template <bool W>
struct QuadFr {
    P2 b, c;
    float wb, wc;
    int d;
};
template <>
struct QuadFr<false> {
    P2 b, c;
    int d;
};
template <bool W>
struct CubicFr {
    P2 b, c, e;
    float wb, wc, we;
    int d;
};
template <>
struct CubicFr<false> {
    P2 b, c, e;
    int d;
};

// Walk the subdivision of a quad (plotter.rs:248-265) in depth-first order.
// Leaves with index in [lo, hi) go to emit(index, point, width).  Returns the
// number of leaves walked (the total when hi == INT_MAX).  `d0`: the depth of (a, b, c)
// in the subdivision of a larger curve (0: the curve itself).
template <bool W, class Emit>
__device__ int quad_walk(P2 a, P2 b, P2 c, float wa, float wb, float wc, float tol_sq, int lo, int hi,
                         int* depth_hit, Emit emit, int d0 = 0) {
    using Fr = QuadFr<W>;
    Fr st[FT_MAX_DEPTH + 1];
    int sp = 0, leaf = 0, d = d0;
    for (;;) {
        P2 ab = pmid(a, b), bc = pmid(b, c), abbc = pmid(ab, bc), ac = pmid(a, c);
        bool within = pdist_sq(abbc, ac) <= tol_sq;
        if (within || d >= FT_MAX_DEPTH) {
            if (!within) *depth_hit = 1;
            if (leaf >= lo && leaf < hi) emit(leaf, c, wc);
            leaf++;
            if (leaf >= hi || sp == 0) break;
            --sp;
            a = c;
            b = st[sp].b;
            c = st[sp].c;
            if constexpr (W) {
                wa = wc;
                wb = st[sp].wb;
                wc = st[sp].wc;
            }
            d = st[sp].d;
        } else {
            float wab = 0, wbc = 0, wabbc = 0;
            if constexpr (W) {
                wab = fmid(wa, wb);
                wbc = fmid(wb, wc);
                wabbc = fmid(wab, wbc);
            }
            st[sp].b = bc;
            st[sp].c = c;
            if constexpr (W) {
                st[sp].wb = wbc;
                st[sp].wc = wc;
            }
            st[sp].d = d + 1;
            sp++;
            b = ab;
            c = abbc;
            if constexpr (W) {
                wb = wab;
                wc = wabbc;
            }
            d++;
        }
    }
    return leaf;
}

// The same for a cubic (plotter.rs:311-332).
template <bool W, class Emit>
__device__ int cubic_walk(P2 a, P2 b, P2 c, P2 e, float wa, float wb, float wc, float we, float tol_sq, int lo,
                          int hi, int* depth_hit, Emit emit, int d0 = 0) {
    using Fr = CubicFr<W>;
    Fr st[FT_MAX_DEPTH + 1];
    int sp = 0, leaf = 0, d = d0;
    for (;;) {
        P2 ab = pmid(a, b), bc = pmid(b, c), cd = pmid(c, e);
        P2 abbc = pmid(ab, bc), bccd = pmid(bc, cd);
        P2 pe = pmid(abbc, bccd);
        P2 ad = pmid(a, e);
        bool within = pdist_sq(pe, ad) <= tol_sq;
        if (within || d >= FT_MAX_DEPTH) {
            if (!within) *depth_hit = 1;
            if (leaf >= lo && leaf < hi) emit(leaf, e, we);
            leaf++;
            if (leaf >= hi || sp == 0) break;
            --sp;
            a = e;
            b = st[sp].b;
            c = st[sp].c;
            e = st[sp].e;
            if constexpr (W) {
                wa = we;
                wb = st[sp].wb;
                wc = st[sp].wc;
                we = st[sp].we;
            }
            d = st[sp].d;
        } else {
            float wab = 0, wbc = 0, wcd = 0, wabbc = 0, wbccd = 0, wpe = 0;
            if constexpr (W) {
                wab = fmid(wa, wb);
                wbc = fmid(wb, wc);
                wcd = fmid(wc, we);
                wabbc = fmid(wab, wbc);
                wbccd = fmid(wbc, wcd);
                wpe = fmid(wabbc, wbccd);
            }
            st[sp].b = bccd;
            st[sp].c = cd;
            st[sp].e = e;
            if constexpr (W) {
                st[sp].wb = wbccd;
                st[sp].wc = wcd;
                st[sp].we = we;
            }
            st[sp].d = d + 1;
            sp++;
            b = ab;
            c = abbc;
            e = pe;
            if constexpr (W) {
                wb = wab;
                wc = wabbc;
                we = wpe;
            }
            d++;
        }
    }
    return leaf;
}

// ------------------------------------------------------------- CTA state
struct CState {
    // path walk carried between op chunks
    float pen_x, pen_y, pen_w, sw;
    int last_pc_kind;  // kind of the last Move/Line/Quad/Cubic/Close op, -1 none
    // figure builder
    int count;
    int has_prev, prev_x, prev_y;  // previous raw vertex
    int rf_x, rf_y, rf_pos;        // first vertex of the current sub-figure and its id
    int capped;
    int flags;     // 1: depth cap reached, 2: bad argument
    // figure summary
    int top_row;
    int dir;  // 0 forward, 1 reverse
    int last_pw;
    // stroke points (stroker.rs:204-236)
    int s_count, s_nsubs, s_capped, s_last_op, s_has_prev;
    float s_prev_x, s_prev_y;
    int s_items;  // outline items of all sub-strokes
};

// One chunk of ops whose curves are taken by slots (ft_slots.cuh), in place of the raw window:
// the ops that have slots, and one round of BLOCK leaves.
struct SlotSmem {
    float4 g0[BLOCK], g1[BLOCK];  // transformed control points (a, b), (c, end)
    float2 w[BLOCK];              // strokes: the widths of the pen and of the op
    int off[BLOCK + 32];          // first slot; past the last op INT_MAX
    int info[BLOCK];              // depth | safe << 4 | type << 8 | starts a sub-figure << 10 | Move << 11 | op << 12
    __align__(16) float4 raw[BLOCK];  // leaves: int2 16.16 vertices (fills), or points and widths (strokes)
    int opi[BLOCK];
    unsigned char rs[BLOCK], jp[BLOCK];
};
enum { SLOT_POINT = 0, SLOT_QUAD = 1, SLOT_CUBIC = 2 };

template <int N, int RAW>
struct BuildSmemT {
    int kind[N];
    float pwval[N];
    float penx[N], peny[N], penw[N];
    int scan[2 * NWARP + 2];
    union {
        struct {
            // 16-byte aligned: stroke points are stored here as float4
            __align__(16) int2 raw[RAW];
            unsigned char rs[RAW];
        };
        SlotSmem slots;
    };
};
using BuildSmem = BuildSmemT<BLOCK, RAW_CAP>;

constexpr int MAP_CAP = 4096;  // (edge, row) items mapped per round

struct RasterSmem {
    EdgeRec edges[BLOCK];
    int ya[BLOCK];
    int off[BLOCK + 1];
    int scan[2 * NWARP + 2];
    unsigned char map[MAP_CAP];  // item -> edge slot of the current chunk
};
static_assert(((sizeof(RasterSmem) + 15) & ~(size_t)15) <= (size_t)RASTER_FIXED_SMEM, "raster smem layout");
static_assert(sizeof(int2) * RAW_CAP >= sizeof(float4) * SRAW && RAW_CAP >= 2 * SRAW, "stroke window layout");
static_assert(offsetof(BuildSmem, raw) % 16 == 0 && sizeof(BuildSmem) % 16 == 0, "build smem alignment");

// ------------------------------------------------------------ figure builder
// Sequential restatement of Fig::add_point / Fig::close (fig.rs:373-461) for one
// group of raw vertices; used for the group in which the 65,535 cap is reached.
__device__ void seq_group(CState& S, const int2* raw, const unsigned char* rsf, int n, int2* pts, int* ss,
                          int cap = PT_CAP) {
    int count = S.count, has_prev = S.has_prev;
    int px = S.prev_x, py = S.prev_y, rfx = S.rf_x, rfy = S.rf_y, rf_pos = S.rf_pos;
    for (int l = 0; l < n; l++) {
        int2 p = raw[l];
        int rs = rsf[l];
        // a close event precedes a vertex that starts a sub-figure: pop when the
        // last vertex equals the sub-figure start (fig.rs:373-383)
        if (rs && has_prev && rfx == px && rfy == py) count -= 1;
        if (count >= cap) {
            // add_point is ignored from here on (fig.rs:430).  The next close —
            // an explicit one or the one Plotter::fill ends with — pops the last
            // vertex if it equals the open sub-figure's start.
            if (!rs && rfx == px && rfy == py) count -= 1;
            S.capped = 1;
            break;
        }
        if (rs) {
            rfx = p.x;
            rfy = p.y;
            rf_pos = count;
            pts[count] = p;
            ss[count] = count;
            count++;
        } else if (p.x != px || p.y != py) {
            pts[count] = p;
            ss[count] = rf_pos;
            count++;
        }
        px = p.x;
        py = p.y;
        has_prev = 1;
    }
    S.count = count;
    S.has_prev = has_prev;
    S.prev_x = px;
    S.prev_y = py;
    S.rf_x = rfx;
    S.rf_y = rfy;
    S.rf_pos = rf_pos;
}

// Append one window of raw vertices to the figure, 256 per step, one per thread.  A vertex is
// kept when it starts a sub-figure or differs from the previous raw vertex; a sub-figure whose
// last vertex equals its first loses that vertex when it is closed.
// Cross-lane questions (latest sub-figure start at or before a vertex, next kept
// vertex, next run end) are answered from per-warp ballot masks in shared memory.
struct CompactSmem {
    unsigned rsm[NWARP], km[NWARP], em[NWARP], pm[NWARP];
    int posv[BLOCK];
    int scan[2 * NWARP + 2];
};

// first set bit of the block-wide mask at index >= i (block-local), or BLOCK
__device__ __forceinline__ int mask_next(const unsigned* m, int i) {
    int w = i >> 5;
    unsigned bits = m[w] & (0xFFFFFFFFu << (i & 31));
    while (!bits) {
        if (++w >= NWARP) return BLOCK;
        bits = m[w];
    }
    return (w << 5) + __ffs(bits) - 1;
}
// last set bit at index <= i (block-local), or -1
__device__ __forceinline__ int mask_prev(const unsigned* m, int i) {
    int w = i >> 5;
    int sh = i & 31;
    unsigned bits = m[w] & (sh == 31 ? 0xFFFFFFFFu : ((2u << sh) - 1u));
    while (!bits) {
        if (--w < 0) return -1;
        bits = m[w];
    }
    return (w << 5) + 31 - __clz(bits);
}

__device__ void compact_window_block(CState& S, const int2* raw, const unsigned char* rsf, int m, int2* pts,
                                     int* ss, CompactSmem& C, int cap = PT_CAP) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int base = 0; base < m; base += BLOCK) {
        const int k = base + tid;
        const bool valid = k < m;
        const int2 p = valid ? raw[k] : make_int2(0, 0);
        const int rs = valid ? rsf[k] : 0;
        const int count0 = S.count, has_prev = S.has_prev;
        const int prevx = S.prev_x, prevy = S.prev_y, rfx0 = S.rf_x, rfy0 = S.rf_y, rfpos0 = S.rf_pos;
        const int nb = min(BLOCK, m - base);  // vertices in this step
        // close of the run that ended with the previous step (pop if it returned to its start)
        int count_b = count0;
        if (rsf[base] && has_prev && rfx0 == prevx && rfy0 == prevy) count_b -= 1;
        int2 q = make_int2(prevx, prevy);
        if (tid > 0 && valid) q = raw[k - 1];
        const bool keep = valid && (rs || p.x != q.x || p.y != q.y);
        // runs ending at the step's last vertex are closed at the next step (as above)
        const bool endk = valid && (tid + 1 < nb) && rsf[k + 1];
        const unsigned RS = __ballot_sync(FULL, valid && rs), K = __ballot_sync(FULL, keep),
                       E = __ballot_sync(FULL, endk);
        if (lane == 0) {
            C.rsm[w] = RS;
            C.km[w] = K;
            C.em[w] = E;
        }
        __syncthreads();
        const int jf = mask_prev(C.rsm, tid);  // first vertex of this vertex's run, in this block
        int rfx = rfx0, rfy = rfy0;
        if (jf >= 0) {
            const int2 f = raw[base + jf];
            rfx = f.x;
            rfy = f.y;
        }
        const bool pop = endk && p.x == rfx && p.y == rfy;
        const unsigned PM = __ballot_sync(FULL, pop);
        if (lane == 0) C.pm[w] = PM;
        int tot;
        const int ex = block_excl_sum((keep ? 1 : 0) - (pop ? 1 : 0), C.scan, tot);
        const int pos = count_b + ex;
        C.posv[tid] = pos;
        const int capped = __syncthreads_or(keep && pos >= cap);
        if (capped) {
            if (tid == 0) seq_group(S, raw + base, rsf + base, nb, pts, ss, cap);
            __syncthreads();
            return;
        }
        // a vertex disappears when it is the last kept one of a run that pops in this block
        bool write = keep;
        if (keep) {
            const int e = mask_next(C.em, tid);
            if (e < BLOCK && ((C.pm[e >> 5] >> (e & 31)) & 1u)) {
                const int nk = tid < BLOCK - 1 ? mask_next(C.km, tid + 1) : BLOCK;
                if (nk > e) write = false;
            }
        }
        if (write) {
            pts[pos] = p;
            ss[pos] = jf >= 0 ? C.posv[jf] : rfpos0;
        }
        __syncthreads();
        if (tid == 0) {
            const int n = nb;
            S.count = count_b + tot;
            const int2 l = raw[base + n - 1];
            S.prev_x = l.x;
            S.prev_y = l.y;
            S.has_prev = 1;
            const int lr = mask_prev(C.rsm, n - 1);
            if (lr >= 0) {
                const int2 f = raw[base + lr];
                S.rf_x = f.x;
                S.rf_y = f.y;
                S.rf_pos = C.posv[lr];
            }
        }
        __syncthreads();
    }
}

// Stroke points, block-wide (Stroke::add_point / close, stroker.rs:204-236): a point is
// kept when it starts a sub-stroke or its f32 position differs from the previous raw
// point; no closing point is popped; points past 65,535 are dropped and start nothing.
// `jpf[k]` is the `joined` value the close events before a sub-stroke start leave on
// the previous sub-stroke (false after a Move, true after a Close).
__device__ void compact_stroke_block(CState& S, const float4* raw, const unsigned char* rsf,
                                     const unsigned char* jpf, const int* opi, int m, float4* spts, SubRec* subs,
                                     CompactSmem& C) {
    const int tid = threadIdx.x;
    for (int base = 0; base < m; base += BLOCK) {
        const int k = base + tid;
        const bool valid = k < m;
        const int nb = min(BLOCK, m - base);
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        int rs = 0;
        if (valid) {
            p = raw[k];
            rs = rsf[k];
        }
        const int count0 = S.s_count, nsub0 = S.s_nsubs;
        float qx = S.s_prev_x, qy = S.s_prev_y;
        if (tid > 0 && valid) {
            qx = raw[k - 1].x;
            qy = raw[k - 1].y;
        }
        const bool keep = valid && (rs || !(p.x == qx && p.y == qy));
        int tot;
        const int pos = count0 + block_excl_sum(keep ? 1 : 0, C.scan, tot);
        const bool acc = keep && pos < PT_CAP;
        int tot_rs;
        const int sid = nsub0 + block_excl_sum((acc && rs) ? 1 : 0, C.scan, tot_rs);
        if (acc) spts[pos] = p;
        if (acc && rs) {
            subs[sid].start = pos;
            if (sid > 0) subs[sid - 1].joined = jpf[k];  // the last sub-stroke's is set by finish_subs
        }
        const int la = block_incl_max(acc ? tid : -1, C.scan);  // last accepted point of the step
        const int capped = __syncthreads_or(keep && pos >= PT_CAP);
        if (tid == BLOCK - 1) {
            S.s_count = min(count0 + tot, PT_CAP);
            S.s_nsubs = nsub0 + tot_rs;
            const float4 l = raw[base + nb - 1];
            S.s_prev_x = l.x;
            S.s_prev_y = l.y;
            S.s_has_prev = 1;
            if (la >= 0) S.s_last_op = opi[base + la];
            if (capped) S.s_capped = 1;
        }
        __syncthreads();
        if (capped) return;
    }
}

// Sizes of the sub-strokes and their outline items (stroker.rs:87-96, 239-262).  The
// last sub-stroke is joined when the last close event after its last point was a
// Close; when the 65,535 cap stopped the point stream, that is the last Close or Move
// op after the op of the last kept point.
__device__ void finish_subs(const KParams& P, const ft_path_desc& d, CState& S, SubRec* subs, int* tmp) {
    const int tid = threadIdx.x;
    const int nsub = S.s_nsubs, count = S.s_count;
    if (S.s_capped) {
        int last = -1;
        for (int i = S.s_last_op + 1 + tid; i < (int)d.n_ops; i += BLOCK) {
            const int kd = P.ops[d.op_begin + i].kind;
            if (kd == FT_OP_CLOSE || kd == FT_OP_MOVE) last = max(last, i);
        }
        last = block_incl_max(last, tmp);
        if (tid == BLOCK - 1 && nsub > 0)
            subs[nsub - 1].joined = last >= 0 ? (P.ops[d.op_begin + last].kind == FT_OP_CLOSE) : 0;
    } else if (tid == 0 && nsub > 0) {
        subs[nsub - 1].joined = S.last_pc_kind == FT_OP_CLOSE;
    }
    __syncthreads();
    int carry = 0;
    for (int s0 = 0; s0 < nsub; s0 += BLOCK) {
        const int si = s0 + tid;
        int items = 0;
        if (si < nsub) {
            SubRec r = subs[si];
            r.n = (si + 1 < nsub ? subs[si + 1].start : count) - r.start;
            // SubStroke::len with u16 arithmetic: n + 1 wraps at 65,536
            r.len = r.joined ? ((r.n + 1) & 0xFFFF) : (r.n > 0 ? r.n - 1 : 0);
            items = r.len > 0 ? 2 * r.len + 2 : 0;
            subs[si].n = r.n;
            subs[si].len = r.len;
        }
        int tot;
        const int off = block_excl_sum(items, tmp, tot);
        if (si < nsub) subs[si].item_off = carry + off;
        carry += tot;
    }
    if (tid == 0) S.s_items = carry;
    __syncthreads();
}

// stroke_offset (stroker.rs:301-309): both ends of segment (p0, p1) moved right by w/2
__device__ __forceinline__ void seg_offset(float4 p0, float4 p1, P2* r0, P2* r1) {
    const P2 vr = pnormalize(pright(psub(p2(p1.x, p1.y), p2(p0.x, p0.y))));
    *r0 = padd(p2(p0.x, p0.y), pscale(vr, __fmul_rn(p0.z, 0.5f)));
    *r1 = padd(p2(p1.x, p1.y), pscale(vr, __fmul_rn(p1.z, 0.5f)));
}

// Round-join arc (stroker.rs:399-416) walked depth first; leaves in [lo, hi) go to
// emit(index, point).  Returns the leaves walked.
template <class Emit>
__device__ int arc_walk(float4 p, P2 a, P2 b, float tol_sq, int lo, int hi, int* depth_hit, Emit emit) {
    struct Fr {
        P2 a, b;
        int d;
    };
    Fr st[FT_MAX_DEPTH + 1];
    int sp = 0, leaf = 0, d = 0;
    const float hw = __fmul_rn(p.z, 0.5f);
    for (;;) {
        const P2 vr = pnormalize(pright(psub(b, a)));
        const P2 c = padd(p2(p.x, p.y), pscale(vr, hw));
        const P2 ab = pmid(a, b);
        const bool leafy = !pfinite(c) || pdist_sq(c, ab) <= tol_sq;
        if (leafy || d >= FT_MAX_DEPTH) {
            if (!leafy) *depth_hit = 1;
            if (leaf >= lo && leaf < hi) emit(leaf, b);
            leaf++;
            if (leaf >= hi || sp == 0) break;
            --sp;
            a = st[sp].a;
            b = st[sp].b;
            d = st[sp].d;
        } else {
            st[sp].a = c;
            st[sp].b = b;
            st[sp].d = d + 1;
            sp++;
            b = c;
            d++;
        }
    }
    return leaf;
}

// One outline item of a sub-stroke: the start point, one join, or the end point of a
// side (stroker.rs:265-295, 323-396).  Emits its points in order through emit(k, pt)
// for k in [lo, hi) and returns how many it has.
template <class Emit>
__device__ int outline_item(const KParams& P, const float4* spts, const SubRec& sr, int u, int lo, int hi,
                            int* depth_hit, Emit emit) {
    const int len = sr.len, n = sr.n, s = sr.start;
    const bool joined = sr.joined != 0;
    const bool rev = u > len;
    const int j = rev ? u - len - 1 : u;  // iteration on this side; j == len is the end item
    // point k modulo n (k - n .. k + n without a division: all there is unless len wrapped)
    auto at = [&](int k) {
        k = k < 0 ? k + n : (k >= n ? k - n : k);
        return s + ((unsigned)k < (unsigned)n ? k : (k % n + n) % n);
    };
    auto v0 = [&](int jj) { return at(rev ? n - 1 - jj : jj); };
    auto v1 = [&](int jj) { return at(rev ? n - 2 - jj : jj + 1); };
    auto seg = [&](int jj, P2* r0, P2* r1) { seg_offset(spts[v0(jj)], spts[v1(jj)], r0, r1); };
    if (j == len) {  // end of an open side: the last offset point
        if (joined) return 0;
        P2 r0, r1;
        seg(len - 1, &r0, &r1);
        if (lo <= 0 && 0 < hi) emit(0, r1);
        return 1;
    }
    if (j == 0) {  // start of an open side: butt end
        if (joined) return 0;
        P2 r0, r1;
        seg(0, &r0, &r1);
        if (lo <= 0 && 0 < hi) emit(0, r0);
        return 1;
    }
    P2 a0, a1, b0, b1;
    seg(j - 1, &a0, &a1);
    seg(j, &b0, &b1);
    if (P.join == FT_JOIN_MITER) {  // stroker.rs:340-367 (the decision as ft_fmath.h takes it)
        const P2 u = psub(a1, a0), v = psub(b0, b1);
        P2 xp;
        if (ft_miter_join(u.x, u.y, v.x, v.y, P.miter_g) && pline_x(a0, a1, b0, b1, &xp)) {
            if (lo <= 0 && 0 < hi) emit(0, xp);
            return 1;
        }
    } else if (P.join == FT_JOIN_ROUND) {  // stroker.rs:380-396
        const P2 u = psub(a1, a0), v = psub(b0, b1);
        if (ft_round_join_arc(u.x, u.y, v.x, v.y)) {
            if (lo <= 0 && 0 < hi) emit(0, a1);
            const int na = arc_walk(spts[v0(j)], a1, b0, P.tol_sq, max(lo - 1, 0), hi - 1, depth_hit,
                                    [&](int k, P2 q) { emit(k + 1, q); });
            return 1 + na;
        }
    }
    // bevel (stroker.rs:370-373)
    if (lo <= 0 && 0 < hi) emit(0, a1);
    if (lo <= 1 && 1 < hi) emit(1, b0);
    return 2;
}

// Stroke outline -> figure: outline items in chunks of BLOCK (count, scan, then emit
// window by window through the second transform, plotter.rs:356-365 / 219-224) into
// the same figure builder a fill uses.
__device__ void build_outline(const KParams& P, CState& S, const float4* spts, const SubRec* subs, BuildSmem& B,
                              CompactSmem& Cs, int2* pts, int* ss) {
    const int tid = threadIdx.x;
    const int total_items = S.s_items, nsub = S.s_nsubs;
    if (tid == 0) {
        S.count = 0;
        S.has_prev = 0;
        S.prev_x = S.prev_y = 0;
        S.rf_x = S.rf_y = 0;
        S.rf_pos = 0;
        S.capped = 0;
    }
    __syncthreads();
    for (int t0 = 0; t0 < total_items; t0 += BLOCK) {
        const int t = t0 + tid;
        int n = 0, si = -1, u = 0, rsk = -1;  // rsk: index of this item's point that starts a figure run
        SubRec sr;
        int depth_hit = 0;
        P2 c0 = p2(0.f, 0.f), c1 = p2(0.f, 0.f);  // the item's first two points, kept for the emit pass
        if (t < total_items) {
            // the last sub-stroke with item_off <= t owns item t (empty ones share the
            // next one's offset and come before it)
            int lo = 0, hi = nsub - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (subs[mid].item_off <= t)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            si = lo;
            sr = subs[si];
            u = t - sr.item_off;
            n = outline_item(P, spts, sr, u, 0, INT_MAX, &depth_hit, [&](int k, P2 q) {
                if (k == 0) c0 = q;
                if (k == 1) c1 = q;
            });
            // a figure run starts at each side's first point after a Close: the forward
            // side always (after the previous sub-stroke's Close, or first), the reverse
            // side when the sub-stroke is joined (stroker.rs:255-260)
            const bool rev = u > sr.len;
            const int j = rev ? u - sr.len - 1 : u;
            const bool joined = sr.joined != 0;
            if (!rev && ((!joined && j == 0) || (joined && j == 1))) rsk = 0;
            if (rev && joined && j == 1) rsk = 0;
        }
        if (depth_hit) atomicOr(&S.flags, 1);
        int total;
        const int off = block_excl_sum(n, B.scan, total);
        for (int w0 = 0; w0 < total; w0 += RAW_CAP) {
            const int w1 = min(w0 + RAW_CAP, total);
            if (n > 0 && off < w1 && off + n > w0) {
                const int lo = max(w0, off) - off, hi = min(w1, off + n) - off;
                auto put = [&](int k, P2 q) {
                    const int idx = off + k - w0;
                    const P2 tq = xform(P.xf, q);  // the outline is transformed again (F9)
                    B.raw[idx] = make_int2(f2fx(tq.x), f2fx(tq.y));
                    B.rs[idx] = (k == rsk) ? (unsigned char)1 : (unsigned char)0;
                };
                if (n <= 2) {  // an end, a miter or a bevel: the points of the count pass
                    for (int k = lo; k < hi; k++) put(k, k == 0 ? c0 : c1);
                } else {
                    int dh = 0;
                    outline_item(P, spts, sr, u, lo, hi, &dh, put);
                }
            }
            __syncthreads();
            compact_window_block(S, B.raw, B.rs, w1 - w0, pts, ss, Cs);
            __syncthreads();
            if (S.capped) break;
        }
        __syncthreads();
        if (S.capped) break;
    }
    // Plotter::fill ends with fig.close() (plotter.rs:347)
    if (tid == 0 && !S.capped && S.has_prev && S.rf_x == S.prev_x && S.rf_y == S.prev_y) S.count -= 1;
    __syncthreads();
}

// Path walk + flattening by the thread group G.
// Fill (Plotter::fill, plotter.rs:339-350): builds the figure in pts[0..S.count) / ss[];
// `limit` is the figure's vertex cap.
// STROKE (Plotter::stroke, plotter.rs:356-365, first half): collects the stroke points
// with their widths in spts[0..S.s_count) and the sub-strokes in subs[0..S.s_nsubs).
// Global raw store of a CTA figure build (SCR_RAWG ...); null: windows of raw
// vertices in shared memory, each emitted by re-walking the ops that reach it.
struct RawStore {
    float4* p4 = nullptr;
    unsigned char* rs = nullptr;
    unsigned char* jp = nullptr;
    int* opi = nullptr;
};
__device__ __forceinline__ RawStore raw_store(unsigned char* scr, const ScrLayout& L = scr_layout(PT_CAP)) {
    RawStore r;
    r.p4 = reinterpret_cast<float4*>(scr + L.rawg);
    r.rs = scr + L.rsg;
    r.jp = scr + L.jpg;
    r.opi = reinterpret_cast<int*>(scr + L.opig);
    return r;
}

template <class G, bool STROKE = false>
__device__ void build_fill(const KParams& P, const ft_path_desc& d, float sw0, BuildSmemT<G::N, G::RAW>& B,
                           CompactSmem* Cs, CState& S, int2* pts, int* ss, int limit, float4* spts = nullptr,
                           SubRec* subs = nullptr, int* opi = nullptr, RawStore rg = RawStore()) {
    constexpr int N = G::N;
    const int tid = G::rank();
    if (tid == 0) {
        S.pen_x = 0.f;
        S.pen_y = 0.f;
        S.pen_w = sw0;
        S.sw = sw0;
        S.last_pc_kind = -1;
        S.count = 0;
        S.has_prev = 0;
        S.prev_x = S.prev_y = 0;
        S.rf_x = S.rf_y = 0;
        S.rf_pos = 0;
        S.capped = 0;
        S.flags = 0;
        S.s_count = S.s_nsubs = S.s_capped = S.s_has_prev = 0;
        S.s_last_op = -1;
        S.s_prev_x = S.s_prev_y = 0.f;
    }
    G::sync();
    constexpr int WIN = STROKE ? SRAW : G::RAW;
    const ft_op* ops = P.ops + d.op_begin;
    const int n_ops = (int)d.n_ops;
    const float tol_sq = P.tol_sq;
    for (int c0 = 0; c0 < n_ops; c0 += N) {
        const int i = c0 + tid;
        const bool valid = i < n_ops;
        ft_op op;
        if (valid) {
            const int4* src = reinterpret_cast<const int4*>(ops + i);
            int4 q0 = __ldg(src), q1 = __ldg(src + 1);
            op.kind = q0.x;
            op.v[0] = __int_as_float(q0.y);
            op.v[1] = __int_as_float(q0.z);
            op.v[2] = __int_as_float(q0.w);
            op.v[3] = __int_as_float(q1.x);
            op.v[4] = __int_as_float(q1.y);
            op.v[5] = __int_as_float(q1.z);
        } else {
            op.kind = -1;
            for (int j = 0; j < 6; j++) op.v[j] = 0.f;
        }
        int kind = op.kind;
        if (kind < -1 || kind > FT_OP_PEN_WIDTH) {
            atomicOr(&S.flags, 2);
            kind = -1;
        }
        const bool isPW = kind == FT_OP_PEN_WIDTH;
        const bool isPC = kind >= FT_OP_CLOSE && kind <= FT_OP_CUBIC;
        B.kind[tid] = kind;
        B.pwval[tid] = op.v[0];
        // pen width in effect at this op (last PenWidth at or before it)
        const int lpw = G::incl_max(isPW ? tid : -1, B.scan);
        G::sync();
        const float sw_i = lpw >= 0 ? B.pwval[lpw] : S.sw;
        if (isPC) {
            float ex = 0.f, ey = 0.f;  // Close resets the pen to the origin (plotter.rs:200-203)
            if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
                ex = op.v[0];
                ey = op.v[1];
            } else if (kind == FT_OP_QUAD) {
                ex = op.v[2];
                ey = op.v[3];
            } else if (kind == FT_OP_CUBIC) {
                ex = op.v[4];
                ey = op.v[5];
            }
            B.penx[tid] = ex;
            B.peny[tid] = ey;
            B.penw[tid] = sw_i;
        }
        // pen before this op = pen after the last Move/Line/Quad/Cubic/Close before it
        int lpc_inc, lpc;
        G::max_scan(isPC ? tid : -1, B.scan, lpc_inc, lpc);
        G::sync();
        float pen_x, pen_y, pen_w;
        int prev_pc_kind;
        if (lpc >= 0) {
            pen_x = B.penx[lpc];
            pen_y = B.peny[lpc];
            pen_w = B.penw[lpc];
            prev_pc_kind = B.kind[lpc];
        } else {
            pen_x = S.pen_x;
            pen_y = S.pen_y;
            pen_w = S.pen_w;
            prev_pc_kind = S.last_pc_kind;
        }
        // widths of a curve's control points (plotter.rs:235-236, 294-298)
        float wa = pen_w, wb = 0.f, wc = 0.f, wd = sw_i;
        if (STROKE) {
            if (kind == FT_OP_QUAD) {
                wb = __fmul_rn(__fadd_rn(pen_w, sw_i), 0.5f);
                wc = sw_i;
            } else if (kind == FT_OP_CUBIC) {
                wb = __fadd_rn(sw_i, __fmul_rn(__fsub_rn(pen_w, sw_i), 1.0f / 3.0f));
                wc = __fadd_rn(sw_i, __fmul_rn(__fsub_rn(pen_w, sw_i), 2.0f / 3.0f));
            }
        }
        // the first vertex of this op starts a sub-figure after a close event
        const int rs = (kind == FT_OP_MOVE) || prev_pc_kind == FT_OP_CLOSE || prev_pc_kind == -1;

        // ---- count the vertices this op adds
        int n = 0;
        int depth_hit = 0;
        bool nonfinite = false;
        constexpr int LC = LEAF_CACHE_CTA;
        int2 cache[LC];  // leaves of the count pass, reused by the emit pass
        auto keep_leaf = [&](int k, P2 q, float) {
            if (k < LC) cache[k] = make_int2(f2fx(q.x), f2fx(q.y));
        };
        int D_slots = 0, safe = 0;  // the curve's slots: 2^D_slots
        P2 A = p2(0, 0), Bq = p2(0, 0), C = p2(0, 0), D = p2(0, 0);
        if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
            A = xform(P.xf, p2(op.v[0], op.v[1]));
            n = 1;
        } else if (kind == FT_OP_QUAD || kind == FT_OP_CUBIC) {
            A = xform(P.xf, p2(pen_x, pen_y));
            Bq = xform(P.xf, p2(op.v[0], op.v[1]));
            C = xform(P.xf, p2(op.v[2], op.v[3]));
            D = kind == FT_OP_CUBIC ? xform(P.xf, p2(op.v[4], op.v[5])) : C;
            nonfinite = !pfinite(A) || !pfinite(Bq) || !pfinite(C) || !pfinite(D);
            n = 1;
            if (!nonfinite) D_slots = curve_depth(A, Bq, C, D, kind == FT_OP_CUBIC, P.tol, safe);
        }
        if (nonfinite) atomicOr(&S.flags, 2);
        if (!__syncthreads_or(D_slots > SLOT_DEPTH)) {
            // ---- the chunk's leaves by slots, BLOCK at a time
            SlotSmem& Q = B.slots;
            const unsigned slots = n ? 1u << D_slots : 0u;
            unsigned inc = slots | ((slots ? 1u : 0u) << 22);
            const unsigned own = inc;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const unsigned t = __shfl_up_sync(FULL, inc, s);
                if ((tid & 31) >= s) inc += t;
            }
            if ((tid & 31) == 31) B.scan[tid >> 5] = (int)inc;
            __syncthreads();
            unsigned pre = 0, sum = 0;
#pragma unroll
            for (int k = 0; k < NWARP; k++) {
                const unsigned v = (unsigned)B.scan[k];
                if (k < tid >> 5) pre += v;
                sum += v;
            }
            const int listed = (int)(sum >> 22), total = (int)(sum & ((1u << 22) - 1));
            if (slots && ck((pre + inc - own) >> 22 < (unsigned)N, 20)) {
                const unsigned ex = pre + inc - own;
                const int at = (int)(ex >> 22);
                const bool curve = (kind == FT_OP_QUAD || kind == FT_OP_CUBIC) && !nonfinite;
                if (curve) Q.g0[at] = make_float4(A.x, A.y, Bq.x, Bq.y);
                const P2 end = kind == FT_OP_MOVE || kind == FT_OP_LINE ? A : D;
                Q.g1[at] = make_float4(C.x, C.y, end.x, end.y);
                if (STROKE) Q.w[at] = make_float2(pen_w, sw_i);
                Q.off[at] = (int)(ex & ((1u << 22) - 1));
                Q.info[at] = (curve ? D_slots : 0) | (safe << 4) |
                             ((!curve ? SLOT_POINT : kind == FT_OP_QUAD ? SLOT_QUAD : SLOT_CUBIC) << 8) | (rs << 10) |
                             ((kind == FT_OP_MOVE ? 1 : 0) << 11) | (tid << 12);
            }
            if (tid < 32) Q.off[listed + tid] = INT_MAX;
            // carry the path-walk state to the next chunk (everyone has read S by now)
            if (tid == N - 1) {
                S.sw = sw_i;
                const int last_pc = isPC ? tid : lpc;
                if (last_pc >= 0) {
                    S.pen_x = B.penx[last_pc];
                    S.pen_y = B.peny[last_pc];
                    S.pen_w = B.penw[last_pc];
                    S.last_pc_kind = B.kind[last_pc];
                }
            }
            __syncthreads();
            int j0 = 0;
            for (int w0 = 0; w0 < total; w0 += N) {
                const int s = w0 + tid;
                int at = -1, info = 0, idx = 0;
                P2 z = p2(0, 0);
                float zw = 0.f;
                if (w0 + (tid & ~31) < total) {
                    const int j = slot_op(Q.off, w0 + (tid & ~31), j0);
                    if (s < total) {
                        info = Q.info[j];
                        idx = s - Q.off[j];
                        const float4 g1 = Q.g1[j];
                        const int depth = info & 15, sf = (info >> 4) & 15, type = (info >> 8) & 3;
                        z = p2(g1.z, g1.w);
                        float2 w = make_float2(0.f, 0.f);
                        if (STROKE) w = Q.w[j];
                        zw = w.y;
                        if (type == SLOT_POINT) {
                            at = 0;
                        } else {
                            const float4 g0 = Q.g0[j];
                            P2 a = p2(g0.x, g0.y);
                            float w0v = w.x;
                            // widths of a curve's control points (plotter.rs:235-236, 294-298)
                            if (type == SLOT_QUAD)
                                at = quad_slot<STROKE>(a, p2(g0.z, g0.w), z, w0v, __fmul_rn(__fadd_rn(w.x, w.y), 0.5f), zw,
                                                       idx, depth, sf, tol_sq);
                            else
                                at = cubic_slot<STROKE>(a, p2(g0.z, g0.w), p2(g1.x, g1.y), z, w0v,
                                                        __fadd_rn(w.y, __fmul_rn(__fsub_rn(w.x, w.y), 1.0f / 3.0f)),
                                                        __fadd_rn(w.y, __fmul_rn(__fsub_rn(w.x, w.y), 2.0f / 3.0f)), zw,
                                                        idx, depth, sf, tol_sq);
                        }
                    }
                }
                int m;
                const int pos = block_excl_sum(at >= 0 ? 1 : 0, B.scan, m);
                if (at >= 0 && ck(pos < N, 28)) {
                    Q.rs[pos] = (unsigned char)(idx == 0 ? (info >> 10) & 1 : 0);
                    if (STROKE) {
                        Q.raw[pos] = make_float4(z.x, z.y, zw, 0.f);
                        Q.jp[pos] = (unsigned char)(((info >> 11) & 1) ^ 1);
                        Q.opi[pos] = c0 + (info >> 12);
                    } else {
                        reinterpret_cast<int2*>(Q.raw)[pos] = make_int2(f2fx(z.x), f2fx(z.y));
                    }
                }
                __syncthreads();
                if (STROKE)
                    compact_stroke_block(S, Q.raw, Q.rs, Q.jp, Q.opi, m, spts, subs, *Cs);
                else
                    compact_window_block(S, reinterpret_cast<const int2*>(Q.raw), Q.rs, m, pts, ss, *Cs, limit);
                __syncthreads();
                if (S.capped || S.s_capped) break;
            }
            __syncthreads();
            if (S.capped || S.s_capped) break;
            continue;
        }
        // ---- a curve deeper than a slot walk: the whole chunk depth first
        if (kind == FT_OP_QUAD && !nonfinite) {
            if (STROKE)
                n = quad_walk<true>(A, Bq, C, wa, wb, wc, tol_sq, 0, INT_MAX, &depth_hit, [](int, P2, float) {});
            else
                n = quad_walk<false>(A, Bq, C, 0.f, 0.f, 0.f, tol_sq, 0, INT_MAX, &depth_hit, keep_leaf);
        } else if (kind == FT_OP_CUBIC && !nonfinite) {
            if (STROKE)
                n = cubic_walk<true>(A, Bq, C, D, wa, wb, wc, wd, tol_sq, 0, INT_MAX, &depth_hit,
                                     [](int, P2, float) {});
            else
                n = cubic_walk<false>(A, Bq, C, D, 0.f, 0.f, 0.f, 0.f, tol_sq, 0, INT_MAX, &depth_hit, keep_leaf);
        }
        if (depth_hit) atomicOr(&S.flags, 1);
        int total;
        const int off = G::excl_sum(n, B.scan, total);
        // carry the path-walk state to the next chunk (everyone has read S by now)
        if (tid == N - 1) {
            S.sw = sw_i;
            int last_pc = isPC ? tid : lpc;
            if (last_pc >= 0) {
                S.pen_x = B.penx[last_pc];
                S.pen_y = B.peny[last_pc];
                S.pen_w = B.penw[last_pc];
                S.last_pc_kind = B.kind[last_pc];
            }
        }
        if (rg.p4 && total > WIN) {
            // ---- a chunk of several windows: emit every op's vertices once into the raw
            //      store (super-windows of RAWG when the chunk has more), then compact the
            //      store window by window
            for (int g0 = 0; g0 < total; g0 += RAWG) {
                const int g1 = min(g0 + RAWG, total);
                if (n > 0 && off < g1 && off + n > g0) {
                    const int lo = max(g0, off) - off, hi = min(g1, off + n) - off;
                    if (STROKE) {
                        auto emit = [&](int k, P2 q, float w) {
                            const int idx = off + k - g0;
                            rg.p4[idx] = make_float4(q.x, q.y, w, 0.f);
                            rg.rs[idx] = (k == 0) ? (unsigned char)rs : (unsigned char)0;
                            rg.jp[idx] = (unsigned char)(kind != FT_OP_MOVE);
                            rg.opi[idx] = i;
                        };
                        if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
                            emit(0, A, sw_i);
                        } else if (nonfinite) {
                            emit(0, kind == FT_OP_QUAD ? C : D, kind == FT_OP_QUAD ? wc : wd);
                        } else if (kind == FT_OP_QUAD) {
                            int dh = 0;
                            quad_walk<true>(A, Bq, C, wa, wb, wc, tol_sq, lo, hi, &dh, emit);
                        } else {
                            int dh = 0;
                            cubic_walk<true>(A, Bq, C, D, wa, wb, wc, wd, tol_sq, lo, hi, &dh, emit);
                        }
                    } else {
                        int2* raw2 = reinterpret_cast<int2*>(rg.p4);
                        auto emit = [&](int k, P2 q, float) {
                            const int idx = off + k - g0;
                            raw2[idx] = make_int2(f2fx(q.x), f2fx(q.y));
                            rg.rs[idx] = (k == 0) ? (unsigned char)rs : (unsigned char)0;
                        };
                        if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
                            emit(0, A, 0.f);
                        } else if (nonfinite) {
                            emit(0, kind == FT_OP_QUAD ? C : D, 0.f);
                        } else if (n <= LC) {
                            for (int k = lo; k < hi; k++) {
                                const int idx = off + k - g0;
                                raw2[idx] = cache[k];
                                rg.rs[idx] = (k == 0) ? (unsigned char)rs : (unsigned char)0;
                            }
                        } else if (kind == FT_OP_QUAD) {
                            int dh = 0;
                            quad_walk<false>(A, Bq, C, 0.f, 0.f, 0.f, tol_sq, lo, hi, &dh, emit);
                        } else {
                            int dh = 0;
                            cubic_walk<false>(A, Bq, C, D, 0.f, 0.f, 0.f, 0.f, tol_sq, lo, hi, &dh, emit);
                        }
                    }
                }
                G::sync();
                for (int w0 = g0; w0 < g1; w0 += WIN) {
                    const int w1 = min(w0 + WIN, g1), o = w0 - g0;
                    if (STROKE)
                        compact_stroke_block(S, rg.p4 + o, rg.rs + o, rg.jp + o, rg.opi + o, w1 - w0, spts, subs, *Cs);
                    else
                        compact_window_block(S, reinterpret_cast<const int2*>(rg.p4) + o, rg.rs + o, w1 - w0, pts, ss,
                                             *Cs, limit);
                    G::sync();
                    if (S.capped || S.s_capped) break;
                }
                if (S.capped || S.s_capped) break;
            }
        } else {
            // ---- emit and compact window by window
            for (int w0 = 0; w0 < total; w0 += WIN) {
                const int w1 = min(w0 + WIN, total);
                if (n > 0 && off < w1 && off + n > w0) {
                    const int lo = max(w0, off) - off, hi = min(w1, off + n) - off;
                    if (STROKE) {
                        // stroke points keep f32 coordinates and their width (stroker.rs:204-225)
                        float4* raw4 = reinterpret_cast<float4*>(B.raw);
                        auto emit = [&](int k, P2 q, float w) {
                            const int idx = off + k - w0;
                            raw4[idx] = make_float4(q.x, q.y, w, 0.f);
                            B.rs[idx] = (k == 0) ? (unsigned char)rs : (unsigned char)0;
                            // a Move closes the previous sub-stroke open, a Close joined (F7)
                            B.rs[SRAW + idx] = (unsigned char)(kind != FT_OP_MOVE);
                            opi[idx] = i;
                        };
                        if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
                            emit(0, A, sw_i);
                        } else if (nonfinite) {
                            emit(0, kind == FT_OP_QUAD ? C : D, kind == FT_OP_QUAD ? wc : wd);
                        } else if (kind == FT_OP_QUAD) {
                            int dh = 0;
                            quad_walk<true>(A, Bq, C, wa, wb, wc, tol_sq, lo, hi, &dh, emit);
                        } else {
                            int dh = 0;
                            cubic_walk<true>(A, Bq, C, D, wa, wb, wc, wd, tol_sq, lo, hi, &dh, emit);
                        }
                    } else {
                        auto emit = [&](int k, P2 q, float) {
                            int idx = off + k - w0;
                            B.raw[idx] = make_int2(f2fx(q.x), f2fx(q.y));
                            B.rs[idx] = (k == 0) ? (unsigned char)rs : (unsigned char)0;
                        };
                        if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
                            emit(0, A, 0.f);
                        } else if (nonfinite) {
                            emit(0, kind == FT_OP_QUAD ? C : D, 0.f);
                        } else if (n <= LC) {
                            for (int k = lo; k < hi; k++) {
                                const int idx = off + k - w0;
                                B.raw[idx] = cache[k];
                                B.rs[idx] = (k == 0) ? (unsigned char)rs : (unsigned char)0;
                            }
                        } else if (kind == FT_OP_QUAD) {
                            int dh = 0;
                            quad_walk<false>(A, Bq, C, 0.f, 0.f, 0.f, tol_sq, lo, hi, &dh, emit);
                        } else {
                            int dh = 0;
                            cubic_walk<false>(A, Bq, C, D, 0.f, 0.f, 0.f, 0.f, tol_sq, lo, hi, &dh, emit);
                        }
                    }
                }
                G::sync();
                if constexpr (STROKE) {
                    compact_stroke_block(S, reinterpret_cast<const float4*>(B.raw), B.rs, B.rs + SRAW, opi, w1 - w0,
                                         spts, subs, *Cs);
                } else {
                    compact_window_block(S, B.raw, B.rs, w1 - w0, pts, ss, *Cs, limit);
                }
                G::sync();
                if (S.capped || S.s_capped) break;
            }
        }
        G::sync();
        if (S.capped || S.s_capped) break;
    }
    if (STROKE) {
        G::sync();
        return;
    }
    // Plotter::fill ends with fig.close() (plotter.rs:347)
    if (tid == 0 && !S.capped && S.has_prev && S.rf_x == S.prev_x && S.rf_y == S.prev_y)
        S.count -= 1;
    G::sync();
}

// Direction of a figure from its top vertex `top` (fig.rs:402-411): the vertex after it
// and the one before it in its sub-figure.
__device__ int fig_dir(int top, int count, const int2* pts, const int* ss) {
    const int s = ss[top];
    const int nf = (top + 1 < count && ss[top + 1] == s) ? top + 1 : s;
    int nr;
    if (top > s) {
        nr = top - 1;
    } else {
        // last vertex of the sub-figure: ss[] is non-decreasing
        int lo = top, hi = count - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (ss[mid] == s)
                lo = mid;
            else
                hi = mid - 1;
        }
        nr = lo;
    }
    int2 p = pts[top], p0 = pts[nf], p1 = pts[nr];
    int ax = wsub(p1.x, p.x), ay = wsub(p1.y, p.y);
    int cx = wsub(p0.x, p.x), cy = wsub(p0.y, p.y);
    // (p1 - p).widdershins(p0 - p) -> Forward   (fig.rs:116-119)
    return (fxmul(ax, cy) > fxmul(cx, ay)) ? 0 : 1;
}

// Top vertex (min (y, x, id)) and figure direction (fig.rs:402-411, 493-496).
template <class G>
__device__ void top_and_dir(CState& S, const int2* pts, const int* ss, int* tmp3) {
    const int tid = G::rank(), lane = threadIdx.x & 31, w = tid >> 5;
    const int count = S.count;
    int by = INT_MAX, bx = INT_MAX, bi = INT_MAX;
    for (int i = tid; i < count; i += G::N) {
        int2 p = pts[i];
        if (p.y < by || (p.y == by && (p.x < bx || (p.x == bx && i < bi)))) {
            by = p.y;
            bx = p.x;
            bi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        int oy = __shfl_down_sync(FULL, by, o), ox = __shfl_down_sync(FULL, bx, o), oi = __shfl_down_sync(FULL, bi, o);
        if (oy < by || (oy == by && (ox < bx || (ox == bx && oi < bi)))) {
            by = oy;
            bx = ox;
            bi = oi;
        }
    }
    if (G::N > 32) {
        if (lane == 0) {
            tmp3[3 * w] = by;
            tmp3[3 * w + 1] = bx;
            tmp3[3 * w + 2] = bi;
        }
        G::sync();
    }
    if (tid == 0) {
        for (int k = 1; k < G::N / 32; k++) {
            int oy = tmp3[3 * k], ox = tmp3[3 * k + 1], oi = tmp3[3 * k + 2];
            if (oy < by || (oy == by && (ox < bx || (ox == bx && oi < bi)))) {
                by = oy;
                bx = ox;
                bi = oi;
            }
        }
        S.dir = fig_dir(bi, count, pts, ss);
        S.top_row = by >> 16;
    }
    G::sync();
}

// One edge per non-horizontal segment (fig.rs:179-201, 576-600).
// Edge from vertex i to the next vertex of its sub-figure (fig.rs:179-210, 402-411): its
// rows, slope and direction relative to the figure's; horizontal and degenerate edges
// have ed == 0.
__device__ __forceinline__ EdgeRec edge_rec(int i, int count, int figdir, const int2* pts, const int* ss) {
    const int s = ss[i];
    const int nx = (i + 1 < count && ss[i + 1] == s) ? i + 1 : s;
    EdgeRec e;
    e.ed = 0;
    e.y_upper = e.y_lower = e.x_bot0 = e.inv_slope = e.step_pix = e.start_row = e.end_row = 0;
    if (nx != i) {
        int2 a = pts[i], b = pts[nx];
        if (a.y != b.y) {
            int2 up, lo;
            int edir;
            if (b.y > a.y) {
                up = a;
                lo = b;
                edir = 0;
            } else {
                up = b;
                lo = a;
                edir = 1;
            }
            const int dx = wsub(lo.x, up.x), dy = wsub(lo.y, up.y);
            const int step = dx != 0 ? min(fxabs(fxdiv(dy, dx)), FX_ONE) : 0;
            const int inv = fxdiv(dx, dy);
            const int ybot = wsub(fxfloor(wadd(up.y, FX_ONE)), up.y);
            e.y_upper = up.y;
            e.y_lower = lo.y;
            e.x_bot0 = wadd(up.x, fxmul(inv, ybot));
            e.inv_slope = inv;
            e.step_pix = step;
            e.ed = (edir == figdir) ? 1 : -1;
            e.start_row = up.y >> 16;
            e.end_row = lo.y >> 16;
        }
    }
    return e;
}

// The segments of seg_w pixels that an edge's cells can reach: its x-range between its ends, two
// pixels more to each side for the rounding of its slope, and the longest walk of a row to the
// right of it.  Edges whose x could wrap take every segment.
__device__ __forceinline__ int2 edge_segs(const EdgeRec& e, int segs, int seg_w) {
    const int inv = e.inv_slope, fu = fxfract(e.y_upper), fl = fxfract(e.y_lower);
    const long long end = (long long)(e.end_row - e.start_row) * inv + e.x_bot0 - fxmul(inv, FX_ONE - fl);
    constexpr int FAR = 1 << 29;
    if (abs(end) >= FAR || abs((long long)e.x_bot0) >= FAR || abs((long long)inv) >= FAR) return make_int2(0, segs - 1);
    const int a = e.x_bot0 - fxmul(inv, FX_ONE - fu), z = (int)end;
    const int cells = e.step_pix > 0 ? (int)__fdividef(65536.0f * 1.01f, (float)e.step_pix) + 3 : 4;
    const int lo = (min(a, z) >> 16) - 2, hi = (max(a, z) >> 16) + 2 + cells;
    int2 g = make_int2(0, 0);
    for (int k = 1; k < segs; k++) {
        g.x += lo >= k * seg_w;
        g.y += hi >= k * seg_w;
    }
    return g;
}

// `segs` > 1: an edge's direction goes into the low byte of ed, its segments above it.
template <class G>
__device__ void build_edges(const CState& S, const int2* pts, const int* ss, EdgeRec* edges, int segs = 1, int seg_w = 0) {
    const int count = S.count, figdir = S.dir;
    for (int i = G::rank(); i < count; i += G::N) {
        EdgeRec e = edge_rec(i, count, figdir, pts, ss);
        if (segs > 1 && e.ed) {
            const int2 g = edge_segs(e, segs, seg_w);
            e.ed = (e.ed & 0xFF) | (g.x << 8) | (g.y << 12);
        }
        edges[i] = e;
    }
}

// Signed cell areas of one edge on one scan row (fig.rs:238-321), added into
// `area` (the band row of width W).  The edge on this row: x_bot where it leaves the
// row, its inverse slope, whether the row is its first (st) or last (en), the 16.16
// fractions of its upper and lower y, the cell step (1 .. ONE) and its direction ed.
__device__ __forceinline__ void scan_row(int x_bot, int inv, bool st, bool en, int fu, int fl, int step, int ed,
                                         int* area, int W) {
    const int ccov = en ? pixel_cov(fl) : 256;
    const int cov = st ? ccov - pixel_cov(fu) : ccov;
    if (cov <= 0) return;
    const int x0 = st ? wsub(x_bot, fxmul(inv, wsub(FX_ONE, fu))) : wsub(x_bot, inv);
    // fxceil(y_lower) - y_lower, from the fraction alone
    const int x1 = en ? wsub(x_bot, fxmul(inv, fl ? FX_ONE - fl : 0)) : x_bot;
    const int mnx = min(x0, x1), mxx = max(x0, x1);
    const int minp = mnx >> 16, maxp = mxx >> 16;
    if (minp >= W) return;
    const int full = cov << 8;
    const int r = (minp == maxp) ? fxmul(wsub(FX_ONE, fxfract(fxavg(mxx, mnx))), full)
                                 : fxmul(wsub(FX_ONE, fxfract(mnx)), FX_HALF);
    const int first = fxmul(r, step);  // fxmul(r, ONE) == r
    // fig.rs:292-301: x_cov runs first, first + step, ... capped at ONE; each cell
    // gets the growth of min(pixel_cov(x_cov), cov) until it reaches cov
    const int jmax = W - 1 - minp;  // the loop also stops at the raster's last cell
    int j, prev, x_cov;
    if (minp < 0) {
        // cells left of the raster all land in cell 0 (fig.rs:295): their sum telescopes
        j = -minp;
        long long v = (long long)first + (long long)j * step;
        x_cov = v > FX_ONE ? FX_ONE : (int)v;
        prev = min(pixel_cov(x_cov), cov);
        if (prev && ck(W > 0, 1)) atomicAdd(&area[0], ed * prev);
        j++;
        x_cov = min(x_cov + step, FX_ONE);
    } else {
        j = 0;
        prev = 0;
        x_cov = first;
    }
    if (prev < cov) {
        for (; j <= jmax; j++) {
            const int v = min(pixel_cov(x_cov), cov);
            const int p = v - prev;
            prev = v;
            if (p && ck(minp + j >= 0 && minp + j < W, 2)) atomicAdd(&area[minp + j], ed * p);
            if (v >= cov) break;
            x_cov = min(x_cov + step, FX_ONE);
        }
    }
}

// The cell step of an edge, step_cov(ONE) (fig.rs:315-321): step_pix when positive,
// else ONE; first_cov's r * step equals step_cov(r) for both.
__device__ __forceinline__ int cell_step(const EdgeRec& E) { return E.step_pix > 0 ? E.step_pix : FX_ONE; }

__device__ __forceinline__ void scan_item(const EdgeRec& E, int y, int* area, int W) {
    const int x_bot = wadd(E.x_bot0, wmul(y - E.start_row, E.inv_slope));
    scan_row(x_bot, E.inv_slope, y == E.start_row, y == E.end_row, fxfract(E.y_upper), fxfract(E.y_lower),
             cell_step(E), E.ed, area, W);
}

// Resolve one band row and write it (fig.rs:621-665, imgbuf.rs:38-199).
__device__ __forceinline__ void resolve_row(const int* arow, int W, int Wp, uint8_t* drow, int rule, int fmt,
                                            unsigned clr) {
    const int lane = threadIdx.x & 31;
    unsigned carry = 0;
    for (int x0 = 0; x0 < W; x0 += 128) {
        const int x = x0 + lane * 4;
        int4 a = make_int4(0, 0, 0, 0);
        if (x < Wp) a = *reinterpret_cast<const int4*>(arow + x);
        const unsigned s0 = (unsigned)a.x;
        const unsigned s1 = s0 + (unsigned)a.y;
        const unsigned s2 = s1 + (unsigned)a.z;
        const unsigned s3 = s2 + (unsigned)a.w;
        const unsigned inc = warp_incl_sum_u(s3);
        const unsigned ex = inc - s3 + carry;
        carry += __shfl_sync(FULL, inc, 31);
        const unsigned v0 = resolve_cov(s0 + ex, rule), v1 = resolve_cov(s1 + ex, rule);
        const unsigned v2 = resolve_cov(s2 + ex, rule), v3 = resolve_cov(s3 + ex, rule);
        if (x >= W) continue;
        if (fmt == FT_MATTE8) {
            uint8_t* dp = drow + x;
            if (x + 3 < W && ((reinterpret_cast<uintptr_t>(dp) & 3) == 0)) {
                // masks are written once and not read back: stream them past L2 (evict first),
                // leaving L2 to the rasterisers' figure scratch
                __stcs(reinterpret_cast<unsigned*>(dp), v0 | (v1 << 8) | (v2 << 16) | (v3 << 24));
            } else {
                dp[0] = (uint8_t)v0;
                if (x + 1 < W) dp[1] = (uint8_t)v1;
                if (x + 2 < W) dp[2] = (uint8_t)v2;
                if (x + 3 < W) dp[3] = (uint8_t)v3;
            }
            continue;
        }
        unsigned* dp = reinterpret_cast<unsigned*>(drow) + x;
        const unsigned vv[4] = {v0, v1, v2, v3};
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (x + c < W) dp[c] = srcover_rgba(dp[c], clr, vv[c]);
    }
}

// Rasterise rows [lo, hi) of the built figure, `R` rows per band.
__device__ void raster_rows(const KParams& P, const ft_path_desc& d, const CState& S, const EdgeRec* edges, int lo,
                            int hi, int R, unsigned char* smem) {
    RasterSmem& Rs = *reinterpret_cast<RasterSmem*>(smem);
    int* area = reinterpret_cast<int*>(smem + ((sizeof(RasterSmem) + 15) & ~(size_t)15));
    const int tid = threadIdx.x, warp = tid >> 5;
    const int W = (int)d.width;
    const int Wp = (W + 3) & ~3;
    const int tmin = min(S.top_row, 0);
    const int count = S.count;
    const unsigned clr = (unsigned)d.clr[0] | ((unsigned)d.clr[1] << 8) | ((unsigned)d.clr[2] << 16) |
                         ((unsigned)d.clr[3] << 24);
    uint8_t* base = P.rasters + d.raster_offset;
    for (int r0 = lo; r0 < hi; r0 += R) {
        const int r1 = min(r0 + R, hi);
        const int nr = r1 - r0;
        int4* a4 = reinterpret_cast<int4*>(area);
        for (int i = tid; i < nr * Wp / 4; i += BLOCK) a4[i] = make_int4(0, 0, 0, 0);
        __syncthreads();
        const int yb0 = r0 + tmin, yb1 = r1 + tmin;
        for (int e0 = 0; e0 < count; e0 += BLOCK) {
            const int e = e0 + tid;
            int nrow = 0, ya = 0;
            EdgeRec E;
            E.ed = 0;
            if (e < count) {
                E = edges[e];
                if (E.ed) {
                    ya = max(E.start_row, yb0);
                    const int yb = min(E.end_row, yb1 - 1);
                    nrow = max(yb - ya + 1, 0);
                }
            }
            Rs.edges[tid] = E;
            Rs.ya[tid] = ya;
            int tot;
            const int o = block_excl_sum(nrow, Rs.scan, tot);
            Rs.off[tid] = o;
            // spread the chunk's (edge, row) items over the threads: each edge writes
            // its slot into a run of the item map, then every thread takes items
            for (int m0 = 0; m0 < tot; m0 += MAP_CAP) {
                const int ia = max(o, m0), ib = min(o + nrow, m0 + MAP_CAP);
                for (int k = ia; k < ib; k++) Rs.map[k - m0] = (unsigned char)tid;
                __syncthreads();
                const int n = min(MAP_CAP, tot - m0);
                for (int it = tid; it < n; it += BLOCK) {
                    const int jj = Rs.map[it];
                    const int y = Rs.ya[jj] + (m0 + it - Rs.off[jj]);
                    scan_item(Rs.edges[jj], y, area + (size_t)(y - yb0) * Wp, W);
                }
                __syncthreads();
            }
        }
        for (int rr = r0 + warp; rr < r1; rr += NWARP)
            resolve_row(area + (size_t)(rr - r0) * Wp, W, Wp, base + (size_t)rr * d.stride, P.rule, P.fmt, clr);
        __syncthreads();
    }
}

template <bool STROKE>
__global__ void __launch_bounds__(BLOCK) k_raster(KParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CState S;
    __shared__ int s_item;
    __shared__ int s_tmp3[3 * NWARP];
    const int tid = threadIdx.x;
    unsigned char* scr = P.scratch + (size_t)blockIdx.x * SCRATCH_BYTES_PER_CTA;
    int2* pts = reinterpret_cast<int2*>(scr + SCR_PTS);
    int* ss = reinterpret_cast<int*>(scr + SCR_SS);
    EdgeRec* edges = reinterpret_cast<EdgeRec*>(scr + SCR_EDGES);
    float4* spts = reinterpret_cast<float4*>(scr + SCR_SPTS);
    SubRec* subs = reinterpret_cast<SubRec*>(scr + SCR_SUBS);
    // paths the tile rasteriser handed over (it ran before this kernel)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int n_over = P.overflow && !P.single ? (int)*(volatile uint32_t*)&P.queue[2] : 0;
    for (int round = 0;; round++) {
        WorkItem wi;
        ft_path_desc d;
        if (P.single) {  // CTA b's rows of the one path, unless the tile rasteriser drew them
            if (round || (P.overflow && !*(volatile uint32_t*)&P.overflow[blockIdx.x])) break;
            d = P.d;
            wi = WorkItem{0, (uint32_t)(blockIdx.x * P.rows_per),
                          min(d.height, (uint32_t)((blockIdx.x + 1) * P.rows_per)), 0};
        } else {
            if (tid == 0) s_item = (int)atomicAdd(&P.queue[0], 1u);
            __syncthreads();
            const int it = s_item;
            __syncthreads();
            if (it >= (int)P.n_items + n_over) break;
            if (it < (int)P.n_items) {
                wi = P.items[it];
            } else {
                wi = P.items_w[P.overflow[it - (int)P.n_items]];
                wi.band_rows = 0;
            }
            d = P.paths[wi.path];
        }
        if (wi.band_rows == 0) {
            const int wp4 = (int)(((d.width + 3) & ~3u) * 4);
            wi.band_rows = (uint32_t)max(1, min((P.smem_bytes - RASTER_FIXED_SMEM) / max(wp4, 4), (int)d.height));
        }
        const float sw0 = P.sw_chain ? *P.sw_chain : d.s_width;
        BuildSmem& B = *reinterpret_cast<BuildSmem*>(smem);
        const size_t cs_off = (sizeof(BuildSmem) + 15) & ~(size_t)15;
        CompactSmem* Cs = reinterpret_cast<CompactSmem*>(smem + cs_off);
        if (STROKE) {
            // Plotter::stroke: stroke points, sub-strokes, outline, then the NonZero fill
            int* opi = reinterpret_cast<int*>(smem + cs_off + ((sizeof(CompactSmem) + 15) & ~(size_t)15));
            build_fill<BlockG, true>(P, d, sw0, B, Cs, S, pts, ss, PT_CAP, spts, subs, opi, raw_store(scr));
            finish_subs(P, d, S, subs, B.scan);
            build_outline(P, S, spts, subs, B, *Cs, pts, ss);
        } else {
            build_fill<BlockG>(P, d, sw0, B, Cs, S, pts, ss, PT_CAP, nullptr, nullptr, nullptr, raw_store(scr));
        }
        if (S.count > 0) {
            top_and_dir<BlockG>(S, pts, ss, s_tmp3);
            build_edges<BlockG>(S, pts, ss, edges);
            __syncthreads();
            const int row_begin = max(S.top_row, 0);
            const int lo = max((int)wi.row_begin, row_begin);
            const int hi = min((int)wi.row_end, (int)d.height);
            if (lo < hi && d.width > 0) raster_rows(P, d, S, edges, lo, hi, (int)wi.band_rows, smem);
        }
        // pen width after the call: the last PenWidth op of the path
        if (P.sw_out && wi.row_begin == 0) {
            int lp = -1;
            for (int i = tid; i < (int)d.n_ops; i += BLOCK)
                if (P.ops[d.op_begin + i].kind == FT_OP_PEN_WIDTH) lp = max(lp, i);
            lp = block_incl_max(lp, reinterpret_cast<BuildSmem*>(smem)->scan);
            if (tid == BLOCK - 1) P.sw_out[wi.path] = lp >= 0 ? P.ops[d.op_begin + lp].v[0] : sw0;
        }
        const int st = S.flags ? ((S.flags & 1) ? FT_ERR_DEPTH : FT_ERR_ARG) : FT_OK;
        if (tid == 0 && P.single) {
            if (wi.row_begin == 0) P.status[0] = st;
        } else if (tid == 0 && S.flags) {
            atomicMax(&P.status[wi.path], st);
        }
        __syncthreads();
    }
}

// Shared-memory carve-out (percent of the SM's unified L1) when a launch has at most
// one CTA per SM: the rest stays L1 for the curve walks' local-memory stacks.
constexpr int FEW_CTAS_CARVEOUT = 25;

cudaError_t launch_raster(const KParams& p, int grid, int smem_bytes, cudaStream_t s, bool few_ctas, bool chained) {
    auto kern = p.stroke ? k_raster<true> : k_raster<false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                         few_ctas ? FEW_CTAS_CARVEOUT : (int)cudaSharedmemCarveoutDefault);
    if (chained) return launch_chain(kern, grid, BLOCK, smem_bytes, s, p);
    kern<<<grid, BLOCK, smem_bytes, s>>>(p);
    return cudaGetLastError();
}

// The occupancy query honours the kernel's carve-out preference: a launch of at most one
// CTA per SM leaves FEW_CTAS_CARVEOUT set, under which the query would report one CTA per
// SM, the next grid would again be one CTA per SM and keep that carve-out for good.  The
// query is made with no preference; each launch then sets its own.
int raster_blocks_per_sm(int smem_bytes, bool stroke) {
    auto kern = stroke ? k_raster<true> : k_raster<false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutDefault);
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, BLOCK, smem_bytes) != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

int raster_max_smem() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    int stat = 0;
    if (cudaFuncGetAttributes(&fa, k_raster<true>) == cudaSuccess) stat = (int)fa.sharedSizeBytes;
    return v - stat;
}

}  // namespace ftk

namespace ftk {

// ===========================================================================
// Ordered composite of many paths onto one raster: footile's repeated
// Plotter::fill / Plotter::stroke calls on one Plotter (plotter.rs:339-365).
//
// k_cbuild: one CTA per path builds its figure and edges as k_raster does, then
// bins the edges by raster band into a device pool.  k_cbands (Matte8) draws of each
// row the last call that reaches it.  k_ctile (Rgba8p) walks the paths in call order;
// for each it accumulates the tile's cell areas, resolves its rows and composites.
// Every call of footile composites every pixel from its top row down, alpha 0
// included, and SrcOver with alpha 0 maps each premultiplied channel d to
// ch8_mul(d, 255), which changes only d in 1..15 and is the identity after 15
// applications.  So a tile keeps, per row, the number of
// calls so far and, per four pixels, the call count at their last visit: covered
// pixels first take the alpha-0 maps they missed in one step, uncovered pixels are
// not touched, and the tile ends with one pending flush.

// Bin the built figure's edges by raster band, and by segment of the row where the compositor's
// warps share a row (bins of a band one after another), into the pool (block-wide).
__device__ void bin_edges(const KParams& P, uint32_t path, const CState& S, const EdgeRec* edges, int* hist,
                          int* tmp) {
    const int tid = threadIdx.x;
    const int count = S.count, H = (int)P.canvas_h, R = P.band_rows, segs = P.bin_segs, nb = P.n_bands * segs;
    const int tmin = min(S.top_row, 0);
    const int rb = count > 0 ? max(S.top_row, 0) : H;  // first raster row footile writes
    for (int b = tid; b < nb; b += BLOCK) hist[b] = 0;
    __syncthreads();
    // several edges per thread per step, loaded before they are used (one CTA may bin
    // a whole figure alone: keep several L2 loads in flight); the count pass reads only
    // the half of each record with its rows (step_pix, ed, start_row, end_row)
    auto rows_of = [&](const int4& q, int& lo, int& hi) {
        lo = max(q.z - tmin, rb);
        hi = min(q.w - tmin, H - 1);
        return q.y != 0 && lo <= hi;
    };
    auto segs_of = [&](const int4& q) {
        return segs > 1 ? make_int2((q.y >> 8) & 15, (q.y >> 12) & 15) : make_int2(0, 0);
    };
    // f(bin) for every bin of an edge, unless it has more than LONG: true, and none.
    constexpr int LONG = 128;
    auto each_bin = [&](const int4& q, auto f) {
        int lo, hi;
        if (!rows_of(q, lo, hi)) return false;
        const int b1 = hi / R;
        int b = lo / R;
        const int2 g = segs_of(q);
        if ((b1 - b + 1) * (g.y - g.x + 1) > LONG) return true;
        for (; b <= b1; b++)
            for (int k = g.x; k <= g.y; k++) f(b * segs + k);
        return false;
    };
    const int4* erec = reinterpret_cast<const int4*>(edges);
    // f(bin, edge's record halves) for every bin of the edges that each_bin left out, each over the lanes
    // of a warp: one thread walks the closing line of a fill on 2048 x 2048 through 500 bands and
    // their segments in turn, twice (10 such fills, build and binning: 117 us, by band alone 71 us,
    // this way 41 us).  Edges of fewer bins are done sooner by a thread each.
    auto long_edges = [&](auto f) {
        for (int e0 = tid & ~31; e0 < count; e0 += BLOCK) {
            const int e = e0 + (tid & 31);
            int lo = 0, hi = 0;
            const int4 q = e < count ? erec[2 * e + 1] : make_int4(0, 0, 0, 0);
            int2 g = segs_of(q);
            const bool on = rows_of(q, lo, hi) && (hi / R - lo / R + 1) * (g.y - g.x + 1) > LONG;
            for (unsigned m = __ballot_sync(FULL, on); m; m &= m - 1) {
                const int j = e0 + __ffs(m) - 1;
                const int4 a = erec[2 * j], c = erec[2 * j + 1];
                rows_of(c, lo, hi);
                g = segs_of(c);
                for (int b = lo / R + (tid & 31); b <= hi / R; b += 32)
                    for (int k = g.x; k <= g.y; k++) f(b * segs + k, a, c);
            }
        }
    };
    bool left = false;
    constexpr int EU = 4;
    for (int e0 = 0; e0 < count; e0 += BLOCK * EU) {
        int4 q[EU];
#pragma unroll
        for (int u = 0; u < EU; u++) {
            const int e = e0 + u * BLOCK + tid;
            q[u] = e < count ? erec[2 * e + 1] : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < EU; u++) left |= each_bin(q[u], [&](int b) { atomicAdd(&hist[b], 1); });
    }
    left = __syncthreads_or(left);
    if (left) {
        long_edges([&](int b, const int4&, const int4&) { atomicAdd(&hist[b], 1); });
        __syncthreads();
    }
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += BLOCK) {
        const int b = b0 + tid;
        int tot;
        const int off = block_excl_sum(b < nb ? hist[b] : 0, tmp, tot);
        if (b < nb) hist[b] = carry + off;
        carry += tot;
    }
    __shared__ unsigned long long s_base;
    if (tid == 0) s_base = atomicAdd(P.pool_used, (unsigned long long)carry);
    __syncthreads();
    const unsigned long long base = s_base;
    const bool fits = base + (unsigned long long)carry <= P.pool_cap;
    // bin offsets bin-major (bandoff[b * n_items + path]): the compositors read 32 calls'
    // offsets of one bin as one coalesced load
    for (int b = tid; b <= nb; b += BLOCK)
        P.bandoff[(size_t)b * P.n_items + path] = fits ? (b < nb ? hist[b] : carry) : 0;
    if (tid == 0) {
        P.crec[path] = make_int4(rb, tmin, (int)(unsigned)(base & 0xFFFFFFFFull), (int)(unsigned)(base >> 32));
        if (!fits) atomicMax(&P.status[path], FT_ERR_CAP);  // the host grows the pool and runs again
    }
    __syncthreads();
    if (fits) {
        auto put = [&](int b, const int4& a, const int4& c) {
            const unsigned long long k = base + (unsigned)atomicAdd(&hist[b], 1);
            if (!ck(k < P.pool_cap, 11)) return;
            int4* dst = reinterpret_cast<int4*>(P.pool + k);
            dst[0] = a;
            dst[1] = make_int4(c.x, (int)(signed char)c.y, c.z, c.w);
        };
        constexpr int FU = 2;
        for (int e0 = 0; e0 < count; e0 += BLOCK * FU) {
            int4 q0[FU], q1[FU];
#pragma unroll
            for (int u = 0; u < FU; u++) {
                const int e = e0 + u * BLOCK + tid;
                q0[u] = e < count ? erec[2 * e] : make_int4(0, 0, 0, 0);
                q1[u] = e < count ? erec[2 * e + 1] : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < FU; u++) each_bin(q1[u], [&](int b) { put(b, q0[u], q1[u]); });
        }
        if (left) long_edges(put);
    }
    __syncthreads();
}

// Four CTAs per SM (56 registers for strokes, no spills; 101 unbounded, two CTAs): the
// builds of an ordered composite are latency-bound chains of block scans.
template <bool STROKE>
__global__ void __launch_bounds__(BLOCK, 4) k_cbuild(KParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CState S;
    __shared__ int s_item;
    __shared__ int s_tmp3[3 * NWARP];
    const int tid = threadIdx.x;
    const ScrLayout L = P.L;
    unsigned char* scr = P.scratch + (size_t)blockIdx.x * L.bytes;
    int2* pts = reinterpret_cast<int2*>(scr + L.pts);
    int* ss = reinterpret_cast<int*>(scr + L.ss);
    EdgeRec* edges = reinterpret_cast<EdgeRec*>(scr + L.edges);
    float4* spts = reinterpret_cast<float4*>(scr + L.spts);
    SubRec* subs = reinterpret_cast<SubRec*>(scr + L.subs);
    BuildSmem& B = *reinterpret_cast<BuildSmem*>(smem);
    const size_t cs_off = (sizeof(BuildSmem) + 15) & ~(size_t)15;
    CompactSmem* Cs = reinterpret_cast<CompactSmem*>(smem + cs_off);
    for (;;) {
        if (tid == 0) s_item = (int)atomicAdd(&P.queue[0], 1u);
        __syncthreads();
        const int it = s_item;
        __syncthreads();
        if (it >= (int)P.n_items) break;
        const ft_path_desc d = P.paths[it];
        const float sw0 = P.sw_chain ? *P.sw_chain : d.s_width;
        if (STROKE) {
            int* opi = reinterpret_cast<int*>(smem + cs_off + ((sizeof(CompactSmem) + 15) & ~(size_t)15));
            build_fill<BlockG, true>(P, d, sw0, B, Cs, S, pts, ss, PT_CAP, spts, subs, opi, raw_store(scr, L));
            finish_subs(P, d, S, subs, B.scan);
            build_outline(P, S, spts, subs, B, *Cs, pts, ss);
        } else {
            build_fill<BlockG>(P, d, sw0, B, Cs, S, pts, ss, P.pt_cap, nullptr, nullptr, nullptr,
                               raw_store(scr, L));
        }
        if (P.split_bin) {
            // the figure's edges are built and binned by launch_figure_bins
            if (S.count > 0) top_and_dir<BlockG>(S, pts, ss, s_tmp3);
            __syncthreads();
            if (tid == 0) P.fig_state[it] = make_int4(S.count, S.dir, S.top_row, 0);
        } else {
            if (S.count > 0) {
                top_and_dir<BlockG>(S, pts, ss, s_tmp3);
                build_edges<BlockG>(S, pts, ss, edges, P.bin_segs, P.seg_w);
            }
            __syncthreads();
            bin_edges(P, (uint32_t)it, S, edges, reinterpret_cast<int*>(smem), s_tmp3);
        }
        if (P.sw_out) {  // pen width after the call: the last PenWidth op of the path
            int lp = -1;
            for (int i = tid; i < (int)d.n_ops; i += BLOCK)
                if (P.ops[d.op_begin + i].kind == FT_OP_PEN_WIDTH) lp = max(lp, i);
            lp = block_incl_max(lp, s_tmp3);
            if (tid == BLOCK - 1) P.sw_out[it] = lp >= 0 ? P.ops[d.op_begin + lp].v[0] : sw0;
        }
        if (tid == 0 && S.flags) atomicMax(&P.status[it], (S.flags & 1) ? FT_ERR_DEPTH : FT_ERR_ARG);
        __syncthreads();
    }
}

// Per-warp shared memory of the Matte8 band compositor for rows of `width` pixels: the
// row's i32 cell areas.
__host__ __device__ constexpr int row_smem_bytes(int width) { return (int)align256((size_t)((width + 3) & ~3) * 4); }

// Accumulate the cells of the `ne` band edges that cross scan row y into `row`
// (one warp; each lane takes edges).
__device__ __forceinline__ void row_items(const EdgeRec* edges, int ne, int y, int* row, int W) {
    const int lane = threadIdx.x & 31;
    for (int e = lane; e < ne; e += 32) {
        const EdgeRec E = edges[e];
        if (E.start_row <= y && y <= E.end_row) scan_item(E, y, row, W);
    }
}

// Resolve one Matte8 row (imgbuf.rs:38-199) and overwrite every pixel of it
// (fig.rs:629-636).
__device__ __forceinline__ void matte_row(const int* row, int W, int Wp, uint8_t* drow, int rule) {
    const int lane = threadIdx.x & 31;
    unsigned carry = 0;
    for (int x0 = 0; x0 < W; x0 += 128) {
        const int x = x0 + lane * 4;
        int4 a = make_int4(0, 0, 0, 0);
        if (x < Wp) a = *reinterpret_cast<const int4*>(row + x);
        const unsigned s0 = (unsigned)a.x, s1 = s0 + (unsigned)a.y, s2 = s1 + (unsigned)a.z, s3 = s2 + (unsigned)a.w;
        const unsigned inc = warp_incl_sum_u(s3);
        const unsigned ex = inc - s3 + carry;
        carry += __shfl_sync(FULL, inc, 31);
        const unsigned av[4] = {resolve_cov(s0 + ex, rule), resolve_cov(s1 + ex, rule), resolve_cov(s2 + ex, rule),
                                resolve_cov(s3 + ex, rule)};
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (x + c < W) drow[x + c] = (uint8_t)av[c];
    }
}

// Matte8 ordered composite: every call overwrites its rows from its top row down
// (fig.rs:629-636), so a raster row shows only the last call that reaches it.  One CTA per
// band of P.band_rows rows, one warp per row: the warp finds that call and draws it.  (A single
// call goes to launch_band_single.)
__global__ void __launch_bounds__(BLOCK) k_cbands(KParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = (int)P.canvas_w, H = (int)P.canvas_h, Wp = (W + 3) & ~3;
    const int R = P.band_rows, b = blockIdx.x;
    const int r = b * R + warp;  // this warp's raster row
    if (warp >= R || r >= H) return;
    int* row = reinterpret_cast<int*>(smem + (size_t)warp * row_smem_bytes(W));
    for (int x = lane * 4; x < Wp; x += 128) *reinterpret_cast<int4*>(row + x) = make_int4(0, 0, 0, 0);
    __syncwarp();
    uint8_t* drow = P.rasters + (size_t)r * P.canvas_stride;
    const int n = (int)P.n_items;
    int found = -1;
    for (int c1 = n; c1 > 0 && found < 0; c1 -= 32) {
        const int i = c1 - 32 + lane;
        const bool hit = i >= 0 && P.crec[i].x <= r;
        const unsigned m = __ballot_sync(FULL, hit);
        if (m) found = c1 - 32 + 31 - __clz(m);
    }
    if (found < 0) return;
    const int4 cr = P.crec[found];
    const int o0 = P.bandoff[(size_t)b * n + found], o1 = P.bandoff[(size_t)(b + 1) * n + found];
    const unsigned long long first = ((unsigned long long)(unsigned)cr.z | ((unsigned long long)(unsigned)cr.w << 32)) + o0;
    row_items(P.pool + first, o1 - o0, r + cr.y, row, W);
    __syncwarp();
    matte_row(row, W, Wp, drow, P.rule);
}

// ===========================================================================
// Rgba8p ordered composite on tiles (ft_composite_batch).
//
// A tile is a few rows of one or more segments of P.seg_w pixels, one warp per row and segment,
// its canvas pixels in shared memory: loaded by TMA (cp.async.bulk.tensor.2d, boxes of at most
// 256 pixels wide, completion on an mbarrier) when the canvas allows a tensor map, stored back by
// TMA at the end.  Each warp walks the calls in order.  For a call, the edges crossing its row
// are spread over its lanes; an edge's cells go into the segment's i32 areas in shared memory
// (atomics).  The row is then resolved sparsely: only the 8-pixel chunks that received cells are
// summed (32 at a time, one per lane, a warp scan placing them), and the untouched gap after a
// chunk holds that chunk's final running sum, so it is one run of a single alpha.
//
// Up to CT_MAX_SEGS segments cover the whole row: the build then bins each edge under the
// segments that its cells reach (bin_edges), no warp sees another's edges, and the running sum
// at the end of a segment is handed to the next one's warp through a ring of 64 words, so the
// warps of a row only follow one another.  Wider rows are cut into tiles of one segment, each
// walking all the band's edges: the closed form of an edge's walk gives what it leaves to the
// left of the segment (the cumulative cell sum through column c of an (edge, row) item is
// min(pixel_cov(min(first + (c - minp) * step, ONE)), cov), fig.rs:285-321).
//
// What is composited are quads, four pixels a lane as one 16-byte word, those of the chunks that
// hold any coverage and those of the runs, queued until all lanes have one.  The alpha-0 SrcOver
// footile applies to every other pixel from the call's top row down is applied lazily: a quad
// keeps the number of calls at its last visit (mod 256), and what it missed since is one packed
// step, because the alpha-0 map takes one from channels 1..15 and leaves the rest.
//
// Bound by the instructions issued, at 20 warps per SM (9 KB of shared memory per 1,024 pixels
// would hold 24).  16,384 strokes on 2048 x 2048, 31.5 million (call, row) pairs of 45 edges and 175
// covered pixels each: every warp walking all the band's edges, a queue of single pixels and a
// table for the alpha-0 powers 118 ms; quads, two warps sharing the row's edges between barriers
// 92 ms; one warp resolving a whole row and one compositing behind it 129 ms; this way 80 ms.

constexpr int CT_QN = 96;       // queued quads of a warp: 31 left over and a round's 64
constexpr int CT_CHAIN = 64;    // sums under way from a segment's warp to the next one's

// Tile rows (they divide the band's) and segments: four warps where the band has the rows, never
// more.
struct CTileShape {
    int rows, segs;
};
__host__ __device__ inline CTileShape ctile_shape(int R, int bin_segs) {
    const int want = bin_segs == 1 ? 4 : (bin_segs == 2 ? 2 : 1);
    int rows = want < R ? want : R;
    while (R % rows) rows--;
    return {rows, bin_segs};
}
struct CTileLayout {
    int tile, area, q, runs, bmap, chain, mbar, qi, clist, last, bytes;
};
// Shared memory of a compositor CTA; `staged`: the canvas tile is held in shared memory.
__host__ __device__ inline CTileLayout ctile_layout(CTileShape t, int sw, bool staged) {
    CTileLayout L;
    const int warps = t.rows * t.segs;
    int o = 0;
    L.tile = o;  // canvas pixels, [box][row][box width]
    if (staged) o += warps * sw * 4;
    L.area = o;  // per warp: sw i32 cell areas
    o += warps * sw * 4;
    L.bmap = o;  // per warp: touched 8-pixel chunks, one bit each
    o += warps * 16;
    L.mbar = o;
    o += 16;
    L.q = o;  // per warp: the alphas of queued quads
    o += warps * CT_QN * 4;
    L.runs = o;  // per warp: the gap runs of a round
    o += warps * 32 * 4;
    L.chain = o;  // per row and segment but the last: sums handed on, and how many were taken
    o += t.rows * (t.segs - 1) * (CT_CHAIN + 1) * 4;
    L.qi = o;  // per warp: which quads are queued
    o += warps * CT_QN;
    L.clist = o;  // per warp: touched chunks
    o += warps * (sw / 8);
    L.last = o;  // per warp: calls so far (mod 256) at each quad's last visit
    o += warps * (sw / 4);
    L.bytes = (o + 15) & ~15;
    return L;
}

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// Wait on an mbarrier phase for at most about 0.2 s of GPU time (the global timer);
// false when it did not complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, unsigned parity) {
    const unsigned a = smem_u32(mbar);
    unsigned long long t0 = 0;
    for (int it = 0; it < (1 << 22); it++) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if ((it & 255) == 255) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (!t0) t0 = t;
            if (t - t0 > 200000000ull) break;
        }
    }
    return false;
}

// Wait until `done(word)` of a word in shared memory that another warp writes; false when it gives
// up (CT_POLLS_SMEM).
template <class F>
__device__ __forceinline__ bool smem_wait(const unsigned* word, unsigned& v, F done) {
    Patience p;
    do {
        v = *reinterpret_cast<const volatile unsigned*>(word);
        if (done(v)) return true;
    } while (!p.ends(v, CT_POLLS_SMEM));
    return false;
}

// Wait until a tile's `batch` batches are done; false when it gives up (CT_POLLS_TILE).
__device__ __forceinline__ bool tile_wait(const unsigned* done, const unsigned* rounds, unsigned batch) {
    Patience p;
    unsigned v, r;
    do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(done) : "memory");
        if (v >= batch) return true;
        __nanosleep(200);
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(r) : "l"(rounds) : "memory");
    } while (!p.ends(r, CT_POLLS_TILE));
    return false;
}

// k (at most 15) alpha-0 composites of a pixel: channels 1..15 each lose one per composite
// down to 0 (ch8_mul(d, 255)), channels of 16 and more stay.
__device__ __forceinline__ unsigned alpha0_pow(unsigned d, int k) {
    // bytes whose high nibble is zero, as 0x00 / 0xFF masks
    const unsigned hi = (((d & 0x70707070u) + 0x70707070u) | d) & 0x80808080u;
    unsigned high;  // the top bit of each byte, spread over it
    asm("prmt.b32 %0, %1, %1, 0xBA98;" : "=r"(high) : "r"(hi));
    const unsigned low = ~high;
    const unsigned t = ((d & low) | 0x10101010u) - (unsigned)k * 0x01010101u;  // bit 4: not below 0
    const unsigned ge = (t >> 4) & 0x01010101u;
    return (d & ~low) | (t & 0x0F0F0F0Fu & (ge * 15u) & low);
}
// srcover_rgba with the colour's channels widened (wide8 of each, c0 .. c3), two channels per word
__device__ __forceinline__ unsigned wide8(unsigned v) { return (v << 4) | (v >> 4); }
__device__ __forceinline__ unsigned srcover_wide(unsigned d, unsigned c0, unsigned c1, unsigned c2, unsigned c3,
                                                 unsigned alpha) {
    const unsigned ra = wide8(alpha);
    const unsigned p3 = c3 * ra;
    const unsigned se = __byte_perm(c0 * ra, c2 * ra, 0x7632), so = __byte_perm(c1 * ra, p3, 0x7632);
    const unsigned ri = wide8(255u - (p3 >> 16));
    const unsigned e = d & 0x00FF00FFu, o = (d >> 8) & 0x00FF00FFu;
    const unsigned le = (e << 4) | ((e >> 4) & 0x000F000Fu), lo = (o << 4) | ((o >> 4) & 0x000F000Fu);
    const unsigned de = __byte_perm((le & 0xFFFFu) * ri, (le >> 16) * ri, 0x7632);
    const unsigned dd = __byte_perm((lo & 0xFFFFu) * ri, (lo >> 16) * ri, 0x7632);
    return __vminu2(se + de, 0x00FF00FFu) | (__vminu2(so + dd, 0x00FF00FFu) << 8);
}

// Cells of one (edge, row) item inside [s0, s1) of a raster row (fig.rs:238-321): the cells'
// growths, scaled by 2^16, into `area` (cells from s0 on), the touched 8-pixel chunks into
// `bmap`, and what the item leaves left of s0 into `left0`.
__device__ __forceinline__ void row_cells(const int4 ha, const int4 hb, int y, int* area, unsigned* bmap, int s0, int s1,
                                          unsigned& left0) {
    const int inv = ha.w;
    const bool st = y == hb.z, en = y == hb.w;
    const int fu = fxfract(ha.x), fl = fxfract(ha.y);
    const int cov = (en ? (fl + 128) >> 8 : 256) - (st ? (fu + 128) >> 8 : 0);
    const int xb = wadd(ha.z, wmul(y - hb.z, inv));
    const int x0 = st ? wsub(xb, fxmul(inv, FX_ONE - fu)) : wsub(xb, inv);
    const int x1 = en && fl ? wsub(xb, fxmul(inv, FX_ONE - fl)) : xb;
    const int mnx = min(x0, x1), mxx = max(x0, x1);
    const int minp = mnx >> 16, maxp = mxx >> 16;
    if (cov <= 0 || minp >= s1) return;
    const unsigned step = hb.x > 0 ? hb.x : FX_ONE;
    const unsigned r = minp == maxp ? ((unsigned)(FX_ONE - fxfract(fxavg(mxx, mnx))) * (unsigned)cov) >> 8
                                    : (unsigned)(FX_ONE - fxfract(mnx)) >> 1;
    const unsigned xc0 = (unsigned)(((unsigned long long)r * step) >> 16) + 128u;
    // 256 * the cumulative sum left of cell x > minp, before the cap at cov
    auto upto = [&](int x) {
        const unsigned long long v = xc0 + (unsigned long long)(unsigned)(x - 1 - minp) * step;
        return v > FX_ONE + 128 ? (unsigned)FX_ONE + 128u : (unsigned)v;
    };
    const unsigned ed = (unsigned)hb.y << 16;
    unsigned xc = xc0;
    int prev = 0, c = minp;
    if (minp < s0) {
        c = s0;
        xc = upto(s0);
        if (s0 > 0) {
            prev = min((int)(xc >> 8), cov);
            left0 += ed * (unsigned)prev;
            if (prev >= cov) return;
        }
        xc = min(xc + step, (unsigned)FX_ONE + 128u);
    }
    const int k0 = (c - s0) >> 3;
    int v;
    do {  // four cells a step
#pragma unroll
        for (int u = 0; u < 4; u++) {
            v = min((int)(xc >> 8), cov);
            if (v != prev && c + u < s1 && ck(c + u >= s0, 6)) atomicAdd(area + (c + u - s0), (v - prev) * (int)ed);
            prev = v;
            xc += step;
        }
        c += 4;
    } while (v < cov && c < s1);
    const int k1 = (min(c, s1) - 1 - s0) >> 3;
    for (int w = k0 >> 5; w <= (k1 >> 5); w++) {  // the chunks k0 .. k1
        const int lo = max(k0 - 32 * w, 0), hi = min(k1 - 32 * w, 31);
        if (ck(w >= 0 && w < 4, 7)) atomicOr(&bmap[w], (0xFFFFFFFFu >> (31 - hi)) & (0xFFFFFFFFu << lo));
    }
}

// A barrier of warp `warp` (0 .. 3) alone.  Written out: a barrier number in a register reserves
// all 16, and the SM's 64 then hold four CTAs (81.4 ms; five, with 96 registers, 79.6; six, with
// 80, 85.8).
__device__ __forceinline__ void warp_barrier(int warp) {
    if (warp == 0)
        asm volatile("bar.sync 1, 32;" ::: "memory");
    else if (warp == 1)
        asm volatile("bar.sync 2, 32;" ::: "memory");
    else if (warp == 2)
        asm volatile("bar.sync 3, 32;" ::: "memory");
    else
        asm volatile("bar.sync 4, 32;" ::: "memory");
}

template <bool STAGED, int RULE>
__global__ void __launch_bounds__(128, 5) k_ctile(KParams P, const __grid_constant__ CUtensorMap tmap) {
    extern __shared__ __align__(128) unsigned char smem_tma[];  // TMA destinations: 128-byte aligned
    unsigned char* smem = smem_tma;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = (int)P.canvas_w, H = (int)P.canvas_h, R = P.band_rows, sw = P.seg_w;
    const CTileShape T = ctile_shape(R, P.bin_segs);
    const int span = T.segs * sw, per_row = (W + span - 1) / span;
    const int n_tiles = (H + T.rows - 1) / T.rows * per_row;
    const int wrow = warp / T.segs, seg = warp % T.segs;
    const CTileLayout L = ctile_layout(T, sw, STAGED);
    const int BW = sw < 256 ? sw : 256;  // TMA box width (pixels)
    const int bw_shift = BW == 256 ? 8 : 7;
    unsigned* tile = reinterpret_cast<unsigned*>(smem + L.tile);
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + L.mbar);
    int* area = reinterpret_cast<int*>(smem + L.area) + warp * sw;
    unsigned* q = reinterpret_cast<unsigned*>(smem + L.q) + warp * CT_QN;
    unsigned char* qi = smem + L.qi + warp * CT_QN;
    unsigned* runs = reinterpret_cast<unsigned*>(smem + L.runs) + warp * 32;
    uint4* bmap = reinterpret_cast<uint4*>(smem + L.bmap) + warp;
    unsigned char* clist = smem + L.clist + warp * (sw / 8);
    unsigned char* last = smem + L.last + warp * (sw / 4);
    // sums to the next segment's warp, and from the one before
    unsigned* out = reinterpret_cast<unsigned*>(smem + L.chain) + (wrow * (T.segs - 1) + seg) * (CT_CHAIN + 1);
    unsigned* in = out - (CT_CHAIN + 1);
    const bool has_out = seg + 1 < T.segs, has_in = seg > 0;
    const unsigned lt = (1u << lane) - 1u;
    const int n = (int)P.n_items;
    __shared__ int s_unit;
    if (STAGED && threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int x = lane * 4; x < sw; x += 128) *reinterpret_cast<int4*>(area + x) = make_int4(0, 0, 0, 0);
    if (lane == 0) *bmap = make_uint4(0, 0, 0, 0);
    if (has_out)
        for (int k = lane; k <= CT_CHAIN; k += 32) out[k] = 0;
    bool ok = true;
    unsigned m = 0;  // sums handed on so far
    for (unsigned phase = 0;; phase ^= 1) {
        // the next unit: tile `unit % n_tiles`, call batch `unit / n_tiles`, once the tile's batch before
        // is on the canvas (its CTA took it from the queue earlier, so it is running or done)
        if (threadIdx.x == 0) {
            const int u = (int)atomicAdd(&P.queue[3], 1u);
            s_unit = u;
            if (u >= n_tiles && u < n_tiles * P.tile_batches &&
                !tile_wait(P.tile_done + u % n_tiles, P.tile_done + n_tiles + u % n_tiles, (unsigned)(u / n_tiles)))
                ok = false;
        }
        ok = __syncthreads_and(ok) != 0;
        const int unit = s_unit;
        if (unit >= n_tiles * P.tile_batches) break;
        const int tix = unit % n_tiles, batch = unit / n_tiles;
        const int X0 = tix % per_row * span;  // the tile's pixels: rows y0 .., columns X0 ..
        const int y0 = tix / per_row * T.rows;
        const int r = y0 + wrow, x0 = X0 + seg * sw;
        unsigned* crow = reinterpret_cast<unsigned*>(P.rasters + (size_t)r * P.canvas_stride) + x0;
        const int xend = min(sw, W - x0);                 // the segment's pixels on the canvas
        const int qend = xend > 0 ? (xend + 3) >> 2 : 0;  // and quads
        const int n_box = (min(span, W - X0) + BW - 1) / BW;
        // a quad of this warp: in the shared tile (staged by TMA; pixels right of the canvas are
        // never stored), or in place in global memory, pixel by pixel
        auto quad = [&](int k) {
            const int x = seg * sw + 4 * k;
            return reinterpret_cast<uint4*>(tile + (((x >> bw_shift) * T.rows + wrow) << bw_shift) + (x & (BW - 1)));
        };
        auto get = [&](int k) {
            if (STAGED) return *quad(k);
            const unsigned* p = crow + 4 * k;
            const int left = xend - 4 * k;
            return make_uint4(p[0], left > 1 ? p[1] : 0u, left > 2 ? p[2] : 0u, left > 3 ? p[3] : 0u);
        };
        auto put = [&](int k, uint4 v) {
            if (STAGED) {
                *quad(k) = v;
                return;
            }
            unsigned* p = crow + 4 * k;
            const int left = xend - 4 * k;
            p[0] = v.x;
            if (left > 1) p[1] = v.y;
            if (left > 2) p[2] = v.z;
            if (left > 3) p[3] = v.w;
        };
        if (STAGED && ok && threadIdx.x == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");  // the canvas, acquired, before the copy reads it
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)),
                         "r"(n_box * T.rows * BW * 4)
                         : "memory");
            for (int bx = 0; bx < n_box; bx++)
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                    "%3}], [%4];" ::"r"(smem_u32(tile + bx * T.rows * BW)),
                    "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(X0 + bx * BW), "r"(y0), "r"(smem_u32(mbar))
                    : "memory");
        }
        for (int k = lane; k < sw / 4; k += 32) last[k] = 0;
        if (STAGED && ok) ok = mbar_wait(mbar, phase);
        ok = __syncthreads_and(ok) != 0;
        if (ok && r < H) {
            // the segment's bin of the band, and the band's bins (a call with edges in any of them is
            // walked by all of the row's warps)
            const int b = r / R, s1 = x0 + max(xend, 0);
            const int *bin = P.bandoff + (size_t)(b * T.segs + seg) * n, *bin0 = P.bandoff + (size_t)(b * T.segs) * n;
            const int call0 = (int)((long long)n * batch / P.tile_batches);
            const int call1 = (int)((long long)n * (batch + 1) / P.tile_batches);
            int G = 0;  // calls so far that reach this row
            for (int c0 = call0; c0 < call1; c0 += 32) {
                // 32 calls' records at once, one per lane
                const int i = c0 + lane;
                const int4 cr = i < call1 ? P.crec[i] : make_int4(INT_MAX, 0, 0, 0);
                const bool reach = cr.x <= r;
                int o0 = 0, o1 = 0;
                bool any = false;
                if (i < call1) {
                    o0 = bin[i];
                    o1 = bin[i + n];
                    any = T.segs > 1 ? bin0[i] < bin0[i + (size_t)T.segs * n] : o0 < o1;
                }
                const unsigned rmask = __ballot_sync(FULL, reach);
                unsigned dmask = __ballot_sync(FULL, reach && any);
                const unsigned long long my_first =
                    ((unsigned long long)(unsigned)cr.z | ((unsigned long long)(unsigned)cr.w << 32)) + (unsigned)o0;
                unsigned my_clr = 0;
                if (reach && any) my_clr = *reinterpret_cast<const unsigned*>(P.paths[i].clr);
                if (has_out && ok) {  // room for the sums of these 32 calls
                    unsigned v;
                    ok = __all_sync(FULL, smem_wait(out + CT_CHAIN, v, [&](unsigned d) { return m - d <= CT_CHAIN - 32; }));
                }
                __syncwarp();
                while (dmask) {
                    const int j = __ffs(dmask) - 1;
                    dmask &= dmask - 1;
                    const unsigned long long first = __shfl_sync(FULL, my_first, j);
                    const int ne = __shfl_sync(FULL, o1 - o0, j);
                    const int y = r + __shfl_sync(FULL, cr.y, j);
                    const int4* E = reinterpret_cast<const int4*>(P.pool + first);
                    if (dmask) {  // the next call's first edges, on their way meanwhile
                        const int nj = __ffs(dmask) - 1;
                        const unsigned long long nf = __shfl_sync(FULL, my_first, nj);
                        const int nn = ct_ahead(__shfl_sync(FULL, o1 - o0, nj));
                        if (lane < nn && ck(nf + lane < P.pool_cap, 17))
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(P.pool + nf + lane));
                    }
                    unsigned base = 0;  // the running sum entering the segment
                    for (int e = lane; e < ne; e += 32) {
                        const int4 hb = E[2 * e + 1];  // step_pix, ed, start_row, end_row
                        const int4 ha = E[2 * e];      // y_upper, y_lower, x_bot0, inv_slope
                        if (hb.z <= y && y <= hb.w) row_cells(ha, hb, y, area, reinterpret_cast<unsigned*>(bmap), x0, s1, base);
                    }
                    base = X0 ? __reduce_add_sync(FULL, base) : 0u;
                    // a barrier of this warp alone: after the edge loops' divergent ends the lanes went on
                    // in groups through all that follows, which __syncwarp did not undo (5.9 / 3.7 ms for
                    // 768 strokes)
                    warp_barrier(warp);
                    // the touched chunks, in order
                    const uint4 bw = *bmap;
                    const unsigned bws[4] = {bw.x, bw.y, bw.z, bw.w};
                    int nt = 0;
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        const int at = nt + __popc(bws[w] & lt);
                        if (((bws[w] >> lane) & 1u) && ck(at < sw / 8, 8)) clist[at] = (unsigned char)(32 * w + lane);
                        nt += __popc(bws[w]);
                    }
                    __syncwarp();
                    if (lane == 0) *bmap = make_uint4(0, 0, 0, 0);
                    __syncwarp();
                    const unsigned clr = __shfl_sync(FULL, my_clr, j);
                    const unsigned w0 = wide8(clr & 0xFFu), w1 = wide8((clr >> 8) & 0xFFu),
                                   w2 = wide8((clr >> 16) & 0xFFu), w3 = wide8(clr >> 24);
                    const int Gj = G + __popc(rmask & ((1u << j) - 1u));
                    m++;
                    if (has_in && ok) {  // sums are multiples of 2^16: the count is in the lower half
                        unsigned v = 0;
                        ok = __all_sync(FULL, smem_wait(in + (m & (CT_CHAIN - 1)), v,
                                                        [&](unsigned d) { return ((d ^ m) & 0xFFFFu) == 0; }));
                        base = v & 0xFFFF0000u;
                    }
                    __syncwarp();
                    // the run at hand (quads [run_k, run_e) of alpha run_a, in every byte): at first the
                    // one before the first touched chunk, which holds the sum entering the segment
                    unsigned run_a = resolve4<RULE>((int)base, (int)base, (int)base, (int)base);
                    int run_k = 0, run_e = run_a ? min(nt ? (int)clist[0] * 2 : qend, qend) : 0;
                    unsigned gm = 0;      // runs of the round still to be queued
                    int t0 = 0, cnt = 0;  // chunks done, quads queued
                    bool sent = !has_out;
                    for (;;) {
                        if (cnt < 32) {
                            if (run_k >= run_e && gm) {
                                const unsigned rec = runs[__ffs(gm) - 1];
                                gm &= gm - 1;
                                run_k = (int)(rec >> 20);
                                run_e = (int)((rec >> 8) & 0xFFF);
                                run_a = (rec & 0xFFu) * 0x01010101u;
                            }
                            if (run_k < run_e) {
                                const int k = run_k + lane, add = min(run_e - run_k, 32);
                                if (k < run_e && ck(cnt + lane < CT_QN, 9)) {
                                    q[cnt + lane] = run_a;
                                    qi[cnt + lane] = (unsigned char)k;
                                }
                                run_k += add;
                                cnt += add;
                                __syncwarp();
                                continue;
                            }
                            if (t0 < nt) {
                                const int t = t0 + lane;
                                const bool valid = t < nt;
                                const int ch = valid ? clist[t] : 0;
                                unsigned s[8], inc;
                                take8(area + ch * 8, valid, lane, s, inc);
                                const uint2 px = pixels8<RULE>(s, inc - s[7] + base, 1);
                                base += __shfl_sync(FULL, inc, 31);
                                // the gap after this chunk up to the next touched one holds its last sum
                                const int g0 = ch * 2 + 2, g1 = min((t + 1 < nt ? (int)clist[t + 1] : sw / 8) * 2, qend);
                                const unsigned ga = px.y >> 24;
                                gm = __ballot_sync(FULL, valid && ga && g0 < g1);
                                if (valid) runs[lane] = ((unsigned)g0 << 20) | ((unsigned)g1 << 8) | ga;
                                const bool a0 = valid && px.x && ch * 2 < qend, a1 = valid && px.y && ch * 2 + 1 < qend;
                                const unsigned m0 = __ballot_sync(FULL, a0), m1 = __ballot_sync(FULL, a1);
                                const int at = cnt + __popc(m0 & lt) + __popc(m1 & lt), at1 = at + (a0 ? 1 : 0);
                                if (a0 && ck(at < CT_QN, 9)) {
                                    q[at] = px.x;
                                    qi[at] = (unsigned char)(ch * 2);
                                }
                                if (a1 && ck(at1 < CT_QN, 9)) {
                                    q[at1] = px.y;
                                    qi[at1] = (unsigned char)(ch * 2 + 1);
                                }
                                cnt += __popc(m0) + __popc(m1);
                                t0 += 32;
                                __syncwarp();
                                continue;
                            }
                            if (!sent) {
                                if (lane == 0)
                                    *reinterpret_cast<volatile unsigned*>(out + (m & (CT_CHAIN - 1))) = base | (m & 0xFFFFu);
                                sent = true;
                                __syncwarp();
                            }
                            if (cnt == 0) break;
                        }
                        // composite 32 queued quads (the last of a call: what there is)
                        const int at = max(cnt - 32, 0) + lane;
                        if (at < cnt) {
                            const unsigned a = q[at];
                            const int k = qi[at];
                            if (ck(k < qend, 10)) {
                                uint4 d = get(k);
                                const int kk = min((Gj - (int)last[k]) & 255, 15);
                                last[k] = (unsigned char)(Gj + 1);
                                d.x = srcover_wide(alpha0_pow(d.x, kk), w0, w1, w2, w3, a & 0xFFu);
                                d.y = srcover_wide(alpha0_pow(d.y, kk), w0, w1, w2, w3, (a >> 8) & 0xFFu);
                                d.z = srcover_wide(alpha0_pow(d.z, kk), w0, w1, w2, w3, (a >> 16) & 0xFFu);
                                d.w = srcover_wide(alpha0_pow(d.w, kk), w0, w1, w2, w3, a >> 24);
                                put(k, d);
                            }
                        }
                        cnt = max(cnt - 32, 0);
                        __syncwarp();
                    }
                }
                __syncwarp();
                if (has_in && lane == 0) *reinterpret_cast<volatile unsigned*>(in + CT_CHAIN) = m;
                if (P.tile_batches > 1 && lane == 0) atomicAdd(P.tile_done + n_tiles + tix, 1u);
                const int G0 = G;
                G += __popc(rmask);
                if ((G0 >> 6) != (G >> 6)) {
                    // every 64 calls: pending counts of 15 or more saturate, so a quad's stamp
                    // moves up to 15 calls behind; the u8 differences then stay below 256
                    for (int k = lane; k < sw / 4; k += 32)
                        if (((G - (int)last[k]) & 255) > 15) last[k] = (unsigned char)(G - 15);
                    __syncwarp();
                }
            }
            // the alpha-0 composites still pending since each quad's last visit
            for (int k = lane; k < qend; k += 32) {
                const int kk = min((G - (int)last[k]) & 255, 15);
                if (kk) {
                    uint4 d = get(k);
                    d.x = alpha0_pow(d.x, kk);
                    d.y = alpha0_pow(d.y, kk);
                    d.z = alpha0_pow(d.z, kk);
                    d.w = alpha0_pow(d.w, kk);
                    put(k, d);
                }
            }
        }
        if (STAGED) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        ok = __syncthreads_and(ok) != 0;
        if (threadIdx.x == 0) {
            if (!ok) atomicMax(&P.status[0], FT_ERR_TIMEOUT);
            if (STAGED && ok) {
                for (int bx = 0; bx < n_box; bx++)
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                                     reinterpret_cast<uint64_t>(&tmap)),
                                 "r"(X0 + bx * BW), "r"(y0), "r"(smem_u32(tile + bx * T.rows * BW))
                                 : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                asm volatile("fence.proxy.async;" ::: "memory");
            }
            __threadfence();
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(P.tile_done + tix), "r"((unsigned)batch + 1u) : "memory");
        }
    }
}

// ===========================================================================
// SrcOver of one call from its coverage mask (single large Rgba8p calls).
//
// footile's rasterize_row composites every pixel of the call's rows from its top row down
// with the row's coverage (fig.rs:637-643; alpha 0 where nothing covers).  With the
// call's Matte8 coverage already in a mask (the band compositor writes it), this pass
// streams the canvas and the mask through shared memory by TMA: per tile of 8 rows x
// 256 pixels, a 2-D tensor load of the canvas (u32 pixels) and of the mask (bytes)
// completing on the stage's mbarrier, SrcOver in place, a 2-D tensor store; three stages
// per CTA and six CTAs per SM keep loads, compute and stores in flight together (the
// fastest of 8 / 16 / 32-row tiles with 2 to 6 stages on the 4096x4096 scene).  A pixel with coverage 0
// takes the alpha-0 map, which changes only channel values 1..15: the common case of no
// such channel leaves the pixel as it is.

constexpr int SO_STAGES = 3;  // SO_ROWS x SO_COLS tiles: ft_kernels.cuh (the host's tensor-map boxes)
constexpr int SO_CANVAS_BYTES = SO_ROWS * SO_COLS * 4, SO_MASK_BYTES = SO_ROWS * SO_COLS;
constexpr int SO_STAGE_BYTES = SO_CANVAS_BYTES + SO_MASK_BYTES;
constexpr int SO_SMEM = SO_STAGES * SO_STAGE_BYTES + 128 + 1024;  // stages, mbarriers, colour table

// ch8_mul(d, b) of the four channels of d, b's 12-bit expansion (b << 4 | b >> 4) given
__device__ __forceinline__ unsigned ch8_mul4(unsigned d, unsigned bx) {
    const unsigned e = d & 0x00FF00FFu, o = (d >> 8) & 0x00FF00FFu;  // two channels per word
    const unsigned le = (e << 4) | ((e >> 4) & 0x000F000Fu), lo = (o << 4) | ((o >> 4) & 0x000F000Fu);
    return __byte_perm((le & 0xFFFFu) * bx, (le >> 16) * bx, 0x7632) |
           (__byte_perm((lo & 0xFFFFu) * bx, (lo >> 16) * bx, 0x7632) << 8);
}

// Warps 0..7 composite; warp 8 moves the tiles (one lane issues every TMA operation):
// full[s] completes when stage s holds a loaded tile, done[s] when the eight compositing
// warps have finished it (each warp fences its shared-memory writes for the async proxy
// first), so no CTA-wide barrier sits in the loop.
constexpr int SO_CWARPS = 8;
constexpr int SO_THREADS = 32 * (SO_CWARPS + 1);

__global__ void __launch_bounds__(SO_THREADS, 6) k_srcover_mask(const __grid_constant__ CUtensorMap tm_canvas,
                                                                 const __grid_constant__ CUtensorMap tm_mask, int W,
                                                                 int H, int r0, unsigned clr, int32_t* status) {
    extern __shared__ __align__(128) unsigned char smem_tma[];  // TMA destinations: 128-byte aligned
    unsigned char* smem = smem_tma;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + SO_STAGES * SO_STAGE_BYTES);
    uint64_t* done = full + SO_STAGES;
    // src[a]: the colour's four channels times coverage a (pix's ch8_mul), packed; its
    // alpha byte is the SrcOver's source alpha
    unsigned* src = reinterpret_cast<unsigned*>(smem + SO_STAGES * SO_STAGE_BYTES + 128);
    for (int a = threadIdx.x; a < 256; a += SO_THREADS) src[a] = ch8_mul4(clr, ((unsigned)a << 4) | ((unsigned)a >> 4));
    const int tx = (W + SO_COLS - 1) / SO_COLS, ty = (H - r0 + SO_ROWS - 1) / SO_ROWS;
    const int ntiles = tx * ty;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t cmap = reinterpret_cast<uint64_t>(&tm_canvas), mmap = reinterpret_cast<uint64_t>(&tm_mask);
    auto canvas_s = [&](int st) { return reinterpret_cast<unsigned*>(smem + st * SO_STAGE_BYTES); };
    auto mask_s = [&](int st) { return smem + st * SO_STAGE_BYTES + SO_CANVAS_BYTES; };
    auto tile_x = [&](int t) { return (t % tx) * SO_COLS; };
    auto tile_y = [&](int t) { return r0 + (t / tx) * SO_ROWS; };
    if (threadIdx.x == 0) {
        for (int st = 0; st < SO_STAGES; st++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(full + st)) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(done + st)), "r"(SO_CWARPS)
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // this CTA's tiles: blockIdx.x, blockIdx.x + gridDim.x, ...
    const int mine = ntiles > (int)blockIdx.x ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    auto tile_of = [&](int k) { return (int)blockIdx.x + k * (int)gridDim.x; };
    if (warp == SO_CWARPS) {
        if (lane != 0) return;
        auto load = [&](int k, int st) {
            const int t = tile_of(k);
            const unsigned mb = smem_u32(full + st);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(SO_STAGE_BYTES)
                         : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                "%3}], [%4];" ::"r"(smem_u32(canvas_s(st))),
                "l"(cmap), "r"(tile_x(t)), "r"(tile_y(t)), "r"(mb)
                : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                "%3}], [%4];" ::"r"(smem_u32(mask_s(st))),
                "l"(mmap), "r"(tile_x(t)), "r"(tile_y(t)), "r"(mb)
                : "memory");
        };
        for (int k = 0; k < SO_STAGES && k < mine; k++) load(k, k);
        for (int k = 0; k < mine; k++) {
            const int st = k % SO_STAGES;
            if (!mbar_wait(done + st, (unsigned)((k / SO_STAGES) & 1))) {
                atomicMax(status, FT_ERR_TIMEOUT);
                break;
            }
            const int t = tile_of(k);
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(cmap),
                         "r"(tile_x(t)), "r"(tile_y(t)), "r"(smem_u32(canvas_s(st)))
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            // the stage of tile k - 1 is free once its store has read it: reload it
            if (k >= 1 && k - 1 + SO_STAGES < mine) {
                asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                load(k - 1 + SO_STAGES, (k - 1) % SO_STAGES);
            }
        }
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        return;
    }
    const unsigned whole = src[255];
    const bool opaque = whole >> 24 == 255u;
    for (int k = 0; k < mine; k++) {
        const int st = k % SO_STAGES;
        if (!mbar_wait(full + st, (unsigned)((k / SO_STAGES) & 1))) {
            if (lane == 0) atomicMax(status, FT_ERR_TIMEOUT);
            break;
        }
        unsigned* cv = canvas_s(st);
        const unsigned* mk = reinterpret_cast<const unsigned*>(mask_s(st));
        // four pixels per step: one mask word, four canvas words
        for (int i = threadIdx.x; i < SO_ROWS * SO_COLS / 4; i += 32 * SO_CWARPS) {
            const unsigned m4 = mk[i];
            const uint4 d = reinterpret_cast<const uint4*>(cv)[i];
            unsigned dv[4] = {d.x, d.y, d.z, d.w};
            // alpha 0 changes only channels in 1..15: four pixels unchanged
            if (!m4 && !(low_channels(dv[0]) | low_channels(dv[1]) | low_channels(dv[2]) | low_channels(dv[3]))) continue;
            if (opaque && m4 == 0xFFFFFFFFu) {  // replaced (an opaque fill: 35 us without this, 30.5 with it)
                reinterpret_cast<uint4*>(cv)[i] = make_uint4(whole, whole, whole, whole);
                continue;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                // pix SrcOver: clr * a + d * (255 - clr_alpha * a), channel by channel.  Of pixels that
                // change and that do not alike: with branches the lanes went through it in turns
                // (4096 x 4096 stroke, 40.7 us; all four pixels, and channels by pairs, 31.1 us)
                const unsigned s4 = src[(m4 >> (8 * j)) & 0xFFu];
                const unsigned inv = 255u - (s4 >> 24);
                dv[j] = __vaddus4(s4, ch8_mul4(dv[j], (inv << 4) | (inv >> 4)));
            }
            reinterpret_cast<uint4*>(cv)[i] = make_uint4(dv[0], dv[1], dv[2], dv[3]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(done + st)) : "memory");
    }
}

cudaError_t launch_srcover_mask(const CUtensorMap& canvas, const CUtensorMap& mask, int W, int H, int r0,
                                unsigned clr, int32_t* status, int sm_count, cudaStream_t s) {
    const int ntiles = ((W + SO_COLS - 1) / SO_COLS) * ((H - r0 + SO_ROWS - 1) / SO_ROWS);
    if (ntiles <= 0) return cudaSuccess;
    const int grid = std::max(1, std::min(ntiles, 6 * sm_count));
    k_srcover_mask<<<grid, SO_THREADS, SO_SMEM, s>>>(canvas, mask, W, H, r0, clr, status);
    return cudaGetLastError();
}

int composite_tile_rows(int band_rows, int bin_segs) { return ctile_shape(band_rows, bin_segs).rows; }
int composite_tile_smem(int band_rows, int bin_segs, int seg_w, bool staged) {
    return ctile_layout(ctile_shape(band_rows, bin_segs), seg_w, staged).bytes;
}
int composite_tiles(const KParams& p) {
    const CTileShape t = ctile_shape(p.band_rows, p.bin_segs);
    const int span = t.segs * p.seg_w;
    return ((int)p.canvas_h + t.rows - 1) / t.rows * (((int)p.canvas_w + span - 1) / span);
}

cudaError_t launch_composite_tiles(KParams p, const CUtensorMap& tmap, int sm_count, cudaStream_t s) {
    const bool staged = p.use_tma != 0, odd = p.rule == FT_EVENODD;
    const CTileShape t = ctile_shape(p.band_rows, p.bin_segs);
    const int smem = ctile_layout(t, p.seg_w, staged).bytes;
    auto kern = staged ? (odd ? k_ctile<true, FT_EVENODD> : k_ctile<true, FT_NONZERO>)
                       : (odd ? k_ctile<false, FT_EVENODD> : k_ctile<false, FT_NONZERO>);
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    const int threads = 32 * t.rows * t.segs;
    int per_sm = 0;
    cudaError_t e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem)) != cudaSuccess) return e;
    const int tiles = composite_tiles(p), slots = std::max(1, per_sm) * sm_count;
    // A tile beyond the resident ones would be composited alone, from the first call to the last
    // (1,024 tiles on 912 places take twice as long as 912): the calls are cut into batches, every
    // tile's first batch goes before any second, and the count with the least left over is taken.
    p.tile_batches = 1;
    auto rounds = [&](int nb) { return (double)(((long long)tiles * nb + slots - 1) / slots) / nb; };
    if (tiles > slots)
        for (int nb = 2; nb <= 16 && (int)p.n_items >= 32 * nb; nb++)
            if (rounds(nb) < 0.97 * rounds(p.tile_batches)) p.tile_batches = nb;
    if (p.tile_batches > 1 && (e = cudaMemsetAsync(p.tile_done, 0, 2 * sizeof(unsigned) * tiles, s)) != cudaSuccess) return e;
    kern<<<(int)std::min<long long>((long long)tiles * p.tile_batches, slots), threads, smem, s>>>(p, tmap);
    return cudaGetLastError();
}

int composite_bands_smem(int band_rows, int width) {
    return std::max(band_rows * row_smem_bytes(width), band_single_smem(band_rows, width));
}

// ---- edges and band bins of one path's figure over the whole GPU (split_bin); the
//      figure was built by CTA 0 of k_cbuild.  Band rows follow bin_edges.
struct FigBins {
    int count, figdir, H, R, nb, tmin, rb;
};
__device__ __forceinline__ FigBins fig_bins(const KParams& P) {
    const int4 fs = P.fig_state[0];
    FigBins f;
    f.count = fs.x;
    f.figdir = fs.y;
    f.H = (int)P.canvas_h;
    f.R = P.band_rows;
    f.nb = P.n_bands;
    f.tmin = min(fs.z, 0);
    f.rb = f.count > 0 ? max(fs.z, 0) : f.H;
    return f;
}

// Bands counted in shared memory by each CTA of the edge binning (one global atomic per
// CTA and band instead of one per edge and band); more bands count in global memory.  In
// shared memory an edge adds +1 at its first band and -1 after its last (a difference
// array, two atomics per edge), and a prefix sum gives the counts.
constexpr int BIN_SMEM_BANDS = 8192;

// Counts of this CTA's edges per band: sh[0 .. nb] difference array -> counts in sh[0 .. nb).
__device__ void fig_bin_prefix(int* sh, int nb, int* tmp) {
    __syncthreads();
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += BLOCK) {
        const int b = b0 + threadIdx.x;
        int tot;
        const int v = b < nb ? sh[b] : 0;
        const int ex = block_excl_sum(v, tmp, tot);
        if (b < nb) sh[b] = carry + ex + v;
        carry += tot;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(BLOCK) k_fig_edges(KParams P) {
    chain_link();
    extern __shared__ int sh_bins[];  // n_bands + 1 differences (when n_bands <= BIN_SMEM_BANDS)
    __shared__ int tmp[2 * NWARP + 2];
    const FigBins f = fig_bins(P);
    const bool local = f.nb <= BIN_SMEM_BANDS;
    const unsigned char* scr = P.scratch;
    const int2* pts = reinterpret_cast<const int2*>(scr + P.L.pts);
    const int* ss = reinterpret_cast<const int*>(scr + P.L.ss);
    EdgeRec* edges = reinterpret_cast<EdgeRec*>(P.scratch + P.L.edges);
    if (local) {
        for (int b = threadIdx.x; b <= f.nb; b += BLOCK) sh_bins[b] = 0;
        __syncthreads();
    }
    for (int e = blockIdx.x * BLOCK + threadIdx.x; e < f.count; e += gridDim.x * BLOCK) {
        const EdgeRec E = edge_rec(e, f.count, f.figdir, pts, ss);
        edges[e] = E;
        if (!E.ed) continue;
        const int lo = max(E.start_row - f.tmin, f.rb), hi = min(E.end_row - f.tmin, f.H - 1);
        if (lo > hi) continue;
        if (local) {
            atomicAdd(&sh_bins[lo / f.R], 1);
            atomicAdd(&sh_bins[hi / f.R + 1], -1);
        } else {
            for (int b = lo / f.R; b <= hi / f.R; b++) atomicAdd(&P.bin_hist[b], 1);
        }
    }
    if (local) {
        fig_bin_prefix(sh_bins, f.nb, tmp);
        for (int b = threadIdx.x; b < f.nb; b += BLOCK)
            if (sh_bins[b]) atomicAdd(&P.bin_hist[b], sh_bins[b]);
    }
}

__global__ void __launch_bounds__(BLOCK) k_fig_bin_scan(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ unsigned long long s_base;
    const FigBins f = fig_bins(P);
    const int tid = threadIdx.x;
    int carry = 0;
    for (int b0 = 0; b0 < f.nb; b0 += BLOCK) {
        const int b = b0 + tid;
        int tot;
        const int off = block_excl_sum(b < f.nb ? P.bin_hist[b] : 0, tmp, tot);
        if (b < f.nb) P.bin_hist[f.nb + b] = carry + off;  // fill cursors
        carry += tot;
    }
    if (tid == 0) s_base = atomicAdd(P.pool_used, (unsigned long long)carry);
    __syncthreads();
    const unsigned long long base = s_base;
    const bool fits = base + (unsigned long long)carry <= P.pool_cap;
    for (int b = tid; b <= f.nb; b += BLOCK) P.bandoff[b] = fits ? (b < f.nb ? P.bin_hist[f.nb + b] : carry) : 0;
    if (tid == 0) {
        P.crec[0] = make_int4(f.rb, f.tmin, (int)(unsigned)(base & 0xFFFFFFFFull), (int)(unsigned)(base >> 32));
        P.fig_state[0].w = fits ? 1 : 0;
        if (!fits) atomicMax(&P.status[0], FT_ERR_CAP);  // the host grows the pool and runs again
    }
    // what the host decides on, straight into its memory
    if (tid == 0) {
        *reinterpret_cast<unsigned long long*>(P.summary) = base + (unsigned long long)carry;
        *reinterpret_cast<int4*>(P.summary + 16) = P.crec[0];
    }
    if (P.gb.done && tid < GB_STATE / 8)
        reinterpret_cast<unsigned long long*>(P.summary + GB_STATE)[tid] =
            reinterpret_cast<const unsigned long long*>(P.gb.done)[tid];
}

// (edge, band) pairs of 256 edges at a time spread over the CTA (run-length item map):
// an edge spanning many bands no longer holds one thread for all of them.
struct BinStage {
    int4 q[2 * BLOCK];  // the edges' two halves
    int b0[BLOCK];      // first band
    int off[BLOCK];
    int scan[2 * NWARP + 2];
    unsigned char map[MAP_CAP];
};

__global__ void __launch_bounds__(BLOCK) k_fig_bin_fill(KParams P) {
    chain_link();
    // n_bands + 1 counts, then n_bands cursors (n_bands <= BIN_SMEM_BANDS), then the stage
    extern __shared__ __align__(16) int sh_bins[];
    const FigBins f = fig_bins(P);
    if (!P.fig_state[0].w) return;
    const bool local = f.nb <= BIN_SMEM_BANDS;
    const int4 cr = P.crec[0];
    const unsigned long long base = (unsigned long long)(unsigned)cr.z | ((unsigned long long)(unsigned)cr.w << 32);
    const int4* erec = reinterpret_cast<const int4*>(P.scratch + P.L.edges);
    int* cursor = P.bin_hist + f.nb;
    auto rows_of = [&](const int4& q1, int& lo, int& hi) {
        lo = max(q1.z - f.tmin, f.rb);
        hi = min(q1.w - f.tmin, f.H - 1);
        return q1.y != 0 && lo <= hi;
    };
    if (!local) {
        for (int e = blockIdx.x * BLOCK + threadIdx.x; e < f.count; e += gridDim.x * BLOCK) {
            const int4 q1 = erec[2 * e + 1];  // step_pix, ed, start_row, end_row
            int lo, hi;
            if (!rows_of(q1, lo, hi)) continue;
            const int4 q0 = erec[2 * e];
            for (int b = lo / f.R; b <= hi / f.R; b++) {
                const unsigned long long k = base + (unsigned)atomicAdd(&cursor[b], 1);
                if (!ck(k < P.pool_cap, 12)) continue;
                int4* dst = reinterpret_cast<int4*>(P.pool + k);
                dst[0] = q0;
                dst[1] = q1;
            }
        }
        return;
    }
    const int stage_at = (2 * f.nb + 1 + 3) & ~3;  // ints, 16-byte aligned
    BinStage& Bs = *reinterpret_cast<BinStage*>(sh_bins + stage_at);
    // this CTA's edges per band, then one run of slots per band taken from the cursors
    for (int b = threadIdx.x; b <= f.nb; b += BLOCK) sh_bins[b] = 0;
    __syncthreads();
    for (int e = blockIdx.x * BLOCK + threadIdx.x; e < f.count; e += gridDim.x * BLOCK) {
        int lo, hi;
        if (!rows_of(erec[2 * e + 1], lo, hi)) continue;
        atomicAdd(&sh_bins[lo / f.R], 1);
        atomicAdd(&sh_bins[hi / f.R + 1], -1);
    }
    fig_bin_prefix(sh_bins, f.nb, Bs.scan);
    for (int b = threadIdx.x; b < f.nb; b += BLOCK)
        sh_bins[f.nb + 1 + b] = sh_bins[b] ? atomicAdd(&cursor[b], sh_bins[b]) : 0;
    __syncthreads();
    int* lcur = sh_bins + f.nb + 1;
    for (int e0 = blockIdx.x * BLOCK; e0 < f.count; e0 += gridDim.x * BLOCK) {
        const int e = e0 + threadIdx.x;
        int n = 0, b0 = 0;
        int4 q0 = make_int4(0, 0, 0, 0), q1 = q0;
        if (e < f.count) {
            q1 = erec[2 * e + 1];
            int lo, hi;
            if (rows_of(q1, lo, hi)) {
                q0 = erec[2 * e];
                b0 = lo / f.R;
                n = hi / f.R - b0 + 1;
            }
        }
        Bs.q[2 * threadIdx.x] = q0;
        Bs.q[2 * threadIdx.x + 1] = q1;
        Bs.b0[threadIdx.x] = b0;
        int tot;
        const int o = block_excl_sum(n, Bs.scan, tot);
        Bs.off[threadIdx.x] = o;
        for (int m0 = 0; m0 < tot; m0 += MAP_CAP) {
            const int ia = max(o, m0), ib = min(o + n, m0 + MAP_CAP);
            for (int k = ia; k < ib; k++) Bs.map[k - m0] = (unsigned char)threadIdx.x;
            __syncthreads();
            const int nm = min(MAP_CAP, tot - m0);
            for (int it = threadIdx.x; it < nm; it += BLOCK) {
                const int jj = Bs.map[it];
                const int b = Bs.b0[jj] + (m0 + it - Bs.off[jj]);
                if (!ck(b >= 0 && b < f.nb, 12)) continue;
                const unsigned long long k = base + (unsigned)atomicAdd(&lcur[b], 1);
                if (!ck(k < P.pool_cap, 12)) continue;
                int4* dst = reinterpret_cast<int4*>(P.pool + k);
                dst[0] = Bs.q[2 * jj];
                dst[1] = Bs.q[2 * jj + 1];
            }
            __syncthreads();
        }
    }
}

cudaError_t launch_figure_bins(const KParams& p, int grid, cudaStream_t s) {
    const bool local = p.n_bands <= BIN_SMEM_BANDS;
    const int sm_e = local ? (p.n_bands + 1) * (int)sizeof(int) : 0;
    const int sm_f = local ? ((2 * p.n_bands + 1 + 3) & ~3) * (int)sizeof(int) + (int)sizeof(BinStage) : 0;
    cudaError_t e;
    if ((e = launch_chain(k_fig_edges, grid, BLOCK, sm_e, s, p)) != cudaSuccess) return e;
    if ((e = launch_chain(k_fig_bin_scan, 1, BLOCK, 0, s, p)) != cudaSuccess) return e;
    return launch_chain(k_fig_bin_fill, grid, BLOCK, sm_f, s, p);
}

// ---- grid-wide figure build of one fill path
//
// footile builds the figure sequentially (Fig::add_point / Fig::close, fig.rs:373-461):
// a raw vertex is kept when it starts a sub-figure or differs from the raw vertex before
// it, and a close event (a Move or a Close before the next vertex, and the close that
// Plotter::fill ends with, plotter.rs:347) pops the last vertex when it equals the
// sub-figure's first.  Each of these decisions is a function of the raw stream alone:
//   keep(k) = starts(k) or raw(k) != raw(k-1)
//   pop(k)  = (starts(k+1) or k is the last raw vertex) and raw(k) == raw(R(k)),
//             R(k) the last sub-figure start at or before k,
// and the vertex count when raw vertex l is reached (the pops before it applied) is the
// exclusive prefix sum pos(l) of keep - pop.  A kept vertex goes to position pos(k) with
// sub-figure start pos(R(k)), unless it is the last kept vertex of a sub-figure that pops
// (the next sub-figure's first vertex takes its position).  The cap (65,535, or
// ft_set_figure_cap's) is reached at the first l with pos(l) >= cap: raw vertices from l
// on are ignored, and the count is the cap less one when l starts no sub-figure and
// raw(l-1) equals its sub-figure's first vertex (the close after the cap, as seq_group
// takes it).  Without the cap the count is the sum of keep - pop over all raw vertices.
//
// pos(k) and pos(R(k)) come out of one scan under an associative combination of
// (s: sum of keep - pop, h: has a sub-figure start, r: pos of the last start relative
// to the range's beginning, mp: largest exclusive prefix in the range); mp finds the
// first tile that reaches the cap.  Kernels, in stream order (each scan is run by the
// last CTA of its kernel to finish):
//   k_gb_ops    resets; per 256 ops: the last Move/Line/Quad/Cubic/Close op and the last PenWidth op
//   k_gb_count  every op's pen (the end point of the last such op before it) and raw
//               vertex count (the count walk, 2^d0 lanes per op); scan of the counts
//   k_gb_emit   every op's raw vertices at its offset (the emit walk); per tile of 1,024
//               raw vertices its last sub-figure start, scanned
//   k_gb_keep   keep, pop and R per raw vertex; tile aggregates, scanned
//   k_gb_write  positions, the cap, the vertex and sub-figure start writes
//   k_gb_top    the top vertex (min (y, x, id)), the direction, the figure state
struct PAgg {
    int s, h, r, mp;
};
constexpr int GB_NEG = -(1 << 30);  // mp of the empty range (sums stay within +-2^29)
static_assert(GB_RAW_MAX <= (1ll << 29), "position sums fit the aggregate");
__device__ __forceinline__ PAgg pa_id() { return PAgg{0, 0, 0, GB_NEG}; }
__device__ __forceinline__ PAgg pa_comb(const PAgg& a, const PAgg& b) {
    return PAgg{a.s + b.s, a.h | b.h, b.h ? a.s + b.r : a.r, max(a.mp, a.s + b.mp)};
}
// one raw vertex: keep - pop, and whether it starts a sub-figure
__device__ __forceinline__ PAgg pa_elem(int v, int starts) { return PAgg{v, starts, 0, 0}; }
__device__ __forceinline__ PAgg pa_shfl_up(const PAgg& a, int o) {
    return PAgg{__shfl_up_sync(FULL, a.s, o), __shfl_up_sync(FULL, a.h, o), __shfl_up_sync(FULL, a.r, o),
                __shfl_up_sync(FULL, a.mp, o)};
}
__device__ __forceinline__ PAgg pa_load(const int4* p) {
    const int4 x = __ldcg(p);
    return PAgg{x.x, x.y, x.z, x.w};
}
// Exclusive block scan under pa_comb; `total` receives the whole block's combination.
__device__ PAgg block_scan_pa(PAgg v, PAgg* wt, PAgg& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    PAgg inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const PAgg t = pa_shfl_up(inc, o);
        if (lane >= o) inc = pa_comb(t, inc);
    }
    PAgg ex = pa_shfl_up(inc, 1);
    if (lane == 0) ex = pa_id();
    if (lane == 31) wt[w] = inc;
    __syncthreads();
    PAgg base = pa_id(), all = pa_id();
    for (int k = 0; k < NWARP; k++) {
        if (k == w) base = all;
        all = pa_comb(all, wt[k]);
    }
    total = all;
    __syncthreads();
    return pa_comb(base, ex);
}
__device__ long long block_excl_sum_ll(long long v, long long* tmp, long long& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) tmp[w] = inc;
    __syncthreads();
    long long base = 0, all = 0;
    for (int k = 0; k < NWARP; k++) {
        if (k == w) base = all;
        all += tmp[k];
    }
    total = all;
    __syncthreads();
    return base + inc - v;
}

// True in the last CTA of the grid to get here (after every CTA's global writes).
__device__ bool gb_last_block(unsigned* ticket) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1 ? 1 : 0;
    __syncthreads();
    const bool last = s_last != 0;
    if (last) __threadfence();
    return last;
}

__device__ __forceinline__ ft_op gb_op(const ft_op* ops, int i) {
    const int4* src = reinterpret_cast<const int4*>(ops + i);
    const int4 q0 = __ldg(src), q1 = __ldg(src + 1);
    ft_op op;
    op.kind = q0.x;
    op.v[0] = __int_as_float(q0.y);
    op.v[1] = __int_as_float(q0.z);
    op.v[2] = __int_as_float(q0.w);
    op.v[3] = __int_as_float(q1.x);
    op.v[4] = __int_as_float(q1.y);
    op.v[5] = __int_as_float(q1.z);
    op.reserved = 0;
    return op;
}
// Pen after op j, a Move/Line/Quad/Cubic/Close (a Close puts it at the origin,
// plotter.rs:200-203), and j's kind; j < 0: the origin and kind -1.
__device__ __forceinline__ void gb_pen(const ft_op* ops, int j, float& x, float& y, int& kind) {
    x = 0.f;
    y = 0.f;
    kind = -1;
    if (j < 0) return;
    const ft_op op = gb_op(ops, j);
    kind = op.kind;
    if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
        x = op.v[0];
        y = op.v[1];
    } else if (kind == FT_OP_QUAD) {
        x = op.v[2];
        y = op.v[3];
    } else if (kind == FT_OP_CUBIC) {
        x = op.v[4];
        y = op.v[5];
    }
}
// Raw vertices of a Move/Line/Quad/Cubic op with the pen at (px, py), as build_fill
// flattens them for a fill, split over 2^d0 lanes: lane s takes the subtree of the
// curve's subdivision whose path from the root is the d0 bits of s (left half 0, in
// the depth-first order of the walk); a leaf above that depth goes to the first lane of
// its range, a Move or Line to lane 0.  Each subtree is the walk's own arithmetic, so the
// lanes' leaves in lane order are the walk's leaves.  emit(k, vertex) for the lane's k-th
// leaf; returns the lane's leaf count.  flags: 1 depth cap reached, 2 non-finite control
// point.
template <class Emit>
__device__ int gb_walk(const KParams& P, const ft_op& op, int kind, float px, float py, int lane, int d0, int& flags,
                       Emit emit) {
    if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
        if (lane) return 0;
        const P2 A = xform(P.xf, p2(op.v[0], op.v[1]));
        emit(0, make_int2(f2fx(A.x), f2fx(A.y)));
        return 1;
    }
    P2 a = xform(P.xf, p2(px, py)), b = xform(P.xf, p2(op.v[0], op.v[1])), c = xform(P.xf, p2(op.v[2], op.v[3]));
    auto leaf = [&](int k, P2 q, float) { emit(k, make_int2(f2fx(q.x), f2fx(q.y))); };
    const float tol_sq = P.tol_sq;
    int dh = 0, n;
    if (kind == FT_OP_QUAD) {
        if (!pfinite(a) || !pfinite(b) || !pfinite(c)) {
            if (lane) return 0;
            flags |= 2;
            emit(0, make_int2(f2fx(c.x), f2fx(c.y)));
            return 1;
        }
        for (int d = 0; d < d0; d++) {
            const P2 ab = pmid(a, b), bc = pmid(b, c), abbc = pmid(ab, bc), ac = pmid(a, c);
            const bool within = pdist_sq(abbc, ac) <= tol_sq;
            if (within || d >= FT_MAX_DEPTH) {
                if (lane & ((1 << (d0 - d)) - 1)) return 0;
                if (!within) flags |= 1;
                emit(0, make_int2(f2fx(c.x), f2fx(c.y)));
                return 1;
            }
            if ((lane >> (d0 - 1 - d)) & 1) {
                a = abbc;
                b = bc;
            } else {
                b = ab;
                c = abbc;
            }
        }
        n = quad_walk<false>(a, b, c, 0.f, 0.f, 0.f, tol_sq, 0, INT_MAX, &dh, leaf, d0);
    } else {
        P2 e = xform(P.xf, p2(op.v[4], op.v[5]));
        if (!pfinite(a) || !pfinite(b) || !pfinite(c) || !pfinite(e)) {
            if (lane) return 0;
            flags |= 2;
            emit(0, make_int2(f2fx(e.x), f2fx(e.y)));
            return 1;
        }
        for (int d = 0; d < d0; d++) {
            const P2 ab = pmid(a, b), bc = pmid(b, c), cd = pmid(c, e);
            const P2 abbc = pmid(ab, bc), bccd = pmid(bc, cd);
            const P2 pe = pmid(abbc, bccd), ad = pmid(a, e);
            const bool within = pdist_sq(pe, ad) <= tol_sq;
            if (within || d >= FT_MAX_DEPTH) {
                if (lane & ((1 << (d0 - d)) - 1)) return 0;
                if (!within) flags |= 1;
                emit(0, make_int2(f2fx(e.x), f2fx(e.y)));
                return 1;
            }
            if ((lane >> (d0 - 1 - d)) & 1) {
                a = pe;
                b = bccd;
                c = cd;
            } else {
                b = ab;
                c = abbc;
                e = pe;
            }
        }
        n = cubic_walk<false>(a, b, c, e, 0.f, 0.f, 0.f, 0.f, tol_sq, 0, INT_MAX, &dh, leaf, d0);
    }
    if (dh) flags |= 1;
    return n;
}

__global__ void __launch_bounds__(BLOCK) k_gb_ops(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ int s_tot[3];
    const GridBuildBufs& G = P.gb;
    const int tid = threadIdx.x, i = blockIdx.x * BLOCK + tid;
    // what the kernels behind this one count in
    for (int k = i; k < G.n_tr; k += gridDim.x * BLOCK) G.tr_all[k] = -1;
    for (int k = i; k < P.n_bands; k += gridDim.x * BLOCK) P.bin_hist[k] = 0;
    if (i < 64) P.queue[i] = 0;
    if (i == 0) {
        P.status[0] = 0;
        *P.pool_used = 0;
        P.fig_state[0] = make_int4(0, 0, 0, 0);
    }
    const int kind = i < G.n_ops ? __ldg(&G.ops[i].kind) : -1;
    int mpc, lpc;
    block_max_scan((kind >= FT_OP_CLOSE && kind <= FT_OP_CUBIC) ? i : -1, tmp, mpc, lpc);
    const int mpw = block_incl_max(kind == FT_OP_PEN_WIDTH ? i : -1, tmp);
    const int mcm = block_incl_max((kind == FT_OP_CLOSE || kind == FT_OP_MOVE) ? i : -1, tmp);
    if (i < G.n_ops) {
        G.opi[i].x = lpc;  // the block's part; k_gb_count adds the blocks before
        G.opw[i] = mpw;
    }
    if (tid == BLOCK - 1) G.opa[blockIdx.x] = make_int4(mpc, mpw, mcm, 0);
    if (!gb_last_block(&G.done[0])) return;
    // exclusive max over the blocks, in place
    const int nb = (int)gridDim.x;
    int cpc = -1, cpw = -1, ccm = -1;
    for (int b0 = 0; b0 < nb; b0 += BLOCK) {
        const int b = b0 + tid;
        const int4 a = b < nb ? __ldcg(&G.opa[b]) : make_int4(-1, -1, -1, 0);
        int ipc, epc, ipw, epw, icm, ecm;
        block_max_scan(a.x, tmp, ipc, epc);
        if (tid == BLOCK - 1) s_tot[0] = ipc;
        block_max_scan(a.y, tmp, ipw, epw);
        if (tid == BLOCK - 1) s_tot[1] = ipw;
        block_max_scan(a.z, tmp, icm, ecm);
        if (tid == BLOCK - 1) s_tot[2] = icm;
        __syncthreads();
        if (b < nb) G.opa[b] = make_int4(max(cpc, epc), max(cpw, epw), max(ccm, ecm), 0);
        cpc = max(cpc, s_tot[0]);
        cpw = max(cpw, s_tot[1]);
        ccm = max(ccm, s_tot[2]);
        __syncthreads();
    }
    if (tid == 0) {
        // pen width after the call: the last PenWidth op of the path
        if (P.sw_out) P.sw_out[0] = cpw >= 0 ? G.ops[cpw].v[0] : *G.s_width;
        if (P.gs.st) {
            P.gs.st[3] = cpc;
            P.gs.st[4] = ccm;
        }
    }
}

// A lane's op of block `blk` of the walks (2^d0 lanes an op) and its pen.
struct GbOp {
    int i, lane, kind, lpc, rs;
    float px, py;
    ft_op op;
};
__device__ __forceinline__ GbOp gb_op_of(const GridBuildBufs& G, int blk, int& flags) {
    GbOp o;
    o.i = (int)(((unsigned)blk * BLOCK + threadIdx.x) >> G.d0);
    o.lane = (int)(threadIdx.x & ((1u << G.d0) - 1u));
    o.kind = -1;
    o.lpc = -1;
    o.rs = 0;
    o.px = o.py = 0.f;
    if (o.i >= G.n_ops) return o;
    o.op = gb_op(G.ops, o.i);
    o.kind = o.op.kind;
    if (o.kind < -1 || o.kind > FT_OP_PEN_WIDTH) {
        if (o.lane == 0) flags |= 2;
        o.kind = -1;
    }
    o.lpc = max(G.opi[o.i].x, G.opa[o.i / BLOCK].x);
    int pk = -1;
    if (o.kind >= FT_OP_MOVE && o.kind <= FT_OP_CUBIC) gb_pen(G.ops, o.lpc, o.px, o.py, pk);
    // the first vertex of this op starts a sub-figure after a close event
    o.rs = o.kind == FT_OP_MOVE || pk == FT_OP_CLOSE || pk == -1;
    return o;
}

__global__ void __launch_bounds__(BLOCK) k_gb_count(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ long long ltmp[NWARP];
    const GridBuildBufs& G = P.gb;
    if (G.skip && *G.skip) return;  // a probe over a prefix of the ops completed the figure
    const int tid = threadIdx.x;
    int flags = 0;
    for (int blk = blockIdx.x; blk < gb_ctas(G.n_ops); blk += gridDim.x) {
        const GbOp o = gb_op_of(G, blk, flags);
        int n = 0;
        if (o.kind >= FT_OP_MOVE && o.kind <= FT_OP_CUBIC)
            n = gb_walk(P, o.op, o.kind, o.px, o.py, o.lane, G.d0, flags, [](int, int2) {});
        // the lanes' offsets within the op, the ops' offsets within the CTA
        int inc = n;
        const int lanes = 1 << G.d0;
        for (int d = 1; d < lanes; d <<= 1) {
            const int t = __shfl_up_sync(FULL, inc, d, lanes);
            if (o.lane >= d) inc += t;
        }
        const int n_op = __shfl_sync(FULL, inc, lanes - 1, lanes);
        int tot;
        const int ex = block_excl_sum(o.lane == 0 ? n_op : 0, tmp, tot);
        if (o.i < G.n_ops) {
            G.opl[(o.i << G.d0) + o.lane] = inc - n;
            if (o.lane == 0) G.opi[o.i].y = ex;
        }
        if (tid == 0) G.opn[blk] = tot;
    }
    if (flags) atomicMax(&P.status[0], (flags & 1) ? FT_ERR_DEPTH : FT_ERR_ARG);
    if (!gb_last_block(&G.done[1])) return;
    // exclusive sum over the blocks, in place; the total is the path's raw vertex count
    const int nb = gb_ctas(G.n_ops);
    long long carry = 0;
    for (int b0 = 0; b0 < nb; b0 += BLOCK) {
        const int b = b0 + tid;
        long long t;
        const long long e = block_excl_sum_ll(b < nb ? __ldcg(&G.opn[b]) : 0ll, ltmp, t);
        if (b < nb) G.opn[b] = carry + e;
        carry += t;
    }
    if (tid == 0) *G.n_raw = carry;
}

// Exclusive max of the tiles' last sub-figure starts, in place (one CTA).
__device__ void gb_scan_tr(const GridBuildBufs& G, long long n_raw, int* tmp, int& s_c) {
    const int tid = threadIdx.x, nt = (int)((n_raw + GB_TILE - 1) / GB_TILE);
    int carry = -1;
    for (int b0 = 0; b0 < nt; b0 += BLOCK) {
        const int b = b0 + tid;
        int inc, exc;
        block_max_scan(b < nt ? __ldcg(&G.tr[b]) : -1, tmp, inc, exc);
        if (tid == BLOCK - 1) s_c = inc;
        __syncthreads();
        if (b < nt) G.tr[b] = max(carry, exc);
        carry = max(carry, s_c);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(BLOCK) k_gb_emit(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ int s_c;
    const GridBuildBufs& G = P.gb;
    if (G.skip && *G.skip) return;  // a probe over a prefix of the ops completed the figure
    const long long n_raw = *G.n_raw;
    if (n_raw > G.raw_cap) return;  // every CTA: the caller grows the arrays
    int flags = 0;
    for (int blk = blockIdx.x; blk < gb_ctas(G.n_ops); blk += gridDim.x) {
        const GbOp o = gb_op_of(G, blk, flags);
        if (o.kind >= FT_OP_MOVE && o.kind <= FT_OP_CUBIC) {
            const long long off0 = G.opn[blk] + G.opi[o.i].y;
            const int off = (int)(off0 + G.opl[(o.i << G.d0) + o.lane]);
            int2* raw = G.raw;
            unsigned char* fl = G.fl;
            const int cap = G.raw_cap;
            const unsigned char rs0 = (o.lane == 0 && o.rs) ? 1 : 0;
            gb_walk(P, o.op, o.kind, o.px, o.py, o.lane, G.d0, flags, [&](int k, int2 q) {
                if (ck(off + k < cap, 13) && off + k < cap) {
                    raw[off + k] = q;
                    fl[off + k] = k == 0 ? rs0 : (unsigned char)0;
                }
            });
            if (rs0 && ck(off < cap, 13) && off < cap) atomicMax(&G.tr[off / GB_TILE], off);
        }
    }
    if (!gb_last_block(&G.done[2])) return;
    gb_scan_tr(G, n_raw, tmp, s_c);
}

__global__ void __launch_bounds__(BLOCK) k_gb_keep(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ PAgg wt[NWARP];
    const GridBuildBufs& G = P.gb;
    if (G.skip && *G.skip) return;  // a probe over a prefix of the ops completed the figure
    const long long n_raw = *G.n_raw;
    if (n_raw > G.raw_cap) return;
    const int M = (int)n_raw, nt = (M + GB_TILE - 1) / GB_TILE, tid = threadIdx.x;
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const int k0 = t * GB_TILE + GB_PER * tid;
        int2 p[GB_PER];
        int rl[GB_PER];
        int st = 0, run = -1;
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            p[j] = make_int2(0, 0);
            if (k < M) {
                p[j] = G.raw[k];
                if (G.fl[k] & 1) {
                    st |= 1 << j;
                    run = k;
                }
            }
            rl[j] = run;
        }
        int inc, exc;
        block_max_scan(run, tmp, inc, exc);
        const int carry = max(G.tr[t], exc);
        int2 q = (k0 > 0 && k0 <= M) ? G.raw[k0 - 1] : make_int2(0, 0);  // raw predecessor
        PAgg a = pa_id();
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            if (k < M) {
                const int R = max(0, max(carry, rl[j]));  // raw vertex 0 always starts one
                const int2 f = G.raw[R];
                const int s = (st >> j) & 1;
                const bool keep = s || p[j].x != q.x || p[j].y != q.y;
                const bool ends = k + 1 >= M || (G.fl[k + 1] & 1);
                const bool pop = ends && p[j].x == f.x && p[j].y == f.y;
                G.kp[k] = (unsigned char)((keep ? 1 : 0) | (pop ? 2 : 0));
                G.rk[k] = R;
                a = pa_comb(a, pa_elem((keep ? 1 : 0) - (pop ? 1 : 0), s));
            }
            q = p[j];
        }
        PAgg tot;
        block_scan_pa(a, wt, tot);
        if (tid == 0) G.tp[t] = make_int4(tot.s, tot.h, tot.r, tot.mp);
    }
    if (!gb_last_block(&G.done[3])) return;
    // exclusive scan of the tiles, in place, GB_PER tiles a thread; the total is the
    // vertex count when the cap is not reached
    PAgg carry = pa_id();
    for (int b0 = 0; b0 < nt; b0 += GB_TILE) {
        const int b = b0 + GB_PER * tid;
        PAgg v[GB_PER], a = pa_id();
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            v[j] = b + j < nt ? pa_load(&G.tp[b + j]) : pa_id();
            a = pa_comb(a, v[j]);
        }
        PAgg tot;
        PAgg ex = pa_comb(carry, block_scan_pa(a, wt, tot));
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            if (b + j < nt) G.tp[b + j] = make_int4(ex.s, ex.h, ex.r, ex.mp);
            ex = pa_comb(ex, v[j]);
        }
        carry = pa_comb(carry, tot);
    }
    if (tid == 0) *G.count = carry.s;
}

__global__ void __launch_bounds__(BLOCK) k_gb_write(KParams P) {
    chain_link();
    __shared__ PAgg wt[NWARP];
    __shared__ int s_l;
    const GridBuildBufs& G = P.gb;
    if (G.skip && *G.skip) return;  // a probe over a prefix of the ops completed the figure
    const long long n_raw = *G.n_raw;
    if (n_raw > G.raw_cap) return;
    const int M = (int)n_raw, nt = (M + GB_TILE - 1) / GB_TILE, tid = threadIdx.x, cap = P.pt_cap;
    int2* pts = reinterpret_cast<int2*>(P.scratch + P.L.pts);
    int* ss = reinterpret_cast<int*>(P.scratch + P.L.ss);
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const PAgg C = pa_load(&G.tp[t]);
        if (C.mp >= cap) continue;  // the cap was reached before this tile
        const int k0 = t * GB_TILE + GB_PER * tid;
        int kp[GB_PER], st[GB_PER];
        PAgg a = pa_id();
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            kp[j] = 0;
            st[j] = 0;
            if (k < M) {
                kp[j] = G.kp[k];
                st[j] = G.fl[k] & 1;
                a = pa_comb(a, pa_elem((kp[j] & 1) - ((kp[j] >> 1) & 1), st[j]));
            }
        }
        if (tid == 0) s_l = INT_MAX;
        PAgg tot;
        PAgg run = pa_comb(C, block_scan_pa(a, wt, tot));
        int pos[GB_PER], posr[GB_PER], lc = INT_MAX;
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            pos[j] = run.s;
            if (k < M) {
                if (run.s >= cap) lc = min(lc, k);
                run = pa_comb(run, pa_elem((kp[j] & 1) - ((kp[j] >> 1) & 1), st[j]));
            }
            posr[j] = run.r;
        }
        if (lc != INT_MAX) atomicMin(&s_l, lc);
        __syncthreads();
        const int l = s_l;  // first raw vertex at the cap, INT_MAX: not in this tile
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            if (k >= M || k >= l || !(kp[j] & 1)) continue;
            const int2 v = G.raw[k], f = G.raw[G.rk[k]];
            bool gone = false;
            if (v.x == f.x && v.y == f.y) {
                // the last kept vertex of a sub-figure that pops: the next kept vertex
                // starts a sub-figure (or there is none)
                int m = k + 1;
                while (m < M && !(G.kp[m] & 1)) m++;
                gone = m >= M || (G.fl[m] & 1);
            }
            if (!gone && ck(pos[j] >= 0 && pos[j] < cap, 14) && pos[j] >= 0 && pos[j] < cap) {
                pts[pos[j]] = v;
                ss[pos[j]] = posr[j];
            }
        }
        if (l != INT_MAX && l >= k0 && l < k0 + GB_PER) {
            // the close after the cap pops the last vertex if it equals its sub-figure's first
            const int2 v = G.raw[l - 1], f = G.raw[G.rk[l - 1]];
            *G.count = cap - ((!(G.fl[l] & 1) && v.x == f.x && v.y == f.y) ? 1 : 0);
            if (G.final_flag) *G.final_flag = 1;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(BLOCK) k_gb_top(KParams P) {
    chain_link();
    __shared__ int4 wb[NWARP];
    const GridBuildBufs& G = P.gb;
    if (G.skip && *G.skip) return;  // a probe over a prefix of the ops completed the figure
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int count = *G.n_raw > G.raw_cap ? 0 : *G.count;
    const int2* pts = reinterpret_cast<const int2*>(P.scratch + P.L.pts);
    const int* ss = reinterpret_cast<const int*>(P.scratch + P.L.ss);
    int by = INT_MAX, bx = INT_MAX, bi = INT_MAX;
    for (int i = blockIdx.x * BLOCK + tid; i < count; i += gridDim.x * BLOCK) {
        const int2 p = pts[i];
        if (top_less(p.y, p.x, i, by, bx, bi)) {
            by = p.y;
            bx = p.x;
            bi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int oy = __shfl_down_sync(FULL, by, o), ox = __shfl_down_sync(FULL, bx, o),
                  oi = __shfl_down_sync(FULL, bi, o);
        if (top_less(oy, ox, oi, by, bx, bi)) {
            by = oy;
            bx = ox;
            bi = oi;
        }
    }
    if (lane == 0) wb[w] = make_int4(by, bx, bi, 0);
    __syncthreads();
    if (tid == 0) {
        int4 b = wb[0];
        for (int k = 1; k < NWARP; k++)
            if (top_less(wb[k].x, wb[k].y, wb[k].z, b.x, b.y, b.z)) b = wb[k];
        G.top[blockIdx.x] = b;
    }
    if (!gb_last_block(&G.done[4])) return;
    by = bx = bi = INT_MAX;
    for (int k = tid; k < (int)gridDim.x; k += BLOCK) {
        const int4 o = __ldcg(&G.top[k]);
        if (top_less(o.x, o.y, o.z, by, bx, bi)) {
            by = o.x;
            bx = o.y;
            bi = o.z;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int oy = __shfl_down_sync(FULL, by, o), ox = __shfl_down_sync(FULL, bx, o),
                  oi = __shfl_down_sync(FULL, bi, o);
        if (top_less(oy, ox, oi, by, bx, bi)) {
            by = oy;
            bx = ox;
            bi = oi;
        }
    }
    __syncthreads();
    if (lane == 0) wb[w] = make_int4(by, bx, bi, 0);
    __syncthreads();
    if (tid == 0) {
        int4 b = wb[0];
        for (int k = 1; k < NWARP; k++)
            if (top_less(wb[k].x, wb[k].y, wb[k].z, b.x, b.y, b.z)) b = wb[k];
        P.fig_state[0] = count > 0 ? make_int4(count, fig_dir(b.z, count, pts, ss), b.x >> 16, 0)
                                   : make_int4(0, 0, 0, 0);
    }
}

cudaError_t launch_grid_build(const KParams& p, int sm_count, cudaStream_t s, const KParams* probe) {
    const int nbo = (p.gb.n_ops + BLOCK - 1) / BLOCK;
    if (nbo <= 0 || p.gb.raw_cap % GB_TILE || p.gb.raw_cap > GB_RAW_MAX) return cudaErrorInvalidValue;
    if (probe && (probe->gb.n_ops <= 0 || probe->gb.n_ops > p.gb.n_ops)) return cudaErrorInvalidValue;
    const int gt = std::max(1, 4 * sm_count);
    cudaError_t e;
    if ((e = launch_chain(k_gb_ops, nbo, BLOCK, 0, s, p)) != cudaSuccess) return e;  // pens of every op (the probe's too) and the pen width after
    for (const KParams* q : {probe, &p}) {
        if (!q) continue;
        const int nbw = std::min(gb_ctas(q->gb.n_ops), 8 * sm_count);  // all resident: a skipped build only launches these
        if ((e = launch_chain(k_gb_count, nbw, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gb_emit, nbw, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gb_keep, gt, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gb_write, gt, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gb_top, GB_TOP_BLOCKS, BLOCK, 0, s, *q)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ---- grid-wide build of one stroke path
//
// Plotter::stroke (plotter.rs:356-365) collects the stroke points (Stroke::add_point and
// close, stroker.rs:204-236), makes every sub-stroke's outline (stroker.rs:239-416) and
// fills it NonZero.  Over the whole GPU, in stream order:
//   k_gb_ops    pens, the last PenWidth op at or before each op, the last Close/Move op
//   k_gs_count  every op's raw stroke points (the walk carrying widths, 2^d0 lanes
//               per op), scanned
//   k_gs_emit   the raw points (x, y, width), whether each starts a sub-stroke, its op
//   k_gs_keep   per raw point: kept when it starts a sub-stroke or its f32 position
//               differs from the raw point before it (no closing point is popped); per
//               tile the kept points and sub-stroke starts, scanned
//   k_gs_write  a kept point's position is the kept points before it and its sub-stroke
//               the starts before it; points from 65,535 on are dropped and start
//               nothing; a start sets its sub-stroke's first point and the joined flag the
//               close events before it leave on the sub-stroke before
//   k_gs_subs   per sub-stroke: its points, the last one's joined flag (the last Close or
//               Move op after its last point when the cap stopped the points, else the
//               path's last Move/Line/Quad/Cubic/Close op), SubStroke::len in u16
//               arithmetic and 2 len + 2 outline items, scanned
//   k_go_count  every outline item's points (outline_item), their number scanned, the first
//               two kept (all there are but for arcs; computed again for the emit: 23 / 26 us
//               on the 65,535 points of a capped stroke from a cold cache, kept 21 / 17 us)
//   k_go_emit   the outline's raw vertices through the second transform (plotter.rs:
//               219-224), the figure runs' starts per tile, scanned
// then k_gb_keep, k_gb_write and k_gb_top build the outline's figure as they do a fill's.

// width in effect at op j: its path's last PenWidth op at or before it, else the width
// the path starts with
__device__ __forceinline__ float gs_width(const GridBuildBufs& G, int j) {
    if (j < 0) return *G.s_width;
    const int lpw = max(G.opw[j], G.opa[j / BLOCK].y);
    return lpw >= 0 ? __ldg(&G.ops[lpw].v[0]) : *G.s_width;
}

// Raw stroke points of a Move/Line/Quad/Cubic op with the pen at (px, py) and widths
// pen_w (at the pen) and sw (at the op), as build_fill's STROKE walk makes them
// (plotter.rs:233-236, 294-298), split over 2^d0 lanes as gb_walk splits a fill's:
// emit(k, point, width) for the lane's k-th leaf; returns the lane's leaf count.
template <class Emit>
__device__ int gs_walk(const KParams& P, const ft_op& op, int kind, float px, float py, float pen_w, float sw,
                       int lane, int d0, int& flags, Emit emit) {
    if (kind == FT_OP_MOVE || kind == FT_OP_LINE) {
        if (lane) return 0;
        emit(0, xform(P.xf, p2(op.v[0], op.v[1])), sw);
        return 1;
    }
    P2 a = xform(P.xf, p2(px, py)), b = xform(P.xf, p2(op.v[0], op.v[1])), c = xform(P.xf, p2(op.v[2], op.v[3]));
    const float tol_sq = P.tol_sq;
    int dh = 0, n;
    if (kind == FT_OP_QUAD) {
        float wa = pen_w, wb = __fmul_rn(__fadd_rn(pen_w, sw), 0.5f), wc = sw;
        if (!pfinite(a) || !pfinite(b) || !pfinite(c)) {
            if (lane) return 0;
            flags |= 2;
            emit(0, c, wc);
            return 1;
        }
        for (int d = 0; d < d0; d++) {
            const P2 ab = pmid(a, b), bc = pmid(b, c), abbc = pmid(ab, bc), ac = pmid(a, c);
            const bool within = pdist_sq(abbc, ac) <= tol_sq;
            if (within || d >= FT_MAX_DEPTH) {
                if (lane & ((1 << (d0 - d)) - 1)) return 0;
                if (!within) flags |= 1;
                emit(0, c, wc);
                return 1;
            }
            const float wab = fmid(wa, wb), wbc = fmid(wb, wc), wabbc = fmid(wab, wbc);
            if ((lane >> (d0 - 1 - d)) & 1) {
                a = abbc;
                b = bc;
                wa = wabbc;
                wb = wbc;
            } else {
                b = ab;
                c = abbc;
                wb = wab;
                wc = wabbc;
            }
        }
        n = quad_walk<true>(a, b, c, wa, wb, wc, tol_sq, 0, INT_MAX, &dh, emit, d0);
    } else {
        P2 e = xform(P.xf, p2(op.v[4], op.v[5]));
        float wa = pen_w, wb = __fadd_rn(sw, __fmul_rn(__fsub_rn(pen_w, sw), 1.0f / 3.0f)),
              wc = __fadd_rn(sw, __fmul_rn(__fsub_rn(pen_w, sw), 2.0f / 3.0f)), we = sw;
        if (!pfinite(a) || !pfinite(b) || !pfinite(c) || !pfinite(e)) {
            if (lane) return 0;
            flags |= 2;
            emit(0, e, we);
            return 1;
        }
        for (int d = 0; d < d0; d++) {
            const P2 ab = pmid(a, b), bc = pmid(b, c), cd = pmid(c, e);
            const P2 abbc = pmid(ab, bc), bccd = pmid(bc, cd);
            const P2 pe = pmid(abbc, bccd), ad = pmid(a, e);
            const bool within = pdist_sq(pe, ad) <= tol_sq;
            if (within || d >= FT_MAX_DEPTH) {
                if (lane & ((1 << (d0 - d)) - 1)) return 0;
                if (!within) flags |= 1;
                emit(0, e, we);
                return 1;
            }
            const float wab = fmid(wa, wb), wbc = fmid(wb, wc), wcd = fmid(wc, we);
            const float wabbc = fmid(wab, wbc), wbccd = fmid(wbc, wcd), wpe = fmid(wabbc, wbccd);
            if ((lane >> (d0 - 1 - d)) & 1) {
                a = pe;
                b = bccd;
                c = cd;
                wa = wpe;
                wb = wbccd;
                wc = wcd;
            } else {
                b = ab;
                c = abbc;
                e = pe;
                wb = wab;
                wc = wabbc;
                we = wpe;
            }
        }
        n = cubic_walk<true>(a, b, c, e, wa, wb, wc, we, tol_sq, 0, INT_MAX, &dh, emit, d0);
    }
    if (dh) flags |= 1;
    return n;
}

__device__ __forceinline__ bool gs_over(const GridStrokeBufs& S) { return *S.n_sraw > S.sraw_cap; }

__global__ void __launch_bounds__(BLOCK) k_gs_count(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ long long ltmp[NWARP];
    const GridBuildBufs& G = P.gb;
    const GridStrokeBufs& S = P.gs;
    if (S.skip && *S.skip) return;  // a probe over a prefix of the ops completed the points
    const int tid = threadIdx.x;
    int flags = 0;
    for (int blk = blockIdx.x; blk < gb_ctas(G.n_ops); blk += gridDim.x) {
        const GbOp o = gb_op_of(G, blk, flags);
        int n = 0;
        if (o.kind >= FT_OP_MOVE && o.kind <= FT_OP_CUBIC)
            n = gs_walk(P, o.op, o.kind, o.px, o.py, gs_width(G, o.lpc), gs_width(G, o.i), o.lane, G.d0, flags,
                        [](int, P2, float) {});
        int inc = n;
        const int lanes = 1 << G.d0;
        for (int d = 1; d < lanes; d <<= 1) {
            const int t = __shfl_up_sync(FULL, inc, d, lanes);
            if (o.lane >= d) inc += t;
        }
        const int n_op = __shfl_sync(FULL, inc, lanes - 1, lanes);
        int tot;
        const int ex = block_excl_sum(o.lane == 0 ? n_op : 0, tmp, tot);
        if (o.i < G.n_ops) {
            G.opl[(o.i << G.d0) + o.lane] = inc - n;
            if (o.lane == 0) G.opi[o.i].y = ex;
        }
        if (tid == 0) G.opn[blk] = tot;
    }
    if (flags) atomicMax(&P.status[0], (flags & 1) ? FT_ERR_DEPTH : FT_ERR_ARG);
    if (!gb_last_block(&S.done[0])) return;
    const int nb = gb_ctas(G.n_ops);
    long long carry = 0;
    for (int b0 = 0; b0 < nb; b0 += BLOCK) {
        const int b = b0 + tid;
        long long t;
        const long long e = block_excl_sum_ll(b < nb ? __ldcg(&G.opn[b]) : 0ll, ltmp, t);
        if (b < nb) G.opn[b] = carry + e;
        carry += t;
    }
    if (tid == 0) *S.n_sraw = carry;
}

__global__ void __launch_bounds__(BLOCK) k_gs_emit(KParams P) {
    chain_link();
    const GridBuildBufs& G = P.gb;
    const GridStrokeBufs& S = P.gs;
    if (S.skip && *S.skip) return;  // a probe over a prefix of the ops completed the points
    if (gs_over(S)) return;  // every CTA: the caller grows the arrays
    int flags = 0;
    for (int blk = blockIdx.x; blk < gb_ctas(G.n_ops); blk += gridDim.x) {
        const GbOp o = gb_op_of(G, blk, flags);
        if (o.kind < FT_OP_MOVE || o.kind > FT_OP_CUBIC) continue;
        const long long off0 = G.opn[blk] + G.opi[o.i].y;
        const int off = (int)(off0 + G.opl[(o.i << G.d0) + o.lane]);
        const int cap = S.sraw_cap;
        // a Move ends the sub-stroke before it open, a Close joined (stroker.rs:87-96)
        const unsigned char f0 = (unsigned char)(((o.lane == 0 && o.rs) ? 1 : 0) | (o.kind != FT_OP_MOVE ? 2 : 0));
        const unsigned char f1 = (unsigned char)(o.kind != FT_OP_MOVE ? 2 : 0);
        float4* raw4 = S.raw4;
        unsigned char* sfl = S.sfl;
        int* sopi = S.sopi;
        const int i = o.i;
        gs_walk(P, o.op, o.kind, o.px, o.py, gs_width(G, o.lpc), gs_width(G, o.i), o.lane, G.d0, flags,
                [&](int k, P2 q, float w) {
                    if (ck(off + k < cap, 13) && off + k < cap) {
                        raw4[off + k] = make_float4(q.x, q.y, w, 0.f);
                        sfl[off + k] = k == 0 ? f0 : f1;
                        sopi[off + k] = i;
                    }
                });
    }
}

// Kept raw stroke points and sub-stroke starts per tile, packed (kept << 32 | starts).
__global__ void __launch_bounds__(BLOCK) k_gs_keep(KParams P) {
    chain_link();
    __shared__ long long ltmp[NWARP];
    const GridStrokeBufs& S = P.gs;
    if (S.skip && *S.skip) return;  // a probe over a prefix of the ops completed the points
    if (gs_over(S)) return;
    const int M = (int)*S.n_sraw, nt = (M + GB_TILE - 1) / GB_TILE, tid = threadIdx.x;
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const int k0 = t * GB_TILE + GB_PER * tid;
        long long v = 0;
        float2 q = make_float2(0.f, 0.f);
        if (k0 > 0 && k0 <= M) {
            const float4 p = S.raw4[k0 - 1];
            q = make_float2(p.x, p.y);
        }
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            if (k >= M) break;
            const float4 p = S.raw4[k];
            const int rs = S.sfl[k] & 1;
            const bool keep = rs || !(p.x == q.x && p.y == q.y);
            v += ((long long)(keep ? 1 : 0) << 32) | rs;
            q = make_float2(p.x, p.y);
        }
        long long tot;
        block_excl_sum_ll(v, ltmp, tot);
        if (tid == 0) S.stile[t] = make_int2((int)(tot >> 32), (int)(tot & 0xFFFFFFFFll));
    }
    if (!gb_last_block(&S.done[1])) return;
    long long carry = 0;
    for (int b0 = 0; b0 < nt; b0 += BLOCK) {
        const int b = b0 + tid;
        long long x = 0;
        if (b < nt) {
            const int2 a = __ldcg(&S.stile[b]);
            x = ((long long)a.x << 32) | (unsigned)a.y;
        }
        long long t;
        const long long e = carry + block_excl_sum_ll(x, ltmp, t);
        if (b < nt) S.stile[b] = make_int2((int)(e >> 32), (int)(e & 0xFFFFFFFFll));
        carry += t;
    }
    if (tid == 0) {
        const int kept = (int)(carry >> 32);
        S.st[0] = min(kept, PT_CAP);
        S.st[6] = kept > PT_CAP ? 1 : 0;
        if (S.final_flag && kept > PT_CAP) *S.final_flag = 1;
    }
}

__global__ void __launch_bounds__(BLOCK) k_gs_write(KParams P) {
    chain_link();
    __shared__ long long ltmp[NWARP];
    const GridStrokeBufs& S = P.gs;
    if (S.skip && *S.skip) return;  // a probe over a prefix of the ops completed the points
    if (gs_over(S)) return;
    const int M = (int)*S.n_sraw, nt = (M + GB_TILE - 1) / GB_TILE, tid = threadIdx.x;
    const int count = S.st[0];
    float4* spts = reinterpret_cast<float4*>(P.scratch + P.L.spts);
    SubRec* subs = reinterpret_cast<SubRec*>(P.scratch + P.L.subs);
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const int2 c = S.stile[t];
        const int k0 = t * GB_TILE + GB_PER * tid;
        float4 p[GB_PER];
        int f[GB_PER], keep = 0;
        long long v = 0;
        float2 q = make_float2(0.f, 0.f);
        if (k0 > 0 && k0 <= M) {
            const float4 pp = S.raw4[k0 - 1];
            q = make_float2(pp.x, pp.y);
        }
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            const int k = k0 + j;
            p[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            f[j] = 0;
            if (k < M) {
                p[j] = S.raw4[k];
                f[j] = S.sfl[k];
                const int rs = f[j] & 1;
                if (rs || !(p[j].x == q.x && p[j].y == q.y)) keep |= 1 << j;
                v += ((long long)((keep >> j) & 1) << 32) | rs;
                q = make_float2(p[j].x, p[j].y);
            }
        }
        long long tot;
        const long long e = block_excl_sum_ll(v, ltmp, tot);
        int pos = c.x + (int)(e >> 32), sid = c.y + (int)(e & 0xFFFFFFFFll);
#pragma unroll
        for (int j = 0; j < GB_PER; j++) {
            if (!((keep >> j) & 1)) continue;
            const int rs = f[j] & 1;
            if (pos < PT_CAP) {
                spts[pos] = p[j];
                if (rs) {
                    subs[sid].start = pos;
                    if (sid > 0) subs[sid - 1].joined = (f[j] >> 1) & 1;
                    atomicMax(&S.st[1], sid + 1);
                }
                if (pos == count - 1) S.st[2] = S.sopi[k0 + j];  // the op of the last kept point
            }
            pos++;
            sid += rs;
        }
    }
}

// Sub-strokes (stroker.rs:87-96, 239-262), 256 a CTA step.
__global__ void __launch_bounds__(BLOCK) k_gs_subs(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    const GridBuildBufs& G = P.gb;
    const GridStrokeBufs& S = P.gs;
    if (gs_over(S)) return;
    const int tid = threadIdx.x, nsub = S.st[1], count = S.st[0];
    SubRec* subs = reinterpret_cast<SubRec*>(P.scratch + P.L.subs);
    const int nc = (nsub + BLOCK - 1) / BLOCK;
    for (int c = blockIdx.x; c < nc; c += gridDim.x) {
        const int si = c * BLOCK + tid;
        int items = 0;
        if (si < nsub) {
            const SubRec r = subs[si];
            const int n = (si + 1 < nsub ? subs[si + 1].start : count) - r.start;
            int joined = r.joined;
            if (si == nsub - 1) {
                // the last sub-stroke: the close events after its last point
                const int cm = S.st[4], pc = S.st[3];
                if (S.st[6])
                    joined = cm > S.st[2] ? (__ldg(&G.ops[cm].kind) == FT_OP_CLOSE) : 0;
                else
                    joined = pc >= 0 ? (__ldg(&G.ops[pc].kind) == FT_OP_CLOSE) : 0;
                subs[si].joined = joined;
            }
            // SubStroke::len with u16 arithmetic: n + 1 wraps at 65,536
            const int len = joined ? ((n + 1) & 0xFFFF) : (n > 0 ? n - 1 : 0);
            items = len > 0 ? 2 * len + 2 : 0;
            subs[si].n = n;
            subs[si].len = len;
        }
        int tot;
        const int off = block_excl_sum(items, tmp, tot);
        if (si < nsub) subs[si].item_off = off;
        if (tid == 0) S.subt[c] = tot;
    }
    if (!gb_last_block(&S.done[2])) return;
    int carry = 0;
    for (int b0 = 0; b0 < nc; b0 += BLOCK) {
        const int b = b0 + tid;
        int tot;
        const int e = block_excl_sum(b < nc ? __ldcg(&S.subt[b]) : 0, tmp, tot);
        if (b < nc) S.subt[b] = carry + e;
        carry += tot;
    }
    if (tid == 0) S.st[5] = carry;
}

// Outline item t: its sub-stroke (the last with item offset <= t: empty sub-strokes share
// the next one's offset and come before it) and its index u in it.
__device__ __forceinline__ SubRec go_item(const GridStrokeBufs& S, const SubRec* subs, int nsub, int t, int& u) {
    int lo = 0, hi = nsub - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (subs[mid].item_off + S.subt[mid / BLOCK] <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    SubRec sr = subs[lo];
    sr.item_off += S.subt[lo / BLOCK];
    u = t - sr.item_off;
    return sr;
}

__global__ void __launch_bounds__(BLOCK) k_go_count(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ long long ltmp[NWARP];
    const GridBuildBufs& G = P.gb;
    const GridStrokeBufs& S = P.gs;
    if (gs_over(S)) return;
    const int tid = threadIdx.x, nsub = S.st[1], n_items = min(S.st[5], GS_ITEMS_CAP);
    const float4* spts = reinterpret_cast<const float4*>(P.scratch + P.L.spts);
    const SubRec* subs = reinterpret_cast<const SubRec*>(P.scratch + P.L.subs);
    const int nc = (n_items + BLOCK - 1) / BLOCK;
    int depth_hit = 0;
    for (int c = blockIdx.x; c < nc; c += gridDim.x) {
        const int t = c * BLOCK + tid;
        int n = 0;
        bool starts = false;
        if (t < n_items) {
            int u;
            const SubRec sr = go_item(S, subs, nsub, t, u);
            float4 two = make_float4(0.f, 0.f, 0.f, 0.f);
            n = outline_item(P, spts, sr, u, 0, INT_MAX, &depth_hit, [&](int k, P2 q) {
                if (k == 0) two.x = q.x, two.y = q.y;
                if (k == 1) two.z = q.x, two.w = q.y;
            });
            S.itp[t] = two;
            // a figure run starts at each side's first point after a Close: the forward side
            // always (after the previous sub-stroke's Close, or first), the reverse side when
            // the sub-stroke is joined (stroker.rs:255-260)
            const bool rev = u > sr.len, joined = sr.joined != 0;
            const int j = rev ? u - sr.len - 1 : u;
            starts = (!rev && ((!joined && j == 0) || (joined && j == 1))) || (rev && joined && j == 1);
        }
        int tot;
        const int off = block_excl_sum(n, tmp, tot);
        if (t < n_items) S.itoff[t] = make_int2(off, n | (starts ? INT_MIN : 0));
        if (tid == 0) S.itc[c] = tot;
    }
    if (depth_hit) atomicMax(&P.status[0], FT_ERR_DEPTH);
    if (!gb_last_block(&S.done[3])) return;
    long long carry = 0;
    for (int b0 = 0; b0 < nc; b0 += BLOCK) {
        const int b = b0 + tid;
        long long t;
        const long long e = block_excl_sum_ll(b < nc ? (long long)__ldcg(&S.itc[b]) : 0ll, ltmp, t);
        if (b < nc) S.itc[b] = (int)min(carry + e, (long long)INT_MAX);
        carry += t;
    }
    if (tid == 0) *G.n_raw = carry;
}

__global__ void __launch_bounds__(BLOCK) k_go_emit(KParams P) {
    chain_link();
    __shared__ int tmp[2 * NWARP + 2];
    __shared__ int s_c;
    const GridBuildBufs& G = P.gb;
    const GridStrokeBufs& S = P.gs;
    if (gs_over(S)) return;
    const long long n_raw = *G.n_raw;
    if (n_raw > G.raw_cap) return;
    const int tid = threadIdx.x, nsub = S.st[1], n_items = min(S.st[5], GS_ITEMS_CAP), cap = G.raw_cap;
    const float4* spts = reinterpret_cast<const float4*>(P.scratch + P.L.spts);
    const SubRec* subs = reinterpret_cast<const SubRec*>(P.scratch + P.L.subs);
    for (int t = blockIdx.x * BLOCK + tid; t < n_items; t += gridDim.x * BLOCK) {
        const int2 it = S.itoff[t];
        const int off = S.itc[t / BLOCK] + it.x, n = it.y & INT_MAX;
        const bool starts = it.y < 0;
        auto put = [&](int k, P2 q) {
            const P2 tq = xform(P.xf, q);  // the outline is transformed again (F9)
            if (ck(off + k < cap, 16) && off + k < cap) {
                G.raw[off + k] = make_int2(f2fx(tq.x), f2fx(tq.y));
                G.fl[off + k] = k == 0 && starts ? (unsigned char)1 : (unsigned char)0;
            }
        };
        if (n <= 2) {  // kept by k_go_count
            const float4 two = S.itp[t];
            if (n > 0) put(0, p2(two.x, two.y));
            if (n > 1) put(1, p2(two.z, two.w));
        } else {  // an arc: again
            int u, dh = 0;
            const SubRec sr = go_item(S, subs, nsub, t, u);
            outline_item(P, spts, sr, u, 0, INT_MAX, &dh, put);
        }
        if (starts && n > 0 && off < cap) atomicMax(&G.tr[off / GB_TILE], off);
    }
    if (!gb_last_block(&G.done[2])) return;
    gb_scan_tr(G, n_raw, tmp, s_c);
}

cudaError_t launch_grid_stroke(const KParams& p, int sm_count, cudaStream_t s, const KParams* probe) {
    const int nbo = (p.gb.n_ops + BLOCK - 1) / BLOCK;
    if (nbo <= 0 || p.gb.raw_cap % GB_TILE || p.gb.raw_cap > GB_RAW_MAX || p.gs.sraw_cap % GB_TILE ||
        p.gs.sraw_cap > GB_RAW_MAX || !p.gs.st || p.pt_cap != PT_CAP)
        return cudaErrorInvalidValue;
    if (probe && (probe->gb.n_ops <= 0 || probe->gb.n_ops > p.gb.n_ops)) return cudaErrorInvalidValue;
    const int gt = std::max(1, 4 * sm_count);
    cudaError_t e;
    if ((e = launch_chain(k_gb_ops, nbo, BLOCK, 0, s, p)) != cudaSuccess) return e;  // pens and widths of every op (the probe's too)
    for (const KParams* q : {probe, &p}) {
        if (!q) continue;
        const int nbw = std::min(gb_ctas(q->gb.n_ops), 8 * sm_count);  // all resident: a skipped build only launches these
        if ((e = launch_chain(k_gs_count, nbw, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gs_emit, nbw, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gs_keep, gt, BLOCK, 0, s, *q)) != cudaSuccess) return e;
        if ((e = launch_chain(k_gs_write, gt, BLOCK, 0, s, *q)) != cudaSuccess) return e;
    }
    if ((e = launch_chain(k_gs_subs, std::max(1, std::min(gt, PT_CAP / BLOCK + 1)), BLOCK, 0, s, p)) != cudaSuccess) return e;
    if ((e = launch_chain(k_go_count, gt, BLOCK, 0, s, p)) != cudaSuccess) return e;
    if ((e = launch_chain(k_go_emit, gt, BLOCK, 0, s, p)) != cudaSuccess) return e;
    if ((e = launch_chain(k_gb_keep, gt, BLOCK, 0, s, p)) != cudaSuccess) return e;
    if ((e = launch_chain(k_gb_write, gt, BLOCK, 0, s, p)) != cudaSuccess) return e;
    if ((e = launch_chain(k_gb_top, GB_TOP_BLOCKS, BLOCK, 0, s, p)) != cudaSuccess) return e;
    return cudaSuccess;
}

cudaError_t launch_composite_build(const KParams& p, int grid, int smem_bytes, cudaStream_t s, bool few_ctas) {
    auto kern = p.stroke ? k_cbuild<true> : k_cbuild<false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                         few_ctas ? FEW_CTAS_CARVEOUT : (int)cudaSharedmemCarveoutDefault);
    kern<<<grid, BLOCK, smem_bytes, s>>>(p);
    return cudaGetLastError();
}

// As raster_blocks_per_sm: the query is made with no carve-out preference.
int composite_build_blocks_per_sm(int smem_bytes, bool stroke) {
    auto kern = stroke ? k_cbuild<true> : k_cbuild<false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutDefault);
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, BLOCK, smem_bytes) != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

cudaError_t launch_composite_bands(const KParams& p, int smem_bytes, cudaStream_t s) {
    k_cbands<<<p.n_bands, 32 * p.band_rows, smem_bytes, s>>>(p);
    return cudaGetLastError();
}

cudaError_t allow_smem(const void* kern) {
    int dev = 0, most = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kern);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes);
    return e;
}
cudaError_t setup_kernels() {
    const void* kernels[] = {(const void*)k_raster<false>,  (const void*)k_raster<true>,
                             (const void*)k_cbuild<false>,  (const void*)k_cbuild<true>,
                             (const void*)k_cbands,         (const void*)k_srcover_mask,
                             (const void*)k_fig_edges,      (const void*)k_fig_bin_fill,
                             (const void*)k_ctile<true, FT_NONZERO>,  (const void*)k_ctile<true, FT_EVENODD>,
                             (const void*)k_ctile<false, FT_NONZERO>, (const void*)k_ctile<false, FT_EVENODD>};
    for (const void* k : kernels) {
        const cudaError_t e = allow_smem(k);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ftk

// ===========================================================================
// Allocation-free single-path fill (ft_fill_noalloc).
//
// For callers that may not allocate device memory themselves or through this
// library: a host whose device memory belongs to another runtime's allocator (a game
// engine's or a language runtime's pool that must see every allocation), or a
// process held to a fixed device-memory budget.  The figure scratch of one CTA lives
// in a file-scope device array that every GPU loading this library holds until the
// process exits; the caller passes only inputs and outputs.  One CTA rasterises the
// whole path.
namespace ftk {

// vertices, sub-figure starts and edges of one figure of up to FT_MAX_POINTS vertices
constexpr size_t NOALLOC_SCRATCH_BYTES = align256(SCR_EDGES + (size_t)PT_CAP * sizeof(EdgeRec));
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

__global__ void __launch_bounds__(BLOCK) k_fill_noalloc(KParams P, ft_path_desc d, unsigned char* scratch,
                                                        int32_t* status_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CState S;
    __shared__ int s_tmp3[3 * NWARP];
    int2* pts = reinterpret_cast<int2*>(scratch + SCR_PTS);
    int* ss = reinterpret_cast<int*>(scratch + SCR_SS);
    EdgeRec* edges = reinterpret_cast<EdgeRec*>(scratch + SCR_EDGES);
    BuildSmem& B = *reinterpret_cast<BuildSmem*>(smem);
    CompactSmem* Cs = reinterpret_cast<CompactSmem*>(smem + ((sizeof(BuildSmem) + 15) & ~(size_t)15));
    build_fill<BlockG>(P, d, d.s_width, B, Cs, S, pts, ss, PT_CAP);
    if (S.count > 0) {
        top_and_dir<BlockG>(S, pts, ss, s_tmp3);
        build_edges<BlockG>(S, pts, ss, edges);
        __syncthreads();
        const int lo = max(S.top_row, 0), hi = (int)d.height;
        const int wp4 = (int)(((d.width + 3) & ~3u) * 4);
        const int R = max(1, min((P.smem_bytes - RASTER_FIXED_SMEM) / max(wp4, 4), max(hi, 1)));
        if (lo < hi && d.width > 0) raster_rows(P, d, S, edges, lo, hi, R, smem);
    }
    if (threadIdx.x == 0 && status_out)
        *status_out = S.flags ? ((S.flags & 1) ? FT_ERR_DEPTH : FT_ERR_ARG) : FT_OK;
}

}  // namespace ftk

#include <cuda.h>
#include <mutex>

namespace {
// Set-up of ft_fill_noalloc per device: the device address of g_noalloc_scratch and the
// kernel's dynamic shared-memory limit, both belonging to the device's current context.
// A device reset (cudaDeviceReset) destroys that context and unloads the module, so the
// set-up is keyed by the context's unique id and done again in a new context.
constexpr int NOALLOC_MAX_DEVICES = 64;
struct NoallocDev {
    unsigned long long ctx_id = 0;  // 0: not set up
    void* scratch = nullptr;
    int smem_max = 0;
};
NoallocDev g_noalloc[NOALLOC_MAX_DEVICES];
std::mutex g_noalloc_mu;

typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long*);

// Unique id of the calling thread's current context (0 when none is current yet),
// through the runtime's driver entry points (no link against the driver library).
unsigned long long current_ctx_id() {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<CtxGetIdFn>(f);
    });
    CUcontext cu = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&cu) != CUDA_SUCCESS || !cu || get_id(cu, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

// The set-up of `dev` (current) for its current context; false when a CUDA call fails.
bool noalloc_setup(int dev, NoallocDev& out) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoallocDev& D = g_noalloc[dev];
    unsigned long long id = current_ctx_id();
    if (id == 0 || id != D.ctx_id) {
        void* p = nullptr;
        // also makes the device's primary context current when none was
        if (cudaGetSymbolAddress(&p, ftk::g_noalloc_scratch) != cudaSuccess || !p) return false;
        int optin = 0;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return false;
        const int smem_max = optin - 1024;
        if (cudaFuncSetAttribute(ftk::k_fill_noalloc, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max) !=
            cudaSuccess)
            return false;
        id = current_ctx_id();
        if (id == 0) return false;
        D.ctx_id = id;
        D.scratch = p;
        D.smem_max = smem_max;
    }
    out = D;
    return true;
}
}  // namespace

extern "C" FT_API int ft_fill_noalloc(int32_t rule, const ft_op* ops, uint32_t n_ops, int32_t fmt,
                                      const uint8_t clr[4], uint8_t* raster, uint32_t w, uint32_t h,
                                      uint32_t stride, const float transform[6], float tolerance, float pen_width,
                                      int32_t* status, void* stream) {
    if ((rule != FT_NONZERO && rule != FT_EVENODD) || (fmt != FT_MATTE8 && fmt != FT_RGBA8P)) return FT_ERR_ARG;
    if ((n_ops && !ops) || (w && h && !raster)) return FT_ERR_ARG;
    if (w > FT_MAX_WIDTH) return FT_ERR_CAP;  // one band row of cell areas must fit in shared memory
    const uint32_t bpp = fmt == FT_RGBA8P ? 4 : 1;
    if (h && stride < (uint64_t)w * bpp) return FT_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(ops) & 15) ||
        (fmt == FT_RGBA8P && ((reinterpret_cast<uintptr_t>(raster) | stride) & 3)))
        return FT_ERR_ARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return FT_ERR_CUDA;
    NoallocDev D;
    if (!noalloc_setup(dev, D)) return FT_ERR_CUDA;
    ft_path_desc d;
    memset(&d, 0, sizeof(d));
    d.n_ops = n_ops;
    d.width = w;
    d.height = h;
    d.stride = stride;
    d.s_width = pen_width;
    if (clr) memcpy(d.clr, clr, 4);
    ftk::KParams p;
    memset(&p, 0, sizeof(p));
    p.ops = ops;
    p.rasters = raster;
    p.rule = rule;
    p.fmt = fmt;
    static const float ident[6] = {1, 0, 0, 0, 1, 0};
    for (int i = 0; i < 6; i++) p.xf[i] = transform ? transform[i] : ident[i];
    const float t = tolerance > 0.01f ? tolerance : 0.01f;
    p.tol = t;
    p.tol_sq = t * t;
    const int wp = (int)((w + 3) & ~3u);
    int smem = std::max(ftk::RASTER_FIXED_SMEM + 16 * wp * 4, 40 * 1024);
    smem = std::min(smem, D.smem_max);
    p.smem_bytes = smem;
    unsigned char* scratch = static_cast<unsigned char*>(D.scratch);
    // the launch's own status: an error some earlier, unrelated call left in the runtime
    // is neither consumed nor reported here
    void* args[] = {&p, &d, &scratch, &status};
    const cudaError_t e = cudaLaunchKernel(reinterpret_cast<const void*>(ftk::k_fill_noalloc), dim3(1),
                                           dim3(ftk::BLOCK), args, (size_t)smem, static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? FT_OK : FT_ERR_CUDA;
}

// Check build: the first failing bounds check's site since the last call (0: none), and
// whether the checks are compiled in.  No counterpart in footile.
extern "C" FT_API int ft_check_failures(int32_t* site, int32_t* compiled_in) {
    if (compiled_in) *compiled_in = FT_CHECK;
    if (!site) return FT_OK;
    ftk::CheckState s;
    for (auto take : {ftk::take_check, ftk::take_check_tile, ftk::take_check_bands, fta::take_check_adjoint}) {
        ftk::CheckState t;
        if (take(&t, false) != cudaSuccess) return FT_ERR_CUDA;
        if (!s.failed) s.failed = t.failed;
    }
    *site = s.failed;
    return FT_OK;
}

#if FT_CHECK
// The check build alone: the sites whose checks ran since the last call, a bit each.
extern "C" FT_API int ft_check_reached(unsigned long long* sites) {
    *sites = 0;
    for (auto take : {ftk::take_check, ftk::take_check_tile, ftk::take_check_bands, fta::take_check_adjoint}) {
        ftk::CheckState t;
        if (take(&t, true) != cudaSuccess) return FT_ERR_CUDA;
        *sites |= t.reached;
    }
    return FT_OK;
}
#endif
