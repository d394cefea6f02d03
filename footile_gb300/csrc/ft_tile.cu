// ft_tile.cu — the tile rasteriser: fills of small canvases, one CTA per path (or per row
// range of a path), the figure never sorted or compacted.
//
// footile builds a figure vertex by vertex (fig.rs:373-461): coincident vertices are
// dropped, a closing vertex equal to the sub-figure's first is popped, the vertices are
// sorted and an active-edge list is swept (fig.rs:493-617).  None of that order reaches the
// mask: the cell areas are wrapping sums, a zero-length segment gives no edge whether its
// vertex was kept or not, and only two things depend on the vertex list, both functions of
// the non-zero segments alone:
//   - the top row, the least y of a vertex that starts a non-zero segment (a sub-figure
//     whose points all coincide is popped whole, and has no such segment);
//   - the direction of the figure (fig.rs:402-411): the top vertex is the start of the
//     first non-zero segment with the least (y, x); the vertex after it is that segment's
//     end, the vertex before it is the start of the non-zero segment before it in its
//     sub-figure, cyclically.
// The direction only flips the sign of every cell sum, so it is applied at the resolve.
//
// So every leaf of a curve's subdivision is an edge by itself: the subdivision node's start
// and end points (the start is the end of the leaf before, bit for bit).  Leaves are taken by
// address (ft_slots.cuh): 2^D slots per curve, one thread each; slots that own no leaf stay
// empty (zero-length segments).
//
// The segments (16 bytes: both end points in 16.16) go to the CTA's scratch in order.  Bands
// of raster rows are then accumulated in shared memory: each warp takes 32 segments at a time
// that reach the band, works out slope and step once per segment, and spreads the (edge, row)
// items over its lanes.  The rows are resolved 8 pixels per lane, as many rows per warp as
// fit, and written once.
//
// A path whose slots exceed the scratch, or with a curve not known to be flat at SLOT_DEPTH, is
// handed to k_raster through the overflow list.
#include <climits>
#include <cstddef>

#include "ft_items.cuh"
#include "ft_slots.cuh"

namespace ftk {
namespace {


static_assert(TILE_THREADS_FEW * ((1 << SLOT_DEPTH) + 1) < (1 << 22) && TILE_THREADS_FEW <= 512,
              "slots and listed ops of a chunk fit one word");

// ------------------------------------------------------------------- state
template <int NT>
struct TileBuild {  // one chunk of NT ops; g0, g1, off and info of the ops that have slots
    float4 g0[NT], g1[NT];  // transformed control points (a, b), (c, end)
    float2 endp[NT];        // the pen after the op
    int off[NT + 33];       // first slot; past the last op: INT_MAX
    int info[NT];           // depth | safe << 4 | type << 8 | closing slot << 10 | starts a sub-figure << 11
    int kind[NT];
};
enum { TY_POINT = 0, TY_QUAD = 1, TY_CUBIC = 2 };
constexpr int TILE_END = 16;  // kind of the virtual op after the last one

struct TileWarp {  // one warp's segments while a band is accumulated
    int4 q[64];    // segments that reach the band
    int4 rec[64];  // two records per segment in work
};

template <int NT>
struct TileState {
    static constexpr int NW = NT / 32;
    unsigned pcm[NW], vom[NW], rsm[NW];
    unsigned wsum[NW];
    // the walk, carried from chunk to chunk
    int c_kind, c_vo, c_rs;  // kind of the last Move/Line/Quad/Cubic/Close op; last vertex op; last sub-figure start
    float c_px, c_py;        // pen after the last Move/Line/Quad/Cubic/Close op
    int flags, item, last_pw;
    unsigned long long top;  // least (y, x) a non-zero segment starts from
    int top_slot;            // the first slot of such a segment
};

template <int NW>
__device__ __forceinline__ int prev_bit(const unsigned* m, int i) {  // last set bit at or below i, or -1
    if (i < 0) return -1;
    int w = i >> 5;
    unsigned v = m[w] & (ALL >> (31 - (i & 31)));
    while (!v) {
        if (--w < 0) return -1;
        v = m[w];
    }
    return (w << 5) + 31 - __clz(v);
}

__device__ __forceinline__ ft_op tile_op(const ft_op* ops, int i) {
    const int4* src = reinterpret_cast<const int4*>(ops + i);
    const int4 q0 = __ldg(src), q1 = __ldg(src + 1);
    ft_op o;
    o.kind = q0.x;
    o.v[0] = __int_as_float(q0.y);
    o.v[1] = __int_as_float(q0.z);
    o.v[2] = __int_as_float(q0.w);
    o.v[3] = __int_as_float(q1.x);
    o.v[4] = __int_as_float(q1.y);
    o.v[5] = __int_as_float(q1.z);
    o.reserved = 0;
    return o;
}
__device__ __forceinline__ P2 op_end(const ft_op& o) {
    if (o.kind == FT_OP_QUAD) return p2(o.v[2], o.v[3]);
    if (o.kind == FT_OP_CUBIC) return p2(o.v[4], o.v[5]);
    return p2(o.v[0], o.v[1]);
}
// The first vertex of the sub-figure that op j starts: its point, or for a curve right
// after a Close (or at the path's start), whose pen is the origin, its first leaf.
__device__ P2 first_vertex(const TileParams& P, const ft_op* ops, int j) {
    const ft_op o = tile_op(ops, j);
    const P2 end = xform(P.xf, op_end(o));
    if (o.kind != FT_OP_QUAD && o.kind != FT_OP_CUBIC) return end;
    P2 a = xform(P.xf, p2(0.f, 0.f)), b = xform(P.xf, p2(o.v[0], o.v[1])), c = xform(P.xf, p2(o.v[2], o.v[3]));
    if (!pfinite(a) || !pfinite(b) || !pfinite(c) || !pfinite(end)) return end;
    float w = 0.f;
    if (o.kind == FT_OP_QUAD) {
        quad_slot(a, b, c, w, w, w, 0, SLOT_DEPTH, 0, P.tol_sq);
        return c;
    }
    P2 e = end;
    cubic_slot(a, b, c, e, w, w, w, w, 0, SLOT_DEPTH, 0, P.tol_sq);
    return e;
}
__device__ __forceinline__ unsigned long long top_key(int x, int y) {
    return ((unsigned long long)((unsigned)y ^ 0x80000000u) << 32) | ((unsigned)x ^ 0x80000000u);
}

// -------------------------------------------------------------------- build
// Segments of the path into E (slots in order, 32-slot groups; empty slots are zero-length)
// and `ends` (per group the slots that close a sub-figure).  Returns the slots, a multiple of
// 32, or -1: the path is not for this kernel.  S.top and S.top_slot are set.
template <int NT>
__device__ __noinline__ int tile_build(const TileParams& P, const ft_path_desc& d, TileState<NT>& S, TileBuild<NT>& B, int4* E,
                          unsigned* ends) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const ft_op* ops = P.ops + d.op_begin;
    const int n = (int)d.n_ops;
    const float tol_sq = P.tol_sq;
    if (tid == 0) {
        S.c_kind = -1;
        S.c_vo = S.c_rs = -1;
        S.c_px = S.c_py = 0.f;
        S.flags = 0;
        S.top = ~0ull;
        S.top_slot = INT_MAX;
        S.last_pw = -1;
    }
    __syncthreads();
    // the top vertex so far: least (y, x), then the first slot
    int by = INT_MAX, bx = INT_MAX, best_slot = INT_MAX;
    auto consider = [&](int4 e, int slot) {
        if ((e.x != e.z || e.y != e.w) && top_less(e.y, e.x, slot, by, bx, best_slot)) {
            by = e.y;
            bx = e.x;
            best_slot = slot;
        }
    };
    int base = 0, bad = 0;
    for (int c0 = 0; c0 <= n; c0 += NT) {
        const int i = c0 + tid;
        ft_op o;
        o.kind = -1;
        if (i < n) {
            o = tile_op(ops, i);
            if (o.kind < 0 || o.kind > FT_OP_PEN_WIDTH) {
                atomicOr(&S.flags, 2);
                o.kind = -1;
            }
        } else if (i == n) {
            o.kind = TILE_END;
        }
        const int kind = o.kind;
        const bool vo = kind >= FT_OP_MOVE && kind <= FT_OP_CUBIC;
        const bool pc = vo || kind == FT_OP_CLOSE;
        if (P.sw_out && kind == FT_OP_PEN_WIDTH) atomicMax(&S.last_pw, i);
        const unsigned pcb = __ballot_sync(ALL, pc), vob = __ballot_sync(ALL, vo);
        if (lane == 0) {
            S.pcm[w] = pcb;
            S.vom[w] = vob;
        }
        B.kind[tid] = kind;
        const P2 end = vo ? op_end(o) : p2(0.f, 0.f);  // Close puts the pen at the origin (plotter.rs:200-203)
        if (pc) B.endp[tid] = make_float2(end.x, end.y);
        __syncthreads();
        // the pen before this op
        const int lpc = prev_bit<NW>(S.pcm, tid - 1);
        const int pk = lpc >= 0 ? B.kind[lpc] : S.c_kind;
        const P2 pen = lpc >= 0 ? p2(B.endp[lpc].x, B.endp[lpc].y) : p2(S.c_px, S.c_py);
        const bool rs = vo && (kind == FT_OP_MOVE || pk == FT_OP_CLOSE || pk == -1);
        const unsigned rsb = __ballot_sync(ALL, rs);
        if (lane == 0) S.rsm[w] = rsb;
        const int lvo = prev_bit<NW>(S.vom, tid - 1);
        const int lvo_op = lvo >= 0 ? c0 + lvo : S.c_vo;
        const bool closes = (rs || kind == TILE_END) && lvo_op >= 0;  // closes the sub-figure before
        __syncthreads();
        const int lrs = prev_bit<NW>(S.rsm, tid - 1);
        const int lrs_op = lrs >= 0 ? c0 + lrs : S.c_rs;
        // slots of this op
        int slots = closes ? 1 : 0, D = 0, safe = 0, type = TY_POINT;
        float4 ga = make_float4(0.f, 0.f, 0.f, 0.f), gb = ga;
        if (vo) {
            const P2 a = xform(P.xf, pen), e = xform(P.xf, end);
            P2 b = a, c = e;
            if (kind == FT_OP_QUAD || kind == FT_OP_CUBIC) {
                b = xform(P.xf, p2(o.v[0], o.v[1]));
                c = xform(P.xf, p2(o.v[2], o.v[3]));
                if (!pfinite(a) || !pfinite(b) || !pfinite(c) || !pfinite(e)) {
                    atomicOr(&S.flags, 2);
                } else {
                    type = kind == FT_OP_QUAD ? TY_QUAD : TY_CUBIC;
                    D = curve_depth(a, b, c, e, type == TY_CUBIC, P.tol, safe);
                    if (D > SLOT_DEPTH) {
                        bad = 1;
                        D = safe = 0;
                    }
                }
            }
            ga = make_float4(a.x, a.y, b.x, b.y);
            gb = make_float4(c.x, c.y, e.x, e.y);
            slots += 1 << D;
        }
        // slot offsets and places in the list of ops with slots, in one scan
        const unsigned mine = (unsigned)slots | ((slots ? 1u : 0u) << 22);
        unsigned inc = mine;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const unsigned t = __shfl_up_sync(ALL, inc, s);
            if (lane >= s) inc += t;
        }
        if (lane == 31) S.wsum[w] = inc;
        __syncthreads();
        unsigned pre = 0, sum = 0;
#pragma unroll
        for (int k = 0; k < NW; k++) {
            const unsigned v = S.wsum[k];
            if (k < w) pre += v;
            sum += v;
        }
        const int listed = (int)(sum >> 22), total = (int)(sum & ((1u << 22) - 1));
        const unsigned excl = pre + inc - mine;
        const int off = (int)(excl & ((1u << 22) - 1));
        if (slots && ck(excl >> 22 < (unsigned)NT, 20)) {
            const int at = (int)(excl >> 22);
            B.g0[at] = ga;
            B.g1[at] = gb;
            B.off[at] = off;
            B.info[at] = D | (safe << 4) | (type << 8) | ((closes ? 1 : 0) << 10) | ((rs ? 1 : 0) << 11);
        }
        if (tid < 32) B.off[listed + tid] = INT_MAX;
        const int padded = (total + 31) & ~31;
        // (not foretold from the ops so far: dense ones often come first, and a path that fits after
        // all takes k_raster up to five times as long, 700 x 700 under 600 curves, then 3,000 lines
        // 114 / 469 us; foreseen, 30,000 curves took 1,861 us instead of 2,016)
        if (base + padded > P.cap) bad = 1;
        if (__syncthreads_or(bad)) break;
        if (closes) {  // last vertex -> first vertex of the sub-figure that ends here
            const P2 l = xform(P.xf, lvo >= 0 ? p2(B.endp[lvo].x, B.endp[lvo].y) : op_end(tile_op(ops, S.c_vo)));
            const P2 f = first_vertex(P, ops, lrs_op);
            const int4 e = make_int4(to_fx(l.x), to_fx(l.y), to_fx(f.x), to_fx(f.y));
            if (ck(base + off < P.cap, 21)) E[base + off] = e;
            consider(e, base + off);
        }
        __syncthreads();
        if (tid == NT - 1) {  // carry (the arrays below are read-only until the next chunk)
            const int p = prev_bit<NW>(S.pcm, NT - 1);
            if (p >= 0) {
                S.c_kind = B.kind[p];
                S.c_px = B.endp[p].x;
                S.c_py = B.endp[p].y;
            }
            const int v = prev_bit<NW>(S.vom, NT - 1);
            if (v >= 0) S.c_vo = c0 + v;
            const int r = prev_bit<NW>(S.rsm, NT - 1);
            if (r >= 0) S.c_rs = c0 + r;
        }
        // one slot per thread, 32 slots per warp at a time
        int j0 = 0;
        for (int s0 = w * 32; s0 < padded; s0 += NT) {
            const int s = s0 + lane;
            const int lo = slot_op(B.off, s0, j0);
            int4 e = make_int4(0, 0, 0, 0);
            bool close_slot = false;
            if (s < total) {
                const int info = B.info[lo];
                const int idx = s - B.off[lo] - ((info >> 10) & 1);
                close_slot = idx < 0;
                if (!close_slot && !(((info >> 11) & 1) && idx == 0 && ((info >> 8) & 3) == TY_POINT)) {
                    const float4 g0 = B.g0[lo], g1 = B.g1[lo];
                    P2 a = p2(g0.x, g0.y), z = p2(g1.z, g1.w);
                    const int type = (info >> 8) & 3, D = info & 15, safe = (info >> 4) & 15;
                    float w = 0.f;
                    int at = 0;  // the leaf's depth, -1: none
                    if (type == TY_QUAD)
                        at = quad_slot(a, p2(g0.z, g0.w), z, w, w, w, idx, D, safe, tol_sq);
                    else if (type == TY_CUBIC)
                        at = cubic_slot(a, p2(g0.z, g0.w), p2(g1.x, g1.y), z, w, w, w, w, idx, D, safe, tol_sq);
                    // the first vertex of a sub-figure ends no segment
                    if (at >= 0 && !(((info >> 11) & 1) && idx == 0))
                        e = make_int4(to_fx(a.x), to_fx(a.y), to_fx(z.x), to_fx(z.y));
                }
            }
            const unsigned cm = __ballot_sync(ALL, close_slot);
            if (lane == 0) ends[(base + s) >> 5] = cm;
            if (!close_slot && ck(base + s < P.cap, 22)) E[base + s] = e;
            consider(e, base + s);
        }
        base += padded;
        __syncthreads();
    }
    if (__syncthreads_or(bad)) return -1;
    const unsigned long long best = best_slot != INT_MAX ? top_key(bx, by) : ~0ull;
    unsigned long long k = best;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        const unsigned long long t = __shfl_xor_sync(ALL, k, s);
        k = t < k ? t : k;
    }
    if (lane == 0 && k != ~0ull) atomicMin(&S.top, k);
    __syncthreads();
    if (best != ~0ull && best == S.top) atomicMin(&S.top_slot, best_slot);
    __syncthreads();
    return base;
}

// Direction of the figure (fig.rs:402-411, 116-119), by one warp: the non-zero segment out
// of the top vertex and the one into it.
__device__ __noinline__ int tile_dir(const int4* E, const unsigned* ends, int n_slots, int top) {
    const int lane = threadIdx.x & 31;
    const int4 out = E[top];
    int4 in = out;
    bool found = false, edge = false;  // edge: the sub-figure's first slot was passed
    auto back = [&](int hi, int lo) {  // the last non-zero segment of slots hi, hi - 1, ... lo
        for (int e = hi; e >= lo && !found && !edge; e -= 32) {
            const int k = e - lane;
            int4 v = make_int4(0, 0, 0, 0);
            bool closing = false;
            if (k >= lo) {
                v = E[k];
                closing = k < top && ((ends[k >> 5] >> (k & 31)) & 1);
            }
            const unsigned nz = __ballot_sync(ALL, v.x != v.z || v.y != v.w), cl = __ballot_sync(ALL, closing);
            const int f = nz ? __ffs(nz) - 1 : 32, c = cl ? __ffs(cl) - 1 : 32;
            if (f < c) {
                in.x = __shfl_sync(ALL, v.x, f);
                in.y = __shfl_sync(ALL, v.y, f);
                found = true;
            }
            edge = c < 32 && !found;
        }
    };
    back(top - 1, 0);
    if (!found) {
        // the top is its sub-figure's first vertex: backwards from the sub-figure's closing slot
        int last = n_slots - 1;
        for (int g = top >> 5; g < n_slots >> 5; g += 32) {
            unsigned m = g + lane < n_slots >> 5 ? ends[g + lane] : 0u;
            if (g + lane == top >> 5) m &= ALL << (top & 31);
            const unsigned any = __ballot_sync(ALL, m != 0);
            if (any) {
                const int f = __ffs(any) - 1;
                last = ((g + f) << 5) + __ffs(__shfl_sync(ALL, m, f)) - 1;
                break;
            }
        }
        edge = false;
        back(last, top);
    }
    const int ax = wsub(in.x, out.x), ay = wsub(in.y, out.y), cx = wsub(out.z, out.x), cy = wsub(out.w, out.y);
    return fxmul(ax, cy) > fxmul(cx, ay) ? 0 : 1;
}

// ------------------------------------------------------------------- raster
// Items of the first m segments in Q.q (all reach rows [yb0, yb1)) into `area`.
__device__ __forceinline__ void tile_items(TileWarp& Q, int m, int yb0, int yb1, int* area, int cells, int pitch, int W) {
    const int lane = threadIdx.x & 31;
    SegRec s;
    s.n_items = 0;
    s.ra = s.rb = make_int4(0, 0, 0, 0);
    if (lane < m) {
        const int4 e = Q.q[lane];
        const bool down = e.w > e.y;
        const int ux = down ? e.x : e.z, uy = down ? e.y : e.w, lx = down ? e.z : e.x, ly = down ? e.w : e.y;
        const int dx = wsub(lx, ux), dy = wsub(ly, uy);
        const unsigned ady = uabs(dy), adx = uabs(dx);
        // fig.rs:187-199; a slope of ONE and above is ONE
        int step = FX_ONE;
        if (ady < adx) {
            step = (int)fx_quot(ady, adx);
        } else if (adx != 0 && (ady >> 15) >= adx) {  // 32,768 and more: the wrapped low half decides
            step = min(fxabs(fx_div(dy, dx)), FX_ONE);
        }
        if (step <= 0) step = FX_ONE;  // step_cov(ONE) (fig.rs:315-321)
        s = seg_items(ux, fxfract(uy), fxfract(ly), uy >> 16, ly >> 16, fx_div(dx, dy), step, !down, yb0, yb1, pitch, W);
    }
    run_items(Q.rec, s, area, cells, pitch, W);
}

struct TileOut {  // where a band's rows go (in shared memory: it would only hold registers)
    uint8_t* base;   // the raster
    unsigned stride, clr;
    int W, pitch, rule, fmt;
    int neg;         // the figure runs in reverse: cell sums change sign
    int lprl;        // log2 of the lanes per row, eight pixels each
    int cells;       // of the area; the staged bytes are as many and 256 more
    bool host;       // mapped host memory: Matte8 rows leave as aligned words
    bool words;      // rows on 4-byte boundaries
    unsigned char* stg;
};

// Resolve rows r0 .. r0 + nr - 1 (imgbuf.rs:38-199) from `area`, clearing it, and write them
// (fig.rs:621-665).  Matte8 in device memory, rows of at most 256 pixels on 4-byte
// boundaries: each lane eight pixels, as many rows a warp as fit, straight-line.
template <int NT, int RULE>
__device__ __noinline__ void tile_rows_matte(const TileOut& T, int* area, int r0, int nr) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = lane & ((1 << T.lprl) - 1), rpw = 32 >> T.lprl, first = warp * rpw + (lane >> T.lprl);
    const int nb = T.W - 8 * l, sg = T.neg ? -1 : 1;
    int* ap = area + first * T.pitch + 8 * l;
    uint8_t* dp = T.base + (size_t)(r0 + first) * T.stride + 8 * l;
    for (int q = warp * rpw; q < nr; q += NW * rpw) {
        const bool in = nb > 0 && q + (lane >> T.lprl) < nr && ck(ap + 8 - area <= T.cells, 25);
        unsigned s[8], inc;
        take8(ap, in, l, s, inc);
        const uint2 px = pixels8<RULE>(s, inc - s[7], sg);
        if (in) {  // written once and not read back
            if (nb >= 4) __stcs(reinterpret_cast<unsigned*>(dp), px.x);
            if (nb >= 8)
                __stcs(reinterpret_cast<unsigned*>(dp + 4), px.y);
            else if (nb & 3)
                store_tail(dp + (nb & 4), nb < 4 ? px.x : px.y, nb & 3);
        }
        ap += NW * rpw * T.pitch;
        dp += (size_t)(NW * rpw) * T.stride;
    }
}

// Every other row: Rgba8p, host rasters, unaligned or wide Matte8; `o0`: with contiguous host
// rows, the staged byte of row r0's first pixel.
template <int NT, int RULE>
__device__ __noinline__ void tile_rows(const TileOut& T, int* area, int r0, int nr, bool contig, int o0) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = T.W, lpr = 1 << T.lprl, rpw = 32 >> T.lprl, l = lane & (lpr - 1), sub = lane >> T.lprl;
    for (int q = warp * rpw; q < nr; q += NW * rpw) {
        const int rr = q + sub;
        const bool valid = rr < nr;
        int* arow = area + rr * T.pitch;
        uint8_t* drow = T.base + (size_t)(r0 + rr) * T.stride;
        unsigned carry = 0;
        for (int x0 = 0; x0 < W; x0 += lpr * 8) {
            const int x = x0 + l * 8, nb = min(W - x, 8);
            const bool in = valid && nb > 0 && ck(arow + x + 8 - area <= T.cells, 25);
            unsigned s[8], inc;
            take8(arow + x, in, l, s, inc);
            const uint2 px = pixels8<RULE>(s, inc - s[7] + carry, T.neg ? -1 : 1);
            carry += __shfl_sync(ALL, inc, lpr - 1, lpr);
            if (!in) continue;
            if (contig) {
                unsigned char* sp = T.stg + o0 + rr * W + x;
                if (ck(o0 + rr * W + x + nb <= T.cells + 256, 24)) for (int k = 0; k < nb; k++) sp[k] = (uint8_t)((k < 4 ? px.x : px.y) >> (8 * (k & 3)));
            } else if (T.fmt == FT_MATTE8 && !T.host && T.words) {
                if (nb >= 4) __stcs(reinterpret_cast<unsigned*>(drow + x), px.x);
                if (nb >= 8)
                    __stcs(reinterpret_cast<unsigned*>(drow + x + 4), px.y);
                else if (nb & 3)
                    store_tail(drow + x + (nb & 4), nb < 4 ? px.x : px.y, nb & 3);
            } else if (T.fmt == FT_MATTE8 && !T.host) {
                for (int k = 0; k < nb; k++) drow[x + k] = (uint8_t)((k < 4 ? px.x : px.y) >> (8 * (k & 3)));
            } else {
                if (ck(rr * T.pitch + x + 8 <= T.cells + 256, 24)) *reinterpret_cast<uint2*>(T.stg + rr * T.pitch + x) = px;
            }
        }
        if (contig || (T.fmt == FT_MATTE8 && !T.host)) continue;
        __syncwarp();
        if (valid) {
            const unsigned char* sp = T.stg + rr * T.pitch;
            if (T.fmt == FT_RGBA8P) {
                unsigned* dp = reinterpret_cast<unsigned*>(drow);
                for (int x = l; x < W; x += 4 * lpr) {  // four loads in flight per lane
                    unsigned v[4], av[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int at = x + k * lpr;
                        v[k] = at < W ? dp[at] : 0u;  // a pixel of 0 under no coverage stays
                        av[k] = at < W ? sp[at] : 0u;
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (av[k] || low_channels(v[k])) dp[x + k * lpr] = srcover_rgba(v[k], T.clr, av[k]);
                }
            } else {  // aligned words of a host row, its ends byte by byte
                const int mis = (int)(reinterpret_cast<uintptr_t>(drow) & 3);
                for (int x = 4 * l - mis; x < W; x += 4 * lpr) {
                    if (x >= 0 && x + 4 <= W) {
                        *reinterpret_cast<unsigned*>(drow + x) = (unsigned)sp[x] | ((unsigned)sp[x + 1] << 8) |
                                                                 ((unsigned)sp[x + 2] << 16) | ((unsigned)sp[x + 3] << 24);
                    } else {
                        for (int k = max(x, 0); k < min(x + 4, W); k++) drow[k] = sp[k];
                    }
                }
            }
        }
        __syncwarp();
    }
}

template <int NT>
struct TileLayout {
    static constexpr int build = (int)((sizeof(TileBuild<NT>) + 15) & ~(size_t)15);
    static constexpr int warps = (int)sizeof(TileWarp) * (NT / 32);
    // the build's arrays and the raster's queues, cells and staged bytes share the space
    static int bytes(int area_ints, bool staged) {
        const int raster = warps + area_ints * 4 + (staged ? area_ints + 256 : 0);
        return raster > build ? raster : build;
    }
};

template <int NT>
__global__ void __launch_bounds__(NT, NT == 32 ? 32 : NT == 128 ? 8 : 2) k_tile(TileParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ TileState<NT> S;
    __shared__ TileOut T;
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned char* scr = P.scratch + (size_t)blockIdx.x * tile_scratch(P.cap);
    int4* E = reinterpret_cast<int4*>(scr);
    unsigned* ends = reinterpret_cast<unsigned*>(scr + (size_t)P.cap * sizeof(int4));
    TileBuild<NT>& B = *reinterpret_cast<TileBuild<NT>*>(smem);
    TileWarp& Q = reinterpret_cast<TileWarp*>(smem)[warp];
    int* area = reinterpret_cast<int*>(smem + TileLayout<NT>::warps);
    // k_raster, behind this kernel, may be set up (it waits for this kernel's end)
    if (P.single) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int round = 0;; round++) {
        int it = blockIdx.x;
        WorkItem wi;
        ft_path_desc d;
        if (P.single) {
            if (round) break;
            d = P.d;
            wi = WorkItem{0, (uint32_t)(it * P.rows_per), min(d.height, (uint32_t)((it + 1) * P.rows_per)), 0};
        } else {
            if (tid == 0) S.item = (int)atomicAdd(&P.queue[1], 1u);
            __syncthreads();
            it = S.item;
            if (it >= (int)P.n_items) break;
            wi = P.items[it];
            d = P.paths[wi.path];
        }
        const float sw0 = P.sw_chain ? *P.sw_chain : d.s_width;
        const int n_slots = tile_build<NT>(P, d, S, B, E, ends);
        if (P.single && tid == 0) P.overflow[it] = n_slots < 0;
        if (n_slots < 0) {  // these rows go to k_raster
            if (!P.single && tid == 0) P.overflow[atomicAdd(&P.queue[2], 1u)] = (uint32_t)it;
            __syncthreads();
            continue;
        }
        if (tid == 0 && wi.row_begin == 0) {
            if (P.single)
                P.status[0] = S.flags ? FT_ERR_ARG : FT_OK;
            else if (S.flags)
                atomicMax(&P.status[wi.path], FT_ERR_ARG);
            if (P.sw_out) P.sw_out[wi.path] = S.last_pw >= 0 ? P.ops[d.op_begin + S.last_pw].v[0] : sw0;
        }
        const int W = (int)d.width, H = (int)d.height;
        if (S.top != ~0ull && W > 0) {
            const int top_row = (int)((unsigned)(S.top >> 32) ^ 0x80000000u) >> 16;
            const int tmin = min(top_row, 0);
            const int lo = max((int)wi.row_begin, max(top_row, 0)), hi = min((int)wi.row_end, H);
            const int pitch = tile_pitch(W);
            const int R = max(1, min(P.area_ints / pitch, 1024));
            uint8_t* const base = P.rasters + d.raster_offset;
            const bool host = P.host_rasters != 0;
            if (tid == 0) {
                T.base = base;
                T.stride = d.stride;
                T.clr = (unsigned)d.clr[0] | ((unsigned)d.clr[1] << 8) | ((unsigned)d.clr[2] << 16) |
                        ((unsigned)d.clr[3] << 24);
                T.W = W;
                T.pitch = pitch;
                T.cells = P.area_ints;
                T.rule = P.rule;
                T.fmt = P.fmt;
                T.host = host;
                T.stg = smem + TileLayout<NT>::warps + P.area_ints * 4;
                T.lprl = W <= 8 ? 0 : min(32 - __clz((W - 1) >> 3), 5);
            }
            const bool words = (((unsigned)reinterpret_cast<uintptr_t>(base) | d.stride) & 3) == 0;
            const bool quick = P.fmt == FT_MATTE8 && !host && W <= 256 && words;
            if (tid == 0) T.words = words;
            // contiguous host rows: whole 128-byte lines leave from the staging bytes
            const bool contig = host && P.fmt == FT_MATTE8 && d.stride == d.width;
            uint8_t* const g0 = base + (size_t)lo * d.stride;
            uint8_t* const g1 = base + (size_t)hi * d.stride;
            uint8_t* L0 = reinterpret_cast<uint8_t*>(reinterpret_cast<uintptr_t>(g0) & ~(uintptr_t)127);
            if (lo < hi) {
                const int cells = min(R, hi - lo) * pitch;
                for (int x = tid * 4; x < cells; x += NT * 4) *reinterpret_cast<int4*>(area + x) = make_int4(0, 0, 0, 0);
                __syncthreads();
                if (warp == 0) {
                    const int dir = tile_dir(E, ends, n_slots, S.top_slot);
                    if (lane == 0) T.neg = dir;
                }
                for (int r0 = lo; r0 < hi; r0 += R) {
                    const int nr = min(R, hi - r0), yb0 = r0 + tmin, yb1 = yb0 + nr;
                    int cnt = 0;
                    for (int g = warp;; g += NW) {
                        const bool more = g < n_slots >> 5;
                        if (more) {
                            const int4 e = E[g * 32 + lane];
                            const int y0 = min(e.y, e.w), y1 = max(e.y, e.w);
                            const bool on = y0 != y1 && (y0 >> 16) < yb1 && ((y1 - 1) >> 16) >= yb0;
                            const unsigned m = __ballot_sync(ALL, on);
                            const int at = cnt + __popc(m & ((1u << lane) - 1u));
                            if (on && ck(at < 64, 23)) Q.q[at] = e;
                            cnt += __popc(m);
                            __syncwarp();
                        }
                        if (cnt >= 32 || (!more && cnt > 0)) {
                            tile_items(Q, min(cnt, 32), yb0, yb1, area, P.area_ints, pitch, W);
                            cnt -= 32;
                            if (lane < cnt) Q.q[lane] = Q.q[32 + lane];
                            __syncwarp();
                        }
                        if (!more) break;
                    }
                    __syncthreads();
                    const int o0 = contig ? (int)(base + (size_t)r0 * d.stride - L0) : 0;
                    if (quick && P.rule == FT_NONZERO)
                        tile_rows_matte<NT, FT_NONZERO>(T, area, r0, nr);
                    else if (quick)
                        tile_rows_matte<NT, FT_EVENODD>(T, area, r0, nr);
                    else if (P.rule == FT_NONZERO)
                        tile_rows<NT, FT_NONZERO>(T, area, r0, nr, contig, o0);
                    else
                        tile_rows<NT, FT_EVENODD>(T, area, r0, nr, contig, o0);
                    __syncthreads();
                    if (contig) {
                        const bool last = r0 + nr >= hi;
                        const int fill = o0 + nr * W, lines = last ? (fill + 127) >> 7 : fill >> 7;
                        for (int x = tid * 16; x < lines * 128 && ck(x + 16 <= P.area_ints + 256, 24); x += NT * 16) {
                            uint8_t* a = L0 + x;
                            const uint4 v = *reinterpret_cast<const uint4*>(T.stg + x);
                            if (a >= g0 && a + 16 <= g1) {
                                *reinterpret_cast<uint4*>(a) = v;
                            } else {
                                for (int k = 0; k < 16; k++)
                                    if (a + k >= g0 && a + k < g1) a[k] = T.stg[x + k];
                            }
                        }
                        if (!last && lines > 0) {  // the partial line moves to the front
                            const int rest = fill - lines * 128;
                            __syncthreads();
                            if (tid * 16 < rest)
                                *reinterpret_cast<uint4*>(T.stg + tid * 16) =
                                    *reinterpret_cast<const uint4*>(T.stg + lines * 128 + tid * 16);
                            L0 += lines * 128;
                        }
                        __syncthreads();
                    }
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace

static_assert(TILE_THREADS_TINY == 32 && TILE_THREADS == 128 && TILE_THREADS_FEW == 512, "the kernels there are");
int tile_smem(int threads, int area_ints, bool staged) {
    if (threads == 32) return TileLayout<32>::bytes(area_ints, staged);
    return threads == 128 ? TileLayout<128>::bytes(area_ints, staged) : TileLayout<512>::bytes(area_ints, staged);
}

int tile_blocks_per_sm(int threads, int smem) {
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &n, threads == 32 ? k_tile<32> : threads == 128 ? k_tile<128> : k_tile<512>, threads, smem);
    return e == cudaSuccess && n > 0 ? n : 1;
}

cudaError_t take_check_tile(CheckState* s, bool reached) { return take_check(s, reached); }

cudaError_t setup_tile() {
    const cudaError_t e = allow_smem((const void*)k_tile<128>);  // (k_tile<32> stays within 48 KB)
    return e == cudaSuccess ? allow_smem((const void*)k_tile<512>) : e;
}

cudaError_t launch_tile(const TileParams& p, int threads, int grid, int smem, cudaStream_t s) {
    auto kern = threads == 32 ? k_tile<32> : threads == 128 ? k_tile<128> : k_tile<512>;
    kern<<<grid, threads, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace ftk
