// Slab level step: image model + N propagation sub-steps + update + S smoothing iterations of
// one pyramid level, one CTA per slab of 128 columns x `rows` rows, held in shared memory.
//
// The CTA loads the previous frame's state over its slab plus a halo into shared memory, one
// plane per channel and row, and runs the stages there one after the other, each over the
// rows the later stages need (one stencil radius fewer per stage):
//
//   N x (upwind X/Y sub-step pair)   rows +- (N - k + 2S), in place
//   image model and update           rows +- 2S, in place; stores delta / old image / flow
//   S x (box X, box Y)               rows +- 2 (S - s), ping-pong; the last Y pass stores
//
// Lanes take four adjacent columns each (16-byte shared-memory accesses; horizontal neighbours
// by warp shuffles), so a warp takes whole rows of the slab, and the rows of a stage are split
// over the warps as one run of consecutive rows each: the Y sub-step's row window stays in
// registers down a run.  Columns outside the slab are not exchanged between slabs: the outer
// HX columns on each side are recomputed by the neighbour.
//
// Why this shape: a stage is one loop that all warps run at the same time, small enough for the
// instruction cache (a kernel that gave every stage its own warps, rows handed over in shared
// memory, ran out of it: 98 us where this one takes 89), and four pixels per lane give
// independent work that covers latency with 8 warps an SM.  It issues 40% fewer instructions
// than the tile kernel (640x480, N 4 S 2: 9.0 M against 14.6 M), whose lanes index every pixel
// of every stage.  Bound by latency within the stages: 37% of the issue slots, stalls on
// shared-memory loads and shuffles, DRAM idle.
// Measured alone on a delta level (us, this / streaming / tile kernel): 640x480 N 4 S 2
// 26.1 / 58.9 / 34.3, 1001x701 N 3 S 2 32.2 / 50.7 / 46.6, 1280x720 N 4 S 2 45.3 / 62.9 / 69.4.
//
// Reads outside the image are clamped to the edge, as the reference's textures do; rows and
// slabs away from the edges and the propagation border run a body without any of that
// handling.  The arithmetic is the per-stage kernels' operation for operation (common.cuh),
// so results are bit-identical to them.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace ffb {
namespace slab {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kCols = 128;          // columns of a slab with its halo, 4 per lane
constexpr int kPlane = kCols * 4;   // bytes of one channel of a row
constexpr int kWarps = 8;           // warps of a slab: the row windows take over 128 registers

__host__ __device__ constexpr int halo_x(int N, int S) { return ((2 * S + (N > 2 ? N : 2)) + 3) & ~3; }
// columns from a window to the next
__host__ __device__ constexpr int slab_cols(int N, int S) { return kCols - 2 * halo_x(N, S); }
// planes of a row: the propagated channels U, V, I, DX, DY (delta levels); U, V and the
// smoothing passes' second pair (top levels)
__host__ __device__ constexpr int planes(bool delta) { return delta ? 5 : 4; }
// shared memory of a slab: its rows with halo and one spare row per warp
__host__ __device__ constexpr int slab_smem(bool delta, int N, int S, int rows) {
    return (rows + 2 * (N + 2 * S) + kWarps) * planes(delta) * kPlane;
}

// The slabs of a level: nwx windows across, the inner ones cut into bands of `rows` rows, the
// first and last (where the image edges are, and a row costs more) into bands of rows_e.
struct Geom {
    int N, S;
    int nwx, rows, rows_e;
    int nby_e, ne;  // bands of an edge window; edge windows (1 or 2)
    __host__ __device__ int slabs(int H) const { return ne * nby_e + (nwx - ne) * ((H + rows - 1) / rows); }
    // window, first row and row count of slab i (edge slabs first: they start earliest)
    __device__ __forceinline__ void at(int i, int& wx, int& ys, int& n) const {
        if (i < ne * nby_e) {
            wx = i < nby_e ? 0 : nwx - 1;
            n = rows_e;
            ys = (i < nby_e ? i : i - nby_e) * rows_e;
        } else {
            i -= ne * nby_e;
            wx = 1 + i % (nwx - ne);
            n = rows;
            ys = i / (nwx - ne) * rows;
        }
    }
};

extern __shared__ __align__(16) char slab_smem_[];

// four pixels of one channel: a = (pixel 0, pixel 1), b = (pixel 2, pixel 3)
struct Q {
    float2 a, b;
};
__device__ __forceinline__ Q ldq(unsigned off) {
    const float4 v = *reinterpret_cast<const float4*>(slab_smem_ + off);
    return Q{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void stq(unsigned off, const Q& q) {
    *reinterpret_cast<float4*>(slab_smem_ + off) = make_float4(q.a.x, q.a.y, q.b.x, q.b.y);
}

// p + y * pitch for a row y >= 0; pitches are below 2^32 bytes, so the offset is one
// 32 x 32 -> 64-bit multiply-add
template <typename T>
__device__ __forceinline__ T* rowp(T* p, unsigned pitch, int y) {
    using B = std::conditional_t<std::is_const_v<T>, const char, char>;
    return reinterpret_cast<T*>(reinterpret_cast<B*>(p) + (unsigned long long)(unsigned)y * pitch);
}

__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }

__device__ __forceinline__ void cp16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp8(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}

struct Ctx {
    int W, H, border, lane, warp;
    int c0;             // first pixel column of this lane
    int wcol;           // first column of its 4-pixel loads, inside the image
    int ys, ye;         // output rows
    int nout;           // pixels this lane stores (0 outside the slab's output columns)
    bool vec;           // all four at once (flow rows 32-byte, scalar rows 16-byte aligned)
    unsigned l16;       // 16 * lane
    int cin;            // bit j: pixel j outside the propagation border columns
    bool e_l, e_r;      // c0 == 0; c0 + 3 == W - 1
    int rag;            // W - 1 - c0 where column W - 1 is pixel 0..2 of this lane, else -1
    bool edge;          // block-uniform: some lane is at an image edge, a border column or outside
    bool rows_edge;     // block-uniform: edge, or rows of the propagation border
    int sy0;            // first row in shared memory
    unsigned spare;     // the warp's spare row
    // rows of radius r around the output, cut to the image, split over the warps
    __device__ __forceinline__ void run_of(int r, int& y0, int& y1) const {
        const int a = max(0, ys - r), n = min(H, ye + r) - a;
        y0 = a + n * warp / kWarps;
        y1 = a + n * (warp + 1) / kWarps;
    }
};

// the slab's output columns of a row: lanes store all four pixels, or (at a ragged right
// edge, or with unaligned rows) n of them one by one
__device__ __forceinline__ void store_f2(bool vec, int n, float2* row, const Q& u, const Q& v) {
    if (vec) {  // one 32-byte store: whole sectors, half the store instructions of 16-byte ones
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(row), "f"(u.a.x), "f"(v.a.x),
                     "f"(u.a.y), "f"(v.a.y), "f"(u.b.x), "f"(v.b.x), "f"(u.b.y), "f"(v.b.y)
                     : "memory");
    } else {
        if (n > 0) row[0] = make_float2(u.a.x, v.a.x);
        if (n > 1) row[1] = make_float2(u.a.y, v.a.y);
        if (n > 2) row[2] = make_float2(u.b.x, v.b.x);
        if (n > 3) row[3] = make_float2(u.b.y, v.b.y);
    }
}
__device__ __forceinline__ void store_f1(bool vec, int n, float* row, const Q& v) {
    if (vec) {
        *reinterpret_cast<float4*>(row) = make_float4(v.a.x, v.a.y, v.b.x, v.b.y);
    } else {
        if (n > 0) row[0] = v.a.x;
        if (n > 1) row[1] = v.a.y;
        if (n > 2) row[2] = v.b.x;
        if (n > 3) row[3] = v.b.y;
    }
}

// Where a forward that is differentiated later keeps its intermediates, dense images of the
// level: the propagated channels after every X and Y sub-step, the image gradient, and the
// input of every smoothing pass.
struct Tape {
    float *f, *s, *v;  // sub-step 0's flow, scalar and vector payload (delta levels)
    size_t step;       // elements from a sub-step to the next
    float* grad;
    float* sm;         // smoothing pass 0's input
    size_t sm_step;
};

// ---------------------------------------------------------------- propagation
template <bool DELTA>
struct Prop {
    static constexpr int NC = DELTA ? 5 : 2;  // propagated channels: U, V [, I, DX, DY]
    static constexpr unsigned ROWB = planes(DELTA) * kPlane;  // unsigned: a row index times it may pass 2^31, and the offsets are differences
    static constexpr int CU = 0, CV = 1;
    // channels whose upwind step the reference build fuses into one fma: all but the last
    // channel each reference kernel writes (flow .y of flowPropagate{X,Y}_k, vector .y of
    // flowPropagatePayload{X,Y}_k)
    static constexpr bool fused(int ch) { return ch != NC - 1; }
    struct Row {
        Q q[NC];
    };

    // v - |t| (v - n) with the negated |t| of the pair (scalar: the packed two-lane form needs
    // the selected neighbours in register pairs, and the moves cost what it saves)
    template <bool FUSED>
    __device__ __forceinline__ static float2 up2(float2 v, float2 n, float2 nat) {
        const float dx = __fsub_rn(v.x, n.x), dy = __fsub_rn(v.y, n.y);
        if (FUSED) return make_float2(__fmaf_rn(nat.x, dx, v.x), __fmaf_rn(nat.y, dy, v.y));
        return make_float2(__fadd_rn(v.x, __fmul_rn(nat.x, dx)), __fadd_rn(v.y, __fmul_rn(nat.y, dy)));
    }
    // the neighbour before pixel 0 and after pixel 3, clamped at the image edges (E)
    template <bool E>
    __device__ __forceinline__ static void around(const Ctx& c, const Q& v, float& L, float& R) {
        L = __shfl_up_sync(kFull, v.b.y, 1);
        R = __shfl_down_sync(kFull, v.a.x, 1);
        if (E) {
            L = c.e_l ? v.a.x : L;
            R = c.e_r ? v.b.y : R;
        }
    }

    // X sub-step of a row (flowPropagateX_k / flowPropagatePayloadX_k)
    template <bool E, int FROM>
    __device__ __forceinline__ static void xstep(const Ctx& c, float dt, const Row& v, Row& o) {
        float L[NC], R[NC];
#pragma unroll
        for (int ch = 0; ch < NC; ++ch)
            if (ch >= FROM || ch == CU) around<E>(c, v.q[ch], L[ch], R[ch]);
        // the neighbour after pixels 0..2 (E: the pixel itself at a ragged right edge)
        auto right0 = [&](int ch) { return E && c.rag == 0 ? v.q[ch].a.x : v.q[ch].a.y; };
        auto right1 = [&](int ch) { return E && c.rag == 1 ? v.q[ch].a.y : v.q[ch].b.x; };
        auto right2 = [&](int ch) { return E && c.rag == 2 ? v.q[ch].b.x : v.q[ch].b.y; };
        const Q& u = v.q[CU];
        const float v0 = dominant(L[CU], right0(CU)), v1 = dominant(u.a.x, right1(CU));
        const float v2 = dominant(u.a.y, right2(CU)), v3 = dominant(u.b.x, R[CU]);
        const bool f0 = v0 >= 0.0f, f1 = v1 >= 0.0f, f2 = v2 >= 0.0f, f3 = v3 >= 0.0f;
        const float2 na = make_float2(__fmul_rn(dt, -fabsf(v0)), __fmul_rn(dt, -fabsf(v1)));
        const float2 nb = make_float2(__fmul_rn(dt, -fabsf(v2)), __fmul_rn(dt, -fabsf(v3)));
#pragma unroll
        for (int ch = FROM; ch < NC; ++ch) {
            const Q& x = v.q[ch];
            const float2 n0 = make_float2(f0 ? L[ch] : right0(ch), f1 ? x.a.x : right1(ch));
            const float2 n1 = make_float2(f2 ? x.a.y : right2(ch), f3 ? x.b.x : R[ch]);
            Q r;
            if (fused(ch)) {
                r.a = up2<true>(x.a, n0, na);
                r.b = up2<true>(x.b, n1, nb);
            } else {
                r.a = up2<false>(x.a, n0, na);
                r.b = up2<false>(x.b, n1, nb);
            }
            if (E) freeze(c, x, r);
            o.q[ch] = r;
        }
    }

    // border columns keep their value (propagation_k.cu:59-65)
    __device__ __forceinline__ static void freeze(const Ctx& c, const Q& v, Q& o) {
        o.a.x = c.cin & 1 ? o.a.x : v.a.x;
        o.a.y = c.cin & 2 ? o.a.y : v.a.y;
        o.b.x = c.cin & 4 ? o.b.x : v.b.x;
        o.b.y = c.cin & 8 ? o.b.y : v.b.y;
    }

    // Y sub-step of row `cur` from the rows before and after it
    template <bool E, int FROM>
    __device__ __forceinline__ static void ystep(const Ctx& c, float dt, const Row& prev, const Row& cur,
                                                 const Row& next, Row& o) {
        const Q &m = prev.q[CV], &p = next.q[CV];
        const float v0 = dominant(m.a.x, p.a.x), v1 = dominant(m.a.y, p.a.y), v2 = dominant(m.b.x, p.b.x), v3 = dominant(m.b.y, p.b.y);
        const bool f0 = v0 >= 0.0f, f1 = v1 >= 0.0f, f2 = v2 >= 0.0f, f3 = v3 >= 0.0f;
        const float2 na = make_float2(__fmul_rn(dt, -fabsf(v0)), __fmul_rn(dt, -fabsf(v1)));
        const float2 nb = make_float2(__fmul_rn(dt, -fabsf(v2)), __fmul_rn(dt, -fabsf(v3)));
#pragma unroll
        for (int ch = FROM; ch < NC; ++ch) {
            const Q &x = cur.q[ch], &mm = prev.q[ch], &pp = next.q[ch];
            const float2 n0 = make_float2(f0 ? mm.a.x : pp.a.x, f1 ? mm.a.y : pp.a.y);
            const float2 n1 = make_float2(f2 ? mm.b.x : pp.b.x, f3 ? mm.b.y : pp.b.y);
            Q r;
            if (fused(ch)) {
                r.a = up2<true>(x.a, n0, na);
                r.b = up2<true>(x.b, n1, nb);
            } else {
                r.a = up2<false>(x.a, n0, na);
                r.b = up2<false>(x.b, n1, nb);
            }
            if (E) freeze(c, x, r);
            o.q[ch] = r;
        }
    }

    __device__ __forceinline__ static void load(unsigned s, Row& x) {
#pragma unroll
        for (int ch = 0; ch < NC; ++ch) x.q[ch] = ldq(s + ch * kPlane);
    }

    // One sub-step pair over the rows of radius r, in place.  LAST: the pair before the update,
    // which reads only the payload of a delta level, so its flow channels are not computed.
    // E: the slab has lanes at image edges or border columns, or rows of the border.
    // TAPE: X and Y results of the slab's own rows also go to the tape, as sub-steps 2k, 2k + 1.
    template <bool LAST, bool E, bool TAPE>
    __device__ __forceinline__ static void pass(const Ctx& c, float dt, int r, const Tape& tape, int k) {
        constexpr int FX = LAST && DELTA ? CV : 0, FY = LAST && DELTA ? 2 : 0;  // first channels of X and Y
        int y0, y1;
        c.run_of(r, y0, y1);
        const bool act = y0 < y1;
        const unsigned base = c.l16 - (unsigned)(c.sy0 * ROWB);
        // the rows before and after the run belong to other warps, which overwrite them: before
        // anyone writes, the row before is read and the row after copied to the warp's own
        // spare row (clamped at the image edges, where the row's own X result is the
        // neighbour's)
        const int yt = max(y0 - 1, 0), yb = min(y1, c.H - 1);
        const unsigned spare = c.spare + c.l16;
        Row w0, w1, w2;
        if (act) {
            load(base + yb * ROWB, w0);
#pragma unroll
            for (int ch = 0; ch < NC; ++ch) stq(spare + ch * kPlane, w0.q[ch]);
            load(base + yt * ROWB, w0);
        }
        __syncthreads();
        if (act) {
            auto inside = [&](int r) { return !E || (r >= c.border && r < c.H - c.border); };
            if (inside(yt)) xstep<E, FX>(c, dt, w0, w0);
            // X of row q + 1 (row `next` of the window), then Y of row q
            unsigned s = base + y0 * ROWB;  // row q + 1
            int q = y0 - 1;
            auto keep = [&](const Row& v, int y, int sub) {
                if (TAPE && y >= c.ys && y < c.ye && c.nout > 0) {
                    const size_t at = (size_t)sub * tape.step, n = (size_t)y * c.W + c.c0;
                    store_f2(c.vec, c.nout, reinterpret_cast<float2*>(tape.f + at) + n, v.q[0], v.q[1]);
                    if constexpr (DELTA) {
                        store_f1(c.vec, c.nout, tape.s + at + n, v.q[2]);
                        store_f2(c.vec, c.nout, reinterpret_cast<float2*>(tape.v + at) + n, v.q[3], v.q[4]);
                    }
                }
            };
            auto row = [&](const Row& prev, const Row& cur, Row& next) {
                const bool end = q + 1 == y1;
                load(end ? spare : s, next);
                if (inside(end ? yb : q + 1)) xstep<E, FX>(c, dt, next, next);
                if (!end) keep(next, q + 1, 2 * k);
                if (q >= y0) {
                    Row y;
                    if (inside(q)) ystep<E, FY>(c, dt, prev, cur, next, y);
                    else y = cur;
#pragma unroll
                    for (int ch = FY; ch < NC; ++ch) stq(s - ROWB + ch * kPlane, y.q[ch]);
                    keep(y, q, 2 * k + 1);
                }
                s += ROWB;
                return ++q == y1;
            };
            if constexpr (E) {
                // the longer body of edge slabs once, its window shifting: three copies of it
                // do not fit the instruction cache
                Row prev = w0, cur = w0;
#pragma unroll 1
                while (!row(prev, cur, w1)) {
                    prev = cur;
                    cur = w1;
                }
            } else {
                // three rows a turn, so the window rotates without moves
#pragma unroll 1
                for (;;) {
                    if (row(w2, w0, w1)) break;
                    if (row(w0, w1, w2)) break;
                    if (row(w1, w2, w0)) break;
                }
            }
        }
        __syncthreads();
    }
};

// offsets -2 .. +5 around the lane's four pixels
struct Ext {
    float2 l, m1, c0, m2, c1, m3, r;  // pairs (-2,-1) (-1,0) (0,1) (1,2) (2,3) (3,4) (4,5)
};
__device__ __forceinline__ Ext extend(const Q& v) {
    Ext e;
    e.l = make_float2(__shfl_up_sync(kFull, v.b.x, 1), __shfl_up_sync(kFull, v.b.y, 1));
    e.r = make_float2(__shfl_down_sync(kFull, v.a.x, 1), __shfl_down_sync(kFull, v.a.y, 1));
    e.c0 = v.a;
    e.c1 = v.b;
    e.m1 = make_float2(e.l.y, v.a.x);
    e.m2 = make_float2(v.a.y, v.b.x);
    e.m3 = make_float2(v.b.y, e.r.x);
    return e;
}
// clamp-to-edge columns of the extended pixels (lanes at an image edge)
__device__ __forceinline__ void clamp_ext(const Ctx& c, Ext& e) {
    if (c.e_l) e.l = make_float2(e.c0.x, e.c0.x);
    // columns after W - 1 read column W - 1; last = W - 1 - c0 (5 and up: none of these pixels)
    const int last = c.W - 1 - c.c0;
    if (last >= 0 && last < 5) {
        if (last < 1) e.c0.y = e.c0.x;
        if (last < 2) e.c1.x = e.c0.y;
        if (last < 3) e.c1.y = e.c1.x;
        if (last < 4) e.r.x = e.c1.y;
        e.r.y = e.r.x;
    }
    e.m1 = make_float2(e.l.y, e.c0.x);
    e.m2 = make_float2(e.c0.y, e.c1.x);
    e.m3 = make_float2(e.c1.y, e.r.x);
}
__device__ __forceinline__ Q smooth_x(const Ext& e) {
    return Q{smooth5_pair(e.l, e.m1, e.c0, e.m2, e.c1), smooth5_pair(e.c0, e.m2, e.c1, e.m3, e.r)};
}
__device__ __forceinline__ Q diff_x(const Ext& e) {
    return Q{diff5_pair(e.l, e.m1, e.c0, e.m2, e.c1), diff5_pair(e.c0, e.m2, e.c1, e.m3, e.r)};
}
__device__ __forceinline__ Q smooth_y(const Q& a, const Q& b, const Q& cc, const Q& d, const Q& e) {
    return Q{smooth5_pair(a.a, b.a, cc.a, d.a, e.a), smooth5_pair(a.b, b.b, cc.b, d.b, e.b)};
}
__device__ __forceinline__ Q diff_y(const Q& a, const Q& b, const Q& cc, const Q& d, const Q& e) {
    return Q{diff5_pair(a.a, b.a, cc.a, d.a, e.a), diff5_pair(a.b, b.b, cc.b, d.b, e.b)};
}

// ---------------------------------------------------------------- image model and update

// the lane's four pixels of an image row, clamped at the image edges
template <typename P>
struct Image;
template <>
struct Image<uint8_t> {
    const uint8_t* p;  // the lane's first column
    unsigned pitch, sel;
    int H;
    using Raw = uint32_t;
    __device__ __forceinline__ Image(const LevelArgs& a, const Ctx& c)
        : p(reinterpret_cast<const uint8_t*>(a.img) + c.wcol), pitch((unsigned)a.img_pitch), sel(0), H(c.H) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sel |= (unsigned)(min(max(c.c0 + j, 0), c.W - 1) - c.wcol) << (4 * j);
    }
    // the aligned word holding the columns (rows are 4-byte aligned and padded to words)
    __device__ __forceinline__ Raw raw(int y) const {
        return ld_waited(reinterpret_cast<const uint32_t*>(rowp(p, pitch, min(max(y, 0), H - 1))));
    }
    __device__ __forceinline__ Q unit(Raw w) const {
        w = __byte_perm(w, 0, sel);
        return Q{make_float2(u8_to_unit(w & 0xffu), u8_to_unit((w >> 8) & 0xffu)),
                 make_float2(u8_to_unit((w >> 16) & 0xffu), u8_to_unit(w >> 24))};
    }
};
template <>
struct Image<float> {
    const float* p;
    unsigned pitch;
    int H, o1, o2, o3;  // clamped columns of pixels 1..3 relative to p
    bool vec;
    using Raw = float4;
    __device__ __forceinline__ Image(const LevelArgs& a, const Ctx& c)
        : pitch((unsigned)a.img_pitch), H(c.H), vec(a.img_vec && !c.edge) {
        const int first = min(max(c.c0, 0), c.W - 1);
        p = reinterpret_cast<const float*>(a.img) + first;
        o1 = min(max(c.c0 + 1, 0), c.W - 1) - first;
        o2 = min(max(c.c0 + 2, 0), c.W - 1) - first;
        o3 = min(max(c.c0 + 3, 0), c.W - 1) - first;
    }
    __device__ __forceinline__ Raw raw(int y) const {
        const float* r = rowp(p, pitch, min(max(y, 0), H - 1));
        if (vec) return ld_waited(reinterpret_cast<const float4*>(r));
        return make_float4(ld_waited(r), ld_waited(r + o1), ld_waited(r + o2), ld_waited(r + o3));
    }
    __device__ __forceinline__ Q unit(const Raw& v) const {
        return Q{make_float2(v.x, v.y), make_float2(v.z, v.w)};
    }
};

template <bool DELTA, typename P>
struct Update {
    static constexpr unsigned ROWB = planes(DELTA) * kPlane;
    // solve2 (common.cuh) of a pixel pair; nothing but the reciprocal is per lane
    __device__ __forceinline__ static void solve_pair(float2 g, float2 ax, float2 ay, float2 yt, float2 fx, float2 fy,
                                                      float2& ox, float2& oy) {
        const float2 n00 = __ffma2_rn(ay, ay, g), n11 = __ffma2_rn(ax, ax, g);
        const float2 den = __fmul2_rn(g, __ffma2_rn(ay, ay, n11));
        const float2 n01 = __fmul2_rn(neg2(ax), ay);
        const float2 rdet = make_float2(__frcp_rn(den.x), __frcp_rn(den.y));
        const float2 qx = __ffma2_rn(g, fx, __fmul2_rn(ax, yt));
        const float2 qy = __ffma2_rn(ay, yt, __fmul2_rn(g, fy));
        ox = __fmul2_rn(__ffma2_rn(n00, qx, __fmul2_rn(n01, qy)), rdet);
        oy = __fmul2_rn(__ffma2_rn(n01, qx, __fmul2_rn(n11, qy)), rdet);
    }
    // deltaFlowUpdate_k's clamps and coarse flow (update_k.cu:136-164), one channel
    __device__ __forceinline__ static float2 clamp_delta(float2 o, float hm) {
        return make_float2(clampm(sanitize(o.x), hm), clampm(sanitize(o.y), hm));
    }
    __device__ __forceinline__ static float2 add_coarse(float2 d, float c0, float c1, float m) {
        return make_float2(clampm(__fadd_rn(d.x, __fmul_rn(2.0f, c0)), m),
                           clampm(__fadd_rn(d.y, __fmul_rn(2.0f, c1)), m));
    }
    __device__ __forceinline__ static float2 clamp_top(float2 o, float m) {
        return make_float2(sanitize(clampm(o.x, m)), sanitize(clampm(o.y, m)));
    }

    // rows of radius 2S: the model from the image (its vertical windows in registers down the
    // warp's run), the update from the propagated state; the new flow replaces planes U, V
    template <bool TAPE>
    __device__ __forceinline__ static void pass(const Ctx& c, const LevelArgs& a, int r2, const Tape& tape) {
        const int nout = c.nout;
        int y0, y1;
        c.run_of(r2, y0, y1);
        if (y0 < y1) {
            const Image<P> img(a, c);
            const float gamma = a.gamma_dev ? ld_waited(a.gamma_dev) : a.gamma;
            const float2 g = make_float2(gamma, gamma);
            const float m = a.maxflow, hm = __fmul_rn(0.5f, m);
            const bool first = a.first != 0, vec = c.vec;
            float* const io_out = a.io_out + c.c0;
            float2* const f_out = reinterpret_cast<float2*>(DELTA ? a.d_out : a.fu_out) + c.c0;
            const unsigned f_pitch = (unsigned)(DELTA ? a.d_out_pitch : a.fu_out_pitch);
            const bool f_store = DELTA || a.fu_out;
            // top levels read the old image in place
            int cc[4];
            unsigned cx[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int x = min(max(c.c0 + j, 0), c.W - 1);
                cc[j] = x;
                cx[j] = DELTA ? 8u * (unsigned)upmap_index(x, c.W, a.Wc) : 0u;
            }
            auto around = [&](const Q& v) {
                Ext e = extend(v);
                if (c.edge) clamp_ext(c, e);  // block-uniform
                return e;
            };
            Q im[4], bx[4];
            typename Image<P>::Raw nxt = img.raw(y0 + 2);
            // the coarse flow (delta levels) or old image (top levels) of a row, fetched a row
            // ahead; the coarse row two rows ahead
            float2 u0, u1, u2, u3;
            Q old_top;
            // the coarse row of a row, from the level's table where it has one
            auto coarse_row = [&](int y) {
                return a.coarse_rows ? __ldg(a.coarse_rows + y) : upmap_index(y, c.H, a.Hc);
            };
            int crow = DELTA ? coarse_row(y0) : 0;
            auto fetch = [&](int y) {
                if constexpr (DELTA) {
                    const char* row = rowp(reinterpret_cast<const char*>(a.coarse), (unsigned)a.coarse_pitch, crow);
                    crow = coarse_row(min(y + 1, c.H - 1));
                    u0 = ld_waited(reinterpret_cast<const float2*>(row + cx[0]));
                    u1 = ld_waited(reinterpret_cast<const float2*>(row + cx[1]));
                    u2 = ld_waited(reinterpret_cast<const float2*>(row + cx[2]));
                    u3 = ld_waited(reinterpret_cast<const float2*>(row + cx[3]));
                } else {
                    const float* row = rowp(a.io_in, (unsigned)a.io_in_pitch, min(y, c.H - 1));
                    if (a.vec) {
                        const float4 v = ld_waited(reinterpret_cast<const float4*>(row + c.wcol));
                        old_top = Q{make_float2(v.x, v.y), make_float2(v.z, v.w)};
                    } else {
                        old_top = Q{make_float2(ld_waited(row + cc[0]), ld_waited(row + cc[1])),
                                    make_float2(ld_waited(row + cc[2]), ld_waited(row + cc[3]))};
                    }
                }
            };
            fetch(y0);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                im[k] = img.unit(img.raw(y0 - 2 + k));
                bx[k] = smooth_x(around(im[k]));
            }
#pragma unroll 1
            for (int y = y0; y < y1; ++y) {
                const typename Image<P>::Raw now = nxt;
                nxt = img.raw(y + 3);
                const unsigned s = (unsigned)((y - c.sy0) * ROWB) + c.l16;
                const float2 c0 = u0, c1 = u1, c2 = u2, c3 = u3;
                Q old = DELTA ? ldq(s + 2 * kPlane) : old_top;
                fetch(y + 1);
                const Q fx = ldq(s + (DELTA ? 3 : 0) * kPlane), fy = ldq(s + (DELTA ? 4 : 1) * kPlane);
                // image model (imagemodel_k.cu:31-133)
                const Q i4 = img.unit(now);
                const Q b4 = smooth_x(around(i4));
                const Ext e = around(smooth_y(im[0], im[1], im[2], im[3], i4));
                const Q ay = diff_y(bx[0], bx[1], bx[2], bx[3], b4);
                const Q a0 = smooth_x(e), ax = diff_x(e);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    im[k] = im[k + 1];
                    bx[k] = bx[k + 1];
                }
                im[3] = i4;
                bx[3] = b4;
                if (first) old = a0;
                Q ox, oy, fu, fv;
                solve_pair(g, ax.a, ay.a, __fadd2_rn(old.a, neg2(a0.a)), fx.a, fy.a, ox.a, oy.a);
                solve_pair(g, ax.b, ay.b, __fadd2_rn(old.b, neg2(a0.b)), fx.b, fy.b, ox.b, oy.b);
                if constexpr (DELTA) {
                    ox = Q{clamp_delta(ox.a, hm), clamp_delta(ox.b, hm)};
                    oy = Q{clamp_delta(oy.a, hm), clamp_delta(oy.b, hm)};
                    fu = Q{add_coarse(ox.a, c0.x, c1.x, m), add_coarse(ox.b, c2.x, c3.x, m)};
                    fv = Q{add_coarse(oy.a, c0.y, c1.y, m), add_coarse(oy.b, c2.y, c3.y, m)};
                } else {
                    // flowUpdate_k (update_k.cu:65-78)
                    fu = ox = Q{clamp_top(ox.a, m), clamp_top(ox.b, m)};
                    fv = oy = Q{clamp_top(oy.a, m), clamp_top(oy.b, m)};
                }
                stq(s, fu);
                stq(s + kPlane, fv);
                if (y >= c.ys && y < c.ye && nout > 0) {
                    store_f1(vec, nout, rowp(io_out, (unsigned)a.io_out_pitch, y), a0);
                    if (f_store) store_f2(vec, nout, rowp(f_out, f_pitch, y), ox, oy);
                    if (TAPE) {
                        const size_t n = (size_t)y * c.W + c.c0;
                        store_f2(vec, nout, reinterpret_cast<float2*>(tape.grad) + n, ax, ay);
                        store_f2(vec, nout, reinterpret_cast<float2*>(tape.sm) + n, fu, fv);
                    }
                    if (!DELTA && a.d_out) {  // a state field that top levels pass on unchanged
                        const float2* d = rowp(reinterpret_cast<const float2*>(a.d_in), (unsigned)a.d_in_pitch, y) + c.c0;
                        float2* o = rowp(reinterpret_cast<float2*>(a.d_out), (unsigned)a.d_out_pitch, y) + c.c0;
                        for (int j = 0; j < nout; ++j) o[j] = ld_waited(d + j);
                    }
                }
            }
        }
        __syncthreads();
    }
};

// ---------------------------------------------------------------- smoothing
template <bool DELTA>
struct Smooth {
    static constexpr unsigned ROWB = planes(DELTA) * kPlane;
    struct W5 {
        float k[5];
    };
    __device__ __forceinline__ static float2 chain(const W5& w, float2 a, float2 b, float2 cc, float2 d, float2 e) {
        return chain5_pair(w.k[0], w.k[1], w.k[2], w.k[3], w.k[4], a, b, cc, d, e);
    }
    template <bool E>
    __device__ __forceinline__ static Q box_x(const Ctx& c, const W5& w, const Q& v) {
        Ext e = extend(v);
        if (E) clamp_ext(c, e);
        return Q{chain(w, e.l, e.m1, e.c0, e.m2, e.c1), chain(w, e.c0, e.m2, e.c1, e.m3, e.r)};
    }
    __device__ __forceinline__ static Q box_y(const W5& w, const Q& a, const Q& b, const Q& cc, const Q& d, const Q& e) {
        return Q{chain(w, a.a, b.a, cc.a, d.a, e.a), chain(w, a.b, b.b, cc.b, d.b, e.b)};
    }

    // X: planes U, V -> the next two, rows of radius r + 2
    // (pass j: the index of what it writes in the tape)
    template <bool E, bool TAPE>
    __device__ __forceinline__ static void pass_x(const Ctx& c, const W5& w, int r, const Tape& tape, int j) {
        int y0, y1;
        c.run_of(r + 2, y0, y1);
        unsigned s = (unsigned)((y0 - c.sy0) * ROWB) + c.l16;
#pragma unroll 2
        for (int y = y0; y < y1; ++y, s += ROWB) {
            const Q u = box_x<E>(c, w, ldq(s)), v = box_x<E>(c, w, ldq(s + kPlane));
            stq(s + 2 * kPlane, u);
            stq(s + 3 * kPlane, v);
            if (TAPE && y >= c.ys && y < c.ye && c.nout > 0)
                store_f2(c.vec, c.nout, reinterpret_cast<float2*>(tape.sm + j * tape.sm_step) + (size_t)y * c.W + c.c0, u, v);
        }
        __syncthreads();
    }
    // Y: back to planes U, V, or (LAST) to the smoothed flow, rows of radius r
    template <bool LAST, bool TAPE>
    __device__ __forceinline__ static void pass_y(const Ctx& c, const LevelArgs& a, const W5& w, int r, const Tape& tape,
                                                  int j) {
        int y0, y1;
        c.run_of(r, y0, y1);
        const bool vec = c.vec;
        const int nout = c.nout;
        float2* const fs_out = reinterpret_cast<float2*>(a.fs_out) + c.c0;
        float2* const y_out = a.y_out ? reinterpret_cast<float2*>(a.y_out) + c.c0 : nullptr;
        const unsigned base = 2 * kPlane + c.l16 - (unsigned)(c.sy0 * ROWB);
        auto src = [&](int y) { return base + (unsigned)(min(max(y, 0), c.H - 1) * ROWB); };
        if (y0 < y1) {
            Q u[4], v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned s = src(y0 - 2 + k);
                u[k] = ldq(s);
                v[k] = ldq(s + kPlane);
            }
            auto row = [&](int y, Q& u0, Q& u1, Q& u2, Q& u3, Q& v0, Q& v1, Q& v2, Q& v3) {
                const unsigned s = src(y + 2);
                const Q u4 = ldq(s), v4 = ldq(s + kPlane);
                const Q ou = box_y(w, u0, u1, u2, u3, u4), ov = box_y(w, v0, v1, v2, v3, v4);
                u0 = u4;  // the newest row replaces the oldest
                v0 = v4;
                if (LAST) {
                    if (nout > 0) {
                        store_f2(vec, nout, rowp(fs_out, (unsigned)a.fs_out_pitch, y), ou, ov);
                        if (y_out) store_f2(vec, nout, rowp(y_out, (unsigned)a.fs_out_pitch, y), ou, ov);
                    }
                } else {
                    const unsigned o = base - 2 * kPlane + (unsigned)(y * ROWB);
                    stq(o, ou);
                    stq(o + kPlane, ov);
                    if (TAPE && y >= c.ys && y < c.ye && nout > 0)
                        store_f2(vec, nout, reinterpret_cast<float2*>(tape.sm + j * tape.sm_step) + (size_t)y * c.W + c.c0,
                                 ou, ov);
                }
            };
            // four rows a turn, so the window rotates without moves
#pragma unroll 1
            for (int y = y0; y < y1;) {
                row(y, u[0], u[1], u[2], u[3], v[0], v[1], v[2], v[3]);
                if (++y == y1) break;
                row(y, u[1], u[2], u[3], u[0], v[1], v[2], v[3], v[0]);
                if (++y == y1) break;
                row(y, u[2], u[3], u[0], u[1], v[2], v[3], v[0], v[1]);
                if (++y == y1) break;
                row(y, u[3], u[0], u[1], u[2], v[3], v[0], v[1], v[2]);
                ++y;
            }
        }
        if (!LAST) __syncthreads();
    }
};

// ---------------------------------------------------------------- one slab
// geometry of slab i: lanes, rows, and which edge handling it needs; sy1 = end of its rows in
// shared memory
template <bool DELTA>
__device__ __forceinline__ void make_ctx(const LevelArgs& a, const Geom& g, int i, Ctx& c, int& sy1) {
    constexpr int ROWB = planes(DELTA) * kPlane;
    const int N = g.N, S = g.S;
    c.W = a.W;
    c.H = a.H;
    c.border = a.border;
    c.lane = threadIdx.x & 31;
    c.warp = __shfl_sync(kFull, (int)(threadIdx.x >> 5), 0);
    c.l16 = 16 * c.lane;
    int wx, ys, rows;
    g.at(i, wx, ys, rows);
    // window wx starts at column x0; its outer HX columns belong to its neighbours, if it has any
    const int HX = halo_x(N, S), x0 = wx * slab_cols(N, S);
    const int xo = wx == 0 ? 0 : x0 + HX, xe = wx == g.nwx - 1 ? a.W : x0 + kCols - HX;
    c.c0 = x0 + 4 * c.lane;
    c.wcol = min(max(c.c0, 0), (c.W - 1) & ~3);
    c.ys = ys;
    c.ye = min(ys + rows, a.H);
    c.e_l = c.c0 == 0;
    c.e_r = c.c0 + 3 == a.W - 1;
    const int last = a.W - 1 - c.c0;
    c.rag = last >= 0 && last < 3 ? last : -1;
    c.cin = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) c.cin |= (c.c0 + j >= a.border && c.c0 + j < a.W - a.border) << j;
    c.edge = x0 <= 0 || x0 + kCols >= a.W || x0 < a.border || x0 + kCols > a.W - a.border;
    c.nout = c.c0 >= xo && c.c0 < xe ? min(4, a.W - c.c0) : 0;
    c.vec = c.nout == 4 && a.vec;
    const int R = N + 2 * S;
    c.sy0 = max(0, ys - R);
    sy1 = min(a.H, c.ye + R);
    c.spare = (unsigned)((sy1 - c.sy0 + c.warp) * ROWB);
    c.rows_edge = c.edge || c.sy0 < a.border || sy1 > a.H - a.border;

}

// the previous frame's state of the slab's rows into the planes, all rows in flight at once
// (the filters' own rows are always aligned, so a load that runs before grid_dep_wait() comes from
// L2, where the writes of completed kernels are)
template <bool DELTA>
__device__ __forceinline__ void load_state(const LevelArgs& a, const Ctx& c, int sy1) {
    constexpr int ROWB = planes(DELTA) * kPlane;
    {
        const char* fs = reinterpret_cast<const char*>(a.fs_in) + 8 * (size_t)c.wcol;
        const char* d = reinterpret_cast<const char*>(a.d_in) + 8 * (size_t)c.wcol;
        const char* io = reinterpret_cast<const char*>(a.io_in) + 4 * (size_t)c.wcol;
        const unsigned sm = (unsigned)__cvta_generic_to_shared(slab_smem_) + c.l16;
        if (a.vec) {
#pragma unroll 2
            for (int y = c.sy0 + c.warp; y < sy1; y += kWarps) {
                const unsigned s = sm + (unsigned)((y - c.sy0) * ROWB);
                const char* pf = rowp(fs, (unsigned)a.fs_in_pitch, y);
                cp16(s, pf);
                cp16(s + kPlane, pf + 16);
                if constexpr (DELTA) {
                    const char* pd = rowp(d, (unsigned)a.d_in_pitch, y);
                    cp16(s + 2 * kPlane, rowp(io, (unsigned)a.io_in_pitch, y));
                    cp16(s + 3 * kPlane, pd);
                    cp16(s + 4 * kPlane, pd + 16);
                }
            }
        } else {  // rows without 16-byte alignment: pixel by pixel, at clamped columns
            int o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = min(max(c.c0 + j, 0), c.W - 1) - c.wcol;
#pragma unroll 1
            for (int y = c.sy0 + c.warp; y < sy1; y += kWarps) {
                const unsigned s = sm + (unsigned)((y - c.sy0) * ROWB);
                const char* pf = rowp(fs, (unsigned)a.fs_in_pitch, y);
#pragma unroll
                for (int j = 0; j < 4; ++j) cp8(s + (j >> 1) * kPlane + 8 * (j & 1), pf + 8 * o[j]);
                if constexpr (DELTA) {
                    const char* pd = rowp(d, (unsigned)a.d_in_pitch, y);
                    const char* pi = rowp(io, (unsigned)a.io_in_pitch, y);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        cp8(s + (3 + (j >> 1)) * kPlane + 8 * (j & 1), pd + 8 * o[j]);
                        cp4(s + 2 * kPlane + 4 * j, pi + 4 * o[j]);
                    }
                }
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        // pixel pairs (u, v) to planes, each lane its own pixels
#pragma unroll 1
        for (int y = c.sy0 + c.warp; y < sy1; y += kWarps) {
            const unsigned s = (unsigned)((y - c.sy0) * ROWB) + c.l16;
#pragma unroll
            for (int ch = 0; ch < (DELTA ? 6 : 3); ch += 3) {
                const Q p = ldq(s + ch * kPlane), q = ldq(s + (ch + 1) * kPlane);
                stq(s + ch * kPlane, Q{make_float2(p.a.x, p.b.x), make_float2(q.a.x, q.b.x)});
                stq(s + (ch + 1) * kPlane, Q{make_float2(p.a.y, p.b.y), make_float2(q.a.y, q.b.y)});
            }
        }
    }
    __syncthreads();
}

// N sub-step pairs, dt = 1/N (FlowPropagator::setIterations, propagation.cu:146-147), from rows of
// radius R.  FULL: every channel of the last pair too (the update reads only the payload of a
// delta level).
template <bool DELTA, bool TAPE, bool FULL = TAPE>
__device__ __forceinline__ void propagate(const Ctx& c, int N, int R, const Tape& tape) {
    const float dt = 1.0f / (float)N;
#pragma unroll 1
    for (int k = 1; k < N + (FULL ? 1 : 0); ++k) {
        if (c.rows_edge) Prop<DELTA>::template pass<false, true, TAPE>(c, dt, R - k, tape, k - 1);
        else Prop<DELTA>::template pass<false, false, TAPE>(c, dt, R - k, tape, k - 1);
    }
    if (!FULL) {
        if (c.rows_edge) Prop<DELTA>::template pass<true, true, false>(c, dt, R - N, tape, N - 1);
        else Prop<DELTA>::template pass<true, false, false>(c, dt, R - N, tape, N - 1);
    }
}

// S smoothing iterations of planes U, V; the last stores the smoothed flow
template <bool DELTA, bool TAPE>
__device__ __forceinline__ void smooth(const Ctx& c, const LevelArgs& a, int S, const Tape& tape) {
    typename Smooth<DELTA>::W5 w;
#pragma unroll
    for (int j = 0; j < 5; ++j) w.k[j] = a.weights ? ld_waited(a.weights + j) : kBox;
#pragma unroll 1
    for (int s = 1; s <= S; ++s) {
        const int r = 2 * (S - s);
        if (c.edge) Smooth<DELTA>::template pass_x<true, TAPE>(c, w, r, tape, 2 * s - 1);
        else Smooth<DELTA>::template pass_x<false, TAPE>(c, w, r, tape, 2 * s - 1);
        if (s < S) Smooth<DELTA>::template pass_y<false, TAPE>(c, a, w, r, tape, 2 * s);
        else Smooth<DELTA>::template pass_y<true, TAPE>(c, a, w, r, tape, 2 * s);
    }
}

// slab i of the level step (a, g), by the whole block
template <bool DELTA, typename P, bool TAPE = false>
__device__ __forceinline__ void level_slab(const LevelArgs& a, const Geom& g, int i, const Tape& tape = Tape{}) {
    // ordering with the preceding kernel: see LevelArgs::pdl_late_wait (everything before the
    // update reads only the previous frame's state and an image that was complete before)
    if (!a.pdl_late_wait) grid_dep_wait();
    if (a.pdl_early_trigger) grid_dep_launch();
    const int N = g.N, S = g.S;
    Ctx c;
    int sy1;
    make_ctx<DELTA>(a, g, i, c, sy1);
    const int R = N + 2 * S;
    load_state<DELTA>(a, c, sy1);

    propagate<DELTA, TAPE>(c, N, R, tape);

    // ---- image model and update
    if (a.pdl_late_wait) grid_dep_wait();
    Update<DELTA, P>::template pass<TAPE>(c, a, 2 * S, tape);
    // the next kernel in the stream may start scheduling its blocks from here on
    if (!a.pdl_early_trigger) grid_dep_launch();

    smooth<DELTA, TAPE>(c, a, S, tape);
}

}  // namespace slab
}  // namespace ffb
