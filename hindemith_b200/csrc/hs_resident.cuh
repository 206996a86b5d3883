// hs_resident.cuh -- the resident form of the Horn-Schunck sweeps: the whole image lives on
// the chip for all sweeps of a call, one tile per CTA and one CTA per SM, in a cooperative
// launch.
//
// The streaming kernels (hs_stream.cuh, hs_stream4.cuh) read and write every plane once per
// pass of T sweeps, and near L2-resident sizes they spend about half of their instructions on
// the temporal halo, the rings and the copies.  An image of up to about 2 Mpx fits the 148 SMs:
//   - the state (u, v) of a tile of 128 columns x (NW * R) rows sits in registers, R rows of 4
//     adjacent columns per lane (a warp owns R whole rows of the tile);
//   - the four coefficients of each pixel (Ix, Iy, It and the negated denominator term) sit in
//     tensor memory: 16 words per lane and row, 512 columns x 128 lanes for the largest tile.
//     Every warp reads back only what it wrote; tcgen05.ld delivers about 900 B per clock and
//     SM, where shared memory, which the shuffles also use, delivers 128;
//   - within a sweep, horizontal neighbours come from warp shuffles, vertical ones from the
//     lane's own rows; a warp publishes its first and last row's contribution to its two
//     neighbour warps through shared memory (one block barrier per sweep);
//   - every kResT sweeps the CTAs exchange a ring of kResT pixels around their tiles through
//     global memory (L2); between exchanges a tile runs kResT sweeps on its own, the valid
//     region shrinking into the kResT-pixel halo.
// Every cell sees the operations of the streaming kernels in their order, so the results are
// the same bit for bit, in both forms.
//
// Image sides.  The lane at column 0 and the lane at column W-1 substitute their own value for
// the missing neighbour (two selects per row and plane, in the tiles at a side only).  Row -1
// and row H are kept equal to rows 0 and H-1 (copied after every sweep), so no row of the sweep
// itself is special.
//
// Exchange.  The warps put their ring into shared memory, then all threads of the CTA send and
// receive it together, three messages each, and the halo goes back through shared memory: one
// round trip to L2 per exchange.  (Each warp receiving its own halo took a round trip per
// message in the warps that hold halo rows: 14000 clocks per exchange at 1080p.)  A message is
// 16 bytes, three state values and the exchange's number, stored and loaded as one 128-bit
// access: a reader polls the message itself until it carries the number it waits for, so no
// flag and no fence stands between the store and the load.  Exchange e = 1, 2, ... uses half
// e % 2 of a tile's outbox.  A tile writes a half again at e + 2, after it has received e + 1
// from all its neighbours, which they sent after a block barrier behind their reads of e.  The
// outboxes are cleared before the launch (numbers start at 1).  Every wait is bounded
// (hs_resident.cu).
#pragma once

#include "hs_stream.cuh"
#include "hs_tmem.cuh"

namespace hs {

constexpr int kResT = 4;                      // sweeps between exchanges = halo pixels
constexpr int kResCols = 128;                 // columns of a tile, halo included (4 per lane)
constexpr int kResChunks = kResCols / 4 - 2;  // 4-column chunks of a tile's own region, at most

constexpr int kMaxResImages = 32;  // images of one launch

// What a launch's waits share.
struct ResWait {
    unsigned *abort_flag;  // raised by a wait that ran out
    int *status;           // if set: HS_ERR_TIMEOUT goes here then
    int polls;             // of one message, at most
};

// Set to HS_ERR_TIMEOUT, too, when a wait of any launch runs out, until hs_wait_status reads it.  (One
// word per translation unit: a device pointer to a single one would take host work in every call.)
static __device__ int g_wait_status;

// *out: the word, which is cleared, or what is there already if it is set.
static __global__ void wait_status_kernel(int *out, int first) {
    const int word = atomicExch(&g_wait_status, 0);
    if (first || word) *out = word;
}

struct ResImage {
    const float *I0, *I1;        // if set: the images; the kernel forms the derivatives itself
    float *Ix, *Iy, *It;         // else the derivative planes; with the images: where to keep them, or null
    float *u, *v;                // state: read at the start (unless zero_start), written at the end
    float *ckpt;                 // if set: checkpoint c, the state after c * ckpt_every sweeps and at
                                 // the end, goes to plane 2c (u) and 2c + 1 (v) from here
    float4 *box;                 // outboxes of the image's tiles
    const float *alpha_dev;      // if set, alpha2 = alpha_dev[0] squared
    float alpha2;
    int H, W, ld;
    int ntx, nty;                // tiles across and down
    int iters, nblocks;          // the sweeps run in nblocks blocks of at most kResT
};

struct ResidentTable {
    ResImage img[kMaxResImages];
    int first[kMaxResImages + 1];  // tiles of the images before image i
    int n;
    ResWait wait;
    size_t ckpt_plane;           // floats between checkpoint planes
    int ckpt_every;
    float we, wc;
    int zero_start;
};

// The chunks (4 pixels of u and of v, 8 floats) a tile sends and receives in one exchange:
//   row blocks    [up, down][kResT rows][32 lanes]  sent: its first / last kResT own rows;
//                                                   received: the rows above / below them
//   column blocks [left, right][rows of the tile]   its first / last own chunk of every row;
//                                                   the chunks beside them
// A chunk is three messages: message m holds floats 3m .. 3m+2 and the exchange's number.
constexpr int kResRowChunks = kResT * 32;
__host__ __device__ constexpr int res_chunks(int rows) { return 2 * kResRowChunks + 2 * rows; }
__host__ __device__ constexpr int res_msgs(int rows) { return 3 * res_chunks(rows); }

// first pixel row of tile row j of n over H rows; first 4-column chunk likewise
__host__ __device__ inline int res_split(int j, int n, int total) {
    return (int)((long long)j * total / n);
}

__device__ __forceinline__ float2 lo2(float4 a) { return make_float2(a.x, a.y); }
__device__ __forceinline__ float2 hi2(float4 a) { return make_float2(a.z, a.w); }
__device__ __forceinline__ float4 cat4(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }

// Per-lane constants of a tile.
struct ResLane {
    int lane, warp;
    bool first, last;  // the lane holds column 0 / column W-1
    int row0;          // image row of the warp's first row
    int H;
    unsigned tmem;     // the warp's tensor memory
};

// Left and right neighbours of a lane's 4 columns (E, O) = ((c0, c1), (c2, c3)) across the
// warp.  SIDE: -1 = no image side in the tile; else the lane column (0..3) that W-1 falls on.
template <int SIDE>
__device__ __forceinline__ void res_neighbours(const ResLane &t, float2 E, float2 O, float2 &lE, float2 &rE,
                                               float2 &lO, float2 &rO) {
    const float lsh = __shfl_up_sync(kFull, O.y, 1);
    const float rsh = __shfl_down_sync(kFull, E.x, 1);
    float L0 = lsh, R0 = E.y, R1 = O.x, R2 = O.y, R3 = rsh;
    if constexpr (SIDE >= 0) L0 = t.first ? E.x : L0;
    if constexpr (SIDE == 0) R0 = t.last ? E.x : R0;
    if constexpr (SIDE == 1) R1 = t.last ? E.y : R1;
    if constexpr (SIDE == 2) R2 = t.last ? O.x : R2;
    if constexpr (SIDE == 3) R3 = t.last ? O.y : R3;
    lE = make_float2(L0, E.x);
    rE = make_float2(R0, R1);
    lO = make_float2(E.y, O.x);
    rO = make_float2(R2, R3);
}

// What a row contributes to the rows around it, for one plane and column pair.
//   fast : h = left + right and Y = we c + wc h (the row's term as an upper or lower row)
//   exact: the five products of the taps and the running sum `up` of the three upper taps
template <bool FAST>
struct RowTerm;
template <>
struct RowTerm<true> {
    float2 h, Y;
};
template <>
struct RowTerm<false> {
    float2 tl, tc, tr, ml, mr, up;
};

template <int SIDE>
__device__ __forceinline__ void row_terms(const ResLane &t, float2 E, float2 O, float2 we, float2 wc,
                                          RowTerm<true> (&o)[2]) {
    float2 lE, rE, lO, rO;
    res_neighbours<SIDE>(t, E, O, lE, rE, lO, rO);
    o[0].h = make_float2(__fadd_rn(lE.x, rE.x), __fadd_rn(lE.y, rE.y));
    o[1].h = make_float2(__fadd_rn(lO.x, rO.x), __fadd_rn(lO.y, rO.y));
    o[0].Y = fma2(we, E, mul2(wc, o[0].h));
    o[1].Y = fma2(we, O, mul2(wc, o[1].h));
}
template <int SIDE>
__device__ __forceinline__ void row_terms(const ResLane &t, float2 E, float2 O, float2 we, float2 wc,
                                          RowTerm<false> (&o)[2]) {
    float2 l[2], r[2];
    res_neighbours<SIDE>(t, E, O, l[0], r[0], l[1], r[1]);
    const float2 c[2] = {E, O};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        o[j].tl = mul2r(wc, l[j]);
        o[j].tc = mul2r(we, c[j]);
        o[j].tr = mul2r(wc, r[j]);
        o[j].ml = mul2r(we, l[j]);
        o[j].mr = mul2r(we, r[j]);
        o[j].up = add2(add2(add2(f2(0.f, 0.f), o[j].tl), o[j].tc), o[j].tr);
    }
}

// Jacobi update of a column pair from its averages; (cx, cy, ct, nd) as in the streaming
// kernels: nd = -1/den (fast) or -den (exact).
template <bool FAST>
__device__ __forceinline__ void res_update(float2 ubar, float2 vbar, float2 cx, float2 cy, float2 ct, float2 nd,
                                           float2 &u, float2 &v) {
    if constexpr (FAST) {
        const float2 nt = mul2(fma2(cx, ubar, fma2(cy, vbar, ct)), nd);
        u = fma2(cx, nt, ubar);
        v = fma2(cy, nt, vbar);
    } else {
        const float2 r = add2(add2(mul2r(cx, ubar), mul2r(cy, vbar)), ct);
        const float2 nt = f2(__fdiv_rn(r.x, nd.x), __fdiv_rn(r.y, nd.y));
        u = add2(ubar, mul2r(cx, nt));
        v = add2(vbar, mul2r(cy, nt));
    }
}

// The block barrier of a sweep.  Warps reach it from different variants of res_sweep (image
// sides and edges), so it is the named-barrier instruction itself: it counts warps, not places.
__device__ __forceinline__ void res_barrier() { asm volatile("bar.sync 0;" ::: "memory"); }

// One sweep of the warp's R rows.  pub: this sweep's half of the publication buffer,
// [NW][4][32] float4 (first row's u, v terms, last row's u, v terms).
//   fast : the first and the last row's Y
//   exact: the first row itself (its three lower taps are added one by one) and the last
//          row's `up`
// UPDATE = false: only the average, A (the adjoint's use).
template <bool FAST, int NW, int R, int SIDE, bool UPDATE = true>
__device__ __forceinline__ void res_sweep(const ResLane &t, float2 (&cu)[R][2][2], float4 *pub, float wef,
                                          float wcf) {
    const float2 we = f2(wef, wef), wc = f2(wcf, wcf);
    RowTerm<FAST> cur[2][2];  // [plane][pair]: terms of the row being finished
    RowTerm<FAST> lst[2][2];  // of the last row
    float4 *mine = pub + t.warp * 128 + t.lane;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        row_terms<SIDE>(t, cu[0][q][0], cu[0][q][1], we, wc, cur[q]);
        if constexpr (R > 1) row_terms<SIDE>(t, cu[R - 1][q][0], cu[R - 1][q][1], we, wc, lst[q]);
        else { lst[q][0] = cur[q][0]; lst[q][1] = cur[q][1]; }
        if constexpr (FAST) {
            mine[32 * q] = cat4(cur[q][0].Y, cur[q][1].Y);
            mine[64 + 32 * q] = cat4(lst[q][0].Y, lst[q][1].Y);
        } else {
            mine[32 * q] = cat4(cu[0][q][0], cu[0][q][1]);
            mine[64 + 32 * q] = cat4(lst[q][0].up, lst[q][1].up);
        }
    }
    res_barrier();
    // the tile's outermost rows have no neighbour warp: any value, they are halo (or outside)
    const float4 *above = pub + max(t.warp - 1, 0) * 128 + 64 + t.lane;
    const float4 *below = pub + min(t.warp + 1, NW - 1) * 128 + t.lane;
    // row 0 as the warp's first row has itself above it, row H-1 as its last row itself below
    const bool top = t.row0 == 0, bottom = t.row0 + R == t.H;

    float2 acc[2][2];  // fast: Z = Y(r-1) + we h(r); exact: upper and middle taps of row r
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float4 a4 = above[32 * q];
        const float2 a[2] = {lo2(a4), hi2(a4)};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if constexpr (FAST) {
                const float2 up = top ? cur[q][j].Y : a[j];
                acc[q][j] = fma2(we, cur[q][j].h, up);
            } else {
                const float2 up = top ? cur[q][j].up : a[j];
                acc[q][j] = add2(add2(up, cur[q][j].ml), cur[q][j].mr);
            }
        }
    }
    float co[16];
    if constexpr (UPDATE) tmem_ld16(co, t.tmem);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        // terms of row r + 1
        RowTerm<FAST> nxt[2][2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (r + 1 < R - 1) {
                row_terms<SIDE>(t, cu[r + 1 < R ? r + 1 : 0][q][0], cu[r + 1 < R ? r + 1 : 0][q][1], we, wc, nxt[q]);
            } else if (r + 1 == R - 1) {
                nxt[q][0] = lst[q][0];
                nxt[q][1] = lst[q][1];
            } else {  // the row below the warp's last row
                const float4 b4 = below[32 * q];
                if constexpr (FAST) {
                    nxt[q][0].Y = bottom ? cur[q][0].Y : lo2(b4);
                    nxt[q][1].Y = bottom ? cur[q][1].Y : hi2(b4);
                } else {
                    const float2 b0 = bottom ? cu[r][q][0] : lo2(b4), b1 = bottom ? cu[r][q][1] : hi2(b4);
                    row_terms<SIDE>(t, b0, b1, we, wc, nxt[q]);
                }
            }
        }
        float2 avg[2][2];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if constexpr (FAST) {
                    avg[q][j] = add2(acc[q][j], nxt[q][j].Y);
                    if (r + 1 < R) acc[q][j] = fma2(we, nxt[q][j].h, cur[q][j].Y);
                } else {
                    avg[q][j] = add2(add2(add2(acc[q][j], nxt[q][j].tl), nxt[q][j].tc), nxt[q][j].tr);
                    if (r + 1 < R) acc[q][j] = add2(add2(cur[q][j].up, nxt[q][j].ml), nxt[q][j].mr);
                }
            }
        if constexpr (UPDATE) {
            tmem_wait_ld(co);
            float cn[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) cn[i] = co[i];
            if (r + 1 < R) tmem_ld16(co, t.tmem + 16 * (r + 1));
#pragma unroll
            for (int j = 0; j < 2; ++j)
                res_update<FAST>(avg[0][j], avg[1][j], f2(cn[2 * j], cn[2 * j + 1]), f2(cn[4 + 2 * j], cn[5 + 2 * j]),
                                 f2(cn[8 + 2 * j], cn[9 + 2 * j]), f2(cn[12 + 2 * j], cn[13 + 2 * j]), cu[r][0][j],
                                 cu[r][1][j]);
        } else {
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int j = 0; j < 2; ++j) cu[r][q][j] = avg[q][j];
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j) cur[q][j] = nxt[q][j];
    }
}

// The ghost rows: row -1 follows row 0 and row H row H-1, where both lie in this warp.  (Row 0
// as a warp's first row and row H-1 as its last one are handled in the sweep.)
template <int R>
__device__ __forceinline__ void res_ghost_rows(const ResLane &t, float2 (&cu)[R][2][2]) {
#pragma unroll
    for (int r = 0; r + 1 < R; ++r) {
        if (t.row0 + r == -1) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                cu[r][q][0] = cu[r + 1][q][0];
                cu[r][q][1] = cu[r + 1][q][1];
            }
        }
        if (t.row0 + r == t.H - 1) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                cu[r + 1][q][0] = cu[r][q][0];
                cu[r + 1][q][1] = cu[r][q][1];
            }
        }
    }
}

// n sweeps of the warp's rows; pub: both halves of the publication buffer, `half` the one to use.
// (The loop is inside the variant: its state registers need not agree with another variant's
// after every sweep.)
template <bool FAST, int NW, int R, int SIDE, bool UPDATE = true>
__device__ __forceinline__ void res_sweeps(const ResLane &t, float2 (&cu)[R][2][2], float4 *pub, int half, int n,
                                           bool ghosts, float wef, float wcf) {
#pragma unroll 1
    for (int i = 0; i < n; ++i, half ^= 1) {
        if (ghosts) res_ghost_rows<R>(t, cu);
        res_sweep<FAST, NW, R, SIDE, UPDATE>(t, cu, pub + half * (NW * 128), wef, wcf);
    }
}

// The lane's 4 columns of a row, the first n of them when the image ends inside the chunk
// (columns past W may belong to other data of the caller).
__device__ __forceinline__ void res_store(float *U, float *V, size_t off, int n, const float2 (&c)[2][2]) {
    if (n >= 4) {
        *reinterpret_cast<float4 *>(U + off) = cat4(c[0][0], c[0][1]);
        *reinterpret_cast<float4 *>(V + off) = cat4(c[1][0], c[1][1]);
    } else {
        const float a[3] = {c[0][0].x, c[0][0].y, c[0][1].x}, b[3] = {c[1][0].x, c[1][0].y, c[1][1].x};
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (j < n) {
                U[off + j] = a[j];
                V[off + j] = b[j];
            }
    }
}

// A row's coefficients into tensor memory: c holds Ix, Iy, It of the lane's 4 columns, the
// negated denominator term joins them.
template <bool FAST>
__device__ __forceinline__ void res_coefficients(unsigned tmem, float (&c)[16], float alpha2, bool in) {
    // cells outside the image: never used, but the exact form's division should see ordinary
    // numbers (a zero numerator takes the division's slow branch for the whole warp)
    if (!in) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            c[j] = c[4 + j] = 0.f;
            c[8 + j] = 1.f;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if constexpr (FAST) {
            c[12 + j] = -rcp_approx(fmaf(c[4 + j], c[4 + j], fmaf(c[j], c[j], alpha2)));
        } else {
            c[12 + j] = -__fadd_rn(__fadd_rn(alpha2, __fmul_rn(c[j], c[j])), __fmul_rn(c[4 + j], c[4 + j]));
        }
    }
    tmem_st16(tmem, c);
}

// columns a CTA of NW warps x R rows allocates
template <int NW, int R>
constexpr int res_tmem_cols() {
    constexpr int words = (NW / 4) * R * 16;
    static_assert(NW % 4 == 0 && words <= 512, "the coefficients of a tile fit tensor memory");
    return words <= 32 ? 32 : words <= 64 ? 64 : words <= 128 ? 128 : words <= 256 ? 256 : 512;
}

// A wait (of kResPolls polls, hs_stream.cuh) can only run out if a neighbour's CTA has stopped: the
// CTAs of a cooperative launch are resident together, and start together (measured on B200: with
// another kernel on five SMs none of 148 CTAs started before the five were free, then all within a
// microsecond).  The tile then raises the abort flag, sets the status words and stops waiting, and
// the tiles that see the flag write NaN as their result.

// One 128-bit access of a message (single-copy atomic).
__device__ __forceinline__ void msg_store(float4 *p, float a, float b, float c, unsigned e) {
    asm volatile(
        "{\n\t.reg .b128 q;\n\t.reg .b64 lo, hi;\n\t"
        "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 q, {lo, hi};\n\t"
        "st.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p), "f"(a), "f"(b), "f"(c), "r"(e)
        : "memory");
}
__device__ __forceinline__ void msg_load(const float4 *p, float (&f)[3], unsigned &e) {
    asm volatile(
        "{\n\t.reg .b128 q;\n\t.reg .b64 lo, hi;\n\t"
        "ld.relaxed.gpu.global.b128 q, [%4];\n\tmov.b128 {lo, hi}, q;\n\t"
        "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=r"(e)
        : "l"(p)
        : "memory");
}

// A chunk (8 floats, 16-byte aligned) to and from the lane's columns of a row.
__device__ __forceinline__ void put_chunk(float *s, const float2 (&c)[2][2]) {
    reinterpret_cast<float4 *>(s)[0] = cat4(c[0][0], c[0][1]);
    reinterpret_cast<float4 *>(s)[1] = cat4(c[1][0], c[1][1]);
}
__device__ __forceinline__ void get_chunk(const float *s, float2 (&c)[2][2]) {
    const float4 u = reinterpret_cast<const float4 *>(s)[0], v = reinterpret_cast<const float4 *>(s)[1];
    c[0][0] = lo2(u);
    c[0][1] = hi2(u);
    c[1][0] = lo2(v);
    c[1][1] = hi2(v);
}

// Shared memory of a CTA: the sweeps' publications, the chunks sent, the chunks received and,
// for every message received, where it comes from.
template <int NW, int R>
struct ResSmem {
    static constexpr int chunks = res_chunks(NW * R), msgs = res_msgs(NW * R);
    static constexpr int out = 2 * NW * 128 * 16;        // bytes
    static constexpr int in = out + chunks * 32 + 16;    // (a chunk's third message reads 1 float past it)
    static constexpr int src = in + chunks * 32 + 16;
    static constexpr int bytes = src + msgs * 4;
};

// A CTA's tile of its image, seen from one lane.
struct ResTile {
    int tile, tx, ty, ntx, nty;
    int H, W, ld;
    int y0, y1;            // its own rows
    int own;               // lanes 1 .. own hold its own columns
    int xa;                // the lane's first column (a multiple of 4)
    bool nl, nr, nu, nd;   // neighbours
    bool own_col, col_in;  // the lane's columns are the tile's own / start inside the image
    int side;              // res_neighbours' SIDE
    bool ghosts;           // the warp holds a ghost row
};

template <int R>
__device__ __forceinline__ void res_tile(ResTile &g, ResLane &t, int tile, int ntx, int nty, int H, int W, int ld,
                                         unsigned tmem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    g.tile = tile;
    g.ntx = ntx;
    g.nty = nty;
    g.tx = tile % ntx;
    g.ty = tile / ntx;
    g.H = H;
    g.W = W;
    g.ld = ld;
    const int chunks = (W + 3) / 4;
    const int x0 = 4 * res_split(g.tx, ntx, chunks), x1 = 4 * res_split(g.tx + 1, ntx, chunks);
    g.y0 = res_split(g.ty, nty, H);
    g.y1 = res_split(g.ty + 1, nty, H);
    g.own = (x1 - x0) / 4;
    g.xa = x0 - 4 + 4 * lane;
    g.nl = g.tx > 0;
    g.nr = g.tx + 1 < ntx;
    g.nu = g.ty > 0;
    g.nd = g.ty + 1 < nty;
    // every plane row holds whole chunks (ld % 4 == 0), so a chunk that starts inside the image
    // may be read; other chunks are never needed
    g.col_in = g.xa >= 0 && g.xa < W;
    g.own_col = lane >= 1 && lane <= g.own;
    g.side = g.nl && g.nr ? -1 : (W - 1) & 3;
    t.lane = lane;
    t.warp = warp;
    t.first = g.xa == 0;
    t.last = g.xa <= W - 1 && g.xa + 4 > W - 1;
    t.row0 = g.y0 - kResT + warp * R;
    t.H = H;
    t.tmem = tmem + ((unsigned)(warp & 3) << 21) + (unsigned)(warp >> 2) * (R * 16);
    g.ghosts = (t.row0 < 0 && t.row0 + R > 0) || (t.row0 < H && t.row0 + R > H);
}

// Where each message a tile receives comes from: its index in all outboxes' first half, -1: none;
// and the chunks nobody sends stay 0 (cells that are never used, but garbage there, a NaN, would
// send whole warps through the exact form's general division).
template <int NW, int R>
__device__ __forceinline__ void res_sources(const ResTile &g, int *src, float *in) {
    using S = ResSmem<NW, R>;
    const int chunks = (g.W + 3) / 4;
    const int lown = g.nl ? res_split(g.tx, g.ntx, chunks) - res_split(g.tx - 1, g.ntx, chunks) : 0;
    for (int i = threadIdx.x; i < S::msgs; i += NW * 32) {
        const int c = i / 3, m = i % 3;
        int dx = 0, dy = 0, from = -1;  // the neighbour and its chunk
        if (c < 2 * kResRowChunks) {
            const int blk = c / kResRowChunks, l = c % 32;  // 0: above, from that tile's last rows
            dy = blk == 0 ? -1 : 1;
            dx = l == 0 ? -1 : l == g.own + 1 ? 1 : 0;
            if (l <= g.own + 1)
                from = (1 - blk) * kResRowChunks + (c % kResRowChunks) - l + (l == 0 ? lown : l == g.own + 1 ? 1 : l);
        } else {
            const int k = c - 2 * kResRowChunks, sd = k >= NW * R, lr = k - sd * (NW * R);
            dx = sd ? 1 : -1;
            const int row = g.y0 - kResT + lr;
            if (row >= g.y0 && row < g.y1) from = 2 * kResRowChunks + (1 - sd) * (NW * R) + lr;
        }
        const int nx = g.tx + dx, ny = g.ty + dy;
        if (nx < 0 || nx >= g.ntx || ny < 0 || ny >= g.nty) from = -1;
        src[i] = from < 0 ? -1 : (ny * g.ntx + nx) * S::msgs + 3 * from + m;
    }
    for (int i = threadIdx.x; i < S::chunks * 8; i += NW * 32) in[i] = 0.f;
}

// Exchange e of a tile (all threads of the CTA): the ring of cu to the neighbours, their rings into
// its halo.  FENCE: what this CTA wrote to global memory before the exchange is visible to its
// neighbours after it.  false: a wait ran out.
template <int NW, int R, bool FENCE>
__device__ __forceinline__ bool res_exchange(const ResLane &t, const ResTile &g, float2 (&cu)[R][2][2], float *out,
                                             float *in, const int *src, float4 *box, unsigned e, int *stop,
                                             const ResWait &w) {
    using S = ResSmem<NW, R>;
    // (uniform in the warp) rows of the ring, and rows of the halo, among the warp's
    const int row_end = t.row0 + R;
    const bool up_rows = t.row0 < g.y0 + kResT && row_end > g.y0;
    const bool down_rows = t.row0 < g.y1 && row_end > g.y1 - kResT;
    const bool above_rows = t.row0 < g.y0, below_rows = t.row0 < g.y1 + kResT && row_end > g.y1;
    if constexpr (FENCE) __threadfence();
    if ((t.lane == 1 && g.nl) || (t.lane == g.own && g.nr)) {  // (own >= 2 in a tile with neighbours beside it)
        float *f = out + 8 * (2 * kResRowChunks + (t.lane == 1 ? 0 : NW * R) + t.warp * R);
#pragma unroll
        for (int r = 0; r < R; ++r) put_chunk(f + 8 * r, cu[r]);
    }
    if (up_rows || down_rows) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int j = t.row0 + r - g.y0, k = t.row0 + r - (g.y1 - kResT);
            if (j >= 0 && j < kResT) put_chunk(out + 8 * (32 * j + t.lane), cu[r]);
            if (k >= 0 && k < kResT) put_chunk(out + 8 * (kResRowChunks + 32 * k + t.lane), cu[r]);
        }
    }
    __syncthreads();
    float4 *boxes = box + ((e & 1u) ? (size_t)g.ntx * g.nty * S::msgs : 0);
    float4 *mine = boxes + (size_t)g.tile * S::msgs;
    constexpr int kPer = (S::msgs + NW * 32 - 1) / (NW * 32);  // messages per thread
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int m = threadIdx.x + i * NW * 32;
        if (m < S::msgs) {
            const float *f = out + 8 * (m / 3) + 3 * (m % 3);
            msg_store(mine + m, f[0], f[1], f[2], e);
        }
    }
    // receive: all of the thread's loads in flight, until each carries e
    int from[kPer];
    float got[kPer][3];
    unsigned tag[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int m = threadIdx.x + i * NW * 32;
        from[i] = m < S::msgs ? src[m] : -1;
        tag[i] = e;
        if (from[i] >= 0) msg_load(boxes + from[i], got[i], tag[i]);
    }
    for (int polls = 0;;) {
        bool all = true;
#pragma unroll
        for (int i = 0; i < kPer; ++i) all = all && tag[i] == e;
        if (all) break;
        if (++polls > w.polls ||
            ((polls & 1023) == 0 && (*(volatile int *)stop || *(volatile unsigned *)w.abort_flag))) {
            atomicExch(w.abort_flag, 1u);
            if (w.status) atomicCAS(w.status, 0, (int)HS_ERR_TIMEOUT);
            atomicCAS(&g_wait_status, 0, (int)HS_ERR_TIMEOUT);
            *(volatile int *)stop = 1;
            break;
        }
#pragma unroll
        for (int i = 0; i < kPer; ++i)
            if (tag[i] != e) msg_load(boxes + from[i], got[i], tag[i]);
    }
    if constexpr (FENCE) __threadfence();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int m = threadIdx.x + i * NW * 32;
        if (from[i] >= 0) {
            float *f = in + 8 * (m / 3) + 3 * (m % 3);
            f[0] = got[i][0];
            f[1] = got[i][1];
            if (m % 3 < 2) f[2] = got[i][2];
        }
    }
    __syncthreads();
    if (*(volatile int *)stop) return false;
    if ((t.lane == 0 && g.nl) || (t.lane == g.own + 1 && g.nr)) {
        const float *f = in + 8 * (2 * kResRowChunks + (t.lane == 0 ? 0 : NW * R) + t.warp * R);
#pragma unroll
        for (int r = 0; r < R; ++r) get_chunk(f + 8 * r, cu[r]);
    }
    if ((above_rows && g.nu) || (below_rows && g.nd)) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int j = t.row0 + r - (g.y0 - kResT), k = t.row0 + r - g.y1;
            if (g.nu && j < kResT) get_chunk(in + 8 * (32 * j + t.lane), cu[r]);
            if (g.nd && k >= 0 && k < kResT) get_chunk(in + 8 * (kResRowChunks + 32 * k + t.lane), cu[r]);
        }
    }
    __syncwarp();
    return true;
}

// n sweeps in the variant of the tile's side (uniform in the CTA; one block barrier per sweep).
template <bool FAST, int NW, int R, bool UPDATE = true>
__device__ __forceinline__ void res_run(const ResLane &t, const ResTile &g, float2 (&cu)[R][2][2], float4 *pub,
                                        int half, int n, float we, float wc) {
    switch (g.side) {
        case -1: res_sweeps<FAST, NW, R, -1, UPDATE>(t, cu, pub, half, n, g.ghosts, we, wc); break;
        case 0: res_sweeps<FAST, NW, R, 0, UPDATE>(t, cu, pub, half, n, g.ghosts, we, wc); break;
        case 1: res_sweeps<FAST, NW, R, 1, UPDATE>(t, cu, pub, half, n, g.ghosts, we, wc); break;
        case 2: res_sweeps<FAST, NW, R, 2, UPDATE>(t, cu, pub, half, n, g.ghosts, we, wc); break;
        default: res_sweeps<FAST, NW, R, 3, UPDATE>(t, cu, pub, half, n, g.ghosts, we, wc); break;
    }
}

// The tile's own pixels of the state to planes U, V.
template <int R>
__device__ __forceinline__ void res_store_own(const ResLane &t, const ResTile &g, const float2 (&cu)[R][2][2],
                                              float *U, float *V) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = t.row0 + r;
        if (row >= g.y0 && row < g.y1 && g.own_col) res_store(U, V, (size_t)row * g.ld + g.xa, g.W - g.xa, cu[r]);
    }
    __syncwarp();
}

}  // namespace hs
