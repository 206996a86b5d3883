// hs_resident.cu -- the cooperative launch of the resident Horn-Schunck sweeps
// (hs_resident.cuh): tile shapes, the exchange between tiles and the host's choice of tiling.
//
// Measured on one B200 (hs_forward, us per call, streaming passes at their default depth ->
// resident):
//   1920x1080 x 500 sweeps, fast   2001 -> 1207      1901x1037 x 200, exact  1463 -> 970
//   320x240 x 100, fast             171 ->  107       640x480 x 200, exact    856 -> 310
// Bound (1080p, fast, 16 x 8 rows): of 2.4 us per sweep, 1.7 us are the sweep itself (the FP32
// pipe and the register reads of its packed operations: fma.rn.f32x2 with three distinct
// operands issues every 3.1 clocks, with a shared one every 2.2) and 0.7 us the exchange's share
// (a quarter of 2.8 us: shared-memory staging and one round trip to L2).  16 warps of 128
// registers run it faster than 8 of 255 (1.72 against 2.14 us per sweep): the state of R = 16
// rows leaves too few warps to cover the shuffles.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "hs_resident.cuh"

namespace hs {

// Polls of one message, at most: a few seconds.  A wait can only run out if a neighbour's CTA
// has stopped (all CTAs of the cooperative launch are resident together); the tile then raises
// the abort flag, stops waiting, and the tiles that see the flag write NaN as their result.
constexpr int kResPolls = 1 << 22;

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

template <bool FAST, int NW, int R>
__global__ void __launch_bounds__(NW * 32, 1) hs_resident_kernel(const __grid_constant__ ResidentTable tab) {
    using S = ResSmem<NW, R>;
    extern __shared__ float4 smem[];
    __shared__ unsigned tmem_base;
    __shared__ int stop;
    float4 *pub = smem;
    float *out = reinterpret_cast<float *>(smem) + S::out / 4, *in = reinterpret_cast<float *>(smem) + S::in / 4;
    int *src = reinterpret_cast<int *>(smem) + S::src / 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kCols = res_tmem_cols<NW, R>();
    if (warp == 0) {
        tmem_alloc(&tmem_base, kCols);
        if (lane == 0) stop = 0;
    }
    const unsigned tmem = tmem_base_of(&tmem_base);

    int image = 0;
    while (image + 1 < tab.n && tab.first[image + 1] <= (int)blockIdx.x) ++image;
    const ResImage &p = tab.img[image];
    const int tile = blockIdx.x - tab.first[image], tx = tile % p.ntx, ty = tile / p.ntx;
    const float alpha2 = p.alpha_dev ? __fmul_rn(__ldg(p.alpha_dev), __ldg(p.alpha_dev)) : p.alpha2;
    const int chunks = (p.W + 3) / 4;
    const int x0 = 4 * res_split(tx, p.ntx, chunks), x1 = 4 * res_split(tx + 1, p.ntx, chunks);
    const int y0 = res_split(ty, p.nty, p.H), y1 = res_split(ty + 1, p.nty, p.H);
    const int xa = x0 - 4 + 4 * lane;  // the lane's first column (a multiple of 4)
    const int own = (x1 - x0) / 4;     // lanes 1 .. own hold the tile's own columns

    ResLane t;
    t.lane = lane;
    t.warp = warp;
    t.first = xa == 0;
    t.last = xa <= p.W - 1 && xa + 4 > p.W - 1;
    t.row0 = y0 - kResT + warp * R;
    t.H = p.H;
    t.tmem = tmem + ((unsigned)(warp & 3) << 21) + (unsigned)(warp >> 2) * (R * 16);
    // every plane row holds whole chunks (ld % 4 == 0), so a chunk that starts inside the image
    // may be read; other chunks are never needed
    const bool col_in = xa >= 0 && xa < p.W;
    const bool own_col = lane >= 1 && lane <= own;

    // start state and coefficients
    float2 cu[R][2][2];
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    // a row of one image: the lane's 4 columns and the next one (clamped to column W-1)
    auto image_row = [&](const float *I, int row, float (&f)[5]) {
        row = min(max(row, 0), p.H - 1);
        const float4 a = col_in ? __ldg(reinterpret_cast<const float4 *>(I + (size_t)row * p.ld + xa)) : z4;
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
        f[4] = __shfl_down_sync(kFull, a.x, 1);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (xa + j == p.W - 1) f[j + 1] = f[j];
    };
    float i0[5], i1[5];
    if (p.I0) {
        image_row(p.I0, t.row0, i0);
        image_row(p.I1, t.row0, i1);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = t.row0 + r;
        const bool in = col_in && row >= 0 && row < p.H;
        const size_t off = (size_t)(in ? row : 0) * p.ld + (in ? xa : 0);
        float c[16];
        if (p.I0) {
            float n0[5], n1[5];  // the next row (row H-1 stands in for row H)
            image_row(p.I0, row + 1, n0);
            image_row(p.I1, row + 1, n1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float a[4] = {i0[j], i0[j + 1], n0[j], n0[j + 1]};
                const float b[4] = {i1[j], i1[j + 1], n1[j], n1[j + 1]};
                hs_derivs_taps(a, b, c[j], c[4 + j], c[8 + j]);
            }
            if (p.Ix && own_col && row >= y0 && row < y1) {  // (scratch planes: whole chunks)
                *reinterpret_cast<float4 *>(p.Ix + off) = make_float4(c[0], c[1], c[2], c[3]);
                *reinterpret_cast<float4 *>(p.Iy + off) = make_float4(c[4], c[5], c[6], c[7]);
                *reinterpret_cast<float4 *>(p.It + off) = make_float4(c[8], c[9], c[10], c[11]);
            }
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                i0[j] = n0[j];
                i1[j] = n1[j];
            }
        } else {
            const float4 ix = __ldg(reinterpret_cast<const float4 *>(p.Ix + off));
            const float4 iy = __ldg(reinterpret_cast<const float4 *>(p.Iy + off));
            const float4 it = __ldg(reinterpret_cast<const float4 *>(p.It + off));
            c[0] = ix.x; c[1] = ix.y; c[2] = ix.z; c[3] = ix.w;
            c[4] = iy.x; c[5] = iy.y; c[6] = iy.z; c[7] = iy.w;
            c[8] = it.x; c[9] = it.y; c[10] = it.z; c[11] = it.w;
        }
        res_coefficients<FAST>(t.tmem + 16 * r, c, alpha2, in);
        float4 u = z4, v = z4;
        if (in && !tab.zero_start) {
            u = __ldcg(reinterpret_cast<const float4 *>(p.u + off));
            v = __ldcg(reinterpret_cast<const float4 *>(p.v + off));
        }
        cu[r][0][0] = lo2(u);
        cu[r][0][1] = hi2(u);
        cu[r][1][0] = lo2(v);
        cu[r][1][1] = hi2(v);
    }
    tmem_wait_st();
    // a neighbour that has heard from this tile may overwrite what was just read (u, v, or
    // images that share memory with them): the reads come before every message
    __threadfence();
    __syncwarp();

    const bool nl = tx > 0, nr = tx + 1 < p.ntx, nu = ty > 0, nd = ty + 1 < p.nty;
    const int side = nl && nr ? -1 : (p.W - 1) & 3;
    const bool ghosts = (t.row0 < 0 && t.row0 + R > 0) || (t.row0 < p.H && t.row0 + R > p.H);
    // where each message received comes from: its index in all outboxes' first half, -1: none
    const int half_msgs = p.ntx * p.nty * S::msgs;
    if (p.nblocks > 1) {
        const int lown = nl ? res_split(tx, p.ntx, chunks) - res_split(tx - 1, p.ntx, chunks) : 0;
        for (int i = threadIdx.x; i < S::msgs; i += NW * 32) {
            const int c = i / 3, m = i % 3;
            int dx = 0, dy = 0, from = -1;  // the neighbour and its chunk
            if (c < 2 * kResRowChunks) {
                const int blk = c / kResRowChunks, l = c % 32;  // 0: above, from that tile's last rows
                dy = blk == 0 ? -1 : 1;
                dx = l == 0 ? -1 : l == own + 1 ? 1 : 0;
                if (l <= own + 1)
                    from = (1 - blk) * kResRowChunks + (c % kResRowChunks) - l + (l == 0 ? lown : l == own + 1 ? 1 : l);
            } else {
                const int k = c - 2 * kResRowChunks, sd = k >= NW * R, lr = k - sd * (NW * R);
                dx = sd ? 1 : -1;
                const int row = y0 - kResT + lr;
                if (row >= y0 && row < y1) from = 2 * kResRowChunks + (1 - sd) * (NW * R) + lr;
            }
            const int nx = tx + dx, ny = ty + dy;
            if (nx < 0 || nx >= p.ntx || ny < 0 || ny >= p.nty) from = -1;
            src[i] = from < 0 ? -1 : (ny * p.ntx + nx) * S::msgs + 3 * from + m;
        }
        // chunks that nobody sends stay 0: cells that are never used, but garbage there (a NaN)
        // would send whole warps through the exact form's general division
        for (int i = threadIdx.x; i < S::chunks * 8; i += NW * 32) in[i] = 0.f;
    }
    // (uniform in the warp) rows of the ring, and rows of the halo, among the warp's
    const int row_end = t.row0 + R;
    const bool up_rows = t.row0 < y0 + kResT && row_end > y0, down_rows = t.row0 < y1 && row_end > y1 - kResT;
    const bool above_rows = t.row0 < y0, below_rows = t.row0 < y1 + kResT && row_end > y1;
    // the tile's own pixels of the state to planes U, V
    auto store_own = [&](float *U, float *V) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = t.row0 + r;
            if (row >= y0 && row < y1 && own_col) res_store(U, V, (size_t)row * p.ld + xa, p.W - xa, cu[r]);
        }
        __syncwarp();
    };
    if (p.ckpt) store_own(p.ckpt, p.ckpt + tab.ckpt_plane);  // checkpoint 0: the start state
    int done = 0, ck = 1;  // ck: the next checkpoint
    for (int b = 0; b < p.nblocks; ++b) {
        const int upto = res_split(b + 1, p.nblocks, p.iters);
        while (done < upto) {
            const int next = p.ckpt ? min(upto, ck * tab.ckpt_every) : upto, n = next - done;
            // (uniform in the CTA; every variant runs one block barrier per sweep)
            switch (side) {
                case -1: res_sweeps<FAST, NW, R, -1>(t, cu, pub, done & 1, n, ghosts, tab.we, tab.wc); break;
                case 0: res_sweeps<FAST, NW, R, 0>(t, cu, pub, done & 1, n, ghosts, tab.we, tab.wc); break;
                case 1: res_sweeps<FAST, NW, R, 1>(t, cu, pub, done & 1, n, ghosts, tab.we, tab.wc); break;
                case 2: res_sweeps<FAST, NW, R, 2>(t, cu, pub, done & 1, n, ghosts, tab.we, tab.wc); break;
                default: res_sweeps<FAST, NW, R, 3>(t, cu, pub, done & 1, n, ghosts, tab.we, tab.wc); break;
            }
            done = next;
            if (p.ckpt && (done == ck * tab.ckpt_every || done == p.iters)) {
                store_own(p.ckpt + (size_t)(2 * ck) * tab.ckpt_plane, p.ckpt + (size_t)(2 * ck + 1) * tab.ckpt_plane);
                ++ck;
            }
        }
        if (b + 1 == p.nblocks) break;
        if (p.ntx * p.nty == 1) continue;  // no neighbours

        // exchange e: the ring into shared memory
        const unsigned e = (unsigned)(b + 1);
        if ((lane == 1 && nl) || (lane == own && nr)) {  // (own >= 2 in a tile with neighbours beside it)
            float *f = out + 8 * (2 * kResRowChunks + (lane == 1 ? 0 : NW * R) + warp * R);
#pragma unroll
            for (int r = 0; r < R; ++r) put_chunk(f + 8 * r, cu[r]);
        }
        if (up_rows || down_rows) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int j = t.row0 + r - y0, k = t.row0 + r - (y1 - kResT);
                if (j >= 0 && j < kResT) put_chunk(out + 8 * (32 * j + lane), cu[r]);
                if (k >= 0 && k < kResT) put_chunk(out + 8 * (kResRowChunks + 32 * k + lane), cu[r]);
            }
        }
        __syncthreads();
        float4 *boxes = p.box + ((e & 1u) ? (size_t)half_msgs : 0);
        float4 *mine = boxes + (size_t)tile * S::msgs;
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
            if (++polls > kResPolls ||
                ((polls & 1023) == 0 && (*(volatile int *)&stop || *(volatile unsigned *)tab.abort_flag))) {
                atomicExch(tab.abort_flag, 1u);
                if (tab.status) atomicCAS(tab.status, 0, (int)HS_ERR_TIMEOUT);
                *(volatile int *)&stop = 1;
                break;
            }
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (tag[i] != e) msg_load(boxes + from[i], got[i], tag[i]);
        }
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
        if (stop) break;
        if ((lane == 0 && nl) || (lane == own + 1 && nr)) {
            const float *f = in + 8 * (2 * kResRowChunks + (lane == 0 ? 0 : NW * R) + warp * R);
#pragma unroll
            for (int r = 0; r < R; ++r) get_chunk(f + 8 * r, cu[r]);
        }
        if ((above_rows && nu) || (below_rows && nd)) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int j = t.row0 + r - (y0 - kResT), k = t.row0 + r - y1;
                if (nu && j < kResT) get_chunk(in + 8 * (32 * j + lane), cu[r]);
                if (nd && k >= 0 && k < kResT) get_chunk(in + 8 * (kResRowChunks + 32 * k + lane), cu[r]);
            }
        }
        __syncwarp();
    }
    __syncthreads();
    bool ok = true;
    if (p.nblocks > 1) ok = stop == 0 && *(volatile unsigned *)tab.abort_flag == 0u;
    if (!ok) {
        const float2 nan2 = f2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) cu[r][q][0] = cu[r][q][1] = nan2;
    }
    store_own(p.u, p.v);
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kCols);
}

// ------------------------------------------------------------------ host side

template <bool FAST, int NW, int R>
static hs_status launch_resident(const ResidentTable &tab, cudaStream_t s) {
    auto fn = hs_resident_kernel<FAST, NW, R>;
    constexpr int smem = ResSmem<NW, R>::bytes;
    static std::mutex mu;
    static bool attr[64] = {};
    int dev = 0;
    HS_CUDA_CHECK(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev >= 64 || !attr[dev]) {
            HS_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
            if (dev < 64) attr[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tab.first[tab.n]);
    cfg.blockDim = dim3(NW * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeCooperative;
    a[0].val.cooperative = 1;
    cfg.attrs = a;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, tab);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs at hand than the device has
        cudaGetLastError();
        return HS_ERR_UNSUPPORTED;
    }
    HS_CUDA_CHECK(e);
    return HS_OK;
}

// Tile shapes: 16 warps of r rows; a tile's own rows, at most.
constexpr int kResWarps = 16, kResMinR = 2, kResMaxR = 8;
constexpr int res_rows(int r) { return kResWarps * r - 2 * kResT; }

int resident_tiles(int H, int W, int r, int *ntx, int *nty) {
    const int chunks = (W + 3) / 4;
    *ntx = (chunks + kResChunks - 1) / kResChunks;
    *nty = (H + res_rows(r) - 1) / res_rows(r);
    const long tiles = (long)*ntx * *nty;
    return (int)std::min(tiles, 1L << 30);
}

size_t resident_box_bytes(int tiles, int r) {
    if (tiles == 1) return 0;
    return (size_t)2 * tiles * res_msgs(kResWarps * r) * sizeof(float4) + 256;
}

// The tiling of an H x W image: the smallest tiles that the SMs hold all at once and whose
// outboxes fit the scratch.
bool resident_plan(int H, int W, int iters, size_t scratch_bytes, ResidentPlan &pl) {
    if (iters < 2) return false;
    for (int r = kResMinR; r <= kResMaxR; ++r) {
        const int tiles = resident_tiles(H, W, r, &pl.ntx, &pl.nty);
        if (tiles > sm_count()) continue;
        pl.r = r;
        pl.box_bytes = resident_box_bytes(tiles, r);
        if (pl.box_bytes <= scratch_bytes) return true;
    }
    return false;
}

// Clears the outboxes of a launch's tiles: block i those of tile i.
__global__ void __launch_bounds__(256) res_clear_kernel(const __grid_constant__ ResidentTable tab, int msgs) {
    int image = 0;
    while (image + 1 < tab.n && tab.first[image + 1] <= (int)blockIdx.x) ++image;
    const ResImage &p = tab.img[image];
    const int tiles = p.ntx * p.nty, tile = blockIdx.x - tab.first[image];
    if (blockIdx.x == 0 && threadIdx.x == 0) *tab.abort_flag = 0u;
    if (tiles == 1) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int h = 0; h < 2; ++h)
        for (int i = threadIdx.x; i < msgs; i += blockDim.x) p.box[(size_t)(h * tiles + tile) * msgs + i] = z;
}

// Launches the table (img, n, ckpt_* and abort_flag filled in; every image tiled for r rows per
// warp).  An image of several tiles has at least one exchange, so that no tile writes its result
// before its neighbours have read their inputs; an image of a single tile needs none.
static hs_status launch_table(ResidentTable &tab, int r, bool zero_start, const ResolvedConfig &rc, cudaStream_t s) {
    tab.first[0] = 0;
    bool several = false;
    for (int i = 0; i < tab.n; ++i) {
        ResImage &p = tab.img[i];
        const int tiles = p.ntx * p.nty;
        tab.first[i + 1] = tab.first[i] + tiles;
        several |= tiles > 1;
        p.nblocks = tiles > 1 ? std::max(2, (p.iters + kResT - 1) / kResT) : 1;
    }
    tab.we = rc.we;
    tab.wc = rc.wc;
    tab.zero_start = zero_start ? 1 : 0;
    if (several && tab.n == 1) {  // the flag lies behind the one image's outboxes
        const size_t bytes = resident_box_bytes(tab.first[1], r);
        HS_CUDA_CHECK(cudaMemsetAsync(tab.img[0].box, 0, bytes, s));
    } else if (several) {
        res_clear_kernel<<<tab.first[tab.n], 256, 0, s>>>(tab, res_msgs(kResWarps * r));
        HS_LAUNCH_CHECK("res_clear_kernel");
    }
    switch (r) {
#define HS_RES(RR) \
    case RR: return rc.fast ? launch_resident<true, kResWarps, RR>(tab, s) : launch_resident<false, kResWarps, RR>(tab, s);
        HS_RES(2) HS_RES(3) HS_RES(4) HS_RES(5) HS_RES(6) HS_RES(7) HS_RES(8)
#undef HS_RES
    }
    HS_FAIL(HS_ERR_INVALID_ARG, "internal: no resident kernel for %d rows", r);
}

hs_status run_resident(const float *I0, const float *I1, const float *Ix, const float *Iy, const float *It, int H,
                       int W, int ld, float alpha2, int iters, float *u, float *v, void *scratch, bool zero_start,
                       const ResolvedConfig &rc, const ResidentPlan &pl, cudaStream_t s) {
    ResidentTable tab;
    memset(&tab, 0, sizeof(tab));
    tab.n = 1;
    ResImage &p = tab.img[0];
    p.I0 = I0; p.I1 = I1;
    p.Ix = const_cast<float *>(Ix); p.Iy = const_cast<float *>(Iy); p.It = const_cast<float *>(It);
    p.u = u; p.v = v;
    p.box = reinterpret_cast<float4 *>(scratch);
    p.H = H; p.W = W; p.ld = ld;
    p.alpha2 = alpha2;
    p.ntx = pl.ntx; p.nty = pl.nty;
    p.iters = iters;
    if (pl.box_bytes)
        tab.abort_flag = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(scratch) + pl.box_bytes - 256);
    return launch_table(tab, pl.r, zero_start, rc, s);
}

// ---- many images: groups whose tiles the SMs hold all at once, one launch each

// How the jobs, in their order, are cut into launches: launch k holds jobs end[k-1] .. end[k]-1
// with r[k] rows per warp.  A launch takes as long as its longest image, and a sweep of it about
// 0.65 + 0.22 r us in the fast form, 0.5 + 0.52 r in the exact one, whatever the number of tiles
// (measured at 320x240 .. 1920x1080, r = 2 .. 8): tall tiles put more images into a launch, low
// ones spread an image over more SMs.  The cut that needs the least time in all (dynamic
// programming over the prefixes).  false if an image does not fit.
struct ResidentCut {
    std::vector<int> end, r;
};
static bool resident_cut(const ResidentJob *jobs, int n, bool fast, ResidentCut &cut) {
    std::vector<double> cost(n + 1, -1.0);
    std::vector<int> from(n + 1, 0), rows(n + 1, 0);
    cost[0] = 0.0;
    for (int i = 0; i < n; ++i) {  // a launch that starts with job i
        if (cost[i] < 0.0) continue;
        for (int r = kResMinR; r <= kResMaxR; ++r) {
            const double sweep = fast ? 0.65 + 0.22 * r : 0.5 + 0.52 * r;
            int tiles = 0, longest = 0;
            for (int j = i; j < n && j < i + kMaxResImages; ++j) {
                int ntx, nty;
                const int t = resident_tiles(jobs[j].H, jobs[j].W, r, &ntx, &nty);
                tiles = std::min(tiles + std::min(t, sm_count() + 1), sm_count() + 1);
                if (tiles > sm_count() || resident_box_bytes(t, r) > jobs[j].scratch_bytes) break;
                longest = std::max(longest, jobs[j].iters);
                const double c = cost[i] + sweep * longest + 8.0;  // (and about 8 us for a launch)
                if (cost[j + 1] < 0.0 || c < cost[j + 1]) {
                    cost[j + 1] = c;
                    from[j + 1] = i;
                    rows[j + 1] = r;
                }
            }
        }
    }
    if (cost[n] < 0.0) return false;
    cut.end.clear();
    cut.r.clear();
    for (int j = n; j > 0; j = from[j]) {
        cut.end.insert(cut.end.begin(), j);
        cut.r.insert(cut.r.begin(), rows[j]);
    }
    return true;
}

bool resident_fits(int H, int W, int iters, size_t scratch_bytes) {
    ResidentPlan pl;
    return resident_plan(H, W, iters, scratch_bytes, pl);
}

hs_status run_resident_jobs(const ResidentJob *jobs, int n, int ckpt_every, size_t ckpt_plane, int *status,
                            const ResolvedConfig &rc, cudaStream_t s) {
    for (int i = 0; i < n; ++i)
        if (jobs[i].iters < 2) return HS_ERR_UNSUPPORTED;
    ResidentCut cut;
    if (!resident_cut(jobs, n, rc.fast, cut)) return HS_ERR_UNSUPPORTED;
    for (size_t g = 0; g < cut.end.size(); ++g) {
        const int i0 = g ? cut.end[g - 1] : 0, m = cut.end[g] - i0, r = cut.r[g];
        ResidentTable tab;
        memset(&tab, 0, sizeof(tab));
        tab.n = m;
        tab.ckpt_every = ckpt_every;
        tab.ckpt_plane = ckpt_plane;
        tab.status = status;
        for (int i = 0; i < m; ++i) {
            const ResidentJob &d = jobs[i0 + i];
            ResImage &p = tab.img[i];
            p.I0 = d.I0; p.I1 = d.I1;
            p.Ix = d.Ix; p.Iy = d.Iy; p.It = d.It;
            p.u = d.u; p.v = d.v;
            p.ckpt = d.ckpt;
            p.box = reinterpret_cast<float4 *>(d.scratch);
            p.alpha_dev = d.alpha_dev;
            p.alpha2 = d.alpha2;
            p.H = d.H; p.W = d.W; p.ld = d.ld;
            p.iters = d.iters;
            const int tiles = resident_tiles(d.H, d.W, r, &p.ntx, &p.nty);
            if (tiles > 1)
                tab.abort_flag = reinterpret_cast<unsigned *>(d.scratch + resident_box_bytes(tiles, r) - 256);
        }
        const hs_status st = launch_table(tab, r, true, rc, s);
        if (st != HS_OK) return st;
    }
    return HS_OK;
}

}  // namespace hs
