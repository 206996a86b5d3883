// hs_resident_adj.cu -- the backward of the differentiable Horn-Schunck on the chip: one launch
// reverses all sweeps of a group of images.
//
// The streaming backward (hs_train.cu) runs per checkpoint interval two recompute passes and two
// to three adjoint passes over all images; on small images those are launches, on large ones every
// pass moves lambda, the coefficients and the accumulators.  Here a tile per SM keeps them: the
// coefficients in tensor memory, lambda (or the recomputed state) in registers, the accumulators
// dIx, dIy, dIt of a few sweeps in shared memory.  Per interval, from the last:
//   1. the states of its inner sweeps are recomputed from its checkpoint (the resident sweep, with
//      an exchange every kResT sweeps) and written to the interval's state buffer;
//   2. lambda comes back, and the interval's sweeps are reversed: M pointwise (hs_train.cu's
//      adjoint map, from the state of the sweep, read through L2) and then A.  Lambda's ring is
//      exchanged every kResT sweeps; the first of these exchanges also orders the neighbours'
//      states before their reads in the halo.  The state buffers alternate by interval parity: a
//      neighbour still reading interval b's is done before this tile, having received its
//      messages of interval b-1, writes b-2's;
//   3. lambda is parked in global memory.
// Every `chain` sweeps, whatever the intervals, the accumulators are added to the planes in global
// memory: chains of `chain` terms and then one of iters / chain sums, where the streaming passes
// have chains of 4 and one of iters / 4.
// The arithmetic of a cell is the streaming kernels'.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "hs_resident.cuh"

namespace hs {

constexpr int kAdjWarps = 16;
constexpr int kAdjMaxR = 6;  // the accumulators of a taller tile do not fit shared memory

struct ResAdjImage {
    const float *Ix, *Iy, *It;   // derivatives
    const float *dLdu, *dLdv;    // lambda at the end
    const float *ckpt;           // checkpoint planes, two per checkpoint
    float *states;               // [parity][ckpt_every - 1] x (u, v) planes
    float *park;                 // two planes for lambda between intervals
    float *acc;                  // dIx, dIy, dIt planes
    double *a2part;              // one slot per tile, zero beyond
    float4 *box;
    const float *alpha_dev;
    int H, W, ld, ntx, nty;
};

struct ResAdjTable {
    ResAdjImage img[kMaxResImages];
    int first[kMaxResImages + 1];
    int n;
    ResWait wait;
    size_t plane;                // floats between planes
    int ckpt_every, iters, nslots;
    int chain;                   // sweeps whose terms are summed before they join the planes
    float we, wc;
};

template <int R>
struct ResAdjSmem {
    using S = ResSmem<kAdjWarps, R>;
    static constexpr int rows = kAdjWarps * R - 2 * kResT;   // a tile's own rows, at most
    static constexpr int acc = (S::bytes + 15) / 16 * 16;    // [3][rows][kResChunks] float4
    static constexpr int bytes = acc + 3 * rows * kResChunks * 16;
};

// Rows of state loaded ahead of their use.  One: more (measured with two and with all of a low
// tile's rows) take registers from the sweeps around, and what does not fit goes through L2, the
// cache beside this much shared memory being small (512^2 x 200 backward 1.42 -> 1.61 ms).
template <int R>
constexpr int adj_ahead() { return 1; }

// Row r of planes xu, xv into q; zero outside the image.
__device__ __forceinline__ void adj_fetch(const ResLane &t, const ResTile &g, int r, const float *xu, const float *xv,
                                          float4 (&q)[2]) {
    const int row = t.row0 + r;
    q[0] = q[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g.col_in && row >= 0 && row < g.H) {
        const size_t off = (size_t)row * g.ld + g.xa;
        q[0] = __ldcg(reinterpret_cast<const float4 *>(xu + off));
        q[1] = __ldcg(reinterpret_cast<const float4 *>(xv + off));
    }
}

// One sweep's M on the warp's rows: lambda -> z in place; x: the state after the sweep (planes xu,
// xu + plane), its first rows already in q; next: the state the next call works from, whose first
// rows are loaded into q (or null); acc: the accumulators, of own cells; a2: the lane's
// columns' sums of lr (-t).
template <bool FAST, int R>
__device__ __forceinline__ void adj_rows(const ResLane &t, const ResTile &g, float2 (&cu)[R][2][2],
                                         float4 (&q)[adj_ahead<R>()][2], const float *xu, const float *next,
                                         size_t pl, float4 *acc, int acc_rows, float2 nia2, float alpha2,
                                         float2 (&a2)[2]) {
    constexpr int AH = adj_ahead<R>();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        __syncwarp();
        float c[16];
        tmem_ld16(c, t.tmem + 16 * r);
        const float2 xs[2][2] = {{lo2(q[r % AH][0]), hi2(q[r % AH][0])}, {lo2(q[r % AH][1]), hi2(q[r % AH][1])}};
        if (r + AH < R) adj_fetch(t, g, r + AH, xu, xu + pl, q[r % AH]);
        const int row = t.row0 + r;
        const bool mine = g.own_col && row >= g.y0 && row < g.y1;
        float2 *slot = reinterpret_cast<float2 *>(acc + (row - g.y0) * kResChunks + (t.lane - 1));
        const int plane = 2 * acc_rows * kResChunks;
        tmem_wait_ld(c);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 cx = f2(c[2 * j], c[2 * j + 1]), cy = f2(c[4 + 2 * j], c[5 + 2 * j]);
            const float2 ct = f2(c[8 + 2 * j], c[9 + 2 * j]);
            float2 nw = f2(c[12 + 2 * j], c[13 + 2 * j]);
            if constexpr (!FAST)  // the exact form keeps -den there
                nw = f2(-rcp_approx(fmaf(cy.x, cy.x, fmaf(cx.x, cx.x, alpha2))),
                        -rcp_approx(fmaf(cy.y, cy.y, fmaf(cx.y, cx.y, alpha2))));
            const float2 lu = cu[r][0][j], lv = cu[r][1][j];
            const float2 lr = mul2(fma2(cx, lu, mul2(cy, lv)), nw);
            const float2 zu = fma2(lr, cx, lu), zv = fma2(lr, cy, lv);
            const float2 nt = mul2(fma2(cx, xs[0][j], fma2(cy, xs[1][j], ct)), nia2);
            cu[r][0][j] = zu;
            cu[r][1][j] = zv;
            if (mine) {
                slot[j] = fma2(nt, zu, fma2(lr, xs[0][j], slot[j]));
                slot[plane + j] = fma2(nt, zv, fma2(lr, xs[1][j], slot[plane + j]));
                slot[2 * plane + j] = add2(slot[2 * plane + j], lr);
                a2[j] = fma2(lr, nt, a2[j]);
            }
        }
    }
    if (next) {
#pragma unroll
        for (int r = 0; r < AH; ++r) adj_fetch(t, g, r, next, next + pl, q[r]);
    }
    __syncwarp();
}

template <bool FAST, int R>
__global__ void __launch_bounds__(kAdjWarps * 32, 1) hs_resident_adj_kernel(const __grid_constant__ ResAdjTable tab) {
    constexpr int NW = kAdjWarps;
    using S = ResSmem<NW, R>;
    using A = ResAdjSmem<R>;
    extern __shared__ float4 smem[];
    __shared__ unsigned tmem_base;
    __shared__ int stop;
    __shared__ double part[NW];
    float4 *pub = smem;
    float *out = reinterpret_cast<float *>(smem) + S::out / 4, *in = reinterpret_cast<float *>(smem) + S::in / 4;
    int *src = reinterpret_cast<int *>(smem) + S::src / 4;
    float4 *acc = smem + A::acc / 16;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kCols = res_tmem_cols<NW, R>();
    if (warp == 0) {
        tmem_alloc(&tmem_base, kCols);
        if (lane == 0) stop = 0;
    }
    const unsigned tmem = tmem_base_of(&tmem_base);
    int image = 0;
    while (image + 1 < tab.n && tab.first[image + 1] <= (int)blockIdx.x) ++image;
    const ResAdjImage &p = tab.img[image];
    const int tile = blockIdx.x - tab.first[image], tiles = p.ntx * p.nty;
    const float alpha = __ldg(p.alpha_dev), alpha2 = __fmul_rn(alpha, alpha);
    const float inv_a2 = 1.0f / (alpha * alpha);
    const float2 nia2 = f2(-inv_a2, -inv_a2);
    ResLane t;
    ResTile g;
    res_tile<R>(g, t, tile, p.ntx, p.nty, p.H, p.W, p.ld, tmem);

    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = t.row0 + r;
        const bool inside = g.col_in && row >= 0 && row < p.H;
        const size_t off = (size_t)(inside ? row : 0) * p.ld + (inside ? g.xa : 0);
        const float4 ix = __ldg(reinterpret_cast<const float4 *>(p.Ix + off));
        const float4 iy = __ldg(reinterpret_cast<const float4 *>(p.Iy + off));
        const float4 it = __ldg(reinterpret_cast<const float4 *>(p.It + off));
        float c[16] = {ix.x, ix.y, ix.z, ix.w, iy.x, iy.y, iy.z, iy.w, it.x, it.y, it.z, it.w};
        res_coefficients<FAST>(t.tmem + 16 * r, c, alpha2, inside);
    }
    tmem_wait_st();
    if (tiles > 1) res_sources<NW, R>(g, src, in);
    for (int i = threadIdx.x; i < 3 * A::rows * kResChunks; i += NW * 32) acc[i] = z4;
    __syncthreads();

    const int k = tab.ckpt_every, nb = (tab.iters + k - 1) / k;
    const size_t pl = tab.plane;
    float2 cu[R][2][2];
    // a plane pair into cu: all cells of the tile inside the image, or its own only
    auto load = [&](const float *U, const float *V, bool own) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = t.row0 + r;
            float4 u = z4, v = z4;
            if (own ? g.own_col && row >= g.y0 && row < g.y1 : g.col_in && row >= 0 && row < p.H) {
                const size_t off = (size_t)row * p.ld + g.xa;
                u = __ldcg(reinterpret_cast<const float4 *>(U + off));
                v = __ldcg(reinterpret_cast<const float4 *>(V + off));
            }
            cu[r][0][0] = lo2(u);
            cu[r][0][1] = hi2(u);
            cu[r][1][0] = lo2(v);
            cu[r][1][1] = hi2(v);
        }
        __syncwarp();
    };
    // the accumulators join the planes in global memory (each thread its own cells; the first ones
    // are the planes' start).  Called before a sweep, not after it: the sweep's registers are dead
    // there (after it R = 5 spilled twice as much, 2 x 700^2 x 200 1.96 -> 2.08 ms).
    auto flush = [&](bool first) {
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            const int row = t.row0 + r;
            if (!(g.own_col && row >= g.y0 && row < g.y1)) continue;
            const size_t off = (size_t)row * p.ld + g.xa;
            for (int i = 0; i < 3; ++i) {
                float4 *a = reinterpret_cast<float4 *>(p.acc + i * pl + off);
                float4 *s = acc + (i * A::rows + row - g.y0) * kResChunks + (lane - 1);
                float4 v = *s;
                if (!first) {
                    const float4 w = *a;
                    v = make_float4(w.x + v.x, w.y + v.y, w.z + v.z, w.w + v.w);
                }
                *a = v;
                *s = z4;
            }
        }
        __syncwarp();
    };
    unsigned e = 0;
    int half = 0, left = tab.chain;  // left: sweeps until the accumulators join the planes
    bool first = true, ok = true;
    double a2sum = 0.0;
    for (int b = nb - 1; b >= 0 && ok; --b) {
        const int nsw = min(k, tab.iters - b * k);
        float *states = p.states + (size_t)(b & 1) * (2 * (size_t)(k - 1)) * pl;
        // 1. states of sweeps 1 .. nsw - 1 of the interval
        if (nsw > 1) {
            load(p.ckpt + (size_t)(2 * b) * pl, p.ckpt + (size_t)(2 * b + 1) * pl, false);
            for (int s = 1; s < nsw; ++s) {
                if (s > 1 && (s - 1) % kResT == 0 && tiles > 1)
                    if (!(ok = res_exchange<NW, R, false>(t, g, cu, out, in, src, p.box, ++e, &stop, tab.wait)))
                        break;
                res_run<FAST, NW, R>(t, g, cu, pub, half, 1, tab.we, tab.wc);
                half ^= 1;
                res_store_own<R>(t, g, cu, states + (size_t)(2 * (s - 1)) * pl, states + (size_t)(2 * s - 1) * pl);
            }
            if (!ok) break;
        }
        // 2. lambda, reversed through the interval's sweeps
        if (b == nb - 1) load(p.dLdu, p.dLdv, true);
        else load(p.park, p.park + pl, true);
        // the state after sweep m of the interval
        auto state_of = [&](int m) {
            return m == nsw ? p.ckpt + (size_t)(2 * (b + 1)) * pl : states + (size_t)(2 * (m - 1)) * pl;
        };
        float4 xq[adj_ahead<R>()][2];
#pragma unroll
        for (int r = 0; r < adj_ahead<R>(); ++r) adj_fetch(t, g, r, state_of(nsw), state_of(nsw) + pl, xq[r]);
        for (int m = nsw; m >= 1; --m) {
            if (left == 0) {
                flush(first);
                first = false;
                left = tab.chain;
            }
            --left;
            if ((nsw - m) % kResT == 0 && tiles > 1) {
                ok = m == nsw ? res_exchange<NW, R, true>(t, g, cu, out, in, src, p.box, ++e, &stop, tab.wait)
                              : res_exchange<NW, R, false>(t, g, cu, out, in, src, p.box, ++e, &stop, tab.wait);
                if (!ok) break;
            }
            float2 a2[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
            adj_rows<FAST, R>(t, g, cu, xq, state_of(m), m > 1 ? state_of(m - 1) : nullptr, pl, acc, A::rows, nia2,
                              alpha2, a2);
            float s = 0.f;  // (columns past the image's last one do not count)
            s += g.xa < p.W ? a2[0].x : 0.f;
            s += g.xa + 1 < p.W ? a2[0].y : 0.f;
            s += g.xa + 2 < p.W ? a2[1].x : 0.f;
            s += g.xa + 3 < p.W ? a2[1].y : 0.f;
            a2sum += (double)s;
            res_run<true, NW, R, false>(t, g, cu, pub, half, 1, tab.we, tab.wc);
            half ^= 1;
        }
        if (!ok) break;
        if (b == 0) flush(first);  // (left < chain: at least one sweep is in them)
        // 3. lambda parked (each thread its own cells)
        if (b > 0) res_store_own<R>(t, g, cu, p.park, p.park + pl);
    }
    __syncthreads();
    if (tiles > 1) ok = ok && stop == 0 && *(volatile unsigned *)tab.wait.abort_flag == 0u;
    if (!ok) {  // a wait ran out: NaN gradients
        const float nanf_ = __int_as_float(0x7fc00000);
        for (int r = 0; r < R; ++r) {
            const int row = t.row0 + r;
            if (g.own_col && row >= g.y0 && row < g.y1)
                for (int i = 0; i < 3; ++i)
                    *reinterpret_cast<float4 *>(p.acc + i * pl + (size_t)row * p.ld + g.xa) =
                        make_float4(nanf_, nanf_, nanf_, nanf_);
        }
        a2sum = (double)nanf_;
    }
    // this tile's share of dL/dalpha^2, in a fixed order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a2sum += __shfl_xor_sync(kFull, a2sum, o);
    if (lane == 0) part[warp] = a2sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < NW; ++w) s += part[w];
        p.a2part[tile] = s;
    }
    if (tile == 0)
        for (int i = tiles + threadIdx.x; i < tab.nslots; i += NW * 32) p.a2part[i] = 0.0;
    if (warp == 0) tmem_dealloc(tmem, kCols);
}

// Clears the outboxes of a launch's tiles: block i those of tile i.
__global__ void __launch_bounds__(256) res_adj_clear_kernel(const __grid_constant__ ResAdjTable tab, int msgs) {
    int image = 0;
    while (image + 1 < tab.n && tab.first[image + 1] <= (int)blockIdx.x) ++image;
    const ResAdjImage &p = tab.img[image];
    const int tiles = p.ntx * p.nty, tile = blockIdx.x - tab.first[image];
    if (blockIdx.x == 0 && threadIdx.x == 0) *tab.wait.abort_flag = 0u;
    if (tiles == 1) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int h = 0; h < 2; ++h)
        for (int i = threadIdx.x; i < msgs; i += blockDim.x) p.box[(size_t)(h * tiles + tile) * msgs + i] = z;
}

template <bool FAST, int R>
static hs_status launch_resident_adj(const ResAdjTable &tab, cudaStream_t s) {
    auto fn = hs_resident_adj_kernel<FAST, R>;
    constexpr int smem = ResAdjSmem<R>::bytes;
    static_assert(smem <= 232448 - 1024, "a tile's buffers fit shared memory");
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
    cfg.blockDim = dim3(kAdjWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeCooperative;
    a[0].val.cooperative = 1;
    cfg.attrs = a;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, tab);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return HS_ERR_UNSUPPORTED;
    }
    HS_CUDA_CHECK(e);
    return HS_OK;
}

hs_status resident_adjoint_wait_status(int *device_status, cudaStream_t s) {
    wait_status_kernel<<<1, 1, 0, s>>>(device_status, 0);
    HS_LAUNCH_CHECK("wait_status_kernel");
    return HS_OK;
}

// When the backward runs here and when in the streaming passes (hs_train.cu): the time of a sweep with
// its recompute in one launch here, of r rows per warp and mpx Mpx, and in the passes for n images.
// Both are fits to 752 backwards measured on B200, 64^2 .. 1920x1080, 1 .. 32 images, intervals of 1 ..
// 32 sweeps, both forms (each 10 % r.m.s.).  By this rule they take 0.757 of the passes' time in the
// geometric mean, by the faster way each time 0.754, and none takes more than 1.10 of it.
//   here  : the tile's rows (the exact form divides in its recompute), the states' way through L2 and,
//           past it, through HBM, and an exchange every kResT sweeps or every interval;
//   passes: launches below 0.17 Mpx, the planes' traffic above.  An interval of one sweep recomputes
//           nothing, one of two sweeps takes a pass for its one.
// Measured, us per sweep here / in the passes, intervals of 10, fast form: 320x240 5.4 / 4.9 (exact
// 6.6 / 7.0), 2 of 200x192 3.9 / 5.1, 512^2 6.7 / 8.9 (intervals of 1: 8.5 / 5.8), 4 of 512^2 12.0 / 13.2,
// 16 of 512^2 47.6 / 36.7.
static double adj_sweep_us(int r, double mpx, bool several, int ckpt_every, bool fast) {
    static const double rows[2][kAdjMaxR - 1] = {{2.3, 4.4, 6.1, 7.3, 9.0}, {2.6, 4.3, 4.5, 6.0, 7.0}};
    const double spilled = std::max(0.0, mpx * 16.0 * (ckpt_every - 1) - 120.0);  // MB of states beyond L2
    return rows[fast][r - 2] + (fast ? 2.7 : 3.5) * mpx + (fast ? 0.0014 : 0.0025) * spilled +
           (several ? 2.6 / std::min(ckpt_every, kResT) : 0.0);
}
static double passes_sweep_us(int n, double mpx, int ckpt_every, bool fast) {
    const bool small = mpx < 0.17;
    double us;
    if (ckpt_every == 1) us = small ? 3.3 + 7.0 * mpx : 4.8 + 3.8 * mpx;
    else if (ckpt_every == 2) us = 8.0 + 7.3 * mpx;
    else if (small) us = (ckpt_every == 3 ? 6.5 : ckpt_every == 4 ? 4.2 : fast ? 4.6 : 6.0) + (fast ? 6.0 : 9.0) * mpx;
    else us = fast ? 7.0 + 5.5 * mpx + std::max(0.0, mpx - 2.0) : 8.2 + 8.0 * mpx + std::max(0.0, mpx - 2.0);
    return us + 0.15 * (n - 1);
}

hs_status run_resident_adjoint(const ResidentAdjJob *jobs, int n, int iters, int ckpt_every, size_t plane, int nslots,
                               const ResolvedConfig &rc, cudaStream_t s, int polls) {
    std::vector<ResidentJob> sizes(n);
    for (int i = 0; i < n; ++i) {
        memset(&sizes[i], 0, sizeof(ResidentJob));
        sizes[i].H = jobs[i].H;
        sizes[i].W = jobs[i].W;
        sizes[i].iters = iters;
        sizes[i].scratch_bytes = jobs[i].scratch_bytes;
    }
    ResidentCut cut;
    if (!resident_cut(sizes.data(), n, 1.2, 1.45, kAdjMaxR, cut)) return HS_ERR_UNSUPPORTED;
    double here = 0.0, pixels = 0.0;
    for (size_t l = 0; l < cut.end.size(); ++l) {
        const int r = cut.r[l];
        double px = 0.0;
        bool several = false;
        for (int i = l ? cut.end[l - 1] : 0; i < cut.end[l]; ++i) {
            int ntx, nty;
            px += 1e-6 * jobs[i].H * jobs[i].W;
            several |= resident_tiles(jobs[i].H, jobs[i].W, r, &ntx, &nty) > 1;
        }
        here += adj_sweep_us(r, px, several, ckpt_every, rc.fast);
        pixels += px;
    }
    if (here > passes_sweep_us(n, pixels, ckpt_every, rc.fast)) return HS_ERR_UNSUPPORTED;
    for (size_t l = 0; l < cut.end.size(); ++l) {
        const int i0 = l ? cut.end[l - 1] : 0, m = cut.end[l] - i0, r = cut.r[l];
        ResAdjTable tab;
        memset(&tab, 0, sizeof(tab));
        tab.n = m;
        tab.wait.polls = polls;
        tab.plane = plane;
        tab.ckpt_every = ckpt_every;
        tab.iters = iters;
        // Terms of like size, FP32 on the CPU against 64 bits, relative error of the sums in 1e-8 (the
        // passes' order, chains of 4 / this one / one chain per checkpoint interval of all sweeps):
        // 16 sweeps 4.2 / 4.2 / 6.1, 50 sweeps 5.8 / 4.8 / 10.4, 200 sweeps 10.5 / 5.9 / 20.6.  (An
        // interval each instead: 600x800, 100 sweeps, intervals of 1, 977 us against 727.)
        tab.chain = iters < 32 ? 4 : iters < 64 ? 8 : 16;
        tab.nslots = nslots;
        tab.we = rc.we;
        tab.wc = rc.wc;
        bool several = false;
        for (int i = 0; i < m; ++i) {
            const ResidentAdjJob &d = jobs[i0 + i];
            ResAdjImage &p = tab.img[i];
            p.Ix = d.Ix; p.Iy = d.Iy; p.It = d.It;
            p.dLdu = d.dLdu; p.dLdv = d.dLdv;
            p.ckpt = d.ckpt; p.states = d.states; p.park = d.park; p.acc = d.acc;
            p.a2part = d.a2part;
            p.box = reinterpret_cast<float4 *>(d.scratch);
            p.alpha_dev = d.alpha_dev;
            p.H = d.H; p.W = d.W; p.ld = d.ld;
            const int tiles = resident_tiles(d.H, d.W, r, &p.ntx, &p.nty);
            tab.first[i + 1] = tab.first[i] + tiles;
            if (tiles > 1) {
                several = true;
                tab.wait.abort_flag = reinterpret_cast<unsigned *>(d.scratch + resident_box_bytes(tiles, r) - 256);
            }
            if (tiles > nslots) HS_FAIL(HS_ERR_INVALID_ARG, "internal: %d tiles, %d slots", tiles, nslots);
        }
        if (several) {
            res_adj_clear_kernel<<<tab.first[m], 256, 0, s>>>(tab, res_msgs(kAdjWarps * r));
            HS_LAUNCH_CHECK("res_adj_clear_kernel");
        }
        hs_status st = HS_ERR_UNSUPPORTED;
        switch (r) {
#define HS_RES(RR) \
    case RR: st = rc.fast ? launch_resident_adj<true, RR>(tab, s) : launch_resident_adj<false, RR>(tab, s); break;
            HS_RES(2) HS_RES(3) HS_RES(4) HS_RES(5) HS_RES(6)
#undef HS_RES
        }
        if (st != HS_OK) return st;
    }
    return HS_OK;
}

}  // namespace hs
