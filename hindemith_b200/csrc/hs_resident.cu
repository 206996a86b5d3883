// hs_resident.cu -- the cooperative launch of the resident Horn-Schunck sweeps
// (hs_resident.cuh): tile shapes, the exchange between tiles and the host's choice of tiling.
//
// Measured on one B200 (hs_forward, us per call, streaming passes at their default depth ->
// resident):
//   1920x1080 x 500 sweeps, fast   2002 -> 1240      1901x1037 x 200, exact  1465 -> 945
//   320x240 x 100, fast             170 ->  108       640x480 x 200, exact    858 -> 312
// Bound (1080p, fast, 16 x 8 rows): of 2.4 us per sweep, 1.7 us are the sweep itself (the FP32
// pipe and the register reads of its packed operations: fma.rn.f32x2 with three distinct
// operands issues every 3.1 clocks, with a shared one every 2.2) and 0.7 us the exchange's share
// (a quarter of 2.8 us: shared-memory staging and one round trip to L2).  16 warps of 128
// registers run it faster than 8 of 255 (1.72 against 2.14 us per sweep): the state of R = 16
// rows leaves too few warps to cover the shuffles.  The 128 registers do not hold all: at R = 8 the
// fast form spills 120 B of stores and 276 of loads per thread, the exact one 436 and 672; up to
// R = 4 the fast form spills nothing.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "hs_resident.cuh"

namespace hs {

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
    const int tile = blockIdx.x - tab.first[image];
    const float alpha2 = p.alpha_dev ? __fmul_rn(__ldg(p.alpha_dev), __ldg(p.alpha_dev)) : p.alpha2;
    ResLane t;
    ResTile g;
    res_tile<R>(g, t, tile, p.ntx, p.nty, p.H, p.W, p.ld, tmem);
    const int xa = g.xa;
    const bool col_in = g.col_in;

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
            if (p.Ix && g.own_col && row >= g.y0 && row < g.y1) {  // (scratch planes: whole chunks)
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

    if (p.nblocks > 1) res_sources<NW, R>(g, src, in);
    bool ok = true;
    if (p.ckpt) res_store_own<R>(t, g, cu, p.ckpt, p.ckpt + tab.ckpt_plane);  // checkpoint 0: the start state
    int done = 0, ck = 1;  // ck: the next checkpoint
    for (int b = 0; b < p.nblocks; ++b) {
        const int upto = res_split(b + 1, p.nblocks, p.iters);
        while (done < upto) {
            const int next = p.ckpt ? min(upto, ck * tab.ckpt_every) : upto, n = next - done;
            res_run<FAST, NW, R>(t, g, cu, pub, done & 1, n, tab.we, tab.wc);
            done = next;
            if (p.ckpt && (done == ck * tab.ckpt_every || done == p.iters)) {
                res_store_own<R>(t, g, cu, p.ckpt + (size_t)(2 * ck) * tab.ckpt_plane,
                                 p.ckpt + (size_t)(2 * ck + 1) * tab.ckpt_plane);
                ++ck;
            }
        }
        if (b + 1 == p.nblocks) break;
        if (p.ntx * p.nty == 1) continue;  // no neighbours

        if (!res_exchange<NW, R, false>(t, g, cu, out, in, src, p.box, (unsigned)(b + 1), &stop, tab.wait)) {
            ok = false;
            break;
        }
    }
    if (p.nblocks > 1) ok = ok && *(volatile unsigned *)tab.wait.abort_flag == 0u;
    if (!ok) {
        const float2 nan2 = f2(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) cu[r][q][0] = cu[r][q][1] = nan2;
    }
    res_store_own<R>(t, g, cu, p.u, p.v);
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
    const int sms = sm_count();
    for (int r = kResMinR; r <= kResMaxR; ++r) {
        const int tiles = resident_tiles(H, W, r, &pl.ntx, &pl.nty);
        if (tiles > sms) continue;
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
    if (blockIdx.x == 0 && threadIdx.x == 0) *tab.wait.abort_flag = 0u;
    if (tiles == 1) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int h = 0; h < 2; ++h)
        for (int i = threadIdx.x; i < msgs; i += blockDim.x) p.box[(size_t)(h * tiles + tile) * msgs + i] = z;
}

// Launches the table (img, n, ckpt_* and wait filled in; every image tiled for r rows per
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
        tab.wait.abort_flag = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(scratch) + pl.box_bytes - 256);
    tab.wait.polls = kResPolls;
    return launch_table(tab, pl.r, zero_start, rc, s);
}

// ---- many images: groups whose tiles the SMs hold all at once, one launch each

// How the jobs, in their order, are cut into launches: launch k holds jobs end[k-1] .. end[k]-1
// with r[k] rows per warp.  A launch takes as long as its longest image, and a sweep of it
// base + slope * r us, whatever the number of tiles: tall tiles put more images into a launch, low
// ones spread an image over more SMs.  The cut that needs the least time in all (dynamic
// programming over the prefixes).  false if an image does not fit.
bool resident_cut(const ResidentJob *jobs, int n, double base, double slope, int max_r, ResidentCut &cut) {
    std::vector<double> cost(n + 1, -1.0);
    std::vector<int> from(n + 1, 0), rows(n + 1, 0);
    cost[0] = 0.0;
    // the tiles of every job at every height, formed once (n^2 of them, each asking for the device,
    // made 900 us of host time for 64 images); one more than the SMs where it does not fit
    const int sms = sm_count();
    std::vector<int> need((size_t)n * (max_r + 1));
    for (int j = 0; j < n; ++j)
        for (int r = kResMinR; r <= max_r; ++r) {
            int ntx, nty;
            const int t = resident_tiles(jobs[j].H, jobs[j].W, r, &ntx, &nty);
            need[(size_t)j * (max_r + 1) + r] =
                t <= sms && resident_box_bytes(t, r) <= jobs[j].scratch_bytes ? t : sms + 1;
        }
    for (int i = 0; i < n; ++i) {  // a launch that starts with job i
        if (cost[i] < 0.0) continue;
        for (int r = kResMinR; r <= max_r; ++r) {
            const double sweep = base + slope * r;
            int tiles = 0, longest = 0;
            for (int j = i; j < n && j < i + kMaxResImages; ++j) {
                tiles += need[(size_t)j * (max_r + 1) + r];
                if (tiles > sms) break;
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
                            const ResolvedConfig &rc, cudaStream_t s, int *launched, int polls) {
    *launched = 0;
    for (int i = 0; i < n; ++i)
        if (jobs[i].iters < 2) return HS_ERR_UNSUPPORTED;
    ResidentCut cut;
    // us per sweep, measured at 320x240 .. 1920x1080, r = 2 .. 8
    if (!resident_cut(jobs, n, rc.fast ? 0.65 : 0.5, rc.fast ? 0.22 : 0.52, kResMaxR, cut)) return HS_ERR_UNSUPPORTED;
    for (size_t g = 0; g < cut.end.size(); ++g) {
        const int i0 = g ? cut.end[g - 1] : 0, m = cut.end[g] - i0, r = cut.r[g];
        ResidentTable tab;
        memset(&tab, 0, sizeof(tab));
        tab.n = m;
        tab.ckpt_every = ckpt_every;
        tab.ckpt_plane = ckpt_plane;
        tab.wait.status = status;
        tab.wait.polls = polls;
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
                tab.wait.abort_flag = reinterpret_cast<unsigned *>(d.scratch + resident_box_bytes(tiles, r) - 256);
        }
        const hs_status st = launch_table(tab, r, true, rc, s);
        if (st != HS_OK) return st;
        *launched = i0 + m;
    }
    return HS_OK;
}

}  // namespace hs

using namespace hs;

extern "C" hs_status hs_wait_status(int *device_status, void *stream) {
    clear_error();
    if (!device_status) HS_FAIL(HS_ERR_INVALID_ARG, "device_status is NULL");
    wait_status_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(device_status, 1);
    HS_LAUNCH_CHECK("wait_status_kernel");
    return resident_adjoint_wait_status(device_status, (cudaStream_t)stream);
}
