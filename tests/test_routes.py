"""Which kernels a call takes, on a CPU: the library's host code on a recording CUDA runtime
(fake_cuda).  Pointers are only numbers here."""
import ctypes

import pytest

from fake_cuda import fake_cuda
from hindemith_b200 import _lib as L

P = ctypes.c_void_p
MB = 1 << 20
WS = 1 << 40  # a workspace far from all planes


@pytest.fixture()
def fake():
    return fake_cuda()


def pad(W):
    return (W + 3) // 4 * 4


def forward(fake, H, W, iters, I0, I1, u, v, cfg=None):
    cfg = cfg if cfg is not None else L.make_config(fast_math=True)
    ld = pad(W)
    need = fake.lib.hs_forward_workspace_bytes(H, W, ld)
    assert fake.lib.hs_forward(P(I0), P(I1), H, W, ld, 1.0, iters, P(u), P(v), P(WS), need, ctypes.byref(cfg), None) == L.HS_OK
    return fake.launches()


def batch(fake, specs, cfg=None, planes=None):
    """hs_forward_batched of (H, W, iters) pairs; planes[i] = (I0, I1, u, v), else all apart."""
    cfg = cfg if cfg is not None else L.make_config(fast_math=True)
    arr = (L.hs_pair_desc * len(specs))()
    for i, (d, (H, W, iters)) in enumerate(zip(arr, specs)):
        at = planes[i] if planes else [(1 << 36) + (4 * i + k) * 64 * MB for k in range(4)]
        d.I0, d.I1, d.u, d.v = at
        d.H, d.W, d.ld, d.alpha, d.iters = H, W, pad(W), 1.0, iters
    need = fake.lib.hs_forward_batched_workspace_bytes(arr, len(specs), ctypes.byref(cfg))
    assert need > 0
    assert fake.lib.hs_forward_batched(arr, len(specs), P(WS), need, ctypes.byref(cfg), None, None) == L.HS_OK
    return fake.launches()


def train_pairs(shapes, planes=None):
    arr = (L.hs_train_pair * len(shapes))()
    for i, (d, (H, W)) in enumerate(zip(arr, shapes)):
        at = planes[i] if planes else [(1 << 36) + (8 * i + k) * 64 * MB for k in range(4)]
        d.I0, d.I1, d.u, d.v = at
        base = (1 << 37) + 8 * i * 64 * MB
        d.dLdu, d.dLdv, d.dI0, d.dI1 = (base + k * 64 * MB for k in range(4))
        d.alpha, d.dalpha = 1 << 35, (1 << 35) + 256 + 4 * i
        d.H, d.W, d.ld = H, W, pad(W)
    return arr


def train(fake, shapes, iters, ckpt, cfg=None, planes=None, backward=False):
    cfg = cfg if cfg is not None else L.make_config(fast_math=True)
    arr = train_pairs(shapes, planes)
    need = fake.lib.hs_train_workspace_bytes(arr, len(shapes), iters, ckpt)
    call = fake.lib.hs_backward_batched if backward else fake.lib.hs_forward_train_batched
    assert call(arr, len(shapes), iters, ckpt, P(WS), need, ctypes.byref(cfg), None) == L.HS_OK
    return fake.launches()


def kernels(launches):
    return {x.kernel for x in launches}


# ------------------------------------------------------------------ outputs over images

A, B, C, D = ((k + 1) << 32 for k in range(4))


@pytest.mark.parametrize("u,v,resident", [(C, D, True), (A, B, True), (B, A, True), (A, C, True),
                                          (A + 1280, C, False), (C, B - 1280, False), (A - 480 * 640 * 4, B + 480 * 640 * 4, True),
                                          (A - 480 * 640 * 4 + 16, C, False)])
def test_forward_with_an_output_inside_an_image(fake, u, v, resident):
    """In the place of an image, or apart: on the chip.  At an offset: the passes, which have read
    all of the images before they write."""
    ks = kernels(forward(fake, 480, 640, 20, A, B, u, v))
    assert ("hs_resident_kernel" in ks) == resident
    assert ("derivs_kernel" in ks) == (not resident)


def test_batch_with_an_output_over_another_pairs_image(fake):
    """Frames of a sequence, the flow of pair 0 over a frame that pair 1 reads: no pair may write
    before all have read."""
    H, W = 240, 320
    frames = [(1 << 36) + k * 64 * MB for k in range(3)]
    out = [(1 << 37) + k * 64 * MB for k in range(4)]
    pairs = [(frames[0], frames[1], out[0], frames[1]), (frames[1], frames[2], out[2], out[3])]
    apart = [(frames[0], frames[1], out[0], out[1]), (frames[1], frames[2], out[2], out[3])]
    own = [(frames[0], frames[1], frames[0], out[1]), (frames[1], frames[2], out[2], frames[2])]
    assert "batch_derivs_kernel" in kernels(batch(fake, [(H, W, 20)] * 2, planes=pairs))
    for ok in (apart, own):
        fake.reset()
        assert kernels(batch(fake, [(H, W, 20)] * 2, planes=ok)) == {"res_clear_kernel", "hs_resident_kernel"}


def test_training_forward_with_an_output_over_another_pairs_image(fake):
    H, W = 240, 320
    frames = [(1 << 36) + k * 64 * MB for k in range(3)]
    out = [(1 << 38) + k * 64 * MB for k in range(4)]
    pairs = [(frames[0], frames[1], out[0], frames[2]), (frames[1], frames[2], out[2], out[3])]
    apart = [(frames[0], frames[1], out[0], out[1]), (frames[1], frames[2], out[2], out[3])]
    ks = kernels(train(fake, [(H, W)] * 2, 20, 5, planes=pairs))
    assert "derivs_kernel" in ks and "hs_resident_kernel" not in ks
    fake.reset()
    assert "hs_resident_kernel" in kernels(train(fake, [(H, W)] * 2, 20, 5, planes=apart))


# ------------------------------------------------------------------ fewer SMs than the device has

def in_place(n):
    """Pairs whose flow takes the place of their images."""
    at = [((1 << 36) + 2 * i * 64 * MB, (1 << 36) + (2 * i + 1) * 64 * MB) for i in range(n)]
    return [(a, b, a, b) for a, b in at]


def refused_from(ls, planes):
    """The first pair of the first refused launch, after at least one that was made."""
    ls = [x for x in ls if x.kernel == "hs_resident_kernel"]
    assert [x.refused for x in ls[:2]] == [False, True]
    return [at[0] for at in planes].index(ls[1].first)


def test_batch_redoes_only_what_was_not_launched(fake):
    """Two launches of different size on a device that holds the first one's tiles only: the pairs
    of the first have their flow where their images were, and are not read again."""
    specs = [(500, 700, 40)] * 6 + [(900, 1300, 30)]
    planes = in_place(len(specs))
    tiles = [x.grid for x in batch(fake, specs, planes=planes) if x.kernel == "hs_resident_kernel"]
    assert len(tiles) == 2 and tiles[0] < tiles[1]
    fake.reset(max_cooperative_blocks=tiles[0])
    ls = batch(fake, specs, planes=planes)
    k = refused_from(ls, planes)
    again = [x.first for x in ls if not x.refused and x.kernel in ("derivs_kernel", "hs_resident_kernel")][1:]
    assert k > 0 and again == [at[0] for at in planes[k:]]


def test_training_forward_redoes_only_what_was_not_launched(fake):
    shapes = [(500, 700)] * 6 + [(900, 1300)]
    planes = in_place(len(shapes))
    tiles = [x.grid for x in train(fake, shapes, 40, 10, planes=planes) if x.kernel == "hs_resident_kernel"]
    assert len(tiles) == 2 and tiles[0] < tiles[1]
    fake.reset(max_cooperative_blocks=tiles[0])
    ls = train(fake, shapes, 40, 10, planes=planes)
    k = refused_from(ls, planes)
    assert k > 0 and [x.first for x in ls if x.kernel == "derivs_kernel"] == [at[0] for at in planes[k:]]


# ------------------------------------------------------------------ host work of a batch

@pytest.mark.parametrize("n,H,W", [(64, 64, 64), (128, 240, 320)])
def test_batch_planning_asks_for_the_device_a_few_times_per_pair(fake, n, H, W):
    batch(fake, [(H, W, 100)] * n)
    assert fake.lib.fake_queries() <= 8 * n


def test_training_planning_asks_for_the_device_a_few_times_per_pair(fake):
    for backward in (False, True):
        fake.reset()
        train(fake, [(128, 128)] * 32, 50, 5, backward=backward)
        assert fake.lib.fake_queries() <= 8 * 32


# ------------------------------------------------------------------ pairs that do not run on the chip

@pytest.mark.parametrize("specs,most", [([(16, 16, 0)] * 64, 1), ([(64, 64, 1)] * 64, 1 + 64),
                                        ([(3, 3000, 9)] * 12, 3 + 12), ([(8, 20000, 8)] * 12, 3),
                                        ([(240, 320, 50), (64, 64, 0), (300, 400, 1), (2200, 2000, 14)], 2 + 3 + 2)])
def test_batch_of_pairs_without_a_resident_form_shares_its_launches(fake, specs, most):
    """No sweep or one, images whose exchange their scratch does not hold or whose shape cuts into
    more tiles than SMs: one derivative launch and the persistent kernel for all of them, and a
    launch per remainder of the depth."""
    ls = batch(fake, specs)
    assert len(ls) <= most
    assert sum(x.kernel == "batch_derivs_kernel" for x in ls) == 1
    assert sum(x.kernel == "derivs_kernel" for x in ls) == sum(H * W > 4e6 for H, W, _ in specs)


def test_batch_of_large_pairs_and_small_ones_does_each_once(fake):
    """Every pair in exactly one of the three ways."""
    specs = [(2200, 2000, 14), (240, 320, 50), (3, 3000, 9), (16, 16, 0)]
    ls = batch(fake, specs)
    at = [(1 << 36) + 4 * i * 64 * MB for i in range(4)]
    assert [x.first for x in ls if x.kernel == "derivs_kernel"] == at[:1]
    assert [x.first for x in ls if x.kernel == "hs_resident_kernel"] == at[1:2]
    assert [x.first for x in ls if x.kernel == "batch_derivs_kernel"] == at[2:3]


# ------------------------------------------------------------------ rows per work item

def pass_items(f, H, W, cfg, T):
    """Work items of the passes of 2 T sweeps (one warp each)."""
    ld = pad(W)
    need = f.lib.hs_sweeps_workspace_bytes(H, W, ld)
    planes = [P((1 << 36) + k * 256 * MB) for k in range(5)]
    f.reset()
    assert f.lib.hs_sweeps(*planes[:3], H, W, ld, 1.0, 2 * T, *planes[3:], P(WS), need, ctypes.byref(cfg), None) == L.HS_OK
    out = {x.grid * (x.threads // 32) for x in f.launches()}
    assert len(out) == 1
    return out.pop()


@pytest.mark.parametrize("held", [8, 12, 16, 19, 28])
@pytest.mark.parametrize("H,W", [(1080, 1920), (1811, 2048), (2160, 3840), (64, 30000)])
@pytest.mark.parametrize("T", [1, 5, 7])
@pytest.mark.parametrize("layout", [1, 2])
def test_passes_fill_the_warps_the_kernel_holds(held, H, W, T, layout):
    """Items for 16 warps per SM (4 columns per lane: 12, 8 beyond depth 4) where the SMs hold them
    at once, else as many as they hold in whole strips; a kernel never holds less than its launch
    bound."""
    f = fake_cuda(held)
    bound = (12 if T <= 4 else 8) if layout == 2 else (16 if T <= 4 else 12 if T <= 6 else 8)
    want = bound if layout == 2 else 16
    slots = max(held, bound) * 148
    strips = -(-W // (128 - 2 * ((T + 3) // 4 * 4))) if layout == 2 else -(-W // (64 - 2 * (T + T % 2)))
    items = pass_items(f, H, W, L.make_config(fast_math=True, sweeps_per_pass=T, layout=layout), T)
    items -= items % strips  # (the last CTA of four warps may not be full)
    seg = lambda n: -(-H // max(-(-H // n), 2 * T, 8))
    full = seg(-(-148 * want // strips))
    assert items == strips * (full if full * strips <= slots else seg(max(1, slots // strips)))


def test_training_passes_fill_the_warps_the_kernel_holds():
    """Two intervals' recompute passes of 16 x 512^2: 16 warps per SM where they are held."""
    for held, most in ((16, 16 * 148), (12, 12 * 148)):
        f = fake_cuda(held)
        ls = train(f, [(512, 512)] * 16, 20, 10, cfg=L.make_config(fast_math=True, sweeps_per_pass=5), backward=True)
        items = {x.grid * (x.threads // 32) for x in ls if x.kernel == "hs_table_pass_kernel" and x.args[0] == 5}
        assert len(items) == 1 and 0.75 * most < items.pop() <= most


@pytest.mark.parametrize("T,rows,kernel", [(2, 0, "hs_stream_tm_kernel"), (2, 64, "hs_stream_w_kernel"), (3, 64, "hs_stream_w_kernel"),
                                           (2, 128, "hs_stream_tm_kernel"), (2, 32, "hs_stream_tm_kernel"),
                                           (1, 64, "hs_stream_tm_kernel"), (4, 64, "hs_stream_tm_kernel")])
def test_large_images_at_small_depths_avoid_a_small_second_wave(T, rows, kernel):
    f = fake_cuda(12)
    H = W = 4096
    need = f.lib.hs_sweeps_workspace_bytes(H, W, W)
    planes = [P((1 << 36) + k * 256 * MB) for k in range(5)]
    cfg = L.make_config(fast_math=True, sweeps_per_pass=T, layout=2, rows_per_segment=rows)
    assert f.lib.hs_sweeps(*planes[:3], H, W, W, 1.0, 2 * T, *planes[3:], P(WS), need, ctypes.byref(cfg), None) == L.HS_OK
    assert kernels(f.launches()) == {kernel}


# ------------------------------------------------------------------ the backward's two ways

def single(fake, H, W, iters, ckpt, fast):
    """Kernels of hs_backward for one pair."""
    cfg = L.make_config(fast_math=fast)
    ld = pad(W)
    need = fake.lib.hs_backward_workspace_bytes(H, W, ld, ckpt)
    a = [P((1 << 36) + k * 64 * MB) for k in range(8)]
    fake.reset()
    assert fake.lib.hs_backward(a[0], H, W, ld, a[1], iters, ckpt, a[2], a[3], a[4], a[5], a[6], a[7], P(WS), need,
                                ctypes.byref(cfg), None) == L.HS_OK
    return fake.launches()


# measured on B200, us: the passes against the chip (in brackets the one not taken)
@pytest.mark.parametrize("shapes,iters,ckpt,fast,resident", [
    ([(240, 320)], 200, 10, True, False),         # 948 (1065)
    ([(240, 320)], 200, 10, False, True),         # (1368) 1310
    ([(64, 64)] * 2, 200, 10, True, False),       # 4.98 (5.68) a sweep
    ([(128, 128)] * 2, 200, 10, True, False),     # 959 (1101)
    ([(512, 512)] * 8, 50, 5, True, False),       # 1066 (1275)
    ([(512, 512)] * 16, 50, 5, True, False),      # 2037 (2529)
    ([(512, 512)] * 16, 50, 5, False, False),     # 2564 (3042)
    ([(600, 800)], 100, 1, True, False),          # 603 (977): no recompute in the passes
    ([(512, 512)] * 4, 100, 1, False, False),     # 809 (1837)
    ([(437, 613)], 100, 10, False, True),         # (1044) 860
    ([(256, 256)] * 4, 200, 10, True, True),      # (1885) 760
    ([(512, 512)] * 2, 200, 10, True, True),      # (2260) 1094
    ([(512, 512)] * 4, 100, 16, False, True),     # (1996) 1449
    ([(128, 128)] * 32, 200, 10, True, True),     # (2746) 1562
])
def test_backward_takes_the_faster_way(fake, shapes, iters, ckpt, fast, resident):
    if len(shapes) == 1:
        ls = single(fake, *shapes[0], iters, ckpt, fast)
    else:
        ls = train(fake, shapes, iters, ckpt, cfg=L.make_config(fast_math=fast), backward=True)
    assert ("hs_resident_adj_kernel" in kernels(ls)) == resident
    assert ("hs_adjoint_pass_kernel" in kernels(ls)) == (not resident)


# ------------------------------------------------------------------ what the GPU tests of training reach

@pytest.mark.parametrize("fast", [True, False])
def test_training_cases_take_their_tile_heights(fake, fast):
    from resident_cases import CKPT, GROUPS, ITERS, SINGLE

    cfg = L.make_config(fast_math=fast)
    for H, W, rows in SINGLE:
        assert [x.args for x in single(fake, H, W, ITERS, CKPT, fast) if x.kernel == "hs_resident_adj_kernel"] == [(fast, rows)]
    assert {rows for _, _, rows in SINGLE} == {2, 3, 4, 5, 6}
    for shapes, forward_rows, backward_rows in GROUPS:
        for name, back, rows in (("hs_resident_kernel", False, forward_rows), ("hs_resident_adj_kernel", True, backward_rows)):
            fake.reset()
            ls = train(fake, shapes, ITERS, CKPT, cfg=cfg, backward=back)
            assert [x.args[-1] for x in ls if x.kernel == name] == rows


# ------------------------------------------------------------------ the wait status

def test_wait_status_argument_checks():
    lib = L.lib()
    assert lib.hs_wait_status(None, None) == L.HS_ERR_INVALID_ARG
    arr = train_pairs([(300, 402)])
    need = lib.hs_train_workspace_bytes(arr, 1, 20, 5)
    cfg = ctypes.byref(L.make_config())
    assert lib.hs_selftest_resident_wait(arr, 1, 20, 5, P(WS), need, cfg, -1, None) == L.HS_ERR_INVALID_ARG
    assert lib.hs_selftest_resident_wait(arr, 1, 20, 5, P(WS), need, cfg, (1 << 22) + 1, None) == L.HS_ERR_INVALID_ARG
    assert lib.hs_selftest_resident_wait(arr, 1, 20, 5, P(WS), need - 1, cfg, 0, None) == L.HS_ERR_WORKSPACE
    assert lib.hs_selftest_resident_wait(arr, 1, 20, 5, P(WS + 16), need, cfg, 0, None) == L.HS_ERR_ALIGNMENT
    arr[0].dLdu = None
    assert lib.hs_selftest_resident_wait(arr, 1, 20, 5, P(WS), need, cfg, 0, None) == L.HS_ERR_INVALID_ARG


def test_wait_status_asks_both_directions(fake):
    assert fake.lib.hs_wait_status(P(1 << 36), None) == L.HS_OK
    assert [x.first for x in fake.launches()] == [1 << 36] * 2


# ------------------------------------------------------------------ what the benchmark reports

@pytest.mark.parametrize("H,W", [(16, 16), (240, 320), (480, 640), (1080, 1920), (1100, 1925), (2048, 2048), (3, 3000), (20000, 60)])
@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("T,layout", [(0, 0), (0, 1), (3, 0), (5, 1), (7, 2)])
def test_benchmark_names_the_launches_of_its_step(fake, H, W, fast, T, layout):
    """Launches, kernel and depth as hs_forward makes them, at every size and with every tuning."""
    import bench

    if layout == 2 and not fast:
        pytest.skip("the exact form has 2 columns per lane")
    cfg = L.make_config(sweeps_per_pass=T, fast_math=fast, layout=layout)
    ls = forward(fake, H, W, 500, A, B, C, D, cfg)
    launches, kernel, chip = bench.sweep_launches(fake.lib, H, W, pad(W), 500, cfg)
    sweeps = [x for x in ls if x.kernel.startswith(("hs_resident", "hs_stream"))]
    assert (len(sweeps), chip) == (launches, sweeps[0].kernel == "hs_resident_kernel")
    if chip:
        assert len(ls) == 1 and kernel == "hs_resident_kernel"
    else:
        args = ",".join([str(sweeps[0].args[0])] + ["true" if a else "false" for a in sweeps[0].args[1:]])
        assert kernel == f"{sweeps[0].kernel}<{args}>"


def test_sweeps_per_launch_argument_checks():
    q = L.lib().hs_sweeps_per_launch
    cfg = L.make_config()
    assert q(0, 8, 8, 5, ctypes.byref(cfg)) == 0
    assert q(8, 8, 6, 5, ctypes.byref(cfg)) == 0
    assert q(8, 8, 8, -1, ctypes.byref(cfg)) == 0
    assert q(8, 8, 8, 5, ctypes.byref(L.make_config(sweeps_per_pass=9))) == 0
    assert q(8, 8, 8, 1, ctypes.byref(cfg)) == 4
    assert q(8, 8, 8, 50, ctypes.byref(L.make_config(sweeps_per_pass=3))) == 3
