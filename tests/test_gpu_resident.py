"""The resident form (an image held on the chip for all sweeps; hs_config left to the library)
against the streaming passes, bit for bit, and against the C oracle: every tile shape, image
sides at every position within a lane's four columns, one tile and many, both forms, from zero
and from a given state."""
import numpy as np
import pytest
import torch

from conftest import assert_bitexact
from hindemith_b200 import _lib as L
from hindemith_b200 import device as D
from oracle import hs_oracle as O

pytestmark = pytest.mark.gpu

# (H, W, sweeps): tiny, single tiles, the smallest two-tile images, ragged widths, and sizes that
# take each tile height on 148 SMs (16 warps x 2 .. 8 rows)
SHAPES = [(1, 1, 5), (1, 200, 7), (24, 120, 9), (25, 121, 2), (13, 500, 12), (31, 122, 3), (200, 30, 21),
          (65, 127, 40), (240, 320, 33), (300, 518, 37), (33, 1003, 16), (480, 642, 10), (600, 800, 9),
          (720, 1280, 9), (900, 1301, 8), (955, 1500, 6), (1000, 1498, 7), (1080, 1920, 9), (1037, 1901, 6)]


def planes(shape, n, pad=0, seed=0):
    H, W = shape
    rng = np.random.default_rng(seed + H * 7 + W)
    ld = (W + 3) // 4 * 4 + 4 * pad
    buf = torch.from_numpy(rng.standard_normal((n, H, ld)).astype(np.float32)).cuda()
    return [buf[i, :, :W] for i in range(n)]


def same(a, b, what):
    """Equal bits, NaN where the other is NaN."""
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert np.array_equal(np.isnan(a), np.isnan(b)), what
    m = ~np.isnan(a)
    assert_bitexact(a[m], b[m], what)


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("H,W,iters", SHAPES)
def test_resident_equals_streaming(cuda, H, W, iters, fast):
    stream = L.make_config(fast_math=fast, sweeps_per_pass=3, layout=1)
    auto = L.make_config(fast_math=fast)
    I0, I1 = planes((H, W), 2)
    u, v = D.hs_forward(I0, I1, 0.4, iters, auto)
    ru, rv = D.hs_forward(I0, I1, 0.4, iters, stream)
    same(u, ru, "u")
    same(v, rv, "v")
    # from a given state on padded rows; the columns beyond W stay as they are
    Ix, Iy, It, a, b = planes((H, W), 5, pad=1, seed=3)
    got = [t.as_strided((H, t.stride(0)), (t.stride(0), 1)).clone() for t in (a, b)]
    ref = [t.clone() for t in got]
    for pair, cfg in ((got, auto), (ref, stream)):
        D.hs_sweeps(Ix, Iy, It, 0.16, iters, pair[0][:, :W], pair[1][:, :W], cfg)
    same(got[0], ref[0], "u of hs_sweeps")
    same(got[1], ref[1], "v of hs_sweeps")


@pytest.mark.parametrize("H,W,iters", [(65, 127, 40), (517, 731, 21), (240, 320, 100)])
def test_resident_exact_equals_the_oracle(cuda, H, W, iters):
    I0, I1 = planes((H, W), 2, seed=5)
    u, v = D.hs_forward(I0, I1, 0.9, iters)
    ru, rv = O.c_hs_forward(I0.cpu().numpy(), I1.cpu().numpy(), np.float32(0.9), iters)
    assert_bitexact(u.cpu().numpy(), ru, "u")
    assert_bitexact(v.cpu().numpy(), rv, "v")


@pytest.mark.parametrize("iters", [0, 1, 2, 3, 4, 5, 8])
def test_resident_short_calls(cuda, iters):
    I0, I1 = planes((130, 250), 2, seed=iters)
    for fast in (True, False):
        u, v = D.hs_forward(I0, I1, 1.0, iters, L.make_config(fast_math=fast))
        ru, rv = D.hs_forward(I0, I1, 1.0, iters, L.make_config(fast_math=fast, sweeps_per_pass=1, layout=1))
        same(u, ru, "u")
        same(v, rv, "v")


def test_resident_nan_input_and_flat_image(cuda):
    I0, I1 = planes((150, 300), 2, seed=1)
    I0 = I0.clone()
    I0[70, 119:122] = float("nan")
    flat = torch.full((150, 300), 0.25, device="cuda")
    for a, b in ((I0, I1), (flat, flat)):
        for fast in (True, False):
            u, v = D.hs_forward(a, b, 1.0, 14, L.make_config(fast_math=fast))
            ru, rv = D.hs_forward(a, b, 1.0, 14, L.make_config(fast_math=fast, sweeps_per_pass=2, layout=1))
            same(u, ru, "u")
            same(v, rv, "v")


def test_resident_output_over_an_input(cuda):
    """hs_forward may write its flow over the images' own planes."""
    I0, I1 = planes((300, 700), 2, seed=2)
    ru, rv = D.hs_forward(I0, I1, 1.0, 20)
    a, b = D._like(I0), D._like(I1)
    a.copy_(I0)
    b.copy_(I1)
    D.hs_forward(a, b, 1.0, 20, out=(a, b))
    same(a, ru, "u")
    same(b, rv, "v")


def test_resident_streams_and_graph(cuda):
    """Calls of several streams at once, and a captured call replayed, give the plain results."""
    sizes = [(240, 320), (480, 640), (600, 800), (300, 500)]
    ins = [planes(s, 2, seed=10 + i) for i, s in enumerate(sizes)]
    refs = [D.hs_forward(a, b, 1.0, 60) for a, b in ins]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()
    for _ in range(3):
        outs = [D.hs_forward(a, b, 1.0, 60, stream=s) for (a, b), s in zip(ins, streams)]
    torch.cuda.synchronize()
    for (u, v), (ru, rv) in zip(outs, refs):
        same(u, ru, "u")
        same(v, rv, "v")
    a, b = ins[1]
    out = D.empty_planes(2, *sizes[1])
    s = streams[1]
    with torch.cuda.stream(s):
        D.hs_forward(a, b, 1.0, 60, out=(out[0], out[1]))
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            D.hs_forward(a, b, 1.0, 60, out=(out[0], out[1]))
    for _ in range(3):
        out.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        same(out[0], refs[1][0], "u")
        same(out[1], refs[1][1], "v")


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("shapes,iters,ckpt", [([(24, 31), (70, 130), (300, 401), (1, 9)], 23, 7),
                                               ([(300, 500)] * 7, 12, 5), ([(250, 130)], 9, 4),
                                               ([(40, 50), (130, 40)], 2, 1)])
def test_resident_training_equals_streaming(cuda, shapes, iters, ckpt, fast):
    """The training forward on the chip (one launch for many images, several groups of them)
    keeps the same checkpoints: flows and gradients equal those of the streaming passes."""
    from hindemith_b200.autograd import horn_schunck, horn_schunck_batch

    ims = [planes(s, 2, seed=50 + i) for i, s in enumerate(shapes)]
    lam = [planes(s, 2, seed=90 + i) for i, s in enumerate(shapes)]

    def run(cfg):
        a = torch.tensor(0.8, device="cuda", requires_grad=True)
        xs = [tuple(t.clone().requires_grad_(True) for t in p) for p in ims]
        outs = ([horn_schunck(*xs[0], a, iters, ckpt, cfg)] if len(xs) == 1 else
                horn_schunck_batch(xs, a, iters, ckpt, cfg))
        loss = sum((u * p).sum() + (v * q).sum() for (u, v), (p, q) in zip(outs, lam))
        return [t for o in outs for t in o], torch.autograd.grad(loss, [t for x in xs for t in x] + [a])

    (f0, g0), (f1, g1) = run(L.make_config(fast_math=fast)), run(L.make_config(fast_math=fast, sweeps_per_pass=4))
    for a, b in zip(f0, f1):
        same(a.detach(), b.detach(), "flow")
    for a, b in zip(g0, g1):
        assert (a - b).norm() <= 1e-5 * b.norm(), "gradient"


@pytest.mark.parametrize("shape", [(1811, 2048), (1650, 2003), (2600, 1282)])
@pytest.mark.parametrize("T", range(1, 9))
def test_wide_passes_with_the_ring_in_tensor_memory(cuda, shape, T):
    """From 3.3 Mpx up the wide layout keeps its coefficient ring in tensor memory: equal to the
    2-column layout bit for bit, at W % 4 = 0, 3 and 2, with partial last passes."""
    H, W = shape
    assert H * W >= 3300000
    Ix, Iy, It, a, b = planes(shape, 5, seed=T)
    got, ref = [a.clone(), b.clone()], [a.clone(), b.clone()]
    for pair, layout in ((got, 2), (ref, 1)):
        pair[:] = [D.as_plane(t) for t in pair]
        D.hs_sweeps(Ix, Iy, It, 0.3, 2 * T + 1, *pair, L.make_config(fast_math=True, sweeps_per_pass=T, layout=layout))
    same(got[0], ref[0], "u")
    same(got[1], ref[1], "v")


@pytest.mark.parametrize("scale", [1e-30, 1e-20, 1e-12, 1e-6, 1.0, 1e6, 1e12, 1e18])
@pytest.mark.parametrize("alpha", [0.0, 1e-18, 1e-7, 1e-3, 1.0, 1e6, 1e12])
def test_resident_exact_division_over_the_float_range(cuda, scale, alpha):
    """The exact form's quotient equals the IEEE division of the streaming passes wherever its
    numerators and denominators lie: tiny, huge, zero and non-finite ones included."""
    I0, I1 = planes((70, 260), 2, seed=7)
    I0, I1 = D.as_plane(I0 * scale), D.as_plane(I1 * scale)
    I0[30:40, 50:90] = 0.5 * scale  # a flat patch: zero derivatives
    I1[30:40, 50:90] = 0.5 * scale
    with np.errstate(all="ignore"):
        u, v = D.hs_forward(I0, I1, alpha, 13)
        ru, rv = D.hs_forward(I0, I1, alpha, 13, L.make_config(sweeps_per_pass=2, layout=1))
    same(u, ru, "u")
    same(v, rv, "v")
