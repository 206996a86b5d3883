"""Calls of the resident form beyond one plain image: outputs over images, mixed batches, several
launches, the backward at every tile height."""
import numpy as np
import pytest
import torch

from conftest import assert_bitexact
from resident_cases import CKPT, GROUPS, ITERS, SINGLE
from hindemith_b200 import _lib as L
from hindemith_b200 import device as D

pytestmark = pytest.mark.gpu


def images(shape, n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    p = D.empty_planes(n, *shape)
    for q in p:
        q.copy_(torch.rand(shape, device="cuda", generator=g))
    return [q for q in p]


def equal(a, b, what):
    assert_bitexact(a.detach().cpu().numpy(), b.detach().cpu().numpy(), what)


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("rows", [1, 40, -40])
def test_forward_writing_inside_its_images_memory(cuda, fast, rows):
    """The flow goes to a plane that begins `rows` rows behind (or before) the first image."""
    H, W = 480, 640
    I0, I1 = images((H, W), 2, 1)
    cfg = L.make_config(fast_math=fast)
    ru, rv = D.hs_forward(I0, I1, 1.0, 40, cfg)
    buf = torch.zeros((H + 2 * 40, W), device="cuda")
    a, u = buf[40:40 + H], buf[40 + rows:40 + rows + H]
    v = D.empty_plane(H, W)
    for _ in range(3):
        a.copy_(I0)
        D.hs_forward(a, I1, 1.0, 40, cfg, out=(u, v))
        equal(u, ru, "u")
        equal(v, rv, "v")


# ------------------------------------------------------------------ the backward's sums

def poisoned(n):
    """n bytes of NaN."""
    return torch.full((n,), 255, dtype=torch.uint8, device="cuda")


class SinglePair:
    """hs_forward_train and hs_backward on buffers of the test's own, whose parts it reads."""

    def __init__(self, H, W, iters, ckpt, cfg, seed):
        import ctypes

        self.lib, self.cfg, self.ct = L.lib(), ctypes.byref(cfg), ctypes
        self.H, self.W, self.ld, self.iters, self.ckpt = H, W, (W + 3) // 4 * 4, iters, ckpt
        self.I0, self.I1 = images((H, W), 2, seed)
        self.stride = (H * self.ld * 4 + 255) // 256 * 256
        self.alpha = torch.tensor([0.9], device="cuda")
        self.flow = images((H, W), 2, 0)
        u, v = self.flow
        nd = self.lib.hs_derivs_bytes(H, W, self.ld)
        nc = self.lib.hs_checkpoint_bytes(H, W, self.ld, iters, ckpt)
        nw = self.lib.hs_forward_train_workspace_bytes(H, W, self.ld)
        self.derivs, self.planes, ws = (poisoned(n) for n in (nd, nc, nw))
        L.check(self.lib.hs_forward_train(D.ptr(self.I0), D.ptr(self.I1), H, W, self.ld, D.ptr(self.alpha), iters, ckpt,
                                          D.ptr(u), D.ptr(v), D.ptr(self.derivs), D.ptr(self.planes), D.ptr(ws), nw,
                                          self.cfg, D.stream_handle()), "hs_forward_train")

    def plane(self, buf, k):
        b = buf[k * self.stride:k * self.stride + self.H * self.ld * 4].view(torch.float32)
        return b.view(self.H, self.ld)[:, :self.W]

    def backward(self, first, iters, ckpt, lu, lv, cfg=None):
        """The sweeps from checkpoint plane `first` on: (accumulators, lambda parked before the first
        interval, gradients)."""
        need = self.lib.hs_backward_workspace_bytes(self.H, self.W, self.ld, ckpt)
        ws = poisoned(need)
        out = images((self.H, self.W), 2, 0)
        da = torch.zeros(1, device="cuda")
        at = self.ct.c_void_p(self.planes.data_ptr() + 2 * first * self.stride)
        L.check(self.lib.hs_backward(D.ptr(self.derivs), self.H, self.W, self.ld, D.ptr(self.alpha), iters, ckpt, at, D.ptr(lu),
                                     D.ptr(lv), D.ptr(out[0]), D.ptr(out[1]), D.ptr(da), D.ptr(ws), need,
                                     self.cfg if cfg is None else self.ct.byref(cfg), D.stream_handle()), "hs_backward")
        lam = 4 * (ckpt - 1)
        return ([self.plane(ws, lam + 4 + i).clone() for i in range(3)],
                [D.as_plane(self.plane(ws, lam + i).clone()) for i in range(2)], [*out, da])


@pytest.mark.parametrize("ckpt", [1, 10, 100])
def test_backward_sums_no_further_off_than_the_passes_order(cuda, ckpt):
    """dIx, dIy, dIt over 100 sweeps: the same terms as 25 backwards of 4 sweeps each.  Against
    these added in 64 bits, the sums of one call are no further off than these added in 32 bits one
    after the other, the order of the streaming passes (10 % for the sample)."""
    H, W, n = 600, 800, 100
    cfg = L.make_config(fast_math=True)
    lam = images((H, W), 2, 7)
    four = SinglePair(H, W, n, 4, cfg, 3)
    one = SinglePair(H, W, n, ckpt, cfg, 3)
    got = one.backward(0, n, ckpt, *lam)[0]
    sum64, sum32 = [0.0] * 3, None
    l = lam
    for c in range(n // 4 - 1, -1, -1):
        acc = four.backward(c, 4, 4, *l)[0]
        sum64 = [s + a.double() for s, a in zip(sum64, acc)]
        sum32 = [s + a for s, a in zip(sum32, acc)] if sum32 else acc
        if c:
            l = four.backward(c - 1, 8, 4, *l)[1]
    for k in range(3):
        off = [float((s.double() - sum64[k]).norm()) for s in (got[k], sum32[k])]
        assert off[0] <= 1.1 * off[1], (k, off)


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("H,W,rows", SINGLE)
def test_single_pair_at_every_tile_height(cuda, H, W, rows, fast):
    """Forward and backward of one pair on the chip and in the passes, in all four combinations, on
    buffers full of NaN: the same flow bit for bit, gradients within 1e-5 of their norm."""
    auto, passes = L.make_config(fast_math=fast), L.make_config(fast_math=fast, sweeps_per_pass=4)
    lam = images((H, W), 2, 7)
    pairs = [SinglePair(H, W, ITERS, CKPT, cfg, 3) for cfg in (passes, auto)]
    for a, b in zip(pairs[0].flow, pairs[1].flow):
        equal(b, a, "flow")
    ref = pairs[0].backward(0, ITERS, CKPT, *lam, cfg=passes)[2]
    for p, cfg in ((pairs[0], auto), (pairs[1], passes), (pairs[1], auto)):
        for g, r in zip(p.backward(0, ITERS, CKPT, *lam, cfg=cfg)[2], ref):
            assert (g - r).norm() <= 1e-5 * r.norm()


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("shapes", [g[0] for g in GROUPS])
def test_training_batches_of_several_launches(cuda, shapes, fast):
    from hindemith_b200.autograd import horn_schunck_batch

    ims = [images(s, 2, 20 + i) for i, s in enumerate(shapes)]
    lam = [images(s, 2, 80 + i) for i, s in enumerate(shapes)]

    def run(cfg):
        nan = torch.full((1 << 28,), float("nan"), device="cuda")  # what the call's buffers hold
        del nan
        a = torch.tensor(0.8, device="cuda", requires_grad=True)
        xs = [tuple(t.clone().requires_grad_(True) for t in p) for p in ims]
        outs = [t for o in horn_schunck_batch(xs, a, ITERS, CKPT, cfg) for t in o]
        return outs, torch.autograd.grad(outs, [t for x in xs for t in x] + [a], [t for p in lam for t in p])

    (f0, g0), (f1, g1) = run(L.make_config(fast_math=fast)), run(L.make_config(fast_math=fast, sweeps_per_pass=4))
    for a, b in zip(f0, f1):
        equal(a, b, "flow")
    for a, b in zip(g0, g1):
        assert (a - b).norm() <= 1e-5 * b.norm()


# ------------------------------------------------------------------ the batched call's default

MIXED = [(1, 1, 1.0, 3), (7, 130, 0.5, 9), (65, 127, 1.7, 40), (300, 518, 0.8, 37), (130, 7, 1.2, 0), (240, 320, 2.0, 100),
         (480, 640, 0.6, 23), (33, 65, 1.0, 8), (200, 90, 0.9, 1), (3, 3000, 1.1, 9), (25, 121, 1.0, 2)]
BATCHES = {
    "mixed": MIXED,
    "with an image above 2 Mpx": MIXED[:4] + [(1100, 1925, 0.7, 9)] + MIXED[4:],
    "more than 32 small images": [(20 + 3 * k, 30 + 7 * k, 1.0, 4 + k % 5) for k in range(40)],
    "several launches": [(500, 701, 1.0, 12)] * 6 + [(900, 1301, 0.8, 7), (720, 1280, 1.3, 9)],
    "no sweep or one": [(40, 52, 1.0, 0), (41, 53, 1.0, 1)] * 5,
}


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("name", list(BATCHES))
def test_batch_by_default_equals_per_pair_passes(cuda, name, fast):
    """Eager and as a replayed graph, into outputs full of NaN."""
    from hindemith_b200.batched import BatchPlan

    specs = BATCHES[name]
    plan = BatchPlan(specs, L.make_config(fast_math=fast))
    refs = []
    for i, (H, W, alpha, iters) in enumerate(specs):
        for t, x in zip((plan.I0[i], plan.I1[i]), images((H, W), 2, 100 + i)):
            t.copy_(x)
        refs.append(D.hs_forward(plan.I0[i], plan.I1[i], alpha, iters, L.make_config(fast_math=fast, sweeps_per_pass=3, layout=1)))

    def run(go):
        for t in plan.u + plan.v:
            t.fill_(float("nan"))
        go()
        plan.check()
        for i, (ru, rv) in enumerate(refs):
            equal(plan.u[i], ru, f"u of pair {i}")
            equal(plan.v[i], rv, f"v of pair {i}")

    run(plan.run)
    plan.capture()
    for _ in range(2):
        run(plan.replay)


# ------------------------------------------------------------------ waits that run out

def test_waits_that_run_out_leave_nan_and_a_status(cuda):
    """Training on the chip with waits of 0 polls: tiles give up on one another, every wait ends, the
    flow and the gradients say so, and the calls after it are right."""
    import ctypes

    lib = L.lib()
    shapes = [(600, 799), (300, 402)]
    cfg = L.make_config(fast_math=True)
    planes = [images(s, 8, 40 + i) for i, s in enumerate(shapes)]
    alpha, dalpha = torch.tensor([0.9], device="cuda"), torch.zeros(2, device="cuda")
    arr = (L.hs_train_pair * 2)()
    for i, (d, p) in enumerate(zip(arr, planes)):
        d.I0, d.I1, d.u, d.v, d.dLdu, d.dLdv, d.dI0, d.dI1 = (t.data_ptr() for t in p)
        d.alpha, d.dalpha = alpha.data_ptr(), dalpha.data_ptr() + 4 * i
        d.H, d.W, d.ld = p[0].shape[0], p[0].shape[1], p[0].stride(0)
    need = lib.hs_train_workspace_bytes(arr, 2, ITERS, CKPT)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")

    def run(polls):
        L.check(lib.hs_selftest_resident_wait(arr, 2, ITERS, CKPT, D.ptr(ws), need, ctypes.byref(cfg), polls,
                                              D.stream_handle()), "hs_selftest_resident_wait")
        return [t.clone() for p in planes for t in (p[2], p[3], p[6], p[7])] + [dalpha.clone()]

    D.check_waits()
    ref = run(1 << 22)
    D.check_waits()
    assert all(torch.isfinite(t).all() for t in ref)
    out = run(0)
    with pytest.raises(L.HSError) as e:
        D.check_waits()
    assert e.value.status == L.HS_ERR_TIMEOUT
    assert any(torch.isnan(t).any() for t in out[:4]) and torch.isnan(out[-1]).any()
    D.check_waits()  # read once
    for a, b in zip(run(1 << 22), ref):
        equal(a, b, "the next call")
    D.check_waits()


def test_first_call_of_a_process_can_be_captured(cuda):
    """hs_forward and the batched call set their kernels up inside a capture, too."""
    import subprocess
    import sys

    code = """
import torch
from hindemith_b200 import _lib as L, device as D
a, b, u, v = (t for t in D.empty_planes(4, 300, 402))
a.copy_(torch.rand(300, 402)); b.copy_(torch.rand(300, 402))
D.workspace(L.lib().hs_forward_workspace_bytes(300, 402, 404), a.device)
s = torch.cuda.Stream()
with torch.cuda.stream(s):
    D.workspace(L.lib().hs_forward_workspace_bytes(300, 402, 404), a.device)
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    D.hs_forward(a, b, 1.0, 30, out=(u, v))
g.replay(); torch.cuda.synchronize()
x, y = D.hs_forward(a, b, 1.0, 30)
assert torch.equal(x, u) and torch.equal(y, v)
print("captured")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert "captured" in r.stdout, r.stderr[-2000:]
