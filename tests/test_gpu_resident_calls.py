"""Calls of the resident form beyond one plain image: outputs over images, mixed batches, several
launches, the backward at every tile height."""
import numpy as np
import pytest
import torch

from conftest import assert_bitexact
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

class SinglePair:
    """hs_forward_train and hs_backward on buffers of the test's own, whose parts it reads."""

    def __init__(self, H, W, iters, ckpt, cfg, seed):
        import ctypes

        self.lib, self.cfg, self.ct = L.lib(), ctypes.byref(cfg), ctypes
        self.H, self.W, self.ld, self.iters, self.ckpt = H, W, (W + 3) // 4 * 4, iters, ckpt
        self.I0, self.I1 = images((H, W), 2, seed)
        self.stride = (H * self.ld * 4 + 255) // 256 * 256
        self.alpha = torch.tensor([0.9], device="cuda")
        u, v = images((H, W), 2, 0)
        nd = self.lib.hs_derivs_bytes(H, W, self.ld)
        nc = self.lib.hs_checkpoint_bytes(H, W, self.ld, iters, ckpt)
        nw = self.lib.hs_forward_train_workspace_bytes(H, W, self.ld)
        self.derivs, self.planes, ws = (torch.zeros(n, dtype=torch.uint8, device="cuda") for n in (nd, nc, nw))
        L.check(self.lib.hs_forward_train(D.ptr(self.I0), D.ptr(self.I1), H, W, self.ld, D.ptr(self.alpha), iters, ckpt,
                                          D.ptr(u), D.ptr(v), D.ptr(self.derivs), D.ptr(self.planes), D.ptr(ws), nw,
                                          self.cfg, D.stream_handle()), "hs_forward_train")

    def plane(self, buf, k):
        b = buf[k * self.stride:k * self.stride + self.H * self.ld * 4].view(torch.float32)
        return b.view(self.H, self.ld)[:, :self.W]

    def backward(self, first, intervals, iters, ckpt, lu, lv):
        """The sweeps from checkpoint plane `first` on; (accumulators, lambda parked before the first
        interval)."""
        need = self.lib.hs_backward_workspace_bytes(self.H, self.W, self.ld, ckpt)
        ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
        out = images((self.H, self.W), 2, 0)
        da = torch.zeros(1, device="cuda")
        at = self.ct.c_void_p(self.planes.data_ptr() + 2 * first * self.stride)
        L.check(self.lib.hs_backward(D.ptr(self.derivs), self.H, self.W, self.ld, D.ptr(self.alpha), iters, ckpt, at, D.ptr(lu),
                                     D.ptr(lv), D.ptr(out[0]), D.ptr(out[1]), D.ptr(da), D.ptr(ws), need, self.cfg,
                                     D.stream_handle()), "hs_backward")
        lam = 4 * (ckpt - 1)
        return ([self.plane(ws, lam + 4 + i).clone() for i in range(3)],
                [D.as_plane(self.plane(ws, lam + i).clone()) for i in range(2)])


@pytest.mark.parametrize("ckpt", [1, 100])
def test_backward_sums_no_further_off_than_the_passes_order(cuda, ckpt):
    """dIx, dIy, dIt over 100 sweeps: the same terms as 25 backwards of 4 sweeps each.  Against
    these added in 64 bits, the sums of one call are no further off than these added in 32 bits one
    after the other, the order of the streaming passes (10 % for the sample)."""
    H, W, n = 600, 800, 100
    cfg = L.make_config(fast_math=True)
    lam = images((H, W), 2, 7)
    four = SinglePair(H, W, n, 4, cfg, 3)
    one = SinglePair(H, W, n, ckpt, cfg, 3)
    got, _ = one.backward(0, n // ckpt, n, ckpt, *lam)
    sum64, sum32 = [0.0] * 3, None
    l = lam
    for c in range(n // 4 - 1, -1, -1):
        acc, _ = four.backward(c, 1, 4, 4, *l)
        sum64 = [s + a.double() for s, a in zip(sum64, acc)]
        sum32 = [s + a for s, a in zip(sum32, acc)] if sum32 else acc
        if c:
            l = four.backward(c - 1, 2, 8, 4, *l)[1]
    for k in range(3):
        off = [float((s.double() - sum64[k]).norm()) for s in (got[k], sum32[k])]
        assert off[0] <= 1.1 * off[1], (k, off)


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
