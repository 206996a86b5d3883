"""Performance cases of the Horn-Schunck path: what a program using this package has it do,
called through the package's public entry points.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges.  For a case,
``prepare`` makes the inputs (and the plan or handle a program would keep), ``run`` does one
pass and returns its outputs whole, ``work`` gives the bytes and operations the pass cannot do
without and ``exact`` the outputs in 64-bit arithmetic, by plain torch.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from hindemith_b200 import hm, hs_average_stencil, hs_derivative_stencils, make_config, synthetic
from hindemith_b200 import device as D
from hindemith_b200 import flow as FL
from hindemith_b200.autograd import horn_schunck, horn_schunck_batch
from hindemith_b200.batched import BatchPlan
from hindemith_b200.cg import hs_matrix_powers
from hindemith_b200.loss import mean_epe_batch
from hindemith_b200.pyramid import coarse_to_fine

# operations per pixel: one Jacobi sweep (two 3x3 averages with shared weights, the residual
# and the update), its adjoint with the gradient terms, one power of the linear operator
SWEEP_FLOPS = 27
ADJOINT_FLOPS = 45
POWER_FLOPS = 25


def listed():
    return [
        # the smallest frame of the batch workload, one quick call: launches and latency count
        dict(name="forward_240x320", kind="forward", H=240, W=320, iters=100, fast=True, alpha=1.0),
        # the default (bit-exact) form on a VGA frame
        dict(name="forward_480x640_exact", kind="forward", H=480, W=640, iters=200, fast=False, alpha=1.0),
        # the headline: one full HD pair, 500 sweeps
        dict(name="forward_1080x1920", kind="forward", H=1080, W=1920, iters=500, fast=True, alpha=1.0),
        # an odd, ragged frame (rows not a multiple of 16 bytes) in the default form
        dict(name="forward_1037x1901_exact", kind="forward", H=1037, W=1901, iters=200, fast=False, alpha=0.7),
        # a large frame
        dict(name="forward_2048x2048", kind="forward", H=2048, W=2048, iters=200, fast=True, alpha=1.5),
        # the drop-in surface: the program as a Hindemith user writes it, default form
        dict(name="hm_480x640", kind="hm", H=480, W=640, iters=200, fast=False, alpha=1.0),
        # a served batch of pairs of mixed sizes, weights and sweep counts (one graph replay)
        dict(name="batch_16_mixed", kind="batch", n=16, specs=2024, fast=True),
        # a training step of 16 crops: loss, backward, gradients of images and alpha
        dict(name="train_16x512x512", kind="train", n=16, H=512, W=512, iters=200, ckpt=10, fast=True, alpha=1.0),
        # one ragged pair through the single-pair differentiable call, default form
        dict(name="train_437x613_exact", kind="train", n=1, H=437, W=613, iters=100, ckpt=10, fast=False, alpha=0.8),
        # large displacements: coarse to fine with the reverse mode through all levels
        dict(name="pyramid_2x1024x1024", kind="pyramid", n=2, H=1024, W=1024, levels=4, iters=100, fast=True, alpha=1.0),
        # the linear-system form: Krylov basis of an s-step solver
        dict(name="powers_2048x2048", kind="powers", H=2048, W=2048, steps=9),
        # the local method on the same substrate
        dict(name="lk_1080x1920", kind="lk", H=1080, W=1920, radius=5),
    ]


def _size(rng, lo, hi):
    """(H, W) with lo..hi pixels, spread over the logarithm, aspect 1:2 to 2:1, odd sizes too."""
    px = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    r = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
    return max(16, round(math.sqrt(px / r))), max(16, round(math.sqrt(px * r)))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "hm", "batch", "train", "train", "pyramid", "powers", "lk"])
    alpha = round(rng.uniform(0.5, 2.0), 3)
    if kind == "forward":
        H, W = _size(rng, 240 * 320, 2048 * 2048)
        iters = min(rng.choice([50, 100, 200, 500]) + rng.randrange(4), 10 ** 9 // (H * W))
        return dict(kind=kind, H=H, W=W, iters=iters, fast=rng.random() < 0.5, alpha=alpha)
    if kind == "hm":
        H, W = _size(rng, 240 * 320, 1080 * 1920)
        return dict(kind=kind, H=H, W=W, iters=200, fast=rng.random() < 0.3, alpha=alpha)
    if kind == "batch":
        return dict(kind=kind, n=rng.randrange(3, 14), specs=rng.randrange(10 ** 6), fast=rng.random() < 0.7)
    if kind == "train":
        n = rng.choice([1, 1, 2, 4, 8, 16])
        H, W = _size(rng, 128 * 128, min(16 * 512 * 512 // n, 1080 * 1920))
        return dict(kind=kind, n=n, H=H, W=W, iters=rng.choice([50, 100, 137, 200]), ckpt=rng.choice([5, 10, 16]),
                    fast=rng.random() < 0.6, alpha=alpha)
    if kind == "pyramid":
        n = rng.choice([1, 2, 4])
        H, W = _size(rng, 256 * 256, 2 * 1024 * 1024 // n)
        return dict(kind=kind, n=n, H=H, W=W, levels=rng.choice([2, 3, 4]), iters=rng.choice([30, 60, 100]),
                    fast=rng.random() < 0.7, alpha=alpha)
    if kind == "powers":
        H, W = _size(rng, 240 * 320, 2048 * 2048)
        return dict(kind=kind, H=H, W=W, steps=rng.randrange(2, 10))
    H, W = _size(rng, 240 * 320, 1080 * 1920)
    return dict(kind="lk", H=H, W=W, radius=rng.randrange(2, 6))


# ------------------------------------------------------------------ inputs


def _smooth(n, H, W, cell, g):
    """n smooth random fields in [0, 1], features of about `cell` pixels."""
    c = torch.rand((n, 1, H // cell + 2, W // cell + 2), device="cuda", generator=g)
    return F.interpolate(c, size=(H, W), mode="bilinear", align_corners=True)


def _pairs(n, H, W, seed, amplitude=1.5):
    """n image pairs: a textured image in [0, 1], the same moved by a smooth flow of up to
    `amplitude` pixels plus sensor noise, and that flow.  Each of shape (n, H, W), float32."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    a = 0.6 * _smooth(n, H, W, 8, g) + 0.4 * _smooth(n, H, W, 3, g)
    f = (2.0 * torch.cat([_smooth(n, H, W, 48, g), _smooth(n, H, W, 48, g)], 1) - 1.0) * amplitude
    y, x = torch.meshgrid(torch.arange(H, device="cuda", dtype=torch.float32),
                          torch.arange(W, device="cuda", dtype=torch.float32), indexing="ij")
    at = torch.stack([2 * (x - f[:, 0]) / max(W - 1, 1) - 1, 2 * (y - f[:, 1]) / max(H - 1, 1) - 1], -1)
    b = F.grid_sample(a, at, mode="bilinear", padding_mode="border", align_corners=True)
    b = b + 0.01 * torch.randn(b.shape, device="cuda", generator=g)
    return a[:, 0].contiguous(), b[:, 0].contiguous(), f[:, 0].contiguous(), f[:, 1].contiguous()


def _batch_specs(case):
    return [(s.H, s.W, s.alpha, s.iters) for s in synthetic.batch_mixed(case["n"], case["specs"])]


def _planes(n, H, W, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return [torch.rand((H, W), device="cuda", generator=g) - 0.5 for _ in range(n)]


def hs_program(I0, I1, Dx, Dy, Dt, A, alpha, u, v):
    alpha2 = alpha * alpha
    Ix = Dx * I0 + Dx * I1
    Iy = Dy * I0 + Dy * I1
    It = Dt * I1 - Dt * I0
    den = alpha2 + Ix * Ix + Iy * Iy
    for i in range(200):
        ubar = A * u
        vbar = A * v
        t = (Ix * ubar + Iy * vbar + It) / den
        u = ubar - Ix * t
        v = vbar - Iy * t
    return u, v


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("forward", "hm", "train", "pyramid"):
        n, H, W = case.get("n", 1), case["H"], case["W"]
        I0, I1, ut, vt = _pairs(n, H, W, seed, 12.0 if kind == "pyramid" else 1.5)
        s["config"] = make_config(fast_math=True) if case["fast"] else None
        if kind in ("train", "pyramid"):
            s["images"] = [(a.clone().requires_grad_(True), b.clone().requires_grad_(True)) for a, b in zip(I0, I1)]
            s["targets"] = [(a.clone(), b.clone()) for a, b in zip(ut, vt)]
            s["alpha"] = torch.tensor(float(case["alpha"]), device="cuda", requires_grad=True)
        else:
            s["I0"], s["I1"] = I0[0], I1[0]
    if kind == "hm":
        Dx, Dy, Dt = hs_derivative_stencils()
        z = torch.zeros_like(s["I0"])
        s["fn"] = _hm_flow
        s["kw"] = dict(I0=s["I0"], I1=s["I1"], Dx=Dx, Dy=Dy, Dt=Dt, A=hs_average_stencil(),
                       alpha=np.float32(case["alpha"]), u=z, v=z)
        _set_hm(case)
        s["fn"](**s["kw"])  # parses, compiles and tunes for this shape once per process
    elif kind == "batch":
        specs = _batch_specs(case)
        plan = BatchPlan(specs, make_config(fast_math=case["fast"]))
        for i, (H, W, _, _) in enumerate(specs):
            a, b, _, _ = _pairs(1, H, W, 100 * seed + i)
            plan.I0[i].copy_(a[0])
            plan.I1[i].copy_(b[0])
        plan.capture()
        s["plan"] = plan
    elif kind == "powers":
        s["planes"] = _planes(4, case["H"], case["W"], seed)
    elif kind == "lk":
        s["planes"] = _planes(3, case["H"], case["W"], seed)
    return s


_hm_flow = hm(hs_program)


def _set_hm(case):
    """The tuning keys are the module-wide `defines`, as a program sets them before its calls."""
    from hindemith_b200 import defines

    if case["fast"]:
        defines["hs_fast_math"] = True
    else:
        defines.pop("hs_fast_math", None)


def run(s):
    kind = s["kind"]
    if kind == "forward":
        return D.hs_forward(s["I0"], s["I1"], s["alpha"], s["iters"], s["config"])
    if kind == "hm":
        _set_hm(s)
        return s["fn"](**s["kw"])
    if kind == "batch":
        s["plan"].replay()
        return {"u": s["plan"].u, "v": s["plan"].v}
    if kind in ("train", "pyramid"):
        leaves = [t for pair in s["images"] for t in pair] + [s["alpha"]]
        if kind == "pyramid":
            flows = coarse_to_fine(s["images"], s["alpha"], s["levels"], s["iters"], config=s["config"])
        elif s["n"] == 1:
            flows = [horn_schunck(*s["images"][0], s["alpha"], s["iters"], s["ckpt"], s["config"])]
        else:
            flows = horn_schunck_batch(s["images"], s["alpha"], s["iters"], s["ckpt"], s["config"])
        loss = mean_epe_batch(flows, s["targets"])
        grads = torch.autograd.grad(loss, leaves)
        out = {"loss": loss.detach(), "grads": list(grads)}
        if s["n"] == 1:
            out["flow"] = [t.detach() for t in flows[0]]
        return out
    if kind == "powers":
        return hs_matrix_powers(1.0, *s["planes"], s["steps"])
    return FL.lk_least_squares(*s["planes"], s["radius"])


# ------------------------------------------------------------------ work


def work(case):
    kind = case["kind"]
    px = case.get("n", 1) * case.get("H", 0) * case.get("W", 0)
    if kind in ("forward", "hm"):  # two images in, two flow planes out
        return {"bytes": 16.0 * px, "flops": float(SWEEP_FLOPS) * px * case["iters"]}
    if kind == "batch":
        specs = _batch_specs(case)
        return {"bytes": 16.0 * sum(H * W for H, W, _, _ in specs),
                "flops": float(SWEEP_FLOPS) * sum(H * W * n for H, W, _, n in specs)}
    if kind == "train":  # images and targets in, image gradients out; forward + adjoint sweeps
        return {"bytes": 24.0 * px, "flops": float(SWEEP_FLOPS + ADJOINT_FLOPS) * px * case["iters"]}
    if kind == "pyramid":
        levels = sum(0.25 ** k for k in range(case["levels"]))
        return {"bytes": 24.0 * px, "flops": float(SWEEP_FLOPS + ADJOINT_FLOPS) * px * case["iters"] * levels}
    if kind == "powers":
        return {"bytes": px * (16.0 + 8.0 * case["steps"]), "flops": float(POWER_FLOPS) * px * (case["steps"] - 1)}
    return {"bytes": 20.0 * px, "flops": 10.0 * px * (2 * case["radius"]) ** 2}


# ------------------------------------------------------------------ 64-bit outputs

# the program's constants are 32-bit floats
_WE, _WC = float(np.float32(1 / 6)), float(np.float32(1 / 12))


def _pad(x, left, right, top, bottom):
    return F.pad(x[:, None], (left, right, top, bottom), mode="replicate")[:, 0]


def _average(x):
    p = _pad(x, 1, 1, 1, 1)
    h = p[:, :, :-2] + p[:, :, 2:]
    v = _WE * p[:, :, 1:-1] + _WC * h
    return v[:, :-2] + _WE * h[:, 1:-1] + v[:, 2:]


def _derivatives(I0, I1):
    a, b = _pad(I0, 0, 1, 0, 1), _pad(I1, 0, 1, 0, 1)
    s = a + b
    Ix = 0.25 * ((s[:, :-1, 1:] - s[:, :-1, :-1]) + (s[:, 1:, 1:] - s[:, 1:, :-1]))
    Iy = 0.25 * ((s[:, 1:, :-1] - s[:, :-1, :-1]) + (s[:, 1:, 1:] - s[:, :-1, 1:]))
    d = b - a
    It = 0.25 * (d[:, :-1, :-1] + d[:, :-1, 1:] + d[:, 1:, :-1] + d[:, 1:, 1:])
    return Ix, Iy, It


def _flow64(I0, I1, alpha, iters):
    Ix, Iy, It = _derivatives(I0, I1)
    den = alpha * alpha + Ix * Ix + Iy * Iy
    u = v = torch.zeros_like(I0)
    for _ in range(iters):
        ub, vb = _average(u), _average(v)
        t = (Ix * ub + Iy * vb + It) / den
        u, v = ub - Ix * t, vb - Iy * t
    return u, v


def _epe64(u, v, ut, vt):
    return torch.sqrt((u - ut) ** 2 + (v - vt) ** 2 + 1e-12).mean(dim=(1, 2)).mean()


def _blur_down64(x):
    w = torch.tensor([1.0, 4.0, 6.0, 4.0, 1.0], dtype=x.dtype, device=x.device) / 16
    p = _pad(x, 2, 2, 2, 2)
    r = sum(w[k] * p[:, :, k:k + x.shape[2]] for k in range(5))
    return sum(w[k] * r[:, k:k + x.shape[1]] for k in range(5))[:, ::2, ::2]


def _upsample64(c, H, W):
    def axis(n, nc):
        p = (torch.arange(n, device=c.device, dtype=c.dtype) + 0.5) / 2 - 0.5
        i = torch.floor(p)
        return i.long().clamp(0, nc - 1), (i.long() + 1).clamp(0, nc - 1), p - i

    y0, y1, fy = axis(H, c.shape[1])
    x0, x1, fx = axis(W, c.shape[2])
    fy = fy[:, None]
    top = (1 - fx) * c[:, y0][:, :, x0] + fx * c[:, y0][:, :, x1]
    bottom = (1 - fx) * c[:, y1][:, :, x0] + fx * c[:, y1][:, :, x1]
    return 2.0 * ((1 - fy) * top + fy * bottom)


def _warp64(src, ox, oy):
    n, H, W = src.shape
    mx, my = torch.floor(ox.detach()).long(), torch.floor(oy.detach()).long()
    xf, yf = ox - mx, oy - my
    y = torch.arange(H, device=src.device)[:, None] + my
    x = torch.arange(W, device=src.device) + mx
    ok = (x >= 0) & (x + 1 < W) & (y >= 0) & (y + 1 < H)
    base = torch.arange(n, device=src.device)[:, None, None] * H * W
    q = base + torch.where(ok, y * W + x, 0)
    s = src.reshape(-1)

    def at(k):
        return s[(q + k).clamp(max=s.numel() - 1)]

    o = ((1 - xf) * (1 - yf) * at(0) + xf * (1 - yf) * at(1) + (1 - xf) * yf * at(W) + xf * yf * at(W + 1))
    return torch.where(ok, o, src)


def _coarse_to_fine64(I0, I1, alpha, levels, iters):
    p0, p1 = [I0], [I1]
    for _ in range(levels - 1):
        p0.append(_blur_down64(p0[-1]))
        p1.append(_blur_down64(p1[-1]))
    u, v = _flow64(p0[-1], p1[-1], alpha, iters)
    for k in range(levels - 2, -1, -1):
        H, W = p0[k].shape[1:]
        u, v = _upsample64(u, H, W), _upsample64(v, H, W)
        du, dv = _flow64(p0[k], _warp64(p1[k], u, v), alpha, iters)
        u, v = u + du, v + dv
    return u, v


def _powers64(lam, Ix, Iy, u, v, steps):
    def laplacian(x):
        p = _pad(x, 1, 1, 1, 1)  # an absent neighbour's copy of the pixel adds nothing
        return 4 * x - p[:, 1:-1, :-2] - p[:, 1:-1, 2:] - p[:, :-2, 1:-1] - p[:, 2:, 1:-1]

    U, V = [u], [v]
    for _ in range(steps - 1):
        g = Ix * U[-1] + Iy * V[-1]
        U, V = U + [Ix * g + lam * laplacian(U[-1])], V + [Iy * g + lam * laplacian(V[-1])]
    return torch.cat(U), torch.cat(V)


def _lk64(err, Ix, Iy, r):
    def window(x):  # sums over [-r, r) x [-r, r)
        c = F.pad(x, (r + 1, r, r + 1, r)).cumsum(0).cumsum(1)
        return c[2 * r:-1, 2 * r:-1] - c[:-2 * r - 1, 2 * r:-1] - c[2 * r:-1, :-2 * r - 1] + c[:-2 * r - 1, :-2 * r - 1]

    xx, yy, xy, xt, yt = (window(p) for p in (Ix * Ix, Iy * Iy, Ix * Iy, Ix * err, Iy * err))
    det = xx * yy - xy * xy
    inside = torch.zeros_like(det, dtype=torch.bool)
    inside[r:det.shape[0] - r, r:det.shape[1] - r] = True
    ok = inside & (det != 0)
    zero = torch.zeros_like(det)
    return torch.where(ok, (xt * yy - xy * yt) / det, zero), torch.where(ok, (xx * yt - xy * xt) / det, zero)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        u, v = [], []
        for i, (H, W, alpha, iters) in enumerate(_batch_specs(case)):
            a, b, _, _ = _pairs(1, H, W, 100 * seed + i)
            x, y = _flow64(a.double(), b.double(), float(np.float32(alpha)), iters)
            u.append(x[0])
            v.append(y[0])
        return {"u": u, "v": v}
    if kind == "powers":
        return _powers64(1.0, *(p.double()[None] for p in _planes(4, case["H"], case["W"], seed)), case["steps"])
    if kind == "lk":
        return _lk64(*(p.double() for p in _planes(3, case["H"], case["W"], seed)), case["radius"])
    a, b, ut, vt = (t.double() for t in _pairs(case.get("n", 1), case["H"], case["W"], seed, 12.0 if kind == "pyramid" else 1.5))
    alpha = float(np.float32(case["alpha"]))
    if kind in ("forward", "hm"):
        u, v = _flow64(a, b, alpha, case["iters"])
        return u[0], v[0]
    a.requires_grad_(True)
    b.requires_grad_(True)
    al = torch.tensor(alpha, dtype=torch.float64, device="cuda", requires_grad=True)
    if kind == "pyramid":
        u, v = _coarse_to_fine64(a, b, al, case["levels"], case["iters"])
    else:
        u, v = _flow64(a, b, al, case["iters"])
    loss = _epe64(u, v, ut, vt)
    ga, gb, gal = torch.autograd.grad(loss, [a, b, al])
    grads = [t for pair in zip(ga, gb) for t in pair] + [gal]
    out = {"loss": loss.detach(), "grads": grads}
    if case["n"] == 1:
        out["flow"] = [u[0].detach(), v[0].detach()]
    return out
