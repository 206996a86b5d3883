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
