"""The level accumulation operators on both sides of every line between their kernels, at last passes of one to three
triangles for each number of triangles a pass, against the oracle: forward bit for bit (the same products in the same
order), adjoint within 1e-5 (chains of at most a few hundred FP32 products); infinities and NaN in the adjoint."""

import numpy as np
import pytest
import torch

from diffsoup_b200 import _core, multires
from oracle import cpu

pytestmark = pytest.mark.gpu

# (T, lo, hi, target, C)
SIZES = [
    # forward, a pass of one CTA on 148 SMs: 4,736, 2,368 and 1,184 triangles at four, two and one a pass
    (4735, 0, 2, 2, 7), (4736, 0, 2, 2, 7), (4737, 0, 2, 2, 7), (4738, 0, 2, 2, 8), (4739, 0, 3, 3, 3),
    (2367, 0, 3, 3, 16), (2368, 0, 3, 3, 16), (2369, 0, 3, 3, 16), (1183, 0, 4, 4, 8), (1184, 0, 4, 4, 8),
    (1185, 0, 4, 4, 16),
    # few values a triangle, and sources of which few are read
    (5000, 0, 0, 0, 8), (5000, 0, 0, 0, 11), (6000, 0, 3, 1, 3), (6000, 0, 3, 2, 3), (3000, 0, 5, 2, 4),
    # adjoint, around 1.5 million products: 45 * 4 * 7 a triangle, 153 * 8, 15 * 3 * 3
    (1190, 0, 3, 3, 7), (1191, 0, 3, 3, 7), (1225, 4, 4, 4, 8), (1226, 4, 4, 4, 8), (11112, 0, 2, 2, 3),
]


@pytest.mark.parametrize("T,lo,hi,target,C", SIZES)
def test_both_sides_of_the_lines(T, lo, hi, target, C):
    rng = np.random.default_rng(T + C)
    S, ST = _core.total_feats(lo, hi), _core.feats_at_level(target)
    src = rng.normal(size=(T, S, C)).astype(np.float32)
    g = rng.normal(size=(T, ST, C)).astype(np.float32)
    feat = torch.from_numpy(src).cuda().requires_grad_()
    out = multires.accumulate_to_level(lo, hi, feat, target)
    want = cpu.accumulate_forward(lo, hi, target, src, precision="f32")
    np.testing.assert_array_equal(out.detach().cpu().numpy().view(np.uint32), want.view(np.uint32))
    out.backward(torch.from_numpy(g).cuda())
    ref = cpu.accumulate_backward(lo, hi, target, T, g)
    rel = lambda a: np.linalg.norm(a - ref) / np.linalg.norm(ref)  # noqa: E731
    assert rel(feat.grad.cpu().numpy()) < 1e-5
    acc = torch.ones(T, S, C, device="cuda")  # the accumulating entry point adds to what is there
    _core.accumulate_to_level_backward(lo, hi, target, acc, torch.from_numpy(g).cuda())
    assert rel(acc.cpu().numpy() - 1.0) < 1e-5


@pytest.mark.parametrize("T", [300, 30000])
def test_infinities_in_the_adjoint(T):
    """Each source whose cell touches a target with an infinite or NaN gradient gets what the sum over all corners
    gives, with either kernel: 0 * inf is NaN."""
    lo, hi, C = 0, 2, 3
    g = np.random.default_rng(6).normal(size=(T, _core.feats_at_level(hi), C)).astype(np.float32)
    g[17, 4, 1], g[T // 2, 0, 2], g[T - 1, 14, 0] = np.nan, np.inf, -np.inf
    grad = torch.empty(T, _core.total_feats(lo, hi), C, device="cuda")
    _core.accumulate_to_level_backward_set(lo, hi, hi, grad, torch.from_numpy(g).cuda())
    want = cpu.accumulate_backward(lo, hi, hi, T, g)
    got = grad.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(want).sum() > 3
    assert np.array_equal(got[np.isinf(got)], want[np.isinf(want)])
    ok = np.isfinite(want)
    assert np.linalg.norm(got[ok] - want[ok]) < 1e-5 * np.linalg.norm(want[ok])
