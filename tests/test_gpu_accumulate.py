"""Level accumulation operators over both of their kernels (the table-driven
map and the one-thread-per-sample kernels) against the oracle: forward bit for
bit (same products in the same order), adjoint within 1e-5 (chains of at most a
few hundred FP32 products)."""

import numpy as np
import pytest
import torch

from oracle import cpu
from diffsoup_b200 import _core, multires

pytestmark = pytest.mark.gpu

# (T, lo, hi, target, C): a single triangle; a last warp pass of 1-3 triangles; one, two and four triangles a
# pass; target lattices below, at and above the finest level; lattices beyond the tables
SIZES = [(1, 0, 0, 0, 1), (138, 0, 2, 2, 7), (139, 0, 2, 2, 8), (685, 0, 3, 3, 7), (257, 0, 3, 3, 16),
         (33, 0, 4, 4, 16), (1367, 1, 3, 1, 3), (501, 0, 2, 4, 5), (2050, 2, 2, 2, 1), (9, 0, 6, 6, 2)]


@pytest.mark.parametrize("T,lo,hi,target,C", SIZES)
def test_accumulate_matches_oracle(T, lo, hi, target, C):
    rng = np.random.default_rng(T * 31 + C)
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
    # the accumulating entry point adds to what is there
    acc = torch.ones(T, S, C, device="cuda")
    _core.accumulate_to_level_backward(lo, hi, target, acc, torch.from_numpy(g).cuda())
    assert rel(acc.cpu().numpy() - 1.0) < 1e-5


def test_accumulate_zero_weights_carry_nan():
    """0 * NaN and 0 * inf reach the samples whose cell touches the corner, as the sum over all corners gives."""
    T, lo, hi, C = 700, 0, 2, 3
    rng = np.random.default_rng(5)
    src = rng.normal(size=(T, _core.total_feats(lo, hi), C)).astype(np.float32)
    src[17, 4, 1], src[300, 0, 2], src[699, 23, 0] = np.nan, np.inf, -np.inf
    out = multires.accumulate_to_level(lo, hi, torch.from_numpy(src).cuda()).cpu().numpy()
    with np.errstate(invalid="ignore"):
        want = cpu.accumulate_forward(lo, hi, hi, src, precision="f32")
    np.testing.assert_array_equal(out, want)
    assert np.isnan(out).sum() > 3
