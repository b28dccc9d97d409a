"""The opacity gradient of triangles large enough for their contributions to be summed over a warp: levels with one
cell, a few pixels' cells and cells smaller than a pixel block, triangles on both sides of the line, and views of a
single block, against the oracle."""

import numpy as np
import pytest
import torch

import diffsoup_b200 as ds
from oracle import cpu

pytestmark = pytest.mark.gpu


def layers(n, size, spread, seed):
    rng = np.random.default_rng(seed)
    corner = np.array([[-1, -1], [3, -1], [-1, 3]], np.float32) * size
    xy = rng.uniform(-spread, spread, (n, 1, 2)) + corner + 0.05 * size * rng.normal(size=(n, 3, 2))
    z = np.broadcast_to(rng.permutation(np.linspace(-0.8, 0.8, n))[:, None, None], (n, 3, 1))
    return np.concatenate([xy, z, np.ones((n, 3, 1))], -1).astype(np.float32).reshape(1, 3 * n, 4)


# (triangles, size in NDC, spread of their centres, height, width)
@pytest.mark.parametrize("n,size,spread,H,W", [(1, 1.0, 0.0, 96, 160), (2, 1.0, 0.0, 8, 4), (40, 1.0, 0.1, 65, 97),
                                               (60, 0.3, 0.8, 150, 131), (300, 0.1, 0.9, 97, 160)])
@pytest.mark.parametrize("level", [0, 2, 4])
@pytest.mark.parametrize("opacity", [0.1, 0.7])
def test_matches_oracle(n, size, spread, H, W, level, opacity):
    rng = np.random.default_rng(n * 7 + level)
    S = ds.feats_at_level(level)
    pos, tri = layers(n, size, spread, seed=n), np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    alpha = np.clip(opacity + 0.05 * rng.normal(size=(n, S)), 0.02, 0.98).astype(np.float32)
    color, target = rng.uniform(size=(2, 1, H, W, 3)).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    a3 = t(alpha[..., None]).requires_grad_(True)
    rast = ds.rasterize_multires_triangle_alpha((H, W), t(pos), t(tri), level, a3.detach(), stochastic=False)
    ds.opacity_aux_loss(t(color), t(target), rast, t(pos), t(tri), level, a3).backward()
    want = cpu.opacity_aux(color, target, rast.cpu().numpy(), pos, tri, level, alpha, precision="f32") / color.size
    got = a3.grad.cpu().numpy().reshape(want.shape)
    # a sample sums up to 15,000 pixels' FP32 contributions of one sign, in another order than the oracle's
    assert np.linalg.norm(got - want) <= 2e-5 * np.linalg.norm(want) + 1e-12
    assert np.abs(want).max() > 0
