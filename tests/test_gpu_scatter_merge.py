"""The feature scatter at one level, whose pixels of a lattice cell are summed before the atomics, on barycentrics that
vary smoothly over a view as a rasterizer's do: one triangle, two that alternate from pixel to pixel, small ones and one a
pixel, in every width of staged rows and of lattice, against the oracle."""

import numpy as np
import pytest
import torch

from diffsoup_b200 import _core
from oracle import cpu

pytestmark = pytest.mark.gpu
T = 40


def raster(kind, H, W, seed):
    """B=2 views: IDs by `kind`, a tenth of the pixels background; barycentrics a linear function of the pixel."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[:H, :W].astype(np.float32)
    ids = {"one": np.ones((H, W)), "two": 1 + (x + y) % 2, "small": 1 + (y // 3 * 7 + x // 4) % T,
           "pixel": rng.integers(1, T + 1, (H, W))}[kind]
    u, v = (x + 0.5) / (W + 1), (y + 0.5) / (H + 1)
    b0, b1 = 0.9 * u * (1 - v), 0.9 * v
    rast = np.stack([b0, b1, np.zeros_like(u), ids], -1).astype(np.float32)[None].repeat(2, 0)
    rast[rng.random((2, H, W)) < 0.1] = 0
    return rast


@pytest.mark.parametrize("kind", ["one", "two", "small", "pixel"])
@pytest.mark.parametrize("H,W", [(4, 8), (37, 61)])
@pytest.mark.parametrize("C", [4, 7, 8, 12, 16, 20, 28, 32])
def test_matches_oracle(kind, H, W, C):
    rast = raster(kind, H, W, seed=C)
    r = torch.from_numpy(rast).cuda()
    for level in (0, 1, 2, 4, 8):
        g = np.random.default_rng(level).normal(size=(2, H, W, C)).astype(np.float32)
        acc = torch.zeros(T, _core.feats_at_level(level), C, device="cuda")
        _core.backward_multires_triangle_color(r, level, level, acc, torch.from_numpy(g).cuda())
        want = cpu.multires_color_backward(rast, level, level, T, g)
        # up to 4,514 FP32 products a sample
        assert np.linalg.norm(acc.cpu().numpy() - want) < 1e-5 * np.linalg.norm(want) + 1e-6
