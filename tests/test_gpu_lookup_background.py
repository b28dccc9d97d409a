"""The feature lookup that writes every pixel, over the ways a warp's pixels can be covered (none, all, one, every
other, runs), in each of its forms of storing rows, against the lookup that adds to a zeroed buffer (one thread per pixel
and channel, the same sums in the same order: equal bit for bit)."""

import numpy as np
import pytest
import torch

from diffsoup_b200 import _core

pytestmark = pytest.mark.gpu


def rast_of(cover, T, seed):
    rng = np.random.default_rng(seed)
    n = cover.size
    b = rng.dirichlet((1, 1, 1), size=n).astype(np.float32)
    r = np.stack([b[:, 0], b[:, 1], rng.uniform(-1, 1, n), rng.integers(1, T + 1, n)], -1).astype(np.float32)
    return torch.from_numpy(r * cover[:, None].astype(np.float32)).cuda().view(1, 1, n, 4)


def patterns():
    lane = np.arange(32)
    warps = [lane < 0, lane >= 0, lane == 0, lane == 31, lane == 17, lane % 2 == 0, lane % 5 == 3, lane < 16, lane >= 7]
    return np.concatenate(warps * 3 + [lane[:13] >= 0])  # a last warp of 13 pixels


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("C", [1, 3, 4, 6, 7, 8, 20, 24, 25, 28, 31, 32, 33, 36, 63, 64])
@pytest.mark.parametrize("lo,hi", [(2, 2), (0, 2)])
def test_every_pixel_is_written(C, lo, hi, shift):
    T, cover = 9, patterns()
    for c in (cover, cover[13:], cover[:1], ~cover[:32], np.zeros(77, bool)):
        rast = rast_of(c, T, C)
        S, n = _core.total_feats(lo, hi), c.size
        g = torch.Generator(device="cuda").manual_seed(C)
        feat = torch.randn(T * S * C + shift, generator=g, device="cuda")[shift:].view(T, S, C)
        want = torch.zeros(1, 1, n, C, device="cuda")
        _core.multires_triangle_color(rast, lo, hi, feat, want)
        room = torch.full((n * C + shift + 8,), float("nan"), device="cuda")
        out = room[shift:shift + n * C].view(1, 1, n, C)
        _core.multires_triangle_color_set(rast, lo, hi, feat, out)
        assert torch.equal(out, want)
        assert torch.isnan(room[:shift]).all() and torch.isnan(room[shift + n * C:]).all()
