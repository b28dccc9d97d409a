"""Per-pixel feature lookup, its scatter and the view encodings over their kernels (four-channel vectors, seven-channel
rows, rows through shared memory, one thread per channel) at ragged sizes and unaligned buffers, against the
oracle."""

import numpy as np
import pytest
import torch

from oracle import cpu
from diffsoup_b200 import _core, multires, rasterize

pytestmark = pytest.mark.gpu


def buffer(a, shift):
    """A contiguous device copy of a whose first element sits `shift` floats past an aligned address."""
    flat = torch.empty(a.size + shift, device="cuda")
    flat[shift:] = torch.from_numpy(a.reshape(-1)).cuda()
    return flat[shift:].view(*a.shape)


def make(B, H, W, T, lo, hi, C, seed):
    rng = np.random.default_rng(seed)
    b = rng.dirichlet((1, 1, 1), size=(B, H, W)).astype(np.float32)
    ids = np.repeat(rng.integers(0, T + 1, size=(B, H, (W + 4) // 5)), 5, axis=2)[:, :, :W]
    rast = np.stack([b[..., 0], b[..., 1], rng.uniform(-1, 1, (B, H, W)), ids], -1).astype(np.float32)
    rast[ids == 0] = 0
    S = _core.total_feats(lo, hi)
    return rast, rng.normal(size=(T, S, C)).astype(np.float32), rng.normal(size=(B, H, W, C)).astype(np.float32)


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("B,H,W,lo,hi,C", [(1, 1, 1, 2, 2, 7), (2, 7, 9, 2, 2, 7), (1, 16, 64, 0, 0, 7),
                                           (3, 33, 65, 0, 3, 7), (2, 31, 33, 2, 2, 4), (1, 40, 40, 1, 2, 16),
                                           (2, 5, 13, 3, 3, 1), (1, 29, 31, 0, 1, 5), (1, 9, 11, 2, 2, 32),
                                           (1, 9, 11, 2, 2, 33)])
def test_lookup_and_scatter(B, H, W, lo, hi, C, shift):
    T = 11
    rast, feat, g = make(B, H, W, T, lo, hi, C, seed=C * 7 + W)
    r, f, gd = torch.from_numpy(rast).cuda(), buffer(feat, shift), buffer(g, shift)
    ref = torch.zeros(B, H, W, C, device="cuda")
    _core.multires_triangle_color(r, lo, hi, f, ref)
    out = buffer(np.full((B, H, W, C), np.nan, np.float32), shift)
    _core.multires_triangle_color_set(r, lo, hi, f, out)
    assert torch.equal(out, ref)
    acc = buffer(np.zeros_like(feat), shift)
    _core.backward_multires_triangle_color(r, lo, hi, acc, gd)
    want = cpu.multires_color_backward(rast, lo, hi, T, g)
    # a few hundred FP32 products per sample
    assert np.linalg.norm(acc.cpu().numpy() - want) < 1e-5 * np.linalg.norm(want) + 1e-6


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 5, 7), (1, 8, 32), (3, 17, 96), (2, 33, 31)])
def test_encodings_write_every_pixel(B, H, W):
    rast, _, _ = make(B, H, W, 9, 0, 0, 1, seed=W)
    rng = np.random.default_rng(W)
    inv = np.linalg.inv(np.eye(4) + 0.2 * rng.normal(size=(B, 4, 4))).astype(np.float32)
    r, m = torch.from_numpy(rast).cuda(), torch.from_numpy(inv).cuda()
    for sh, fn in ((True, rasterize.encode_view_dir_sh2), (False, rasterize.encode_view_dir)):
        want = cpu.encode_view(rast, inv, sh=sh)
        torch.full((B * H * W * 9,), float("nan"), device="cuda")  # leaves NaN in the allocator's block
        got = fn(r, m).cpu().numpy()
        assert np.abs(got - want).max() < 2e-5  # rsqrtf and the FP32 chain of two projections
        assert (got[rast[..., 3] == 0] == 0).all()
        keep = torch.full_like(torch.from_numpy(want).float().cuda(), 7.0)  # background keeps what was there
        (_core.encode_view_dir_sh2 if sh else _core.encode_view_dir)(r, m, keep)
        k = keep.cpu().numpy()
        assert (k[rast[..., 3] == 0] == 7).all() and np.array_equal(k[rast[..., 3] > 0], got[rast[..., 3] > 0])
