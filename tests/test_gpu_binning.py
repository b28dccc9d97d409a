"""Tile lists of the binning passes against brute force: each tile's list holds its triangles once, in depth
order up to 512 entries, over both widths of the passes, list lengths around the sort's sizes and rects of more than 64
tiles."""

import numpy as np
import pytest
import torch

from oracle import cpu
from diffsoup_b200 import _core, scenes, tiles
import diffsoup_b200 as ds

pytestmark = pytest.mark.gpu


def al(n):
    return (n + 255) // 256 * 256


def lists_of(b):
    """Per tile the (zlo, record) pairs in list order, and the tile's sorted flag, from the bins' workspace."""
    ws, n, nt = b.workspace.cpu().numpy(), b.B * b.T, b.num_tiles
    o = al(16 * n) + al(48 * n) + al(32 * n) + al(32 * n) + al(4 * nt)
    off = ws[o:o + 8 * (nt + 1)].view(np.int64)
    o += al(8 * (nt + 1)) + al(4 * nt)
    flags = ws[o:o + 4 * nt].view(np.int32)
    o += al(4 * nt) + 256 + al(8 * ((nt + 2047) // 2048 + 1))
    ent = ws[o:o + 16 * int(off[-1])].view(np.int32).reshape(-1, 4)
    return off, flags, ent[:, 2].view(np.float32), ent[:, 3]


# stacks of n triangles on one tile: around every sort size; 70,000 records take the wide passes
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512, 513, 700])
def test_list_lengths(n):
    rng = np.random.default_rng(n)
    z = rng.permutation(n).astype(np.float32) / (n + 1) - 0.5
    tri_xy = np.array([[-1, -1], [3, -1], [-1, 3]], np.float32)  # covers the whole 16x16 view
    pos = np.concatenate([np.broadcast_to(tri_xy, (n, 3, 2)), np.broadcast_to(z[:, None, None], (n, 3, 1)),
                          np.ones((n, 3, 1), np.float32)], -1).reshape(1, 3 * n, 4).astype(np.float32)
    tri = torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(n, 3)
    b = tiles.bin_views(torch.from_numpy(pos.copy()).cuda(), tri, [(16, 16)], reuse=False)
    off, flags, zlo, rec = lists_of(b)
    assert off[-1] == n and sorted(rec.tolist()) == list(range(n))
    assert flags[0] == (1 if n <= 512 else 0)
    if n <= 512:
        assert (np.diff(zlo) >= 0).all() and (z[rec] == np.sort(z)).all()


@pytest.mark.parametrize("T,views,hw,scale", [(37, 1, (333, 517), 1.0), (1501, 2, (240, 321), 12.0),
                                              (30001, 3, (96, 131), 3.0)])
def test_wide_and_narrow_passes(T, views, hw, scale):
    """Small and large rects (scale widens the triangles to hundreds of tiles): the ID buffer equals the oracle's."""
    sc = scenes.make_scene(1, seed=T, num_tris=T, num_views=views, resolution=hw, with_targets=False)
    c = sc.verts.reshape(-1, 3, 3).mean(1, keepdims=True)
    verts = (c + scale * (sc.verts.reshape(-1, 3, 3) - c)).reshape(-1, 3).astype(np.float32)
    pos = cpu.project(verts, sc.mvps())
    alpha = np.random.default_rng(3).uniform(0, 1, (T, 15)).astype(np.float32)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    got = ds.rasterize_multires_triangle_alpha(hw, d(pos), d(sc.tri), 2, d(alpha[..., None]), stochastic=False)
    for v in range(views):
        want, _ = cpu.rasterize_alpha(hw[0], hw[1], pos[v:v + 1], sc.tri, 2, alpha, False, view0=v)
        assert np.array_equal(got[v:v + 1].cpu().numpy().view(np.uint32), want.view(np.uint32))
