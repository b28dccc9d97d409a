"""Tile lists of views of many tiles, from passes of 8 and of 32 triangles a warp and with rects of more than 64 tiles:
every triangle with a fragment in a tile is in the tile's list once, none is there twice, and lists marked as sorted
are in depth order."""

import numpy as np
import pytest
import torch

from diffsoup_b200 import scenes, tiles
from oracle import cpu
from test_gpu_binning import lists_of

pytestmark = pytest.mark.gpu


# (triangles, views): 24,000 pairs and one more, three views of a wide pass; scale 12 widens rects to hundreds of tiles
@pytest.mark.parametrize("T,views,hw,scale", [(24000, 1, (90, 330), 1.0), (24001, 1, (90, 330), 1.0),
                                              (8001, 3, (160, 250), 12.0), (2000, 1, (400, 517), 12.0),
                                              (12500, 2, (333, 517), 6.0)])
def test_lists_hold_every_fragment_once(T, views, hw, scale):
    H, W = hw
    sc = scenes.make_scene(1, seed=T, num_tris=T, num_views=views, resolution=hw, with_targets=False)
    c = sc.verts.reshape(-1, 3, 3).mean(1, keepdims=True)
    grow = np.where(np.arange(T) % 16 == 0, scale, 1.0)[:, None, None]  # a sixteenth of the triangles
    verts = (c + grow * (sc.verts.reshape(-1, 3, 3) - c)).reshape(-1, 3).astype(np.float32)
    pos = cpu.project(verts, sc.mvps())
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    b = tiles.bin_views(d(pos), d(sc.tri), [hw] * views, reuse=False)
    off, flags, zlo, rec = lists_of(b)
    per, tx = b.num_tiles // views, (W + 15) // 16
    widest = 0
    for v in range(views):
        fpix, fattr = cpu.compute_fragments(H, W, pos[v:v + 1], sc.tri)
        tile = fpix[:, 1] // 16 * tx + fpix[:, 2] // 16
        want = np.unique(tile.astype(np.int64) * T + fattr[:, 3].astype(np.int64) - 1)
        got = np.concatenate([i * T + rec[off[v * per + i]:off[v * per + i + 1]] - v * T for i in range(per)])
        assert len(np.unique(got)) == len(got)
        assert np.isin(want, got).all()
        widest = max(widest, np.bincount(got % T, minlength=T).max())
    assert scale == 1.0 or widest > 64
    for i in range(b.num_tiles):
        z = zlo[off[i]:off[i + 1]]
        assert flags[i] == (len(z) <= 512)
        assert not flags[i] or (np.diff(z) >= 0).all()
