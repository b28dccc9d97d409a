"""Edge gradients of three-channel images (the staged kernel) against the one-thread-per-pixel kernel, which the
same image with a zero fourth channel takes: the same pairs with the same arithmetic, sums in another order."""

import pytest
import torch

from diffsoup_b200 import _core, scenes
import diffsoup_b200 as ds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,T,views,hw", [(1, 1, 1, (1, 1)), (1, 40, 2, (15, 17)), (1, 3000, 1, (16, 32)),
                                               (2, 4000, 3, (97, 130)), (3, 2000, 2, (255, 241))])
def test_staged_kernel_matches_per_pixel_kernel(config, T, views, hw):
    sc = scenes.make_scene(config, seed=T, num_tris=T, num_views=views, resolution=hw, with_targets=False)
    pos = torch.from_numpy(sc.clip_positions()).cuda()
    tri = torch.from_numpy(sc.tri).cuda()
    g = torch.Generator(device="cuda").manual_seed(T)
    alpha = torch.rand(sc.T, 15, 1, generator=g, device="cuda")
    rast = ds.rasterize_multires_triangle_alpha(hw, pos, tri, 2, alpha, stochastic=False)
    color = torch.rand(views, *hw, 3, generator=g, device="cuda")
    color[:, ::3] = 0.5  # equal neighbours: pairs without an adjoint
    grad = torch.randn(views, *hw, 3, generator=g, device="cuda")
    got, want = torch.zeros_like(pos), torch.zeros_like(pos)
    _core.backward_edge_grad(color, grad, rast, pos, got, tri)
    wide = lambda t: torch.nn.functional.pad(t, (0, 1)).contiguous()  # noqa: E731
    _core.backward_edge_grad(wide(color), wide(grad), rast, pos, want, tri)
    # FP32 sums of a few dozen contributions per vertex in another order; their magnitudes cancel at most 100-fold
    assert float((got - want).norm()) <= 1e-5 * float(want.norm()) + 1e-12
