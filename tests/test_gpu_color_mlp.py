"""The fused ColorMLP kernels against the module's own torch operations in FP64, and the calls that keep to the
torch operations."""

import copy

import pytest
import torch

from diffsoup_b200 import ColorMLP, multires

pytestmark = pytest.mark.gpu
DEV = "cuda"


def make(cin, layers, shape, cover, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    torch.manual_seed(seed)
    mlp = ColorMLP(cin, 3, 16, layers).to(DEV)
    with torch.no_grad():
        for p in mlp.parameters():
            p.add_(0.1 * torch.randn(p.shape, generator=g, device=DEV))
    x = torch.rand(*shape, cin, generator=g, device=DEV)
    mask = None if cover is None else torch.rand(*shape, generator=g, device=DEV) < cover
    if mask is not None:  # a pixel whose hidden sum is zero within FP32 rounding has no FP64 gradient to compare with
        h = x.double()
        for lin in [m for m in mlp.mlp if isinstance(m, torch.nn.Linear)][:-1]:
            z = h @ lin.weight.double().T + lin.bias.double()
            mask &= (z.abs() > 1e-5).all(-1)
            h = torch.relu(z)
    return mlp, x, mask, torch.randn(*shape, 3, generator=g, device=DEV)


def run(mlp, x, mask, gout):
    x = x.detach().clone().requires_grad_(True)
    out = mlp(x, mask=mask)
    grads = torch.autograd.grad(out, [x] + list(mlp.parameters()), gout)
    return [out.detach()] + list(grads)


# every padded input width, both depths, pixel counts around a warp's and a CTA's, more than one pass of the grid
@pytest.mark.parametrize("cin", [4, 11, 12, 13, 16, 19, 20])
@pytest.mark.parametrize("layers", [1, 2])
@pytest.mark.parametrize("shape,cover", [((1, 1, 1), None), ((1, 3, 11), 0.5), ((2, 16, 17), 0.02), ((1, 401, 397), 0.6)])
def test_matches_torch_in_fp64(cin, layers, shape, cover):
    mlp, x, mask, g = make(cin, layers, shape, cover, seed=cin)
    assert mlp._fused_layers(x, mask) is not None
    got = run(mlp, x, mask, g)
    d = copy.deepcopy(mlp).double()
    assert d._fused_layers(x.double(), mask) is None
    want = run(d, x.double(), mask, g.double())
    for a, b in zip(got, want):
        # chains of 16 to 20 FP32 products; the parameters' gradients sum up to 160,000 pixels (pairwise by CTA)
        assert float((a.double() - b).norm()) < 1e-5 * float(b.norm()) + 1e-7
    if mask is not None:
        assert (got[0][~mask] == 0).all() and (got[1][~mask] == 0).all()


def test_rows_that_are_not_vectors_and_repeat_runs():
    mlp, x, mask, g = make(16, 2, (1, 57, 63), 0.7)
    flat = torch.empty(x.numel() + 1, device=DEV)
    flat[1:] = x.reshape(-1)
    shifted = flat[1:].view_as(x)  # 4 bytes past an aligned address
    ref = run(mlp, x, mask, g)
    with torch.no_grad():
        assert torch.equal(mlp(shifted, mask=mask), ref[0])
    wide = torch.cat([x, x], -1)[..., :16]  # strided rows
    assert torch.equal(mlp(wide, mask=mask), ref[0])
    for a, b in zip(ref, run(mlp, x, mask, g)):
        assert torch.equal(a, b)


def test_second_derivatives_and_frozen_parameters():
    mlp, x, mask, _ = make(11, 2, (1, 5, 7), 0.8)
    d = copy.deepcopy(mlp).double()

    def penalty(m, x):
        x = x.detach().clone().requires_grad_(True)
        (gx,) = torch.autograd.grad(m(x, mask=mask).square().sum(), x, create_graph=True)
        return torch.autograd.grad(gx.square().sum(), [x] + list(m.parameters()), allow_unused=True)

    for a, b in zip(penalty(mlp, x), penalty(d, x.double())):
        if b is None:
            assert a is None or float(a.abs().max()) == 0
        else:
            assert float((a.double() - b).norm()) < 1e-4 * float(b.norm()) + 1e-7
    for p in mlp.parameters():
        p.requires_grad_(False)
    assert not mlp(x, mask=mask).requires_grad
    x.requires_grad_(True)
    out = mlp(x, mask=mask)
    with torch.no_grad():
        x.zero_()  # the masked call works on its own copy of the rows
    out.sum().backward()
    assert float(x.grad.abs().sum()) > 0


def test_other_calls_keep_the_torch_operations():
    mlp, x, mask, _ = make(16, 2, (1, 8, 9), 0.5)
    assert not mlp(x, mask=torch.zeros_like(mask)).requires_grad  # nothing covered: plain zeros
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert mlp._fused_layers(x, mask) is None
    seen = []
    h = mlp.mlp[0].register_forward_hook(lambda *a: seen.append(1))
    mlp(x, mask=mask)
    h.remove()
    assert seen == [1]
    assert mlp._fused_layers(x.half(), mask) is None and mlp._fused_layers(x, mask.float()) is None
    params = {k: v.detach() for k, v in mlp.named_parameters()}
    f = lambda p: torch.func.functional_call(mlp, p, (x,)).sum()  # noqa: E731
    gr = torch.func.grad(f)(params)
    ref = run(mlp, x, None, torch.ones(1, 8, 9, 3, device=DEV))[2:]
    for a, b in zip(gr.values(), ref):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)
    assert multires.ColorMLP(16, 3, 64, 2).to(DEV)._fused_layers(x, mask) is None
    assert multires.ColorMLP(16, 4, 16, 2).to(DEV)._fused_layers(x, mask) is None
