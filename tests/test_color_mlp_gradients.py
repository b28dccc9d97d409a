"""ColorMLP's torch form of the fused kernels, which a differentiable backward goes through: values of pixels that the
mask leaves out reach no gradient."""

import types

import pytest
import torch

from diffsoup_b200 import ColorMLP, multires


def rows(dev, n=60, cin=11):
    g = torch.Generator().manual_seed(3)
    torch.manual_seed(3)
    mlp = ColorMLP(cin, 3, 16, 2).to(dev)
    x, mask = torch.rand(1, 1, n, cin, generator=g), torch.rand(1, 1, n, generator=g) < 0.6
    mask[0, 0, :3] = False
    clean = x.clone()
    x[0, 0, 0], x[0, 0, 1, 5], x[0, 0, 2, 3] = float("nan"), float("inf"), float("-inf")
    return mlp, x.to(dev), clean.to(dev), mask.to(dev), torch.randn(1, 1, n, 3, generator=g).to(dev)


def backward_on(mlp, x, mask, g):
    """_ColorMLPFn.backward with gradients enabled, as create_graph runs it: gradients of x, biases and weights."""
    lins = [m for m in mlp.mlp if isinstance(m, torch.nn.Linear)]
    saved = (x.view(-1, x.shape[-1]), None if mask is None else mask.view(-1), torch.cat([m.bias for m in lins]),
             *[m.weight for m in lins])
    ctx = types.SimpleNamespace(saved_tensors=saved, needs_input_grad=[True, False] + [True] * (len(lins) + 1))
    gx, _, gb, *gw = multires._ColorMLPFn.backward(ctx, g.view(-1, 3))
    return [gx.view_as(x), gb, *gw]


def test_differentiable_backward_leaves_masked_rows_out():
    """First gradients with create_graph, and a second derivative, against the module on rows without infinities and
    NaN."""
    mlp, x, clean, mask, g = rows("cpu")
    lins = [m for m in mlp.mlp if isinstance(m, torch.nn.Linear)]
    weights = [m.weight for m in lins]

    def second(first):
        return torch.autograd.grad(first[0][mask].square().sum() + first[2].square().sum(), weights)

    x.requires_grad_(True)
    got = backward_on(mlp, x, mask, g)
    clean.requires_grad_(True)
    want = torch.autograd.grad(mlp(clean, mask=mask), [clean, *[m.bias for m in lins], *weights], g, create_graph=True)
    want = [want[0], torch.cat(want[1:4]), *want[4:]]
    for a, b in zip([*got, *second(got)], [*want, *second(want)]):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("layers", [1, 2])
@pytest.mark.parametrize("cover", [None, 0.0, 0.5, 1.0])
def test_differentiable_backward_is_the_modules(layers, cover):
    """Every gradient, and the gradients of a function of them, in FP64 (chains of at most 60 products and sums)."""
    torch.manual_seed(layers)
    mlp = ColorMLP(7, 3, 16, layers).double()
    x = torch.randn(1, 6, 10, 7, dtype=torch.float64, requires_grad=True)
    g = torch.randn(1, 6, 10, 3, dtype=torch.float64, requires_grad=True)
    mask = None if cover is None else torch.rand(1, 6, 10) < cover
    lins = [m for m in mlp.mlp if isinstance(m, torch.nn.Linear)]
    weights, biases = [m.weight for m in lins], [m.bias for m in lins]
    got = backward_on(mlp, x, mask, g)
    y = mlp(x, mask=mask) + 0.0 * sum(t.sum() for t in (x, *weights, *biases))  # nothing covered: zero gradients
    want = torch.autograd.grad(y, [x, *biases, *weights], g, create_graph=True)
    want = [want[0], torch.cat(want[1:len(lins) + 1]), *want[len(lins) + 1:]]
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, rtol=1e-11, atol=1e-13)
    second = [torch.autograd.grad(sum(t.sin().sum() for t in first), [x, g, *weights, *biases], materialize_grads=True)
              for first in (got, want)]
    for a, b in zip(*second):
        torch.testing.assert_close(a, b, rtol=1e-10, atol=1e-12)


class TorchForward(torch.autograd.Function):
    """_ColorMLPFn with the module's own operations in the forward, so that its backward runs without a GPU."""

    @staticmethod
    def forward(ctx, x, mask, biases, *weights):
        ctx.save_for_backward(x, mask, biases, *weights)
        mlp = ColorMLP(x.shape[1], 3, 16, len(weights) - 1)
        with torch.no_grad():
            for lin, w, b in zip([m for m in mlp.mlp if isinstance(m, torch.nn.Linear)], weights,
                                 biases.split([w.shape[0] for w in weights])):
                lin.weight.copy_(w), lin.bias.copy_(b)
            return mlp(x[None, None], None if mask is None else mask[None, None])[0, 0]

    backward = staticmethod(multires._ColorMLPFn.backward)


def batched(out, inputs, gs):
    """The three ways to ask for a batch of gradients, each against one gradient at a time."""
    want = [torch.stack(t) for t in zip(*(torch.autograd.grad(out, inputs, g, retain_graph=True) for g in gs))]
    one = lambda g: torch.autograd.grad(out, inputs, g, retain_graph=True)  # noqa: E731
    for got in (torch.autograd.grad(out, inputs, gs, retain_graph=True, is_grads_batched=True),
                torch.func.vmap(one)(gs),
                torch.autograd.grad(out, inputs, gs, retain_graph=True, is_grads_batched=True, create_graph=True)):
        for a, b in zip(got, want):
            torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("masked", [False, True])
def test_batched_gradients(masked):
    mlp, _, x, mask, _ = rows("cpu")
    lins = [m for m in mlp.mlp if isinstance(m, torch.nn.Linear)]
    weights, x, mask = [m.weight for m in lins], x.view(-1, 11).requires_grad_(True), mask.view(-1) if masked else None
    out = TorchForward.apply(x, mask, torch.cat([m.bias for m in lins]), *weights)
    want = mlp(x[None, None], None if mask is None else mask[None, None])[0, 0]
    gs = torch.randn(4, *out.shape, generator=torch.Generator().manual_seed(0))
    inputs = [x, *mlp.parameters()]
    for g in gs:  # backward without create_graph needs the kernels: compared through the batch of one
        for a, b in zip(torch.autograd.grad(out, inputs, g[None], retain_graph=True, is_grads_batched=True),
                        torch.autograd.grad(want, inputs, g, retain_graph=True)):
            torch.testing.assert_close(a[0], b, rtol=1e-5, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("masked", [False, True])
def test_batched_gradients_of_the_fused_call(masked):
    mlp, _, x, mask, _ = rows("cuda")
    x.requires_grad_(True)
    out = mlp(x, mask=mask if masked else None)
    assert "_ColorMLPFn" in str(out.grad_fn.next_functions)
    gs = torch.randn(4, *out.shape, generator=torch.Generator().manual_seed(0)).cuda()
    batched(out, [x, *mlp.parameters()], gs)


@pytest.mark.gpu
def test_create_graph_leaves_masked_rows_out():
    """The call with create_graph=True, on the rows with infinities and NaN, against the clean rows without it."""
    mlp, x, clean, mask, g = rows("cuda")
    assert mlp._fused_layers(x, mask) is not None

    def grads(x, create_graph):
        x = x.clone().requires_grad_(True)
        return torch.autograd.grad(mlp(x, mask=mask), [x, *mlp.parameters()], g, create_graph=create_graph)

    for a, b in zip(grads(x, True), grads(clean, False)):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)
