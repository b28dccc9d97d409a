"""Multi-resolution triangle features: opacity, colour, level accumulation and
the shading MLP.

Drop-in for kenji-tojo/diffsoup python/diffsoup/multires.py (same public
functions, signatures, layouts and assertions).  rasterize_multires_triangle_alpha
runs the tiled rasterizer of csrc/tiled.cu with a counter-based stochastic
threshold instead of the fragment list plus torch.rand of the reference.
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch
from torch import nn

from . import _core
from . import tiles as _tiles


def feats_at_level(level: int) -> int:
    """Lattice samples per triangle at one level (multires.py:16-23)."""
    assert level >= 0
    return 3 if level == 0 else ((1 << (level - 1)) + 1) * ((1 << level) + 1)


def build_multires_triangle_color(T: int, min_level: int, max_level: int, feat_dim: int) -> torch.Tensor:
    """Zero (T, S, feat_dim) float32 buffer for levels [min_level, max_level] (multires.py:26-45)."""
    S = sum(feats_at_level(l) for l in range(min_level, max_level + 1))
    return torch.zeros(T, S, feat_dim, dtype=torch.float32)


# ---------------------------------------------------------------------------
#  Stochastic-opacity rasterisation (multires.py:52-102)
# ---------------------------------------------------------------------------

_iteration = 0


def _rng_state(device: torch.device) -> torch.Tensor:
    """Device (seed, iteration) for the Philox threshold.  The seed is drawn
    from torch's default CPU generator, so torch.manual_seed makes the masks
    reproducible."""
    global _iteration
    seed = int(torch.randint(0, 2 ** 62, (1,)).item())
    _iteration += 1
    return torch.tensor([seed, _iteration], dtype=torch.int64, device=device)


def rasterize_multires_triangle_alpha(resolution: Tuple[int, int], pos: torch.Tensor, tri: torch.Tensor, level: int,
                                      alpha_src: torch.Tensor, stochastic: bool = True) -> torch.Tensor:
    """Rasterise with per-fragment multires opacity and depth testing.

    Returns rast (B, H, W, 4) float32 = (b0, b1, z_ndc, tri_id + 1), 0 where
    nothing passes.  A fragment is kept when its opacity is >= its threshold:
    0.5 when stochastic is False (bit-identical IDs to the reference), else a
    uniform draw keyed by (seed, iteration, view, pixel, triangle).
    """
    H, W = resolution
    B, V, _ = pos.shape
    T, _ = tri.shape
    _, S, _ = alpha_src.shape
    dev = pos.device
    assert pos.shape == (B, V, 4) and pos.dtype == torch.float32 and pos.is_contiguous()
    assert tri.shape == (T, 3) and tri.dtype == torch.int32 and tri.is_contiguous()
    assert alpha_src.shape == (T, S, 1) and alpha_src.dtype == torch.float32 and alpha_src.is_contiguous()
    assert S == feats_at_level(level)
    assert pos.is_cuda and tri.device == dev and alpha_src.device == dev
    rast = torch.empty(B, H, W, 4, dtype=torch.float32, device=dev)
    if B == 0:
        return rast
    bins = _tiles.bin_views(pos, tri, [(H, W)] * B)
    a2 = alpha_src.view(T, S)
    if stochastic:
        _tiles.rasterize(bins, level, a2, rast, thr_mode=1, rng=_rng_state(dev))
    else:
        _tiles.rasterize(bins, level, a2, rast, thr_mode=0, thr_const=0.5)
    return rast


# ---------------------------------------------------------------------------
#  Colour MLP (multires.py:109-207)
# ---------------------------------------------------------------------------

def _gradients(x: torch.Tensor, mask: Optional[torch.Tensor], biases: torch.Tensor, weights, grad_out: torch.Tensor,
               need_x: bool):
    """The backward kernels' gradients of flat rows x [n,in] (None unless need_x), biases and weights in torch
    operations, which are differentiable.  Only the rows that mask covers are computed, as the kernels do: an
    infinity or NaN of another row would turn its zero gradient into NaN."""
    xs, g = x, grad_out
    if mask is not None:
        rows = mask.nonzero().squeeze(1)
        xs, g = x.index_select(0, rows), grad_out.index_select(0, rows)
    hs, b = [xs], biases.split([w.shape[0] for w in weights])
    for w, bw in zip(weights[:-1], b):
        hs.append(torch.relu(nn.functional.linear(hs[-1], w, bw)))
    y = torch.sigmoid(nn.functional.linear(hs[-1], weights[-1], b[-1]))
    res, aten = xs[:, 3:4], torch.ops.aten
    d = aten.sigmoid_backward(res * g, y)
    gw, gb = [], []
    for i in range(len(weights) - 1, -1, -1):
        gw.append(d.t() @ hs[i])
        gb.append(d.sum(0))
        if i > 0:
            d = aten.threshold_backward(d @ weights[i], hs[i], 0.0)
    gx = None
    if need_x:
        blend = torch.cat([(1.0 - res) * g, (g * (y - xs[:, :3])).sum(1, keepdim=True)], 1)
        gx = d @ weights[0] + nn.functional.pad(blend, (0, x.shape[1] - 4))
        if mask is not None:
            gx = torch.zeros_like(x).index_copy(0, rows, gx)
    return gx, torch.cat(gb[::-1]), gw[::-1]


class _ColorMLPFn(torch.autograd.Function):
    """ColorMLP on flat rows by ds_color_mlp_forward / _backward (csrc/color_mlp.cu)."""

    @staticmethod
    def forward(ctx, x, mask, biases, *weights):
        n, cin = x.shape
        out = torch.empty(n, 3, dtype=torch.float32, device=x.device)
        p = _core.ptr
        w1 = weights[1] if len(weights) == 3 else None
        _core.check(_core.lib.ds_color_mlp_forward(n, cin, 16, len(weights) - 1, p(x), p(mask), p(weights[0]), p(w1),
                                                   p(weights[-1]), p(biases), p(out), _core.stream()))
        ctx.save_for_backward(x, mask, biases, *weights)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        x, mask, biases, *weights = ctx.saved_tensors
        # create_graph, and a batch of gradients (vmap): the gradient in torch operations
        if torch.is_grad_enabled() or not _plain_call(grad_out):
            gx, gb, gw = _gradients(x, mask, biases, weights, grad_out, ctx.needs_input_grad[0])
            return (gx, None, gb, *gw)
        n, cin = x.shape
        layers = len(weights) - 1
        grad_out = grad_out.contiguous()
        gx = torch.empty_like(x) if ctx.needs_input_grad[0] else None
        gb = torch.empty_like(biases)
        gw = [torch.empty_like(w) for w in weights]
        ws = _core.workspace(_core.lib.ds_color_mlp_backward_workspace(n, cin, layers), x.device)
        p, two = _core.ptr, len(weights) == 3
        _core.check(_core.lib.ds_color_mlp_backward(
            n, cin, 16, layers, p(x), p(mask), p(weights[0]), p(weights[1] if two else None), p(weights[-1]), p(biases),
            p(grad_out), p(gx), p(gw[0]), p(gw[1] if two else None), p(gw[-1]), p(gb), p(ws), ws.numel(),
            _core.stream()))
        return (gx, None, gb, *gw)


def _plain_call(*tensors) -> bool:
    """Whether nothing watches or transforms torch operations on these tensors (tracing, compilation, function
    transforms, the batched gradients of autograd, forward-mode AD, dispatch modes), so that a kernel may take
    their place."""
    return (all(type(t) in (torch.Tensor, nn.Parameter) and not torch._C._functorch.is_legacy_batchedtensor(t)
                for t in tensors)
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling()
            and torch._C._functorch.peek_interpreter_stack() is None
            and torch.autograd.forward_ad._current_level < 0
            and torch._C._len_torch_dispatch_stack() == 0 and torch._C._len_torch_function_stack() == 0)


def _no_hooks(module: nn.Module) -> bool:
    return not (module._forward_hooks or module._forward_pre_hooks or module._backward_hooks
                or module._backward_pre_hooks or "forward" in module.__dict__)


class ColorMLP(nn.Module):
    """Per-pixel shading MLP with a residual blend.

    output = (1 - x[..., 3]) * x[..., :3] + x[..., 3] * sigmoid(MLP(x)), where
    MLP = n_layers hidden Linear+ReLU layers of width hidden_dim and a final
    Linear.  Module layout (``mlp`` = Sequential of Linear/ReLU/.../Sigmoid) and
    initialisation (Kaiming-uniform hidden layers, Xavier-uniform or zero output
    layer, zero biases) follow multires.py:128-167 so checkpoints interchange.
    """

    def __init__(self, input_dim: int, output_dim: int, hidden_dim: int = 16, n_layers: int = 2,
                 zero_last: bool = False):
        super().__init__()
        dims = [input_dim] + [hidden_dim] * n_layers
        mods = []
        for a, b in zip(dims[:-1], dims[1:]):
            mods += [nn.Linear(a, b), nn.ReLU()]
        mods += [nn.Linear(dims[-1], output_dim), nn.Sigmoid()]
        self.input_dim = input_dim
        self.output_dim = output_dim
        self.mlp = nn.Sequential(*mods)
        self._init_weights(zero_last)

    def _init_weights(self, zero_last: bool = False) -> None:
        lins = [m for m in self.mlp if isinstance(m, nn.Linear)]
        for lin in lins[:-1]:
            nn.init.kaiming_uniform_(lin.weight, a=0.0, mode="fan_in", nonlinearity="relu")
            nn.init.zeros_(lin.bias)
        last = lins[-1]
        if zero_last:
            nn.init.zeros_(last.weight)
        else:
            nn.init.xavier_uniform_(last.weight, gain=1.0)
        nn.init.zeros_(last.bias)

    def _fused_layers(self, x: torch.Tensor, mask: Optional[torch.Tensor]):
        """The Linear layers when the fused kernels compute exactly this call: FP32 on the current CUDA device,
        4 to 20 inputs, one or two hidden layers of 16, three outputs, and the plain module as built here."""
        mods = list(self.mlp) if type(self.mlp) is nn.Sequential else []
        kinds = [type(m) for m in mods]
        if kinds not in ([nn.Linear, nn.ReLU] * n + [nn.Linear, nn.Sigmoid] for n in (1, 2)):
            return None
        lins = mods[0::2]
        shapes = [(16, self.input_dim)] + [(16, 16)] * (len(lins) - 2) + [(3, 16)]
        g = nn.modules.module
        if (not 4 <= self.input_dim <= 20 or self.output_dim != 3 or x.numel() == 0
                or not (x.is_cuda and x.dtype == torch.float32 and x.device.index == torch.cuda.current_device())
                or (mask is not None and not (type(mask) is torch.Tensor and mask.dtype == torch.bool
                                              and mask.device == x.device))
                or g._global_forward_hooks or g._global_forward_pre_hooks or g._global_backward_hooks
                or g._global_backward_pre_hooks or torch.is_autocast_enabled("cuda") or not all(_no_hooks(m) for m in mods + [self.mlp])):
            return None
        for lin, shape in zip(lins, shapes):
            if lin.bias is None or tuple(lin.weight.shape) != shape or any(
                    t.device != x.device or t.dtype != torch.float32 or not t.is_contiguous()
                    for t in (lin.weight, lin.bias)):
                return None
        return lins if _plain_call(x, *(t for lin in lins for t in (lin.weight, lin.bias))) else None

    def forward(self, x: torch.Tensor, mask: Optional[torch.Tensor] = None) -> torch.Tensor:
        B, H, W, _ = x.shape
        assert x.shape == (B, H, W, self.input_dim)
        assert mask is None or mask.shape == (B, H, W)
        lins = self._fused_layers(x, mask)
        if lins is not None:
            weights = [lin.weight for lin in lins]
            biases = torch.cat([lin.bias for lin in lins])
            if mask is None:
                return _ColorMLPFn.apply(x.reshape(-1, self.input_dim).contiguous(), None, biases,
                                         *weights).view(B, H, W, 3)
            if not mask.any():
                return torch.zeros(B, H, W, 3, device=x.device, dtype=x.dtype)
            rows, flags = x.reshape(-1, self.input_dim).contiguous(), mask.reshape(-1).contiguous()
            if torch.is_grad_enabled():
                # copies: writing to x or mask before backward is allowed here, as it is when rows are gathered
                rows, flags = rows.clone(), flags.clone()
            return _ColorMLPFn.apply(rows, flags, biases, *weights).view(B, H, W, 3)
        rgb, res = x[..., :3], x[..., 3:4]
        if mask is None:
            y = self.mlp(x.reshape(-1, self.input_dim)).view(B, H, W, self.output_dim)
            return (1.0 - res) * rgb + res * y
        flat = x.reshape(-1, self.input_dim)
        m = mask.reshape(-1)
        out = torch.zeros(B * H * W, self.output_dim, device=x.device, dtype=x.dtype)
        if m.any():
            sel = flat[m]
            y = self.mlp(sel)
            r = sel[:, 3:4]
            out[m] = (1.0 - r) * sel[:, :3] + r * y
        return out.view(B, H, W, self.output_dim)


# ---------------------------------------------------------------------------
#  Per-pixel feature interpolation (multires.py:214-272)
# ---------------------------------------------------------------------------

class _MultiresTriangleColorFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, rast, min_level, max_level, feat):
        B, H, W, _ = rast.shape
        out = torch.empty((B, H, W, feat.shape[2]), dtype=torch.float32, device=rast.device)
        _core.multires_triangle_color_set(rast, min_level, max_level, feat, out)
        ctx.save_for_backward(rast)
        ctx.levels = (min_level, max_level)
        ctx.feat_shape = tuple(feat.shape)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        (rast,) = ctx.saved_tensors
        lo, hi = ctx.levels
        grad_feat = torch.zeros(ctx.feat_shape, dtype=torch.float32, device=rast.device)
        _core.backward_multires_triangle_color(rast, lo, hi, grad_feat, grad_out.contiguous())
        return None, None, None, grad_feat


def multires_triangle_color(rast: torch.Tensor, level: int, feat: torch.Tensor) -> torch.Tensor:
    """Interpolate (T, S, C) features at one level per pixel: (B, H, W, C)."""
    B, H, W, _ = rast.shape
    _, S, _ = feat.shape
    dev = rast.device
    assert rast.shape == (B, H, W, 4) and rast.dtype == torch.float32 and rast.is_contiguous()
    assert feat.dim() == 3 and feat.dtype == torch.float32 and feat.is_contiguous()
    assert S == feats_at_level(level)
    assert rast.is_cuda and feat.device == dev
    return _MultiresTriangleColorFn.apply(rast, level, level, feat)


# ---------------------------------------------------------------------------
#  Cross-level accumulation (multires.py:279-339)
# ---------------------------------------------------------------------------

class _AccumulateToLevelFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, min_level, max_level, target_level, feat):
        T, _, Cd = feat.shape
        out = torch.empty(T, feats_at_level(target_level), Cd, dtype=torch.float32, device=feat.device)
        _core.accumulate_to_level_forward(min_level, max_level, target_level, feat, out)
        ctx.levels = (min_level, max_level, target_level)
        ctx.feat_shape = tuple(feat.shape)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        lo, hi, tl = ctx.levels
        grad_feat = torch.empty(ctx.feat_shape, dtype=torch.float32, device=grad_out.device)
        _core.accumulate_to_level_backward_set(lo, hi, tl, grad_feat, grad_out.contiguous())
        return None, None, None, grad_feat


def accumulate_to_level(min_level: int, max_level: int, feat: torch.Tensor,
                        target_level: Optional[int] = None) -> torch.Tensor:
    """Evaluate levels [min_level, max_level] on the lattice of target_level
    (default max_level): (T, S_target, C)."""
    assert min_level >= 0
    assert feat.ndim == 3 and feat.dtype == torch.float32
    assert feat.is_contiguous() and feat.is_cuda
    if target_level is None:
        target_level = max_level
    return _AccumulateToLevelFn.apply(min_level, max_level, target_level, feat)
