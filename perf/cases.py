"""The work that users of diffsoup_b200 have it do, as cases that can be timed and compared.

Twelve listed cases cover the package's public entry points over the sizes of its benchmark
configurations and tests: whole training steps (`TrainStep`), the operators of a training loop written
with autograd (rasterisation, feature lookup, level accumulation, edge and opacity gradients), the optimiser
updates, the inference render and the resampling pass.  `draw` gives further cases of the same ranges.

  kind       entry points                                                     range
  step       TrainStep.run, eager or captured                                 500 - 200,000 triangles, 1 - 8 views
  view       the operators of one training iteration on one view, autograd    1,000 - 60,000 triangles
  raster     rasterize_multires_triangle_alpha                                500 - 60,000 triangles
  levels     accumulate_to_level, forward and backward                        500 - 200,000 triangles, 1 - 16 channels
  features   multires_triangle_color (both ways), encode_view_dir_sh2         1 - 8 views, 4 - 16 channels
  hooks      edge_grad and opacity_aux_loss, forward and backward             1 - 4 views
  adam       VectorAdam and Adam over a soup's parameters                     500 - 200,000 triangles
  render     viewer.Renderer: frames of a soup                                1 - 8 views, LUT level 3 - 5
  resample   count_visible_triangles and split_triangle_soup_clip_until       1,000 - 60,000 triangles

`exact` restates the paths in 64-bit torch: fragments of every triangle, nearest fragment per pixel,
shading with autograd, and the edge and opacity estimators.  Visibility is decided there in 64 bits too, so a
few pixels on triangle borders differ from any FP32 rasterizer.
"""

import math

import numpy as np
import torch
import torch.nn.functional as F

import diffsoup_b200 as ds
from diffsoup_b200 import optimize, remesh, scenes, viewer, visibility
from diffsoup_b200.step import TrainStep

# Shading models that have fused training kernels: feature channels, view encoding, hidden width and
# layers, lattice levels.  "ref" is the reference's own model.
MODELS = {
    "dir8": dict(C=8, enc="dir3", hidden=16, layers=1, lo=0, hi=2),
    "ref": dict(C=7, enc="sh2", hidden=16, layers=2, lo=0, hi=2),
    "wide16": dict(C=16, enc="dir3", hidden=64, layers=2, lo=0, hi=3),
}


def listed():
    return [
        # one small view a step: launches and latency (5,000-triangle uniform soup, 256x256)
        dict(name="step_tiny", kind="step", soup="box", tris=5000, views=1, height=256, width=256, ragged=False,
             model="dir8", precision="split", u8=False, graph=True),
        # the benchmark workload: 8 views of 800x800 of a 15,000-triangle shell, 8-bit targets, replayed
        dict(name="step_batch", kind="step", soup="shell", tris=15000, views=8, height=800, width=800, ragged=False,
             model="dir8", precision="split", u8=True, graph=True),
        # unbounded-scene captures: clustered soup, views of uneven size (so not captured), the reference's model
        dict(name="step_ragged", kind="step", soup="cluster", tris=60000, views=6, height=799, width=1065,
             ragged=True, model="ref", precision="split", u8=True, graph=False),
        # the largest: 200,000 triangles, full-HD views, the wide MLP in BF16
        dict(name="step_wide", kind="step", soup="cluster", tris=200000, views=3, height=1080, width=1920,
             ragged=False, model="wide16", precision="bf16", u8=False, graph=True),
        # a training loop on the drop-in operators: one view, autograd, the reference's model
        dict(name="view_ops", kind="view", soup="shell", tris=15000, views=1, height=800, width=800, model="ref"),
        # the smallest call: the ID buffer of a small view, e.g. for previews and picking
        dict(name="raster_small", kind="raster", soup="box", tris=1500, views=1, height=200, width=255, hi=2),
        # features of a soup brought to the finest lattice, and the gradient back to all levels
        dict(name="levels_mid", kind="levels", tris=60000, C=7, lo=0, hi=3),
        # per-pixel shading inputs of a batch and their gradient
        dict(name="features_batch", kind="features", soup="shell", tris=15000, views=4, height=800, width=800, C=7,
             hi=2),
        # the two gradient hooks of the training loop on a small batch
        dict(name="hooks_batch", kind="hooks", soup="shell", tris=15000, views=2, height=601, width=803, hi=2),
        # the parameter update after a step on a large soup
        dict(name="adam_large", kind="adam", tris=60000, C=7, lo=0, hi=2),
        # frames of a trained soup at the viewer's level and size
        dict(name="render_view", kind="render", soup="shell", tris=15000, views=1, height=1200, width=1200, level=5,
             graph=False),
        # densification between training phases: visible faces of the training views, then the longest edges
        # of one view split under a cap on the soup's growth
        dict(name="resample", kind="resample", soup="shell", tris=15000, views=16, height=800, width=800, hi=2,
             tau=0.01, cap=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "view", "raster", "levels", "features", "hooks", "adam", "render",
                       "resample"])
    c = dict(kind=kind)
    if kind in ("levels", "adam"):
        c.update(tris=_log(rng, 500, 200000), C=rng.choice([1, 3, 4, 7, 8, 16]), lo=rng.choice([0, 0, 1]),
                 hi=rng.choice([2, 3]))
        if kind == "adam":
            c["C"] = rng.choice([7, 8])
        return c
    side = _log(rng, 64, 1100)
    aspect = rng.choice([1.0, 4 / 3, 16 / 9, 0.75, 1.1])
    c.update(soup=rng.choice(["box", "shell", "cluster"]), height=side, width=max(16, int(side * aspect) + rng.randint(-3, 3)))
    pixels = c["height"] * c["width"]
    most = max(1, min(8, int(5_000_000 // pixels)))  # pixels of a batch: at most the benchmark's
    c["views"] = rng.randint(1, most)
    if kind == "step":
        c["model"] = rng.choice(["dir8", "ref", "wide16"])
        c["precision"] = "bf16" if c["model"] == "wide16" else rng.choice(["split", "split", "bf16"])
        c["tris"] = _log(rng, 500, 60000 if c["views"] > 2 else 200000)
        c["ragged"] = rng.random() < 0.4 and c["views"] > 1
        c["u8"] = rng.random() < 0.5
        c["graph"] = not c["ragged"]
        return c
    c["tris"] = _log(rng, 1000, 60000)
    c["hi"] = rng.choice([2, 2, 3])
    if kind == "view":
        c.update(views=1, model="ref")
        del c["hi"]
    elif kind == "raster":
        c["tris"] = _log(rng, 500, 60000)
    elif kind == "features":
        c["C"] = rng.choice([4, 7, 8, 16])
    elif kind == "hooks":
        c["views"] = min(c["views"], 4)
    elif kind == "render":
        c["level"] = rng.choice([3, 4, 5])
        c["tris"] = min(c["tris"], 20000)
        c["graph"] = rng.random() < 0.5
        del c["hi"]
    elif kind == "resample":
        c.update(tau=0.005, cap=c["tris"] // 32)
    return c


# ---------------------------------------------------------------------------
#  Inputs
# ---------------------------------------------------------------------------

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _soup(case, g):
    """Soup vertices [3T,3] and faces [T,3]: centres uniform in a box, on a noisy shell, or clustered, and the
    three corners of each face spread around its centre (as diffsoup_b200.scenes draws them)."""
    T, dev = case["tris"], _dev()
    n = lambda *s: torch.randn(*s, generator=g, device=dev)  # noqa: E731
    u = lambda *s: torch.rand(*s, generator=g, device=dev) * 2 - 1  # noqa: E731
    if case["soup"] == "box":
        centres = u(T, 3)
    elif case["soup"] == "shell":
        centres = F.normalize(n(T, 3), dim=1) * (1 + 0.1 * n(T, 1))
    else:
        lab = torch.randint(0, 20, (T,), generator=g, device=dev)
        centres = (3 * u(20, 3))[lab] + 0.3 * n(T, 3)
    verts = (centres[:, None] + 0.05 * n(T, 3, 3)).reshape(-1, 3).contiguous()
    return verts, torch.arange(3 * T, device=dev, dtype=torch.int32).reshape(T, 3)


def _sizes(case):
    """Heights and widths of the views: uneven sizes shrink from the first view's by a fixed sequence."""
    h, w = case["height"], case["width"]
    if not case.get("ragged"):
        return [(h, w)] * case["views"]
    k = [1.0, 0.62, 0.87, 0.45, 0.93, 0.71, 0.55, 0.8]
    return [(max(1, int(h * k[b % 8]) - b % 3), max(1, int(w * k[(b + 3 * (b % 2)) % 8]))) for b in range(case["views"])]


def _cameras(case, seed):
    """Row-major MVPs and inverses, a camera ring around the soup whose start follows the seed."""
    r = np.random.default_rng(seed + 31)
    radius = {"box": 3.0, "shell": 4.0, "cluster": 5.0}[case["soup"]]
    turn, mvps = r.uniform(0, 2 * math.pi), []
    for b, (h, w) in enumerate(_sizes(case)):
        a = turn + 2 * math.pi * b / case["views"]
        eye = radius * np.array([math.cos(a), math.sin(a), 0.3])
        mvps.append(scenes.projection_matrix(40.0, w, h) @ np.linalg.inv(scenes.look_at_c2w(eye)))
    m = np.stack(mvps)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(_dev())  # noqa: E731
    return t(m), t(np.linalg.inv(m))


def _mlp(C_in, hidden, layers, seed):
    ws = scenes.mlp_weights(C_in, 3, hidden, layers, seed=seed)
    return [(torch.from_numpy(W).to(_dev()), torch.from_numpy(b).to(_dev())) for W, b in ws]


def _opacity(case, g):
    """Opacities [T,S] of the finest level, as a sigmoid of level-accumulated logits gives them."""
    S = scenes.feats_at_level(case["hi"])
    return torch.sigmoid(1.2 * torch.randn(case["tris"], S, generator=g, device=_dev()))


def _clip(verts, mvp):
    return torch.einsum("bij,nj->bni", mvp, F.pad(verts, (0, 1), value=1.0)).contiguous()


def prepare(case, seed):
    g, dev, kind = _gen(seed), _dev(), case["kind"]
    s = dict(case=case)
    if kind == "levels":
        S = scenes.total_feats(case["lo"], case["hi"])
        s["feat"] = (0.1 * torch.randn(case["tris"], S, case["C"], generator=g, device=dev)).requires_grad_()
        s["grad"] = torch.randn(case["tris"], scenes.feats_at_level(case["hi"]), case["C"], generator=g, device=dev)
        return s
    if kind == "adam":
        S = scenes.total_feats(case["lo"], case["hi"])
        n = lambda *z: torch.randn(*z, generator=g, device=dev)  # noqa: E731
        shapes = [(case["tris"], S, case["C"]), (case["tris"], S, 1), (16, case["C"] + 9), (16,), (16, 16), (16,),
                  (3, 16), (3,)]
        s["verts"] = n(3 * case["tris"], 3).requires_grad_()
        s["params"] = [(0.1 * n(*z)).requires_grad_() for z in shapes]
        for p in [s["verts"]] + s["params"]:
            p.grad = 1e-3 * n(*p.shape)
        s["opts"] = [optimize.VectorAdam([s["verts"]], lr=1e-3), optimize.Adam(s["params"], lr=5e-3)]
        return s
    s["verts"], s["tri"] = _soup(case, g)
    s["mvp"], s["inv"] = _cameras(case, seed)
    H, W, B = case["height"], case["width"], case["views"]
    if kind == "step":
        m = MODELS[case["model"]]
        S = scenes.total_feats(m["lo"], m["hi"])
        hw = _sizes(case)
        step = TrainStep(case["tris"], 3 * case["tris"], hw, m["C"], m["lo"], m["hi"], m["hidden"], m["layers"],
                         stochastic=True, seed=seed, precision=case["precision"], view_enc=m["enc"],
                         target_u8=case["u8"])
        P = step.num_pixels
        s["feat"] = 0.1 * torch.randn(case["tris"], S, m["C"], generator=g, device=dev)
        s["alpha"] = torch.randn(case["tris"], S, generator=g, device=dev)
        s["mlp"] = _mlp(m["C"] + (9 if m["enc"] == "sh2" else 3), m["hidden"], m["layers"], seed)
        flat = torch.cat([t.reshape(-1) for wb in s["mlp"] for t in wb])
        s["target"] = (torch.randint(0, 256, (P, 3), generator=g, device=dev, dtype=torch.uint8) if case["u8"]
                       else torch.rand(P, 3, generator=g, device=dev))
        s["step"], s["flat"] = step, flat
        s["args"] = (s["verts"], s["tri"], s["mvp"], s["inv"], s["feat"], s["alpha"], flat, s["target"])
        if case["graph"]:  # fixed shapes: a program tunes and captures its step once
            step.autotune(*s["args"])
            s["graph"] = step.capture(*s["args"])
        else:
            step.fit_capacity(*s["args"])
        step.rng[1] = 0
        step.status.zero_()
        return s
    if kind == "view":
        m = MODELS[case["model"]]
        S = scenes.total_feats(m["lo"], m["hi"])
        s["verts"].requires_grad_()
        s["feat"] = (0.1 * torch.randn(case["tris"], S, m["C"], generator=g, device=dev)).requires_grad_()
        s["alpha"] = torch.randn(case["tris"], S, 1, generator=g, device=dev).requires_grad_()
        s["mlp"] = ds.ColorMLP(m["C"] + 9, 3, m["hidden"], m["layers"]).to(dev)
        lins = [x for x in s["mlp"].modules() if isinstance(x, torch.nn.Linear)]
        with torch.no_grad():
            for lin, (w, b) in zip(lins, _mlp(m["C"] + 9, m["hidden"], m["layers"], seed)):
                lin.weight.copy_(w)
                lin.bias.copy_(b)
        s["target"] = torch.rand(B, H, W, 3, generator=g, device=dev)
        return s
    if kind == "render":
        S, T = scenes.feats_at_level(case["level"]), case["tris"]
        lut = torch.rand(T * S, 8, generator=g, device=dev)
        lut[:, 7] = torch.sigmoid(0.5 + 2 * torch.randn(T * S, generator=g, device=dev))
        lut0, lut1 = viewer.quantize_lut(viewer.pack_face_color_lut(lut[:, :7], lut[:, 7:], T, case["level"]))
        mlp = [t.cpu() for wb in _mlp(16, 16, 2, seed) for t in wb]
        s["r"] = viewer.Renderer(s["verts"], s["tri"], lut0, lut1, *mlp, level=case["level"])
        s["mvp_host"] = s["mvp"].cpu()
        s["frame"] = s["r"].frame(s["mvp_host"], H, W)
        if case["graph"]:
            s["graph"] = s["frame"].capture()
        return s
    s["opacity"] = _opacity(case, g)
    if kind == "resample":
        return s
    s["pos"] = _clip(s["verts"], s["mvp"])
    if kind == "raster":
        s["opacity"] = s["opacity"].unsqueeze(-1)
        return s
    s["rast"] = ds.rasterize_multires_triangle_alpha((H, W), s["pos"], s["tri"], case["hi"],
                                                     s["opacity"].unsqueeze(-1), stochastic=False)
    if kind == "features":
        S = scenes.feats_at_level(case["hi"])
        s["feat"] = torch.rand(case["tris"], S, case["C"], generator=g, device=dev).requires_grad_()
        s["grad"] = torch.randn(B, H, W, case["C"], generator=g, device=dev) / (B * H * W)
    else:
        s["pos"].requires_grad_()
        s["alpha"] = s["opacity"].unsqueeze(-1).clone().requires_grad_()
        s["target"] = torch.rand(B, H, W, 3, generator=g, device=dev)
        mask = (s["rast"][..., 3:] > 0).float()
        smooth = 0.5 + 0.3 * torch.sin(0.7 * s["rast"][..., 3:] + torch.arange(3, device=dev)) + 0.1 * s["rast"][..., :1]
        s["color"] = (mask * smooth + (1 - mask)).contiguous().requires_grad_()
        s["grad"] = (2 * (s["color"].detach() - s["target"]) / s["target"].numel()).contiguous()
    return s


# ---------------------------------------------------------------------------
#  One pass
# ---------------------------------------------------------------------------

def run(s):
    case, kind = s["case"], s["case"]["kind"]
    H, W = case.get("height"), case.get("width")
    if kind == "step":
        step = s["step"]
        if case["graph"]:
            s["graph"].replay()
        else:
            step.run(*s["args"])
        return dict(loss=step.loss, verts=step.grad_verts, feat=step.grad_feat_src, alpha=step.grad_alpha_src,
                    mlp=step.grad_mlp)
    if kind == "levels":
        out = ds.accumulate_to_level(case["lo"], case["hi"], s["feat"])
        (grad,) = torch.autograd.grad(out, s["feat"], s["grad"])
        return dict(out=out, grad=grad)
    if kind == "features":
        out = ds.multires_triangle_color(s["rast"], case["hi"], s["feat"])
        enc = ds.encode_view_dir_sh2(s["rast"], s["inv"])
        (grad,) = torch.autograd.grad(out, s["feat"], s["grad"])
        return dict(out=out, enc=enc, grad=grad)
    if kind == "raster":
        return ds.rasterize_multires_triangle_alpha((H, W), s["pos"], s["tri"], case["hi"], s["opacity"],
                                                    stochastic=False)
    if kind == "hooks":
        aux = ds.opacity_aux_loss(s["color"].detach(), s["target"], s["rast"], s["pos"].detach(), s["tri"],
                                  case["hi"], s["alpha"])
        out = ds.edge_grad(s["color"], s["rast"], s["pos"], s["tri"])
        (ga,) = torch.autograd.grad(aux, s["alpha"])
        gc, gp = torch.autograd.grad(out, (s["color"], s["pos"]), s["grad"])
        return dict(aux=aux, alpha=ga, color=gc, pos=gp)
    if kind == "view":
        m = MODELS[case["model"]]
        alpha = ds.accumulate_to_level(m["lo"], m["hi"], s["alpha"]).sigmoid()
        feat = ds.accumulate_to_level(m["lo"], m["hi"], s["feat"]).sigmoid()
        pos = _clip(s["verts"], s["mvp"])
        with torch.no_grad():
            rast = ds.rasterize_multires_triangle_alpha((H, W), pos, s["tri"], m["hi"], alpha, stochastic=False)
            mask = rast[..., 3] > 0
            enc = ds.encode_view_dir_sh2(rast, s["inv"])
        x = torch.cat([ds.multires_triangle_color(rast, m["hi"], feat), enc], -1)
        mk = mask.unsqueeze(-1).float()
        color = (mk * s["mlp"](x, mask=mask) + (1 - mk)).contiguous()
        loss = ds.opacity_aux_loss(color.detach(), s["target"], rast, pos.detach(), s["tri"], m["hi"], alpha)
        loss = loss + F.mse_loss(ds.edge_grad(color, rast, pos, s["tri"]), s["target"])
        params = list(s["mlp"].parameters())
        grads = torch.autograd.grad(loss, [s["verts"], s["feat"], s["alpha"]] + params)
        return dict(loss=loss, verts=grads[0], feat=grads[1], alpha=grads[2].squeeze(-1),
                    mlp=torch.cat([x.reshape(-1) for x in grads[3:]]))
    if kind == "adam":
        for o in s["opts"]:
            o.step()
        ps = [s["verts"]] + s["params"]
        st = [o.state[p] for o, group in zip(s["opts"], ([s["verts"]], s["params"])) for p in group]
        return dict(params=ps, first=[x.get("g1", x.get("exp_avg")) for x in st],
                    second=[x.get("g2", x.get("exp_avg_sq")) for x in st])
    if kind == "render":
        if case["graph"]:
            s["graph"].replay()
            return s["frame"].rgba8
        return s["r"].render(s["mvp_host"], H, W)
    counts = visibility.count_visible_triangles((H, W), s["mvp"], s["verts"], s["tri"], case["hi"], s["opacity"])
    valid = (counts > 0).int()
    return (counts,) + tuple(remesh.split_triangle_soup_clip_until((H, W), s["mvp"][0], s["verts"], s["tri"], valid,
                                                                   case["tau"], hard_cap=case["cap"]))


def work(case):
    """Bytes that one pass reads and writes at least once (parameters, gradients, per-pixel inputs and outputs)
    and the operations of its shading MLPs."""
    kind, T = case["kind"], case["tris"]
    if kind in ("levels", "adam"):
        S = scenes.total_feats(case["lo"], case["hi"])
        if kind == "levels":  # forward: source and result; backward: their gradients
            ST = scenes.feats_at_level(case["hi"])
            n = 8 * T * (S + ST) * case["C"]
            return dict(bytes=n, flops=12 * T * ST * case["C"] * (case["hi"] - case["lo"] + 1))
        n = T * S * (case["C"] + 1) + 16 * (case["C"] + 9) + 16 + 272 + 51
        return dict(bytes=28 * n + 68 * 3 * T + 8 * 3 * T, flops=12 * n + 14 * 9 * T)
    P, B = sum(h * w for h, w in _sizes(case)), case["views"]
    if kind in ("step", "view"):
        m = MODELS[case["model"]]
        S = scenes.total_feats(m["lo"], m["hi"])
        k = m["C"] + (9 if m["enc"] == "sh2" else 3)
        mac = k * m["hidden"] + (m["layers"] - 1) * m["hidden"] ** 2 + 3 * m["hidden"]
        target = 3 if case.get("u8") else 12
        # vertices, faces, parameters and their gradients; targets; per view the clip positions
        return dict(bytes=T * (2 * 36 + 12) + 8 * T * S * (m["C"] + 1) + B * 32 * 3 * T + P * target, flops=6 * mac * P)
    if kind == "render":  # vertices and faces, the texture pair once, an RGBA8 frame
        return dict(bytes=T * 48 + 8 * T * scenes.feats_at_level(case["level"]) + 4 * P, flops=2 * (16 * 35) * P)
    ST = scenes.feats_at_level(case["hi"])
    if kind == "raster":
        return dict(bytes=B * T * 48 + 12 * T + 4 * T * ST + 16 * P, flops=60 * P)
    if kind == "features":  # ID buffer both ways, features and gradient, per-pixel result, encoding and adjoint
        return dict(bytes=P * (32 + 8 * case["C"] + 36) + 8 * T * ST * case["C"], flops=12 * case["C"] * P)
    if kind == "hooks":  # ID buffer, colour, target, adjoint in and out; positions and opacities with gradients
        return dict(bytes=P * (16 + 12 + 12 + 12 + 12) + B * 96 * T + 8 * T * ST + 12 * T, flops=100 * P)
    return dict(bytes=B * T * 48 + 12 * T + 4 * T * ST + 8 * T + 84 * T, flops=60 * P)  # resample


# ---------------------------------------------------------------------------
#  The same in 64 bits
# ---------------------------------------------------------------------------

def _lattice(b0, b1, level):
    """Sample indices [...,3] and weights [...,3] of the lattice cell that holds (b0, b1)."""
    res = 1 << level
    x = (b0 * res).floor().long().clamp(0, res - 1)
    y = torch.minimum((b1 * res).floor().long().clamp(min=0), res - 1 - x)
    f0, f1 = b0 * res - x, b1 * res - y
    flip = f0 + f1 > 1
    x2 = x + flip
    y2 = torch.minimum(y + flip, res - x2)
    at = lambda i, j: (i + j) * (i + j + 1) // 2 + j  # noqa: E731
    w0, w1 = torch.where(flip, 1 - f1, f0), torch.where(flip, 1 - f0, f1)
    return torch.stack([at(x + 1, y), at(x, y + 1), at(x2, y2)], -1), torch.stack([w0, w1, 1 - w0 - w1], -1)


def _level_matrix(lo, hi):
    """[S_target, S]: the samples of levels lo..hi evaluated at the vertices of level hi's lattice."""
    R = 1 << hi
    xy = [(s - y, y) for s in range(R + 1) for y in range(s + 1)]
    b = torch.tensor(xy, dtype=torch.float64, device=_dev()) / R
    M = torch.zeros(len(xy), scenes.total_feats(lo, hi), dtype=torch.float64, device=_dev())
    off = 0
    for level in range(lo, hi + 1):
        idx, w = _lattice(b[:, 0], b[:, 1], level)
        M.scatter_add_(1, off + idx, w)
        off += scenes.feats_at_level(level)
    return M


def _lookup(table, t, b0, b1, level):
    """Interpolated [n,C] rows of table [T,S,C]."""
    idx, w = _lattice(b0, b1, level)
    return sum(w[:, k, None] * table[t, idx[:, k]] for k in range(3))


def _cover(P, nx, ny):
    """Barycentrics, depth and w of clip triangles P [n,3,4] at NDC points; covered or not."""
    q = P[..., :2] - torch.stack([nx, ny], -1)[:, None] * P[..., 3:]
    cross = lambda a, b: a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]  # noqa: E731
    A = torch.stack([cross(q[:, 1], q[:, 2]), cross(q[:, 2], q[:, 0]), cross(q[:, 0], q[:, 1])], -1)
    b = A / A.sum(-1, keepdim=True)
    z, w = (b * P[..., 2]).sum(-1), (b * P[..., 3]).sum(-1)
    return b, z, w, (b[:, 0] >= 0) & (b[:, 1] >= 0) & (b[:, 0] + b[:, 1] <= 1)


def _fragments(pos, tri, H, W):
    """Every fragment of one view: pixel, triangle, b0, b1, depth (pos [V,4] in 64 bits)."""
    P = pos[tri.long()]
    ok = (P[..., 3] > 0).all(1)
    ndc = (P[..., :3] / P[..., 3:]).clamp(-1, 1)
    out = ((P[..., :3] < -P[..., 3:]).all(1) | (P[..., :3] > P[..., 3:]).all(1)).any(1)
    lo = ((ndc.amin(1)[:, :2] + 1) / 2 * P.new_tensor([W, H])).floor().long().clamp(min=0)
    hi = ((ndc.amax(1)[:, :2] + 1) / 2 * P.new_tensor([W, H])).floor().long()
    hi = torch.minimum(hi, torch.tensor([W - 1, H - 1], device=P.device))
    n = (hi - lo + 1).clamp(min=0)
    count = torch.where(ok & ~out, n[:, 0] * n[:, 1], torch.zeros_like(n[:, 0]))
    parts, ends = [], count.cumsum(0)
    starts = torch.arange(0, int(ends[-1]) + 1, 8_000_000, device=P.device)
    cuts = torch.unique(torch.cat([torch.searchsorted(ends, starts), ends.new_tensor([len(count)])])).tolist()
    for a, z in zip([0] + cuts[:-1], cuts):
        t = torch.repeat_interleave(torch.arange(a, z, device=P.device), count[a:z])
        if not t.numel():
            continue
        k = torch.arange(t.numel(), device=P.device) - (ends - count)[t] + (ends - count)[a]
        x, y = lo[t, 0] + k % n[t, 0], lo[t, 1] + k // n[t, 0]
        b, cz, cw, hit = _cover(P[t], -1 + (2 * x + 1).double() / W, -1 + (2 * y + 1).double() / H)
        depth = cz / cw
        hit &= (depth >= -1) & (depth <= 1)
        parts.append([v[hit] for v in (y * W + x, t, b[:, 0], b[:, 1], depth)])
    if not parts:
        e = torch.zeros(0, dtype=torch.long, device=P.device)
        return e, e, e.double(), e.double(), e.double()
    return [torch.cat(v) for v in zip(*parts)]


def _uniform(seed, iteration, view, pix, t):
    """Philox-4x32-10 word 0 of (pixel, triangle, view, iteration) under the seed, as [0, 1) in 24 bits."""
    M = 0xFFFFFFFF

    def wide(a, c):  # 32 x 32 -> high and low words, in 64-bit integers
        lo = a * (c & 0xFFFF)
        hi = a * (c >> 16) + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    c = [pix.clone(), t.clone(), torch.full_like(t, view), torch.full_like(t, iteration)]
    k0, k1 = seed & M, (seed >> 32) & M
    for _ in range(10):
        h0, l0 = wide(c[0], 0xD2511F53)
        h1, l1 = wide(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return (c[0] >> 8).double() / 2 ** 24


def _surface(frag, opacity, level, n, draw_u):
    """Per pixel the nearest fragment whose opacity reaches its threshold: index into frag, or -1."""
    pix, t, b0, b1, z = frag
    a = _lookup(opacity.unsqueeze(-1), t, b0, b1, level)[:, 0]
    thr = draw_u(pix, t) if draw_u is not None else 0.5
    keep = ((a >= thr) & (z > -1)).nonzero()[:, 0]
    order = keep[torch.argsort(z[keep], stable=True)]
    order = order[torch.argsort(pix[order], stable=True)]
    first = torch.ones(len(order), dtype=torch.bool, device=pix.device)
    first[1:] = pix[order][1:] != pix[order][:-1]
    win = torch.full((n,), -1, dtype=torch.long, device=pix.device)
    win[pix[order][first]] = order[first]
    return win, a


def _rast(frag, win, H, W):
    r = torch.zeros(H * W, 4, dtype=torch.float64, device=win.device)
    hit = win >= 0
    k = win[hit]
    r[hit] = torch.stack([frag[2][k], frag[3][k], frag[4][k], (frag[1][k] + 1).double()], -1)
    return r.reshape(H, W, 4)


def _aux_grad(frag, a, rast, l1, level, S, T, scale):
    """Opacity gradient: L/alpha for the visible fragment of a pixel, -L/(1-alpha) for those in front of it."""
    pix, t, b0, b1, z = frag
    tp, zp = rast.reshape(-1, 4)[pix, 3].long() - 1, rast.reshape(-1, 4)[pix, 2]
    seen = tp == t
    # the surface itself is given in FP32 in some cases: its own fragment counts as level with it
    keep = (tp < 0) | seen | (z <= zp)
    loss = l1[pix]
    g = torch.where(seen, loss / a.clamp(min=1e-5), -loss / (1 - a).clamp(min=1e-5)) * scale
    g = torch.where(keep, g, torch.zeros_like(g))
    idx, w = _lattice(b0, b1, level)
    out = torch.zeros(T * S, dtype=torch.float64, device=pix.device)
    for k in range(3):
        out.index_add_(0, t * S + idx[:, k], g * w[:, k])
    return out.reshape(T, S)


def _normal(P):
    X = P[..., :3] / P[..., 3:]
    n = torch.linalg.cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0])
    return n / n.norm(dim=1, keepdim=True).clamp(min=1e-300)


def _edge_pos_grad(color, grad, rast, pos, tri):
    """Silhouette, opacity-edge, intersection and interior gradients of one view at the clip positions."""
    H, W, _ = rast.shape
    ids, out = rast[..., 3].long() - 1, torch.zeros_like(pos)
    tri = tri.long()
    for dx, dy in ((1, 0), (-1, 0), (0, -1), (0, 1)):
        y, x = (ids >= 0).nonzero(as_tuple=True)
        inside = (x + dx >= 0) & (x + dx < W) & (y + dy >= 0) & (y + dy < H)
        y, x = y[inside], x[inside]
        adj = (0.5 * (grad[y, x] + grad[y + dy, x + dx]) * (color[y, x] - color[y + dy, x + dx])).sum(-1)
        y, x, adj = y[adj != 0], x[adj != 0], adj[adj != 0]
        i0, i1 = ids[y, x], ids[y + dy, x + dx]
        z0, z1 = rast[y, x, 2], rast[y + dy, x + dx, 2]
        n0 = torch.stack([-1 + (2 * x + 1).double() / W, -1 + (2 * y + 1).double() / H], -1)
        n1 = n0 + n0.new_tensor([2 * dx / W, 2 * dy / H])
        g = torch.stack([adj * dx * W / 2, adj * dy * H / 2, torch.zeros_like(adj)], -1)
        P0, P1 = pos[tri[i0]], pos[tri[i1.clamp(min=0)]]
        _, cz, cw, cover = _cover(P0, n1[:, 0], n1[:, 1])
        same = i1 == i0
        front = (i1 < 0) | (z0 < z1)
        crossing = cover & (i1 >= 0) & (z1 < cz / cw)
        _, ez, ew, ecover = _cover(P1, n0[:, 0], n0[:, 1])
        isect = ~same & crossing & ecover & (z0 < ez / ew)
        mid = same | isect | (~same & cover & ~crossing & front)
        # intersections: the boundary moves along the line where the two planes meet
        a = 0 if dx else 1
        na, nb = _normal(P0), _normal(P1)
        na, nb = F.normalize(na[:, [a, 2]], dim=1, eps=1e-15), F.normalize(nb[:, [a, 2]], dim=1, eps=1e-15)
        den = -nb[:, 1] * na[:, 0] + nb[:, 0] * na[:, 1]
        k = torch.where(den.abs() > 1e-12, -nb[:, 1] / den, torch.zeros_like(den))
        ga = g[:, a]
        gi = torch.zeros_like(g)
        gi[:, a], gi[:, 2] = ga * k * na[:, 0], ga * k * na[:, 1]
        gm = torch.where(isect[:, None], gi, g)
        nm = 0.5 * (n0 + n1)
        b, mz, mw, mcover = _cover(P0, nm[:, 0], nm[:, 1])
        mid = mid & mcover
        u = b / mw[:, None]
        pull = (gm[:, :2] * nm).sum(-1) + torch.where(isect, gm[:, 2] * mz / mw, torch.zeros_like(mz))
        add = torch.cat([u[..., None] * gm[:, None], (-u * pull[:, None])[..., None]], -1)
        add = torch.where(mid[:, None, None], add, torch.zeros_like(add))
        # silhouettes: the triangle edge that the segment between the centres crosses first in (01, 12, 20)
        todo = ~same & ~cover & front
        ndc, d = P0[..., :2] / P0[..., 3:], n1 - n0
        for i, j in ((0, 1), (1, 2), (2, 0)):
            p, e = ndc[:, i], ndc[:, j] - ndc[:, i]
            den = d[:, 0] * e[:, 1] - d[:, 1] * e[:, 0]
            q = p - n0
            t = (q[:, 0] * e[:, 1] - q[:, 1] * e[:, 0]) / den
            s = (q[:, 0] * d[:, 1] - q[:, 1] * d[:, 0]) / den
            eps = 1e-7
            hit = todo & (den.abs() > eps) & (t >= -eps) & (t <= 1 + eps) & (s >= -eps) & (s <= 1 + eps)
            todo = todo & ~hit
            at = n0 + t[:, None] * d
            A, D = P0[:, i], P0[:, j] - P0[:, i]
            av, bv = A[:, :2] - at * A[:, 3:], D[:, :2] - at * D[:, 3:]
            bb = (bv * bv).sum(-1)
            s1 = torch.where(bb != 0, -(av * bv).sum(-1) / bb, torch.full_like(bb, 0.5))
            c = A + s1[:, None] * D
            iw = 1 / c[:, 3]
            pull = (g[:, :2] * c[:, :2]).sum(-1) * iw * iw
            for v, sv in ((i, 1 - s1), (j, s1)):
                w = torch.cat([sv[:, None] * g[:, :2] * iw[:, None], torch.zeros_like(iw)[:, None],
                               (-sv * pull)[:, None]], -1)
                add[:, v] += torch.where(hit[:, None], w, torch.zeros_like(w))
        out.index_add_(0, tri[i0].reshape(-1), add.reshape(-1, 4))
    return out


def _direction(inv, H, W):
    """Unit view directions [H,W,3] from the far plane to the camera through the pixel centres."""
    y, x = torch.meshgrid(torch.arange(H, device=_dev()), torch.arange(W, device=_dev()), indexing="ij")
    n = torch.stack([-1 + (2 * x + 1).double() / W, -1 + (2 * y + 1).double() / H], -1)
    ends = []
    for z in (-1.0, 1.0):
        c = torch.cat([n, torch.full_like(n[..., :1], z), torch.ones_like(n[..., :1])], -1) @ inv.T
        ends.append(c[..., :3] / c[..., 3:])
    return F.normalize(ends[0] - ends[1], dim=-1)


def _sh2(d):
    x, y, z = d.unbind(-1)
    c0, c1 = math.sqrt(1 / math.pi) / 2, math.sqrt(3 / math.pi) / 2
    a, b, c = math.sqrt(15 / math.pi) / 2, math.sqrt(5 / math.pi) / 4, math.sqrt(15 / math.pi) / 4
    return torch.stack([torch.full_like(x, c0), -c1 * y, c1 * z, -c1 * x, a * x * y, -a * y * z,
                        b * (2 * z * z - x * x - y * y), -a * x * z, c * (x * x - y * y)], -1)


def _exact_step(s, m, hw, alpha, feat, mlp, target, draw_u, u8):
    """Loss and gradients of a training step over views of sizes hw."""
    d = lambda t: t.detach().double()  # noqa: E731
    M = _level_matrix(m["lo"], m["hi"])
    alpha, feat = d(alpha).requires_grad_(), d(feat).requires_grad_()
    op, ft = torch.sigmoid(alpha @ M.T), torch.sigmoid(torch.einsum("ks,tsc->tkc", M, feat))
    ws = [d(t).requires_grad_() for t in mlp]
    S, T = op.shape[1], op.shape[0]
    n_all = sum(h * w for h, w in hw) * 3
    loss, g_op, g_verts, at = 0.0, torch.zeros_like(op), torch.zeros_like(d(s["verts"])), 0
    g_ft, g_ws = torch.zeros_like(ft), [torch.zeros_like(w) for w in ws]
    for b, (H, W) in enumerate(hw):
        mvp, inv = d(s["mvp"][b]), d(s["inv"][b])
        pos = F.pad(d(s["verts"]), (0, 1), value=1.0) @ mvp.T
        frag = _fragments(pos, s["tri"], H, W)
        win, a = _surface(frag, op.detach(), m["hi"], H * W, None if draw_u is None else (lambda p, t: draw_u(b, p, t)))
        rast = _rast(frag, win, H, W)
        hit = (win >= 0).nonzero()[:, 0]
        r = rast.reshape(-1, 4)[hit]
        dirs = _direction(inv, H, W).reshape(-1, 3)[hit]
        ftd, wd = ft.detach().requires_grad_(), [w.detach().requires_grad_() for w in ws]
        x = torch.cat([_lookup(ftd, r[:, 3].long() - 1, r[:, 0], r[:, 1], m["hi"]),
                       _sh2(dirs) if m["enc"] == "sh2" else dirs], -1)
        h = x
        for k in range(0, len(wd) - 2, 2):
            h = F.relu(h @ wd[k].T + wd[k + 1])
        y = torch.sigmoid(h @ wd[-2].T + wd[-1])
        shade = (1 - x[:, 3:4]) * x[:, :3] + x[:, 3:4] * y
        color = torch.ones(H * W, 3, dtype=torch.float64, device=_dev())
        color[hit] = shade.detach()
        tgt = target[at:at + H * W].double() / (255.0 if u8 else 1.0)
        at += H * W
        diff = color - tgt
        loss = loss + (diff * diff).sum() / n_all
        grad = 2 * diff / n_all
        gs = torch.autograd.grad(shade, [ftd] + wd, grad[hit])
        g_ft += gs[0]
        for k, v in enumerate(gs[1:]):
            g_ws[k] += v
        g_op += _aux_grad(frag, a, rast, diff.abs().sum(-1), m["hi"], S, T, 1.0 / n_all)
        gp = _edge_pos_grad(color.reshape(H, W, 3), grad.reshape(H, W, 3), rast, pos, s["tri"])
        g_verts += (gp @ mvp)[:, :3]
    ga, gf = torch.autograd.grad([op, ft], [alpha, feat], [g_op, g_ft])
    return dict(loss=loss.reshape(1), verts=g_verts, feat=gf, alpha=ga, mlp=torch.cat([w.reshape(-1) for w in g_ws]))


def exact(case, seed):
    kind = case["kind"]
    # no 64-bit value: frames and counts are whole numbers, and a soup's pieces are bisected by FP32 rules;
    # steps and views of dense full-size batches take too long
    if kind in ("render", "resample"):
        return None
    if kind in ("step", "view") and case["tris"] * case["views"] > 400000:
        return None
    s = prepare(case, seed)
    d = lambda t: t.detach().double()  # noqa: E731
    H, W = case.get("height"), case.get("width")
    if kind == "levels":
        M = _level_matrix(case["lo"], case["hi"])
        return dict(out=torch.einsum("ks,tsc->tkc", M, d(s["feat"])), grad=torch.einsum("ks,tkc->tsc", M, d(s["grad"])))
    if kind == "adam":
        out = dict(params=[], first=[], second=[])
        for i, p in enumerate([s["verts"]] + s["params"]):
            g, lr = d(p.grad), 1e-3 if i == 0 else 5e-3
            m, v = 0.1 * g, 0.001 * (g * g).sum(-1, keepdim=True) if i == 0 else 0.001 * g * g
            out["params"].append(d(p) - lr * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8))
            out["first"].append(m)
            out["second"].append(v)
        return out
    if kind == "features":
        feat = d(s["feat"]).requires_grad_()
        outs, encs = [], []
        for r, inv in zip(d(s["rast"]), d(s["inv"])):
            hit = r[..., 3] > 0
            o = torch.zeros(H, W, case["C"], dtype=torch.float64, device=_dev())
            q = r[hit]
            outs.append(o.index_put((hit,), _lookup(feat, q[:, 3].long() - 1, q[:, 0], q[:, 1], case["hi"])))
            encs.append(_sh2(_direction(inv, H, W)) * hit[..., None])
        out = torch.stack(outs)
        (grad,) = torch.autograd.grad(out, feat, d(s["grad"]))
        return dict(out=out, enc=torch.stack(encs), grad=grad)
    if kind == "raster":
        rs = []
        for p in d(s["pos"]):
            frag = _fragments(p, s["tri"], H, W)
            win, _ = _surface(frag, d(s["opacity"]).squeeze(-1), case["hi"], H * W, None)
            rs.append(_rast(frag, win, H, W))
        return torch.stack(rs)
    if kind == "hooks":
        op = d(s["opacity"])
        ga, gp = torch.zeros_like(op), []
        for p, r, c, t, g in zip(d(s["pos"]), d(s["rast"]), d(s["color"]), d(s["target"]), d(s["grad"])):
            frag = _fragments(p, s["tri"], H, W)
            a = _lookup(op.unsqueeze(-1), frag[1], frag[2], frag[3], case["hi"])[:, 0]
            ga += _aux_grad(frag, a, r, (c - t).abs().sum(-1).reshape(-1), case["hi"], op.shape[1], op.shape[0],
                            1.0 / s["color"].numel())
            gp.append(_edge_pos_grad(c, g, r, p, s["tri"]))
        return dict(aux=torch.zeros(1, dtype=torch.float64), alpha=ga.unsqueeze(-1), color=d(s["grad"]), pos=torch.stack(gp))
    m = MODELS[case["model"]]
    if kind == "view":
        return _exact_step(s, m, [(H, W)], s["alpha"].squeeze(-1), s["feat"], list(s["mlp"].parameters()),
                           s["target"].reshape(-1, 3), None, False)
    return _exact_step(s, m, _sizes(case), s["alpha"], s["feat"], [t for wb in s["mlp"] for t in wb], s["target"],
                       lambda b, p, t: _uniform(seed, 0, b, p, t), case["u8"])
