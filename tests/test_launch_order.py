"""Kernels that may be set up while their predecessor in the stream still runs follow a kernel (or a memset or copy) of
the same library call: never an event wait, after which there is more than one thing to wait for, and never whatever
the caller put on the stream."""

import pytest

from fake_runtime import run

# name -> calls; each prints its recorded operations
CALLS = {
    "step": "train_step()",
    "step_without_records": "train_step(frag_records=0.0)",
    "step_without_tables": "train_step(hi=4, C_=8)",
    "step_wide": "train_step(hi=3, C_=16, hidden=64, layers=2, precision=0, frag_records=0.0)",
    "step_few_triangles": "train_step(T=1, B=1, H=8, W=8, frag_records=0.0)",
    "step_many_tiles": "train_step(B=8, H=800, W=800)",
    "step_one_stream": "(lib.ds_train_step_set_events((C.c_void_p * 8)(*range(1, 9)), 8), train_step())[1]",
    "step_one_stream_without_records":
        "(lib.ds_train_step_set_events((C.c_void_p * 8)(*range(1, 9)), 8), train_step(frag_records=0.0))[1]",
    "bin": "tiles('ds_tiles_bin_report', 'p', 900, 'p', 300, 'p', 'p', *ws, 'p', stream())",
    "rasterize": "tiles('ds_tiles_rasterize', 'p', 900, 'p', 300, 'p', 2, 15, 'p', 0, 0.5, None, 'p', 'p', *ws, stream())",
    "opacity_aux": "tiles('ds_tiles_opacity_aux', 'p', 900, 'p', 300, 'p', 2, 15, 'p', 3, 'p', 'p', 'p', 1.0, 'p', 'p',"
                   " *ws, stream())",
    "render_deferred": "call('ds_render_deferred', 2, 'p', i64(9216), 'p', 2, 'p', 'p', i64(4500), 'p', 'p', 0.0, 0.0,"
                       " 0.0, 'p', 'p', stream())",
    "render_frame": "call('ds_render_frame', 2, 'p', NT, i64(9216), 900, 'p', 300, 'p', 'p', 'p', 2, 'p', 'p', i64(4500),"
                    " 'p', 'p', 0.0, 0.0, 0.0, 'p', 'p', 'p', 'p', C.c_size_t(lib.ds_render_workspace_size(2, 900, 300,"
                    " NT, i64(9600))), i64(9600), 'p', stream())",
    "split_count": "call('ds_split_soup_count', 0, None, 1.0, 0.1, -1, 900, 'p', 300, 'p', None, 'p', C.byref(i64(0)),"
                   " 'p', C.c_size_t(lib.ds_split_soup_workspace_size(300)), 'p', stream())",
    "levels_backward": "call('ds_accumulate_to_level_backward_set', 100, 0, 2, 2, 24, 15, 7, 'p', 'p', stream())",
    "triangle_rects": "call('ds_compute_triangle_rects', 96, 48, 2, 900, 'p', 300, 'p', 'p', 'p', C.byref(C.c_int(0)),"
                      " 'p', C.c_size_t(1 << 20), stream())",
}
SETUP = """
NT = 2 * 6 * 3  # two views of 96x48
ws = (C.c_size_t(lib.ds_tiles_workspace_size(2, 300, NT, i64(9600))), i64(9600))
def tiles(name, views, *rest): return call(name, 2, views, NT, *rest)
"""


@pytest.mark.parametrize("name", CALLS)
def test_chained_launches_follow_a_kernel_of_the_call(tmp_path, name):
    body = SETUP + f"for x in {CALLS[name]}: print(*x)\n"
    before, chained, launches = {}, 0, 0
    for what, stream, *rest in (line.split() for line in run(tmp_path, body).splitlines()):
        if what in ("limit", "record"):
            continue
        if what == "launch":
            launches += 1
            if rest[0] == "1":
                chained += 1
                assert before.get(stream) not in (None, "wait"), rest[2]
        before[stream] = what
    assert launches > 0 and (chained > 0 or name in ("rasterize", "opacity_aux", "render_deferred"))


@pytest.mark.gpu
def test_captured_step_without_records_equals_the_eager_one():
    """The opacity pass starts on the step's second stream there, after an event wait: a captured step, replayed, and
    eager steps give the same gradients (up to the order of the atomics)."""
    import numpy as np
    import torch

    from diffsoup_b200 import scenes
    from diffsoup_b200.step import TrainStep

    sc = scenes.make_scene(2, seed=21, num_tris=2500, num_views=2, resolution=(120, 136))
    mlp = scenes.mlp_weights(sc.mlp_input_dim, 3, sc.hidden_dim, sc.n_layers, seed=21)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, a.dtype)).cuda()  # noqa: E731
    flat = np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in mlp]).astype(np.float32)
    args = (t(sc.verts), t(sc.tri), t(sc.mvps()), t(sc.inv_mvps()), t(sc.feat_src), t(sc.alpha_src[..., 0]), t(flat),
            t(np.concatenate([x.reshape(-1, 3) for x in sc.targets])))
    step = TrainStep(sc.T, sc.verts.shape[0], [(v.height, v.width) for v in sc.views], sc.feat_dim, sc.min_level,
                     sc.max_level, sc.hidden_dim, sc.n_layers, stochastic=True, seed=5, frag_records=0.0)
    step.fit_capacity(*args)

    def grads(run):
        step.rng[1] = 3
        run()
        torch.cuda.synchronize()
        return [g.clone() for g in (step.loss, step.grad_verts, step.grad_feat_src, step.grad_alpha_src, step.grad_mlp)]

    want = grads(lambda: step.run(*args))
    graph = step.capture(*args)
    for _ in range(4):
        for a, b in zip(grads(graph.replay), want):
            assert float((a - b).norm()) <= 2e-6 * float(b.norm())
