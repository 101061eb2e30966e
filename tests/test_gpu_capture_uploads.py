"""Uploads captured in a CUDA graph: a direct run after a replay sees the images that the replay brought.

The host calls that a replay repeats do not run again, so nothing that the context knows of a view's image
(whether its levels are whole numbers, which image its byte copies hold) may outlive a replay.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
from test_gpu_batch import _load, _maps, _same

pytestmark = pytest.mark.gpu


# "replayed": the direct runs follow replays alone; "direct": a direct upload and run come before the replay
@pytest.mark.parametrize("order", ["replayed", "direct"])
@pytest.mark.parametrize("batched", [False, True])
def test_direct_run_after_replayed_upload(order, batched):
    import torch
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=3, width=96, height=72, n_src=2, seed=23, supersample=1)
    first = [synth.gray_float(v.image) for v in scene.views]
    images = [first, [np.ascontiguousarray(255.0 - g) for g in first],
              [np.ascontiguousarray(0.25 + 0.5 * g) for g in first]]
    srcs = [j for j, _ in scene.pairs[0]]

    def run(ctx, cams):
        params = hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[0]), mode=0)
        if batched:
            ctx.run_batch([0], [srcs], params, [5])
        else:
            ctx.run_patchmatch(0, srcs, params, seed=5)
        return _maps(ctx, [0], hpm_b200.MAP_DEPTH)[0]

    want = []
    for im in images:
        with hpm_b200.Context(0) as ctx:
            cams = _load(ctx, scene)
            for i, g in enumerate(im):
                ctx.set_view(i, g, cams[i])
            want.append(run(ctx, cams))
    buffers = [torch.from_numpy(g.copy()).pin_memory() for g in first]
    with hpm_b200.Context(0) as ctx:
        cams = _load(ctx, scene)
        run(ctx, cams)
        stream = torch.cuda.ExternalStream(ctx.stream_handle())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            for i, b in enumerate(buffers):
                ctx.set_view(i, b.numpy(), cams[i])
        for k, im in enumerate(images):
            if order == "direct":
                for i, g in enumerate(images[0]):
                    ctx.set_view(i, g, cams[i])
                assert all(_same(a, b) for a, b in zip(run(ctx, cams), want[0])), k
            for b, g in zip(buffers, im):
                b.copy_(torch.from_numpy(g))
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            assert all(_same(a, b) for a, b in zip(run(ctx, cams), want[k])), k
        del graph
