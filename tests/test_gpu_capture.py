"""A captured run replayed on other images: each replay gives the maps of a direct run on the images that the
views hold at that time, whether the levels are whole numbers, as they were at capture, or not.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
from test_gpu_batch import _load, _maps, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(96, 72), (640, 166)])  # one launch a half-sweep, bands
def test_replay_reads_the_views_images(width, height):
    import torch
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=3, width=width, height=height, n_src=2, seed=23, supersample=1)
    grays = [synth.gray_float(v.image) for v in scene.views]
    images = [grays, [np.ascontiguousarray(255.0 - g) for g in grays],
              [np.ascontiguousarray(0.25 + 0.5 * g) for g in grays]]
    srcs = [j for j, _ in scene.pairs[0]]

    def run(ctx, cams):
        ctx.run_patchmatch(0, srcs, hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[0]), mode=0), seed=5)

    direct = []
    for im in images:
        with hpm_b200.Context(0) as ctx:
            cams = _load(ctx, scene)
            for i, g in enumerate(im):
                ctx.set_view(i, g, cams[i])
            run(ctx, cams)
            direct.append(_maps(ctx, [0], hpm_b200.MAP_DEPTH)[0])
    with hpm_b200.Context(0) as ctx:
        cams = _load(ctx, scene)
        run(ctx, cams)
        ctx.synchronize()
        stream = torch.cuda.ExternalStream(ctx.stream_handle())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            run(ctx, cams)
        for im, want in zip(images, direct):
            for i, g in enumerate(im):
                ctx.set_view(i, g, cams[i])
            ctx.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            for a, b in zip(_maps(ctx, [0], hpm_b200.MAP_DEPTH)[0], want):
                assert _same(a, b)
        del graph
