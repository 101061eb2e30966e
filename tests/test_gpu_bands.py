"""Half-sweeps on several streams.

In bands of rows, as a single run above one wave of blocks takes them,
against the whole-image launches of the batching form on the same views: the maps are equal bit for bit.
The heights give bands of 16 row pairs and more with each remainder of the four-row-pair blocks.

In two groups of a batch's runs, with the large views first, last and alone: the maps of single runs.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
from test_gpu_batch import _load, _maps, _same

pytestmark = pytest.mark.gpu


# 32-pixel columns x four-pair rows of blocks: 444 places on 148 SMs; one band, two, three, four bands
@pytest.mark.parametrize("width,height", [(2250, 47), (1700, 70), (1200, 103), (640, 166), (417, 301)])
@pytest.mark.parametrize("mode", [0, hpm_b200.MODE_GEOM, hpm_b200.MODE_GEOM | hpm_b200.MODE_MAND,
                                  hpm_b200.MODE_PRIOR])
def test_bands_equal_whole_launches(width, height, mode):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=3, width=width, height=height, n_src=2, seed=21, supersample=1)
    srcs = [[j for j, _ in p] for p in scene.pairs]
    refs = [0, 1]
    kind = hpm_b200.MAP_DEPTH_GEOM if mode & hpm_b200.MODE_GEOM else hpm_b200.MAP_DEPTH
    out = []
    for batched in (False, True):
        with hpm_b200.Context(0) as ctx:
            cams = _load(ctx, scene)
            if mode == hpm_b200.MODE_PRIOR:
                for r in refs:
                    ctx.build_prior(r, 0)
            params = [hpm_b200.Params.make(len(srcs[r]) + 1, *hpm_b200.widened_range(cams[r]), mode=mode)
                      for r in refs]
            if batched:
                ctx.run_batch(refs, [srcs[r] for r in refs], params, [31, 32])
            else:
                for k, r in enumerate(refs):
                    ctx.run_patchmatch(r, srcs[r], params[k], seed=31 + k)
            out.append(_maps(ctx, refs, kind))
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.isfinite(x).any() and _same(x, y)


@pytest.mark.parametrize("heights", [(40, 40), (200, 8, 8), (8, 8, 200), (24, 40, 24, 56, 8, 16)])
def test_groups_equal_single_runs(heights):
    from hpm_b200 import synth
    n = len(heights)
    scene = synth.make_scene(n_views=n, width=96, height=72, n_src=1, seed=22, supersample=1,
                             sizes=[(96, h) for h in heights])
    srcs = [[j for j, _ in p] for p in scene.pairs]
    out = []
    for batched in (False, True):
        with hpm_b200.Context(0) as ctx:
            ctx.set_batch_options(0)
            cams = _load(ctx, scene)
            params = [hpm_b200.Params.make(len(srcs[r]) + 1, *hpm_b200.widened_range(cams[r]), mode=0)
                      for r in range(n)]
            if batched:
                ctx.run_batch(list(range(n)), srcs, params, list(range(40, 40 + n)))
            else:
                for r in range(n):
                    ctx.run_patchmatch(r, srcs[r], params[r], seed=40 + r)
            out.append(_maps(ctx, range(n), hpm_b200.MAP_DEPTH))
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert _same(x, y)


def test_graph_replay_after_a_larger_batch():
    """A batch shape replayed after a batch that needed larger tables."""
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=5, width=96, height=72, n_src=2, seed=24, supersample=1)
    srcs = [[j for j, _ in p] for p in scene.pairs]
    with hpm_b200.Context(0) as ctx:
        ctx.set_batch_options(hpm_b200.BATCH_GRAPH)
        cams = _load(ctx, scene)

        def run(n):
            params = [hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[r]), mode=0) for r in range(n)]
            ctx.run_batch(list(range(n)), srcs[:n], params, list(range(60, 60 + n)))
            return _maps(ctx, range(n), hpm_b200.MAP_DEPTH)

        first = run(2)
        run(2)
        run(5)
        for a, b in zip(first, run(2)):
            for x, y in zip(a, b):
                assert _same(x, y)
