"""hpm_eval_costs on both sides of its launch rule: a thread per pixel and view while those are resident
together, a thread per pixel past that.  The pixels of one large call are costed again in small calls, and
some of them by the oracle; every cost has the same bits."""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from conftest import scene_cams, scene_grays

pytestmark = pytest.mark.gpu


# 3 blocks of 128 threads on each of 148 SMs: 147 blocks of pixels x 3 views fit, 148 do not
@pytest.mark.parametrize("n_src,n", [(1, 60001), (3, 147 * 128), (3, 147 * 128 + 1), (10, 12345)])
@pytest.mark.parametrize("levels", ["whole", "halves"])
def test_large_calls_equal_small_ones(n_src, n, levels):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=n_src + 1, width=97, height=61, seed=19, n_src=n_src, supersample=1)
    cams = scene_cams(scene)
    grays = [g if levels == "whole" else np.ascontiguousarray(0.25 + 0.5 * g) for g in scene_grays(scene)]
    rng = np.random.default_rng(n)
    px = np.stack([rng.integers(0, 97, n), rng.integers(0, 61, n)], 1).astype(np.int32)
    normal = rng.normal(0, 0.3, (n, 3)) + [0, 0, -1]
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    K = np.asarray(scene.views[0].K, np.float64)
    ray = np.concatenate([px, np.ones((n, 1))], 1) @ np.linalg.inv(K).T
    depth = rng.uniform(scene.views[0].depth_min, scene.views[0].depth_max, n)
    planes = np.concatenate([normal, -(normal * ray).sum(1, keepdims=True) * depth[:, None]], 1).astype(np.float32)
    params = hpm_b200.Params.make(n_src + 1, *hpm_b200.widened_range(cams[0]))
    srcs = [j for j, _ in scene.pairs[0]]
    with hpm_b200.Context(0) as ctx:
        for i, (g, c) in enumerate(zip(grays, cams)):
            ctx.set_view(i, g, c)
        whole = ctx.eval_costs(0, srcs, params, px, planes)
        parts = [ctx.eval_costs(0, srcs, params, px[k:k + 2500], planes[k:k + 2500]) for k in range(0, n, 2500)]
    assert (whole < 2).mean() > 0.2
    np.testing.assert_array_equal(whole, np.concatenate(parts))
    if levels == "whole":  # a fetch of whole levels has the same bits in the oracle
        some = rng.choice(n, 500, replace=False)
        want = ora.eval_costs([grays[0]] + [grays[j] for j in srcs], [cams[0]] + [cams[j] for j in srcs], params,
                              px[some], planes[some])
        np.testing.assert_array_equal(whole[some], want)
