"""The gradient kernels over source counts: a warp holds 32 / S pixels with one lane per view.

Costs and gradients against the FP64 oracle within the tolerances of tests/test_gpu_grad.py; the
refinement's sums over a pixel's lanes (zero steps write the starting RMS cost) against the costs of
hpm_eval_cost_grad summed in numpy.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from conftest import scene_cams, scene_grays
from test_gpu_grad import _jittered

pytestmark = pytest.mark.gpu


# 32 / S pixels a warp: 32, 16, 10 with 2 lanes over, 2, 2 with none over, 1, 1 with one lane over
@pytest.mark.parametrize("n_src", [1, 2, 3, 11, 16, 17, 31])
def test_lanes_of_every_source_count(n_src):
    from hpm_b200 import synth
    w, h = 67, 51
    scene = synth.make_scene(n_views=n_src + 1, width=w, height=h, seed=12, n_src=n_src, supersample=1)
    cams, grays = scene_cams(scene), scene_grays(scene)
    v0 = scene.views[0]
    srcs = [j for j, _ in scene.pairs[0]]
    params = hpm_b200.Params.make(n_src + 1, *hpm_b200.widened_range(cams[0]))
    rng = np.random.default_rng(2)
    ys, xs = np.nonzero(v0.depth > 0)
    pick = rng.choice(len(xs), 101, replace=False)
    xs, ys = xs[pick], ys[pick]
    th = _jittered(v0, xs, ys, rng, dj=0.003, nj=0.02).astype(np.float32)
    with hpm_b200.Context(0) as ctx:
        for i, (g, c) in enumerate(zip(grays, cams)):
            ctx.set_view(i, g, c)
        px = np.stack([xs, ys], 1).astype(np.int32)
        cost, grad = ctx.eval_cost_grad(0, srcs, params, px, th)
        alone, none = ctx.eval_cost_grad(0, srcs, params, px, th, with_grad=False)
        ctx.set_map(0, hpm_b200.MAP_DEPTH_GEOM, v0.depth)
        ctx.set_map(0, hpm_b200.MAP_NORMAL, v0.normal)
        ctx.set_map(0, hpm_b200.MAP_COST, np.full((h, w), -1, np.float32))
        ctx.gn_refine(0, srcs, params, hpm_b200.MAP_DEPTH_GEOM, 0)
        rms = ctx.get_map(0, hpm_b200.MAP_COST)
        gx, gy = [a.ravel() for a in np.meshgrid(np.arange(w), np.arange(h))]
        n = v0.normal[gy, gx].astype(np.float64) @ v0.R.astype(np.float64).T
        n[n[:, 2] > 0] *= -1
        n /= np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-9)
        full = np.concatenate([v0.depth[gy, gx][:, None], n[:, :2]], 1).astype(np.float32)
        all_costs, _ = ctx.eval_cost_grad(0, srcs, params, np.stack([gx, gy], 1).astype(np.int32), full, with_grad=False)
    np.testing.assert_array_equal(alone, cost)
    assert none is None
    ok = total = 0
    err = []
    for k in range(len(xs)):
        for j, s in enumerate(srcs):
            c64, g64 = ora.cost_grad64(grays[0], cams[0], grays[s], cams[s], params, int(xs[k]), int(ys[k]),
                                       th[k].astype(np.float64))
            err.append(abs(c64 - cost[k, j]))
            if 0.0 < c64 < 2.0:
                total += 3
                ok += int((np.abs(grad[k, j] - g64) <= 2e-3 * np.abs(g64) + 2e-4).sum())
    assert np.quantile(err, 0.99) < 2e-4
    assert ok >= 0.99 * total
    # the refinement's starting cost: pixels with at least two costs in (0, 2), others left alone
    use = (all_costs > 0) & (all_costs < 2)
    count = use.sum(1)
    want = np.sqrt((np.where(use, all_costs, 0).astype(np.float64) ** 2).sum(1) / np.maximum(count, 1)).reshape(h, w)
    seen = (count.reshape(h, w) >= 2) & (v0.depth > 0)
    assert ((rms >= 0) == seen).mean() > 0.999
    both = seen & (rms >= 0)
    # the map's normal is normalised in float here, in double above: costs differ by their rounding
    assert not both.any() or np.quantile(np.abs(rms[both] - want[both]), 0.99) < 2e-4
