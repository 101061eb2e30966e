"""Consistency scans where a source's counted positions lie far apart.

The scans look up the next counted and the last accepted pixel over 32-pixel words, the rest of a
1024-pixel chunk and whole chunks; these maps put the gaps at and around those steps.  All results are
those of the oracle's sequential loop, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from conftest import scene_cams, scene_grays
from test_gpu_stages import noisy_maps

pytestmark = pytest.mark.gpu


# kept pixels of the first view: isolated ones near word and chunk edges, bands of rows, one in many, none
def _keep(kind, n, rng):
    keep = np.zeros(n, bool)
    if kind == "edges":
        for c in range(0, n, 1024):
            keep[[k for k in (c, c + 1, c + 31, c + 32, c + 1023) if k < n]] = True
        keep[3 * 1024:7 * 1024] = False
    elif kind == "bands":
        keep[:3000] = True
        keep[n - 2500:] = True
        keep[9000:9003] = True
    elif kind == "sparse":
        keep[rng.random(n) < 0.004] = True
    return keep


@pytest.mark.parametrize("noise", [0.002, 0.006])
@pytest.mark.parametrize("width,height", [(160, 120), (96, 64), (33, 31)])
@pytest.mark.parametrize("kind", ["edges", "bands", "sparse", "none"])
def test_scans_over_gaps_match_oracle(kind, width, height, noise):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=4, width=width, height=height, seed=3, n_src=3, supersample=1)
    depths, normals = noisy_maps(scene, 9, noise=noise)
    rng = np.random.default_rng(4)
    n = width * height
    for v in (0, 1):
        if n > 9003 or kind in ("sparse", "none", "edges"):
            depths[v] = np.where(_keep(kind, n, rng).reshape(height, width), depths[v], 0).astype(np.float32)
    cams = scene_cams(scene)
    # a source listed twice shares its marks
    srcs = [[j for j, _ in p] for p in scene.pairs]
    srcs[2] = srcs[2] + [srcs[2][0]]
    with hpm_b200.Context(0) as ctx:
        for i, (g, c) in enumerate(zip(scene_grays(scene), cams)):
            ctx.set_view(i, g, c)
            ctx.set_color(i, scene.views[i].image)
            ctx.set_map(i, hpm_b200.MAP_DEPTH, depths[i])
            ctx.set_map(i, hpm_b200.MAP_NORMAL, normals[i])
        ctx.confidence_eval(srcs, hpm_b200.MAP_DEPTH)
        conf = [ctx.get_map(i, hpm_b200.MAP_CONF) for i in range(4)]
        pts, count = ctx.fuse(srcs, hpm_b200.MAP_DEPTH)
    for i, ref in enumerate(ora.confidence_eval(cams, depths, normals, srcs)):
        np.testing.assert_array_equal(conf[i], ref)
    ref, n_ref = ora.fusion(cams, depths, normals, [v.image for v in scene.views], srcs)
    assert count == n_ref
    np.testing.assert_array_equal(pts, ref)
