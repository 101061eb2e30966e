"""Consistency scans over maps that hold two bands of pixels and a few between them, at sizes whose last
chunk of 1024 pixels is full, partial, or the only one.  All results are the oracle's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from conftest import scene_cams, scene_grays
from test_gpu_stages import noisy_maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noise", [0.002, 0.006])
@pytest.mark.parametrize("width,height", [(160, 120), (96, 64), (33, 31), (113, 91)])
def test_scans_over_bands_match_oracle(width, height, noise):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=4, width=width, height=height, seed=3, n_src=3, supersample=1)
    depths, normals = noisy_maps(scene, 9, noise=noise)
    n = width * height
    keep = np.zeros(n, bool)
    keep[:n // 6] = True
    keep[n - n // 7:] = True
    keep[n // 2:n // 2 + 3] = True
    for v in (0, 1):
        depths[v] = np.where(keep.reshape(height, width), depths[v], 0).astype(np.float32)
    cams = scene_cams(scene)
    srcs = [[j for j, _ in p] for p in scene.pairs]
    srcs[2] = srcs[2] + [srcs[2][0]]  # listed twice: shares its marks
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
