"""The sequential pass of the consistency scans, which takes over where the rounds have not settled.

With the rounds capped at 0 every view goes through it, with 1 or 2 those that need more; the other views
settle in rounds, before and after.  All results are those of the oracle's sequential loop, bit for bit,
and those without a cap.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from conftest import scene_cams, scene_grays
from test_gpu_stages import noisy_maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds", [0, 1, 2, 256])
@pytest.mark.parametrize("width,height", [(160, 120), (33, 31), (64, 48)])  # 18.75, 0.99 and 3 chunks of 1024
def test_capped_rounds_match_oracle(width, height, rounds):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=5, width=width, height=height, seed=3, n_src=4, supersample=1)
    depths, normals = noisy_maps(scene, 9, noise=0.006)
    depths[1] = np.where(np.random.default_rng(4).random(depths[1].shape) < 0.05, depths[1], 0).astype(np.float32)
    cams = scene_cams(scene)
    srcs = [[j for j, _ in p] for p in scene.pairs]
    srcs[2] = srcs[2] + [srcs[2][0]]  # listed twice: shares its marks
    srcs[3] = []
    with hpm_b200.Context(0) as ctx:
        for i, (g, c) in enumerate(zip(scene_grays(scene), cams)):
            ctx.set_view(i, g, c)
            ctx.set_color(i, scene.views[i].image)
            ctx.set_map(i, hpm_b200.MAP_DEPTH, depths[i])
            ctx.set_map(i, hpm_b200.MAP_NORMAL, normals[i])
        ctx.debug_scan_rounds(rounds)
        used = ctx.confidence_eval(srcs, hpm_b200.MAP_DEPTH)
        conf = [ctx.get_map(i, hpm_b200.MAP_CONF) for i in range(5)]
        pts, count = ctx.fuse(srcs, hpm_b200.MAP_DEPTH)
    # more rounds than allowed: the pass took over in one view at least
    assert used == rounds + 1 if rounds < 2 else used <= rounds + 1
    for i, ref in enumerate(ora.confidence_eval(cams, depths, normals, srcs)):
        np.testing.assert_array_equal(conf[i], ref)
    ref, n_ref = ora.fusion(cams, depths, normals, [v.image for v in scene.views], srcs)
    assert count == n_ref and count > 0
    np.testing.assert_array_equal(pts, ref)


def test_cap_is_checked():
    with hpm_b200.Context(0) as ctx:
        for bad in (-1, 257):
            with pytest.raises(hpm_b200.HPMError):
                ctx.debug_scan_rounds(bad)
