"""Combinations of modes that a run refuses, with the context usable afterwards.

The hierarchy mode starts from the coarser level's maps and the geometric mode from its own, so a run in
both has no input for one of them.
"""
from __future__ import annotations

import pytest

import hpm_b200
from test_gpu_batch import _load, _maps, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, hpm_b200.MODE_MULTIGEOM, hpm_b200.MODE_MULTIGEOM | hpm_b200.MODE_MAND])
@pytest.mark.parametrize("batched", [False, True])
def test_hierarchy_with_geometric_is_refused(extra, batched):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=3, width=64, height=48, n_src=2, seed=5, supersample=1)

    def params(mode):
        return hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[0]), mode=mode)

    with hpm_b200.Context(0) as ctx:
        cams = _load(ctx, scene)
        mode = hpm_b200.MODE_HIERARCHY | hpm_b200.MODE_GEOM | extra
        with pytest.raises(hpm_b200.HPMError, match="exclude"):
            if batched:
                ctx.run_batch([0, 1], [[1, 2], [0, 2]], params(mode), [1, 2])
            else:
                ctx.run_patchmatch(0, [1, 2], params(mode), seed=1)
        ctx.run_patchmatch(0, [1, 2], params(hpm_b200.MODE_GEOM), seed=1)
        after = _maps(ctx, [0], hpm_b200.MAP_DEPTH_GEOM)[0]
    with hpm_b200.Context(0) as ctx:
        cams = _load(ctx, scene)
        ctx.run_patchmatch(0, [1, 2], params(hpm_b200.MODE_GEOM), seed=1)
        assert all(_same(a, b) for a, b in zip(after, _maps(ctx, [0], hpm_b200.MAP_DEPTH_GEOM)[0]))
