"""Runs before and after a view's byte copies are made.

A run makes the copies once the runs on its reference have work for them, so the same images are sampled as
floats by some runs and as bytes by others.  Every run gives the oracle's maps, whatever ran before it.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
from test_gpu_batch import _same
from test_gpu_edges import _views
from test_gpu_geometric_prior import _inputs, _oracle

pytestmark = pytest.mark.gpu


# iterations of the runs in turn; at 64x48 with two sources a first run of one stays on the float images
@pytest.mark.parametrize("turns", [(0, 1, 0, 1, 3), (3, 0, 1), (0, 0, 0, 2)])
@pytest.mark.parametrize("upload", ["set_view", "prepare_level"])
@pytest.mark.parametrize("batched", [False, True])
def test_runs_in_turn_match_oracle(turns, upload, batched):
    sc, cams, first = _views(3, 64, 48, seed=91)
    inputs = _inputs(sc, cams, 8)
    with hpm_b200.Context(0) as ctx:
        for image in range(2):  # new images start again
            for i, v in enumerate(sc.views):
                if upload == "set_view":
                    ctx.set_view(i, first[i] if image == 0 else np.ascontiguousarray(255 - first[i]), cams[i])
                    ctx.set_canny(i, inputs[i][6])
                else:
                    ctx.set_image(i, np.ascontiguousarray(v.image if image == 0 else 255 - v.image))
                    ctx.prepare_level(i, 64, 48, cams[i])
            levels = [ctx.get_level(i) for i in range(3)]
            grays, canny = [lv[1] for lv in levels], [lv[2] for lv in levels]
            own = [inp[:6] + (c,) for inp, c in zip(inputs, canny)]
            for k, iterations in enumerate(turns):
                ref = k % 2  # each view is a source of the other
                srcs = [j for j in range(3) if j != ref]
                params = hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[ref]))
                params.max_iterations = iterations
                if batched:
                    ctx.run_batch([ref], [srcs], params, [k])
                else:
                    ctx.run_patchmatch(ref, srcs, params, seed=k)
                got = [ctx.get_map(ref, m) for m in (hpm_b200.MAP_DEPTH, hpm_b200.MAP_NORMAL, hpm_b200.MAP_COST)]
                for name, a, b in zip(("depth", "normal", "cost"), got,
                                      _oracle(cams, grays, own, ref, srcs, params, k)):
                    assert _same(a, np.ascontiguousarray(b)), (image, k, name)


@pytest.mark.parametrize("address_mode", [0, 1])
def test_views_through_more_sizes_than_are_kept(address_mode):
    """Level images of six sizes in turn, twice: a view keeps the 8-bit arrays of its last four sizes."""
    sc, cams, _ = _views(3, 96, 72, seed=92)
    sizes = [(96, 72), (48, 36), (64, 48), (33, 25), (80, 60), (41, 52)]
    want = {}
    with hpm_b200.Context(0) as kept:
        kept.set_address_mode(address_mode)
        for i, v in enumerate(sc.views):
            kept.set_image(i, v.image)
        for turn, (w, h) in enumerate(sizes + sizes[::-1] + sizes[:2] * 2):
            for fresh in (True, False):
                if fresh and (w, h) in want:
                    continue
                ctx = hpm_b200.Context(0) if fresh else kept
                if fresh:
                    ctx.set_address_mode(address_mode)
                    for i, v in enumerate(sc.views):
                        ctx.set_image(i, v.image)
                for i, c in enumerate(cams):
                    ctx.prepare_level(i, w, h, c.scaled(w, h, 96, 72))
                params = hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[0]))
                ctx.run_patchmatch(0, [1, 2], params, seed=3)
                maps = [ctx.get_map(0, m) for m in (hpm_b200.MAP_DEPTH, hpm_b200.MAP_NORMAL, hpm_b200.MAP_COST)]
                if fresh:
                    ctx.close()
                    want[(w, h)] = maps
                else:
                    assert all(_same(a, b) for a, b in zip(maps, want[(w, h)])), (turn, w, h)
