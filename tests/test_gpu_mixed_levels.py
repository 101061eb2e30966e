"""Runs in which some images hold whole grey levels and others do not, against the oracle.

An image of whole levels is read as bytes, any other as floats, the reference and each source for itself.
Every fetch from levels that are multiples of 1/2 is a multiple of 1/512 below 256, which a float holds, so
the oracle's filtered samples are the texture unit's and the maps have the same bits.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from test_gpu_batch import _same
from test_gpu_edges import _views
from test_gpu_geometric_prior import _inputs, _load, _oracle

pytestmark = pytest.mark.gpu

GEOM, MAND = hpm_b200.MODE_GEOM, hpm_b200.MODE_GEOM | hpm_b200.MODE_MULTIGEOM | hpm_b200.MODE_MAND


def _halves(g, seed):
    on = (np.random.default_rng(seed).random(g.shape) < 0.3) & (g < 255)
    return np.ascontiguousarray(g + np.float32(0.5) * on)


# one source count of each specialisation
@pytest.mark.parametrize("n_src,size", [(3, (67, 41)), (7, (41, 50)), (11, (96, 72)), (17, (57, 50))])
@pytest.mark.parametrize("mode", [0, GEOM, MAND])
@pytest.mark.parametrize("changed", ["reference", "one source", "all"])
@pytest.mark.parametrize("shifted", [False, True])
def test_run_matches_oracle(mode, n_src, size, changed, shifted):
    sc, cams, grays = _views(n_src + 1, *size, seed=80 + n_src)
    inputs = _inputs(sc, cams, 7)
    which = {"reference": [0], "one source": [2], "all": range(n_src + 1)}[changed]
    grays = [_halves(g, i) if i in which else g for i, g in enumerate(grays)]
    srcs = list(range(1, n_src + 1))
    params = hpm_b200.Params.make(n_src + 1, *hpm_b200.widened_range(cams[0]), mode=mode)
    with hpm_b200.Context(0) as ctx:
        if shifted:
            ctx.set_ncc_mode(hpm_b200.NCC_SHIFTED)
        _load(ctx, cams, grays, inputs, hpm_b200.MAP_DEPTH_GEOM if mode == MAND else hpm_b200.MAP_DEPTH)
        ctx.run_patchmatch(0, srcs, params, seed=9)
        kind = hpm_b200.MAP_DEPTH_GEOM if mode & GEOM else hpm_b200.MAP_DEPTH
        got = [ctx.get_map(0, k) for k in (kind, hpm_b200.MAP_NORMAL, hpm_b200.MAP_COST)]
    ora.set_ncc_shift(shifted)
    try:
        want = _oracle(cams, grays, inputs, 0, srcs, params, 9)
    finally:
        ora.set_ncc_shift(False)
    for name, a, b in zip(("depth", "normal", "cost"), got, want):
        assert np.isfinite(a).any() and _same(a, np.ascontiguousarray(b)), name
