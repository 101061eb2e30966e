"""Runs in the geometric and the prior mode at once, against the oracle.

The two are set independently (HPM::SetGeomConsistencyParams and SetPlanarPriorParams, HPM.cpp:565-587): no
schedule combines them, but a caller may.  Half-sweeps of prior runs take their pixels from work lists, and
those of a geometric run need the source views' geometry.
"""
from __future__ import annotations

import cv2
import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from test_gpu_batch import _same
from test_gpu_edges import _views

pytestmark = pytest.mark.gpu

GEOM, PRIOR, MULTI = hpm_b200.MODE_GEOM, hpm_b200.MODE_PRIOR, hpm_b200.MODE_MULTIGEOM


def _inputs(sc, cams, seed):
    """Per view: depth, world normal, cost, confidence, prior planes (camera frame) and their mask."""
    out = []
    for i, (v, c) in enumerate(zip(sc.views, cams)):
        rng = np.random.default_rng(seed + i)
        h, w = v.depth.shape
        gt = v.depth > 0
        depth = np.where(gt, v.depth * (1 + 0.004 * rng.standard_normal((h, w))), v.depth_max).astype(np.float32)
        normal = v.normal.astype(np.float32).copy()
        normal[np.linalg.norm(normal, axis=-1) < 0.5] = (0.0, 0.0, -1.0)
        cost = rng.uniform(0.0, 0.6, (h, w)).astype(np.float32)
        conf = rng.uniform(0.0, 0.6, (h, w)).astype(np.float32)
        n_cam = normal.astype(np.float64) @ np.asarray(v.R, np.float64).T
        ys, xs = np.mgrid[0:h, 0:w]
        ray = np.stack([xs, ys, np.ones_like(xs)], -1) @ np.linalg.inv(np.asarray(v.K, np.float64)).T
        offset = -(n_cam * ray).sum(-1) * depth
        prior = np.concatenate([n_cam, offset[..., None]], -1).astype(np.float32)
        mask = ((rng.random((h, w)) < 0.7) & gt).astype(np.uint8)
        out.append((depth, normal, cost, conf, prior, mask, cv2.Canny(v.image, 50, 150)))
    return out


def _load(ctx, cams, grays, inputs, kind):
    for i, (g, c, (depth, normal, cost, conf, prior, mask, canny)) in enumerate(zip(grays, cams, inputs)):
        ctx.set_view(i, g, c)
        ctx.set_canny(i, canny)
        ctx.set_map(i, kind, depth)
        ctx.set_map(i, hpm_b200.MAP_NORMAL, normal)
        ctx.set_map(i, hpm_b200.MAP_COST, cost)
        ctx.set_map(i, hpm_b200.MAP_CONF, conf)
        ctx.set_prior(i, prior, mask)


def _maps(ctx, i):
    return [ctx.get_map(i, k) for k in (hpm_b200.MAP_DEPTH_GEOM, hpm_b200.MAP_NORMAL, hpm_b200.MAP_COST)]


def _oracle(cams, grays, inputs, ref, srcs, params, seed):
    depth, normal, cost, conf, prior, mask, canny = inputs[ref]
    h, w = depth.shape
    st = ora.RunState(w, h)
    st.planes[..., :3] = normal
    st.planes[..., 3] = depth
    st.costs[:] = cost
    st.confidences[:] = conf
    st.prior_planes[:] = prior
    st.plane_masks[:] = mask
    st.canny[:] = canny
    ora.run_patchmatch([grays[ref]] + [grays[j] for j in srcs], [None] + [inputs[j][0] for j in srcs],
                       [cams[ref]] + [cams[j] for j in srcs], params, st, seed, ref)
    return [st.planes[..., 3], st.planes[..., :3], st.costs]


# source counts of two specialisations; sizes with a partial block across and down
@pytest.mark.parametrize("n_src,size", [(3, (67, 41)), (11, (40, 33))])
@pytest.mark.parametrize("mode", [GEOM | PRIOR, GEOM | MULTI | PRIOR])
@pytest.mark.parametrize("batched", [False, True])
def test_run_matches_oracle(mode, n_src, size, batched):
    sc, cams, grays = _views(n_src + 1, *size, seed=60 + n_src)
    inputs = _inputs(sc, cams, 5)
    kind = hpm_b200.MAP_DEPTH_GEOM if mode & MULTI else hpm_b200.MAP_DEPTH
    refs = [0] if mode & MULTI else [0, 1]  # a multi-geometry run writes the map that the next one reads
    srcs = [[j for j in range(n_src + 1) if j != r] for r in refs]
    params = [hpm_b200.Params.make(n_src + 1, *hpm_b200.widened_range(cams[r]), mode=mode) for r in refs]
    with hpm_b200.Context(0) as ctx:
        ctx.set_batch_options(0)
        _load(ctx, cams, grays, inputs, kind)
        if batched:
            ctx.run_batch(refs, srcs, params, [70 + r for r in refs])
        else:
            for r in refs:
                ctx.run_patchmatch(r, srcs[r], params[r], seed=70 + r)
        got = [_maps(ctx, r) for r in refs]
    for r in refs:
        want = _oracle(cams, grays, inputs, r, srcs[r], params[r], 70 + r)
        for name, a, b in zip(("depth", "normal", "cost"), got[r], want):
            assert _same(a, np.ascontiguousarray(b)), (r, name)


@pytest.mark.parametrize("tuned", [False, True])
def test_bands_equal_batches(tuned):
    """Four bands of rows against one launch a stage, and the shapes that the batch tuner tries."""
    sc, cams, grays = _views(3, 640, 166, seed=66)
    inputs = _inputs(sc, cams, 6)
    out = []
    for batched in (False, True):
        with hpm_b200.Context(0) as ctx:
            if not tuned:
                ctx.set_batch_options(0)
            _load(ctx, cams, grays, inputs, hpm_b200.MAP_DEPTH)
            params = [hpm_b200.Params.make(3, *hpm_b200.widened_range(cams[r]), mode=GEOM | PRIOR) for r in (0, 1)]
            srcs = [[1, 2], [0, 2]]
            if batched:
                ctx.run_batch([0, 1], srcs, params, [80, 81])
            else:
                for r in (0, 1):
                    ctx.run_patchmatch(r, srcs[r], params[r], seed=80 + r)
            out.append(_maps(ctx, 0) + _maps(ctx, 1))
    for a, b in zip(*out):
        assert np.isfinite(a).any() and _same(a, b)
