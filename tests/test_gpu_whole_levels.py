"""Images of whole grey levels: the byte textures and weight tables the half-sweeps use for them.

A linearly filtered fetch of whole levels is a whole number N of 1/256 levels (8-bit filter weights),
and the same fetch from 8-bit texels is N / 65280 rounded to a multiple of 1/65535, so rounding it times
65280 gives N.  The runs below take every combination of byte and float reference and sources and are
compared bit for bit, or with the oracle.
"""
from __future__ import annotations

import numpy as np
import pytest

import hpm_b200
import hpm_oracle as ora
from conftest import scene_cams, scene_grays


@pytest.mark.parametrize("tie", ["up", "down"])
def test_every_filtered_value_is_recovered(tie):
    """All 65281 values of N, through the float of the unit's 16-bit result and one fused multiply-add."""
    n = np.arange(255 * 256 + 1, dtype=np.int64)
    m = (n * 257 + (128 if tie == "up" else 127)) // 256  # N / 65280 in steps of 1/65535, rounded
    u = (m / 65535.0).astype(np.float32)
    back = (u.astype(np.float64) * 65280.0 + 12582912.0).astype(np.float32) - np.float32(12582912.0)
    np.testing.assert_array_equal(back.astype(np.int64), n)


@pytest.mark.gpu
@pytest.mark.parametrize("address_mode", [0, 1])
@pytest.mark.parametrize("pattern", ["noise", "extremes", "ramp"])
def test_byte_fetch_equals_float_fetch(pattern, address_mode):
    rng = np.random.default_rng(17)
    h, w = 61, 83
    img = {"noise": lambda: rng.integers(0, 256, (h, w)), "extremes": lambda: 255 * rng.integers(0, 2, (h, w)),
           "ramp": lambda: (np.arange(h)[:, None] * 3 + np.arange(w)[None, :]) % 256}[pattern]().astype(np.float32)
    cam = hpm_b200.Camera.make(np.eye(3), np.eye(3), np.zeros(3), w, h, 1, 2)
    xy = np.stack([rng.uniform(-4, w + 4, 200000), rng.uniform(-4, h + 4, 200000)], 1).astype(np.float32)
    xy[:5] = [[np.nan, 3.0], [3.0, np.nan], [np.inf, 2.0], [-np.inf, 2.0], [1e30, 1e30]]
    out = {}
    for fmt in (hpm_b200.TEX_F32, hpm_b200.TEX_U8):
        with hpm_b200.Context(0) as ctx:
            ctx.set_address_mode(address_mode)
            ctx.set_texture_format(fmt)
            ctx.set_view(0, img, cam)
            out[fmt] = ctx.sample_view(0, xy)
    np.testing.assert_array_equal(np.rint(out[hpm_b200.TEX_U8].astype(np.float64) * 65280.0),
                                  out[hpm_b200.TEX_F32].astype(np.float64) * 256.0)


def _scene(n_src, width, height, seed):
    from hpm_b200 import synth
    scene = synth.make_scene(n_views=n_src + 1, width=width, height=height, seed=seed, n_src=n_src, supersample=1)
    return scene, scene_cams(scene), scene_grays(scene)


def _partial(scene, cams, grays, n_half, shifted=False):
    import cv2
    srcs = [j for j, _ in scene.pairs[0]]
    params = hpm_b200.Params.make(len(srcs) + 1, *hpm_b200.widened_range(cams[0]))
    with hpm_b200.Context(0) as ctx:
        if shifted:
            ctx.set_ncc_mode(hpm_b200.NCC_SHIFTED)
        for i, (g, c) in enumerate(zip(grays, cams)):
            ctx.set_view(i, g, c)
        ctx.set_canny(0, cv2.Canny(scene.views[0].image, 50, 150))
        return ctx.run_partial(0, srcs, params, n_half, seed=5)


# one below, at and above each source count the kernels are specialised for; widths around a warp
@pytest.mark.gpu
@pytest.mark.parametrize("n_src,width,height", [(1, 31, 40), (4, 33, 37), (5, 64, 48), (10, 65, 41), (11, 40, 33),
                                                (16, 37, 40), (17, 33, 36)])
def test_half_sweeps_match_oracle(n_src, width, height):
    import cv2
    scene, cams, grays = _scene(n_src, width, height, 40 + n_src)
    g = _partial(scene, cams, grays, 2)
    srcs = [j for j, _ in scene.pairs[0]]
    params = hpm_b200.Params.make(len(srcs) + 1, *hpm_b200.widened_range(cams[0]))
    st = ora.RunState(width, height)
    st.canny[:] = cv2.Canny(scene.views[0].image, 50, 150)
    imgs, cs = [grays[0]] + [grays[j] for j in srcs], [cams[0]] + [cams[j] for j in srcs]
    ora.random_init(imgs, cs, params, st, 5, 0)
    for k in range(2):
        ora.half_sweep(imgs, None, cs, params, st, k & 1, k >> 1, 5, 0)
    np.testing.assert_array_equal(g["rng_draw"], st.rng_draw)
    np.testing.assert_array_equal(g["selected_views"], st.selected_views)
    np.testing.assert_array_equal(g["planes"], st.planes)
    np.testing.assert_array_equal(g["costs"], st.costs)


@pytest.mark.gpu
@pytest.mark.parametrize("shifted", [False, True])
@pytest.mark.parametrize("changed", ["reference", "source"])
def test_float_images_take_the_general_path_with_the_same_bits(changed, shifted):
    """One texel off the whole levels sends an image down the general path; away from that texel nothing
    may change.  The initialisation and one half-sweep read at most 40 px around a pixel."""
    scene, cams, grays = _scene(4, 150, 140, 8)
    whole = _partial(scene, cams, grays, 1, shifted)
    other = [g.copy() for g in grays]
    view = 0 if changed == "reference" else scene.pairs[0][1][0]
    other[view][0, 0] = np.floor(other[view][0, 0]) + (0.5 if other[view][0, 0] < 255 else -0.5)
    mixed = _partial(scene, cams, other, 1, shifted)
    far = np.ones((140, 150), bool)
    if changed == "reference":
        far[:64, :64] = False
        for k in ("planes", "costs", "selected_views", "rng_draw"):
            np.testing.assert_array_equal(mixed[k][far], whole[k][far], err_msg=k)
    else:
        # a hypothesis reads the corner when its patch lands within 6 px of it: about 36 in 21000 positions,
        # for each of the some twenty hypotheses a pixel and its neighbours cost
        for k in ("planes", "costs", "selected_views", "rng_draw"):
            same = (mixed[k] == whole[k]).reshape(140, 150, -1).all(-1)
            assert same.mean() > 0.9, (k, same.mean())
