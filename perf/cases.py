"""The workloads whose speed this repository is held to.

Every case is one call, or one short sequence of calls, that a reconstruction program makes through
the Python binding of the C ABI (hpm-mvs_plusplus_b200/__init__.py):

  patchmatch   one PatchMatch run of a reference view (hpm_run_patchmatch) in one of the modes of the
               schedule, with its hypothesis maps uploaded and its results read back;
  reconstruct  the whole schedule over a small scene (hpm_reconstruct), images uploaded, maps and points
               read back;
  confidence   ConfidenceEvaluation over all views of a level (hpm_confidence_eval);
  fuse         fusion of all views' final maps into points (hpm_fuse);
  cost_grad    costs and their gradients for a batch of hypotheses (hpm_eval_cost_grad_device), the
               forward and backward pass of the torch.autograd binding;
  refine       Gauss-Newton refinement of a view's maps (hpm_gn_refine).

Scenes are the seeded synthetic ones of the benchmark (synth.py): views 7.5 degrees apart on an arc, the
middle one as the reference.  The maps that a pass starts from are the rendered truth with the errors that
an earlier pass leaves: sub-percent depth noise, tilted normals, a share of outliers.
"""
import importlib
import math

import numpy as np
import torch

hpm = importlib.import_module("hpm-mvs_plusplus_b200")
synth = importlib.import_module("hpm-mvs_plusplus_b200.synth")

TEXTURES = {"f32": hpm.TEX_F32, "f16": hpm.TEX_F16, "u8": hpm.TEX_U8}
NCC = {"plain": hpm.NCC_PLAIN, "shifted": hpm.NCC_SHIFTED}
MODES = {
    "photometric": 0,
    "prior": hpm.MODE_PRIOR,
    "hierarchy": hpm.MODE_HIERARCHY,
    "geometric": hpm.MODE_GEOM,
    "mandatory": hpm.MODE_GEOM | hpm.MODE_MULTIGEOM | hpm.MODE_MAND,
}


def _pm(mode, width, height, n_src, texture="f32", ncc="plain", flat=0.0):
    return {"kind": "patchmatch", "mode": mode, "width": width, "height": height, "n_src": n_src,
            "texture": texture, "ncc": ncc, "flat": flat}


def listed():
    cases = [
        # the first pass of a preview: 1280x960 views at scale 4, four sources; one run does not fill the GPU
        ("photometric_320x240_s4", _pm("photometric", 320, 240, 4)),
        # the first pass at the coarse level of the headline scene
        ("photometric_800x600_s10", _pm("photometric", 800, 600, 10)),
        # the first geometric pass on views of an odd size with more sources than usual, 8-bit source textures
        ("geometric_1021x763_s13_u8", _pm("geometric", 1021, 763, 13, texture="u8")),
        # the last passes at the fine level of the headline scene: geometric with mandatory consistency
        ("mandatory_1600x1200_s10", _pm("mandatory", 1600, 1200, 10)),
        # the planar-prior pass at the fine level
        ("prior_1600x1200_s10", _pm("prior", 1600, 1200, 10)),
        # the step from the coarse to the fine level: joint bilateral upsampling, then the hierarchy pass
        ("hierarchy_1600x1200_s10", _pm("hierarchy", 1600, 1200, 10)),
        # a whole preview reconstruction, batched over the views, 8-bit textures: many small launches
        ("reconstruct_5x1280x960_scale4", {"kind": "reconstruct", "views": 5, "width": 1280, "height": 960, "scale": 4,
                                           "n_src": 4, "form": "chosen"}),
        # a whole reconstruction at one level as the command line runs it, view after view
        ("reconstruct_6x640x480", {"kind": "reconstruct", "views": 6, "width": 640, "height": 480, "scale": 1,
                                   "n_src": 5, "form": "plain"}),
        # the consistency check between passes, all views of a scene at the fine level
        ("confidence_11x1600x1200_s10", {"kind": "confidence", "views": 11, "width": 1600, "height": 1200,
                                         "n_src": 10}),
        # the point cloud at the end
        ("fuse_11x800x600_s10", {"kind": "fuse", "views": 11, "width": 800, "height": 600, "n_src": 10}),
        # one optimiser step's costs and gradients at sampled pixels of a 1024x768 view
        ("cost_grad_10000_s10", {"kind": "cost_grad", "n": 10000, "width": 1024, "height": 768, "n_src": 10}),
        # polishing a view's maps after the schedule
        ("refine_640x480_s10", {"kind": "refine", "width": 640, "height": 480, "n_src": 10, "steps": 3}),
    ]
    return [{"name": name, **case} for name, case in cases]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A width between lo and hi and a height of a common aspect ratio; odd sizes among them."""
    w = _log_int(rng, lo, hi)
    return w, max(96, min(int(round(w / rng.uniform(1.25, 1.8))), 3 * w // 4))


def draw(rng):
    kind = rng.choice(["patchmatch"] * 5 + ["reconstruct", "confidence", "fuse", "cost_grad", "refine"])
    if kind == "patchmatch":
        w, h = _size(rng, 200, 1600)
        mode = rng.choice(sorted(MODES))
        n_src = rng.randint(2, 16)
        while n_src * w * h > 10 * 1600 * 1200:
            n_src = rng.randint(2, 16)
        return _pm(mode, w, h, n_src, rng.choice(["f32", "f32", "u8", "f16"]),
                   rng.choice(["plain", "plain", "shifted"]), rng.choice([0.0, 0.0, 0.4]))
    if kind == "reconstruct":
        scale = rng.choice([1, 2, 4])
        w, h = _size(rng, 160 * scale, min(1280, 640 * scale))
        views = rng.randint(3, 6)
        return {"kind": kind, "views": views, "width": w, "height": h, "scale": scale,
                "n_src": rng.randint(2, views - 1), "form": rng.choice(["plain", "chosen"])}
    if kind in ("confidence", "fuse"):
        w, h = _size(rng, 200, 1600 if kind == "confidence" else 1000)
        views = rng.randint(3, 11)
        return {"kind": kind, "views": views, "width": w, "height": h, "n_src": rng.randint(2, views - 1)}
    if kind == "cost_grad":
        w, h = _size(rng, 320, 1024)
        return {"kind": kind, "n": _log_int(rng, 64, 40000), "width": w, "height": h, "n_src": rng.randint(2, 16)}
    w, h = _size(rng, 160, 640)
    return {"kind": kind, "width": w, "height": h, "n_src": rng.randint(2, 10), "steps": rng.randint(1, 3)}


# ---------------------------------------------------------------- inputs


def _scene(views, width, height, n_src, seed, flat=0.0):
    """The seeded scene: `views` views 7.5 degrees apart, sources by angle."""
    return synth.make_scene(n_views=views, width=width, height=height, layout="arc", arc_deg=7.5 * (views - 1),
                            n_src=n_src, seed=seed % (1 << 30), device="cuda" if torch.cuda.is_available() else "cpu",
                            supersample=1, textureless_area=flat)


def _camera(v):
    h, w = v.image.shape[:2]
    return hpm.Camera.make(v.K, v.R, v.t, w, h, v.depth_min, v.depth_max)


def _smooth(g, w, h, cell, dev):
    """A smooth random field in 0..1 with features about `cell` pixels across."""
    coarse = torch.rand(1, 1, h // cell + 2, w // cell + 2, generator=g, device=dev)
    return torch.nn.functional.interpolate(coarse, size=(h, w), mode="bicubic", align_corners=True)[0, 0].clamp(0, 1)


def _maps(v, seed, only_depth=False):
    """Depth, world normal, cost and confidence maps of a view as an earlier pass leaves them."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    h, w = v.depth.shape
    gt = torch.from_numpy(v.depth).to(dev)
    wrong = _smooth(g, w, h, 24, dev) > 0.72          # patches that the earlier pass got wrong
    wrong |= torch.rand(h, w, generator=g, device=dev) < 0.02
    wrong |= gt <= 0
    lo, hi = 0.6 * v.depth_min, 1.2 * v.depth_max
    depth = gt * (1 + 0.0015 * torch.randn(h, w, generator=g, device=dev))
    depth = torch.where(wrong, lo + (hi - lo) * torch.rand(h, w, generator=g, device=dev), depth).float()
    if only_depth:
        return {"depth": depth.cpu().numpy()}
    n = torch.from_numpy(v.normal).to(dev) + 0.05 * torch.randn(h, w, 3, generator=g, device=dev)
    n = torch.where(wrong[..., None], torch.randn(h, w, 3, generator=g, device=dev), n)
    n = torch.nn.functional.normalize(n, dim=-1)
    # the normal faces the camera, as every hypothesis does
    ys, xs = torch.meshgrid(torch.arange(h, device=dev), torch.arange(w, device=dev), indexing="ij")
    ray = torch.stack([(xs - float(v.K[0, 2])) / float(v.K[0, 0]), (ys - float(v.K[1, 2])) / float(v.K[1, 1]),
                       torch.ones(h, w, device=dev)], -1) @ torch.from_numpy(v.R).to(dev)
    n = torch.where((n * ray).sum(-1, keepdim=True) > 0, -n, n)
    spread = torch.rand(h, w, generator=g, device=dev)
    cost = torch.where(wrong, 0.25 + 1.2 * spread, 0.02 + 0.2 * spread * spread)
    conf = (2.0 * (_smooth(g, w, h, 16, dev) - 0.45)).clamp(0, 1) + 0.1 * torch.rand(h, w, generator=g, device=dev)
    conf = torch.where(wrong, torch.zeros_like(conf), conf)
    return {"depth": depth.cpu().numpy(), "normal": n.float().cpu().numpy(), "cost": cost.float().cpu().numpy(),
            "conf": conf.float().cpu().numpy()}


def _pinned(a):
    """The array in page-locked host memory, where a program keeps what it uploads on every call."""
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.pin_memory().numpy() if torch.cuda.is_available() else t.numpy()


def _pinned_empty(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def _load(ctx, scene, views=None):
    """Original images and level images (grey, texture, colour, edges) of the views at full size."""
    cams = [_camera(v) for v in scene.views]
    for i in range(len(cams)) if views is None else views:
        ctx.set_image(i, scene.views[i].image)
        ctx.prepare_level(i, cams[i].width, cams[i].height, cams[i])
    return cams


def _pixels(case, scene, ref, seed):
    """Random pixels of the reference and hypotheses (depth, nx, ny) around the true surface."""
    rng = np.random.default_rng(seed)
    v = scene.views[ref]
    h, w = v.depth.shape
    x = rng.integers(0, w, case["n"])
    y = rng.integers(0, h, case["n"])
    gt = v.depth[y, x].astype(np.float64)
    d = np.where(gt > 0, gt * (1 + rng.normal(0, 0.003, gt.shape)), rng.uniform(v.depth_min, v.depth_max, gt.shape))
    n = v.normal[y, x].astype(np.float64) @ v.R.astype(np.float64).T + rng.normal(0, 0.012, (case["n"], 3))
    n[gt <= 0] = rng.normal(0, 0.3, (int((gt <= 0).sum()), 3)) + [0, 0, -1]
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    n[n[:, 2] > 0] *= -1
    return np.stack([x, y], 1).astype(np.int32), np.concatenate([d[:, None], n[:, :2]], 1).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    ctx = hpm.Context(0)
    st = {"case": case, "ctx": ctx, "seed": seed}
    if kind == "patchmatch":
        ctx.set_texture_format(TEXTURES[case["texture"]])
        ctx.set_ncc_mode(NCC[case["ncc"]])
        w, h, n_src = case["width"], case["height"], case["n_src"]
        scene = _scene(n_src + 1, w, h, n_src, seed, case["flat"])
        ref = (n_src + 1) // 2
        srcs = [j for j, _ in scene.pairs[ref]]
        cams = _load(ctx, scene)
        lo, hi = hpm.widened_range(cams[ref])
        st.update(ref=ref, srcs=srcs, params=hpm.Params.make(n_src + 1, lo, hi, MODES[case["mode"]]), maps=[])
        depth_kind = hpm.MAP_DEPTH_GEOM if case["mode"] in ("geometric", "mandatory") else hpm.MAP_DEPTH
        if case["mode"] == "hierarchy":
            # maps of the coarser level, half the size
            m = {k: a[:h // 2 * 2:2, :w // 2 * 2:2] for k, a in _maps(scene.views[ref], seed + 1).items()}
            st["maps"] = [(hpm.MAP_DEPTH_GEOM, _pinned(m["depth"])), (hpm.MAP_NORMAL, _pinned(m["normal"])),
                          (hpm.MAP_COST, _pinned(m["cost"]))]
        elif case["mode"] != "photometric":
            m = _maps(scene.views[ref], seed + 1)
            inp = hpm.MAP_DEPTH_GEOM if case["mode"] == "mandatory" else hpm.MAP_DEPTH
            st["maps"] = [(inp, _pinned(m["depth"])), (hpm.MAP_NORMAL, _pinned(m["normal"])),
                          (hpm.MAP_COST, _pinned(m["cost"]))]
            ctx.set_map(ref, hpm.MAP_CONF, m["conf"])
            if case["mode"] == "prior":
                for k, a in st["maps"]:
                    ctx.set_map(ref, k, a)
                ctx.build_prior(ref, 0)
            else:
                for j in srcs:
                    ctx.set_map(j, inp, _maps(scene.views[j], seed + 2 + j, only_depth=True)["depth"])
        st["out"] = [(depth_kind, _pinned_empty((h, w))), (hpm.MAP_NORMAL, _pinned_empty((h, w, 3))),
                     (hpm.MAP_COST, _pinned_empty((h, w)))]
    elif kind == "reconstruct":
        w, h = case["width"], case["height"]
        scene = _scene(case["views"], w, h, case["n_src"], seed)
        st["images"] = [_pinned(v.image) for v in scene.views]
        st["cams"] = [_camera(v) for v in scene.views]
        st["srcs"] = [[j for j, _ in p] for p in scene.pairs]
        if case["form"] == "chosen":
            ctx.set_texture_format(hpm.TEX_U8)
            ctx.set_batch_options(hpm.BATCH_AUTOTUNE | hpm.BATCH_GRAPH)
        st["points"] = _pinned_empty((case["views"] * w * h // (2 * case["scale"] ** 2), 9))
        st["points"][:] = 0
        st["batch"] = hpm.RECON_BATCH_EXACT if case["form"] == "chosen" else hpm.RECON_SEQUENTIAL
    elif kind in ("confidence", "fuse"):
        scene = _scene(case["views"], case["width"], case["height"], case["n_src"], seed)
        _load(ctx, scene)
        st["srcs"] = [[j for j, _ in p] for p in scene.pairs]
        st["depth_kind"] = hpm.MAP_DEPTH_GEOM if kind == "fuse" else hpm.MAP_DEPTH
        for i, v in enumerate(scene.views):
            m = _maps(v, seed + 1 + i)
            ctx.set_map(i, st["depth_kind"], m["depth"])
            ctx.set_map(i, hpm.MAP_NORMAL, m["normal"])
        if kind == "confidence":
            st["out"] = [_pinned_empty((case["height"], case["width"])) for _ in scene.views]
        else:
            st["points"] = _pinned_empty((case["views"] * case["width"] * case["height"] // 2, 9))
            st["points"][:] = 0
    else:
        scene = _scene(case["n_src"] + 1, case["width"], case["height"], case["n_src"], seed)
        ref = (case["n_src"] + 1) // 2
        cams = _load(ctx, scene)
        lo, hi = hpm.widened_range(cams[ref])
        st.update(ref=ref, srcs=[j for j, _ in scene.pairs[ref]], params=hpm.Params.make(case["n_src"] + 1, lo, hi))
        if kind == "cost_grad":
            px, theta = _pixels(case, scene, ref, seed + 1)
            st["px"] = torch.from_numpy(px).cuda()
            st["theta"] = torch.from_numpy(theta).cuda()
        else:
            m = _maps(scene.views[ref], seed + 1)
            st["maps"] = [(hpm.MAP_DEPTH_GEOM, _pinned(m["depth"])), (hpm.MAP_NORMAL, _pinned(m["normal"])),
                          (hpm.MAP_COST, _pinned(m["cost"]))]
            h, w = case["height"], case["width"]
            st["out"] = [(hpm.MAP_DEPTH_GEOM, _pinned_empty((h, w))), (hpm.MAP_NORMAL, _pinned_empty((h, w, 3))),
                         (hpm.MAP_COST, _pinned_empty((h, w)))]
    ctx.synchronize()
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "patchmatch":
        for k, a in st["maps"]:
            ctx.set_map(st["ref"], k, a)
        if case["mode"] == "hierarchy":
            ctx.jbu(st["ref"])
        ctx.run_patchmatch(st["ref"], st["srcs"], st["params"], texture_level=0, seed=st["seed"])
        return [ctx.get_map(st["ref"], k, out) for k, out in st["out"]]
    if kind == "reconstruct":
        for i, im in enumerate(st["images"]):
            ctx.set_image(i, im)
        ctx.reconstruct(st["cams"], st["srcs"], initial_image_scale=case["scale"], seed=st["seed"], batch=st["batch"])
        out = [len(ctx.get_points(out=st["points"])), st["points"]]
        for i in range(len(st["images"])):
            out += [ctx.get_map(i, hpm.MAP_DEPTH_GEOM), ctx.get_map(i, hpm.MAP_NORMAL)]
        return out
    if kind == "confidence":
        ctx.confidence_eval(st["srcs"], st["depth_kind"])
        return [ctx.get_map(i, hpm.MAP_CONF, out) for i, out in enumerate(st["out"])]
    if kind == "fuse":
        _, n = ctx.fuse(st["srcs"], st["depth_kind"], capacity=0)  # the points stay on the GPU until they are read
        ctx.get_points(out=st["points"])
        return [n, st["points"]]
    if kind == "cost_grad":
        return ctx.eval_cost_grad_tensors(st["ref"], st["srcs"], st["params"], st["px"], st["theta"])
    for k, a in st["maps"]:
        ctx.set_map(st["ref"], k, a)
    ctx.gn_refine(st["ref"], st["srcs"], st["params"], hpm.MAP_DEPTH_GEOM, case["steps"])
    return [ctx.get_map(st["ref"], k, out) for k, out in st["out"]]


# ---------------------------------------------------------------- work


def work(case):
    """Inputs read once, outputs written once; flops of the algorithm: 31 per warped patch sample (12
    homography, 3 perspective divide, 6 bilinear, 6 moments and the per-hypothesis setup), 36 samples."""
    kind = case["kind"]
    ncc = 36 * 31
    if kind == "patchmatch":
        n, s = case["width"] * case["height"], case["n_src"]
        # initial costs, then three iterations over all pixels: eight neighbours against every source, the
        # current plane and five refinements against the about four sources that view selection keeps
        updated = 0.55 if case["mode"] == "prior" else 1.0
        evals = n * (s + 3 * updated * (8 * s + 6 * min(4, s)))
        maps_in = 0 if case["mode"] == "photometric" else 20 * n
        if case["mode"] in ("geometric", "mandatory"):
            maps_in += 4 * n * s
        return {"bytes": n * (s + 1) + maps_in + 20 * n, "flops": evals * ncc}
    if kind == "reconstruct":
        w, h = case["width"] // case["scale"], case["height"] // case["scale"]
        n, s, v = w * h, case["n_src"], case["views"]
        evals = v * n * 5 * (s + 3 * (8 * s + 6 * min(4, s)))  # photometric, prior and three geometric passes
        return {"bytes": v * (3 * case["width"] * case["height"] + 16 * n + 36 * n // 4), "flops": evals * ncc}
    if kind in ("confidence", "fuse"):
        n = case["width"] * case["height"] * case["views"]
        out = 4 * n if kind == "confidence" else 36 * n // 4
        # per pixel and source: two transforms and projections, a distance, an angle and an exponential
        return {"bytes": 16 * n + out + (3 * n if kind == "fuse" else 0), "flops": 120 * n * case["n_src"]}
    if kind == "cost_grad":
        n, s = case["n"], case["n_src"]
        # the gradient adds the two derivatives of a sample and the chain rule through it
        return {"bytes": n * (8 + 12 + 16 * s) + 4 * (s + 1) * case["width"] * case["height"],
                "flops": n * s * 36 * 60}
    n, s = case["width"] * case["height"], case["n_src"]
    # per step: costs and gradients, then the costs of one trial
    return {"bytes": 40 * n + 4 * n * s, "flops": n * s * (ncc + case["steps"] * (36 * 60 + ncc))}


# ---------------------------------------------------------------- 64-bit values


def _exact_cost_grad(case, seed):
    """The bilateral NCC with exact bilinear sampling and its derivatives with respect to (depth, nx, ny)."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    D = torch.float64
    scene = _scene(case["n_src"] + 1, case["width"], case["height"], case["n_src"], seed)
    ref = (case["n_src"] + 1) // 2
    px, theta = _pixels(case, scene, ref, seed + 1)
    rv = scene.views[ref]
    img = torch.from_numpy(rv.image[..., 0].copy()).to(dev, D)
    H, W = img.shape
    p = torch.from_numpy(px).to(dev)
    th = torch.from_numpy(theta).to(dev, D)
    off = torch.arange(-5, 6, 2, device=dev)
    dx, dy = off.repeat_interleave(6), off.repeat(6)
    gx = (p[:, :1] + dx).clamp(0, W - 1)
    gy = (p[:, 1:] + dy).clamp(0, H - 1)
    r = img[gy, gx]
    centre = img[p[:, 1], p[:, 0]][:, None]
    wt = torch.exp(-torch.sqrt((dx * dx + dy * dy).to(D)) / 50.0 - (r - centre).abs() / 18.0)
    Ws = wt.sum(1)
    mean_r = (wt * r).sum(1) / Ws
    var_r = (wt * (r - mean_r[:, None]) ** 2).sum(1) / Ws
    K, R, t = (torch.from_numpy(a.astype(np.float64)).to(dev) for a in (rv.K, rv.R, rv.t))
    fx, fy, cx, cy = K[0, 0], K[1, 1], K[0, 2], K[1, 2]
    nx, ny = th[:, 1], th[:, 2]
    nz = -torch.sqrt((1 - nx * nx - ny * ny).clamp(min=1e-300))
    n = torch.stack([nx, ny, nz], 1)
    q = p.to(D)
    ray = torch.stack([(q[:, 0] - cx) / fx, (q[:, 1] - cy) / fy, torch.ones_like(nx)], 1)
    nr = (n * ray).sum(1)
    w = -th[:, 0] * nr
    tt = torch.stack([nx / fx, ny / fy, nz - nx * cx / fx - ny * cy / fy], 1)
    m = tt / w[:, None]
    U = torch.stack([q[:, :1] + dx, q[:, 1:] + dy, torch.ones_like(r)], 2)  # n, 36, 3
    Kinv = torch.tensor([[1 / fx, 0, -cx / fx], [0, 1 / fy, -cy / fy], [0, 0, 1]], dtype=D, device=dev)
    costs, grads = [], []
    for j, _ in scene.pairs[ref]:
        sv = scene.views[j]
        Ks, Rs, ts = (torch.from_numpy(a.astype(np.float64)).to(dev) for a in (sv.K, sv.R, sv.t))
        src = torch.from_numpy(sv.image[..., 0].copy()).to(dev, D)
        sh, sw = src.shape
        A = Ks @ Rs @ R.T @ Kinv
        b = Ks @ Rs @ ((-R.T @ t) - (-Rs.T @ ts))
        Hm = A - b[None, :, None] * m[:, None, :]
        c3 = (Hm @ torch.cat([q, torch.ones_like(q[:, :1])], 1)[..., None])[..., 0]
        X0, Y0 = c3[:, 0] / c3[:, 2], c3[:, 1] / c3[:, 2]
        inside = (X0 >= 0) & (X0 < sw) & (Y0 >= 0) & (Y0 < sh)
        P = U @ Hm.transpose(1, 2)
        X, Y, qz = P[..., 0] / P[..., 2], P[..., 1] / P[..., 2], P[..., 2]
        Xc = torch.nan_to_num(X, nan=-2.0).clamp(-2.0, sw + 1.0)
        Yc = torch.nan_to_num(Y, nan=-2.0).clamp(-2.0, sh + 1.0)
        x0, y0 = torch.floor(Xc), torch.floor(Yc)
        ax, ay = Xc - x0, Yc - y0
        xa, xb = x0.long().clamp(0, sw - 1), (x0.long() + 1).clamp(0, sw - 1)
        ya, yb = y0.long().clamp(0, sh - 1), (y0.long() + 1).clamp(0, sh - 1)
        i00, i10, i01, i11 = src[ya, xa], src[ya, xb], src[yb, xa], src[yb, xb]
        v = (1 - ay) * ((1 - ax) * i00 + ax * i10) + ay * ((1 - ax) * i01 + ax * i11)
        vX = (1 - ay) * (i10 - i00) + ay * (i11 - i01)
        vY = (1 - ax) * (i01 - i00) + ax * (i11 - i10)
        Ss = (wt * v).sum(1) / Ws
        var_s = (wt * (v - Ss[:, None]) ** 2).sum(1) / Ws
        cov = (wt * (r - mean_r[:, None]) * (v - Ss[:, None])).sum(1) / Ws
        sig = torch.sqrt(var_r * var_s)
        c = 1 - cov / sig
        dcdv = wt / Ws[:, None] * (-(r - mean_r[:, None]) / sig[:, None]
                                   + (cov / (sig * var_s))[:, None] * (v - Ss[:, None]))
        gb = (vX * b[0] + vY * b[1] - (vX * X + vY * Y) * b[2]) / qz
        dm = (-(dcdv * gb)[..., None] * U).sum(1)
        dw = -(dm * m).sum(1) / w
        dn = torch.stack([dm[:, 0] / fx - dm[:, 2] * cx / fx, dm[:, 1] / fy - dm[:, 2] * cy / fy, dm[:, 2]], 1)
        dn = dn / w[:, None] - (dw * th[:, 0])[:, None] * ray
        g = torch.stack([-dw * nr, dn[:, 0] - dn[:, 2] * nx / nz, dn[:, 1] - dn[:, 2] * ny / nz], 1)
        none = ~inside | (var_r < 1e-5) | (var_s < 1e-5)
        flat = none | (c < 0) | (c > 2)
        costs.append(torch.where(none, torch.full_like(c, 2.0), c.clamp(0, 2)))
        grads.append(torch.where(flat[:, None], torch.zeros_like(g), g))
    return torch.stack(costs, 1), torch.stack(grads, 1)


def exact(case, seed):
    """64-bit values where they exist.  A PatchMatch run, a whole reconstruction, the consistency scans and
    the refinement follow accept-or-reject decisions that rounding moves, so they have none."""
    if case["kind"] == "cost_grad":
        return _exact_cost_grad(case, seed)
    return None
