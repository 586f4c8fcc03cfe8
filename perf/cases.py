"""Performance cases: the work users of this framework have it do, over the
sizes and options they use, each through the public entry points.

Kinds of case (the "kind" key) and what they stand for:

* ``frame``: the render loop.  One pass is one frame of a camera orbit (or of
  a still camera) into a device image, with the reuse state of the frames
  before it: Conditional ReSTIR in both reservoir storages, RestirPt and the
  plain path tracer, optionally tone-mapped and with reprojected temporal
  reuse.
* ``batch``: several views of one scene rendered together, uneven sizes.
* ``trace``: closest-hit and occlusion queries over a scene by a caller with
  rays of its own.
* ``search``: the prefix-endpoint neighbour search over a caller's entries.
* ``tonemap``: one HDR image to sRGB bytes.
* ``pt_adjoint`` / ``restir_adjoint``: one step of inverse rendering: the
  views' images at the current parameters and the gradient of an L2 loss.

Sizes and settings are those of the benchmark's workloads and of the tests;
scenes are the generators of ``crisoptix_b200.scenes``, seeded.
"""
import ctypes
import dataclasses
import math

import numpy as np
import torch

from crisoptix_b200 import Batch, Renderer, Scene, _abi, adjoint, default_params, image, scenes
from crisoptix_b200._abi import check, load

ORBIT = 60  # frames of one camera orbit

#: The renderer types by the names the cases use.
TYPES = {"path_tracer": _abi.PATH_TRACER, "restir_pt": _abi.RESTIR_PT, "conditional": _abi.CONDITIONAL_RESTIR}

#: Work a ray cannot do without: about ten eight-wide nodes and four triangles.
RAY_FLOPS = 10 * 8 * 12 + 4 * 50


def listed():
    return [
        # Interactive preview of a small scene: the benchmark's small workload
        # (still camera, depth 4, no gather neighbours), the lowest-latency frame.
        {"name": "frame_cornell_256", "kind": "frame", "scene": "cornell", "width": 256, "height": 256,
         "type": "conditional", "depth": 4, "prefix": 1, "spatial": 3, "rounds": 1, "k": 0, "window": 30},
        # A path tracer frame of a large scene: what reference images are summed
        # from, one sample per pixel.
        {"name": "frame_path_tracer_960x540", "kind": "frame", "scene": "room", "width": 960, "height": 540,
         "type": "path_tracer", "depth": 8},
        # RestirPt with prefix temporal and spatial reuse over textured materials,
        # at a size no tile divides.
        {"name": "frame_restir_pt_textured_641x479", "kind": "frame", "scene": "textured", "width": 641, "height": 479,
         "type": "restir_pt", "depth": 6, "spatial": 3, "rounds": 2, "window": 10},
        # The benchmark's large workload at half resolution (interactive preview).
        {"name": "frame_room_960x540", "kind": "frame", "scene": "room", "width": 960, "height": 540,
         "type": "conditional", "depth": 8, "prefix": 2, "spatial": 5, "rounds": 2, "k": 8, "window": 10},
        # A viewer's frame: packed reservoirs, reprojected temporal reuse, sRGB
        # bytes out, a ragged size.
        {"name": "frame_room_fp16_reproject_1277x719", "kind": "frame", "scene": "room", "width": 1277, "height": 719,
         "type": "conditional", "depth": 8, "prefix": 2, "spatial": 5, "rounds": 2, "k": 8, "window": 10,
         "storage": 1, "reproject": True, "srgb": True},
        # The benchmark's large workload: 1080p, 1.31 M triangles, depth 8, k = 8.
        {"name": "frame_room_1920x1080", "kind": "frame", "scene": "room", "width": 1920, "height": 1080,
         "type": "conditional", "depth": 8, "prefix": 2, "spatial": 5, "rounds": 2, "k": 8, "window": 10},
        # The batched multiview workload: 16 views of three sizes, packed reservoirs.
        {"name": "batch_16_views_fp16", "kind": "batch", "small": 8, "medium": 4, "large": 4, "storage": 1},
        # A caller's own rays over the large scene: camera rays and bounce rays,
        # nearest hits and occlusion.
        {"name": "trace_1000003_rays", "kind": "trace", "rays": 1000003, "spheres": 64, "subdiv": 5},
        # The endpoint search on its own, at the entry count of a 512 x 512 view.
        {"name": "search_262144", "kind": "search", "entries": 262144, "queries": 262144, "k": 8},
        # One 1080p frame to bytes.
        {"name": "tonemap_1920x1080", "kind": "tonemap", "width": 1920, "height": 1080},
        # An inverse-rendering step with the path tracer: 8 views of 512 x 512.
        {"name": "pt_adjoint_8x512", "kind": "pt_adjoint", "views": 8, "res": 512, "depth": 8},
        # The same with the resampled estimator of rendered frames.
        {"name": "restir_adjoint_8x512", "kind": "restir_adjoint", "views": 8, "res": 512, "depth": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["batch", "trace", "search", "tonemap", "pt_adjoint", "restir_adjoint"])
    if kind == "frame":
        pixels = _log_int(rng, 64 * 48, 1920 * 1080)
        aspect = rng.uniform(1.0, 2.0)
        w = max(8, int(math.sqrt(pixels * aspect)))
        h = max(8, pixels // w)
        c = {"kind": kind, "scene": rng.choice(["cornell", "room", "room", "textured"]), "width": w, "height": h,
             "type": rng.choice(["conditional", "conditional", "conditional", "restir_pt", "path_tracer"])}
        c["depth"] = rng.randint(3, 8)
        if c["type"] != "path_tracer":
            c["spatial"] = rng.randint(1, 5)
            c["rounds"] = rng.randint(1, 2)
            c["window"] = rng.choice([10, 30])
            c["storage"] = rng.randint(0, 1)
            c["reproject"] = rng.random() < 0.4
        if c["type"] == "conditional":
            c["prefix"] = rng.randint(1, 2)
            c["k"] = rng.choice([0, 3, 8])
        c["srgb"] = rng.random() < 0.4
        return c
    if kind == "batch":
        return {"kind": kind, "small": rng.randint(1, 6), "medium": rng.randint(0, 3), "large": rng.randint(0, 3),
                "storage": rng.randint(0, 1)}
    if kind == "trace":
        return {"kind": kind, "rays": _log_int(rng, 1000, 1000003), "spheres": rng.randint(8, 64),
                "subdiv": rng.randint(2, 5)}
    if kind == "search":
        n = _log_int(rng, 1000, 2073600)
        return {"kind": kind, "entries": n, "queries": max(1, int(n * rng.uniform(0.3, 1.0))), "k": rng.choice([1, 4, 8, 16])}
    if kind == "tonemap":
        w = _log_int(rng, 64, 3840)
        return {"kind": kind, "width": w, "height": max(1, int(w * rng.uniform(0.5, 1.0)))}
    return {"kind": kind, "views": rng.randint(1, 8), "res": _log_int(rng, 64, 512), "depth": rng.randint(3, 8)}


# ---- scenes and parameters ----------------------------------------------------------
def _room(seed, aspect, spheres=64, subdiv=5, emitters=256):
    return scenes.sphere_room(num_spheres=spheres, subdiv=subdiv, num_emitters=emitters, seed=1 + seed, aspect=aspect)


def _scene(case, seed):
    """(description, camera) of a frame case; the small scenes are seen from
    a seeded place near their camera."""
    aspect = case["width"] / case["height"]
    if case["scene"] == "room":
        return _room(seed, aspect)
    desc, cam = scenes.cornell_box() if case["scene"] == "cornell" else scenes.textured_cornell_box()
    j = np.random.default_rng(seed).uniform(-0.05, 0.05, 3)
    return desc, dataclasses.replace(cam, pos=tuple(float(a + b) for a, b in zip(cam.pos, j)), aspect=aspect)


def _orbit(cam, start):
    cams = []
    c = cam
    for _ in range(ORBIT):
        cams.append(c)
        c = c.rotate_around_origin((0.0, 1.0, 0.0), 2.0 * math.pi / ORBIT)
    return cams[start:] + cams[:start]


def _params(case, scene_size, seed):
    kind = TYPES[case.get("type", "conditional")]
    kw = dict(renderer_type=kind, nee_prob=0.3, max_path_len=case["depth"], seed=seed, enable_accum=0)
    if kind != _abi.PATH_TRACER:
        kw.update(prefix_len=min(case.get("prefix", 2), case["depth"]), window_radius=case["window"],
                  storage=case.get("storage", 0),
                  motion_mode=_abi.MOTION_REPROJECT if case.get("reproject") else _abi.MOTION_NONE)
    if kind == _abi.RESTIR_PT:
        kw.update(prefix_enable_spatial=1, prefix_spatial_count=case["spatial"], prefix_spatial_rounds=case["rounds"])
    if kind == _abi.CONDITIONAL_RESTIR:
        kw.update(suffix_spatial_count=case["spatial"], suffix_spatial_rounds=case["rounds"], gather_m=case["k"] + 1,
                  gather_radius=0.01)
    return default_params(scene_size, **kw)


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ---- frames -------------------------------------------------------------------------
def _prepare_frame(case, seed):
    w, h = case["width"], case["height"]
    desc, cam = _scene(case, seed)
    sc = Scene(desc)
    s = {"scene": sc, "renderer": Renderer(w, h, sc, _params(case, sc.scene_size, seed)), "frame": 0}
    # the large scene is seen from an orbit, the box by a still camera
    s["cams"] = _orbit(cam, seed % ORBIT) if case["scene"] == "room" else [cam]
    s["rgb"] = torch.zeros(h, w, 3, device="cuda")
    s["srgb"] = torch.zeros(h, w, 3, dtype=torch.uint8, device="cuda") if case.get("srgb") else None
    if s["srgb"] is not None:
        s["renderer"].set_srgb_output(s["srgb"].data_ptr())
    return s


def _run_frame(s):
    cam = s["cams"][s["frame"] % len(s["cams"])]
    s["frame"] += 1
    s["renderer"].launch_frame(cam, s["rgb"].data_ptr(), _stream())
    return {"rgb": s["rgb"], "srgb": s["srgb"]} if s["srgb"] is not None else {"rgb": s["rgb"]}


# ---- batched views ------------------------------------------------------------------
def _sizes(case):
    return [(512, 512)] * case["small"] + [(1280, 720)] * case["medium"] + [(1920, 1080)] * case["large"]


def _prepare_batch(case, seed):
    desc, _ = _room(seed, 1.0)
    sc = Scene(desc)
    views = scenes.multiview_cameras(_sizes(case), seed=2 + seed)
    c = {"type": "conditional", "depth": 8, "prefix": 2, "spatial": 5, "rounds": 2, "k": 8, "window": 10,
         "storage": case["storage"]}
    rs = [Renderer(w, h, sc, _params(c, sc.scene_size, seed + i)) for i, (_, w, h) in enumerate(views)]
    outs = [torch.zeros(h, w, 3, device="cuda") for _, w, h in views]
    return {"scene": sc, "batch": Batch(rs), "cams": [c for c, _, _ in views], "outs": outs}


def _run_batch(s):
    # each view orbits the room's vertical axis, 30 frames per sequence
    s["cams"] = [c.rotate_around_origin((0.0, 1.0, 0.0), 2.0 * math.pi / 30) for c in s["cams"]]
    s["batch"].render(s["cams"], [o.data_ptr() for o in s["outs"]], _stream())
    return s["outs"]


# ---- ray queries --------------------------------------------------------------------
def _prepare_trace(case, seed):
    desc, cam = _room(seed, 1.0, case["spheres"], case["subdiv"])
    n = case["rays"]
    rng = np.random.default_rng(seed)
    # half camera rays in scan order, half bounce rays between places in the room
    m = n // 2
    side = max(1, int(math.ceil(math.sqrt(max(m, 1)))))
    i = np.arange(m)
    f = np.asarray(cam.view_dir, np.float64)
    right = np.cross(f, cam.up)
    right /= np.linalg.norm(right)
    up = np.cross(right, f)
    t = math.tan(cam.fov / 2)
    d = (f + np.outer((2.0 * (i % side + 0.5) / side - 1.0) * t, right) -
         np.outer((2.0 * (i // side + 0.5) / side - 1.0) * t, up))
    o = np.broadcast_to(np.asarray(cam.pos), d.shape)
    half = np.array([9.9, 3.9, 9.9])
    o2 = rng.uniform(-half, half, (n - m, 3))
    d2 = rng.uniform(-half, half, (n - m, 3)) - o2
    o, d = np.concatenate([o, o2]), np.concatenate([d, d2])
    dist = np.linalg.norm(d, axis=1, keepdims=True)
    dist[:m] = 10.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    closest = np.concatenate([o, np.full((n, 1), 1e-3), d, np.full((n, 1), 1e16)], axis=1)
    occlusion = np.concatenate([o, np.full((n, 1), 1e-3), d, dist], axis=1)
    return {"scene": Scene(desc), "n": n,
            "closest": torch.from_numpy(closest.astype(np.float32)).cuda(),
            "occlusion": torch.from_numpy(occlusion.astype(np.float32)).cuda(),
            "hits": torch.zeros(n, 4, device="cuda"), "seen": torch.zeros(n, 4, device="cuda")}


def _run_trace(s):
    st = _stream()
    s["scene"].trace(s["closest"].data_ptr(), s["hits"].data_ptr(), s["n"], False, st)
    s["scene"].trace(s["occlusion"].data_ptr(), s["seen"].data_ptr(), s["n"], True, st)
    return {"prim": s["hits"].view(torch.int32)[:, 0], "tuv": s["hits"][:, 1:], "seen": s["seen"].view(torch.int32)[:, 0]}


# ---- endpoint search ----------------------------------------------------------------
def _surface_points(n, gen):
    """Points on the walls of the large scene's room and on 64 spheres in it."""
    half = torch.tensor([10.0, 4.0, 10.0])
    p = (torch.rand(n, 3, generator=gen) * 2 - 1) * half
    wall = torch.rand(n, generator=gen) < 0.7
    axis = torch.multinomial(torch.tensor([80.0, 200.0, 80.0]), n, replacement=True, generator=gen)
    face = torch.where(torch.rand(n, generator=gen) < 0.5, -half[axis], half[axis])
    w = p.scatter(1, axis[:, None], face[:, None])
    centre = ((torch.rand(64, 3, generator=gen) * 2 - 1) * (half - 1.0))
    radius = 0.2 + 0.8 * torch.rand(64, generator=gen)
    which = torch.randint(0, 64, (n,), generator=gen)
    d = torch.randn(n, 3, generator=gen)
    q = centre[which] + radius[which, None] * d / d.norm(dim=1, keepdim=True)
    return torch.where(wall[:, None], w, q)


def _prepare_search(case, seed):
    gen = torch.Generator().manual_seed(seed)
    pts = _surface_points(case["entries"] + case["queries"], gen)
    pts = pts[torch.randperm(len(pts), generator=gen)]
    n, m = case["entries"], case["queries"]
    # radius = gather radius x path length / 4.5; a tenth of the pixels has no endpoint
    r = 0.01 * (4.0 + 36.0 * torch.rand(n, generator=gen)) / 4.5
    r[torch.rand(n, generator=gen) < 0.1] = -1.0
    return {"entries": torch.cat([pts[:n], r[:, None]], 1).contiguous().cuda(), "queries": pts[n:].contiguous().cuda(),
            "n": n, "m": m, "k": case["k"], "out": torch.zeros(m, case["k"], 2, device="cuda"),
            "count": torch.zeros(m, dtype=torch.int32, device="cuda")}


def _run_search(s):
    check(load().crisb_endpoint_search(s["entries"].data_ptr(), s["n"], s["queries"].data_ptr(), s["m"], s["k"],
                                       s["out"].data_ptr(), s["count"].data_ptr(), ctypes.c_void_p(_stream())))
    return {"count": s["count"], "dist": s["out"][..., 1], "pixel": s["out"].view(torch.int32)[..., 0]}


def _exact_search(case, seed):
    """Distances of the k nearest covering entries, by testing every entry."""
    if case["entries"] * case["queries"] > 8e10:
        return None
    s = _prepare_search(case, seed)
    e, q = s["entries"].double(), s["queries"].double()
    e = e[e[:, 3] >= 0]
    k = min(case["k"], len(e))
    dist = torch.zeros(case["queries"], case["k"], dtype=torch.float64, device=e.device)
    for a in range(0, len(q), 1024):
        d = torch.cdist(q[a:a + 1024], e[:, :3], compute_mode="donot_use_mm_for_euclid_dist")
        d[d > e[:, 3]] = math.inf
        near = d.topk(k, dim=1, largest=False, sorted=True).values
        dist[a:a + 1024, :k] = torch.where(near.isinf(), 0.0, near)
    return {"count": None, "dist": dist, "pixel": None}


# ---- tone mapping -------------------------------------------------------------------
def _prepare_tonemap(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    # HDR radiance: log-normal about mid grey, a tenth of the pixels unlit
    rgb = torch.randn(case["height"], case["width"], 3, device="cuda", generator=gen).mul_(1.5).exp_().mul_(0.2)
    rgb *= torch.rand(case["height"], case["width"], 1, device="cuda", generator=gen) >= 0.1
    return {"rgb": rgb, "out": torch.zeros(case["height"], case["width"], 3, dtype=torch.uint8, device="cuda")}


def _run_tonemap(s):
    return image.tonemap(s["rgb"], s["out"], _stream())


# ---- inverse rendering --------------------------------------------------------------
def _inverse_scene(case, seed):
    desc, _ = _room(seed, 1.0)
    sc = Scene(desc)
    cams = [c for c, _, _ in scenes.multiview_cameras([(case["res"], case["res"])] * case["views"], seed=3 + seed)]
    return desc, sc, cams, adjoint.perturbed_start(desc, seed=3 + seed)


def _set(sc, mats, rgb):
    adjoint.set_materials(sc, mats)
    adjoint.set_emitter_colors(sc, rgb)


def _prepare_pt_adjoint(case, seed):
    desc, sc, cams, (tm, trgb, sm, srgb) = _inverse_scene(case, seed)
    _set(sc, sm, srgb)
    p = default_params(sc.scene_size, max_path_len=case["depth"], nee_prob=0.3, seed=3 + seed)
    adj = adjoint.PtAdjoint(sc, case["res"], case["res"], p)
    _set(sc, tm, trgb)
    target = adj.render(cams)
    _set(sc, sm, srgb)
    return {"scene": sc, "adj": adj, "cams": cams, "target": target}


def _run_pt_adjoint(s):
    img = s["adj"].render(s["cams"])
    g_mat, g_em = s["adj"].gradient(s["cams"], 2.0 * (img - s["target"]))
    return {"image": img, "materials": g_mat, "emitters": g_em}


def _prepare_restir_adjoint(case, seed):
    desc, sc, cams, (tm, trgb, sm, srgb) = _inverse_scene(case, seed)
    _set(sc, sm, srgb)
    p = adjoint.restir_params(sc.scene_size, 3 + seed, max_path_len=case["depth"])
    adj = adjoint.RestirAdjoint(sc, case["res"], case["res"], p, len(cams))
    adj.prepare(cams, 3)
    _set(sc, tm, trgb)
    target = adj.render()
    _set(sc, sm, srgb)
    return {"scene": sc, "adj": adj, "target": target}


def _run_restir_adjoint(s):
    img = s["adj"].render()
    g_mat, g_em = s["adj"].gradient(2.0 * (img - s["target"]))
    return {"image": img, "materials": g_mat, "emitters": g_em}


# ---- work ---------------------------------------------------------------------------
def _frame_work(case, pixels):
    """Per pixel: the reservoirs read and written once and the image, and the
    rays of the paths and of the shifts (a path of d vertices: about d / 2
    extension rays and one light ray)."""
    packed = case.get("storage", 0) == 1
    pre, suf = (80, 64) if packed else (144, 112)
    path = case["depth"] / 2 + 1
    if case["type"] == "path_tracer":
        return 12 * pixels, pixels * path * RAY_FLOPS
    if case["type"] == "restir_pt":
        return pixels * (2 * pre + 12), pixels * (path + 2 * case["spatial"] * case["rounds"]) * RAY_FLOPS
    rays = 2 * path + 1 + 2  # suffix and gather paths, the prefix, the shifts that are left
    return pixels * (2 * pre + 2 * suf + 12), pixels * rays * RAY_FLOPS


def work(case):
    kind = case["kind"]
    if kind == "frame":
        p = case["width"] * case["height"]
        b, f = _frame_work(case, p)
        return {"bytes": b + (3 * p if case.get("srgb") else 0), "flops": f}
    if kind == "batch":
        c = {"type": "conditional", "depth": 8, "storage": case["storage"]}
        b, f = _frame_work(c, sum(w * h for w, h in _sizes(case)))
        return {"bytes": b, "flops": f}
    if kind == "trace":
        return {"bytes": case["rays"] * 2 * (32 + 16), "flops": case["rays"] * 2 * RAY_FLOPS}
    if kind == "search":
        n, m, k = case["entries"], case["queries"], case["k"]
        return {"bytes": 16 * n + 12 * m + 8 * k * m + 4 * m, "flops": 10.0 * m * (k + math.log2(n + 1))}
    if kind == "tonemap":
        return {"bytes": case["width"] * case["height"] * 15, "flops": case["width"] * case["height"] * 3 * 4}
    p = case["views"] * case["res"] * case["res"]
    # the image out, its gradient in; every path traced for the image and again for the gradient
    paths = 2 if kind == "pt_adjoint" else 6
    return {"bytes": 24 * p, "flops": paths * p * (case["depth"] / 2 + 1) * RAY_FLOPS}


# ---- the interface ------------------------------------------------------------------
_PREPARE = {"frame": _prepare_frame, "batch": _prepare_batch, "trace": _prepare_trace, "search": _prepare_search,
            "tonemap": _prepare_tonemap, "pt_adjoint": _prepare_pt_adjoint, "restir_adjoint": _prepare_restir_adjoint}
_RUN = {"frame": _run_frame, "batch": _run_batch, "trace": _run_trace, "search": _run_search, "tonemap": _run_tonemap,
        "pt_adjoint": _run_pt_adjoint, "restir_adjoint": _run_restir_adjoint}


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    # radiance follows the sampling decisions of 32-bit arithmetic, and hits
    # over a large scene would take too long to test one by one
    return _exact_search(case, seed) if case["kind"] == "search" else None
