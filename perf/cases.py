"""The work that programs have this renderer do, as measurable cases.

A case is one pass through the public entry points: a frame of a view, of a stereo pair, of a
foveated headset or of many views at once, an animated frame with its refit, a depth query, a new
per-gaze sample set, or a burst of requests to the render server. `prepare` brings up what such a
program keeps between frames (resident scene, clustered samples, render targets, the first frame
out); `run` is the steady-state pass.

The scene geometry of a given size is one asset (the seeded generator of `hvvr_b200.scenes`); the
seed of a case draws what differs from call to call: the camera poses, the gaze, the animation
phase, the jitter of a sample set.
"""
import ctypes
import functools
import math
import random

import numpy as np
import torch

import hvvr_b200 as hv
from hvvr_b200 import _abi, scenes, workloads

DEVICE = "cuda"
IPD = 0.064


# ---------------------------------------------------------------- the cases
def _view(name, **kw):
    """A frame of one or two pinhole, thin-lens or textured cameras over one scene."""
    case = {"kind": "view", "triangles": 57344, "width": 640, "height": 480, "sampling": "grid", "msaa": 1, "eyes": 1,
            "lens": 0.0, "textures": 0, "rotated_grid": False, "strict": False, "host_image": False, "animate": False}
    case.update(kw)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest call: a depth and triangle query under a small window (picking, compositing);
        # launches and the read-back's latency decide it
        {"name": "pick", "kind": "pick", "triangles": 57344, "width": 160, "height": 120},
        # a desktop window without antialiasing on a small scene, the image left on the device
        _view("window", triangles=57344, width=640, height=480),
        # a ragged window on a medium scene, lens-distorted samples, the image copied to host memory
        _view("host_window", triangles=300000, width=811, height=613, sampling="barrel", msaa=4, host_image=True),
        # the headset frame: both eyes, lens-distorted samples, on a million triangles
        _view("stereo", triangles=995072, width=1080, height=1200, sampling="barrel", msaa=8, eyes=2),
        # an offline-quality still: the highest antialiasing rate, with the rotated-grid pattern
        _view("still", triangles=500000, width=1280, height=720, msaa=32, rotated_grid=True),
        # depth of field
        _view("lens", triangles=57344, width=640, height=480, msaa=8, lens=0.02),
        # textured materials
        _view("textured", triangles=57344, width=960, height=540, msaa=4, textures=8),
        # a simulation's frame: a tenth of the vertices move on the device, the BVH is refit, then a
        # frame of it
        _view("animated", triangles=995072, width=1280, height=720, msaa=2, animate=True),
        # the foveated headset: both eyes' polar sets, resolved with the temporal filter
        {"name": "foveated", "kind": "foveated", "triangles": 995072, "width": 1440, "height": 1600, "msaa": 16,
         "acuity": 1.0, "eyes": 2},
        # a sample set drawn anew for the gaze of this frame: set it, build its hierarchy, render
        {"name": "gaze_samples", "kind": "samples", "triangles": 300000, "width": 1440, "height": 1600,
         "samples": 300007, "msaa": 4},
        # many views of uneven size over several resident scenes as one frame
        {"name": "views", "kind": "views", "triangles": 300000, "scenes": 3, "views": 12},
        # a burst of render requests to the server, a stereo pair of the latency class among them
        {"name": "served", "kind": "served", "triangles": 100000, "scenes": 2, "requests": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view", "view", "view", "view", "pick", "foveated", "samples", "views", "served"])
    triangles = _log(rng, 20000, 1000000)
    if kind == "pick":
        return {"kind": kind, "triangles": _log(rng, 20000, 60000), "width": _log(rng, 64, 320),
                "height": _log(rng, 64, 240)}
    if kind == "foveated":
        return {"kind": kind, "triangles": triangles, "width": _log(rng, 480, 1440), "height": _log(rng, 480, 1600),
                "msaa": rng.choice([1, 4, 8, 16]), "acuity": round(rng.uniform(1.0, 3.0), 2), "eyes": rng.choice([1, 2])}
    if kind == "samples":
        samples = _log(rng, 20000, 600000)
        return {"kind": kind, "triangles": max(20000, min(triangles, 6 * samples)), "width": _log(rng, 480, 1440),
                "height": _log(rng, 480, 1600), "samples": samples, "msaa": rng.choice([1, 4, 8])}
    if kind == "views":
        return {"kind": kind, "triangles": _log(rng, 20000, 300000), "scenes": rng.choice([1, 2, 3]),
                "views": rng.randint(3, 16)}
    if kind == "served":
        return {"kind": kind, "triangles": _log(rng, 20000, 200000), "scenes": rng.choice([1, 2]),
                "requests": rng.randint(6, 24)}
    width, height, eyes = _log(rng, 96, 1920), _log(rng, 96, 1200), rng.choice([1, 1, 2])
    msaa = rng.choice([1, 2, 4, 8, 16, 32])
    while msaa > 1 and width * height * eyes * msaa > 20000000:  # at most the stereo frame's subsamples
        msaa //= 2
    option = rng.choice(["", "", "lens", "textures", "strict", "animate", "rotated_grid"])
    # the detail of an asset follows the view that it is made for
    triangles = max(20000, min(triangles, 6 * width * height))
    if option in ("lens", "textures"):
        triangles = _log(rng, 20000, 120000)
        msaa = min(msaa, 8)
    return _view(None, triangles=triangles, width=width, height=height, sampling=rng.choice(["grid", "barrel", "foveated"]),
                 msaa=msaa, eyes=eyes, lens=0.02 if option == "lens" else 0.0, textures=8 if option == "textures" else 0,
                 strict=option == "strict", animate=option == "animate", rotated_grid=option == "rotated_grid",
                 host_image=rng.random() < 0.25)


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=8)
def _scene(triangles, textures=0):
    """The asset of this size, with its topology (built once, as an asset pipeline does)."""
    if triangles == 995072:
        sc = scenes.scene_c2()
    elif triangles == 57344:
        sc = scenes.scene_c1()
    else:
        sc = scenes.scene_sized(triangles, seed=triangles)
    hv.generate_topology(sc)
    return scenes.with_textures(sc, textures) if textures else sc


@functools.lru_cache(maxsize=1)
def _stream():
    """The program's render stream."""
    s = torch.cuda.Stream()
    return s, ctypes.c_void_p(s.cuda_stream)


def _samples(kind, width, height, rng):
    if kind == "barrel":
        return scenes.barrel_samples(width, height), scenes.viewport_for(width, height)
    if kind == "foveated":
        gaze = (rng.uniform(-10, 10), rng.uniform(-10, 10))
        return (scenes.foveated_samples(max(256, width * height // 2), width, height, 100.0, gaze),
                scenes.viewport_fov(width, height, 100.0))
    return scenes.grid_samples(width, height), scenes.viewport_for(width, height)


def _pose(rng):
    """Eye and target over the terrain: near the ground to well above it, looking across the scene."""
    a, r = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(7.0, 13.0)
    return ((r * math.sin(a), rng.uniform(1.5, 5.0), r * math.cos(a)), (rng.uniform(-3.0, 3.0), 0.0, rng.uniform(-3.0, 3.0)))


def _raycaster(triangles, textures=0, **kw):
    sc = _scene(triangles, textures)
    rc = hv.Raycaster(**kw)
    for i in range(textures):
        rc.create_texture(scenes.texture_rgba8(256 + 64 * i, 256, seed=i))
    model = rc.create_model(sc)
    for light in sc.lights:
        rc.create_light(light)
    return rc, model


def _image(height, width):
    return torch.zeros((height, width), dtype=torch.int32, device=DEVICE)


def _first_frame(rc, handle):
    rc.render(stream=handle)
    rc.synchronize()


def prepare(case, seed):
    torch.cuda.set_device(0)
    rng = random.Random(int(seed))
    state = {"kind": case["kind"], "stream": _stream()[1]}
    return {"view": _prepare_view, "pick": _prepare_pick, "foveated": _prepare_foveated, "samples": _prepare_samples,
            "views": _prepare_views, "served": _prepare_served}[case["kind"]](case, rng, state)


def _add_camera(rc, smp, viewport, width, height, msaa, device=True):
    cam = rc.create_camera(viewport)
    img = _image(height, width) if device else None
    cam.set_render_target(width, height, device_ptr=img.data_ptr() if device else None)
    cam.set_samples(smp)
    cam.set_msaa(msaa)
    return cam, img if device else cam.image


def _prepare_view(case, rng, state):
    w, h = case["width"], case["height"]
    rc, model = _raycaster(case["triangles"], case["textures"],
                           fp_mode=hv.HVVR_FP_STRICT if case["strict"] else hv.HVVR_FP_FMA)
    smp, viewport = _samples(case["sampling"], w, h, rng)
    eye, target = _pose(rng)
    xfs = scenes.stereo_eyes(IPD, eye, target) if case["eyes"] == 2 else [scenes.camera_transform(eye, target)]
    cams, images = [], []
    for _ in xfs:
        cam, img = _add_camera(rc, smp, viewport, w, h, case["msaa"], not case["host_image"])
        if case["lens"]:
            cam.set_lens(case["lens"], 8.0)
        if case["rotated_grid"]:
            cam.set_msaa_pattern(hv.HVVR_MSAA_ROTATED_GRID)
        cams.append(cam)
        images.append(img)
    for cam, xf in zip(cams, xfs):
        cam.set_camera_to_world(xf)
    _first_frame(rc, state["stream"])
    if case["animate"]:
        # this frame's displaced vertices, as the program's simulation left them on the device
        anim = workloads.Animator(torch, model, _scene(case["triangles"]))
        anim.buf[:, 1] = anim.base[:, 1] + workloads.ANIM_AMPLITUDE * torch.sin(anim.phase + rng.uniform(0.0, 6.0))
        torch.cuda.synchronize()
        state.update(model=model, anim=anim)
    state.update(rc=rc, cams=cams, xfs=xfs, images=images)
    return state


def _prepare_pick(case, rng, state):
    w, h = case["width"], case["height"]
    rc, _ = _raycaster(case["triangles"])
    smp, viewport = _samples("grid", w, h, rng)
    cam, img = _add_camera(rc, smp, viewport, w, h, 1)
    cam.set_capture(hv.HVVR_CAPTURE_HITS)
    xf = scenes.camera_transform(*_pose(rng))
    cam.set_camera_to_world(xf)
    _first_frame(rc, state["stream"])
    state.update(rc=rc, cam=cam, xf=xf, image=img, remap=cam.sample_remap().reshape(h, w))
    return state


def _foveated_spec(case):
    # 50 degrees of eccentricity; a foveal acuity of 1 arc minute is the benchmark's pattern, a
    # coarser one has fewer rings and samples
    acuity = case["acuity"] / 60.0
    return hv.foveated_spec(0.5, 50.0, acuity / 5.0, acuity, mode=_abi.HVVR_MODE_FOVEATED_POLAR)


def _prepare_foveated(case, rng, state):
    w, h = case["width"], case["height"]
    rc, _ = _raycaster(case["triangles"], spec=_foveated_spec(case))
    smp, viewport = scenes.grid_samples(w, h), scenes.viewport_fov(w, h, 100.0)
    eye, target = _pose(rng)
    xfs = scenes.stereo_eyes(IPD, eye, target) if case["eyes"] == 2 else [scenes.camera_transform(eye, target)]
    a, b = math.radians(rng.uniform(-10, 10)), math.radians(rng.uniform(-8, 8))
    gaze = (math.sin(a) * math.cos(b), math.sin(b), -math.cos(a) * math.cos(b))
    cams, images = [], []
    for xf in xfs:
        cam, img = _add_camera(rc, smp, viewport, w, h, case["msaa"])
        cam.set_camera_to_world(xf)
        cam.set_eye_dir(gaze)
        cams.append(cam)
        images.append(img)
    _first_frame(rc, state["stream"])
    state.update(rc=rc, cams=cams, xfs=xfs, gaze=gaze, images=images)
    return state


def _prepare_samples(case, rng, state):
    w, h = case["width"], case["height"]
    rc, _ = _raycaster(case["triangles"])
    gaze = (rng.uniform(-10, 10), rng.uniform(-10, 10))
    smp = scenes.foveated_samples(case["samples"], w, h, 100.0, gaze, jitter_seed=rng.randrange(1 << 30))
    cam, img = _add_camera(rc, smp, scenes.viewport_fov(w, h, 100.0), w, h, case["msaa"])
    xf = scenes.camera_transform(*_pose(rng))
    cam.set_camera_to_world(xf)
    _first_frame(rc, state["stream"])
    state.update(rc=rc, cam=cam, xf=xf, image=img, samples=smp)
    return state


_VIEW_KINDS = (("grid", 256, 256, 4), ("grid", 640, 480, 1), ("barrel", 540, 600, 8), ("foveated", 720, 800, 16))


def _prepare_views(case, rng, state):
    rcs = [_raycaster(max(20000, case["triangles"] >> (2 * i)))[0] for i in range(case["scenes"])]
    cams, images, xfs = [], [], []
    for i in range(case["views"]):
        kind, w, h, msaa = _VIEW_KINDS[i % len(_VIEW_KINDS)]
        w, h = w + i % 3, h - i % 5
        smp, viewport = _samples(kind, w, h, rng)
        cam, img = _add_camera(rcs[i % len(rcs)], smp, viewport, w, h, msaa)
        xfs.append(scenes.camera_transform(*_pose(rng)))
        cam.set_camera_to_world(xfs[-1])
        cams.append(cam)
        images.append(img)
    batch = hv.Batch(cameras=cams)
    batch.render(stream=state["stream"])
    batch.synchronize()
    state.update(rcs=rcs, batch=batch, cams=cams, xfs=xfs, images=images)
    return state


def _prepare_served(case, rng, state):
    rcs = [_raycaster(max(20000, case["triangles"] >> (2 * i)))[0] for i in range(case["scenes"])]
    server = hv.Server(rcs, hv.server_config(slots=2, slot_list_capacity=64 << 20))
    views = []
    for s in range(case["scenes"]):
        for kind, w, h, msaa in _VIEW_KINDS:
            smp, viewport = _samples(kind, w, h, rng)
            views.append((server.add_view(s, viewport, smp, w, h), w, h, msaa))
    for vid, _, _, _ in views:
        server.prewarm(vid, 4)
    items, images = [], []
    for i in range(case["requests"]):
        vid, w, h, msaa = views[i % len(views)]
        images.append(_image(h, w))
        items.append((vid, msaa, scenes.camera_transform(*_pose(rng)), None, images[-1].data_ptr(), i))
    vid, w, h, msaa = views[2]  # the stereo pair
    pair = []
    for k, xf in enumerate(scenes.stereo_eyes(IPD, *_pose(rng))):
        images.append(_image(h, w))
        pair.append((vid, msaa, xf, None, images[-1].data_ptr(), 1000 + k))
    torch.cuda.synchronize()
    state.update(rcs=rcs, server=server, items=items, pair=pair, images=images)
    _serve(state)
    return state


# ---------------------------------------------------------------- one pass
def _serve(state):
    server, pair = state["server"], state["pair"]
    for vid, msaa, xf, out, ptr, tag in state["items"]:
        server.submit(vid, msaa, xf, output=out, device_ptr=ptr, tag=tag)
    server.submit_group(pair, priority=1)
    left = len(state["items"]) + len(pair)
    while left:
        for done in server.poll(wait_ms=50.0):
            if done.status != 0:
                raise RuntimeError("request %d: status %d" % (done.tag, done.status))
            left -= 1


def run(state):
    kind, stream = state["kind"], state["stream"]
    if kind == "served":
        _serve(state)
        return state["images"]
    if kind == "views":
        for cam, xf in zip(state["cams"], state["xfs"]):
            cam.set_camera_to_world(xf)
        state["batch"].render(stream=stream)
        return state["images"]
    rc = state["rc"]
    if kind == "pick":
        cam = state["cam"]
        cam.set_camera_to_world(state["xf"])
        rc.render(stream=stream)
        rc.synchronize()
        ids, depth = cam.hits()
        at = state["remap"]
        # disparity, as a compositor stores it: 0 where nothing is hit
        return {"image": state["image"], "triangle": ids[at, 0], "disparity": np.float32(1.0) / depth[at, 0]}
    if kind == "samples":
        cam = state["cam"]
        cam.set_samples(state["samples"])
        cam.set_camera_to_world(state["xf"])
        rc.render(stream=stream)
        return state["image"]
    for cam, xf in zip(state["cams"], state["xfs"]):
        cam.set_camera_to_world(xf)
        if kind == "foveated":
            cam.set_eye_dir(state["gaze"])
    if "anim" in state:
        anim = state["anim"]
        state["model"].update_vertices_device(anim.first, anim.count, anim.buf.data_ptr(), stream)
    rc.render(stream=stream)
    return state["images"]


# ---------------------------------------------------------------- what a pass cannot do without
def _frame_work(samples, pixels, msaa, triangles):
    """Beams (36 bytes a sample) and the scene's triangles and leaf bounds in, the image out; a
    ray-triangle test (16 flops) per subsample, and the test's setup and the shading per sample."""
    return {"bytes": 36.0 * samples + 4.0 * pixels + (36.0 + 12.0) * triangles,
            "flops": float(samples) * (16.0 * msaa + 72.0 + 400.0)}


def _plus(*works):
    return {k: sum(w[k] for w in works) for k in ("bytes", "flops")}


def work(case):
    kind, tris = case["kind"], case["triangles"]
    if kind in ("views", "served"):
        n = case["views"] if kind == "views" else case["requests"] + 2
        parts = [_frame_work(w * h // (2 if k == "foveated" else 1), w * h, msaa, 0)
                 for k, w, h, msaa in (_VIEW_KINDS[i % len(_VIEW_KINDS)] for i in range(n))]
        return _plus({"bytes": 48.0 * sum(max(20000, tris >> (2 * i)) for i in range(case["scenes"])), "flops": 0.0}, *parts)
    pixels = case["width"] * case["height"]
    if kind == "pick":
        return _plus(_frame_work(pixels, pixels, 1, tris), {"bytes": 8.0 * pixels, "flops": 0.0})
    if kind == "samples":
        return _plus(_frame_work(case["samples"], pixels, case["msaa"], tris), {"bytes": 28.0 * case["samples"], "flops": 0.0})
    if kind == "foveated":
        n = 1173612 / case["acuity"] ** 2
        eyes = [_frame_work(n, pixels, case["msaa"], 0)] * case["eyes"]
        # the resolve reads the history and the polar texels and writes the image and the history
        return _plus({"bytes": 48.0 * tris, "flops": 0.0}, *eyes, {"bytes": case["eyes"] * (8.0 * pixels + 24.0 * n), "flops": 0.0})
    n = pixels // 2 if case["sampling"] == "foveated" else pixels
    parts = [_frame_work(n, pixels, case["msaa"], 0)] * case["eyes"]
    if case["animate"]:
        # the displaced vertices in and out, and every triangle, vertex and node written anew
        verts = 1.8 * tris
        parts.append({"bytes": 0.1 * verts * 64.0 + 64.0 * verts + 112.0 * tris + 30.0 * tris, "flops": 60.0 * verts})
    return _plus({"bytes": 48.0 * tris, "flops": 0.0}, *parts)


def exact(case, seed):
    """The depth query in 64 bits, by testing every ray against every triangle. (The renderer's tile
    tests leave out a few grazing hits at tile borders, as the reference's do, so a few pixels differ
    by more than rounding.) The other outputs are 8-bit images and triangle indices, which have no
    value in 64 bits."""
    if case["kind"] != "pick":
        return None
    torch.cuda.set_device(0)
    rng = random.Random(int(seed))
    w, h = case["width"], case["height"]
    sc = _scene(case["triangles"])
    smp, viewport = _samples("grid", w, h, rng)
    eye, target = _pose(rng)
    f64 = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=DEVICE)  # noqa: E731
    # rays: the sample's position and ellipse on the viewport, the one subsample's offset, rotated to world space
    pos, minor, major = (smp[k].astype(np.float64) for k in ("position", "minor", "major"))
    lx, ly, ux, uy = viewport.lower.x, viewport.lower.y, viewport.upper.x, viewport.upper.y
    scale = np.array([ux - lx, ly - uy])
    ext = math.sqrt(0.5)
    mn = minor * ext
    mj = np.stack([-mn[:, 1], mn[:, 0]], 1) * (major * ext / np.hypot(minor[:, 0], minor[:, 1]))[:, None]
    ax, ay = math.cos(0.5 * 6.28) * ext, math.sin(0.5 * 6.28) * ext
    cam = np.empty((len(smp), 3))
    cam[:, :2] = (pos + ax * mj + ay * mn) * scale + np.array([lx, uy])
    cam[:, 2] = -1.0
    x, y, z, q = scenes.look_at_quaternion(eye, target)
    rot = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * q), 2 * (x * z + y * q)],
                    [2 * (x * y + z * q), 1 - 2 * (x * x + z * z), 2 * (y * z - x * q)],
                    [2 * (x * z - y * q), 2 * (y * z + x * q), 1 - 2 * (x * x + y * y)]])
    rays = f64(cam @ rot.T)
    p = f64(sc.verts["pos"])[torch.as_tensor(sc.tri_shade["indices"].astype(np.int64), device=DEVICE)]
    v0, e0, e1 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    rel = f64(np.array([float(np.float32(t)) for t in eye])) - v0
    n = torch.linalg.cross(e0, e1)
    t = (rel * n).sum(1)
    front = t >= 0  # back faces are not seen
    n, rel, e0, e1, t = n[front], rel[front], e0[front], e1[front], t[front]
    gv, gw = torch.linalg.cross(rel, e1), -torch.linalg.cross(rel, e0)
    disparity = torch.empty(len(rays), dtype=torch.float64, device=DEVICE)
    for i in range(0, len(rays), 512):
        d = -rays[i:i + 512]
        denom, v, k = d @ n.T, d @ gv.T, d @ gw.T
        hit = (v >= 0) & (k >= 0) & (denom - v - k >= 0) & (denom > 0)
        disparity[i:i + 512] = 1.0 / torch.where(hit, t / denom, math.inf).amin(1)
    return {"image": None, "triangle": None, "disparity": disparity.cpu().numpy().reshape(h, w)}
