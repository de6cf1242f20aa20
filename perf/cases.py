"""The performance cases of the renderer: the calls a user's program makes, over the range of
sizes and options it makes them with.

Each case is a dict of plain values; "kind" says which public entry points one pass takes:

  frame   Context: one camera, one synchronous frame, the RGBA8 image read back to pinned memory
  stream  Context: a camera path, every frame enqueued over the frame lanes and read back
  open    Context: a 3DGS PLY file loaded, drawn once and read back (time to the first image)
  batch   Batch: many views of resident scenes in one call, the images left on the device
  serve   Server: a burst of requests submitted, waited for, read and released
  sort    the standalone stable sort, on host arrays or on the caller's device arrays

Scenes are synthetic 3DGS captures with the parameter distributions of gsplat_scenes (log-scales,
opacity logits, DC and SH coefficients, a Gaussian mixture of positions; "box" adds the uniform
volume of the large capture, seen from inside). Everything is made from the seed.
"""

import ctypes
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gsplat-rs_b200"))
import gsplat_ffi as ffi  # noqa: E402
import gsplat_scenes  # noqa: E402

LANES = 8  # frame lanes of the streaming program


def _frame(name, splats, degree, width, height, blend="fp32", scene="gmm", packed=False, tile=16):
    return {"name": name, "kind": "frame", "splats": splats, "degree": degree, "width": width,
            "height": height, "blend": blend, "scene": scene, "packed": packed, "tile": tile}


def listed():
    return [
        # The smallest frame in use: a preview or a thumbnail of a small object.
        _frame("frame_16k_256", 16384, 0, 256, 256),
        # The ordinary frame: a captured scene at full HD, both blend modes.
        _frame("frame_279k_1080p", 279199, 3, 1920, 1080),
        _frame("frame_279k_1080p_unorm8", 279199, 3, 1920, 1080, blend="unorm8"),
        # The packed resident format in an odd-sized window.
        _frame("frame_1m_packed_odd", 1000003, 3, 1279, 717, packed=True),
        # The largest frame: the camera inside a 3M-splat capture, 4K.
        _frame("frame_3m_4k", 3000000, 3, 3840, 2160, scene="box"),
        # An interactive viewer or a video export: consecutive frames of a camera path.
        {"name": "stream_279k_1080p", "kind": "stream", "splats": 279199, "degree": 3,
         "width": 1920, "height": 1080, "frames": 24, "scene": "gmm"},
        # Opening a file: 3DGS PLY to the first image.
        {"name": "open_279k", "kind": "open", "splats": 279199, "degree": 3, "width": 1280,
         "height": 720, "scene": "gmm"},
        # Many small views of one small object (a turntable, a dataset's thumbnails).
        {"name": "batch_64_thumbs", "kind": "batch", "splats": "16384", "degree": 0, "views": 64,
         "width": 256, "height": 256, "mixed": False},
        # Many views of scenes of uneven sizes at mixed resolutions.
        {"name": "batch_48_mixed", "kind": "batch", "splats": "50000,279199,1000000",
         "degree": 3, "views": 48, "width": 1920, "height": 1080, "mixed": True},
        # A burst of requests to the render server.
        {"name": "serve_32_mixed", "kind": "serve", "splats": "50000,279199", "degree": 2,
         "views": 32, "width": 1280, "height": 720, "mixed": True},
        # The reference's sort microbenchmark length, on host arrays.
        {"name": "sort_200k_host", "kind": "sort", "items": 200000, "where": "host"},
        # The allocation-free sort of a host that owns its device memory.
        {"name": "sort_1m_device", "kind": "sort", "items": 1000003, "where": "device"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "stream", "batch", "batch", "serve",
                       "open", "sort"])
    if kind == "sort":
        where = rng.choice(["host", "device"])
        return {"kind": kind, "where": where,
                "items": _log_int(rng, 5000, 1 << 20 if where == "device" else 4 << 20)}
    width = _log_int(rng, 240, 2560)
    height = max(128, min(1600, int(width * rng.uniform(0.4, 1.2))))
    degree = rng.randint(0, 4)
    if kind == "frame":
        blend = rng.choice(["fp32", "fp32", "fp32", "unorm8"])
        packed = degree < 4 and rng.random() < 0.2
        # the parity blend has no early exit: its cost grows with every splat behind a pixel
        splats = _log_int(rng, 16000, 600_000 if blend == "unorm8" else 2_500_000)
        # close splats of the box cover hundreds of tiles, four times as many at tile size 8
        scene = rng.choice(["gmm", "gmm", "box"]) if blend == "fp32" else "gmm"
        return {"kind": kind, "splats": splats, "degree": degree, "width": width,
                "height": height, "blend": blend, "packed": packed, "scene": scene,
                "tile": rng.choice([16, 16, 16, 8]) if scene == "gmm" else 16}
    if kind == "stream":
        return {"kind": kind, "splats": _log_int(rng, 16000, 700_000), "degree": degree,
                "width": min(width, 1920), "height": min(height, 1080),
                "frames": rng.randint(4, 24), "scene": "gmm"}
    if kind == "open":
        return {"kind": kind, "splats": _log_int(rng, 16000, 500_000), "degree": min(degree, 3),
                "width": width, "height": height, "scene": "gmm"}
    scenes = ",".join(str(_log_int(rng, 16000, 700_000)) for _ in range(rng.randint(1, 3)))
    return {"kind": kind, "splats": scenes, "degree": degree,
            "views": rng.randint(4, 48 if kind == "batch" else 32),
            "width": min(width, 1280), "height": min(height, 720), "mixed": rng.random() < 0.5}


# ---- inputs ------------------------------------------------------------------

def _scene(splats, degree, shape, seed):
    """A SceneBuffers-shaped dict, drawn on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(mu, sd, *shape):
        return torch.randn(*shape, generator=g, device="cuda") * sd + mu

    n = splats
    if shape == "box":
        pos = torch.rand(n, 3, generator=g, device="cuda") * 10.0 - 5.0
        pos[n // 2:] = normal(0.0, 0.7, n - n // 2, 3)
        log_scale, scale_sd, logit, logit_sd = -3.5, 0.8, 1.0, 1.0
    else:
        sigma = torch.tensor([0.3, 0.6, 0.9, 1.2], device="cuda")
        centre = normal(0.0, 0.5, 4, 3)
        k = torch.randint(0, 4, (n,), generator=g, device="cuda")
        pos = centre[k] + normal(0.0, 1.0, n, 3) * sigma[k, None]
        log_scale, scale_sd, logit, logit_sd = -4.5, 0.7, 0.5, 1.5
    quat = normal(0.0, 1.0, n, 4)
    scene = {
        "positions": pos,
        "opacity": normal(logit, logit_sd, n),
        "scale_xyz": normal(log_scale, scale_sd, n, 3),
        "rotation_xyzw": quat / quat.norm(dim=1, keepdim=True),
        "color_dc": normal(0.0, 0.5, n, 3),
    }
    if degree > 0:
        scene["sh_rest"] = normal(0.0, 0.1, n, gsplat_scenes.sh_rest_width(degree))
    scene = {k: v.cpu().numpy() for k, v in scene.items()}
    scene.setdefault("sh_rest", None)
    scene["sh_degree"] = degree
    return scene


def _cameras(count, shape, seed, path=False):
    """Orbit cameras around the scene, cameras inside the box, or a smooth orbit path."""
    rng = np.random.default_rng(seed)
    if shape == "box":
        return [ffi.GsplatCamera.from_dict(gsplat_scenes.camera(
            rng.uniform(-0.6, 0.6, 3) + np.array([0.0, 0.0, -3.0]), (0.0, 0.0, 0.0), 60.0))
            for _ in range(count)]
    if path:
        yaw, pitch = rng.uniform(0.0, 2 * math.pi), rng.uniform(-0.3, 0.3)
        return [ffi.GsplatCamera.from_dict(gsplat_scenes.camera(
            (4.0 * math.sin(a) * math.cos(pitch), 4.0 * math.sin(pitch),
             -4.0 * math.cos(a) * math.cos(pitch)), (0.0, 0.0, 0.0), 45.0))
            for a in (yaw + 0.02 * k for k in range(count))]
    return [ffi.GsplatCamera.from_dict(gsplat_scenes.orbit_camera(rng, (3.5, 5.0), (40.0, 55.0)))
            for _ in range(count)]


def _pinned(nbytes):
    return torch.empty(nbytes, dtype=torch.uint8, pin_memory=True).numpy()


def _view_sizes(case):
    """Image size of each view: the case's, or in turn it, two thirds and half of it."""
    w, h = case["width"], case["height"]
    sizes = [(w, h), (max(64, 2 * w // 3), max(64, 2 * h // 3)), (max(64, w // 2), max(64, h // 2))]
    return [sizes[k % 3] if case["mixed"] else sizes[0] for k in range(case["views"])]


def _scene_sizes(case):
    return [int(s) for s in str(case["splats"]).split(",")]


def _views(case, seed):
    count = len(_scene_sizes(case))
    cams = _cameras(case["views"], "gmm", seed + 2)
    return [(k * count // case["views"], cam, w, h)
            for k, (cam, (w, h)) in enumerate(zip(cams, _view_sizes(case)))]


def _context(case):
    ctx = ffi.Context(case["width"], case["height"])
    if case.get("tile", 16) != 16:
        ctx.set_tile_size(case["tile"])
    if case.get("blend") == "unorm8":
        ctx.set_blend_mode(ffi.BLEND_UNORM8)
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "sort":
        # depth keys as the frame has them: the bits of positive floats, ties among them
        g = torch.Generator(device="cuda").manual_seed(seed)
        depth = torch.rand(case["items"], generator=g, device="cuda") * 8.0 + 0.01
        depth = (depth * 65536.0).round() / 65536.0
        keys = depth.view(torch.int32)
        order = torch.arange(case["items"], dtype=torch.int32, device="cuda")
        state["where"] = case["where"]
        if case["where"] == "host":
            state["keys"] = keys.cpu().numpy().view(np.uint32)
            state["order"] = order.cpu().numpy().view(np.uint32)
        else:
            state["keys"], state["order"] = keys, order
            state["values"] = torch.empty_like(order)
        return state
    if kind in ("frame", "stream", "open"):
        ctx = state["ctx"] = _context(case)
        scene = _scene(case["splats"], case["degree"], case["scene"], seed)
        nbytes = case["width"] * case["height"] * 4
        if kind == "open":
            state["dir"] = tempfile.TemporaryDirectory(prefix="gsplat_perf_")
            state["path"] = os.path.join(state["dir"].name, "scene.ply")
            gsplat_scenes.write_ply(state["path"], scene)
        elif case.get("packed"):
            ctx.load_scene_packed(scene)
        else:
            ctx.load_scene(scene)
        if kind == "stream":
            state["cams"] = _cameras(case["frames"], case["scene"], seed + 1, path=True)
            state["outs"] = [_pinned(nbytes) for _ in range(case["frames"])]
            # a streaming program draws its first frame synchronously: enqueued frames keep the
            # tile-pair capacity it leaves
            ctx.set_camera(state["cams"][0])
            ctx.render_frame()
            ctx.set_frame_lanes(LANES)
        else:
            state["cam"] = _cameras(1, case["scene"], seed + 1)[0]
            state["out"] = _pinned(nbytes)
        return state
    scenes = [_scene(n, case["degree"], "gmm", seed + 10 * k)
              for k, n in enumerate(_scene_sizes(case))]
    views = _views(case, seed)
    if kind == "batch":
        state["batch"] = ffi.Batch()
        for s in scenes:
            state["batch"].add_scene(s)
        state["views"] = ffi.Batch.make_views(views)
        state["arena"] = None
    else:
        state["server"] = ffi.Server(max_views=64, result_pool_mib=256)
        for s in scenes:
            state["server"].add_scene(s)
        state["views"] = views
        state["outs"] = [np.empty(w * h * 4, np.uint8) for _, _, w, h in views]
    return state


# ---- one pass ----------------------------------------------------------------

class _DeviceImage:
    """An RGBA8 image in a batch's device memory, for torch.as_tensor; keeps the batch alive."""

    def __init__(self, batch, ptr, width, height):
        self.batch = batch
        self.__cuda_array_interface__ = {"shape": (height, width, 4), "typestr": "|u1",
                                         "data": (ptr, False), "version": 3}


def _batch_images(state):
    """The batch's images as torch tensors, wrapped again when the images have moved."""
    batch = state["batch"]
    arena = batch.image_device(0)[0]
    if arena != state["arena"]:
        state["arena"] = arena
        state["images"] = [
            torch.as_tensor(_DeviceImage(batch, batch.image_device(k)[0], w, h), device="cuda")
            for k, (w, h) in enumerate(batch.sizes)]
    return state["images"]


def run(state):
    kind = state["kind"]
    if kind == "frame":
        ctx = state["ctx"]
        ctx.set_camera(state["cam"])
        ctx.render_frame()
        return ctx.readback_rgba8(state["out"])
    if kind == "stream":
        ctx = state["ctx"]
        for cam, out in zip(state["cams"], state["outs"]):
            ctx.set_camera(cam)
            ctx.render_frame_async()
            ctx.readback_rgba8_async(out)
        ctx.sync()
        return state["outs"]
    if kind == "open":
        ctx = state["ctx"]
        ctx.load_scene_path(state["path"])
        ctx.set_camera(state["cam"])
        ctx.render_frame()
        return ctx.readback_rgba8(state["out"])
    if kind == "batch":
        state["batch"].render(state["views"])
        return _batch_images(state)
    if kind == "serve":
        server = state["server"]
        requests = [server.submit(*view) for view in state["views"]]
        images = []
        for rid, out in zip(requests, state["outs"]):
            server.wait(rid)
            images.append(server.read_rgba8(rid, out))
            server.release(rid)
        return images
    if state["where"] == "host":
        return ffi.sort_values_by_keys(state["keys"], state["order"])
    keys, values = state["keys"], state["values"]
    values.copy_(state["order"])
    ffi.check(ffi.lib().gsplat_cuda_sort_values_by_keys_noalloc(
        keys.data_ptr(), values.data_ptr(), keys.numel(),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return values


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """Bytes: every scene a pass draws read once (a file too, for open) and every image written
    once; a sort reads keys and values and writes the values. Operations: the vertex stage of
    every view's splats (projection, and two per SH coefficient and channel); what blending takes
    depends on the camera and is not counted."""
    if case["kind"] == "sort":
        return {"bytes": 12 * case["items"], "flops": 0}
    coeffs = (case["degree"] + 1) ** 2
    per_splat = 4 * (11 + 3 * coeffs)
    if case.get("packed"):
        per_splat = 20 + (48 if case["degree"] else 0)
    ops = 200 + 6 * coeffs
    if case["kind"] in ("frame", "open", "stream"):
        frames = case.get("frames", 1)
        file_bytes = per_splat * case["splats"] if case["kind"] == "open" else 0
        return {"bytes": file_bytes + per_splat * case["splats"]
                + 4 * frames * case["width"] * case["height"],
                "flops": ops * frames * case["splats"]}
    sizes = _scene_sizes(case)
    drawn = [sizes[k * len(sizes) // case["views"]] for k in range(case["views"])]
    pixels = sum(w * h for w, h in _view_sizes(case))
    return {"bytes": per_splat * sum(sizes) + 4 * pixels, "flops": ops * sum(drawn)}


def exact(case, seed):
    """The sorts' order by numpy's stable sort. Images are bytes: they are compared as they are."""
    if case["kind"] != "sort":
        return None
    state = prepare(case, seed)
    keys, order = state["keys"], state["order"]
    if case["where"] == "device":
        keys, order = keys.cpu().numpy().view(np.uint32), order.cpu().numpy()
    return order[np.argsort(-keys.astype(np.int64), kind="stable")]
