"""The calls whose speed is tracked: what users of the renderer have it do, through its public
entry points, over the range of sizes and options that they use.

A case is a dict with an "op" and the op's sizes:

  render   one RayRenderer.render() of a scene that is already set, and its HDR image
  frame    RayRenderer.set_scene() with new geometry, render() and the HDR image: an animation
           frame or an edit in a viewer
  batch    a mix of jobs through RenderServer: submit all, wait, read every image
  closest  RayRenderer.trace_closest() on a batch of rays
  any      RayRenderer.trace_any() on a batch of shadow rays
  atrous   rg_denoise_atrous_noalloc on device buffers
  denoise  Denoiser.apply() on host images (the learned denoiser)
  train    Denoiser.train() steps, and the weights after them
"""
import ctypes
import math
import os
import random

import numpy as np
import torch

from __graft_entry__ import load_package

rg = load_package()


def listed():
    return [
        # a probe of a mid-size scene with a few rays (picking, light baking tests): latency
        {"name": "closest_1k", "op": "closest", "scene": "job", "tris": 20000, "emitters": 8, "rays": 1000},
        # an ambient-occlusion or visibility bake: a million shadow rays at once
        {"name": "any_1m", "op": "any", "scene": "job", "tris": 300000, "emitters": 16, "rays": 1 << 20},
        # the small standard render: the cube room, 256 x 256, 16 samples, depth 5
        {"name": "room_256", "op": "render", "scene": "room", "width": 256, "height": 256, "spp": 16, "depth": 5},
        # the standard benchmark: 4 x 1,003,520-triangle spheres, 1080p, 64 samples, depth 8
        {"name": "spheres_1080p", "op": "render", "scene": "spheres", "tris": 1003520, "width": 1920, "height": 1080,
         "spp": 64, "depth": 8},
        # spheres in fog, adaptive sampling in 16-sample passes, A-Trous denoiser: an image meant to be looked at
        {"name": "fog_adaptive", "op": "render", "scene": "fog", "tris": 250000, "width": 960, "height": 540,
         "spp": 64, "depth": 8, "adaptive": 16, "denoise": "atrous"},
        # an odd-sized still of a mid-size scene, few samples and the learned denoiser: a fast good image
        {"name": "still_learned", "op": "render", "scene": "job", "tris": 150000, "emitters": 24, "width": 517,
         "height": 333, "spp": 33, "depth": 10, "denoise": "learned"},
        # a viewer's preview after an edit: a small scene set anew, 4 samples
        {"name": "edit_20k", "op": "frame", "scene": "job", "tris": 20000, "emitters": 8, "width": 800, "height": 600,
         "spp": 4, "depth": 5},
        # an animation frame of the heavy scene: upload, BVH build, 1080p at 4 samples
        {"name": "frame_4m", "op": "frame", "scene": "spheres", "tris": 1003520, "width": 1920, "height": 1080,
         "spp": 4, "depth": 8},
        # the job server: a heterogeneous mix of small and mid-size images at once
        {"name": "batch_24", "op": "batch", "jobs": 24, "tris": 300000, "side": 384, "spp": 64},
        # the denoiser of an interactive preview, on the application's own device buffers
        {"name": "atrous_1024", "op": "atrous", "width": 1024, "height": 1024, "levels": 5},
        # the learned denoiser on images from elsewhere, 720p
        {"name": "denoise_720p", "op": "denoise", "width": 1280, "height": 720},
        # fitting the denoiser to a studio's own scenes: training steps on 64 x 64 pairs
        {"name": "train_16x64", "op": "train", "size": 64, "examples": 48, "batch": 16, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choices(["render", "frame", "batch", "closest", "any", "atrous", "denoise", "train"],
                     [32, 18, 8, 10, 10, 10, 6, 6])[0]
    if op in ("render", "frame"):
        scene = rng.choice(["room", "job", "job", "spheres", "fog"] if op == "render" else ["job", "job", "spheres"])
        width, height = _log(rng, 64, 1920), _log(rng, 64, 1080)
        # at most the largest listed render's samples, spread over their logarithm
        most = max(1.0, min(256.0, (40e6 if op == "render" else 8e6) / (width * height)))
        c = {"op": op, "scene": scene, "width": width, "height": height, "spp": _log(rng, 1, most),
             "depth": rng.randint(4, 10)}
        if scene == "job":
            c.update(tris=_log(rng, 1000, 1500000), emitters=rng.randint(1, 64))
        elif scene != "room":
            c.update(tris=_log(rng, 1000, 500000))
        if op == "render":
            c["denoise"] = rng.choice(["", "", "atrous", "learned"])
            if scene in ("job", "fog") and rng.random() < 0.3 and c["spp"] >= 8:
                c["adaptive"] = max(4, c["spp"] // 4)
        return c
    if op == "batch":
        return {"op": op, "jobs": rng.randint(4, 24), "tris": _log(rng, 2000, 300000), "side": rng.randint(64, 384),
                "spp": _log(rng, 4, 64)}
    if op in ("closest", "any"):
        return {"op": op, "scene": "job", "tris": _log(rng, 1000, 1000000), "emitters": rng.randint(1, 64),
                "rays": _log(rng, 100, 1500000)}
    if op == "atrous":
        return {"op": op, "width": _log(rng, 40, 1024), "height": _log(rng, 40, 1024), "levels": rng.randint(3, 6)}
    if op == "denoise":
        return {"op": op, "width": _log(rng, 64, 1920), "height": _log(rng, 64, 1080)}
    return {"op": op, "size": rng.choice([32, 48, 64, 96, 128]), "examples": 24, "batch": rng.randint(2, 16),
            "steps": rng.randint(2, 12)}


# ---------------------------------------------------------------- preparing --
_KIND = {"room": 1, "spheres": 2, "fog": 3, "job": 4}


def _scene(case, seed):
    kind = case["scene"]
    params = {"room": None, "spheres": [case.get("tris")], "fog": [case.get("tris")],
              "job": [case.get("tris"), case.get("emitters")]}[kind]
    return rg.Scene.builtin(_KIND[kind], 1 + seed % 100003, params)


def _in_pinned_memory(scene):
    """The scene with its triangle arrays in page-locked memory, as a program that sends a new
    scene for every frame keeps them."""
    d = scene.desc
    keep = [torch.from_numpy(np.array(a)).pin_memory() for a in scene.arrays()]
    out = rg.Scene.from_arrays(*(t.numpy() for t in keep), [d.mesh_object[i] for i in range(d.num_meshes)],
                               [d.objects[i] for i in range(d.num_objects)],
                               [d.materials[i] for i in range(d.num_materials)], d.camera)
    return out, keep


def _settings(case, seed):
    s = rg.RendererSettings(resolutionWidth=case["width"], resolutionHeight=case["height"], samples=case["spp"],
                            maxDepth=case["depth"], rrDepth=3, seed=1 + seed % 100003)
    if case.get("adaptive"):
        s.enableAdaptiveSampling, s.adaptiveBaseSamples = True, case["adaptive"]
    s.enableDenoise = bool(case.get("denoise"))
    return s


def _mix(case):
    """The sizes of a job mix: log-uniform triangles and sides, as many for every seed."""
    rng = random.Random(case["jobs"] * 7919 + case["side"])
    out = []
    for _ in range(case["jobs"]):
        side = _log(rng, min(48, case["side"]), case["side"])
        out.append({"scene": "job", "tris": _log(rng, 1000, case["tris"]), "emitters": rng.randint(1, 64), "side": side,
                    "spp": _log(rng, 1, case["spp"]), "depth": rng.randint(4, 10)})
    return out


def _rays(case, seed):
    """View-space rays of a job scene: half from the camera, half between points of the room."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    o = np.zeros((n, 3), np.float32)
    inner = np.arange(n) % 2 == 1
    lo, hi = np.array([-9.5, -4.5, -19.0], np.float32), np.array([9.5, 4.5, 0.0], np.float32)
    o[inner] = lo + (hi - lo) * rng.random((int(inner.sum()), 3), dtype=np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[~inner, 2] = -np.abs(d[~inner, 2]) - 1.0
    if case["op"] == "any":  # shadow rays run from point to point: the direction carries the distance
        return np.concatenate([o, d * rng.uniform(2.0, 12.0, (n, 1)).astype(np.float32)], 1), np.full(n, 0.99999, np.float32)
    return np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1), None


def _image(w, h, seed):
    """A noisy render and its guides: a few surfaces with normals that vary slowly, fireflies,
    a background; guides are values that half precision holds, as the renderer's are."""
    g = torch.Generator().manual_seed(seed)
    y, x = torch.meshgrid(torch.arange(h) / h, torch.arange(w) / w, indexing="ij")
    p = torch.rand(8, generator=g)
    part = (torch.sin(7 * x + 5 * p[0]) + torch.sin(6 * y + 5 * p[1]) > 0.3).float()
    n = torch.stack([torch.sin(3 * x + 4 * p[2]) * (0.3 + 0.6 * part), torch.cos(4 * y + 4 * p[3]) * 0.4,
                     0.4 + part], -1) + 0.02 * torch.randn((h, w, 3), generator=g)
    normal = (n / n.norm(dim=-1, keepdim=True) * 0.5 + 0.5).half().float()
    depth = (0.3 + 0.3 * x + 0.2 * part + 0.002 * torch.randn((h, w), generator=g)).clamp(0, 1).half().float()
    albedo = (0.2 + 0.6 * torch.rand(3, generator=g) * (0.5 + 0.5 * part[..., None]).expand(h, w, 3)).half().float()
    alpha = ((x - p[4]) ** 2 + (y - p[5]) ** 2 > 0.02).float()
    light = 0.2 + torch.exp(-8 * ((x - p[6]) ** 2 + (y - p[7]) ** 2))[..., None]
    noise = torch.empty((h, w, 3)).exponential_(generator=g)
    color = albedo * light * noise
    color[torch.rand((h, w), generator=g) < 0.001] = 9.0
    return color, normal, depth, albedo, alpha


def _atrous_call():
    f = rg.load_library().rg_denoise_atrous_noalloc
    f.restype = ctypes.c_int32
    f.argtypes = ([ctypes.c_int32] * 2 + [ctypes.c_void_p] * 5 + [ctypes.c_int32] + [ctypes.c_float] * 4
                  + [ctypes.c_void_p] * 2)
    return f


def prepare(case, seed):
    op = case["op"]
    if op in ("render", "frame"):
        scene, keep = _scene(case, seed), None
        r = rg.RayRenderer(_settings(case, seed))
        if op == "frame":
            scene, keep = _in_pinned_memory(scene)
        else:
            r.set_scene(scene)
        if case.get("denoise") == "learned":
            r.set_denoiser(rg.Denoiser.pretrained())
        return {"op": op, "renderer": r, "scene": scene, "keep": keep}
    if op == "batch":
        jobs = [(_scene(j, seed + 31 * k), j, 1 + seed % 100003 + k) for k, j in enumerate(_mix(case))]
        return {"op": op, "server": rg.RenderServer(rg.RendererSettings(rrDepth=3)), "jobs": jobs}
    if op in ("closest", "any"):
        scene = _scene(case, seed)
        r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=64, resolutionHeight=64, samples=1))
        r.set_scene(scene)
        rays, tmax = _rays(case, seed)
        return {"op": op, "renderer": r, "scene": scene, "rays": rays, "tmax": tmax}
    if op == "atrous":
        color, *guides = _image(case["width"], case["height"], seed)
        rgba = torch.cat([color, torch.ones_like(color[..., :1])], -1)
        bufs = [t.contiguous().cuda() for t in (rgba, *guides)]
        return {"op": op, "call": _atrous_call(), "size": (case["width"], case["height"]), "levels": case["levels"],
                "bufs": bufs, "out": torch.empty_like(bufs[0]), "stream": torch.cuda.current_stream().cuda_stream}
    if op == "denoise":
        color, normal, depth, albedo, _ = (t.numpy() for t in _image(case["width"], case["height"], seed))
        rgba = np.concatenate([color, np.ones_like(color[..., :1])], -1)
        return {"op": op, "denoiser": rg.Denoiser.pretrained(), "images": (rgba, normal, albedo, depth)}
    d = rg.Denoiser.pretrained()
    weights = d.params
    for k in range(case["examples"]):
        color, normal, depth, albedo, _ = (t.numpy() for t in _image(case["size"], case["size"], seed * 64 + k))
        d.add_example(color, normal, albedo, depth, color * 0.5 + 0.5 * color.mean((0, 1)), 8.0)
    return {"op": op, "denoiser": d, "weights": weights, "steps": case["steps"], "batch": case["batch"]}


# ------------------------------------------------------------------ running --
def run(state):
    op = state["op"]
    if op == "render":
        state["renderer"].render()
        return state["renderer"].get_hdr_result()
    if op == "frame":
        state["renderer"].set_scene(state["scene"])
        state["renderer"].render()
        return state["renderer"].get_hdr_result()
    if op == "batch":
        srv = state["server"]
        ids = [srv.submit(sc, j["side"], j["side"], j["spp"], max_depth=j["depth"], seed=s) for sc, j, s in state["jobs"]]
        for i in ids:
            srv.wait(i)
        return [srv.result(i) for i in ids]
    if op == "closest":
        tuv, prim = state["renderer"].trace_closest(state["rays"])
        return {"t": tuv[:, 0], "uv": tuv[:, 1:], "prim": prim}
    if op == "any":
        return state["renderer"].trace_any(state["rays"], state["tmax"])
    if op == "atrous":
        rc = state["call"](*state["size"], *(b.data_ptr() for b in state["bufs"]), state["levels"], 0.4, 128.0, 0.1,
                           1.0, state["out"].data_ptr(), state["stream"])
        if rc:
            raise RuntimeError("rg_denoise_atrous_noalloc: %d" % rc)
        return state["out"]
    if op == "denoise":
        return state["denoiser"].apply(*state["images"], spp=8.0)
    d = state["denoiser"]
    d.params = state["weights"]  # every run fits from the same weights
    losses = d.train(state["steps"], state["batch"], 1e-4)
    return {"losses": losses, "weights": d.params}


# --------------------------------------------------------------------- work --
def _trace_work(tris, rays):
    """Operations of tracing `rays` through a hierarchy over `tris` triangles: a box test (6
    multiply-adds, 4 comparisons) per binary level on the way down and 2 triangle tests of 40."""
    return rays * (16.0 * math.log2(max(tris, 2)) + 80.0)


def _render_flops(case):
    tris = {"room": 36, "spheres": 4 * case.get("tris", 0), "fog": 4 * case.get("tris", 0)}.get(case["scene"], case.get("tris", 0))
    samples = case["width"] * case["height"] * case["spp"]
    # per sample about 3.5 path segments, 2.5 shadow rays, and 300 operations of shading a vertex
    return _trace_work(tris, 6.0 * samples) + 300.0 * 3.5 * samples, tris


_NET = 2 * 9 * 32 * (16 + 5 * 32)  # multiply-adds of the denoiser's six convolutions per pixel, as operations


def work(case):
    op = case["op"]
    if op in ("render", "frame"):
        flops, tris = _render_flops(case)
        pixels = case["width"] * case["height"]
        # the image out; the triangles in, once: uploaded (76 B) for a frame, positions and normals (72 B) for a render
        return {"bytes": 16.0 * pixels + (76.0 if op == "frame" else 72.0) * tris,
                "flops": flops + (40.0 * tris * math.log2(max(tris, 2)) if op == "frame" else 0.0)}
    if op == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for j in _mix(case):
            w = work(dict(j, op="frame", width=j["side"], height=j["side"]))
            total = {k: total[k] + w[k] for k in total}
        return total
    if op in ("closest", "any"):
        n = case["rays"]
        return {"bytes": (40.0 if op == "closest" else 29.0) * n + 36.0 * case["tris"], "flops": _trace_work(case["tris"], n)}
    pixels = case.get("width", 0) * case.get("height", 0)
    if op == "atrous":  # colour 16 in and out, normal 12, albedo 12, depth 4, alpha 4; 25 taps of 30 operations a level
        return {"bytes": 64.0 * pixels, "flops": 750.0 * case["levels"] * pixels}
    if op == "denoise":
        return {"bytes": 60.0 * pixels, "flops": float(_NET) * pixels}
    pixels = case["batch"] * case["size"] ** 2 * case["steps"]
    return {"bytes": 64.0 * pixels + 50880 * 16.0 * case["steps"], "flops": 3.0 * _NET * pixels}


# -------------------------------------------------------------------- exact --
def _exact_closest(case, seed):
    if case["rays"] * case["tris"] > 4e9:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    scene = _scene(case, seed)
    pos = torch.from_numpy(np.array(scene.arrays()[0], np.float64)).reshape(-1, 3, 3).to(dev)
    pos = pos - torch.tensor([scene.desc.camera.location[k] for k in range(3)], dtype=torch.float64, device=dev)
    v0, e1, e2 = pos[:, 0], pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 0]
    rays = torch.from_numpy(_rays(case, seed)[0].astype(np.float64)).to(dev)
    chunk = max(1, int(4e6 / len(v0)))
    t_out, uv_out = [], []
    for k in range(0, len(rays), chunk):
        o, d = rays[k:k + chunk, None, :3], rays[k:k + chunk, None, 3:]
        p = torch.linalg.cross(d.expand(-1, len(v0), -1), e2[None].expand(d.shape[0], -1, -1))
        det = (e1 * p).sum(-1)
        s = o - v0
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand(d.shape[0], -1, -1))
        v = (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t >= 0)
        best, i = torch.where(ok, t, torch.full_like(t, math.inf)).min(1)
        hit = torch.isfinite(best)
        t_out.append(torch.where(hit, best, torch.full_like(best, 1e6)))
        uv = torch.stack([u.gather(1, i[:, None])[:, 0], v.gather(1, i[:, None])[:, 0]], 1)
        uv_out.append(torch.where(hit[:, None], uv, torch.zeros_like(uv)))
    return {"t": torch.cat(t_out).cpu().numpy(), "uv": torch.cat(uv_out).cpu().numpy(), "prim": None}


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _shifted(a, dy, dx, fill):
    """a[y + dy, x + dx], `fill` outside."""
    h, w = a.shape[:2]
    out = torch.full_like(a, fill)
    if abs(dy) < h and abs(dx) < w:
        out[max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)] = a[max(0, dy):h + min(0, dy), max(0, dx):w + min(0, dx)]
    return out


def _exact_atrous(case, seed):
    color, normal, depth, albedo, alpha = (t.double() for t in _image(case["width"], case["height"], seed))
    near = torch.zeros_like(depth)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            if dy or dx:
                near = torch.maximum(near, _shifted(_lum(color), dy, dx, 0.0))
    l, cap = _lum(color), 1.5 * near + 0.01
    c = color * torch.where(l > cap, cap / l, torch.ones_like(l))[..., None]
    hit = (alpha > 0.5)[..., None]
    c = torch.where(hit, (c / albedo.clamp(min=0.3)).clamp(max=3.0), c)
    n, taps = normal * 2 - 1, [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    for level in range(case["levels"]):
        step = 1 << level
        total, weights = torch.zeros_like(c), torch.zeros_like(depth)
        for ky in range(5):
            for kx in range(5):
                dy, dx = (ky - 2) * step, (kx - 2) * step
                inside = _shifted(torch.ones_like(depth), dy, dx, 0.0)
                s = _shifted(c, dy, dx, 0.0)
                nd = (_shifted(n, dy, dx, 0.0) * n).sum(-1).clamp(min=0)
                wgt = (taps[ky] * taps[kx] * inside * nd ** 128 * torch.exp(-(_lum(s) - _lum(c)) ** 2 / (2 * 0.4 ** 2 + 1e-8))
                       * torch.exp(-(_shifted(depth, dy, dx, 0.0) - depth).abs() / (0.1 * step + 1e-8)))
                total += s * wgt[..., None]
                weights += wgt
        c = torch.where((weights > 1e-8)[..., None], total / weights.clamp(min=1e-30)[..., None], c)
    out = torch.where(hit, c * albedo, c)
    return torch.cat([out, torch.ones_like(out[..., :1])], -1)


def _exact_denoise(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    color, normal, depth, albedo, _ = (t.double().to(dev) for t in _image(case["width"], case["height"], seed))
    h, w = depth.shape
    x = torch.zeros((h, w, 16), dtype=torch.float64, device=dev)
    x[..., :3], x[..., 3:6], x[..., 6:9], x[..., 9], x[..., 10] = torch.log1p(color.clamp(min=0)), albedo, normal, depth, math.log2(9.0) / 12
    p = torch.from_numpy(np.fromfile(os.path.join(os.path.dirname(rg.__file__), "kpcn_weights.bin"), np.float32)).double().to(dev)
    at = 0
    for layer, cin in enumerate([16, 32, 32, 32, 32, 32]):
        wts = p[at:at + 32 * 9 * cin].reshape(32, 9, cin)
        bias = p[at + 32 * 9 * cin:at + 32 * 9 * cin + 32]
        at += 32 * 9 * cin + 32
        y = bias.expand(h, w, 32).clone()
        for t in range(9):
            y += _shifted(x, t // 3 - 1, t % 3 - 1, 0.0) @ wts[:, t].T
        x = y.clamp(min=0) if layer < 5 else y
    k = torch.softmax(x[..., :25], -1)
    out = torch.zeros_like(color)
    for j in range(25):
        yy = (torch.arange(h, device=dev) + j // 5 - 2).clamp(0, h - 1)
        xx = (torch.arange(w, device=dev) + j % 5 - 2).clamp(0, w - 1)
        out += k[..., j:j + 1] * color[yy][:, xx]
    return torch.cat([out, torch.ones_like(out[..., :1])], -1).cpu()


def exact(case, seed):
    """What run() returns, in 64 bits; None where there is no such value (a path tracer's image is
    a sum over paths whose branches turn on rounding; whole-valued visibility; training steps whose
    batches the network draws itself)."""
    if case["op"] == "closest":
        return _exact_closest(case, seed)
    if case["op"] == "atrous":
        return _exact_atrous(case, seed)
    if case["op"] == "denoise":
        return _exact_denoise(case, seed)
    return None
