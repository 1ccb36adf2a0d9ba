"""The work a user of the renderer has it do, as cases that can be timed and compared.

A case is a dict of plain values.  `kind` says which public entry point it goes through:

  frame   one frame's API calls and sft_present into a host colour buffer (Renderer.render)
  batch   many views of several scenes in one submission (Renderer.render_batch)
  serve   the native request loop, continuous batching over submission lanes (Renderer.serve)
  rays    ray queries against the atrium's models (Renderer.raycast_device / raycast_host)
  poses   skeletal poses (Renderer.pose_eval_device / pose_eval_host)

Scenes have the shapes, sizes and distributions of sofren2_gb300.scenes (static shapes, skinned
characters, lightmapped atrium, the mixed-materials scene).  A scene's models and textures are the
same for every seed, as a program's assets are; the seed draws the cameras, instance placements,
animation times and lights of the frames, the rays and the pose requests.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sofren2_gb300 import runtime, scenes

F32 = np.float32
SIZES = scenes.MULTIVIEW_SIZES
VIEW_SCENES = ("skinned", "atrium")
BUDGET = 150 << 30          # the serving loop's device-memory admission budget, bytes


# --------------------------------------------------------------------------- the cases
def listed() -> list[dict]:
    return [
        # a thumbnail or probe render: launch latency and host work are all there is
        _case("thumbnail_160x90", "frame", scene="static", width=160, height=90, samples=1, lights=1, host="pinned", clear=True),
        # the small plain frame: static shapes, nearest-filtered textures, no MSAA
        _case("static_640x360_1x", "frame", scene="static", width=640, height=360, samples=1, lights=1, host="pinned", clear=True),
        # an editor or thin-client window of odd size: near-plane clipping, NPOT and untextured materials,
        # directional lights, more lights than a tile holds, pixels of the caller kept, pageable buffer
        _case("window_1333x717_2x_keep", "frame", scene="variety", width=1333, height=717, samples=2, lights=18, host="pageable", clear=False),
        # the headline frame: eight skinned characters, 1080p, 2x MSAA
        _case("skinned_1080p_2x", "frame", scene="skinned", width=1920, height=1080, samples=2, lights=4, host="pinned", clear=True),
        # a game frame without MSAA over the large static model, odd size
        _case("atrium_1279x719_1x", "frame", scene="atrium", width=1279, height=719, samples=1, lights=8, host="pinned", clear=True),
        # the heavy frame: 249k triangles, 16 lights on every pixel, lightmaps, 4x MSAA
        _case("atrium_1080p_4x", "frame", scene="atrium", width=1920, height=1080, samples=4, lights=16, host="pinned", clear=True),
        # offline / multi-camera rendering: mixed scenes, resolutions and MSAA in one submission
        _case("multiview_48", "batch", views=48),
        # a burst of requests at a render server
        _case("serve_burst_40", "serve", requests=40, max_batch=8),
        # picking and gameplay queries of one tick: host arrays, latency
        _case("rays_host_600", "rays", n=600, where="host"),
        # visibility or baking queries in bulk, device arrays
        _case("rays_device_1m", "rays", n=1 << 20, where="device"),
        # a scene's characters animated for one frame, host arrays
        _case("poses_host_100", "poses", n=100, where="host"),
        # a crowd or a dataset of poses, device arrays
        _case("poses_device_65536", "poses", n=1 << 16, where="device"),
    ]


def _case(name: str, kind: str, **values) -> dict:
    return {"name": name, "kind": kind, **values}


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame", "frame", "frame", "batch", "serve", "rays", "poses"])
    if kind == "frame":
        scene = rng.choice(["static", "variety", "skinned", "atrium"])
        width = _log_int(rng, 96, 1920)
        height = max(64, min(1080, int(width * rng.uniform(0.45, 0.75))))
        most = {"static": 4, "variety": 20, "skinned": 16, "atrium": 16}[scene]
        clear = rng.random() < 0.75
        return {"kind": kind, "scene": scene, "width": width, "height": height, "samples": rng.choice([1, 2, 4]),
                "lights": rng.randint(1, most), "host": rng.choice(["pinned", "pinned", "pageable"]), "clear": clear}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(2, 48)}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(4, 40), "max_batch": rng.randint(1, 16)}
    where = rng.choice(["host", "device"])
    if kind == "rays":
        return {"kind": kind, "n": _log_int(rng, 1, 1 << 14 if where == "host" else 1 << 20), "where": where}
    return {"kind": kind, "n": _log_int(rng, 1, 1 << 12 if where == "host" else 1 << 16), "where": where}


# --------------------------------------------------------------------------- assets
_KEEP: dict = {}            # this process's renderer and its scenes' assets, made once


def _kept(key, make):
    if key not in _KEEP:
        _KEEP[key] = make()
    return _KEEP[key]


def _renderer() -> runtime.Renderer:
    return _kept("renderer", lambda: runtime.Renderer(640, 360, 1))


def _noise_texture(size: int, seed: int, lattice: int = 16) -> np.ndarray:
    """ARGB8888 value noise: a random lattice every `lattice` texels, smoothstep-bilinear between."""
    rng = np.random.default_rng(seed)
    g = size // lattice + 1
    f = np.arange(lattice, dtype=F32) / F32(lattice)
    s = f * f * (3 - 2 * f)
    out = np.full((size, size), 0xFF000000, np.uint32)
    for shift in (16, 8, 0):
        c = rng.integers(0, 256, (g, g)).astype(F32)
        rows = (c[:-1, None, :] + (c[1:, None, :] - c[:-1, None, :]) * s[None, :, None]).reshape(size, g)
        v = (rows[:, :-1, None] + (rows[:, 1:, None] - rows[:, :-1, None]) * s[None, None, :]).reshape(size, size)
        out |= v.astype(np.uint32) << np.uint32(shift)
    return out


def _assets(kind: str) -> dict:
    """A scene's models, materials and textures with its base frame, and the blob bytes of all but the frames."""
    def make():
        if kind == "static":
            sc, anims = scenes.static_shapes_scene(64, 64, seed=1001), []
        elif kind == "variety":
            sc, anims = scenes.variety_scene(64, 64, seed=4001), []
        elif kind == "skinned":
            sc = scenes.skinned_characters_scene(64, 64, seed=2001)
            anims = [scenes.HumanoidAnim(2001 * 89 + c) for c in range(8)]
        else:
            # its own textures are made here, where the scene's generator takes seconds for them, at 512x512: resident
            # textures stay in the renderer's heap for its life, and every state loads its scene; a frame reads no level
            # but those its pixels are as dense as.  Ray queries read no texture at all.
            size = 512 if kind == "atrium" else 16
            sc = _kept("atrium scene", lambda: scenes.atrium_scene(64, 64, seed=3001, tex_size=64))
            full = sc.textures
            sc = _with_assets(sc, [full[0] if kind == "atrium" else full[0][:16, :16]] +
                              [_noise_texture(size, 3001 + t) for t in range(25)] +
                              [t if kind == "atrium" else t[:16, :16] for t in full[26:]], list(sc.frames))
            anims = [scenes.HumanoidAnim(3001 * 89 + c) for c in range(4)]
        base = sc.frames[0]
        sc.frames = []
        return {"scene": sc, "base": base, "anims": anims, "bytes": sc.to_bytes()[:-4],
                "meshlets": sum(ms.n for mi, _, _ in base.instances for ms in sc.models[mi].meshes)}
    return _kept(("assets", kind), make)


def _lights(kind: str, rng, n: int) -> list:
    u = rng.uniform
    if kind == "static":    # far above the objects, covering all of them
        return [((u(-1, 1), F32(30.0), F32(25) + u(-1, 1)), 1.0, 0.95, 0.9, 1.0, 60.0) for _ in range(n)]
    if kind == "variety":
        return [((u(-4, 4), u(9, 11), u(3, 9)), u(0.3, 1), u(0.3, 1), u(0.3, 1), 0.8, u(12, 20)) for _ in range(n)]
    if kind == "skinned":
        return [((u(-6, 6), u(5, 7), u(3, 11)), u(0.6, 1), u(0.6, 1), u(0.6, 1), 1.0, 14.0) for _ in range(n)]
    return [((u(-12, 12), u(13, 14.5), u(6, 17)), u(0.6, 1), u(0.6, 1), u(0.6, 1), 0.5, 60.0) for _ in range(n)]


def _frame(kind: str, rng, width: int, height: int, lights: int, clear: bool = True, free_camera: bool = False) -> scenes.Frame:
    """One frame of a scene: seeded camera, placements, animation time and lights."""
    a, u = _assets(kind), rng.uniform
    base = a["base"]
    insts = list(base.instances)
    if kind == "skinned":
        pos = (u(-4, 4), u(1.2, 2.6), u(-1, 1.5)) if free_camera else (u(-0.3, 0.3), 1.7, u(-0.3, 0.3))
        tgt = (u(-2, 2), u(0.6, 1.4), u(6, 9)) if free_camera else (0.0, 1.0, 8.0)
    elif kind.startswith("atrium"):
        pos = (u(-5, 5), u(1.5, 4), u(0.2, 2.5)) if free_camera else (u(-0.5, 0.5), 1.7, u(0.3, 0.8))
        tgt = (u(-4, 4), u(1, 5), u(9, 15)) if free_camera else (0.0, 3.0, 12.0)
    else:
        pos, tgt = (0.0, 0.0, 0.0), (0.0, 0.0, 1.0)
        centre, half, size = ((0, 0, 25), (10, 10, 10), (0.5, 2.0)) if kind == "static" else ((0, 0, 3), (3, 2, 3), (0.5, 1.8))
        for k, (mi, _, _) in enumerate(insts):
            p = [F32(c + u(-h, h)) for c, h in zip(centre, half)]
            t = scenes.mat_mul(scenes.mat_scale(F32(u(*size))), scenes.mat_rot_y(F32(u(0, 6.28318))))
            insts[k] = (mi, scenes.mat_mul(t, scenes.mat_translate(*p)), None)
    if a["anims"]:
        t = F32(u(0, 1))
        first = len(insts) - len(a["anims"])
        insts[first:] = [(mi, tr, a["anims"][c].pose(t)) for c, (mi, tr, _) in enumerate(insts[first:])]
    pos, tgt = tuple(F32(x) for x in pos), tuple(F32(x) for x in tgt)
    f = scenes.Frame(width, height, pos, scenes.view_look_at(pos, tgt), scenes.proj(60.0, F32(width) / F32(height), 0.1, 100.0))
    f.ambient, f.clear, f.dir_lights = base.ambient, int(clear), base.dir_lights
    f.point_lights = _lights(kind, rng, lights)
    f.instances = insts
    return f


class _Scene:
    """A scene resident in the renderer, with its frames; its host copy goes with the object."""

    def __init__(self, kind: str, frames: list):
        only = scenes.Scene()
        only.frames = frames
        blob = _assets(kind)["bytes"] + only.to_bytes()[20:]     # 20 bytes: magic, version, no textures, materials, models
        self.kind, self.frames = kind, frames
        self.handle = _renderer().load_scene(blob)

    def __del__(self):
        _renderer().free_scene(self.handle)


def _colour(n: int, host: str) -> torch.Tensor:
    t = torch.zeros(n, dtype=torch.int32)
    return t.pin_memory() if host == "pinned" else t


def _image(t: torch.Tensor, width: int, height: int) -> np.ndarray:
    return t.numpy()[: width * height].reshape(height, width).view(np.uint32)


# --------------------------------------------------------------------------- prepare
def _views(seed: int, n: int) -> list[tuple]:
    """n views, in turn of the skinned and the atrium scene: (scene index, kind, width, height, samples, lights).
    The sizes and sample counts come round in turn, so that the work of a case hardly depends on the seed."""
    rng = np.random.default_rng([seed, 4])
    out = []
    for k in range(n):
        w, h = SIZES[(k * 3 + k // 5) % len(SIZES)]
        out.append((k % 2, VIEW_SCENES[k % 2], w, h, (1, 2, 4)[(k + k // 3) % 3], int(rng.integers(1, 17))))
    return out


def _load_views(seed: int, views: list[tuple]) -> tuple[list, list[int]]:
    """The scenes with the views' frames, and each view's frame index in its scene."""
    rng = np.random.default_rng([seed, 5])
    frames, index = [[] for _ in VIEW_SCENES], []
    for si, kind, w, h, _, lights in views:
        index.append(len(frames[si]))
        frames[si].append(_frame(kind, rng, w, h, lights, free_camera=True))
    return [_Scene(kind, fr) for kind, fr in zip(VIEW_SCENES, frames)], index


def _ray_records(seed: int, n: int, scene: _Scene) -> np.ndarray:
    return scenes.ray_batch(_with_frames("atrium for rays", scene.frames), n, seed=seed)


def _with_assets(src: scenes.Scene, textures: list, frames: list) -> scenes.Scene:
    sc = scenes.Scene()
    sc.textures, sc.materials, sc.models, sc.frames = textures, src.materials, src.models, frames
    return sc


def _with_frames(kind: str, frames: list) -> scenes.Scene:
    src = _assets(kind)["scene"]
    return _with_assets(src, src.textures, frames)


def _pose_records(seed: int, n: int, rig: dict) -> np.ndarray:
    """Requests over both animations: most times inside a few loops of the clip, some before it."""
    rng = np.random.default_rng([seed, 8])
    req = np.zeros(n, runtime.POSE_REQUEST_DTYPE)
    req["animation"] = (rng.random(n) < 0.25).astype(np.int32)
    req["time"] = np.where(rng.random(n) < 0.9, rng.uniform(0, 4, n), rng.uniform(-1, 0, n)).astype(F32)
    return req


def prepare(case: dict, seed: int) -> dict:
    R = _renderer()
    kind = case["kind"]
    st = {"case": case, "renderer": R}
    if kind == "frame":
        w, h = case["width"], case["height"]
        rng = np.random.default_rng([seed, 1])
        st["scene"] = _Scene(case["scene"], [_frame(case["scene"], rng, w, h, case["lights"], case["clear"])])
        st["colour"] = _colour(w * h, case["host"])
        st["image"] = _image(st["colour"], w, h)
        if not case["clear"]:   # the caller's picture; every pass draws over what the buffer then holds
            st["image"][:] = _noise_texture(2048, seed)[:h, :w]
    elif kind == "batch":
        views = _views(seed, case["views"])
        st["scenes"], index = _load_views(seed, views)
        st["views"] = [(st["scenes"][v[0]].handle, i, v[4]) for v, i in zip(views, index)]
        st["colours"] = [_colour(v[2] * v[3], "pinned") for v in views]
        st["images"] = [_image(c, v[2], v[3]) for c, v in zip(st["colours"], views)]
    elif kind == "serve":
        views = _views(seed, case["requests"])
        st["scenes"], index = _load_views(seed, views)
        st["handles"] = [s.handle for s in st["scenes"]]
        need = {k: _assets(k)["meshlets"] for k in ("skinned", "atrium")}
        st["requests"] = [(0.0, si, i, S, lights, runtime.request_device_bytes(w, h, S, need[k]))
                          for (si, k, w, h, S, lights), i in zip(views, index)]
        most = max(w * h for _, _, w, h, _, _ in views)
        st["ring"] = [_colour(most, "pinned") for _ in range(max(len(views), case["max_batch"]))]
        st["images"] = [c.numpy().view(np.uint32) for c in st["ring"]]
        st["colours"] = [c[: v[2] * v[3]] for c, v in zip(st["ring"], views)]
    elif kind == "rays":
        st["scene"] = _Scene("atrium for rays", [_frame("atrium for rays", np.random.default_rng([seed, 6]), 64, 64, 1)])
        rays = _ray_records(seed, case["n"], st["scene"])
        ids = np.array([R.model_device_id(st["scene"].handle, mi) for mi in range(len(_assets("atrium for rays")["scene"].models))], np.int32)
        rays["model"] = ids[rays["model"]]
        if case["where"] == "host":
            st["rays"], st["hits"] = rays, np.zeros(case["n"], runtime.HIT_DTYPE)
        else:
            st["rays"] = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
            st["hits"] = torch.zeros((case["n"], 8), dtype=torch.float32, device="cuda")
    else:
        rig = _kept("rig", lambda: scenes.pose_rig())
        n, nb = case["n"], len(rig["bones"])
        req = _pose_records(seed, n, rig)
        req["skeleton"] = _kept("skeleton", lambda: R.skeleton_upload(rig))
        if case["where"] == "host":
            st["requests"] = req
            st["posed"], st["global"] = np.zeros((n, nb, 16), F32), np.zeros((n, nb, 16), F32)
        else:
            st["requests"] = torch.from_numpy(req.view(np.uint8).copy()).cuda()
            st["offsets"] = torch.arange(0, n * nb, nb, dtype=torch.int32, device="cuda")
            st["posed"] = torch.zeros((n, nb, 16), dtype=torch.float32, device="cuda")
            st["global"] = torch.zeros((n, nb, 16), dtype=torch.float32, device="cuda")
    return st


# --------------------------------------------------------------------------- run
def run(st: dict):
    case, R = st["case"], st["renderer"]
    kind = case["kind"]
    if kind == "frame":
        R.set_samples(case["samples"])
        R.render(st["scene"].handle, 0, st["image"])
        return st["colour"]
    if kind == "batch":
        R.render_batch(st["views"], st["images"])
        return st["colours"]
    if kind == "serve":
        R.serve(st["handles"], st["requests"], case["max_batch"], BUDGET, "overlap", st["images"])
        return st["colours"]
    if kind == "rays":
        if case["where"] == "host":
            h = R.raycast_host(st["rays"], st["hits"])
            return {"hit": h["hit"].view(np.int32), "distance": h["dist"], "pos": h["pos"], "normal": h["nrm"]}
        R.raycast_device(st["rays"].data_ptr(), case["n"], st["hits"].data_ptr())
        h = st["hits"]
        return {"hit": h[:, 0].view(torch.int32), "distance": h[:, 1], "pos": h[:, 2:5], "normal": h[:, 5:8]}
    if case["where"] == "host":
        R.pose_eval_host(st["requests"], st["posed"].reshape(-1), st["global"].reshape(-1))
    else:
        R.pose_eval_device(st["requests"].data_ptr(), st["offsets"].data_ptr(), case["n"], st["posed"].data_ptr(), st["global"].data_ptr())
    return {"posed": st["posed"], "global": st["global"]}


# --------------------------------------------------------------------------- work
def _frame_work(kind: str, w: int, h: int, samples: int, lights: int) -> tuple[float, float]:
    """Bytes and operations of one frame: every meshlet's attributes, indices and bounds (and skin) once,
    one texel and (kept or lightmapped) four bytes more per pixel, the colours out; transform and projection
    per vertex, edge functions and depth per sample, and per pixel about 150 operations of interpolation,
    texturing and blending and 40 per light that reaches a tile (at most 16 do)."""
    m = _assets(kind)["meshlets"]
    px = w * h
    size = m * (2560 + 512 + 32) + px * 12
    ops = m * 64 * 120 + px * (12 * samples + 150 + 40 * min(lights, 16))
    return float(size), float(ops)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "frame":
        b, f = _frame_work(case["scene"], case["width"], case["height"], case["samples"], case["lights"])
    elif kind in ("batch", "serve"):
        each = [_frame_work(k, w, h, S, 8) for _, k, w, h, S, _ in _views(0, case["views" if kind == "batch" else "requests"])]
        b, f = sum(x[0] for x in each), sum(x[1] for x in each)
    elif kind == "rays":    # the records, and per ray about 12 nodes of 8 boxes and 2 triangles
        b, f = case["n"] * (96.0 + 32.0), case["n"] * (12 * 8 * 20.0 + 2 * 60.0)
    else:                   # the requests, and two 4x4 matrices a bone out; three 4x4 products and a slerp a bone
        b, f = case["n"] * (16.0 + 22 * 128.0), case["n"] * 22 * (3 * 112.0 + 60.0)
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------------- exact
def exact(case: dict, seed: int):
    """Poses, and ray queries of a few hundred rays, in 64 bits; colours are whole numbers."""
    if case["kind"] == "poses":
        rig = scenes.pose_rig()
        req = _pose_records(seed, case["n"], rig)
        posed, glob = _poses64(rig, req["animation"], req["time"].astype(np.float64))
        return {"posed": posed, "global": glob}
    if case["kind"] == "rays" and case["n"] <= 2048:
        fr = _frame("atrium for rays", np.random.default_rng([seed, 6]), 64, 64, 1)
        sc = _with_frames("atrium for rays", [fr])
        dist, pos, nrm = _rays64(sc, scenes.ray_batch(sc, case["n"], seed=seed))
        return {"hit": None, "distance": dist, "pos": pos, "normal": nrm}
    return None


def _poses64(rig: dict, anim: np.ndarray, time: np.ndarray):
    n, nb = len(anim), len(rig["bones"])
    glob, posed = np.zeros((n, nb, 4, 4)), np.zeros((n, nb, 4, 4))
    for a, an in enumerate(rig["anims"]):
        at = np.nonzero(anim == a)[0]
        if not len(at):
            continue
        t = np.fmod(time[at], np.float64(an["duration"]))
        val = {}
        for s, node, path in an["channels"]:
            if not 0 <= node < nb:
                continue
            ins, outs, step = an["samplers"][s]
            ins, outs = ins.astype(np.float64), outs.astype(np.float64)
            f0 = np.clip(np.searchsorted(ins, t, side="right") - 1, 0, len(ins) - 1)
            f1 = np.minimum(f0 + 1, len(ins) - 1)
            f1 = np.where(t <= ins[0], 0, f1)
            f0 = np.where(t <= ins[0], 0, f0)
            dt = ins[f1] - ins[f0]
            x = np.where(dt > 0.0001, (t - ins[f0]) / np.where(dt > 0, dt, 1), 0.0)[:, None]
            v0, v1 = outs[f0], outs[f1]
            if step:
                v = v0
            elif path == 1:
                v = _slerp64(v0, v1, x)
            else:
                v = v0 + (v1 - v0) * x
            val[node, path] = v
        local = np.zeros((len(at), nb, 4, 4))
        for b, bone in enumerate(rig["bones"]):
            if not any((b, p) in val for p in range(3)):
                local[:, b] = bone["local_bind"].astype(np.float64)
                continue
            pick = lambda p, rest, k: val[b, p][:, :k] if (b, p) in val else np.broadcast_to(np.asarray(rest, np.float64), (len(at), k))  # noqa: E731
            tr, q, sc = pick(0, bone["base_t"], 3), pick(1, bone["base_r"], 4), pick(2, bone["base_s"], 3)
            x, y, z, w = q.T
            rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y),
                            2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x),
                            2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)
            local[:, b, :3, :3] = sc[:, :, None] * rot
            local[:, b, 3, :3] = tr
            local[:, b, 3, 3] = 1
        g = np.zeros_like(local)
        for b, bone in enumerate(rig["bones"]):     # parents come first in the rig
            g[:, b] = local[:, b] if bone["parent"] < 0 else local[:, b] @ g[:, bone["parent"]]
        glob[at] = g
        posed[at] = np.stack([bone["inverse_bind"].astype(np.float64) for bone in rig["bones"]])[None] @ g
    return posed.reshape(n, nb, 16), glob.reshape(n, nb, 16)


def _slerp64(a, b, t):
    dot = (a * b).sum(-1, keepdims=True)
    b, dot = np.where(dot < 0, -b, b), np.abs(dot)
    th = np.arccos(np.minimum(dot, 1.0))
    sin = np.where(dot > 0.9995, 1.0, np.sin(th))
    far = a * (np.cos(th * t) - dot * np.sin(th * t) / sin) + b * (np.sin(th * t) / sin)
    v = np.where(dot > 0.9995, a + t * (b - a), far)
    return v / np.sqrt((v * v).sum(-1, keepdims=True))


def _rays64(sc: scenes.Scene, rays: np.ndarray):
    """Every ray against every triangle of its model; the nearest hit within the limit."""
    n = len(rays)
    dist, pos, nrm = rays["max_dist"].astype(np.float64), np.zeros((n, 3)), np.zeros((n, 3))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    for mi in np.unique(rays["model"]):
        tris = []
        for ms in sc.models[mi].meshes:
            k = ms.inds.reshape(ms.n, 16, 4, 8)[:, :, :3].transpose(0, 1, 3, 2).reshape(ms.n, 128, 3).astype(np.int64)
            p = ms.attr[:, :3].transpose(0, 2, 1)
            v = np.take_along_axis(p[:, None], k[..., None].reshape(ms.n, 1, 384, 1), 2).reshape(ms.n, 128, 3, 3)
            tris.append(v[k.any(-1)])
        v = torch.from_numpy(np.concatenate(tris)).to(dev, torch.float64)
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        at = np.nonzero(rays["model"] == mi)[0]
        m3 = torch.from_numpy(rays["T"][at].reshape(-1, 4, 4)[:, :3, :3].astype(np.float64)).to(dev)
        o = torch.einsum("rij,rj->ri", m3, torch.from_numpy(rays["o"][at].astype(np.float64)).to(dev))
        d = torch.einsum("rij,rj->ri", m3, torch.from_numpy(rays["d"][at].astype(np.float64)).to(dev))
        scale = 1 / d.norm(dim=-1, keepdim=True)
        d = d * scale
        for c in range(0, len(at), 64):
            oc, dc = o[c : c + 64, None], d[c : c + 64, None]
            p = torch.linalg.cross(dc.expand(-1, len(v), -1), e2.expand(len(oc), -1, -1))
            det = (e1 * p).sum(-1)
            tv = oc - v[:, 0]
            q = torch.linalg.cross(tv, e1.expand(len(oc), -1, -1))
            inv = 1 / torch.where(det.abs() < 1e-6, torch.ones_like(det), det)
            a, b, t = (tv * p).sum(-1) * inv, (dc * q).sum(-1) * inv, (e2 * q).sum(-1) * inv
            far = torch.from_numpy(rays["max_dist"][at[c : c + 64]].astype(np.float64)).to(dev)[:, None] / scale[c : c + 64]
            ok = (det.abs() >= 1e-6) & (a >= 0) & (a <= 1) & (b >= 0) & (a + b <= 1) & (t > 1e-6) & (t < far)
            t, k = torch.where(ok, t, torch.full_like(t, math.inf)).min(-1)
            for r in torch.nonzero(torch.isfinite(t))[:, 0].tolist():
                w = at[c + r]
                dist[w] = float(t[r] * scale[c + r, 0])
                pos[w] = ((o[c + r] + d[c + r] * t[r]) @ m3[c + r]).cpu().numpy()
                x = torch.linalg.cross(e1[k[r]], e2[k[r]])
                x = (x / x.norm()) @ m3[c + r]
                nrm[w] = (x / x.norm()).cpu().numpy()
    return dist, pos, nrm
