"""What a user has this library do, as timed cases.

A case is a dict of plain values.  ``listed()`` gives the standing ones,
``draw(rng)`` more of the same ranges, ``prepare(case, seed)`` what a program
holds before the call (context, resident scenes, rays, targets), ``run(state)``
one pass through the public entry points, ``work(case)`` the bytes and
operations a pass cannot do without and ``exact(case, seed)`` its result in 64
bits where one exists.

Kinds and their ranges:
  room      the 48-triangle Lambert room, 32x32 .. 384x384, 1 .. 32 spp,
            2 .. 8 bounces, Halton or MRG32k3a light draws
  frame     icosphere soups of 1 K .. 1 M triangles, 256 principled materials,
            64x48 .. 1280x720, 1 .. 64 spp, 2 .. 8 bounces; options: tree from
            the host or the device builder, textures, sky light, thin lens,
            image left on the device or copied to the host
  batch     4 .. 16 soups of different size, resolution and spp as one frame
  backward  parameter gradient of a frame (up to 512x512, 16 spp, 4 bounces)
  fit       2 .. 16 scenes' fitting step (forward, L2 loss, gradient)
  closest, any   1 K .. 2 M rays in caller's memory (host or device)
  animate   moved vertices: refit, then a frame of 1 .. 4 spp
  direct    the two direct-lighting integrators
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from globillum_gb300 import gbpt, scenes

FLT_MAX = float(np.finfo(np.float32).max)


# ------------------------------------------------------------------ cases --

def listed() -> list:
    return [
        # the smallest call: a preview of a tiny scene while it is edited
        {"name": "preview_room", "kind": "room", "w": 64, "h": 64, "spp": 4, "bounces": 5, "halton": True, "host": False},
        # the plain workload of the benchmark: Cornell-style room to a host image
        {"name": "room_frame", "kind": "room", "w": 256, "h": 256, "spp": 16, "bounces": 5, "halton": True, "host": True},
        # an asset with diffuse textures under a sky, through a thin lens, at an odd size
        {"name": "textured_sky", "kind": "frame", "spheres": 50, "w": 333, "h": 217, "spp": 8, "bounces": 6, "lights": 1,
         "builder": "host", "textured": True, "sky": True, "lens": True, "host": True},
        # interactive view of a large scene: one sample per pixel of the device-built tree
        {"name": "progressive_1m", "kind": "frame", "spheres": 800, "w": 1280, "h": 720, "spp": 1, "bounces": 8,
         "lights": 4, "builder": "device", "textured": False, "sky": False, "lens": False, "host": False},
        # the headline frame: 1 M triangles, 1280x720, 64 spp, 8 bounces
        {"name": "frame_1m", "kind": "frame", "spheres": 800, "w": 1280, "h": 720, "spp": 64, "bounces": 8, "lights": 4,
         "builder": "host", "textured": False, "sky": False, "lens": False, "host": True},
        # a dataset of many scenes rendered as one frame
        {"name": "batch_mixed", "kind": "batch", "scenes": 12, "max_tris": 100_000, "bounces": 6},
        # inverse rendering of one scene: the gradient of an image loss, odd size
        {"name": "backward_odd", "kind": "backward", "spheres": 160, "w": 509, "h": 511, "spp": 16, "bounces": 4},
        # inverse rendering of many scenes: one fitting step
        {"name": "fit_step", "kind": "fit", "scenes": 8, "spheres": 24, "w": 256, "h": 256, "spp": 8, "bounces": 4},
        # closest-hit queries of another program on device buffers
        {"name": "trace_closest", "kind": "closest", "spheres": 50, "rays": 262_147, "host": False},
        # visibility queries against a large scene
        {"name": "trace_any", "kind": "any", "spheres": 800, "rays": 2_000_003, "host": False},
        # an animated preview: vertices move, the tree is refitted, two samples per pixel
        {"name": "animate", "kind": "animate", "spheres": 160, "w": 640, "h": 360, "spp": 2, "bounces": 4},
        # direct lighting with the hybrid integrator's sampling at an odd size
        {"name": "direct", "kind": "direct", "spheres": 50, "w": 641, "h": 359, "hybrid": True, "camera_samples": 2,
         "light_samples": 8},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo: int, hi_w: int, hi_h: int) -> tuple:
    w = _log(rng, lo, hi_w)
    h = max(lo * 3 // 4, min(hi_h, int(w * rng.uniform(0.5, 1.1))))
    return w, h


def draw(rng) -> dict:
    kind = rng.choice(["room", "room", "frame", "frame", "frame", "batch", "backward", "fit", "closest", "any",
                       "animate", "direct"])
    if kind == "room":
        w, h = _size(rng, 32, 384, 384)
        return {"kind": kind, "w": w, "h": h, "spp": _log(rng, 1, 32), "bounces": rng.randint(2, 8),
                "halton": rng.random() < 0.5, "host": rng.random() < 0.5}
    if kind == "frame":
        w, h = _size(rng, 64, 1280, 720)
        plain = rng.random() < 0.5
        return {"kind": kind, "spheres": _log(rng, 1, 800), "w": w, "h": h, "spp": _log(rng, 1, 64),
                "bounces": rng.randint(2, 8), "lights": rng.randint(1, 4),
                "builder": "device" if rng.random() < 0.4 else "host", "textured": not plain and rng.random() < 0.6,
                "sky": not plain and rng.random() < 0.6, "lens": not plain and rng.random() < 0.5,
                "host": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(4, 16), "max_tris": _log(rng, 4_000, 200_000),
                "bounces": rng.randint(3, 6)}
    if kind == "backward":
        w, h = _size(rng, 64, 512, 512)
        return {"kind": kind, "spheres": _log(rng, 1, 400), "w": w, "h": h, "spp": _log(rng, 1, 16),
                "bounces": rng.randint(2, 6)}
    if kind == "fit":
        return {"kind": kind, "scenes": rng.randint(2, 16), "spheres": _log(rng, 4, 60), "w": _log(rng, 32, 256),
                "h": _log(rng, 32, 256), "spp": _log(rng, 2, 16), "bounces": rng.randint(2, 4)}
    if kind in ("closest", "any"):
        return {"kind": kind, "spheres": _log(rng, 1, 800), "rays": _log(rng, 1_000, 2_000_000),
                "host": rng.random() < 0.5}
    if kind == "animate":
        w, h = _size(rng, 64, 1280, 720)
        return {"kind": kind, "spheres": _log(rng, 4, 400), "w": w, "h": h, "spp": rng.randint(1, 4),
                "bounces": rng.randint(2, 6)}
    w, h = _size(rng, 64, 1280, 720)
    return {"kind": "direct", "spheres": _log(rng, 1, 400), "w": w, "h": h, "hybrid": rng.random() < 0.5,
            "camera_samples": rng.randint(1, 4), "light_samples": rng.randint(1, 16)}


# ----------------------------------------------------------------- scenes --

def _room(case: dict, seed: int) -> scenes.SceneData:
    """The room with seeded albedos; the tall box and the camera move a little."""
    sc = scenes.cornell(case["w"], case["h"], case["spp"], case["bounces"], seed=seed)
    r = np.random.default_rng(seed + 71)
    box = sc.material_index == 6
    sc.positions[box] += np.tile(r.uniform(-0.04, 0.04, 3) * [1, 0, 1], 3).astype(np.float32)
    sc.camera["pos"] = tuple(float(x) for x in np.array([0.5, 0.5, -1.4]) + r.uniform(-0.03, 0.03, 3))
    sc.render["rng_mode"] = gbpt.GB_RNG_HALTON_LIGHT if case["halton"] else gbpt.GB_RNG_MRG32K3A_POOL
    return sc


def _soup(spheres: int, w: int, h: int, spp: int, bounces: int, seed: int, lights: int = 4,
          density_box: bool = True) -> scenes.SceneData:
    """Icospheres at the density of the 800-sphere scene, other geometry,
    materials and lights for every seed."""
    box = 100.0 * (spheres / 800.0) ** (1.0 / 3.0) if density_box else 100.0
    return scenes.icospheres(n_spheres=spheres, width=w, height=h, spp=spp, max_bounces=bounces, n_lights=lights,
                             box=max(box, 12.0), seed_geometry=3 * seed + 1, seed_materials=3 * seed + 2,
                             seed_lights=3 * seed + 3)


def _frame_scene(case: dict, seed: int) -> scenes.SceneData:
    sc = _soup(case["spheres"], case["w"], case["h"], case["spp"], case["bounces"], seed, case["lights"])
    if case["textured"]:
        sc = scenes.with_textures(sc, n_textures=2, size=256, fraction=0.5, scale=0.2, seed=seed)
    if case["sky"]:
        sc.lights.append({"type": gbpt.GB_LIGHT_SKY, "map": scenes.procedural_sky(256, 128, seed=seed), "scale": 0.2,
                          "diameter": 40.0, "power": -1.0})
    if case["lens"]:
        eye = np.array(sc.camera["pos"])
        sc.camera["aperture"] = 0.5
        sc.camera["focus_distance"] = float(np.linalg.norm(eye - np.array([0.5, 0.3, 0.5]) * eye[1] / 0.7))
    return sc


class _State:
    """What a program keeps between passes; gives its scenes and context back."""

    def __init__(self, case: dict):
        self.case = case
        self.ctx = gbpt.Context(0)
        self.scenes = []

    def scene(self, data, **kw) -> gbpt.Scene:
        s = self.ctx.scene(data, **kw)
        self.scenes.append(s)
        return s

    def __del__(self):
        for s in getattr(self, "scenes", []):
            s.close()
        if getattr(self, "ctx", None) is not None:
            self.ctx.close()


def _rays(sc: scenes.SceneData, n: int, seed: int, shadow: bool) -> tuple:
    """Camera rays of an n-pixel square view in pixel order and, after them,
    rays between random points of the scene; shadow rays end at a light."""
    r = np.random.default_rng(seed + 5)
    o, d = scenes.random_rays(sc, n, seed=seed + 6)
    t = np.full(n, FLT_MAX, np.float32)
    if shadow:
        ls = [l for l in sc.lights if l.get("type", gbpt.GB_LIGHT_RECT) == gbpt.GB_LIGHT_RECT]
        k = r.integers(0, len(ls), n)
        c = np.array([l["center"] for l in ls])[k]
        wh = np.array([l["wh"] for l in ls])[k]
        tgt = c + np.stack([r.uniform(-0.5, 0.5, n) * wh[:, 0], np.zeros(n), r.uniform(-0.5, 0.5, n) * wh[:, 1]], 1)
        v = tgt - o
        ln = np.linalg.norm(v, axis=1)
        return o, (v / ln[:, None]).astype(np.float32), ln.astype(np.float32)
    m = n // 2
    side = max(1, int(math.isqrt(m)))
    i = np.arange(m)
    pos, W, U, V, th = _camera(sc.camera)
    u = (((i % side) + r.uniform(0, 1, m)) / side * 2 - 1) * th
    v = (((i // side) + r.uniform(0, 1, m)) / side * 2 - 1) * th
    cd = u[:, None] * U + v[:, None] * V + W
    o[:m] = pos
    d[:m] = cd / np.linalg.norm(cd, axis=1, keepdims=True)
    return o, d, t


def _camera(cam: dict) -> tuple:
    pos = np.array(cam["pos"], np.float64)
    W = np.array(cam["dir"], np.float64)
    W = W / np.linalg.norm(W)
    U = np.cross(np.array(cam["up"], np.float64), W)
    U = U / np.linalg.norm(U)
    return pos, W, U, np.cross(W, U), math.tan(math.pi * cam["fovy_deg"] / 360.0)


def _batch_scenes(case: dict, seed: int) -> list:
    """Sizes of the mixed set (spp 4/16/64, 64^2 .. 512^2 pixels) belong to
    the case; geometry, materials and lights to the seed."""
    r = np.random.default_rng(case["scenes"] * 1_000_003 + case["max_tris"])
    out = []
    for k in range(case["scenes"]):
        tris = math.exp(r.uniform(math.log(1_000), math.log(case["max_tris"])))
        res = int(r.choice([64, 128, 256, 512]))
        spp = int(r.choice([4, 16, 64])) if res < 512 else 4
        out.append(_soup(max(1, round(tris / 1280)), res, res, spp, case["bounces"], seed * 100 + k,
                         int(r.integers(1, 5))))
    return out


def prepare(case: dict, seed: int):
    st = _State(case)
    kind = case["kind"]
    if kind in ("room", "frame"):
        sc = _room(case, seed) if kind == "room" else _frame_scene(case, seed)
        st.cam, st.rdesc = sc.camera, sc.render
        st.s = st.scene(sc, builder=case.get("builder", "host"))
        shape = (case["h"], case["w"], 3)
        if case["host"]:
            st.image = torch.empty(shape, dtype=torch.float32, pin_memory=True)
            st.out = st.image.numpy()
        else:
            st.image = torch.empty(shape, dtype=torch.float32, device="cuda")
    elif kind == "batch":
        data = _batch_scenes(case, seed)
        st.jobs = [(st.scene(sc), sc.camera, sc.render) for sc in data]
        st.images = [torch.empty((sc.render["height"], sc.render["width"], 3), dtype=torch.float32, device="cuda")
                     for sc in data]
    elif kind == "backward":
        sc = _soup(case["spheres"], case["w"], case["h"], case["spp"], case["bounces"], seed)
        st.cam, st.rdesc = sc.camera, sc.render
        st.s = st.scene(sc)
        g = torch.Generator(device="cuda").manual_seed(seed)
        # the gradient of an L2 loss: differences of two noisy images
        st.dimg = torch.randn((case["h"], case["w"], 3), generator=g, device="cuda") * 0.2
    elif kind == "fit":
        jobs, st.targets, st.images, st.params = [], [], [], []
        r = np.random.default_rng(seed)
        for k in range(case["scenes"]):
            sc = _soup(case["spheres"], case["w"], case["h"], case["spp"], case["bounces"], seed * 100 + k, 1 + k % 4)
            s = st.scene(sc)
            jobs.append((s, sc.camera, sc.render))
            st.targets.append(torch.empty((case["h"], case["w"], 3), dtype=torch.float32, device="cuda"))
            st.images.append(torch.empty_like(st.targets[-1]))
            s.render_device(sc.camera, sc.render, st.targets[-1].data_ptr())
            x = s.get_params()
            m = 5 * len(sc.materials)
            x[:m] = np.clip(x[:m] + r.normal(0, 0.1, m), 0.05, 1.0)
            st.params.append(x.astype(np.float32))
        st.ctx.fit_prepare(jobs, [t.data_ptr() for t in st.targets], [t.data_ptr() for t in st.images])
    elif kind in ("closest", "any"):
        sc = _soup(case["spheres"], 64, 64, 1, 1, seed)
        st.s = st.scene(sc)
        st.o, st.d, st.t = _rays(sc, case["rays"], seed, kind == "any")
        if not case["host"]:
            st.o, st.d, st.t = (torch.from_numpy(x).cuda() for x in (st.o, st.d, st.t))
            n = case["rays"]
            st.hits = torch.empty(n, dtype=torch.uint8, device="cuda") if kind == "any" else \
                torch.empty((n, 4), dtype=torch.float32, device="cuda")
    elif kind == "animate":
        sc = _soup(case["spheres"], case["w"], case["h"], case["spp"], case["bounces"], seed)
        st.cam, st.rdesc = sc.camera, sc.render
        st.s = st.scene(sc, builder="device")
        p = sc.positions.reshape(-1, 3).astype(np.float64)
        moved = p + 0.2 * np.sin(p[:, [1, 2, 0]] * 0.35 + seed)
        st.moved = moved.astype(np.float32).reshape(-1, 9)
        st.normals = sc.normals
        st.image = torch.empty((case["h"], case["w"], 3), dtype=torch.float32, device="cuda")
    else:
        sc = _soup(case["spheres"], case["w"], case["h"], 1, 1, seed)
        st.cam, st.rdesc = sc.camera, sc.render
        st.s = st.scene(sc)
    torch.cuda.synchronize()
    return st


def run(st):
    case = st.case
    kind = case["kind"]
    if kind in ("room", "frame"):
        if case["host"]:
            return st.s.render(st.cam, st.rdesc, out=st.out)
        st.s.render_device(st.cam, st.rdesc, st.image.data_ptr())
        return st.image
    if kind == "batch":
        st.ctx.render_batch_device(st.jobs, [t.data_ptr() for t in st.images])
        return st.images
    if kind == "backward":
        return st.s.backward_device(st.cam, st.rdesc, st.dimg.data_ptr())
    if kind == "fit":
        grads, loss = st.ctx.fit_step(st.params)
        return {"gradients": grads, "loss": loss, "images": st.images}
    if kind == "closest":
        if case["host"]:
            h = st.s.trace_closest(st.o, st.d, st.t)
            return {"t": h["t"], "beta": h["beta"], "gamma": h["gamma"], "ref": h["ref"].view(np.int32)}
        lib, p = st.ctx.lib, ctypes.c_void_p
        st.ctx.check(lib.gb_trace_closest(st.ctx.h, st.s.h, case["rays"], p(st.o.data_ptr()), p(st.d.data_ptr()),
                                          p(st.t.data_ptr()), p(st.hits.data_ptr()), 1))
        return {"t": st.hits[:, 0], "beta": st.hits[:, 1], "gamma": st.hits[:, 2],
                "ref": st.hits[:, 3].view(torch.int32)}
    if kind == "any":
        if case["host"]:
            return st.s.trace_any(st.o, st.d, st.t)
        lib, p = st.ctx.lib, ctypes.c_void_p
        st.ctx.check(lib.gb_trace_any(st.ctx.h, st.s.h, case["rays"], p(st.o.data_ptr()), p(st.d.data_ptr()),
                                      p(st.t.data_ptr()), p(st.hits.data_ptr()), 1))
        return st.hits
    if kind == "animate":
        st.s.refit(st.moved, st.normals)
        st.s.render_device(st.cam, st.rdesc, st.image.data_ptr())
        return st.image
    if case["hybrid"]:
        return st.s.render_hybrid_direct(st.cam, st.rdesc, case["camera_samples"], case["light_samples"])
    return st.s.render_direct(st.cam, st.rdesc, case["light_samples"])


# ------------------------------------------------------------------- work --
# Operations per ray: a ray of these scenes visits a few nodes per level of an
# 8-wide tree (24 operations per child box, 8 boxes) and tests about two
# triangles (30 operations); a shaded vertex takes about 300 operations.

def _ray_flops(tris: int) -> float:
    return max(1.0, 0.9 * math.log2(max(tris, 2) / 2.0) * 0.6) * 8 * 24 + 2.3 * 30


def _frame_work(tris: int, pixels: int, spp: int, bounces: int, closed: bool) -> dict:
    paths = float(pixels) * spp
    # closed room: most paths take every bounce; soup: about 0.7 further segments
    more = 0.8 * (bounces - 1) if closed else min(0.7, 0.35 * bounces)
    closest, shaded = paths * (1.0 + more), paths * ((1.0 + more) if closed else 0.7)
    return {"bytes": tris * (36 + 36 + 4) + pixels * 12.0,
            "flops": closest * _ray_flops(tris) + shaded * (0.8 * _ray_flops(tris) + 300)}


def work(case: dict) -> dict:
    kind = case["kind"]
    tris = 48 if kind == "room" else 1280 * case.get("spheres", 0) + 10
    if kind == "room":
        return _frame_work(48, case["w"] * case["h"], case["spp"], case["bounces"], True)
    if kind in ("frame", "animate"):
        return _frame_work(tris, case["w"] * case["h"], case["spp"], case["bounces"], False)
    if kind == "batch":
        r = np.random.default_rng(case["scenes"] * 1_000_003 + case["max_tris"])
        tot = {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["scenes"]):
            t = math.exp(r.uniform(math.log(1_000), math.log(case["max_tris"])))
            res = int(r.choice([64, 128, 256, 512]))
            spp = int(r.choice([4, 16, 64])) if res < 512 else 4
            r.integers(1, 5)
            w = _frame_work(1280 * max(1, round(t / 1280)) + 10, res * res, spp, case["bounces"], False)
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    if kind == "backward":
        w = _frame_work(tris, case["w"] * case["h"], case["spp"], case["bounces"], False)
        paths = case["w"] * case["h"] * case["spp"]
        return {"bytes": w["bytes"], "flops": w["flops"] + paths * 0.7 * 600}
    if kind == "fit":
        w = _frame_work(tris, case["w"] * case["h"], case["spp"], case["bounces"], False)
        paths = case["w"] * case["h"] * case["spp"]
        return {"bytes": case["scenes"] * (w["bytes"] + 12.0 * case["w"] * case["h"]),
                "flops": case["scenes"] * (2 * w["flops"] + paths * 0.7 * 600)}
    if kind in ("closest", "any"):
        return {"bytes": tris * 36 + case["rays"] * (28.0 + (16 if kind == "closest" else 1)),
                "flops": case["rays"] * _ray_flops(tris)}
    pixels = case["w"] * case["h"]
    cams = case["camera_samples"] if case["hybrid"] else 1
    return {"bytes": tris * 76 + pixels * 12.0,
            "flops": pixels * cams * (_ray_flops(tris) + 0.6 * case["light_samples"] * (0.8 * _ray_flops(tris) + 60))}


# ------------------------------------------------------------------ exact --
# The same results in 64 bits: rays against every triangle (no tree), and for
# the Lambert room the whole path: camera, MRG32k3a / Halton draws, light
# sample, cosine lobe, clamped throughput, mean over the samples.

_M1, _M2 = 4294967087, 4294944443  # L'Ecuyer 1999, MRG32k3a


def _matmul(a, b, m):
    return [[sum(a[i][k] * b[k][j] for k in range(3)) % m for j in range(3)] for i in range(3)]


def _mrg_start(n: int) -> tuple:
    """States of streams 0 .. n-1, 2^76 steps apart, from the all-12345 seed."""
    A = [[0, 1, 0], [0, 0, 1], [_M1 - 810728, 1403580, 0]], [[0, 1, 0], [0, 0, 1], [_M2 - 1370589, 0, 527612]]
    out = []
    for a, m in zip(A, (_M1, _M2)):
        for _ in range(76):
            a = _matmul(a, a, m)
        s = np.full((n, 3), 12345, np.uint64)
        idx = np.arange(n)
        for bit in range(max(1, n.bit_length())):
            on = ((idx >> bit) & 1).astype(bool)
            t = np.zeros_like(s[on])
            for i in range(3):
                for k in range(3):
                    t[:, i] = (t[:, i] + s[on, k] * np.uint64(a[i][k]) % np.uint64(m)) % np.uint64(m)
            s[on] = t
            a = _matmul(a, a, m)
        out.append(s)
    return tuple(out)


def _mrg_draws(n: int, updates: int) -> np.ndarray:
    """(updates, n, 3) uniforms in (0, 1], rounded to float as a float sampler gives them."""
    s1, s2 = _mrg_start(n)
    u = np.empty((updates * 3, n))
    m1, m2 = np.uint64(_M1), np.uint64(_M2)
    for k in range(updates * 3):
        p1 = (np.uint64(1403580) * s1[:, 1] + (m1 - np.uint64(810728)) * s1[:, 0] % m1) % m1
        s1 = np.stack([s1[:, 1], s1[:, 2], p1], 1)
        p2 = (np.uint64(527612) * s2[:, 2] + (m2 - np.uint64(1370589)) * s2[:, 0] % m2) % m2
        s2 = np.stack([s2[:, 1], s2[:, 2], p2], 1)
        z = np.where(p1 > p2, p1 - p2, p1 + m1 - p2)
        u[k] = (z.astype(np.float64) / _M1).astype(np.float32)
    return u.reshape(updates, 3, n).transpose(0, 2, 1)


def _halton(i: np.ndarray, base: int) -> np.ndarray:
    r, f, i = np.zeros(i.shape), 1.0 / base, i.copy()
    while (i > 0).any():
        r += f * (i % base)
        i //= base
        f /= base
    return r


def _cross(a, b):
    return torch.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1], a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                        a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _brute(tri, o, d, tmax, pairs: int = 1 << 27):
    """Closest hit of every ray over every triangle (Moller & Trumbore 1997);
    the lowest index wins a tie.  tri (n, 3, 3), o, d (m, 3), tmax (m)."""
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    m, step = o.shape[0], max(1, pairs // max(1, tri.shape[0]))
    T = torch.full((m,), math.inf, dtype=torch.float64, device=o.device)
    B, G = torch.zeros_like(T), torch.zeros_like(T)
    R = torch.full((m,), -1, dtype=torch.int64, device=o.device)
    # t, u, v and the determinant are triple products of o, d and per-triangle
    # vectors, so each is a matrix product over all (ray, triangle) pairs:
    # det = -d . n, t = (o - v0) . n / det, u = d . (e2 x (o - v0)) / det,
    # v = d . ((o - v0) x e1) / det
    n = _cross(e1, e2)
    c0 = (n * v0).sum(1)
    e2v, e1v = _cross(e2, v0), _cross(e1, v0)
    for a in range(0, m, step):
        oo, dd, lim = o[a:a + step], d[a:a + step], tmax[a:a + step]
        od = _cross(oo, dd)  # o x d
        det = -(dd @ n.T)
        inv = 1.0 / det
        t = (oo @ n.T - c0) * inv
        u = (od @ e2.T - dd @ e2v.T) * inv
        v = (dd @ e1v.T - od @ e1.T) * inv
        bad = (det == 0) | ~(u >= 0) | ~(v >= 0) | ~(u + v <= 1) | ~(t > 0) | ~(t <= lim[:, None])
        t = torch.where(bad, math.inf, t)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        r = torch.arange(t.shape[0], device=o.device)
        T[a:a + step] = best
        B[a:a + step] = torch.where(hit, u[r, k], 0.0)
        G[a:a + step] = torch.where(hit, v[r, k], 0.0)
        R[a:a + step] = torch.where(hit, k, -1)
    return T, B, G, R


def _norm(a):
    return a / a.norm(dim=-1, keepdim=True)


def _room_exact(case: dict, seed: int) -> np.ndarray:
    sc = _room(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    w, h, spp, L = case["w"], case["h"], case["spp"], case["bounces"]
    n = w * h
    pool = torch.as_tensor(_mrg_draws(n, spp * L), **f64)
    tri = torch.as_tensor(sc.positions.reshape(-1, 3, 3), **f64)
    nrm = torch.as_tensor(sc.normals.reshape(-1, 3, 3)[:, 0], **f64)
    alb = torch.as_tensor(np.array([m["diffuse"] for m in sc.materials], np.float32), **f64)[
        torch.as_tensor(sc.material_index.astype(np.int64), device=dev)]
    roff, soff = float(np.float32(sc.render["ray_offset"])), float(np.float32(sc.render["shadow_offset"]))
    light = sc.lights[0]
    col = torch.as_tensor(np.array(light["col"], np.float32), **f64)
    ctr = torch.as_tensor(np.array(light["center"], np.float32), **f64)
    lw, lh = light["wh"]
    ldir = torch.tensor([0.0, -1.0, 0.0], **f64)
    cam = dict(sc.camera, pos=np.array(sc.camera["pos"], np.float32))
    pos, W, U, V, th = (torch.as_tensor(x, **f64) for x in _camera(cam))
    i = np.arange(n)
    hal = torch.as_tensor(np.stack([_halton(i + 1, 2), _halton(i + 1, 3)], 1), **f64)
    px, py = torch.as_tensor(i % w, **f64), torch.as_tensor(i // w, **f64)
    inf = torch.full((n,), FLT_MAX, **f64)
    image = torch.zeros((n, 3), **f64)
    for p in range(spp):
        j = pool[p]
        u = ((px + j[:, 0]) / w * 2 - 1) * (th * w / h)
        v = ((py + j[:, 1]) / h * 2 - 1) * th
        d = _norm(u[:, None] * U + v[:, None] * V + W)
        o = pos.expand(n, 3)
        tp, acc = torch.ones((n, 3), **f64), torch.zeros((n, 3), **f64)
        alive = torch.ones(n, dtype=torch.bool, device=dev)
        for b in range(L):
            t, beta, gamma, ref = _brute(tri, o, d, inf)
            miss = alive & (ref < 0)
            acc = torch.where((miss & (tp == 1).all(1))[:, None], acc + tp, acc)
            alive = alive & (ref >= 0)
            r = ref.clamp(min=0)
            P = (1 - beta - gamma)[:, None] * tri[r, 0] + beta[:, None] * tri[r, 1] + gamma[:, None] * tri[r, 2]
            Ng = nrm[r]
            rnd = pool[p * L + b]
            lr = hal if case["halton"] else rnd
            ls = ctr + torch.stack([(lr[:, 0] - 0.5) * lw, torch.zeros(n, **f64), (lr[:, 1] - 0.5) * lh], 1)
            to = ls - P
            ln = to.norm(dim=1)
            to = to / ln[:, None]
            g = lw * lh * (Ng * to).sum(1).clamp(min=0) * (-(ldir * to).sum(1)).clamp(min=0) / (ln * ln)
            so = P + soff * to
            occ = _brute(tri, so, to, ln)[3] >= 0
            N = torch.where(((d * Ng).sum(1) > 0)[:, None], -Ng, Ng)
            f = alb[r] * (1.0 / math.pi)
            add = f * (to * N).sum(1).abs()[:, None] * tp * col * g[:, None]
            acc = torch.where((alive & ~occ)[:, None], acc + add, acc)
            # cosine lobe around N in the tangent frame of the unflipped normal
            sg = torch.where(torch.signbit(Ng[:, 2]), -1.0, 1.0).to(torch.float64)
            a = -1.0 / (sg + Ng[:, 2])
            c = Ng[:, 0] * Ng[:, 1] * a
            Tv = torch.stack([1 + sg * Ng[:, 0] ** 2 * a, sg * c, -sg * Ng[:, 0]], 1)
            Bv = torch.stack([c, sg + Ng[:, 1] ** 2 * a, -Ng[:, 1]], 1)
            ru, ph = rnd[:, 0].sqrt(), 2 * math.pi * rnd[:, 1]
            z = (1 - rnd[:, 0]).clamp(min=0).sqrt()
            wi = _norm((ru * ph.cos())[:, None] * Tv + (ru * ph.sin())[:, None] * Bv + z[:, None] * N)
            pdf = z / math.pi
            tp = torch.where(alive[:, None], (tp * f * (wi * N).sum(1).abs()[:, None] / pdf[:, None]).clamp(max=1.0), tp)
            alive = alive & (pdf > 0)
            o, d = P + roff * N, wi
        image = (image * p + acc) / (p + 1)
    return image.reshape(h, w, 3).cpu().numpy()


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "room" and case["w"] * case["h"] * case["spp"] * case["bounces"] <= 1 << 23:
        return _room_exact(case, seed)
    if kind in ("closest", "any") and case["rays"] * (1280.0 * case["spheres"] + 10) <= 2e10:
        sc = _soup(case["spheres"], 64, 64, 1, 1, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        o, d, t = (torch.as_tensor(x, dtype=torch.float64, device=dev)
                   for x in _rays(sc, case["rays"], seed, kind == "any"))
        tri = torch.as_tensor(sc.positions.reshape(-1, 3, 3), dtype=torch.float64, device=dev)
        T, B, G, R = _brute(tri, o, d, t)
        if kind == "any":
            return None  # bytes: equal to the start's
        T = torch.where(R < 0, FLT_MAX, T)
        # ids are whole numbers: equal to the start's
        return {"t": T.cpu().numpy(), "beta": B.cpu().numpy(), "gamma": G.cpu().numpy(), "ref": None}
    # textured / principled frames, batches, gradients: paths through 64-bit
    # arithmetic and every triangle would take minutes
    return None
