"""The calls this renderer's users make, as cases that can be timed.

A case is a dict of plain values; ``listed()`` names the representative ones
and ``draw(rng)`` gives another of the same ranges.  ``prepare(case, seed)``
builds what a program has in hand before the call (a context with the scene
uploaded, films, ray arrays), ``run(state)`` makes one call through the public
binding or the C ABI and returns its outputs, ``work(case)`` states the bytes
and operations the call cannot do without, and ``exact(case, seed)`` evaluates
ray queries in 64 bits.

Kinds of call:

* ``render``  — ``Context.render``: one call adds ``spp`` samples per pixel to
                the film.  Each pass takes the next sample range, as a
                progressive view does.  ``film`` is "host" (numpy films, copied
                in and out by the call) or "device".
* ``cached``  — the same with the radiance cache: the call also trains the
                network, whose weights are read back.
* ``batch``   — ``Context.render_batch``: requests of different sizes, cameras
                and sample counts on one scene.
* ``queries`` — ``pt_trace_closest`` / ``pt_trace_shadow`` on device arrays of
                incoherent rays (visibility and occlusion queries).
* ``load``    — ``Context.upload`` of a scene followed by a small one-sample
                preview: opening or editing a scene.

Scenes (``pbrt_b200.scenes``): ``room`` (Cornell box with a Disney sphere),
``spheres`` (a grid of Disney UV spheres under an HDR sky), ``fog`` (displaced
spheres of Disney and hair materials, a fog box, a tree larger than the L2),
``hair`` (hair ribbons in a heterogeneous medium) and ``textured`` (every
texture map, an alpha cut-out).
"""

from __future__ import annotations

import ctypes as C
import functools
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "pbrt-renderer-_b200")


def _pt():
    """The binding, registered as pbrt_b200 (its folder is no identifier)."""
    if "pbrt_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("pbrt_b200", os.path.join(_PKG, "__init__.py"),
                                                      submodule_search_locations=[_PKG])
        m = importlib.util.module_from_spec(spec)
        sys.modules["pbrt_b200"] = m
        spec.loader.exec_module(m)
    return sys.modules["pbrt_b200"]


def _scenes():
    _pt()
    return importlib.import_module("pbrt_b200.scenes")


def listed():
    return [
        # A material thumbnail: the smallest call, host film, launches and latency only.
        {"name": "thumbnail_room", "kind": "render", "scene": "room", "size": 0, "width": 64, "height": 64, "spp": 1,
         "depth": 8, "film": "host"},
        # A small still of a closed room, where paths run to the depth limit.
        {"name": "still_room", "kind": "render", "scene": "room", "size": 0, "width": 256, "height": 256, "spp": 16,
         "depth": 8, "film": "device"},
        # One sample per pixel of an interactive view, refined call by call.
        {"name": "preview_spheres", "kind": "render", "scene": "spheres", "size": 8, "width": 1280, "height": 720,
         "spp": 1, "depth": 16, "film": "device"},
        # A final-quality frame: the largest call.
        {"name": "frame_spheres", "kind": "render", "scene": "spheres", "size": 8, "width": 1280, "height": 720,
         "spp": 64, "depth": 16, "film": "device"},
        # A scene larger than the L2 with a homogeneous medium and two material families, odd image size.
        {"name": "frame_fog", "kind": "render", "scene": "fog", "size": 36, "width": 1917, "height": 1079, "spp": 4,
         "depth": 16, "film": "device"},
        # Hair in a heterogeneous medium, the wavefront option.
        {"name": "hair_wavefront", "kind": "render", "scene": "hair", "size": 4000, "width": 512, "height": 512,
         "spp": 8, "depth": 16, "film": "device", "media_wavefront": True},
        # The same scene as a caller gets it by default (the reference's order of draws), small.
        {"name": "hair_default", "kind": "render", "scene": "hair", "size": 4000, "width": 192, "height": 192,
         "spp": 2, "depth": 16, "film": "host"},
        # Texture maps and an alpha cut-out, white-noise sampler and alias-table light sampling.
        {"name": "textured", "kind": "render", "scene": "textured", "size": 0, "width": 641, "height": 479, "spp": 12,
         "depth": 16, "film": "host", "white_noise": True, "alias": True},
        # One call of a cached progressive render: queries, training records, four optimiser steps.
        {"name": "cached_spheres", "kind": "cached", "scene": "spheres", "size": 8, "width": 1280, "height": 720,
         "spp": 8, "depth": 16, "film": "device"},
        # A serving batch: requests of log-uniform sizes and 4 .. 64 samples.
        {"name": "batch_spheres", "kind": "batch", "scene": "spheres", "size": 8, "requests": 12, "side_max": 512,
         "spp_max": 64, "depth": 16},
        # Incoherent closest-hit queries.
        {"name": "queries_closest", "kind": "queries", "scene": "spheres", "size": 8, "rays": 1 << 20, "shadow": False},
        # Opening a scene of 1.3 million triangles with an envmap, up to its first picture.
        {"name": "load_spheres", "kind": "load", "scene": "spheres", "size": 8, "width": 320, "height": 180, "spp": 1,
         "depth": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 5 + ["cached", "batch", "queries", "load"])
    if kind == "render":
        scene = rng.choice(["room", "spheres", "spheres", "fog", "hair", "textured"])
        c = {"kind": kind, "scene": scene, "size": 0, "width": 0, "height": 0, "spp": 0,
             "depth": rng.randint(4, 8) if scene == "room" else rng.randint(8, 16),
             "film": rng.choice(["host", "device"])}
        if scene == "room":
            c["width"], c["height"], c["spp"] = _log_int(rng, 48, 640), _log_int(rng, 48, 480), _log_int(rng, 1, 16)
        elif scene == "spheres":
            c["size"] = rng.randint(2, 8)
            c["width"], c["height"], c["spp"] = _log_int(rng, 160, 1280), _log_int(rng, 90, 720), _log_int(rng, 1, 64)
        elif scene == "fog":
            c["size"] = rng.randint(9, 36)
            c["width"], c["height"], c["spp"] = _log_int(rng, 320, 1920), _log_int(rng, 180, 1080), _log_int(rng, 1, 4)
        elif scene == "hair":
            c["size"] = 4000
            c["media_wavefront"] = rng.random() < 0.6
            side, spp = (512, 8) if c["media_wavefront"] else (192, 2)
            c["width"], c["height"], c["spp"] = _log_int(rng, 48, side), _log_int(rng, 48, side), rng.randint(1, spp)
        else:
            c["width"], c["height"], c["spp"] = _log_int(rng, 96, 800), _log_int(rng, 72, 600), _log_int(rng, 1, 16)
        if scene != "hair":
            c["white_noise"] = rng.random() < 0.25
            c["alias"] = rng.random() < 0.25
        return c
    if kind == "cached":
        return {"kind": kind, "scene": "spheres", "size": rng.randint(4, 8), "width": _log_int(rng, 320, 1280),
                "height": _log_int(rng, 180, 720), "spp": rng.randint(2, 8), "depth": rng.randint(8, 16),
                "film": rng.choice(["host", "device"])}
    if kind == "batch":
        return {"kind": kind, "scene": rng.choice(["room", "spheres"]), "size": 8, "requests": rng.randint(2, 16),
                "side_max": rng.randint(128, 512), "spp_max": rng.randint(8, 64), "depth": rng.randint(6, 12)}
    if kind == "queries":
        return {"kind": kind, "scene": "spheres", "size": rng.randint(4, 8), "rays": _log_int(rng, 1 << 14, 1 << 20),
                "shadow": rng.random() < 0.5}
    return {"kind": kind, "scene": "spheres", "size": rng.randint(2, 8), "width": _log_int(rng, 160, 480),
            "height": _log_int(rng, 90, 270), "spp": 1, "depth": rng.randint(8, 16)}


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _hair_geometry(strands):
    return _scenes().hair_volume(64, 64, strands=strands, segments=32, seed=0, grid_n=128)


def _build_scene(case, seed):
    """(scene, camera at the case's aspect ratio) with the seed's materials, placement and media."""
    pt, scenes = _pt(), _scenes()
    name, size = case["scene"], case["size"]
    w, h = case.get("width", 16), case.get("height", 9)
    rng = np.random.default_rng(seed)
    if name == "room":
        sc, cam = scenes.cornell(w, h)
        sc.materials[4].albedo[:] = tuple(rng.uniform(0.2, 0.9, 3))
        sc.materials[4].roughness = float(rng.uniform(0.1, 0.9))
        return sc, cam
    if name == "spheres":
        return scenes.disney_spheres(w, h, grid=size, seed=seed)
    if name == "fog":
        return scenes.radiance_cache_scene(w, h, instances=size, seed=seed)
    if name == "textured":
        return scenes.textured_scene(w, h, seed=seed)
    base, _ = _hair_geometry(size)
    mats = []
    for m in base.materials:
        n = pt.pt_material()
        C.memmove(C.byref(n), C.byref(m), C.sizeof(m))
        n.albedo[:] = tuple(scenes.eumelanin_to_color(rng.uniform(0.3, 6.0), 0.3))
        mats.append(n)
    vol = pt.pt_volume()
    C.memmove(C.byref(vol), C.byref(base.volumes[0]), C.sizeof(vol))
    vol.phase_g = float(rng.uniform(0.0, 0.8))
    vol.sigma_s[:] = (float(rng.uniform(1.4, 1.8)),) * 3
    grid = np.roll(base.grid_arrays[0], int(rng.integers(0, 16)), axis=2)
    sc = pt.Scene(base.positions, base.indices, mats, normals=base.normals, texcoords=base.texcoords,
                  tangents=base.tangents, env_rgb=base.env_rgb, volumes=[vol], grids=[grid])
    return sc, scenes.look_at_camera((0.0, 0.0, 4.0), (0.0, 0.2, 0.0), (0, 1, 0), 45.0, w / h)


def _orbit_camera(rng, scene, aspect):
    """A view of the room or of the sphere grid, as a serving request asks for."""
    scenes = _scenes()
    if scene == "room":
        eye = (rng.uniform(-0.7, 0.7), rng.uniform(0.3, 1.7), rng.uniform(0.6, 0.95))
        to = (rng.uniform(-0.5, 0.5), rng.uniform(0.2, 1.2), rng.uniform(-1.0, -0.2))
        return scenes.look_at_camera(eye, to, (0, 1, 0), float(rng.uniform(40, 70)), aspect)
    az, el, dist = rng.uniform(0, 2 * np.pi), np.radians(rng.uniform(15, 50)), rng.uniform(12, 30)
    eye = (dist * np.cos(el) * np.sin(az), 1.0 + dist * np.sin(el), dist * np.cos(el) * np.cos(az))
    to = (rng.uniform(-3, 3), 1.0, rng.uniform(-3, 3))
    return scenes.look_at_camera(eye, to, (0, 1, 0), float(rng.uniform(30, 50)), aspect)


def _rays(case, seed):
    """Origins in a slab around the sphere grid, uniform directions: 8 floats per ray."""
    n, half = case["rays"], (case["size"] - 1) * 1.25 + 2.0
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    r = torch.empty((n, 8), device="cuda")
    r[:, 0:3] = torch.rand((n, 3), generator=g, device="cuda") * torch.tensor([2 * half, 4.0, 2 * half], device="cuda")
    r[:, 0:3] -= torch.tensor([half, 0.5, half], device="cuda")
    r[:, 3] = 0.001
    d = torch.randn((n, 3), generator=g, device="cuda")
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    r[:, 7] = 1e4
    return r


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    pt = _pt()
    sc, cam = _build_scene(case, seed)
    ctx = pt.Context(torch.cuda.current_device())
    s = {"case": case, "ctx": ctx}
    kind = case["kind"]
    if kind != "load":
        ctx.upload(sc)
    if kind in ("render", "cached", "load"):
        flags = pt.PT_RENDER_MEDIA_WAVEFRONT if case.get("media_wavefront") else 0
        flags |= pt.PT_RENDER_RADIANCE_CACHE if kind == "cached" else 0
        s["params"] = pt.render_params(case["width"], case["height"], case["spp"], cam, max_depth=case["depth"],
                                       sample_offset=(seed % 1024) * 64, flags=flags,
                                       rng_kind=pt.PT_RNG_PCG_HASH if case.get("white_noise") else pt.PT_RNG_SOBOL_OWEN,
                                       env_sampling=pt.PT_ENV_ALIAS if case.get("alias") else pt.PT_ENV_CDF)
        shape = (case["height"], case["width"], 4)
        if case.get("film") == "device":
            s["film"] = (torch.zeros(shape, device="cuda"), torch.zeros(shape, device="cuda"))
        elif kind != "load":
            s["film"] = (np.zeros(shape, np.float32), np.zeros(shape, np.float32))
        if kind == "cached":
            ctx.cache_init(pt.cache_params(train_records=65536, rough_threshold=0.1, learning_rate=1e-2, ema=0.97,
                                           max_train_fraction=0.1, seed=seed % 65536))
        if kind == "load":
            s["scene"] = sc
    elif kind == "batch":
        rng = np.random.default_rng(seed + 7)
        s["requests"], s["films"] = [], []
        # the shape of the batch is the case's own (the launch plan follows it); views and offsets are the seed's
        shape_rng = np.random.default_rng(case["requests"] * 1000 + case["side_max"])
        for _ in range(case["requests"]):
            w, h = (int(round(math.exp(shape_rng.uniform(math.log(64), math.log(case["side_max"]))))) for _ in range(2))
            spp = int(shape_rng.integers(4, case["spp_max"] + 1))
            s["requests"].append(pt.render_params(w, h, spp, _orbit_camera(rng, case["scene"], w / h),
                                                  max_depth=case["depth"], sample_offset=int(rng.integers(0, 4096))))
            s["films"].append((torch.zeros((h, w, 4), device="cuda"), torch.zeros((h, w, 4), device="cuda")))
    else:
        s["rays"] = _rays(case, seed)
        n = case["rays"]
        if case["shadow"]:
            s["out"] = (torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros((n, 3), device="cuda"))
        else:
            s["out"] = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the films and rays are torch's; the context has a stream of its own
    return s


def run(state):
    pt, ctx, case = _pt(), state["ctx"], state["case"]
    kind = case["kind"]
    if kind in ("render", "cached"):
        p, (fs, fc) = state["params"], state["film"]
        if case["film"] == "device":
            ctx.render(p, fs.data_ptr(), fc.data_ptr(), location=pt.PT_MEM_DEVICE)
        else:
            ctx.render(p, fs, fc)
        p.sample_offset += p.spp
        if kind == "cached":
            return {"film": fs, "weights": ctx.cache_weights()}
        return {"film": fs, "compensation": fc}
    if kind == "batch":
        ptrs = [(a.data_ptr(), b.data_ptr()) for a, b in state["films"]]
        ctx.render_batch(state["requests"], ptrs, location=pt.PT_MEM_DEVICE)
        for p in state["requests"]:
            p.sample_offset += p.spp
        return [a for a, _ in state["films"]]
    if kind == "queries":
        f = C.POINTER(C.c_float)
        rays = C.cast(state["rays"].data_ptr(), f)
        if case["shadow"]:
            occ, tr = state["out"]
            ctx._check(ctx.L.pt_trace_shadow(ctx.h, rays, case["rays"], C.cast(occ.data_ptr(), C.POINTER(C.c_uint32)),
                                             C.cast(tr.data_ptr(), f), pt.PT_MEM_DEVICE))
            return {"occluded": occ, "transmission": tr}
        o = state["out"]
        ctx._check(ctx.L.pt_trace_closest(ctx.h, rays, case["rays"], C.cast(o.data_ptr(), C.POINTER(pt.pt_hit)),
                                          pt.PT_MEM_DEVICE))
        v = o.view(torch.float32)
        return {"t": v[:, 0], "u": v[:, 3], "v": v[:, 4], "ids": o[:, 1:3], "hit": o[:, 5]}
    ctx.upload(state["scene"])
    film, _, _ = ctx.render(state["params"])
    return {"film": film}


# ---------------------------------------------------------------------------
# work and 64-bit results
# ---------------------------------------------------------------------------
_TRIS = {"room": lambda c: 1294, "spheres": lambda c: 20480 * c["size"] ** 2, "fog": lambda c: 81920 * c["size"] + 4,
         "hair": lambda c: 64 * c["size"], "textured": lambda c: 2310}
# rays per path (extension + shadow) measured on these scenes, rounded; per ray the box tests of a balanced
# 8-wide tree (8 children x 12 operations a level) and two triangle tests, per path vertex its shading
_RAYS = {"room": 9.0, "spheres": 1.7, "fog": 3.0, "hair": 6.0, "textured": 3.0}
_TRI_TEST, _SHADE = 45, 400


def _ray_flops(tris):
    return 96.0 * max(1.0, math.log(max(tris, 8) / 3.0, 8)) + 2 * _TRI_TEST


def work(case):
    tris = _TRIS[case["scene"]](case)
    kind = case["kind"]
    if kind == "queries":
        n = case["rays"]
        return {"bytes": n * (32 + (16 if case["shadow"] else 24)) + min(48 * tris, 48 * n), "flops": n * _ray_flops(tris)}
    if kind == "batch":
        rng = np.random.default_rng(case["requests"] * 1000 + case["side_max"])
        pix = paths = 0
        for _ in range(case["requests"]):
            w, h = (int(round(math.exp(rng.uniform(math.log(64), math.log(case["side_max"]))))) for _ in range(2))
            spp = int(rng.integers(4, case["spp_max"] + 1))
            pix, paths = pix + w * h, paths + w * h * spp
    else:
        pix = case["width"] * case["height"]
        paths = pix * case["spp"]
    rays = paths * _RAYS[case["scene"]]
    # film sum and compensation read and written; each triangle that a path can touch read once
    b = 64.0 * pix + 48.0 * min(tris, rays)
    f = rays * (_ray_flops(tris) + _SHADE)
    if kind == "cached":  # about one query per three paths, 65,536 records through forward and backward passes
        f += paths / 3.0 * 43008 + 65536 * 120832.0
    if kind == "load":  # the scene's host arrays in (vertices 44 bytes, indices, envmap), nodes and triangles out
        b += tris * (22 + 12 + 71.0) + 2048 * 1024 * 28.0
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """Closest-hit distances in float64 by brute force over each sphere's triangles (rays that meet its bounding
    sphere).  Films have no such value: a path's random decisions are part of the result."""
    if case["kind"] != "queries" or case["shadow"]:
        return None
    sc, _ = _build_scene(case, seed)
    rays = _rays(case, seed).double()
    o, d, tmin = rays[:, 0:3], rays[:, 4:7], rays[:, 3]
    pos = torch.from_numpy(sc.positions).cuda().double()
    idx = torch.from_numpy(sc.indices.astype(np.int64)).cuda().view(-1, 3)
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device="cuda")
    for m in sc.materials:
        f = idx[m.indexOffset // 3:(m.indexOffset + m.indexCount) // 3] + m.vertexOffset
        p0 = pos[f[:, 0]]
        e1, e2 = pos[f[:, 1]] - p0, pos[f[:, 2]] - p0
        c = 0.5 * (p0.amin(0) + p0.amax(0))
        rad = (p0 - c).norm(dim=1).max() + e1.norm(dim=1).max()
        oc = c - o
        t_mid = (oc * d).sum(1)
        near = torch.nonzero((oc - t_mid[:, None] * d).norm(dim=1) <= rad).flatten()
        for part in near.split(2048):
            oo, dd = o[part], d[part]
            # scalar triple products with the terms that do not depend on the ray taken out
            n = torch.linalg.cross(e1, e2)
            det = -(dd @ n.T)
            s_n = (oo @ n.T) - (p0 * n).sum(1)
            q = torch.linalg.cross(oo, dd)
            # u det = (s x d) . e2 and v det = -(s x d) . e1, with s = o - p0
            u = (q @ e2.T) - (dd @ torch.linalg.cross(e2, p0).T)
            v = -((q @ e1.T) - (dd @ torch.linalg.cross(e1, p0).T))
            inv = 1.0 / det
            t, u, v = s_n * inv, u * inv, v * inv
            ok = (det.abs() > 1e-12) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin[part][:, None])
            best[part] = torch.minimum(best[part], torch.where(ok, t, math.inf).amin(1))
    return {"t": torch.where(torch.isinf(best), 0.0, best), "u": None, "v": None, "ids": None, "hit": None}
