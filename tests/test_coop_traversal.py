"""Traversal with 8 lanes per ray (short queues) against the one-lane form: the
same rays queried a few at a time and all at once, and films rendered in
waves below and above the limit, must agree bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 148 * 32 * 4  # queries up to this many rays take 8 lanes each


def scene(scenes, name):
    if name == "spheres":
        return scenes.disney_spheres(64, 48, grid=3, slices=64, rings=33, env_w=64, env_h=32)[0]
    if name == "hair":
        return scenes.hair_volume(32, 32, strands=300, segments=8, grid_n=16)[0]
    return scenes.textured_scene(64, 48)[0] if name == "textured" else scenes.cornell(32, 32)[0]


def rays(sc, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = sc.positions.min(0), sc.positions.max(0)
    r = np.zeros((n, 8), np.float32)
    r[:, :3] = lo + (hi - lo) * rng.uniform(-0.1, 1.1, (n, 3))
    d = rng.normal(size=(n, 3))
    d[:: 7] = np.eye(3)[rng.integers(0, 3, len(d[:: 7]))] * rng.choice([-1, 1], (len(d[:: 7]), 1))  # along the axes
    at = sc.positions[rng.integers(0, len(sc.positions), n)] - r[:, :3]  # at vertices: ties and grazes
    d[:: 3] = at[:: 3]
    r[:, 4:7] = d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-6)
    r[:, 3] = rng.choice([0.0, 1e-3, -5.0], n)
    r[:, 7] = rng.choice([1e20, 1.5, 0.2, 0.0], n)
    return r


@pytest.mark.parametrize("name", ["cornell", "spheres", "textured", "hair"])
@pytest.mark.parametrize("part", [1, 3, 1000, LIMIT])
def test_queries_in_parts_equal_all_at_once(name, part, scenes, ctx):
    ctx.upload(scene(scenes, name))
    r = rays(ctx.scene, LIMIT + 1, 5)
    hits, (occ, tr) = ctx.trace_closest(r), ctx.trace_shadow(r)
    n = min(LIMIT, 40 * part)
    if name == "textured":  # the alpha test is seeded by a ray's place in its query
        n = part
    for k in range(0, n, part):
        q = r[k:k + part] if name != "textured" else r[:part]
        h, (o, t) = ctx.trace_closest(q), ctx.trace_shadow(q)
        assert h.tobytes() == hits[k:k + part].tobytes()
        assert np.array_equal(o, occ[k:k + part]) and np.array_equal(t, tr[k:k + part])


@pytest.mark.parametrize("name,depth", [("cornell", 8), ("cornell", 14), ("spheres", 16), ("textured", 13)])
def test_films_of_short_and_long_waves_agree(name, depth, pt, scenes, ctx):
    """173 x 139 x 2 paths: one wave above the limit at its first bounces, waves
    of 5,000 paths below it throughout; with and without the tail kernels."""
    w, h = 173, 139
    sc = scene(scenes, name)
    cam = {"spheres": scenes.disney_spheres(w, h, grid=3, slices=8, rings=5, env_w=8, env_h=4)[1],
           "textured": scenes.textured_scene(w, h)[1]}.get(name, scenes.cornell(w, h)[1])
    ctx.upload(sc)
    films = []
    for wave, tail in ((0, 0), (5000, 0), (0, 1), (5000, 1), (5000, 2)):
        ctx.debug_set(pt.PT_DEBUG_TAIL, tail)
        try:
            s, c, st = ctx.render(pt.render_params(w, h, 2, cam, max_depth=depth, sample_offset=4, wave_paths=wave))
        finally:
            ctx.debug_set(pt.PT_DEBUG_TAIL, 0)
        films.append((s, c, st.extension_rays, st.shadow_rays))
    for s, c, e, n in films[1:]:
        assert np.array_equal(s.view(np.uint32), films[0][0].view(np.uint32))
        assert np.array_equal(c.view(np.uint32), films[0][1].view(np.uint32))
        assert (e, n) == films[0][2:]
