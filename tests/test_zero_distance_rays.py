"""Rays that start on a plane of a box and leave it at distance zero: the box
ends at t = -0 where the ray begins at tmin = +0, which counts as entered.
Both forms of a query (8 lanes per ray up to 18,944 rays, one lane above)
against the oracle: the floor, the left and the back wall of the room are the
lower planes of the boxes they lie in, and a ray from them outwards hits at
t = 0."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 148 * 32 * 4  # queries up to this many rays take 8 lanes each


def wall_rays(sc, n, seed, tmax):
    """Rays from inside the axis-parallel triangles, along the axis (both ways)
    or slanted."""
    rng = np.random.default_rng(seed)
    tri = np.concatenate([sc.indices[m.indexOffset:m.indexOffset + m.indexCount].reshape(-1, 3) + m.vertexOffset
                          for m in sc.materials])
    p = sc.positions[tri]
    flat = np.stack([(p[:, 0, a] == p[:, 1, a]) & (p[:, 0, a] == p[:, 2, a]) for a in range(3)], 1)
    p, flat = p[flat.any(1)], flat[flat.any(1)]
    assert len(p) >= 12
    k = rng.integers(0, len(p), n)
    b = rng.dirichlet((4.0, 4.0, 4.0), n).astype(np.float32)  # well inside: no ties with a neighbour
    o = (p[k] * b[:, :, None]).sum(1).astype(np.float32)
    axis = flat[k].argmax(1)
    row = np.arange(n)
    o[row, axis] = p[k, 0, axis]
    d = np.where(rng.uniform(size=n)[:, None] < 0.5, 0.0, rng.normal(size=(n, 3)) * 0.3)
    d[row, axis] = rng.choice([-1.0, 1.0], n)
    r = np.zeros((n, 8), np.float32)
    r[:, :3], r[:, 4:7], r[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), tmax
    return r


@pytest.mark.parametrize("tmax", [1e20, 0.0, -0.0])
@pytest.mark.parametrize("n", [1000, LIMIT, LIMIT + 1])
@pytest.mark.parametrize("plan", [0, 1])
def test_rays_leaving_a_box_at_zero(n, tmax, plan, pt, scenes, ctx, oracle):
    sc = scenes.cornell(16, 16)[0]
    ctx.debug_set(pt.PT_DEBUG_WIDE_PLAN, plan)
    try:
        ctx.upload(sc)
    finally:
        ctx.debug_set(pt.PT_DEBUG_WIDE_PLAN, 0)
    oracle.load(sc)
    r = wall_rays(sc, n, 3, tmax)
    hg, ho = ctx.trace_closest(r), oracle.trace_closest(r)
    assert (ho["hit"] == 1).all() and (ho["t"] == 0.0).all()
    for f in ("hit", "mesh", "prim", "t", "u", "v"):
        assert np.array_equal(hg[f], ho[f]), f
    assert np.array_equal(ctx.trace_shadow(r)[0], oracle.trace_shadow(r)[0])
