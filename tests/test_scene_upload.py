"""Scene upload: index checks on the device, the scene's memory kept from one
upload to the next, the block-per-row envmap tables at their edges."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def film_of(pt, ctx, sc, cam, w=24, h=16):
    ctx.upload(sc)
    return ctx.render(pt.render_params(w, h, 2, cam, max_depth=5))[0]


@pytest.mark.parametrize("mesh,corner", [(0, 0), (1, 2), (4, 1)])
def test_index_out_of_range_is_refused(mesh, corner, pt, scenes, ctx):
    """The first index past a mesh's vertices, in a mesh with and without other
    meshes before it; the context renders a good scene afterwards."""
    sc, cam = scenes.cornell(24, 16)
    want = film_of(pt, ctx, sc, cam)
    bad, _ = scenes.cornell(24, 16)
    m = bad.materials[mesh]
    at = m.indexOffset + m.indexCount - 3 + corner
    bad.indices[at] = m.vertexCount
    with pytest.raises(pt.PTError, match="index out of range"):
        ctx.upload(bad)
    with pytest.raises(pt.PTError, match="no scene"):
        ctx.render(pt.render_params(24, 16, 1, cam, max_depth=5))
    assert np.array_equal(film_of(pt, ctx, sc, cam), want)


def test_uploads_of_other_sizes_in_turn(pt, scenes, ctx):
    """Small, large and small scenes on one context against fresh contexts."""
    made = [scenes.cornell(24, 16), scenes.disney_spheres(24, 16, grid=3, slices=64, rings=33, env_w=256, env_h=128),
            scenes.textured_scene(24, 16), scenes.hair_volume(24, 16, strands=200, segments=8, grid_n=32),
            scenes.cornell(24, 16, subdiv=1)]
    for k in (0, 1, 2, 1, 3, 0, 4, 1, 1, 0):
        sc, cam = made[k]
        fresh = pt.Context(0)
        want = film_of(pt, fresh, sc, cam)
        fresh.close()
        assert np.array_equal(film_of(pt, ctx, sc, cam), want), k


@pytest.mark.parametrize("w,h", [(1, 1), (3, 2), (33, 5), (130, 64), (4097, 3), (6200, 2), (16384, 2), (16385, 2),
                                 (2, 4100)])
@pytest.mark.parametrize("black_row", [False, True])
def test_envmap_tables_edges(w, h, black_row, pt, scenes, ctx, oracle):
    """CDFs bit for bit, and alias-table samples, around the sizes where the
    tables' kernels change (48 KB of shared memory, 16,384 texels) and with
    rows that sum to zero."""
    rng = np.random.default_rng(w * 31 + h)
    env = rng.gamma(0.5, 2.0, (h, w, 3)).astype(np.float32)
    if black_row:
        env[h // 2] = 0.0
    m = pt.make_material(pt.PT_MAT_DIFFUSE)
    m.vertexCount, m.indexCount = 3, 3
    sc = pt.Scene(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), np.array([0, 1, 2]), [m], env_rgb=env)
    ctx.upload(sc)
    oracle.load(sc)
    mg, cg = ctx.env_cdf()
    mo, co = oracle.env_cdf()
    assert np.array_equal(mg, mo) and np.array_equal(cg, co)
    u = rng.uniform(0, 1, (1 << 14, 2)).astype(np.float32)
    dg, _, pg = ctx.env_sample(pt.PT_ENV_ALIAS, u)
    do, _, po = oracle.env_sample(pt.PT_ENV_ALIAS, u)
    assert np.abs(dg - do).max() < 1e-5
    ok = po > 0
    assert np.array_equal(ok, pg > 0)
    assert np.all(np.abs(pg[ok] - po[ok]) <= 1e-4 * po[ok])
