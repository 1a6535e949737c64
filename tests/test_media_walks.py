"""Walks through heterogeneous media in kernels of their own (one step per lane
at a time, finished lanes refilled) against the same walks run to their end in
one thread: free flights against the tail kernel's, deferred ratio tracking
against the shadow kernel's own (which scenes with glass use).  Films must be
equal bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volumes(pt, kinds, sigma):
    """Overlapping boxes in the room; kinds: h heterogeneous, u uniform, e empty."""
    out = []
    for k, kind in enumerate(kinds):
        v = pt.pt_volume()
        v.vmin[:] = (-0.9 + 0.2 * k, 0.1, -0.9)
        v.vmax[:] = (0.9, 1.7 - 0.3 * k, 0.9 - 0.1 * k)
        s = 0.0 if kind == "e" else sigma
        v.sigma_a[:] = (0.1 * s, 0.2 * s, 0.3 * s)
        v.sigma_s[:] = (s, 0.8 * s, 0.6 * s)
        v.phase_g = 0.4 - 0.2 * k
        v.flags = 0 if kind == "u" else pt.PT_VOLUME_HETEROGENEOUS
        v.density_grid = pt.PT_NO_TEXTURE if kind == "u" else 0
        out.append(v)
    return out


def room(pt, scenes, kinds, sigma, glass_inside=False):
    sc, cam = scenes.cornell(70, 50)
    pos, idx, mats = sc.positions, sc.indices, list(sc.materials)
    nrm = sc.normals
    if glass_inside:  # a glass triangle inside the opaque sphere, which no ray reaches
        m = pt.make_material(pt.PT_MAT_DIELECTRIC)
        m.vertexOffset, m.vertexCount, m.indexOffset, m.indexCount = len(pos), 3, len(idx), 3
        tri = np.array([[0, 0.55, -0.1], [0.1, 0.55, -0.1], [0, 0.6, -0.1]], np.float32)
        pos, idx = np.concatenate([pos, tri]), np.concatenate([idx, np.arange(3, dtype=np.uint32)])
        nrm = np.concatenate([nrm, np.zeros((3, 3), np.float32)])
        mats.append(m)
    return pt.Scene(pos, idx, mats, normals=nrm, volumes=volumes(pt, kinds, sigma), grids=[scenes.fbm_grid(32, 4)]), cam


@pytest.mark.parametrize("kinds,sigma", [("h", 2.0), ("hu", 6.0), ("heh", 3.0), ("uhh", 20.0), ("e", 1.0)])
@pytest.mark.parametrize("rng", [0, 1])
def test_flights_of_both_forms_agree(kinds, sigma, rng, pt, scenes, ctx):
    sc, cam = room(pt, scenes, kinds, sigma)
    ctx.upload(sc)
    P = pt.render_params(70, 50, 3, cam, max_depth=14, sample_offset=3, rng_kind=rng)
    films = []
    for tail in (1, 2):  # never; from bounce 4 on
        ctx.debug_set(pt.PT_DEBUG_TAIL, tail)
        try:
            films.append(ctx.render(P))
        finally:
            ctx.debug_set(pt.PT_DEBUG_TAIL, 0)
    assert films[1][2].tail_extension_rays > 0 and films[0][2].tail_extension_rays == 0
    assert np.array_equal(films[0][0].view(np.uint32), films[1][0].view(np.uint32))
    assert np.array_equal(films[0][1].view(np.uint32), films[1][1].view(np.uint32))


@pytest.mark.parametrize("kinds,sigma", [("h", 2.0), ("hu", 6.0), ("heh", 3.0), ("uhh", 20.0)])
@pytest.mark.parametrize("spp", [1, 5])
def test_deferred_ratio_tracking_of_both_forms_agrees(kinds, sigma, spp, pt, scenes, ctx):
    films = []
    for glass in (False, True):
        sc, cam = room(pt, scenes, kinds, sigma, glass_inside=glass)
        ctx.upload(sc)
        films.append(ctx.render(pt.render_params(70, 50, spp, cam, max_depth=9, sample_offset=3,
                                                 flags=pt.PT_RENDER_MEDIA_WAVEFRONT)))
    assert films[0][2].extension_rays == films[1][2].extension_rays
    assert np.array_equal(films[0][0].view(np.uint32), films[1][0].view(np.uint32))
