"""The captured form of a render (parallel branches, the conditional body after
the tail kernel, launch shapes of short queues) against the launches issued
one after the other on one stream (PT_RENDER_STAGE_TIMING): the same films bit
for bit and the same ray counts."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# name, scene, width, height, spp, depth, wave_paths
CASES = [
    ("one pixel", "cornell", 1, 1, 1, 8, 0),
    ("short queues", "cornell", 61, 37, 2, 8, 0),
    ("tail finishes the wave", "spheres", 200, 120, 3, 16, 0),
    ("body runs after the tail bounce", "cornell", 256, 256, 16, 16, 0),
    ("waves on both sides of the tail's limit", "cornell", 192, 128, 24, 14, 192 * 128 * 16),
    ("counter blocks of a deep render", "cornell", 48, 32, 1, 70, 0),
    ("textures and alpha maps", "textured", 150, 110, 5, 13, 0),
    ("homogeneous medium", "fog", 96, 60, 2, 12, 0),
    ("heterogeneous medium", "hair_volume", 48, 48, 2, 13, 0),
]


def make(scenes, name, w, h):
    if name == "cornell":
        return scenes.cornell(w, h)
    if name == "spheres":
        return scenes.disney_spheres(w, h, grid=3, slices=48, rings=25, env_w=256, env_h=128)
    if name == "textured":
        return scenes.textured_scene(w, h)
    if name == "fog":
        return scenes.radiance_cache_scene(w, h, instances=9, subdiv=3)
    return scenes.hair_volume(w, h, strands=300, segments=8, grid_n=32)


@pytest.mark.parametrize("what,name,w,h,spp,depth,wave", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("wavefront", [False, True], ids=["default", "media_wavefront"])
def test_captured_render_equals_serial_launches(what, name, w, h, spp, depth, wave, wavefront, pt, scenes, ctx):
    if wavefront and name != "hair_volume":
        pytest.skip("the option concerns heterogeneous media")
    sc, cam = make(scenes, name, w, h)
    ctx.upload(sc)
    flags = pt.PT_RENDER_MEDIA_WAVEFRONT if wavefront else 0
    P = pt.render_params(w, h, spp, cam, max_depth=depth, sample_offset=5, wave_paths=wave, flags=flags)
    serial, serial_c, st0 = ctx.render(pt.render_params(w, h, spp, cam, max_depth=depth, sample_offset=5,
                                                        wave_paths=wave, flags=flags | pt.PT_RENDER_STAGE_TIMING))
    for _ in range(2):  # the capturing call and a replay
        film, comp, st = ctx.render(P)
        assert np.array_equal(film.view(np.uint32), serial.view(np.uint32))
        assert np.array_equal(comp.view(np.uint32), serial_c.view(np.uint32))
        assert (st.extension_rays, st.shadow_rays, st.launches) == (st0.extension_rays, st0.shadow_rays, st0.launches)
