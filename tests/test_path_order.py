"""The path order groups a call's samples so that a warp's camera rays lie close
together; the film must not depend on it: one call of n samples equals n calls
of one sample bit for bit, for sample counts with every kind of group, images
with and without full 8 x 4 tiles, and waves that cut groups apart."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(3, 2), (8, 4), (37, 21)])
@pytest.mark.parametrize("spp", [2, 7, 12, 31, 33, 79])
def test_one_call_equals_single_samples(w, h, spp, pt, scenes, ctx):
    sc, cam = scenes.cornell(w, h)
    ctx.upload(sc)
    s = np.zeros((h, w, 4), np.float32)
    c = np.zeros((h, w, 4), np.float32)
    for k in range(spp):
        ctx.render(pt.render_params(w, h, 1, cam, max_depth=6, sample_offset=9 + k), s, c)
    for wave in (0, w * h * spp // 37 + 1, w * h * 5):
        s1, c1, st = ctx.render(pt.render_params(w, h, spp, cam, max_depth=6, sample_offset=9, wave_paths=wave))
        assert st.paths == w * h * spp
        assert np.array_equal(s1, s) and np.array_equal(c1, c), wave
