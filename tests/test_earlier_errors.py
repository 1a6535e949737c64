"""A call that was refused has reported its error; the calls after it on the same
thread must not report it again as theirs."""

import numpy as np
import pytest

from test_zz_no_alloc import _call

pytestmark = pytest.mark.gpu


def refused_wave(pt, ctx, cam):
    """921 M paths in one wave need 335 GB."""
    big = pt.render_params(1280, 720, 1000, cam, max_depth=5, wave_paths=1 << 30)
    with pytest.raises(pt.PTError, match="wave buffers"):
        ctx.render(big)


def refused_device(pt, ctx, cam):
    with pytest.raises(pt.PTError):
        pt.Context(99)


@pytest.mark.parametrize("refused", [refused_wave, refused_device])
@pytest.mark.parametrize("call", ["upload", "render", "batch", "noalloc"])
def test_calls_after_a_refused_one(refused, call, pt, scenes):
    sc, cam = scenes.cornell(24, 16)
    P = pt.render_params(24, 16, 2, cam, max_depth=5)
    ctx = pt.Context(0)
    try:
        ctx.upload(sc)
        want = ctx.render(P)[0]
        refused(pt, ctx, cam)
        if call == "upload":
            ctx.upload(sc)
        elif call == "batch":
            films, _, _ = ctx.render_batch([P])
            assert np.array_equal(films[0][0], want)
        elif call == "noalloc":
            w = np.array([[0.0, 0.0, 1.0]], np.float32)
            assert _call(pt, [pt.make_material(pt.PT_MAT_DIFFUSE)], None, w, w, None)[0] == 0
        assert np.array_equal(ctx.render(P)[0], want)
    finally:
        ctx.close()
