"""pt_stats.launches counts every kernel of a call: where a queue's length
decides on the device between the one-lane and the 8-lanes-per-ray kernel, both
are launched and both count; so do the tail's kernels and those of the bounces
that follow it only when it left paths."""

import pytest

pytestmark = pytest.mark.gpu

CLASSES = 4  # the room's: miss, emitter, diffuse, Disney
SHORT, LONG = (64, 48), (200, 200)  # 3,072 paths; 40,000, above 18,944 at bounce 0 only


def launches(pt, scenes, ctx, size, depth, spp=1, tail=0, flags=0, calls=2):
    sc, cam = scenes.cornell(*size)
    ctx.upload(sc)
    ctx.debug_set(pt.PT_DEBUG_TAIL, tail)
    try:
        counts = {ctx.render(pt.render_params(*size, spp, cam, max_depth=depth, flags=f | flags))[2].launches
                  for f in [0] * calls + [pt.PT_RENDER_STAGE_TIMING]}
    finally:
        ctx.debug_set(pt.PT_DEBUG_TAIL, 0)
    assert len(counts) == 1  # captured, replayed and one by one
    return counts.pop()


@pytest.mark.parametrize("depth", [1, 2, 3])
def test_bounces(depth, pt, scenes, ctx):
    """Sample offset, camera rays and film; per bounce the closest-hit kernel,
    one kernel per class and the shadow kernel; both forms of the first and
    the last from the second bounce of the long queue on."""
    short = 3 + depth * (2 + CLASSES)
    assert launches(pt, scenes, ctx, SHORT, depth) == short
    assert launches(pt, scenes, ctx, LONG, depth) == short + 2 * (depth - 1)


def test_tail_finishes(pt, scenes, ctx):
    """13 bounces: the tail takes over at bounce 4 with both of its forms and
    the kernel that closes it.  Switched off, its one-lane form and the closing
    kernel find nothing to do, and all 13 bounces run."""
    assert launches(pt, scenes, ctx, SHORT, 13) == 3 + 4 * (2 + CLASSES) + 3
    assert launches(pt, scenes, ctx, SHORT, 13, tail=1) == 3 + 13 * (2 + CLASSES) + 2


def test_bounces_after_the_tail(pt, scenes, ctx):
    """2^20 paths in a closed room: more than the tail takes are left at bounce
    4, and its kernels come on top of all 16 bounces'; from bounce 3 on
    (2^20 / 4^3 < 18,944) both forms of each traversal kernel."""
    bounces = 16 * (2 + CLASSES) + 2 * 13
    assert launches(pt, scenes, ctx, (256, 256), 16, spp=16) == 3 + bounces + 3
    assert launches(pt, scenes, ctx, (256, 256), 16, spp=16, tail=1) == 3 + bounces + 2


def test_cached_render(pt, scenes, ctx):
    """Two waves: inference and the five kernels of the training targets after
    each, then four times the gradient and the update; the first call sets the
    chance of training."""
    w, h = SHORT
    sc, cam = scenes.cornell(w, h)
    c = pt.Context(0)
    try:
        c.upload(sc)
        c.cache_init(pt.cache_params(seed=1, train_records=512))
        P = pt.render_params(w, h, 2, cam, max_depth=3, wave_paths=w * h, flags=pt.PT_RENDER_RADIANCE_CACHE)
        got = [c.render(P)[2].launches for _ in range(3)]
        call = 1 + 2 * (2 + 3 * (2 + CLASSES) + 1 + 5) + 4 * 2
        assert got == [call + 1, call, call]
    finally:
        c.close()
