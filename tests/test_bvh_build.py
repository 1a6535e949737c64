"""Bottom-up passes of the BVH build: the second arrival at a node finishes it,
so its reads must be ordered after both arrivals' writes, in every lane that
reads.  A missing fence shows on no run that can be asked for, so the order of
the fences, barriers and arrivals is read from the source; on the GPU the same
geometry must give the same tree on every build."""

import os
import re

import numpy as np
import pytest

from conftest import PKG_DIR

# per kernel, one pass of its loop: F fence, B warp barrier, A arrival, T the
# warp's work on a node (reads what other lanes' arrivals made visible)
ORDER = {"k_refit": "FAF", "k_wide_plan": "FAF", "k_treelet": "AFBTBF"}


@pytest.mark.parametrize("kernel", sorted(ORDER))
def test_fences_of_the_bottom_up_passes(kernel):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(PKG_DIR, "csrc", "pt_bvh.cu")).read())
    body = src[re.search(r"__global__ void [^;{]*\b%s\(" % kernel, src).end():]
    body = body[body.index("for (int guard"):]
    body = body[:body.index("\n}")]
    marks = {"__threadfence": "F", "__syncwarp": "B", "atomicAdd": "A", "treelet_restructure": "T"}
    assert "".join(marks[m] for m in re.findall("|".join(marks), body)) == ORDER[kernel]


@pytest.mark.gpu
@pytest.mark.parametrize("plan", [0, 1])
@pytest.mark.parametrize("name", ["spheres", "hair"])
def test_builds_repeat(name, plan, pt, scenes, ctx):
    """Greedy and planned collapse of two scenes, ten builds each: the wide
    tree's size, the order of its triangles and every hit of 20,000 rays."""
    if name == "spheres":
        sc = scenes.disney_spheres(64, 48, grid=4, slices=64, rings=33, env_w=64, env_h=32)[0]
    else:
        sc = scenes.hair_volume(32, 32, strands=1500, segments=8, grid_n=16)[0]
    rng = np.random.default_rng(11)
    lo, hi = sc.positions.min(0), sc.positions.max(0)
    r = np.zeros((20000, 8), np.float32)
    r[:, :3] = lo + (hi - lo) * rng.uniform(-0.1, 1.1, (len(r), 3))
    d = rng.normal(size=(len(r), 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 1e20
    ctx.debug_set(pt.PT_DEBUG_WIDE_PLAN, plan)
    try:
        first = None
        for _ in range(10):
            ctx.upload(sc)
            _, order, _, wide = ctx.bvh()
            got = (wide, order.tobytes(), ctx.trace_closest(r).tobytes())
            first = first or got
            assert got == first
    finally:
        ctx.debug_set(pt.PT_DEBUG_WIDE_PLAN, 0)
