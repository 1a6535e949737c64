"""Memory that uploads keep for the next one (their workspace, the previous
scene's arrays) is given back when an allocation would fail without it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Hold:
    """Holds all of the device's free memory but `left` bytes."""

    def __init__(self, left):
        import torch

        self.torch = torch
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        self.block = torch.empty(max(free - left, 1), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        del self.block
        self.torch.cuda.empty_cache()


def spheres(scenes, grid):
    """grid^2 spheres of 20,480 triangles."""
    return scenes.disney_spheres(64, 36, grid=grid, slices=128, rings=81, env_w=64, env_h=32)


def some_rays(sc, n):
    rng = np.random.default_rng(5)
    lo, hi = sc.positions.min(0), sc.positions.max(0)
    r = np.zeros((n, 8), np.float32)
    r[:, :3] = lo + (hi - lo) * rng.uniform(size=(n, 3))
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[:, 7] = 1e20
    return r


def test_scratch_takes_the_upload_workspace(pt, scenes):
    """A query whose staging fits only once the upload's workspace (190 bytes
    for each of 1.3 M triangles) is given back."""
    sc, _ = spheres(scenes, 8)
    n = 5_000_000  # 56 bytes each in staging: 280 MB
    r = some_rays(sc, n)
    ctx = pt.Context(0)
    try:
        ctx.upload(sc)
        few = ctx.trace_closest(r[:1000])
        with Hold(200 * MB):
            got = ctx.trace_closest(r)
        assert got[:1000].tobytes() == few.tobytes()
    finally:
        ctx.close()


def test_a_larger_scene_takes_the_previous_scenes_memory(pt, scenes):
    """From 0.9 M to 1.3 M triangles with room for the difference only: the new
    arrays do not fit the old ones' places."""
    small, large = spheres(scenes, 7)[0], spheres(scenes, 8)
    w, h = 64, 36
    want = None
    for left in (None, 160 * MB):
        ctx = pt.Context(0)
        try:
            ctx.upload(small)
            if left is None:
                ctx.upload(large[0])
            else:
                with Hold(left):
                    ctx.upload(large[0])
            film = ctx.render(pt.render_params(w, h, 1, large[1], max_depth=4))[0]
            want = film if want is None else want
            assert np.array_equal(film, want)
        finally:
            ctx.close()


def test_a_vertex_takes_52_bytes(pt):
    """Resident after an upload and a render: 16-byte positions and normals,
    texture coordinates and tangents, and not also the arrays that the records
    were made from.  (48 MB beside them: wave buffers and rounding.)"""
    import torch

    n = 8_000_000
    m = pt.make_material(pt.PT_MAT_DIFFUSE)
    m.vertexCount, m.indexCount = 3, 3
    cam = pt.pt_camera()
    P = pt.render_params(64, 64, 1, cam, max_depth=2)
    for nv in (3, n):  # the first: the kernels' own memory
        sc = pt.Scene(np.eye(3, dtype=np.float32)[np.arange(nv) % 3], np.array([0, 1, 2]), [m],
                      normals=np.ones((nv, 3), np.float32))
        free = torch.cuda.mem_get_info()[0]
        ctx = pt.Context(0)
        try:
            ctx.upload(sc)
            ctx.render(P)  # its buffers grow: the workspace is given back
            used = free - torch.cuda.mem_get_info()[0]
        finally:
            ctx.close()
    assert 52 * n <= used <= 60 * n + 48 * MB
