"""Shared memory of the envmap kernels at their first launch: a block holds one
row, up to 196,608 bytes, and above 48 KB (the kernels' static variables
counted in) a launch is refused unless the limit has been raised.  The limit
belongs to the kernel, not to a context: it must not depend on the maps that
were uploaded before, nor on what another thread uploads meanwhile."""

import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# 12 bytes a texel of a row (or row of the map), 8 in the first kernel: 49,152
# bytes lie at 4,096 and at 6,144; the sizes of each kernel in rising order
SIZES = [(4095, 2), (4096, 2), (6143, 2), (6144, 2), (2, 4094), (2, 4095), (2, 4096), (16384, 1), (1, 16384)]


def one_triangle(pt, env):
    m = pt.make_material(pt.PT_MAT_DIFFUSE)
    m.vertexCount, m.indexCount = 3, 3
    return pt.Scene(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), np.array([0, 1, 2]), [m], env_rgb=env)


def check(pt, ctx, oracle, w, h):
    sc = one_triangle(pt, np.random.default_rng(w * 31 + h).gamma(0.5, 2.0, (h, w, 3)).astype(np.float32))
    ctx.upload(sc)
    oracle.load(sc)
    for got, want in zip(ctx.env_cdf(), oracle.env_cdf()):
        assert np.array_equal(got, want)


def test_first_uploads_of_a_process():
    """Each size while its kernel's limit is still what the process began with."""
    code = ("import sys; sys.path.insert(0, 'tests'); import conftest; pt = conftest.load_package()\n"
            "from oracle.oracle import Oracle; import test_envmap_shared_memory as t\n"
            "ctx, o, bad = pt.Context(0), Oracle(pt), []\n"
            "for w, h in t.SIZES:\n"
            "    try: t.check(pt, ctx, o, w, h)\n"
            "    except Exception as e: bad.append((w, h, repr(e)))\n"
            "ctx.close(); print(bad); sys.exit(1 if bad else 0)\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env={**os.environ, "PYTHONPATH": ROOT},
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


def test_uploads_on_two_threads(pt):
    """Two contexts, each on its own thread, a hundred uploads of maps whose
    rows need different amounts."""
    failed = []

    def work(w):
        ctx = pt.Context(0)
        sc = one_triangle(pt, np.ones((1, w, 3), np.float32))
        for _ in range(100):
            try:
                ctx.upload(sc)
            except pt.PTError as e:
                failed.append((w, str(e)))
        ctx.close()

    threads = [threading.Thread(target=work, args=(w,)) for w in (8192, 16384)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, (len(failed), failed[0])
