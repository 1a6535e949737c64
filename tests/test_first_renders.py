"""Contexts on threads of their own whose first renders begin together: the
launch sizes of all kernels are worked out once per process, and no render may
start with a part of them."""

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import sys, threading
sys.path.insert(0, "tests")
import conftest, importlib, numpy as np
pt = conftest.load_package()
scenes = importlib.import_module("pbrt_b200.scenes")
sc, cam = scenes.%s
P = pt.render_params(48, 32, 2, cam, max_depth=6)
ctxs = [pt.Context(0) for _ in range(4)]
for c in ctxs:
    c.upload(sc)
start, films = threading.Barrier(4), [None] * 4
def work(k):
    start.wait()
    films[k] = ctxs[k].render_batch([P])[0][0][0] if k %% 2 else ctxs[k].render(P)[0]
threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
again = ctxs[0].render(P)[0]
assert all(f is not None and np.array_equal(f, again) for f in films)
"""


@pytest.mark.parametrize("scene", ["cornell(48, 32)", "hair_volume(48, 32, strands=200, segments=8, grid_n=16)"])
def test_first_renders_begin_together(scene):
    r = subprocess.run([sys.executable, "-c", CODE % scene], cwd=ROOT, env={**os.environ, "PYTHONPATH": ROOT},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
