"""Allocation-free queries beside a frame in flight, in a process that has run none of their kernels before."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes as C, sys
sys.path[:0] = [sys.argv[1] + "/gpu-pathed_b200", sys.argv[1] + "/tests"]
import numpy as np
import pathed
from _util import seeded_rays

first, n = sys.argv[2], int(sys.argv[3])
s = pathed.Session(1024, 1024)
s.load_config(3, level=6)
assert s.counts().bvh_depth >= 6  # calls of 1024 rays or more share their last queries
rays = seeded_rays(s.export_scene(), n, seed=5)
out = [np.zeros(n, np.int32) for _ in range(3)] + [np.zeros(n, np.float32)]

def static(m):
    s._check(pathed.lib.pt_trace_rays_static(s._h, *[a.ctypes.data for a in rays], m, *[a.ctypes.data for a in out], None))

if first == "trace":
    s.trace_rays(*[a[:16] for a in rays])
s.render(32)
static(1) if first == "trace" else None
s.render_async(32)  # about 110 ms on a B200
static(n)           # less than 1 ms
done = C.c_int(1)
pathed.lib.pt_poll(s._h, C.byref(done), None)
s.wait()
got = [a.copy() for a in out]
static(n)
assert all(np.array_equal(a, b) for a, b in zip(got, out))
print("in flight" if done.value == 0 else "waited")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("n", [100, 30000])
@pytest.mark.parametrize("first", ["trace", "render"])
def test_first_query_does_not_wait_for_the_frame(first, n):
    r = subprocess.run([sys.executable, "-c", PROGRAM, ROOT, first, str(n)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == "in flight"
