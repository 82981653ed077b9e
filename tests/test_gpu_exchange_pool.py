"""The exchange buffers that resident launches share in a process: they are taken by stream,
reused when free, grown to eight per device, then waited for, and marked with 32-bit tags
that go on from launch to launch."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

WRAP = r'''
import os, sys
import numpy as np
for p in ({root!r}, {root!r} + "/tests", {root!r} + "/ausm-webgpu_b200"):
    sys.path.insert(0, p)
from ausm import _lib
from test_gpu_edges import solver

big, small = solver(333, 250), solver(64, 33)
big.step(1)  # tags 1, 2, 3: edges of tags 2 and 3 are left in the cells of its tiles
_lib.check(_lib.lib().ausm_debug_set_exchange_tag(0xfffffffe))
small.step(1)  # three tags, the last past the range's end
big.step(1)  # the first tags again, and the cells that `small` did not reach
big.step(3)
got = big.max_wave_speed(), big.state(), small.state()
os.environ["AUSM_TILE_ROWS"] = "16"
big, small = solver(333, 250), solver(64, 33)
small.step(1)
for n in (1, 1, 3):
    big.step(n)
assert got[0] == big.max_wave_speed()
np.testing.assert_array_equal(got[1], big.state())
np.testing.assert_array_equal(got[2], small.state())
'''

FULL = r'''
import ctypes as C, os, sys
import numpy as np
for p in ({root!r}, {root!r} + "/tests", {root!r} + "/ausm-webgpu_b200"):
    sys.path.insert(0, p)
from ausm import Batch
from test_gpu_edges import solver

def members():
    return [solver(96, 40), solver(65, 33, scheme="AUSM+-up")]

def steps(s, sols, b):
    return [s.step(3), b.step(2), s.step(1), b.step(3), s.state()] + [x.state() for x in sols]

os.environ["AUSM_TILE_ROWS"] = "16"  # the stage kernels, loaded before the memory is taken
s, sols, b = solver(128, 96), members(), Batch(graphs=False)
for x in sols:
    b.add(x)
want = steps(s, sols, b)
b.close()
for x in [s] + sols:
    x.close()
del os.environ["AUSM_TILE_ROWS"]
os.environ["AUSM_AUTOTUNE"] = "0"

cu = C.CDLL("libcuda.so.1")
held = []
def fill(size):
    p = C.c_void_p()
    while cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(size)) == 0:
        held.append(p)
        p = C.c_void_p()

def give_back(n):
    for _ in range(n):
        assert cu.cuMemFree_v2(held.pop()) == 0

for k in range(34, 20, -1):
    fill(1 << k)
give_back(1)
fill(2 << 20)
give_back(3)
fill(8 << 20)  # the rest holds small solvers, but no exchange buffer (9.1 MB)
s, sols, b = solver(128, 96), members(), Batch(graphs=False)
for x in sols:
    b.add(x)
got = steps(s, sols, b)
give_back(len(held))
for x, y in zip(got, want):
    np.testing.assert_array_equal(x, y)
'''


def run(code):
    """In a process of its own, whose exchange buffers are its own."""
    env = {k: v for k, v in os.environ.items() if k != "AUSM_TILE_ROWS"}
    r = subprocess.run([sys.executable, "-c", code.format(root=str(ROOT))], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_tags_start_again_on_a_cleared_buffer():
    """One buffer, first tag 1.  Past the range's end the next launch would read the first
    one's edges as its neighbours' had the buffer not been cleared."""
    run(WRAP)


def test_steps_without_memory_for_a_buffer():
    """A device that has no room for an exchange buffer steps by the stage kernels, which
    need none: the same bits."""
    run(FULL)
