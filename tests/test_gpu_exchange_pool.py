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

def steps(s):
    out = [s.step(3), s.step(1)]
    with Batch(graphs=False) as b:
        b.add(s)
        out += [b.step(2), b.step(3)]
    return out + [s.state()]

os.environ["AUSM_TILE_ROWS"] = "16"  # the stage kernels, loaded before the memory is taken
with solver(300, 200) as s:
    want = steps(s)
del os.environ["AUSM_TILE_ROWS"]
os.environ["AUSM_AUTOTUNE"] = "0"

cu = C.CDLL("libcuda.so.1")
held = []

def take(size):
    p = C.c_void_p()
    if cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(size)):
        return False
    held.append(p)
    return True

def give_back(p):
    held.remove(p)
    assert cu.cuMemFree_v2(p) == 0

for k in range(34, 20, -1):
    while take(1 << k):
        pass
while not take(8 << 20):  # the solver's arrays (6.3 MB)
    give_back(held[-1])
mine = held[-1]
while take(2 << 20):
    pass
for p in [mine] + [p for p in held if p is not mine][-2:]:  # and 4 MiB: less than its exchange buffer
    give_back(p)
s = solver(300, 200)
got = steps(s)
while held:
    give_back(held[-1])
for x, y in zip(got, want):
    np.testing.assert_array_equal(x, y)
'''

KEEP = r'''
import ctypes as C, sys
for p in ({root!r}, {root!r} + "/tests", {root!r} + "/ausm-webgpu_b200"):
    sys.path.insert(0, p)
import ausm
from test_gpu_edges import solver

cu = C.CDLL("libcuda.so.1")

def free():
    a, b = C.c_size_t(), C.c_size_t()
    assert cu.cuMemGetInfo_v2(C.byref(a), C.byref(b)) == 0
    return a.value

for k in range(3):  # the first turn loads the kernels
    with solver(300, 200) as s:
        s.synchronize()
        before = free()
        s.step(2)
        assert k == 0 or free() == before, "a step allocated or freed device memory"
s = solver(300, 200)
s.close()
none = free()
with ausm.Server(1e9, chunk_steps=10, plain=True) as srv:
    for k in range(2):
        srv.submit(ausm.make_request(300, 200, naca4=12, mach=0.5, far_radius=10.0, grid_iters=20, max_steps=20))
        srv.drain()
        held = none - free()
        assert held > 4e6, f"{{held}} bytes held between requests"
assert free() == none, "the buffer was not given back"
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


def test_buffer_is_kept_and_given_back():
    """One solver at a time: the buffer comes with its creation, so that a step allocates
    nothing.  A server keeps it between its requests, also one that serves them singly, and
    gives it back at its end."""
    run(KEEP)


def test_steps_without_memory_for_a_buffer():
    """A device that has no room for an exchange buffer steps by the stage kernels, which
    need none: the same bits."""
    run(FULL)
