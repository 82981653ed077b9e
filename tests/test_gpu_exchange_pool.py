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


def test_tags_start_again_on_a_cleared_buffer():
    """A process of its own: one buffer, first tag 1.  Past the range's end the next launch
    would read the first one's edges as its neighbours' had the buffer not been cleared."""
    env = {k: v for k, v in os.environ.items() if k != "AUSM_TILE_ROWS"}
    r = subprocess.run([sys.executable, "-c", WRAP.format(root=str(ROOT))], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
