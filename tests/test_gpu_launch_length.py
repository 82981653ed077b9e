"""A resident launch takes all SMs, so its length is what a call on another stream may have
to wait: at most 360 steps.  A small solver's steps beside a long call on one of the largest
resident grids wait for one launch at a time (the bound: three of them, in the best of three
tries, since the host's own delays only add), not for a launch as long as the call."""
import time

import pytest

from test_gpu_edges import solver

pytestmark = pytest.mark.gpu


def test_other_streams_wait_for_one_launch():
    big, small = solver(768, 296), solver(64, 33)
    for s in (big, small):
        s.step(3)
        s.step(3)
    one = 1e-3 * big.time_steps(360, 4) / 4  # seconds of a launch
    longest = []
    for _ in range(3):
        waits = []
        big.step(8000, wait=False)
        time.sleep(0.002)
        for _ in range(4):
            t = time.perf_counter()
            small.step(1)
            waits.append(time.perf_counter() - t)
        big.synchronize()
        longest.append(max(waits))
    assert min(longest) <= 3 * one, (longest, one)
    for s in (big, small):
        s.close()
