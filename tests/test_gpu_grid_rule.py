"""Sizes on both sides of the line between one and two multicolour sweeps to a launch (296
tiles of 56 x 40 vertices for even M, 148 of 40 x 32 for odd M), against the oracle."""
import pytest

from test_gpu_grid_sweeps import test_sweeps_match_oracle as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1008, 641), (1010, 641), (561, 289), (561, 290)])
@pytest.mark.parametrize("sweeps", [1, 8])
def test_sizes_at_the_line(M, N, sweeps):
    check(M, N, sweeps)
