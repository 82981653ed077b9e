"""The timeout tests again on the stage kernels: on the grids they use, steps are resident
and only the edge exchange's wait runs out.  With a fixed tile height the waits of the TMA
boxes do, single and batched, at each height, and in a server's round."""
import pytest

import test_gpu_server
from test_gpu_server import alone  # noqa: F401 (a fixture)
from test_gpu_timeout import *  # noqa: F401,F403 (the tests, run here under the fixture below)
from test_gpu_timeout import polls  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=["8", "16", "32"])
def rows(request, monkeypatch):
    monkeypatch.setenv("AUSM_TILE_ROWS", request.param)


def test_failed_round_of_stage_kernels(alone):  # noqa: F811
    test_gpu_server.test_failed_round_ends_only_its_members(alone)
