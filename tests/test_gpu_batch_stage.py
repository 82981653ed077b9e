"""The batch tests again on the stage kernels: members as small as theirs are resident in the
default setting, whatever the graphs' switch says.  Under a fixed tile height they run the
work list, eagerly and from graphs; and a batch whose tiles do not fit on the chip runs it
in the default setting, tuned, from graphs and eagerly, with the bits of the single
solves."""
import numpy as np
import pytest

from test_gpu_batch import (grids, test_batch_graphs_off_identical, test_batch_matches_single_solve_path,  # noqa: F401
                            test_batch_membership_changes, test_batch_residual_norms,
                            test_batch_same_alone_and_in_mix)
from test_gpu_edges import solver

pytestmark = pytest.mark.gpu

LARGE = [(768, 200, "SLAU2"), (500, 301, "AUSM+-up"), (257, 131, "SLAU"), (33, 17, "SLAU2")]  # 1367 tiles of 8 rows


@pytest.fixture(autouse=True)
def rows(request, monkeypatch):
    if "large" not in request.node.name:
        monkeypatch.setenv("AUSM_TILE_ROWS", "8")


def test_large_batch_graphs_eager_and_alone():
    from ausm import Batch
    assert sum(-(-M // 32) * -(-N // 8) for M, N, _ in LARGE) > 888

    def make():
        return [solver(M, N, scheme=sc, mach=1.2) for M, N, sc in LARGE]
    out = []
    for graphs in (True, False):
        sols = make()
        with Batch(graphs=graphs) as b:
            for s in sols:
                b.add(s)
            dts = [b.step(n) for n in (4, 3, 4, 1)]
        out.append(dts + [s.state() for s in sols])
        for s in sols:
            s.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    for k, s in enumerate(make()):
        for n in (4, 3, 4, 1):
            s.step(n)
        np.testing.assert_array_equal(s.state(), out[0][4 + k])
        s.close()
