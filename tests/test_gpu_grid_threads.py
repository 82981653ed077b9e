"""Grids generated on several host threads at once, one handle each: the sweep kernels'
shared-memory limit is a property of the kernel that all threads share, so no launch may
lower it under another one.  Of each pair of sizes, which run the same kernel, the first
takes more shared memory than the second; every grid must equal the one generated alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def generate(M, N, method, sweeps):
    from ausm import Solver
    with Solver(M, N) as s:
        s.set_body_naca4(12, 0.3, -0.7)
        s.set_outer_rect(1.5)
        s.generate_grid(sweeps, method)
        return s.vertices()


@pytest.mark.parametrize("method,sizes", [("jacobi", [(640, 480), (1024, 768)]),
                                          ("multicolor", [(401, 400), (401, 300)])])
def test_concurrent_grids(method, sizes):
    alone = [generate(M, N, method, 1500) for M, N in sizes]
    got, errors = {}, []

    def work(k):
        try:
            for r in range(3):
                got[k, r] = generate(*sizes[k % 2], method, 1500)
        except Exception as e:  # reported below, on the test's own thread
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (k, r), v in got.items():
        np.testing.assert_array_equal(v, alone[k % 2])
