"""More streams with resident steps in flight than there are exchange buffers: buffers are
shared by waiting on the device, and a larger grid takes the place of a smaller one's
buffer.  Every solve must end with the bits it has when it is stepped alone, from one host
thread that only enqueues and from a host thread per solve, small and chip-filling grids
mixed, with a batch among them."""
import threading

import numpy as np
import pytest

from test_gpu_edges import solver

pytestmark = pytest.mark.gpu

SMALL = [(64 + 8 * k, 33 + k) for k in range(10)]
MIXED = [(768, 290), (640, 148), (128, 96), (512, 384), (64, 33), (700, 300), (96, 64), (257, 131), (640, 140), (50, 40),
         (333, 250), (300, 200)]


def enqueue(s, calls=6, n=400):
    for _ in range(calls):
        s.step(n, wait=False)


def alone(sizes, **kw):
    out = []
    for k, (M, N) in enumerate(sizes):
        with solver(M, N, mach=0.6 + 0.1 * k) as s:
            enqueue(s, **kw)
            out.append((s.max_wave_speed(), s.state()))
    return out


def same(sols, want):
    for s, (w, q) in zip(sols, want):
        assert s.max_wave_speed() == w
        np.testing.assert_array_equal(s.state(), q)


def test_streams_beyond_the_buffers_then_a_larger_grid():
    """Ten streams grow the pool to eight buffers of the smallest size; the large grid then
    finds none that it fits in, and all ten still at work."""
    sizes = SMALL + [(768, 296)]
    want = alone(sizes)
    sols = [solver(M, N, mach=0.6 + 0.1 * k) for k, (M, N) in enumerate(SMALL)]
    for s in sols:
        enqueue(s)
    sols.append(solver(*sizes[-1], mach=0.6 + 0.1 * len(SMALL)))
    enqueue(sols[-1])
    same(sols, want)
    for s in sols:
        s.close()


def test_threads_beyond_the_buffers():
    from ausm import Batch
    want = alone(MIXED, calls=3, n=100)
    sols = [solver(M, N, mach=0.6 + 0.1 * k) for k, (M, N) in enumerate(MIXED)]
    errors = []

    def work(step):
        try:
            for _ in range(3):
                step(100)
        except Exception as e:  # reported below, on the test's own thread
            errors.append(e)
    with Batch() as b:
        for s in sols[-2:]:
            b.add(s)
        threads = [threading.Thread(target=work, args=(x.step,)) for x in sols[:-2] + [b]]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors, errors
    same(sols, want)
    for s in sols:
        s.close()
