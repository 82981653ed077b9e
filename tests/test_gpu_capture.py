"""Steps captured into a CUDA graph of the host's own.  A captured step stays on the stage
kernels at any size: a captured resident launch would hold an exchange buffer that other
solvers use between the replays.  Replays beside another solver's direct steps, and direct
steps after them, must give the bits of a twin that is stepped directly throughout, for a
single solve and for a batch (graphs off), both small enough that their direct steps are
resident."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_edges import solver

pytestmark = pytest.mark.gpu

SIZES = [(96, 40, "SLAU2"), (65, 33, "AUSM+-up"), (33, 17, "SLAU")]


class Graph:
    """What fn enqueues on a stream, captured and replayed through the driver API."""

    def __init__(self, stream, fn):
        self.cu, self.stream = C.CDLL("libcuda.so.1"), stream
        g, self.exec = C.c_void_p(), C.c_void_p()
        self.ok(self.cu.cuStreamBeginCapture_v2(stream, 1))  # thread-local
        fn()
        self.ok(self.cu.cuStreamEndCapture(stream, C.byref(g)))
        self.ok(self.cu.cuGraphInstantiateWithFlags(C.byref(self.exec), g, C.c_ulonglong(0)))
        self.ok(self.cu.cuGraphDestroy(g))

    def ok(self, rc):
        assert rc == 0, f"CUDA driver error {rc}"

    def launch(self):
        self.ok(self.cu.cuGraphLaunch(self.exec, self.stream))

    def close(self):
        self.ok(self.cu.cuGraphExecDestroy(self.exec))


def refused(stream, fn, code):
    """fn must fail with `code` inside a capture, and leave the capture itself valid."""
    from ausm import AusmError

    def go():
        with pytest.raises(AusmError) as e:
            fn()
        assert e.value.code == code
    Graph(stream, go).close()


def stream_of(s):
    from ausm import _lib
    st = C.c_void_p()
    s._c(_lib.lib().ausm_stream(s.h, C.byref(st)))
    return st


def test_captured_solver_step_beside_direct_steps():
    a, twin, other, other_twin = (solver(*x) for x in ((96, 40), (96, 40), (257, 131), (257, 131)))
    for s in (a, twin):
        s.step(3)
    g = Graph(stream_of(a), lambda: a.step(3, wait=False))
    for _ in range(5):
        g.launch()
        other.step(30, wait=False)
        twin.step(3)
        other_twin.step(30)
    for s in (a, twin, other, other_twin):
        s.step(4)
    g.close()
    for x, y in ((a, twin), (other, other_twin)):
        assert x.max_wave_speed() == y.max_wave_speed()
        np.testing.assert_array_equal(x.state(), y.state())
    for s in (a, twin, other, other_twin):
        s.close()


def test_captured_batch_step_beside_direct_steps():
    from ausm import Batch
    mine, twins = ([solver(M, N, scheme=sc) for M, N, sc in SIZES] for _ in range(2))
    other, other_twin = solver(257, 131), solver(257, 131)
    with Batch(graphs=False) as b, Batch(graphs=False) as t:
        for s, x in zip(mine, twins):
            b.add(s)
            t.add(x)
        np.testing.assert_array_equal(b.step(3), t.step(3))
        g = Graph(stream_of(mine[0]), lambda: b.step(3, wait=False))
        other.step(30, wait=False)  # whatever the capture left behind is not this solver's error
        other_twin.step(30)
        for _ in range(5):
            g.launch()
            other.step(30, wait=False)
            t.step(3)
            other_twin.step(30)
        np.testing.assert_array_equal(b.step(4), t.step(4))
        b.synchronize()
        g.close()
    for x, y in zip(mine + [other], twins + [other_twin]):
        np.testing.assert_array_equal(x.state(), y.state())
    for s in mine + twins + [other, other_twin]:
        s.close()


def test_captured_batch_step_refuses_to_upload(monkeypatch):
    """A captured step cannot bring the device's tables up to date (a replay would read host
    memory that has changed or gone): before the first direct call, after a parameter change
    and after a membership change it is refused, and a direct step makes it possible again."""
    from ausm import Batch, _lib
    monkeypatch.setenv("AUSM_TILE_ROWS", "8")  # a fixed height: nothing to tune
    sols = [solver(M, N, scheme=sc) for M, N, sc in SIZES]
    st = None
    with Batch(graphs=False) as b:
        def no():
            refused(st, lambda: b.step(3, wait=False), _lib.ERR_STATE)
        for s in sols:
            b.add(s)
        st = stream_of(sols[0])
        no()
        b.step(3)
        sols[0].set_params(mach=0.7)
        no()
        b.step(3)
        b.remove(sols[1])
        no()
        b.step(3)
        g = Graph(st, lambda: b.step(3, wait=False))
        g.launch()
        out = b.step(1)
        g.close()
    assert np.all(np.isfinite(out))
    for s in sols:
        s.close()


def test_captured_tuning_is_refused():
    """Tuning times and waits, which a capture does not allow: a captured step of a grid too
    large to be resident needs its tile height tuned before, and so does ausm_autotune itself
    at any size; a batch needs a step before.  Neither capture nor solver is the worse for the
    attempt."""
    from ausm import Batch, _lib
    for M, N, call in ((1030, 411, lambda s: s.step(3, wait=False)), (71, 37, lambda s: s.autotune())):
        s = solver(M, N)
        refused(stream_of(s), lambda: call(s), _lib.ERR_CUDA)
        assert s.autotune() in (8, 16, 32)
        assert np.isfinite(s.step(2))
        with Batch(graphs=False) as b:
            b.add(s)
            refused(stream_of(s), lambda: b.step(3, wait=False), _lib.ERR_CUDA)
            assert np.all(np.isfinite(b.step(2)))
        s.close()
