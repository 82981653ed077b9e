"""A timeout that the host has not read yet spoils nothing but the steps that timed out: a
solve that is given a new state goes on from it, wave speed and dt included, although the
error flag is still set, and the next call that waits reports the timeout."""
import numpy as np
import pytest

from test_gpu_timeout import expect_timeout, polls, solver  # noqa: F401 (polls: a fixture)

pytestmark = pytest.mark.gpu


def twin():
    s = solver()
    s.step(2)
    s.step(2)
    out = s.max_wave_speed(), s.state()
    s.close()
    return out


def test_solver_steps_on_with_the_flag_set(polls):  # noqa: F811
    want = twin()
    s = solver()
    polls(0)
    s.step(1, wait=False)
    polls(65536)
    s.prepare_state("freestream")
    s.step(2, wait=False)
    s.step(2, wait=False)
    expect_timeout(s.synchronize)
    assert s.max_wave_speed() == want[0]
    np.testing.assert_array_equal(s.state(), want[1])
    s.close()


def test_batch_steps_on_with_the_flag_set(polls):  # noqa: F811
    import ausm
    want = twin()
    sols = [solver() for _ in range(2)]
    with ausm.Batch() as b:
        for s in sols:
            b.add(s)
        b.step(1)
        polls(0)
        b.step(1, wait=False)
        polls(65536)
        for s in sols:
            s.prepare_state("freestream")
        b.step(2, wait=False)
        b.step(2, wait=False)
        expect_timeout(b.synchronize)
    for s in sols:
        assert s.max_wave_speed() == want[0]
        np.testing.assert_array_equal(s.state(), want[1])
        s.close()
