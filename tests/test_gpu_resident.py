"""Grids whose tiles all fit on the chip step in one launch per call (the resident kernel).
Its face, ghost and combination arithmetic is the stage kernels', each expression rounded
alike, so states, dt and wave speed must equal the stage kernels' bit for bit
(AUSM_TILE_ROWS keeps a solve on those): at tile remainders in both directions, one tile
that is its own neighbour, the smallest grid, the last size of 4-row tiles and of 8-row
tiles and the first beyond, for n that rotate the buffers differently (n = 3 writes the
result over the input) and for a call that takes two launches."""
import numpy as np
import pytest

from test_gpu_edges import solver

pytestmark = pytest.mark.gpu

CASES = [(4, 2, "SLAU2", 1), (5, 9, "SLAU", 1), (33, 5, "AUSM+-up", 0), (32, 4, "SLAU2", 0), (65, 33, "AUSM+-up", 1),
         (257, 131, "SLAU", 0), (640, 148, "SLAU2", 1), (640, 149, "SLAU", 1), (768, 296, "AUSM+-up", 1),
         (768, 297, "SLAU2", 1)]


def run(M, N, frames, **kw):
    s = solver(M, N, **kw)
    out = []
    for n in frames:
        dt = s.step(n)
        out.append((dt, s.max_wave_speed(), s.state()))
    s.close()
    return out


@pytest.mark.parametrize("M,N,scheme,muscl", CASES)
def test_resident_steps_bit_identical(M, N, scheme, muscl, monkeypatch):
    frames = (1, 2, 3, 7, 2060) if M * N < 100 else (1, 2, 3, 7)
    got = run(M, N, frames, scheme=scheme, muscl=muscl, mach=1.4, K_p=0.25)
    monkeypatch.setenv("AUSM_TILE_ROWS", "16")
    want = run(M, N, frames, scheme=scheme, muscl=muscl, mach=1.4, K_p=0.25)
    for (dt, w, q), (dt1, w1, q1) in zip(got, want):
        assert dt == dt1 and w == w1
        np.testing.assert_array_equal(q, q1)


def test_resident_batch_bit_identical(monkeypatch):
    """A batch that fits on the chip against the batched stage kernels, with a member leaving
    (more tiles of the lower height then fit) and one large member joining (none fit)."""
    from ausm import Batch
    sizes = [(640, 60, "SLAU2"), (257, 131, "AUSM+-up"), (33, 17, "SLAU"), (128, 96, "SLAU2"), (4, 2, "SLAU2")]

    def go():
        sol = [solver(M, N, scheme=sc, muscl=k % 4 != 3, mach=1.2 + 0.1 * k) for k, (M, N, sc) in enumerate(sizes)]
        big = solver(1024, 400, mach=2.0)
        out = []
        with Batch() as b:
            for s in sol:
                b.add(s)
            for n in (1, 3, 5):
                out.append(b.step(n))
            out.append(b.residual_l2())
            b.remove(sol[0])
            out.append(b.step(4))
            b.add(big)
            out.append(b.step(2))
            b.remove(big)
            out.append(b.step(2))
        out += [s.state() for s in sol + [big]]
        for s in sol + [big]:
            s.close()
        return out
    got = go()
    monkeypatch.setenv("AUSM_TILE_ROWS", "8")
    for a, c in zip(got, go()):
        np.testing.assert_array_equal(a, c)
