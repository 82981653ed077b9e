"""Tiled grid sweeps against the oracle's whole-grid sweeps, where the tiles can go wrong:
sweep counts that leave a shorter last launch, grids narrower than a tile with its halo
(columns wrap several times), odd M (the seam column has colours of its own), tile
remainders, one and two sweeps per launch.  Jacobi (FP32) must equal the float oracle bit
for bit; the multicolour sweeps are FP64 in the oracle's operation order, so the vertices
rounded to float32 may differ by one unit in the last place where a last bit of FP64 turns
a rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(4, 2), (7, 3), (49, 34), (48, 65), (131, 50), (640, 260), (643, 300)]


def grids(M, N, sweeps, method):
    from ausm import Solver
    from oracle.geometry_ref import naca4_boundary, rectangular_outer
    from oracle.oracle import Oracle
    body, outer = naca4_boundary(M, 12, 0.3, -0.7), rectangular_outer(M, 1.5)
    o = Oracle(M, N, "f32" if method == "jacobi" else "f64")
    dt = np.float32 if method == "jacobi" else np.float64
    v = np.zeros((N + 1, M, 2), dt)
    v[0], v[N] = body, outer
    o.set_vertices(v)
    o.grid_interpolate()
    if method == "jacobi":
        o.grid_jacobi(sweeps)
    else:
        o.grid_multicolor(sweeps, 0.0)
    ref = o.vertices()
    o.close()
    s = Solver(M, N)
    s.set_body_points(body)
    s.set_outer_rect(1.5)
    assert s.generate_grid(sweeps, method) == sweeps
    g = s.vertices()
    s.close()
    return g, ref


@pytest.mark.parametrize("M,N", SIZES)
@pytest.mark.parametrize("sweeps", [1, 8, 21])
def test_sweeps_match_oracle(M, N, sweeps):
    g, ref = grids(M, N, sweeps, "jacobi")
    np.testing.assert_array_equal(g, ref)
    g, ref = grids(M, N, sweeps, "multicolor")
    ref = ref.astype(np.float32)
    assert np.all(np.abs(g - ref) <= np.spacing(np.abs(ref)))
