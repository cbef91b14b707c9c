"""Short ghosted 1D grids, whose steps run in one cluster launch: cell counts
around its 128-cell tiles (a last tile of one or two cells shares its ghosts with
the one before) and its limit of 2048 cells, each kind of boundary, RK2 and RK3,
an even and an odd number of steps: bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 5.0 / 3.0


@pytest.mark.parametrize("N", [1, 2, 5, 127, 128, 129, 130, 131, 257, 1024, 2048, 2049])
@pytest.mark.parametrize("rec,rs,rk", [("minmod", 1, 2), ("wenoz", 1, 3), ("ppm", 0, 3), ("wenoz", 0, 2)])
def test_ghosted_tube_bitwise(oracle, N, rec, rs, rk):
    from verona_b200 import Solver

    rng = np.random.default_rng(N)
    dx, dt = 1.0 / 64, 0.3 / 64
    x = np.arange(N + 6) / (N + 6)
    P = np.zeros((3, N + 6), order="F")
    P[0] = np.where(x < 0.5, 8.0, 1.0) * (1 + 0.02 * rng.standard_normal(N + 6))
    P[1] = np.where(x < 0.5, 12.0, 0.05) * (1 + 0.02 * rng.standard_normal(N + 6))
    P[2] = np.where(x > 0.3, 0.1, 0.0) * rng.standard_normal(N + 6)
    faces = [(0, 1, (2, 0.5 * dt, 4.5 * dt, 0.9)), (1, 2, (1.0, 0, 0, 0.5, 0.1, -0.2))]  # decaying ghosts; an inflow
    for bc in ([], faces):
        s = Solver(1, (N,), G, (dx,), recon=rec, riemann=rs, rk=rk, n_iter=50, tol=1e-12, floor=1e-8)
        o = oracle.SolverND(1, (N,), P, G, 1e-8, 50, 1e-12, oracle.RECON[rec], rs, rk)
        o.set_grid(dx)
        for face, kind, par in bc:
            s.set_boundary(face, kind, par)
            o.set_boundary(face, kind, par)
        s.load_prims(P)
        for steps in (3, 4):
            s.step(dt, steps)
            o.step(dt, steps)
            got, ref = s.prims(), o.prims()
            assert np.array_equal(got, ref, equal_nan=True), (bc, steps, np.argwhere(got != ref)[:4])
        assert s.t == o.t
