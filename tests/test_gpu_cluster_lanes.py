"""The 1D cluster kernels where the lanes of a warp leave con2prim at different
times (one Newton step to the limit of n_iter, cells without a root among them)
just before the cluster meets: bit for bit against the oracle, and the counters
of the kernels that run a stage at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 5.0 / 3.0


def _state(N, ghosts, seed):
    """Cells at rest (few Newton steps) with fast, cold ones among them."""
    rng = np.random.default_rng(seed)
    P = np.zeros((3, N + 2 * ghosts), order="F")
    P[0] = 1 + 0.1 * rng.random(N + 2 * ghosts)
    P[1] = 0.5
    fast = rng.random(N + 2 * ghosts) < 0.15
    P[1, fast], P[2, fast] = 1e-4, 8.0 * rng.standard_normal(int(fast.sum()))
    return P


@pytest.mark.parametrize("stats", [0, 1])
@pytest.mark.parametrize("n_iter", [3, 50])
@pytest.mark.parametrize("rs,rk", [(0, 2), (1, 3)])
def test_tube_with_uneven_newton_lengths(oracle, rs, rk, n_iter, stats):
    from verona_b200 import Solver

    N, dx, dt = 300, 1.0 / 300, 0.2 / 300
    P = _state(N, 3, 5)
    out = []
    for per_stage in (False, True):  # profiling takes the stage kernels
        s = Solver(1, (N,), G, (dx,), recon="minmod", riemann=rs, rk=rk, n_iter=n_iter, tol=1e-12, floor=1e-8, stats=stats)
        s.profile(per_stage)
        s.load_prims(P)
        s.step(dt, 4)
        out.append((s.prims(), s.counters()))
    o = oracle.SolverND(1, (N,), P, G, 1e-8, n_iter, 1e-12, oracle.RECON["minmod"], rs, rk)
    o.set_grid(dx)
    o.step(dt, 4)
    for p, _ in out:
        assert np.array_equal(p, o.prims(), equal_nan=True)
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n_iter", [3, 50])
def test_reference_tube_with_uneven_newton_lengths(oracle, n_iter):
    from verona_b200 import Solver

    N = 300
    P = _state(N, 0, 6)
    s = Solver(1, (N,), G, (1.0 / N,), nghost=0, recon="minmod", n_iter=n_iter, tol=1e-12)
    s.load_prims(P)
    o = oracle.Solver1DRef(P[0], P[1], P[2], G, "minmod", n_iter, 1e-12)
    s.step(0.2 / N, 4)
    o.step(0.2 / N, 1.0 / N, 4)
    assert np.array_equal(s.prims(), o.prims(), equal_nan=True)
