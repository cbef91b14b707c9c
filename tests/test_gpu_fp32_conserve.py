"""The FP32-bulk form conserves: a cell's flux differences are formed and summed in
FP64 from the FP32 fluxes, so what leaves one cell enters the next, and the sums of
D, E and S over a grid whose faces see only the static medium keep to FP64 rounding.
With the sum in FP32 they drift by FP32 rounding, 1e3 times the bound and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0
STEPS = 6


def _blob(n):
    """A fast, dense, hot blob in the middle of a static uniform medium; it stays
    6 cells (two stencils) clear of every face for STEPS steps of RK3."""
    d = len(n)
    P = np.zeros((2 + d,) + tuple(m + 6 for m in n), order="F")
    x = np.meshgrid(*[np.arange(m + 6) - 2.5 - m / 2 for m in n], indexing="ij")
    inside = sum((c / (m / 8)) ** 2 for c, m in zip(x, n)) < 1
    P[0], P[1] = np.where(inside, 3.7, 1.0), np.where(inside, 0.9, 0.3)
    for a in range(d):
        P[2 + a] = np.where(inside, 0.6 - 0.25 * a, 0.0)
    return P


@pytest.mark.parametrize("n", [(121, 97), (256, 160)])
@pytest.mark.parametrize("rec,rs,rk", [("wenoz", "hllc", 3), ("ppm", "hll", 2), ("minmod", "hllc", 3)])
@pytest.mark.parametrize("guess", ["previous", "previous_w"])
def test_sums_of_u_keep_to_fp64_rounding(n, rec, rs, rk, guess):
    from verona_b200 import Solver

    d, P = len(n), _blob(n)
    inner = (slice(None),) + (slice(3, -3),) * d
    s = Solver(d, n, G, [1.0 / 64] * d, recon=rec, riemann=rs, rk=rk, precision="fp32", guess=guess, n_iter=50,
               tol=1e-12, floor=1e-8)
    s.load_prims(P)
    U0 = s.cons()[inner]
    s.step(0.2 / (d * 64), STEPS)
    U = s.cons()[inner]
    assert s.counters()[0] == 0 and np.max(np.abs(U - U0)) > 0.05  # it moved
    # per cell and stage: two operations per axis, three of the RK combination, whose
    # weights' rounding counts twice, each at most half an ulp of the largest |U|
    ops = (2 * d + 5) * rk * STEPS * U0[0].size
    for v in range(2 + d):
        bound = ops * 2.0**-53 * np.max(np.abs(U0[v]))
        drift = abs(np.sum(U[v] - U0[v], dtype=np.longdouble))
        assert drift <= bound, (v, float(drift), bound)
