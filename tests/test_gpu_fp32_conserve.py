"""The FP32-bulk form conserves: a cell's flux differences are formed and summed in
FP64 from the FP32 fluxes, so what leaves one cell enters the next, and the sums of
D, E and S over a grid whose faces see only the static medium keep to FP64 rounding.
With the sum in FP32 they drift by FP32 rounding, 1e3 times the bound and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0


def _blob(n):
    """A fast, dense, hot blob in the middle of a static uniform medium, 3/8 of the
    width from every face. A stage moves its effect by 3 cells at most, so
    3 x stages <= 3/8 of the width keeps it from the faces' fluxes. (The medium stays
    uniform because con2prim's Newton ends in FP64, c2p_fp32 = 0: from the network's
    guess the FP32 one leaves it an ulp off the ghosts, and the faces see that.)"""
    d = len(n)
    P = np.zeros((2 + d,) + tuple(m + 6 for m in n), order="F")
    x = np.meshgrid(*[np.arange(m + 6) - 2.5 - m / 2 for m in n], indexing="ij")
    inside = sum((c / (m / 8)) ** 2 for c, m in zip(x, n)) < 1
    P[0], P[1] = np.where(inside, 3.7, 1.0), np.where(inside, 0.9, 0.3)
    for a in range(d):
        P[2 + a] = np.where(inside, 0.6 - 0.25 * a, 0.0)
    return P


def _check(n, steps, rec, rs, rk, guess, **tuning):
    from verona_b200 import Solver, mlp

    assert 3 * rk * steps <= 0.375 * min(n)
    d, P = len(n), _blob(n)
    inner = (slice(None),) + (slice(3, -3),) * d
    s = Solver(d, n, G, [1.0 / 64] * d, recon=rec, riemann=rs, rk=rk, precision="fp32", guess=guess, n_iter=50,
               tol=1e-12, floor=1e-8, c2p_fp32=0)
    s.set_tuning(**tuning)
    if guess == "learned":
        mlp.attach(s)
    s.load_prims(P)
    U0 = s.cons()[inner]
    s.step(0.2 / (d * 64), steps)
    U = s.cons()[inner]
    c = s.counters()
    assert c[0] == 0 and c[4] == 0 and np.max(np.abs(U - U0)) > 0.02  # it moved
    # per cell and stage: two operations per axis, three of the RK combination, whose
    # weights' rounding counts twice, each at most half an ulp of the largest |U|
    ops = (2 * d + 5) * rk * steps * U0[0].size
    for v in range(2 + d):
        bound = ops * 2.0**-53 * np.max(np.abs(U0[v]))
        drift = abs(np.sum(U[v] - U0[v], dtype=np.longdouble))
        assert drift <= bound, (v, float(drift), bound)


SCHEMES = [("wenoz", "hllc", 3), ("ppm", "hll", 2), ("minmod", "hllc", 3)]


@pytest.mark.parametrize("n", [(121, 97), (256, 160)])
@pytest.mark.parametrize("rec,rs,rk", SCHEMES)
@pytest.mark.parametrize("guess", ["previous", "previous_w"])
def test_2d_sums_of_u_keep_to_fp64_rounding(n, rec, rs, rk, guess):
    _check(n, 4, rec, rs, rk, guess)


@pytest.mark.parametrize("n", [(50, 52, 49), (64, 50, 51), (81, 48, 50)])
@pytest.mark.parametrize("rec,rs,rk", SCHEMES)
@pytest.mark.parametrize("guess,tuning", [("previous", {}), ("previous", {"split_con2prim": 0}),
                                          ("previous", {"fp32_pairs": 0}), ("previous_w", {"tma_tiles": 0}),
                                          ("learned", {}), ("learned", {"learned_fused": 0})])
def test_ragged_3d_sums_of_u_keep_to_fp64_rounding(n, rec, rs, rk, guess, tuning):
    """Grids that are no multiple of the 32 x 8 column tiles."""
    _check(n, 2, rec, rs, rk, guess, **tuning)
