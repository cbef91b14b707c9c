"""The 1D reference solver on clusters of 1 to 16 CTAs: cell counts around the
cluster sizes' limits and the tile of a CTA, against the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [6, 7, 63, 64, 65, 127, 500, 1023, 1025, 8191, 20000])
@pytest.mark.parametrize("rec", ["minmod", "ppm", "wenoz"])
def test_ref1d_any_number_of_cells_bitwise(oracle, N, rec):
    from verona_b200 import Solver

    rng = np.random.default_rng(N)
    g, x = 5.0 / 3.0, (np.arange(N) + 0.5) / N
    left = x < 0.45
    rho = np.where(left, 10.0, 1.0) * (1 + 0.02 * rng.standard_normal(N))
    u = np.where(left, 13.33, 1e-2) / (g - 1) * (1 + 0.02 * rng.standard_normal(N))
    ux = 0.1 * rng.standard_normal(N) * (x > 0.2)  # some cells exactly at rest
    s = Solver(1, (N,), g, (1.0 / N,), nghost=0, recon=rec, n_iter=50, tol=1e-12)
    s.load_prims(np.asfortranarray(np.stack([rho, u, ux])))
    o = oracle.Solver1DRef(rho, u, ux, g, rec, 50, 1e-12)
    for steps in (1, 4):  # two calls: the edge states and frozen cells carry over
        s.step(0.3 / N, steps)
        o.step(0.3 / N, 1.0 / N, steps)
        assert np.array_equal(s.prims(), o.prims(), equal_nan=True)
        assert np.array_equal(s.cons(), o.cons(), equal_nan=True)
