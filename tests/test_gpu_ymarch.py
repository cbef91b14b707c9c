"""The y-marching 2D stencil kernel of the FP32-bulk form (warps of 30 columns,
rows in pairs) at the edges of its strips and ranges."""
import numpy as np
import pytest

from helpers import jet_ic, nozzle_params

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0
# one cell per axis; one short of, equal to and one past a strip; several CTAs of strips; odd and many rows
SIZES = [(1, 1), (29, 2), (30, 3), (31, 33), (121, 8), (250, 67)]


def _run(n, rec, rs, rk, precision, **tuning):
    from verona_b200 import Solver

    s = Solver(2, n, G, [1.0 / 64] * 2, recon=rec, riemann=rs, rk=rk, precision=precision, n_iter=50, tol=1e-12,
               floor=1e-8)
    s.set_tuning(**tuning)
    s.set_boundary(0, 2, nozzle_params(2, n + (1,), 3.0, gamma=G))
    s.load_prims(jet_ic(2, n, gamma=G, noise=0.03, seed=9))
    s.step(0.4 / (2 * 64), 4)
    c = s.counters()
    assert c[0] == 0 and c[4] == 0  # no con2prim failure, no row wait ran out
    return s.prims()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("rec,rs,rk", [("wenoz", "hllc", 3), ("ppm", "hll", 2), ("minmod", "hllc", 2)])
def test_fp32_ymarch_rows_by_tma_and_by_loads_and_the_box_kernel(n, rec, rs, rk):
    """Both stagings agree bit for bit; the one-cell-per-thread box kernel to
    FP32 rounding (2e-6 in the mean, as the 3D pair kernel's test); the FP64 run
    to the FP32-bulk bar (L1 of rho and u at most 1e-5)."""
    a = _run(n, rec, rs, rk, "fp32", tma_tiles=1)
    assert np.array_equal(a, _run(n, rec, rs, rk, "fp32", tma_tiles=0))
    box = _run(n, rec, rs, rk, "fp32", fp32_pairs=0)
    ref = _run(n, rec, rs, rk, "fp64")
    for v in range(4):
        scale = np.mean(np.abs(ref[v])) if v < 2 else 1.0
        assert np.mean(np.abs(a[v] - box[v])) <= 2e-6 * scale
    for v in range(2):
        assert np.mean(np.abs(a[v] - ref[v])) <= 1e-5 * np.mean(np.abs(ref[v]))
