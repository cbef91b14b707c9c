"""The z-marching 3D stencil kernels on grids that are no multiple of their
32 x 8 column tiles, down to one cell per axis, in one and several z ranges."""
import numpy as np
import pytest

from helpers import jet_ic, nozzle_params

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0
# one cell per axis; one short of, equal to and one past a tile; two x tiles with a ragged y; odd z
SIZES = [(1, 1, 1), (31, 7, 5), (33, 9, 2), (32, 8, 3), (65, 20, 9), (40, 3, 33)]


def _run(n, steps, precision="fp64", **tuning):
    from verona_b200 import Solver

    dxs = [1.0 / 32] * 3
    s = Solver(3, n, G, dxs, recon="wenoz", riemann="hllc", rk=3, precision=precision, n_iter=50, tol=1e-12,
               floor=1e-8)
    s.set_tuning(**tuning)
    s.set_boundary(0, 2, nozzle_params(3, n, 5.0, gamma=G))
    s.load_prims(jet_ic(3, n, gamma=G, noise=0.03, seed=21))
    s.step(0.4 / (3 * 32), steps)
    assert s.counters()[0] == 0
    return s.prims()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("split", [0, 1])
def test_fp64_ragged_grid_matches_oracle_bitwise(oracle, n, split):
    got = _run(n, 3, split_con2prim=split)
    o = oracle.SolverND(3, n, jet_ic(3, n, gamma=G, noise=0.03, seed=21), G, 1e-8, 50, 1e-12, 2, 1, 3)
    o.set_grid(*[1.0 / 32] * 3)
    o.set_boundary(0, oracle.BC_NOZZLE, nozzle_params(3, n, 5.0, gamma=G))
    o.step(0.4 / (3 * 32), 3)
    assert int(np.sum(got != o.prims())) == 0


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("split", [0, 1])
def test_fp32_ragged_grid_planes_by_tma_and_by_loads(n, split):
    """The two stagings of the z-pair kernel agree bit for bit, and with the
    FP64 run to the FP32-bulk bar (L1 of rho and u at most 1e-5)."""
    a = _run(n, 3, "fp32", split_con2prim=split, tma_tiles=1)
    b = _run(n, 3, "fp32", split_con2prim=split, tma_tiles=0)
    assert np.array_equal(a, b)
    ref = _run(n, 3)
    for v in range(2):
        assert np.mean(np.abs(a[v] - ref[v])) <= 1e-5 * np.mean(np.abs(ref[v]))
