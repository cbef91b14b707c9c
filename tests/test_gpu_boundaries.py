"""Every mixture of face kinds through the one-launch boundary fill, ghost
corners included, against the oracle's face-by-face fill, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 4.0 / 3.0


@pytest.mark.parametrize("dims,n", [(2, (5, 4)), (2, (40, 9)), (3, (4, 5, 3)), (3, (35, 6, 7))])
@pytest.mark.parametrize("seed", range(6))
def test_mixed_face_kinds_with_corners_bitwise(oracle, dims, n, seed):
    from verona_b200 import Solver

    rng = np.random.default_rng(100 * dims + seed)
    shape = (2 + dims,) + tuple(x + 6 for x in n)
    P = np.zeros(shape, order="F")
    P[0] = 1 + 0.1 * rng.standard_normal(shape[1:])
    P[1] = 0.05 * (1 + 0.1 * rng.standard_normal(shape[1:]))
    P[2:] = 0.05 * rng.standard_normal((dims,) + shape[1:])
    P[1].flat[:: 7 + seed] = 1e-9  # below the floor in some cells and ghosts
    dt = 0.2 / (dims * 32)
    s = Solver(dims, n, G, [1.0 / 32] * dims, recon="wenoz", riemann="hllc", rk=3 - seed % 2, n_iter=50, tol=1e-12,
               floor=1e-8)
    o = oracle.SolverND(dims, n, P, G, 1e-8, 50, 1e-12, 2, 1, 3 - seed % 2)
    o.set_grid(*[1.0 / 32] * dims)
    for face in range(2 * dims):
        kind = int(rng.integers(3))
        par = ()
        if kind == 1 and rng.integers(2):
            par = (2, 0.5 * dt, 9 * dt, 0.8)
        if kind == 2:
            vel = [0.0] * dims
            vel[face // 2] = 0.3 if face % 2 == 0 else -0.3
            par = (2.2, n[0 if face > 1 else 1] / 2, n[-1] / 2, 0.4, 0.02, *vel)
        s.set_boundary(face, kind, par)
        o.set_boundary(face, kind, par)
    s.load_prims(P)
    s.step(dt, 3)
    o.step(dt, 3)
    assert np.array_equal(s.prims(), o.prims(), equal_nan=True)
