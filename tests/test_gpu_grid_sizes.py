"""The one-kernel-at-a-time entry points at the edges of their tiles: rows of
fewer and more cells than a warp's 31 faces, columns of one face and of several
marching runs, cell counts beside a multiple of a CTA's. Bit for bit against the
oracle, FP64."""
import numpy as np
import pytest

from test_gpu_grid_kernels import FLOOR, G, _dev, _host, _lib, _p, _state

pytestmark = pytest.mark.gpu

SIZES = [(1, (1,)), (1, (257,)), (2, (1, 1)), (2, (30, 3)), (2, (64, 41)), (3, (1, 1, 1)), (3, (26, 2, 5)),
         (3, (33, 19, 14))]


@pytest.mark.parametrize("dims,n", SIZES)
@pytest.mark.parametrize("rec,rs", [(2, 0), (2, 1), (1, 1), (0, 0)])
def test_grid_kernels_at_tile_edges_bitwise(oracle, dims, n, rec, rs):
    import torch

    lib = _lib()
    P = _state(dims, n, 17)
    nn = tuple(n) + (1,) * (3 - dims)
    d = _dev(P)
    U = torch.zeros_like(d)
    assert lib.vb_grid_prim2con(dims, *nn, _p(d), G, _p(U), None) == 0
    ref_u = oracle.k_ptou(P, G)
    assert np.array_equal(_host(U), ref_u)
    F, ref_f = [], []
    for axis in range(dims):
        f = torch.zeros_like(d)
        assert lib.vb_grid_fluxes(dims, *nn, _p(d), G, FLOOR, axis, rec, rs, _p(f), None) == 0
        F.append(f)
        ref_f.append(oracle.k_fluxes(P, G, FLOOR, axis, rec, rs))
        assert np.array_equal(_host(f), ref_f[-1], equal_nan=True), axis
    out = torch.zeros_like(d)
    Fp = [_p(f) for f in F] + [None] * (3 - dims)
    assert lib.vb_grid_update(dims, *nn, _p(U), *Fp, 1e-3, 0.1, 0.2, 0.3, _p(out), None) == 0
    ref_o = oracle.k_update(ref_u, 1e-3, (0.1, 0.2, 0.3)[:dims], ref_f)
    assert np.array_equal(_host(out), ref_o, equal_nan=True)
    guess = d.clone()
    assert lib.vb_grid_con2prim(dims, *nn, _p(out), G, 50, 1e-12, _p(guess), None, None) == 0
    assert np.array_equal(_host(guess), oracle.k_utop(ref_o, P, G, 50, 1e-12), equal_nan=True)
