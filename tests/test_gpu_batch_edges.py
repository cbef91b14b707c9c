"""Batched problems whose last tile along an axis holds one or two cells, so that
the tile before it has ghosts in its halo too, in every tile variant: states that
vary up to the faces, every kind of boundary, ghosts included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 5.0 / 3.0
OPTS = dict(riemann="hllc", n_iter=50, tol=1e-12, floor=1e-8)
# one and two past a multiple of the tile extents 4, 8, 16, 32, 64 and the pencils 128, 256, 512
SIZES_2D = [(33, 9), (34, 10), (65, 17), (66, 34), (18, 5)]
SIZES_1D = [129, 130, 257, 258, 513, 514]
RECON = ["wenoz", "ppm", "minmod"]


def _problems():
    out = []
    for k, n in enumerate([(m,) for m in SIZES_1D] + SIZES_2D):
        d = len(n)
        rng = np.random.default_rng(50 + k)
        shape = tuple(m + 6 for m in n)
        x = np.meshgrid(*[np.arange(m) / 9.0 for m in shape], indexing="ij")
        wave = sum(np.sin(x[a] * (1 + 0.3 * a) + k) for a in range(d))
        P = np.zeros((2 + d,) + shape, order="F")
        P[0] = 1 + 0.2 * wave + 0.02 * rng.standard_normal(shape)
        P[1] = 0.5 + 0.1 * wave + 0.01 * rng.standard_normal(shape)
        for a in range(d):
            P[2 + a] = 0.3 * np.cos(x[a] + k) + 0.01 * rng.standard_normal(shape)
        dx = 1.0 / 64
        spec = {"dims": d, "n": n, "recon": RECON[k % 3], "dx": dx, "dy": dx, "dt": 0.3 * dx / d}
        nozzle = [2.5, n[-1] / 2 if d == 2 else 0.0, 0.0, 0.7, 0.4, -0.2] + [0.1] * (d - 1)
        decay = (2.0, 0.5 * spec["dt"], 3.5 * spec["dt"], 0.8)
        bcs = []  # outflow on every face
        if k % 3 == 1:
            bcs = [(1, 1, decay), (0, 2, nozzle)] + ([(3, 2, [2.5, n[0] / 2] + nozzle[2:])] if d == 2 else [])
        if k % 3 == 2:
            bcs = [(1, 2, nozzle), (0, 1, ())] + ([(3, 1, decay), (2, 2, [2.5, n[0] / 2] + nozzle[2:])] if d == 2 else [])
        out.append((spec, P, bcs))
    return out


def _batch(probs, rk, precision, variant):
    from verona_b200.batch import Batch

    b = Batch([p[0] for p in probs], G, rk=rk, precision=precision, **OPTS)
    b.set_tuning(variant)
    for i, (_, P, bcs) in enumerate(probs):
        b.load_prims(i, P)
        for face, kind, par in bcs:
            b.set_boundary(i, face, kind, par)
    b.step(2)
    b.step(3)
    assert b.check() == 0 and b.counters()[0] == 0
    out = [b.prims(i) for i in range(len(probs))]
    b.close()
    return out


def _parts(a, d):
    """The interior and, in 2D, the ghosts without their corners."""
    if d == 1:
        return [a]
    return [a[:, 3:-3, 3:-3], a[:, :3, 3:-3], a[:, -3:, 3:-3], a[:, 3:-3, :3], a[:, 3:-3, -3:]]


@pytest.mark.parametrize("rk", [2, 3])
@pytest.mark.parametrize("variant", [0, 1])
def test_fp64_short_last_tiles_match_the_oracle_bitwise(oracle, rk, variant):
    probs = _problems()
    for (spec, P, bcs), got in zip(probs, _batch(probs, rk, "fp64", variant)):
        d = spec["dims"]
        o = oracle.SolverND(d, spec["n"], P, G, OPTS["floor"], OPTS["n_iter"], OPTS["tol"],
                            oracle.RECON[spec["recon"]], oracle.HLLC, rk)
        o.set_grid(spec["dx"], spec["dy"])
        for face, kind, par in bcs:
            o.set_boundary(face, kind, par if kind != 1 or len(par) else (-1.0, 0.0, 0.0, 1.0))
        o.step(spec["dt"], 5)
        for x, y in zip(_parts(got, d), _parts(o.prims(), d)):
            assert np.array_equal(x, y), (spec, bcs, np.argwhere(x != y)[:4])


@pytest.mark.parametrize("rk", [2, 3])
def test_fp32_variants_agree_bitwise_on_short_last_tiles(rk):
    """The tile shapes, whose last tiles are short for different problems, do the
    same arithmetic per cell (the FP64 forms above share their ghost rule)."""
    probs = _problems()
    base = _batch(probs, rk, "fp32", 0)
    for variant in (1, 2, 3):
        for (spec, _, _), x, y in zip(probs, base, _batch(probs, rk, "fp32", variant)):
            for u, v in zip(_parts(x, spec["dims"]), _parts(y, spec["dims"])):
                assert np.array_equal(u, v), (variant, spec, np.argwhere(u != v)[:4])
