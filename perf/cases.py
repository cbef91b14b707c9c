"""Performance cases of the SRHD step library: what its users have it do.

Every case is one stretch of work between two points where a program looks at
its state: the primitives are loaded, a few time steps run, the primitives are
read back (kind "jet", "tube", "tube_reference"); a batch of uneven problems is
advanced (kind "batch"); or one midpoint stage is done kernel by kernel on the
caller's own arrays (kind "kernels"). Sizes come from the repository's tests and
benchmark (tubes of 256 to 8192 cells, 2D grids to 4096^2, 3D grids to 512^3,
odd and ragged ones among them), physics from its jets and shock tubes.

The FP32-bulk form holds its primitives in single precision, so its snapshots
are handed out in single precision; FP64 snapshots in double.

`exact` restates the scheme (reconstruction, HLL / HLLC, midpoint RK2 / SSP-RK3,
con2prim, ghost fill, floors) in plain 64-bit torch.
"""
import ctypes as C
import math

import torch

from verona_b200 import Solver, _lib
from verona_b200 import mlp
from verona_b200.batch import Batch

GAMMA_JET = 4.0 / 3.0
GAMMA_TUBE = 5.0 / 3.0
FLOOR = 1e-8
N_ITER, TOL = 50, 1e-12


# ---- the cases -------------------------------------------------------------------
def _jet(name, dims, n, recon, riemann, rk, precision, guess, steps):
    c = {"kind": "jet", "dims": dims, "nx": n[0], "ny": n[1], "nz": n[2] if dims == 3 else 1, "recon": recon,
         "riemann": riemann, "rk": rk, "precision": precision, "guess": guess, "steps": steps}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The 1D reference solver on the shock tube of the examples: the smallest grid, one launch per call.
        {"name": "tube1d_reference", "kind": "tube_reference", "n": 1024, "recon": "wenoz", "steps": 50},
        # The configured tube, MINMOD + HLLC + RK2 with ghost cells: tiny launches, latency is all there is.
        {"name": "tube1d_hllc", "kind": "tube", "n": 1024, "recon": "minmod", "riemann": "hllc", "rk": 2, "steps": 10},
        # A 2D jet while a setup is being tried out: the reference's own scheme, small and ragged.
        _jet("jet2d_small_fp64", 2, (300, 150), "wenoz", "hll", 2, "fp64", "previous", 5),
        # The 2D production jet in plain FP64, bit-exact.
        _jet("jet2d_large_fp64", 2, (4096, 4096), "wenoz", "hllc", 3, "fp64", "previous", 1),
        # The 2D jet in the FP32-bulk form with its fastest con2prim, on an odd grid.
        _jet("jet2d_odd_fp32", 2, (2047, 1021), "wenoz", "hllc", 3, "fp32", "previous_w", 2),
        # A 3D jet at test resolution, the reference's scheme: few tiles, many launches.
        _jet("jet3d_small_fp64", 3, (64, 48, 48), "wenoz", "hll", 2, "fp64", "previous", 5),
        # A 3D jet in plain FP64 on a grid that is no multiple of any tile.
        _jet("jet3d_ragged_fp64", 3, (200, 100, 100), "wenoz", "hllc", 3, "fp64", "previous", 1),
        # The 3D PPM jet in the FP32-bulk form with the reference con2prim.
        _jet("jet3d_ppm_fp32", 3, (256, 128, 128), "ppm", "hllc", 3, "fp32", "previous", 2),
        # The 3D learned-guess jet on an elongated ragged box, as jets are run.
        _jet("jet3d_ragged_learned", 3, (300, 125, 125), "wenoz", "hllc", 3, "fp32", "learned", 2),
        # The headline: 512^3, WENOZ + HLLC + SSP-RK3, learned guess, FP32 bulk.
        _jet("jet3d_512_learned", 3, (512, 512, 512), "wenoz", "hllc", 3, "fp32", "learned", 2),
        # Uneven 1D tubes and 2D quadrant problems advanced together, FP32 bulk.
        {"name": "batch_mixed", "kind": "batch", "n1d": 36, "n2d": 12, "mix": 7, "precision": "fp32", "steps": 2},
        # A program that replaces the reference's kernels one by one on its own arrays.
        {"name": "kernels3d_fp64", "kind": "kernels", "nx": 120, "ny": 62, "nz": 62, "recon": "wenoz",
         "riemann": "hll"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jet2d", "jet2d", "jet3d", "jet3d", "jet3d", "jet3d", "tube", "tube_reference", "batch",
                       "kernels"])
    recon = rng.choice(["wenoz", "wenoz", "ppm", "minmod"])
    riemann, rk = rng.choice([("hll", 2), ("hllc", 3)])
    if kind == "tube_reference":
        return {"kind": kind, "n": _log(rng, 256, 8192), "recon": recon, "steps": rng.randint(20, 60)}
    if kind == "tube":
        return {"kind": kind, "n": _log(rng, 256, 8192), "recon": recon, "riemann": riemann, "rk": rk,
                "steps": rng.randint(5, 20)}
    if kind == "batch":
        return {"kind": kind, "n1d": rng.randint(8, 40), "n2d": rng.randint(3, 16), "mix": rng.randrange(1 << 20),
                "precision": rng.choice(["fp32", "fp32", "fp64"]), "steps": rng.choice([1, 2, 4])}
    if kind == "kernels":
        return {"kind": kind, "nx": _log(rng, 24, 240), "ny": _log(rng, 24, 130), "nz": _log(rng, 24, 130),
                "recon": recon, "riemann": riemann}
    precision = rng.choice(["fp64", "fp32"])
    steps = rng.choice([1, 2, 3])
    if kind == "jet2d":
        guess = "previous" if precision == "fp64" else rng.choice(["previous", "previous_w"])
        n = (_log(rng, 100, 4096), _log(rng, 60, 2500))
        return _jet(None, 2, n, recon, riemann, rk, precision, guess, steps)
    guess = "previous" if precision == "fp64" else rng.choice(["previous", "previous_w", "learned", "learned"])
    most = 300 if precision == "fp64" else 420
    n = [_log(rng, 40, most), _log(rng, 32, 0.6 * most), _log(rng, 32, 0.6 * most)]
    if rng.random() < 0.4:  # powers of two and their halves are as usual as odd sizes
        n = [max(32, x // 32 * 32) for x in n]
    return _jet(None, 3, n, recon, riemann, rk, precision, guess, steps)


# ---- inputs -----------------------------------------------------------------------
def _dims(case):
    return {"jet": case.get("dims"), "tube": 1, "tube_reference": 1, "kernels": 3}[case["kind"]]


def _size(case):
    if "n" in case:
        return (case["n"],)
    return tuple(case[k] for k in ("nx", "ny", "nz"))[: _dims(case)]


def _gen(seed, device):
    return torch.Generator(device=device).manual_seed(int(seed))


def _beam(case, seed):
    """Beam of a jet: its Lorentz factor, how far it has come, radius in cells."""
    u = torch.rand(2, generator=_gen(seed, "cpu"), dtype=torch.float64)
    n = _size(case)
    return 4.0 + 4.0 * float(u[0]), (0.25 + 0.2 * float(u[1])) * n[0], max(3.0, min(n[1:]) / 16.0)


def _jet_state(case, seed):
    """A jet under way: a beam of light fast gas along x with a sheared edge, in
    a hotter cocoon, in a medium at rest with 3 % density noise. (Nz+6, Ny+6,
    Nx+6, nv) FP64, the library's padded layout."""
    dims, n = _dims(case), _size(case)
    lor, head, radius = _beam(case, seed)
    shape = tuple(m + 6 for m in reversed(n))
    P = torch.zeros(shape + (2 + dims,), dtype=torch.float64, device="cuda")
    x = [(torch.arange(m + 6, dtype=torch.float64, device="cuda") - 2.5) for m in n]
    r2 = (x[1] - n[1] / 2) ** 2
    r2 = r2.view(-1, 1) if dims == 2 else (x[2] - n[2] / 2).view(-1, 1, 1) ** 2 + r2.view(-1, 1)
    along = 0.5 * (1 - torch.tanh((x[0] - head) / 2.0))
    r = torch.sqrt(r2)
    beam = 0.5 * (1 - torch.tanh((r - radius) / 1.5)) * along
    noise = torch.randn(shape, generator=_gen(seed, "cuda"), dtype=torch.float64, device="cuda")
    P[..., 0] = (1 - beam) * (1 + 0.03 * noise) + 0.05 * beam
    P[..., 1] = 1e-3 / (GAMMA_JET - 1) * (1 + 9 * along * torch.exp(-((r / (2 * radius)) ** 2)))
    P[..., 2] = math.sqrt(lor**2 - 1) * torch.where(beam > 1e-6, beam, torch.zeros_like(beam))
    return P


def _nozzle(case, seed):
    lor, _, radius = _beam(case, seed)
    n = _size(case) + (0,)
    return [radius, n[1] / 2, n[2] / 2, 0.05, 1e-2 / (GAMMA_JET - 1), math.sqrt(lor**2 - 1), 0.0, 0.0]


def _tube_state(case, seed):
    """Shock tube 1 of Marti & Mueller, its states varied by the seed."""
    ghosts = 0 if case["kind"] == "tube_reference" else 3
    N = case["n"]
    u = torch.rand(3, generator=_gen(seed, "cpu"), dtype=torch.float64)
    x = torch.arange(N + 2 * ghosts, dtype=torch.float64, device="cuda") - ghosts + 0.5
    left = x < 0.5 * N
    P = torch.zeros((N + 2 * ghosts, 3), dtype=torch.float64, device="cuda")
    P[:, 0] = torch.where(left, 8.0 + 4.0 * float(u[0]), 1.0)
    P[:, 1] = torch.where(left, 10.0 + 5.0 * float(u[1]), 10.0 ** (-6 + 3 * float(u[2]))) / (GAMMA_TUBE - 1)
    return P


def _batch_specs(case):
    """Sizes, reconstructions and time steps of a batch (the same for every seed)."""
    g = _gen(case["mix"], "cpu")
    rnd = lambda lo, hi: int(torch.randint(lo, hi + 1, (1,), generator=g))  # noqa: E731
    specs = []
    for d, count, lo, hi in ((1, case["n1d"], 256, 8192), (2, case["n2d"], 128, 1024)):
        for _ in range(count):
            m = rnd(lo, hi)
            specs.append({"dims": d, "n": (m,) * d, "recon": ("minmod", "ppm", "wenoz")[rnd(0, 2)], "dx": 1.0 / m,
                          "dt": 0.4 / (d * m)})
    return specs


def _batch_states(case, seed):
    """Two states (1D) or four (2D) per problem meeting at the centre: density in
    [0.1, 10], pressure in [1e-2, 20], speed up to 0.6 in any direction."""
    g = _gen(seed, "cpu")
    rnd = lambda lo, hi: lo + (hi - lo) * float(torch.rand(1, generator=g, dtype=torch.float64))  # noqa: E731

    def state(d):
        v, a = rnd(0.0, 0.6), rnd(0.0, 2 * math.pi)
        u = v / math.sqrt(1 - v * v)
        rho, p = 10 ** rnd(-1.0, 1.0), 10 ** rnd(-2.0, math.log10(20.0))
        return [rho, p / (GAMMA_TUBE - 1)] + ([math.copysign(u, math.cos(a))] if d == 1
                                              else [u * math.cos(a), u * math.sin(a)])

    out = []
    for q in _batch_specs(case):
        d, m = q["dims"], q["n"][0]
        s = torch.tensor([state(d) for _ in range(2**d)], dtype=torch.float64, device="cuda")
        hi = (torch.arange(m + 6, device="cuda") - 2.5 > m / 2).long()
        out.append(s[hi] if d == 1 else s[hi.view(1, -1) + 2 * hi.view(-1, 1)])
    return out


def _make_solver(case, seed):
    dims, n = _dims(case), _size(case)
    opts = {"recon": case["recon"], "n_iter": N_ITER, "tol": TOL, "floor": FLOOR}
    if case["kind"] == "tube_reference":
        return Solver(1, n, GAMMA_TUBE, (1.0 / n[0],), nghost=0, **opts)
    opts.update(riemann=case["riemann"], rk=case["rk"])
    if case["kind"] == "tube":
        return Solver(1, n, GAMMA_TUBE, (1.0 / n[0],), **opts)
    s = Solver(dims, n, GAMMA_JET, (1.0 / n[0],) * dims, precision=case["precision"], guess=case["guess"], **opts)
    s.set_boundary("xlo", _lib.BC_NOZZLE, _nozzle(case, seed)[: 5 + dims])
    if case["guess"] == "learned":
        mlp.attach(s)
    return s


def _dt(case):
    return 0.4 / (_dims(case) * _size(case)[0])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = Batch(_batch_specs(case), GAMMA_TUBE, riemann="hllc", rk=3, precision=case["precision"], n_iter=N_ITER,
                  tol=TOL, floor=FLOOR)
        for i, P in enumerate(_batch_states(case, seed)):
            b.load_prims(i, P)
        b.checkpoint()
        outs = [torch.empty(b.device_shape(i), dtype=torch.float64, device="cuda") for i in range(b.nprob)]
        return {"case": case, "batch": b, "outs": outs}
    if kind == "kernels":
        lib = _lib.lib()
        vp, d, i = C.c_void_p, C.c_double, C.c_int
        lib.vb_grid_fluxes.argtypes = [i, i, i, i, vp, d, d, i, i, i, vp, vp]
        lib.vb_grid_update.argtypes = [i, i, i, i, vp, vp, vp, vp, d, d, d, d, vp, vp]
        lib.vb_grid_con2prim.argtypes = [i, i, i, i, vp, d, i, d, vp, vp, vp]
        lib.vb_grid_prim2con.argtypes = [i, i, i, i, vp, d, vp, vp]
        lib.vb_grid_limit.argtypes = [i, i, i, i, vp, d, vp]
        P = _jet_state(case, seed)
        return {"case": case, "lib": lib, "P": P, "work": [torch.zeros_like(P) for _ in range(6)]}
    P = _tube_state(case, seed) if kind.startswith("tube") else _jet_state(case, seed)
    return {"case": case, "solver": _make_solver(case, seed), "P": P, "out": torch.empty_like(P)}


# ---- one pass ---------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.rollback()
        b.step(case["steps"])
        outs = [b.store_prims(i, o) for i, o in enumerate(state["outs"])]
        # the interiors, as a dump has them (a batch never fills the ghost corners)
        outs = [o[3:-3] if o.dim() == 2 else o[3:-3, 3:-3] for o in outs]
        return [o.float() for o in outs] if case["precision"] == "fp32" else outs
    if case["kind"] == "kernels":
        return _kernel_stage(state)
    s = state["solver"]
    s.load_prims(state["P"])
    s.step(_dt(case), case["steps"])
    out = s.store_prims(state["out"])
    return out.float() if case.get("precision") == "fp32" else out


def _kernel_stage(state):
    """One midpoint stage, each of the reference's kernels a call of its own."""
    case, lib, P = state["case"], state["lib"], state["P"]
    U, Uh, Ph, Fx, Fy, Fz = state["work"]
    n, ptr = (3, case["nx"], case["ny"], case["nz"]), lambda t: C.c_void_p(t.data_ptr())
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rec, rs = _lib.RECON[case["recon"]], _lib.RIEMANN[case["riemann"]]
    dx = 1.0 / case["nx"]
    Ph.copy_(P)
    rc = lib.vb_grid_prim2con(*n, ptr(P), GAMMA_JET, ptr(U), stream)
    for axis, F in enumerate((Fx, Fy, Fz)):
        rc |= lib.vb_grid_fluxes(*n, ptr(P), GAMMA_JET, FLOOR, axis, rec, rs, ptr(F), stream)
    rc |= lib.vb_grid_update(*n, ptr(U), ptr(Fx), ptr(Fy), ptr(Fz), 0.5 * _dt(case), dx, dx, dx, ptr(Uh), stream)
    rc |= lib.vb_grid_con2prim(*n, ptr(Uh), GAMMA_JET, N_ITER, TOL, ptr(Ph), None, stream)
    rc |= lib.vb_grid_limit(*n, ptr(Ph), FLOOR, stream)
    if rc:
        raise RuntimeError("a grid kernel returned an error")
    return {"U": U, "Fx": Fx, "Fy": Fy, "Fz": Fz, "Uhalf": Uh, "Phalf": Ph}


# ---- what a pass cannot do without --------------------------------------------------
_RECON_OPS = {"minmod": 10, "ppm": 70, "wenoz": 75}
_FLUX_OPS = {"hll": 110, "hllc": 160}


def _stage_ops(dims, recon, riemann):
    return dims * ((2 + dims) * _RECON_OPS[recon] + _FLUX_OPS[riemann]) + 100


def _step_work(cells, dims, recon, riemann, rk, precision, steps):
    """P read and written once per stage, U read and written as the scheme needs it."""
    nv = 2 + dims
    pb = 4 if precision == "fp32" else 8
    u_passes = 8 if rk == 3 else 4
    stages = rk * steps
    return {"bytes": cells * nv * (2 * pb * stages + 8 * u_passes * steps),
            "flops": cells * stages * _stage_ops(dims, recon, riemann)}


def work(case):
    if case["kind"] == "batch":
        total = {"bytes": 0, "flops": 0}
        for q in _batch_specs(case):
            w = _step_work(q["n"][0] ** q["dims"], q["dims"], q["recon"], "hllc", 3, case["precision"], case["steps"])
            total = {k: total[k] + w[k] for k in total}
        return total
    dims, cells = _dims(case), math.prod(_size(case))
    if case["kind"] == "kernels":
        # P read by prim2con, each flux axis, con2prim (and written), limit; U, F, Uhalf written and read
        return {"bytes": cells * 5 * 8 * 14, "flops": cells * _stage_ops(3, case["recon"], case["riemann"])}
    w = _step_work(cells, dims, case["recon"], case.get("riemann", "hll"), case.get("rk", 2),
                   case.get("precision", "fp64"), case["steps"])
    w["bytes"] += cells * (2 + dims) * 8 * 2  # the state in, the state out
    return w


# ---- the scheme in 64 bits, plain torch ------------------------------------------------
def _minmod(a, b, c, d, e):
    s, t = d - c, c - b
    du = 0.25 * (torch.sign(s) + torch.sign(t)) * torch.minimum(s.abs(), t.abs())
    return c - du, c + du


def _weno_side(v0, v1, v2, v3, v4, i0, i1, i2):
    """Face value on the far side of v2 (towards v4) from its ratios tau / beta."""
    a0, a1, a2 = 0.1 * (1 + i0 * i0), 0.6 * (1 + i1 * i1), 0.3 * (1 + i2 * i2)
    num = a0 * (2 * v0 - 7 * v1 + 11 * v2) + a1 * (-v1 + 5 * v2 + 2 * v3) + a2 * (2 * v2 + 5 * v3 - v4)
    return num / (6 * (a0 + a1 + a2))


def _wenoz(a, b, c, d, e):
    b0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    tau, eps = (b0 - b2).abs(), 1e-42
    i0, i1, i2 = tau / (b0 + eps), tau / (b1 + eps), tau / (b2 + eps)
    return _weno_side(e, d, c, b, a, i2, i1, i0), _weno_side(a, b, c, d, e, i0, i1, i2)


def _ppm(a, b, c, d, e):
    """Interface values with their curvature limit, then the parabola's."""
    K = 1.25
    curv = (a + c - 2 * b, b + d - 2 * c, c + e - 2 * d)
    zero = torch.zeros_like(c)

    def same(*q):
        s = torch.sign(q[0])
        ok = torch.ones_like(s, dtype=torch.bool)
        for x in q[1:]:
            ok &= torch.sign(x) == s
        return ok

    def interface(l2, l, r, r2, cl, cr):
        f = 0.5 * (l + r) + (0.5 * (r - l2) - 0.5 * (r2 - l)) / 6
        top = 3 * (l + r - 2 * f)
        lim = torch.minimum(torch.minimum(K * cl.abs(), K * cr.abs()), top.abs())
        lim = torch.where(same(top, cl, cr), torch.sign(top) * lim, zero)
        return torch.where((f - l) * (r - f) < 0, 0.5 * (l + r) - lim / 6, f)

    lo, hi = interface(a, b, c, d, curv[0], curv[1]), interface(b, c, d, e, curv[1], curv[2])
    cf = 6 * (lo + hi - 2 * c)
    dm, dp = c - lo, hi - c
    lim = torch.minimum(torch.minimum(K * curv[0].abs(), K * curv[1].abs()),
                        torch.minimum(K * curv[2].abs(), cf.abs()))
    lim = torch.where(same(cf, *curv), torch.sign(cf) * lim, zero)
    big = torch.stack([x.abs() for x in (a, b, c, d, e)]).amax(0)
    rho = torch.where(cf.abs() > 1e-12 * big, lim / torch.where(cf == 0, torch.ones_like(cf), cf), zero)
    extremum = (dm * dp <= 0) | ((d - c) * (c - b) <= 0)
    scale = extremum & (rho <= 1 - 1e-12)
    qr = torch.where(scale, c - rho * dm, torch.where(~extremum & (dm.abs() >= 2 * dp.abs()), c - 2 * dp, lo))
    ql = torch.where(scale, c + rho * dp, torch.where(~extremum & (dp.abs() >= 2 * dm.abs()), c + 2 * dm, hi))
    return qr, ql


_RECON_FN = {"minmod": _minmod, "ppm": _ppm, "wenoz": _wenoz}


class _Face:
    """One side of the faces: conserved vector, flux along `axis`, signal speeds."""

    def __init__(self, P, axis, g):
        rho, u, m = P[0], P[1], P[2:]
        lor2 = 1 + (m * m).sum(0)
        lor, w, self.p, un = lor2.sqrt(), rho + g * u, (g - 1) * u, m[axis]
        self.U = torch.cat([(lor * rho)[None], (self.p - lor2 * w)[None], m * (lor * w)])
        self.F = torch.cat([(rho * un)[None], (-w * un * lor)[None], m * (un * w)])
        self.F[2 + axis] += self.p
        self.v = un / lor
        cs2 = g * self.p / w
        sig = cs2 / (lor2 * (1 - cs2))
        r = (sig * (1 - self.v**2 + sig)).sqrt()
        self.hi, self.lo = (self.v + r) / (1 + sig), (self.v - r) / (1 + sig)


def _flux(PL, PR, axis, g, riemann):
    L, R = _Face(PL, axis, g), _Face(PR, axis, g)
    hi, lo = torch.maximum(L.hi, R.hi), torch.minimum(L.lo, R.lo)
    F = (hi * L.F - lo * R.F + hi * lo * (R.U - L.U)) / (hi - lo)
    if riemann == "hllc":
        k = 2 + axis
        H = (hi * R.U - lo * L.U - (R.F - L.F)) / (hi - lo)
        E, m, FE, Fm = -H[1], H[k], -F[1], F[k]
        b = E + Fm
        ls = 2 * m / (b + (b * b - 4 * FE * m).clamp(min=0).sqrt())
        ps = Fm - FE * ls
        left = ls >= 0
        U, FK = torch.where(left, L.U, R.U), torch.where(left, L.F, R.F)
        lK, v, p = torch.where(left, lo, hi), torch.where(left, L.v, R.v), torch.where(left, L.p, R.p)
        S = U * ((lK - v) / (lK - ls))
        S[1] = -(-U[1] * (lK - v) + ps * ls - p * v) / (lK - ls)
        S[k] = (U[k] * (lK - v) + ps - p) / (lK - ls)
        good = (ps > 0) & (ls >= lo) & (ls <= hi)
        F = torch.where(good, FK + lK * (S - U), F)
    return torch.where(hi < 0, R.F, torch.where(lo > 0, L.F, F))


def _face_fluxes(P, axis, g, recon, riemann):
    """Fluxes of every face between cells 2 .. n-3 of the padded axis of P."""
    dim = P.dim() - 1 - axis
    n = P.shape[dim]
    sh = [P.narrow(dim, o, n - 4) for o in range(5)]
    both = [_RECON_FN[recon](*[q[v] for q in sh]) for v in range(P.shape[0])]
    qr, ql = torch.stack([x[0] for x in both]), torch.stack([x[1] for x in both])
    del both
    PL, PR = ql.narrow(dim, 0, n - 5), qr.narrow(dim, 1, n - 5)
    PL[:2].clamp_(min=FLOOR)
    PR[:2].clamp_(min=FLOOR)
    return _flux(PL, PR, axis, g, riemann)


def _inner(P, dims, but=()):
    for a in range(dims):
        if a not in but:
            dim = P.dim() - 1 - a
            P = P.narrow(dim, 3, P.shape[dim] - 6)
    return P


def _divergence(P, dims, g, dx, recon, riemann):
    div = 0
    for axis in range(dims):
        F = _face_fluxes(_inner(P, dims, (axis,)), axis, g, recon, riemann)
        dim = P.dim() - 1 - axis
        m = F.shape[dim] - 1
        div = div + (F.narrow(dim, 1, m) - F.narrow(dim, 0, m)) / dx
    return div


def _prim2con(P, g):
    lor2 = 1 + (P[2:] ** 2).sum(0)
    w = P[0] + g * P[1]
    return torch.cat([(lor2.sqrt() * P[0])[None], ((g - 1) * P[1] - lor2 * w)[None], P[2:] * (lor2.sqrt() * w)])


def _con2prim(U, P, g):
    """Newton on W = rho h Gamma^2 from the state P; where none is found, P stays."""
    D, S2, k = U[0], (U[2:] ** 2).sum(0), (g - 1) / g
    low = S2.sqrt() * (1 + 1e-15)
    W = torch.maximum((P[0] + g * P[1]) * (1 + (P[2:] ** 2).sum(0)), low)
    for _ in range(60):
        v2 = (S2 / W**2).clamp(max=1 - 1e-15)
        s = (1 - v2).sqrt()
        f = U[1] + W - k * (W * (1 - v2) - D * s)
        new = W - f / (1 - k * (1 + v2 - D * v2 / (W * s)))
        new = torch.where(new > low, new, 0.5 * (W + low))
        done = bool(((new - W).abs() <= 4e-16 * new).all())
        W = new
        if done:
            break
    s = (1 - S2 / W**2).sqrt()
    rho, u = D * s, (W * s * s - D * s) / g
    out = torch.cat([rho[None], u[None], U[2:] / (W * s)])
    return torch.where(torch.isfinite(out).all(0) & (u > 0), out, P)


def _fill(P, dims, nozzle):
    """Ghost fill at the start of a step: y, z, then x faces; the nozzle on x-lo."""
    for axis in [a for a in (1, 2, 0) if a < dims]:
        dim = P.dim() - 1 - axis
        n = P.shape[dim]
        P.narrow(dim, 0, 3).copy_(P.narrow(dim, 3, 1).expand_as(P.narrow(dim, 0, 3)))
        P.narrow(dim, n - 3, 3).copy_(P.narrow(dim, n - 4, 1).expand_as(P.narrow(dim, n - 3, 3)))
    if nozzle:
        y = torch.arange(P.shape[-2], dtype=torch.float64, device=P.device) - 2.5 - nozzle[1]
        r2 = y * y
        if dims == 3:
            z = torch.arange(P.shape[-3], dtype=torch.float64, device=P.device) - 2.5 - nozzle[2]
            r2 = r2 + z.view(-1, 1) ** 2
        inside = (r2 < nozzle[0] ** 2)[..., None].expand(P.shape[1:-1] + (3,))
        for v in range(2 + dims):
            P[v][..., :3][inside] = nozzle[3 + v]


def _evolve(P, dims, g, dx, dt, steps, recon, riemann, rk, nozzle=None):
    """P: (nv, [Nz+6, [Ny+6,]] Nx+6); the padded state after `steps` steps."""
    U0 = _inner(_prim2con(P, g), dims).clone()

    def stage(P, Us, h, a, b):
        out = P.clone()
        out[:2].clamp_(min=FLOOR)
        U, inner, guess = torch.empty_like(Us), _inner(out, dims), _inner(P, dims)
        slab = Us.shape[1] if dims < 3 else max(1, (1 << 25) // (Us.shape[2] * Us.shape[3]))
        for z in range(0, Us.shape[1], slab):
            m = min(slab, Us.shape[1] - z)
            block = P.narrow(1, z, m + 6) if dims == 3 else P
            sl = (slice(None), slice(z, z + m))
            u = b * (Us[sl] - h * _divergence(block, dims, g, dx, recon, riemann))
            U[sl] = u + a * U0[sl] if a else u
            q = _con2prim(U[sl], guess[sl], g)
            q[:2].clamp_(min=FLOOR)
            inner[sl] = q
        return out, U

    for _ in range(steps):
        _fill(P, dims, nozzle)
        if rk == 3:
            P, U = stage(P, U0, dt, 0.0, 1.0)
            P, U = stage(P, U, dt, 0.75, 0.25)
            P, U0 = stage(P, U, dt, 1 / 3, 2 / 3)
        else:
            half, _ = stage(P, U0, 0.5 * dt, 0.0, 1.0)
            P, U0 = stage(half, U0, dt, 0.0, 1.0)
    return P


def _evolve_reference_tube(P, g, dx, dt, steps, recon):
    """The reference's 1D solver: no ghosts; faces and cells at the ends keep
    what they had, face states are not floored."""
    N, reach = P.shape[1], 1 if recon == "minmod" else 2
    U, PL, PR = _prim2con(P, g), P.clone(), P.clone()

    def stage(P, base, h):
        m = N - 2 * reach
        q = [P[:, max(0, reach + o):][:, :m] for o in range(-2, 3)]  # MINMOD looks at the middle three only
        qr, ql = _RECON_FN[recon](*q)
        PR[:, reach - 1:reach - 1 + m] = qr
        PL[:, reach:reach + m] = ql
        F = _flux(PL, PR, 0, g, "hll")
        U = base.clone()
        U[:, 1:N - 2] -= h / dx * (F[:, 1:N - 2] - F[:, :N - 3])
        return U, _con2prim(U, P, g)

    for _ in range(steps):
        _, half = stage(P, U, 0.5 * dt)
        U, P = stage(half, U, dt)
    return P


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        outs = []
        for q, P in zip(_batch_specs(case), _batch_states(case, seed)):
            P = P.movedim(-1, 0).contiguous()
            P = _evolve(P, q["dims"], GAMMA_TUBE, q["dx"], q["dt"], case["steps"], q["recon"], "hllc", 3)
            outs.append(_inner(P, q["dims"]).movedim(0, -1).contiguous())
        return outs
    dims, dx, dt = _dims(case), 1.0 / _size(case)[0], _dt(case)
    if kind.startswith("tube"):
        P = _tube_state(case, seed).t().contiguous()
        if kind == "tube_reference":
            P = _evolve_reference_tube(P, GAMMA_TUBE, dx, dt, case["steps"], case["recon"])
        else:
            P = _evolve(P, 1, GAMMA_TUBE, dx, dt, case["steps"], case["recon"], case["riemann"], case["rk"])
        return P.t().contiguous()
    P = _jet_state(case, seed).movedim(-1, 0).contiguous()
    if kind == "jet":
        P = _evolve(P, dims, GAMMA_JET, dx, dt, case["steps"], case["recon"], case["riemann"], case["rk"],
                    _nozzle(case, seed))
        return P.movedim(0, -1).contiguous()
    U, Uh, Ph = _prim2con(P, GAMMA_JET), torch.zeros_like(P), P.clone()
    fluxes = []
    for axis in range(3):
        near = P
        for a in range(3):  # faces of the cells 2 .. n-4 on every axis
            if a != axis:
                near = near.narrow(3 - a, 2, P.shape[3 - a] - 5)
        F = torch.zeros_like(P)
        F[:, 2:-3, 2:-3, 2:-3] = _face_fluxes(near, axis, GAMMA_JET, case["recon"], case["riemann"])
        fluxes.append(F)
    _inner(Uh, 3).copy_(_inner(U, 3) - 0.5 * dt * _divergence(P, 3, GAMMA_JET, dx, case["recon"], case["riemann"]))
    _inner(Ph, 3).copy_(_con2prim(_inner(Uh, 3), _inner(P, 3), GAMMA_JET))
    Ph[:2].clamp_(min=FLOOR)
    outs = {"U": U, "Fx": fluxes[0], "Fy": fluxes[1], "Fz": fluxes[2], "Uhalf": Uh, "Phalf": Ph}
    return {k: v.movedim(0, -1).contiguous() for k, v in outs.items()}
