"""Performance cases of the finite-volume step: what a user's program has the library do, through the C ABI.

Families (``kind``):

- ``explicit``: K device-resident explicit steps (``sifv_advance``) in 1D / 2D / 3D, in each arithmetic mode
  (``fp64`` the default, ``fast``, ``mixed``), single- and two-phase, inviscid and viscous, over the boundary kinds.
- ``semi``: one semi-implicit step (``sifv_step``) with IGR and one of the three pressure solvers.
- ``adjoint``: K recorded forward steps and the reverse sweep (gradient of a scalar with respect to U(t0)).
- ``ensemble``: many two-phase water-air tubes of different sizes in one call (``sifv_ensemble_run``).

A pass puts the initial state into the context's device fields, runs the steps and leaves the results in device
memory; nothing but the time step and the step counts comes back to the host.  ``exact`` is the same scheme in
plain torch, double precision.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from semiimplicitfv_b200 import _lib, abi

F64 = torch.float64
PRECISION = {"fp64": abi.PREC_FP64, "fast": abi.PREC_FP64_FAST, "mixed": abi.PREC_MIXED}
RIEMANN = {"hllc": abi.HLLC, "rusanov": abi.RUSANOV, "lf": abi.LF}
BC = {"outflow": abi.BC_OUTFLOW, "periodic": abi.BC_PERIODIC, "slip": abi.BC_SLIPWALL, "noslip": abi.BC_NOSLIPWALL}
SOLVER = {"jacobi": abi.PRESSURE_JACOBI, "gs": abi.PRESSURE_GAUSS_SEIDEL, "pcg": abi.PRESSURE_PCG_MG}
GAMMA = 1.4
PH_GAMMA, PH_PINF, ALPHA_MIN = (4.4, 1.4), (6.0e8, 0.0), 1e-8   # water, air
VEL = (abi.F_VELU, abi.F_VELV, abi.F_VELW)
MOM = (abi.F_RHOU, abi.F_RHOV, abi.F_RHOW)


# ---------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------
def _explicit(nx, ny, nz, steps, precision="fp64", riemann="hllc", bc="outflow", flow="riemann", phases=0, mu=0.0):
    return {"kind": "explicit", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": precision,
            "riemann": riemann, "bc": bc, "flow": flow, "phases": phases, "mu": mu}


def _semi(nx, ny, nz, solver, bc, tol, igr=True):
    return {"kind": "semi", "nx": nx, "ny": ny, "nz": nz, "solver": solver, "bc": bc, "tol": tol, "igr": igr}


def _adjoint(n, m, steps, every, precision="fp64", bc="periodic"):
    return {"kind": "adjoint", "nx": n, "ny": m, "steps": steps, "every": every, "precision": precision, "bc": bc}


def _ensemble(tubes, lo, hi, steps, precision="mixed"):
    return {"kind": "ensemble", "tubes": tubes, "lo": lo, "hi": hi, "steps": steps, "precision": precision}


def listed():
    return [
        # the smallest calls: the 1D Sod tube every new user runs first; launches and latency
        dict(_explicit(1000, 1, 1, 20, flow="tube"), name="sod_1000"),
        # an example-sized 2D run in the default, bit-exact arithmetic
        dict(_explicit(256, 256, 1, 10), name="riemann2d_256"),
        # an ordinary production 2D run in the default arithmetic, ragged sizes, viscous walls
        dict(_explicit(1531, 1021, 1, 2, riemann="rusanov", bc="noslip", mu=0.01, flow="pulse"), name="viscous2d_1531x1021"),
        # the headline workload: four-quadrant Riemann problem 4096^2, fused FP64
        dict(_explicit(4096, 4096, 1, 2, precision="fast"), name="riemann2d_4096_fast"),
        # the same family in mixed precision, periodic vortex-like flow
        dict(_explicit(2048, 2048, 1, 4, precision="mixed", bc="periodic", flow="pulse"), name="pulse2d_2048_mixed"),
        # explicit 3D, odd sizes, fused FP64
        dict(_explicit(203, 160, 131, 2, precision="fast", bc="slip", flow="pulse"), name="pulse3d_203x160x131_fast"),
        # two-phase water / air in 2D (a drop hit by a shock), default arithmetic
        dict(_explicit(480, 352, 1, 3, phases=2, flow="drop"), name="drop2d_480x352"),
        # the semi-implicit workload: 3D low-Mach pulse, IGR, Jacobi, periodic
        dict(_semi(256, 256, 256, "jacobi", "periodic", 1e-6), name="semi3d_256_jacobi"),
        # 2D semi-implicit with the Gauss-Seidel solver of the 2D examples
        dict(_semi(384, 256, 1, "gs", "periodic", 1e-6), name="semi2d_384x256_gs"),
        # semi-implicit with PCG + multigrid, ragged box with walls
        dict(_semi(150, 96, 77, "pcg", "slip", 1e-10), name="semi3d_150x96x77_pcg"),
        # gradient of an objective with respect to the initial state
        dict(_adjoint(256, 256, 12, 6), name="adjoint_256"),
        # a batch of uneven shock tubes
        dict(_ensemble(400, 256, 4096, 40), name="ensemble_400"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["explicit1", "explicit2", "explicit2", "explicit3", "drop", "semi2", "semi3", "adjoint", "ensemble"])
    riemann = rng.choice(["hllc", "hllc", "rusanov", "lf"])
    if kind == "explicit1":
        return _explicit(_log_int(rng, 200, 20000), 1, 1, rng.randint(5, 30), rng.choice(["fp64", "fast"]), riemann,
                         rng.choice(["outflow", "slip"]), "tube")
    if kind == "explicit2":
        prec = rng.choice(["fp64", "fp64", "fast", "mixed"])
        top = 1600 if prec == "fp64" else 3600
        nx, ny = _log_int(rng, 96, top), _log_int(rng, 96, top)
        return _explicit(nx, ny, 1, rng.randint(1, 3), prec, riemann,
                         rng.choice(["outflow", "periodic", "slip", "noslip"]), rng.choice(["riemann", "pulse"]), 0,
                         rng.choice([0.0, 0.01]) if prec == "fp64" else 0.0)
    if kind == "explicit3":
        n = [_log_int(rng, 40, 160) for _ in range(3)]
        return _explicit(*n, rng.randint(1, 2), rng.choice(["fp64", "fast", "mixed"]), riemann,
                         rng.choice(["outflow", "periodic", "slip"]), "pulse")
    if kind == "drop":
        return _explicit(_log_int(rng, 64, 600), _log_int(rng, 64, 600), 1, rng.randint(1, 3), "fp64", riemann,
                         rng.choice(["outflow", "slip"]), "drop", 2)
    if kind == "semi2":
        return _semi(_log_int(rng, 64, 384), _log_int(rng, 64, 256), 1, rng.choice(["gs", "jacobi", "pcg"]),
                     rng.choice(["periodic", "slip", "outflow"]), 1e-6, rng.random() < 0.7)
    if kind == "semi3":
        n = [_log_int(rng, 48, 200) for _ in range(3)]
        return _semi(*n, rng.choice(["jacobi", "jacobi", "pcg"]), rng.choice(["periodic", "slip", "outflow"]), 1e-6,
                     rng.random() < 0.7)
    if kind == "adjoint":
        steps = rng.randint(4, 12)
        return _adjoint(_log_int(rng, 48, 256), _log_int(rng, 48, 256), steps, rng.randint(2, steps),
                        rng.choice(["fp64", "fp64", "mixed"]), rng.choice(["periodic", "outflow"]))
    return _ensemble(_log_int(rng, 30, 400), 200, _log_int(rng, 800, 4096), rng.randint(10, 40),
                     rng.choice(["mixed", "fp64"]))


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _dim(case):
    return 3 if case.get("nz", 1) > 1 else 2 if case.get("ny", 1) > 1 else 1


def _lengths(case):
    """Box [0, L] per axis, cubic cells (dx = 1 / nx)."""
    n = (case["nx"], case.get("ny", 1), case.get("nz", 1))
    return n, tuple(v / n[0] for v in n)


def _config(case):
    k = case["kind"]
    if k == "ensemble":
        return abi.config_defaults(dim=1, nGhost=3, RKOrder=3, reconOrder=abi.WENO5, riemannSolver=abi.HLLC, cfl=0.5,
                                   nPhases=2, phaseGamma=PH_GAMMA, phasePInf=PH_PINF, alphaMin=ALPHA_MIN,
                                   precision=PRECISION[case["precision"]])
    if k == "semi":
        return abi.config_defaults(dim=_dim(case), nGhost=3, RKOrder=1, reconOrder=abi.WENO5, riemannSolver=abi.HLLC,
                                   semiImplicit=1, useIGR=int(case["igr"]), siCfl=0.8, siMaxDt=1e-2,
                                   pressureTol=case["tol"], maxPressureIters=400, alphaCoeff=10.0, IGRIters=5,
                                   IGRWarmStartIters=50)
    if k == "adjoint":
        return abi.config_defaults(dim=2, nGhost=3, RKOrder=3, reconOrder=abi.WENO5, riemannSolver=abi.HLLC, cfl=0.6,
                                   maxDt=1.0)
    cfg = abi.config_defaults(dim=_dim(case), nGhost=3, RKOrder=3, reconOrder=abi.WENO5,
                              riemannSolver=RIEMANN[case["riemann"]], cfl=0.5, precision=PRECISION[case["precision"]],
                              mu=case["mu"])
    if case["phases"]:
        cfg.nPhases, cfg.alphaMin = 2, ALPHA_MIN
        for q in range(2):
            cfg.phaseGamma[q], cfg.phasePInf[q] = PH_GAMMA[q], PH_PINF[q]
    return cfg


def _waves(gen, x, y, z, lengths, modes=4):
    """Sum of a few smooth random modes, about unit amplitude, periodic on the box."""
    r = torch.rand((modes, 4), generator=gen, dtype=F64)
    k = torch.randint(1, 4, (modes, 3), generator=gen)
    out = torch.zeros(torch.broadcast_shapes(x.shape, y.shape, z.shape), dtype=F64, device=x.device)
    for m in range(modes):
        a = 2.0 * math.pi
        arg = (a * int(k[m, 0])) * x / lengths[0]
        if y.numel() > 1:
            arg = arg + (a * int(k[m, 1])) * y / lengths[1]
        if z.numel() > 1:
            arg = arg + (a * int(k[m, 2])) * z / lengths[2]
        out = out + (2.0 * float(r[m, 0]) - 1.0) * torch.sin(arg + a * float(r[m, 1]))
    return out / math.sqrt(modes)


def _initial(case, seed):
    """Interior primitive fields on the GPU: rho, u[dim], p, alpha[phases], sigma; each (nz, ny, nx)."""
    gen = torch.Generator().manual_seed(int(seed) * 1009 + 17)
    n, L = _lengths(case)
    dim = _dim(case)
    x, y, z = ((torch.arange(n[d], dtype=F64, device="cuda") + 0.5) * (L[d] / n[d]) for d in range(3))
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    shape = (n[2], n[1], n[0])
    full = lambda v: torch.as_tensor(v, dtype=F64, device="cuda").expand(shape).clone()
    wave = lambda: _waves(gen, x, y, z, L)
    r = torch.rand(16, generator=gen, dtype=F64).tolist()
    jitter = lambda q, a=0.1: 1.0 + a * (2.0 * r[q] - 1.0)
    flow = case.get("flow", "low_mach" if case["kind"] == "semi" else "vortex")
    alpha = []
    two = lambda at, a, b: torch.where(at, full(a), full(b))
    if flow == "tube":        # Sod states, a little uneven
        left = x < 0.5 + 0.02 * (r[0] - 0.5)
        rho = two(left, 1.0 * jitter(1), 0.125 * jitter(2)) * (1.0 + 0.01 * wave())
        p = two(left, 1.0 * jitter(3), 0.1 * jitter(4))
        vel = [full(0.0)]
    elif flow == "riemann":   # four-quadrant Riemann problem, split at 0.8
        rx, ry = x < 0.8 * L[0], y < 0.8 * L[1]
        pick = lambda a, b, c, d: torch.where(ry, torch.where(rx, c, d), torch.where(rx, b, a))
        t = lambda v, q: torch.tensor(v * jitter(q, 0.03), dtype=F64, device="cuda")
        rho = pick(t(1.5, 0), t(0.5323, 1), t(0.138, 2), t(0.5323, 3)) * (1.0 + 0.01 * wave())
        p = pick(t(1.5, 4), t(0.3, 5), t(0.029, 6), t(0.3, 7))
        vel = [pick(t(0.0, 8), t(1.206, 9), t(1.206, 10), t(0.0, 11)) + 0.01 * wave(),
               pick(t(0.0, 8), t(0.0, 9), t(1.206, 10), t(1.206, 11)) + 0.01 * wave()]
    elif flow == "drop":      # shocked air left, a water drop at rest in the middle
        rr = torch.sqrt((x - (0.5 + 0.05 * (r[0] - 0.5)) * L[0]) ** 2 + (y - 0.5 * L[1]) ** 2)
        prof = 0.5 * (1.0 - torch.tanh((rr - 0.18 * min(L[0], L[1])) / (2.0 / n[0])))
        aw = torch.clamp(prof, ALPHA_MIN, 1.0 - ALPHA_MIN)
        alpha = [aw, 1.0 - aw]
        shock = (x < 0.2).expand(shape)
        p = two(shock, 2.35e5 * jitter(1), 1.0e5 * jitter(2))
        air = two(shock, 2.18 * jitter(3), 1.2 * jitter(4))
        rho = [alpha[0] * 1000.0, alpha[1] * air]
        vel = [two(shock, 225.0 * jitter(5), 0.0) * alpha[1], 1.0 * wave()]
    elif flow == "low_mach":  # low-Mach acoustic pulse
        r2 = (x - (0.4 + 0.2 * r[0]) * L[0]) ** 2
        if dim >= 2:
            r2 = r2 + (y - 0.5 * L[1]) ** 2
        if dim >= 3:
            r2 = r2 + (z - 0.5 * L[2]) ** 2
        p = 1.0 + 1e-3 * jitter(1, 0.3) * torch.exp(-r2 / 0.01)
        rho = full(1.0) * (1.0 + 0.02 * wave())
        vel = [v + 1e-3 * wave() for v in (0.1, 0.05, 0.02)[:dim]]
    elif flow == "vortex":    # isentropic vortex in a free stream (1, 1), R about a tenth of the box
        dx, dy = 10.0 * (x / L[0] - 0.4 - 0.2 * r[0]), 10.0 * (y / L[1] - 0.4 - 0.2 * r[1])
        f = torch.exp(0.5 * (1.0 - dx * dx - dy * dy))
        beta = 5.0 * jitter(2, 0.2)
        T = 1.0 - (GAMMA - 1.0) * beta * beta / (8.0 * GAMMA * math.pi ** 2) * f * f
        rho, p = T ** (1.0 / (GAMMA - 1.0)), T ** (GAMMA / (GAMMA - 1.0))
        vel = [1.0 - beta / (2.0 * math.pi) * dy * f, 1.0 + beta / (2.0 * math.pi) * dx * f]
    else:                     # smooth subsonic waves with a pressure pulse
        r2 = (x - 0.5 * L[0]) ** 2 + ((y - 0.5 * L[1]) ** 2 if dim >= 2 else 0.0) + ((z - 0.5 * L[2]) ** 2 if dim >= 3 else 0.0)
        rho = 1.0 + 0.2 * wave()
        p = 1.0 + 0.5 * jitter(0, 0.3) * torch.exp(-r2 / 0.02) + 0.05 * wave()
        vel = [0.3 * wave() for _ in range(dim)]
    sigma = None
    if case["kind"] == "semi":
        sigma = 1e-5 * (1.0 + 0.5 * wave()) if case["igr"] else full(0.0)
    part = [q.expand(shape).contiguous() for q in rho] if alpha else []
    return {"rho": part[0] + part[1] if alpha else rho.expand(shape).contiguous(),
            "vel": [v.expand(shape).contiguous() for v in vel], "p": p.expand(shape).contiguous(),
            "alpha": [a.expand(shape).contiguous() for a in alpha], "alphaRho": part, "sigma": sigma}


def _conservative(s):
    """Momenta and total energy of the initial primitive state."""
    mom = [s["rho"] * v for v in s["vel"]]
    ke = 0.5 * s["rho"] * sum(v * v for v in s["vel"])
    if s["alpha"]:
        e = sum(a * (s["p"] + g * pi) / (g - 1.0) for a, g, pi in zip(s["alpha"], PH_GAMMA, PH_PINF))
    else:
        e = s["p"] / (GAMMA - 1.0)
    return mom, e + ke


def _field_map(s):
    """Initial state as SIFV_F_* -> interior tensor."""
    mom, energy = _conservative(s)
    f = {abi.F_RHO: s["rho"], abi.F_RHOE: energy, abi.F_PRES: s["p"]}
    for d, (m, v) in enumerate(zip(mom, s["vel"])):
        f[MOM[d]], f[VEL[d]] = m, v
    for q in range(len(s["alpha"])):
        f[abi.F_ALPHARHO(q)], f[abi.F_ALPHA(q)] = s["alphaRho"][q], s["alpha"][q]
    if s["sigma"] is not None:
        f[abi.F_SIGMA] = s["sigma"]
    return f


class _DeviceArray:
    """A field of the context as torch sees it (no copy); a tensor made of it keeps the context alive."""

    def __init__(self, ctx, ptr, shape):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (ptr, False), "version": 2}


def _name(fid):
    names = {abi.F_RHO: "rho", abi.F_RHOU: "rhoU", abi.F_RHOV: "rhoV", abi.F_RHOW: "rhoW", abi.F_RHOE: "rhoE",
             abi.F_VELU: "velU", abi.F_VELV: "velV", abi.F_VELW: "velW", abi.F_PRES: "pres", abi.F_SIGMA: "sigma"}
    return names.get(fid) or ("alphaRho%d" % (fid - 16) if fid < 32 else "alpha%d" % (fid - 32))


def _tubes(case, seed):
    """Water-air tubes: cells log-uniform in [lo, hi], interface, pressure and air density varied."""
    rng = np.random.default_rng(int(seed) + 5)
    k = case["tubes"]
    # the sizes are the case's own: another seed gives other states in the same tubes
    sizes = np.random.default_rng(case["tubes"] * 7919 + case["hi"])
    n = np.exp(sizes.uniform(np.log(case["lo"]), np.log(case["hi"]), k)).astype(int)
    return n, rng.uniform(0.4, 0.6, k), rng.uniform(1e7, 1e9, k), rng.uniform(0.5, 5.0, k)


def _tube_state(n, xi, p_left, rho_air):
    """Interior fields of one tube (numpy)."""
    xc = (np.arange(n) + 0.5) / n
    left = xc < xi
    aw = np.where(left, 1.0 - ALPHA_MIN, ALPHA_MIN)
    aa = 1.0 - aw
    rho = np.where(left, 1000.0, rho_air)
    p = np.where(left, p_left, 1.0e5)
    e = aw * (p + PH_GAMMA[0] * PH_PINF[0]) / (PH_GAMMA[0] - 1.0) + aa * p / (PH_GAMMA[1] - 1.0)
    return {abi.F_ALPHARHO(0): aw * rho, abi.F_ALPHARHO(1): aa * rho, abi.F_ALPHA(0): aw, abi.F_ALPHA(1): aa,
            abi.F_RHO: aw * rho + aa * rho, abi.F_RHOU: np.zeros(n), abi.F_RHOE: e, abi.F_VELU: np.zeros(n),
            abi.F_PRES: p}


ENS_FIELDS = (abi.F_RHO, abi.F_RHOU, abi.F_RHOE, abi.F_VELU, abi.F_PRES, abi.F_ALPHARHO(0), abi.F_ALPHARHO(1),
              abi.F_ALPHA(0), abi.F_ALPHA(1))


class _State:
    pass


def _check(be, st, h, ensemble=False):
    if st < 0:
        msg = be.fn["ensemble_last_error" if ensemble else "last_error"](h)
        raise abi.AbiError(st, msg.decode() if msg else "")


def prepare(case, seed):
    be = abi.Backend(_lib.load(), "sifv_", "cuda")
    s = _State()
    s.case, s.be = case, be
    if case["kind"] == "ensemble":
        n, xi, pl, ra = _tubes(case, seed)
        s.ens = be.create_ensemble(_config(case), [int(v) for v in n], [0.0] * len(n), [1.0] * len(n))
        packed = {f: np.zeros(s.ens.ncells) for f in ENS_FIELDS}
        s.off, s.n = s.ens.offsets, n
        for k in range(len(n)):
            st = _tube_state(int(n[k]), xi[k], pl[k], ra[k])
            at = slice(int(s.off[k]) + 3, int(s.off[k]) + 3 + int(n[k]))
            for f in ENS_FIELDS:
                packed[f][at] = st[f]
        s.init = {f: torch.from_numpy(a).cuda() for f, a in packed.items()}
        s.out = {f: torch.empty_like(a) for f, a in s.init.items()}
        return s
    n, L = _lengths(case)
    dim = _dim(case)
    nodes = [abi.linspace_nodes(n[d], 0.0, L[d]) for d in range(dim)]
    b = BC[case["bc"]]
    s.mesh = abi.MeshSpec(*nodes, bc=[b if d < dim else abi.BC_OUTFLOW for d in (0, 0, 1, 1, 2, 2)])
    s.cfg = _config(case)
    s.ctx = be.create(s.cfg, s.mesh, 0)
    # the copies below and the library's kernels go down one stream
    s.stream = torch.cuda.Stream()
    _check(be, be.fn["set_stream"](s.ctx.h, s.stream.cuda_stream), s.ctx.h)
    if case["kind"] == "semi":
        s.ctx.set_pressure_solver(SOLVER[case["solver"]])
    inner = s.ctx.interior_slices()
    s.init, s.view = {}, {}
    for fid, a in _field_map(_initial(case, seed)).items():
        ptr = C.c_void_p()
        _check(be, be.fn["field_device_ptr"](s.ctx.h, fid, C.byref(ptr)), s.ctx.h)
        s.view[fid] = torch.as_tensor(_DeviceArray(s.ctx, ptr.value, s.ctx.shape), device="cuda")
        s.init[fid] = torch.zeros(s.ctx.shape, dtype=F64, device="cuda")
        s.init[fid][inner] = a
    s.fids = list(s.init)
    s.inner = inner
    s.dst, s.src = [s.view[f] for f in s.fids], [s.init[f] for f in s.fids]
    if case["kind"] == "adjoint":
        if case["precision"] == "mixed":
            s.ctx.adjoint_set_precision(abi.PREC_MIXED)
        s.seed = _adjoint_seed(case, seed)
        s.cons = [abi.F_RHO, abi.F_RHOU, abi.F_RHOV, abi.F_RHOE]
        s.seedFull = {f: torch.zeros(s.ctx.shape, dtype=F64, device="cuda") for f in s.cons}
        for f, a in zip(s.cons, s.seed):
            s.seedFull[f][inner] = a
        s.grad = {f: torch.empty(s.ctx.shape, dtype=F64, device="cuda") for f in s.cons}
    torch.cuda.synchronize()
    return s


def _adjoint_seed(case, seed):
    """dJ/dU(t1): smooth weights over the box."""
    gen = torch.Generator().manual_seed(int(seed) * 31 + 3)
    n, L = _lengths(case)
    x = ((torch.arange(n[0], dtype=F64, device="cuda") + 0.5) * (L[0] / n[0]))[None, None, :]
    y = ((torch.arange(n[1], dtype=F64, device="cuda") + 0.5) * (L[1] / n[1]))[None, :, None]
    z = torch.zeros((1, 1, 1), dtype=F64, device="cuda")
    return [_waves(gen, x, y, z, L) for _ in range(4)]


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def run(s):
    case, be = s.case, s.be
    if case["kind"] == "ensemble":
        h = s.ens.h
        for f in ENS_FIELDS:
            _check(be, be.fn["ensemble_set_field"](h, f, s.init[f].data_ptr(), 1), h, True)
        # every instance takes `steps` steps more than it has taken so far
        s.total = getattr(s, "total", 0) + case["steps"]
        _, steps, _ = s.ens.run(1.0, s.total)
        for f in ENS_FIELDS:
            _check(be, be.fn["ensemble_get_field"](h, f, s.out[f].data_ptr(), 1), h, True)
        return {_name(f): s.out[f] for f in ENS_FIELDS}
    ctx = s.ctx
    with torch.cuda.stream(s.stream):
        torch._foreach_copy_(s.dst, s.src)
    out = {}
    if case["kind"] == "explicit":
        out["time"], _ = ctx.advance(0, 0.0, -1.0, case["steps"])
    elif case["kind"] == "semi":
        out["dt"] = ctx.step(1, 0.0)   # step 1: the ordinary number of IGR sweeps
    else:
        out["time"], _ = ctx.adjoint_forward(0, 0.0, 1e9, case["steps"], case["every"])
        for f in s.cons:
            _check(be, be.fn["adjoint_set_seed"](ctx.h, f, s.seedFull[f].data_ptr(), 1), ctx.h)
        ctx.adjoint_backward()
        for f in s.cons:
            _check(be, be.fn["adjoint_get_gradient"](ctx.h, f, s.grad[f].data_ptr(), 1), ctx.h)
            out["grad_" + _name(f)] = s.grad[f][s.inner]
    for f in s.fids:
        out[_name(f)] = s.view[f][s.inner]
    return out


# ---------------------------------------------------------------------------------------------------------------
# work and tolerances
# ---------------------------------------------------------------------------------------------------------------
def _cells(case):
    if case["kind"] == "ensemble":
        return int(_tubes(case, 0)[0].sum())
    return case["nx"] * case.get("ny", 1) * case.get("nz", 1)


def work(case):
    """Bytes: per step the conservative state in and out once, and the initial state in and the results out; for the
    adjoint the stage states and the adjoint state once per reversed step; for the semi-implicit step its fields
    once, without the solver's own iterations.  Flops: reconstruction of both sides of every face (about 70 per
    value in WENO5), the Riemann solver (about 120) and the update, per stage."""
    n, k = _cells(case), case["kind"]
    dim = 1 if k == "ensemble" else _dim(case)
    ph = 2 if k == "ensemble" else case.get("phases", 0)
    nc = dim + 2 + 2 * ph
    state = 8.0 * n * (2 * dim + 3 + 2 * ph)
    stage = n * dim * (2 * 70.0 * (dim + 2 + ph) + 120.0 + 40.0 * ph) + 20.0 * n * nc
    if k == "semi":
        sweeps = (5 * 30.0 if case["igr"] else 0.0) + 20.0 * 20.0
        return {"bytes": 2.0 * state + 16.0 * n, "flops": stage + n * sweeps}
    steps = case["steps"]
    fwd = {"bytes": 2.0 * state + 16.0 * n * nc * steps, "flops": 3.0 * stage * steps}
    if k == "adjoint":   # recomputed forward, reverse sweep at about three times a forward stage
        return {"bytes": 2.0 * fwd["bytes"] + 24.0 * n * nc * steps, "flops": 5.0 * fwd["flops"]}
    return fwd


def tolerance(case):
    """Relative 2-norm, about four times the largest error against ``exact`` measured over 62 cases of the ranges
    (in brackets): round-off through the steps, single precision in the mixed modes, the stopping rule for PCG."""
    k = case["kind"]
    if k == "explicit":
        if case["precision"] == "mixed":
            return {"rel": 2e-6}                                    # [3.9e-7]
        return {"rel": 1e-11 if case["phases"] else 2e-13}          # [2.2e-12; 4.3e-14]
    if k == "semi":
        return {"rel": 30.0 * case["tol"] if case["solver"] == "pcg" else 1e-13}   # [7.9 tol; 2.6e-14]
    if k == "adjoint":
        return {"rel": 1e-4 if case["precision"] == "mixed" else 1e-12}            # [1.6e-5; 2.7e-13]
    return {"rel": 2e-4 if case["precision"] == "mixed" else 1e-12}                # [3.9e-5; 1.4e-13]


# ---------------------------------------------------------------------------------------------------------------
# the scheme in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------------------------
class _Grid:
    """Boundary handling and cell sizes of the exact scheme; arrays are (nz, ny, nx)."""

    def __init__(self, dim, widths, bc, lengths=None):
        self.dim, self.w, self.bc, self.lengths = dim, widths, bc, lengths

    def pad(self, q, d, g, sign=1.0):
        """q extended by g ghost layers along axis d."""
        ax = 2 - d
        n = q.shape[ax]
        if self.lengths is not None:   # rows of different lengths: zero gradient past each row's last cell
            at = torch.arange(-g, n + g, device=q.device)[None, None, :]
            at = torch.minimum(at.clamp(min=0), self.lengths[None, :, None] - 1)
            return torch.gather(q, ax, at.expand(q.shape[0], q.shape[1], -1))
        if self.bc == "periodic":
            lo, hi = q.narrow(ax, n - g, g), q.narrow(ax, 0, g)
        elif self.bc == "outflow":
            sh = list(q.shape)
            sh[ax] = g
            lo, hi = q.narrow(ax, 0, 1).expand(sh), q.narrow(ax, n - 1, 1).expand(sh)
        else:
            lo, hi = sign * q.narrow(ax, 0, g).flip(ax), sign * q.narrow(ax, n - g, g).flip(ax)
        return torch.cat([lo, q, hi], ax)

    def vel_sign(self, comp, d):
        return -1.0 if self.bc == "noslip" or (self.bc == "slip" and comp == d) else 1.0


def _smax(a, b):
    return torch.where(a < b, b, a)


def _smin(a, b):
    return torch.where(b < a, b, a)


def _weno(v, mirror):
    """WENO5 value at the high face of the middle cell of v[0..4] (mirror: at its low face)."""
    a, b, c, d, e = v[::-1] if mirror else v
    p0 = a / 3.0 - 7.0 / 6.0 * b + 11.0 / 6.0 * c
    p1 = -b / 6.0 + 5.0 / 6.0 * c + d / 3.0
    p2 = c / 3.0 + 5.0 / 6.0 * d - e / 6.0
    b0 = 13.0 / 12.0 * (a - 2.0 * b + c) ** 2 + 0.25 * (a - 4.0 * b + 3.0 * c) ** 2
    b1 = 13.0 / 12.0 * (b - 2.0 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13.0 / 12.0 * (c - 2.0 * d + e) ** 2 + 0.25 * (3.0 * c - 4.0 * d + e) ** 2
    a0, a1, a2 = 0.1 / (1e-6 + b0) ** 2, 0.6 / (1e-6 + b1) ** 2, 0.3 / (1e-6 + b2) ** 2
    return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2)


def _faces(q, d, n):
    """Left and right face values along axis d of q extended by 3 ghosts (n interior cells, n + 1 faces)."""
    ax = 2 - d
    c = [q.narrow(ax, k, n + 1) for k in range(6)]
    return _weno(c[0:5], False), _weno(c[1:6], True)


def _flux(riemann, d, L, R, acoustic):
    """Face flux (mass, momenta, energy, p u, face velocity, alpha u) of two states with keys rho, u, p, g, pi, a."""
    uL, uR = L["u"][d], R["u"][d]

    def energy(W):
        return (W["p"] + W["g"] * W["pi"]) / (W["g"] - 1.0) + 0.5 * W["rho"] * sum(v * v for v in W["u"])

    def sound(W):
        floor = torch.full_like(W["p"], 1e-14)
        return torch.sqrt(W["g"] * _smax(W["p"] + W["pi"], floor) / _smax(W["rho"], floor))

    eL, eR = energy(L), energy(R)
    cL, cR = (sound(L), sound(R)) if acoustic else (0.0, 0.0)
    dim = len(L["u"])

    def plain(W, u, e):
        f = [W["rho"] * u] + [W["rho"] * v * u for v in W["u"]] + [e * u]
        if acoustic:
            f[1 + d] = f[1 + d] + W["p"]
            f[-1] = f[-1] + W["p"] * u
        return f + [W["p"] * u, u] + [a * u for a in W["a"]]

    def cons(W, e):
        return [W["rho"]] + [W["rho"] * v for v in W["u"]] + [e, W["p"], torch.zeros_like(e)] + W["a"]

    if riemann != "hllc":
        if riemann == "rusanov":
            c = _smax(torch.abs(uL) + cL, torch.abs(uR) + cR)
        else:
            mag = lambda W: torch.sqrt(sum(v * v for v in W["u"]))
            c = _smax(mag(L), mag(R)) + (_smax(cL, cR) if acoustic else 0.0)
        return [0.5 * (a + b) - 0.5 * c * (y - x)
                for a, b, x, y in zip(plain(L, uL, eL), plain(R, uR, eR), cons(L, eL), cons(R, eR))]
    if acoustic:
        sL, sR = _smin(uL - cL, uR - cR), _smax(uL + cL, uR + cR)
        sS = (R["p"] - L["p"] + L["rho"] * uL * (sL - uL) - R["rho"] * uR * (sR - uR)) / \
            (L["rho"] * (sL - uL) - R["rho"] * (sR - uR))
    else:
        sL, sR, sS = _smin(uL, uR), _smax(uL, uR), 0.5 * (uL + uR)
    useL, useR, left = sL >= 0, sR <= 0, sS >= 0
    useR = useR & ~useL
    one = torch.ones_like(sS)

    def star(W, u, s, e, used):
        # unused sides get harmless denominators so that their derivatives stay finite
        den = torch.where(used & (s != sS), s - sS, one)
        su = torch.where(used & (s != u), s - u, one)
        r = W["rho"] * (s - u) / den
        f = [W["rho"] * u + s * (r - W["rho"])]
        for i in range(dim):
            v = W["u"][i] + (sS - u) if i == d else W["u"][i]
            m = W["rho"] * W["u"][i] * u + s * (r * v - W["rho"] * W["u"][i])
            f.append(m + W["p"] if acoustic and i == d else m)
        if acoustic:
            E = r * (e / W["rho"] + (sS - u) * (sS + W["p"] / (W["rho"] * su)))
            f.append((e + W["p"]) * u + s * (E - e))
        else:
            f.append(e * u + s * (r * (e / W["rho"] + (sS - u) * sS) - e))
        return f + [W["p"] * sS, sS] + [a * sS for a in W["a"]]

    mid = ~useL & ~useR
    fl, fr = plain(L, uL, eL), plain(R, uR, eR)
    gl, gr = star(L, uL, sL, eL, mid & left), star(R, uR, sR, eR, mid & ~left)
    return [torch.where(useL, a, torch.where(useR, b, torch.where(left, x, y))) for a, b, x, y in zip(fl, fr, gl, gr)]


def _to_prim(U, dim, ph):
    """Primitive state of the conservative one: dict of rho, m, E, ar, a."""
    tiny = torch.full_like(U["E"], 1e-14)
    rs = _smax(sum(U["ar"]) if ph else U["rho"], tiny)
    u = [m / rs for m in U["m"]]
    e = U["E"] - 0.5 * rs * sum(v * v for v in u)
    if ph:
        inv = sum(a / (g - 1.0) for a, g in zip(U["a"], PH_GAMMA))
        pi = sum(a * g * s / (g - 1.0) for a, g, s in zip(U["a"], PH_GAMMA, PH_PINF))
        return {"rho": rs, "u": u, "p": (e - pi) / inv, "a": U["a"], "ar": U["ar"]}
    return {"rho": U["rho"], "u": u, "p": _smax((GAMMA - 1.0) * e, tiny), "a": [], "ar": []}


def _viscous(G, W, mu, d):
    """Viscous stress (momentum components, work) on the faces of axis d, 2D."""
    ax, o = 2 - d, 1 - d
    oax = 2 - o
    n, m = W["u"][0].shape[ax], W["u"][0].shape[oax]
    # both axes extended (corners x then y)
    e = [G.pad(G.pad(v, 0, 1, G.vel_sign(c, 0)), 1, 1, G.vel_sign(c, 1)) for c, v in enumerate(W["u"])]
    mid = lambda q, ax_, n_: q.narrow(ax_, 1, n_)
    dn, dt_ = [], []
    face = []
    for v in e:
        c = mid(v, oax, m)
        dn.append((c.narrow(ax, 1, n + 1) - c.narrow(ax, 0, n + 1)) / G.w[d])
        t = (v.narrow(oax, 2, m) - v.narrow(oax, 0, m)) / (2.0 * G.w[o])
        dt_.append(0.5 * (t.narrow(ax, 0, n + 1) + t.narrow(ax, 1, n + 1)))
        face.append(0.5 * (c.narrow(ax, 0, n + 1) + c.narrow(ax, 1, n + 1)))
    div = dn[d] + dt_[o]
    tau = [None, None]
    tau[d] = mu * (2.0 * dn[d] - 2.0 / 3.0 * div)
    tau[o] = mu * (dn[o] + dt_[d])
    return tau + [tau[0] * face[0] + tau[1] * face[1]]


def _rhs(G, W, riemann, acoustic, mu=0.0):
    """Flux divergence of the primitive state: list mass, m[dim], E, p, a[], ar[]."""
    dim, ph = G.dim, len(W["a"])
    total = None
    for d in range(dim):
        ax = 2 - d
        n = W["rho"].shape[ax]
        ext = lambda q, sgn=1.0: G.pad(q, d, 3, sgn)
        rhoE = ext(W["rho"])
        states = [{}, {}]
        for key, q in [("rho", rhoE), ("p", ext(W["p"]))]:
            states[0][key], states[1][key] = _faces(q, d, n)
        us = [_faces(ext(v, G.vel_sign(c, d)), d, n) for c, v in enumerate(W["u"])]
        al = [_faces(ext(a), d, n) for a in W["a"]]
        for k in range(2):
            states[k]["u"] = [v[k] for v in us]
            states[k]["a"] = [v[k] for v in al]
            if ph:
                inv = sum(a / (g - 1.0) for a, g in zip(states[k]["a"], PH_GAMMA))
                spi = sum(a * g * s / (g - 1.0) for a, g, s in zip(states[k]["a"], PH_GAMMA, PH_PINF))
                states[k]["g"] = 1.0 + 1.0 / inv
                states[k]["pi"] = (states[k]["g"] - 1.0) / states[k]["g"] * spi
            else:
                states[k]["g"], states[k]["pi"] = GAMMA, 0.0
        f = _flux(riemann, d, states[0], states[1], acoustic)
        up = []
        for ar in W["ar"]:
            y = ext(ar) / rhoE
            up.append(torch.where(f[0] >= 0, y.narrow(ax, 2, n + 1), y.narrow(ax, 3, n + 1)) * f[0])
        f = f + up
        if mu > 0:
            t = _viscous(G, W, mu, d)
            for q, v in zip((1, 2, 3), t):
                f[q] = f[q] - v
        r = [(v.narrow(ax, 0, n) - v.narrow(ax, 1, n)) / G.w[d] for v in f]
        total = r if total is None else [a + b for a, b in zip(total, r)]
    div = -total[dim + 3]
    out = total[:dim + 2] + [total[dim + 2] + W["p"] * div]
    out += [r + a * div for r, a in zip(total[dim + 4:dim + 4 + ph], W["a"])]
    return out + total[dim + 4 + ph:]


def _acoustic_dt(G, W, cfl, max_dt, mu):
    """Per-cell limit's minimum; per row for rows of different lengths."""
    tiny = torch.full_like(W["p"], 1e-14)
    if W["a"]:
        s = 0.0
        for a, ar, g, pi in zip(W["a"], W["ar"], PH_GAMMA, PH_PINF):
            rk = _smax(ar, tiny) / _smax(a, tiny)
            s = s + a / (rk * _smax(g * (W["p"] + pi) / rk, tiny))
        c = torch.sqrt(1.0 / (W["rho"] * s))
    else:
        c = torch.sqrt(GAMMA * _smax(W["p"], tiny) / _smax(W["rho"], tiny))
    v = None
    for d in range(G.dim):
        t = G.w[d] / (torch.abs(W["u"][d]) + c)
        v = t if v is None else torch.minimum(v, t)
    v = cfl * v
    if mu > 0:
        w = min(G.w[:G.dim])
        v = torch.minimum(v, cfl * (w * w / (2.0 * G.dim * (mu / W["rho"]))))
    if G.lengths is not None:
        return torch.clamp(v.amin(dim=2, keepdim=True), max=max_dt)
    return torch.clamp(v.amin(), max=max_dt)


def _stack(U):
    return [U["rho"]] + U["m"] + [U["E"]] + U["a"] + U["ar"]


def _unstack(v, dim, ph):
    return {"rho": v[0], "m": list(v[1:1 + dim]), "E": v[1 + dim], "a": list(v[2 + dim:2 + dim + ph]),
            "ar": list(v[2 + dim + ph:])}


def _explicit_steps(G, U, W, riemann, cfl, max_dt, steps, mu=0.0):
    """SSP-RK3 steps with the CFL time step; returns the state, its primitives and the time."""
    dim, ph = G.dim, len(U["a"])
    time = 0.0
    for _ in range(steps):
        dt = _acoustic_dt(G, {k: [q.detach() for q in v] if isinstance(v, list) else v.detach() for k, v in W.items()},
                          cfl, max_dt, mu)
        U0 = _stack(U)
        for c1, c2, c4 in ((1.0, 0.0, 1.0), (1.0, 3.0, 4.0), (2.0, 1.0, 3.0)):
            Wp = _to_prim(U, dim, ph)
            r = _rhs(G, Wp, riemann, True, mu)
            r = r[:dim + 2] + r[dim + 3:]
            cur = _stack(U)
            if ph:
                cur[0] = Wp["rho"]
            c3 = 2.0 if c1 == 2.0 else 1.0
            new = [(c1 * a + c2 * b + c3 * dt * q) / c4 for a, b, q in zip(cur, U0, r)]
            U = _unstack(new, dim, ph)
            if ph:
                tiny = torch.full_like(U["E"], 1e-14)
                U["ar"] = [_smax(v, tiny) for v in U["ar"]]
                U["rho"] = sum(U["ar"])
                a = [v.clamp(min=ALPHA_MIN) for v in U["a"]]
                U["a"] = [v / sum(a) for v in a]
        W = _to_prim(U, dim, ph)
        if ph:
            U["rho"] = W["rho"]
        time = time + dt
    return U, W, time


def _outputs(U, W):
    out = {"rho": W["rho"], "rhoE": U["E"], "pres": W["p"]}
    for d, (m, v) in enumerate(zip(U["m"], W["u"])):
        out[_name(MOM[d])], out[_name(VEL[d])] = m, v
    for q in range(len(U["a"])):
        out["alphaRho%d" % q], out["alpha%d" % q] = U["ar"][q], U["a"][q]
    return out


def _start(case, seed):
    s = _initial(case, seed)
    mom, energy = _conservative(s)
    U = {"rho": s["rho"], "m": mom, "E": energy, "a": s["alpha"], "ar": s["alphaRho"]}
    W = {"rho": s["rho"], "u": s["vel"], "p": s["p"], "a": s["alpha"], "ar": s["alphaRho"]}
    n, L = _lengths(case)
    return _Grid(_dim(case), [L[d] / n[d] for d in range(3)], case["bc"]), U, W, s


def _neighbours(q, periodic, dim):
    """Values one cell lower and higher along each axis (zero gradient outside)."""
    out = []
    for d in range(dim):
        ax = 2 - d
        n = q.shape[ax]
        if periodic:
            out.append((q.roll(1, ax), q.roll(-1, ax)))
        else:
            out.append((torch.cat([q.narrow(ax, 0, 1), q.narrow(ax, 0, n - 1)], ax),
                        torch.cat([q.narrow(ax, 1, n - 1), q.narrow(ax, n - 1, 1)], ax)))
    return out


def _lexicographic(q, rhs, den, coef, sweeps, periodic, dim, tol=None):
    """In-place sweeps in storage order of q = (rhs + sum coef q_nb) / den, plane i + j + k = const at a time; the
    neighbours outside the box hold the values from before the sweep.  Stops after the sweep whose largest change
    is below tol."""
    shape = q.shape
    pad = [1, 1, 1, 1] + ([1, 1] if dim == 3 else [0, 0])
    ext = [s + (2 if dim == 3 or ax > 0 else 0) for ax, s in enumerate(shape)]
    ii = torch.arange(shape[2], device=q.device)[None, None, :]
    jj = torch.arange(shape[1], device=q.device)[None, :, None]
    kk = torch.arange(shape[0], device=q.device)[:, None, None]
    plane = (ii + jj + kk).expand(shape).reshape(-1)
    order = torch.argsort(plane, stable=True)
    counts = torch.bincount(plane).tolist()
    e = ((kk + (1 if dim == 3 else 0)) * ext[1] + jj + 1) * ext[2] + ii + 1
    at = e.expand(shape).reshape(-1)[order]
    step = [1, ext[2], ext[1] * ext[2]][:dim]
    st = torch.tensor([o for v in step for o in (-v, v)], device=q.device)
    R, D = rhs.reshape(-1)[order], den.reshape(-1)[order]
    K = torch.stack([c.expand(shape).reshape(-1)[order] for pair in coef for c in pair])
    cuts = np.cumsum([0] + counts)
    parts = [(at[a:b], at[a:b][None, :] + st[:, None], R[a:b], D[a:b], K[:, a:b]) for a, b in zip(cuts[:-1], cuts[1:])]
    mode = "circular" if periodic else "replicate"
    for done in range(sweeps):
        buf = torch.nn.functional.pad(q[None, None], pad, mode=mode)[0, 0].contiguous()
        flat = buf.view(-1)
        for c, nb, r, dd, k in parts:
            flat[c] = (r + (k * flat[nb]).sum(0)) / dd
        new = buf[1:-1, 1:-1, 1:-1] if dim == 3 else buf[:, 1:-1, 1:-1]
        change = (new - q).abs().amax() if tol is not None else None
        q = new.contiguous()
        if tol is not None and float(change) < tol:
            break
    return q


def _semi_step(case, seed):
    G, U, W, s = _start(case, seed)
    dim, per = G.dim, case["bc"] == "periodic"
    w = G.w
    dt = 0.8 * min(float((w[d] / W["u"][d].abs().clamp(min=1e-14)).amin()) for d in range(dim))
    dt = min(max(dt, 1e-12), 1e-2)
    W = _to_prim(U, dim, 0)
    sigma = s["sigma"]

    def central(v, c, d):
        e = G.pad(v, d, 1, G.vel_sign(c, d))
        n = v.shape[2 - d]
        return e.narrow(2 - d, 2, n), e.narrow(2 - d, 0, n)

    rho = W["rho"]
    rn = _neighbours(rho, per, dim)
    if case["igr"]:
        alpha = 10.0 * w[0] * w[0]
        g = [[(lambda h, l: (h - l) * (0.5 / w[d]))(*central(W["u"][c], c, d)) for d in range(dim)] for c in range(dim)]
        rhs = alpha * (sum(g[a][b] * g[b][a] for a in range(dim) for b in range(dim)) + sum(g[a][a] for a in range(dim)) ** 2)
        coef = [[alpha / (w[d] * w[d]) / (0.5 * (rho + r)) for r in rn[d]] for d in range(dim)]
        sigma = _lexicographic(sigma, rhs, 1.0 / rho + sum(c for pair in coef for c in pair), coef, 5, per, dim)
    r = _rhs(G, W, "hllc", False)
    rho = U["rho"] + dt * r[0]
    star = [m + dt * q for m, q in zip(U["m"], r[1:1 + dim])]
    p_adv = W["p"] + dt * r[dim + 2]
    vel = [m / rho for m in star]
    rhoc2 = rho * (GAMMA * W["p"] / rho)
    div = 0.0
    for d in range(dim):
        hi, lo = central(vel[d], d, d)
        div = div + (0.5 * (vel[d] + hi) - 0.5 * (lo + vel[d])) / w[d]
    rhs = p_adv - rhoc2 * dt * div
    rn = _neighbours(rho, per, dim)
    face = [[1.0 / (0.5 * (rho + q) * w[d] * w[d]) for q in rn[d]] for d in range(dim)]
    cf = rhoc2 * dt * dt
    den = 1.0 + cf * sum(c for pair in face for c in pair)
    p = W["p"]
    if case["solver"] == "jacobi":
        for _ in range(400):
            nb = _neighbours(p, per, dim)
            new = (rhs + cf * sum(c * q for pc, pq in zip(face, nb) for c, q in zip(pc, pq))) / den
            change = float((new - p).abs().amax())
            p = new
            if change < case["tol"]:
                break
    elif case["solver"] == "gs":
        p = _lexicographic(p, rhs, den, [[cf * c for c in pair] for pair in face], 400, per, dim, case["tol"])
    else:   # the solution itself: conjugate gradients on the symmetric form, zero-flux walls
        if not per:
            for d in range(dim):
                face[d] = [c.clone() for c in face[d]]
                face[d][0].narrow(2 - d, 0, 1).zero_()
                face[d][1].narrow(2 - d, p.shape[2 - d] - 1, 1).zero_()
        diag = 1.0 / cf + sum(c for pair in face for c in pair)
        A = lambda q: diag * q - sum(c * v for pc, pv in zip(face, _neighbours(q, per, dim)) for c, v in zip(pc, pv))
        b = rhs / cf
        res = b - A(p)
        z = res / diag
        k, rz = z, (res * z).sum()
        for _ in range(2000):
            q = A(k)
            a = rz / (k * q).sum()
            p, res = p + a * k, res - a * q
            if float(res.norm() / b.norm()) < 1e-13:
                break
            z = res / diag
            new = (res * z).sum()
            k, rz = z + (new / rz) * k, new
    total = p + sigma
    mom = [m - dt * (0.5 * (total + hi) - 0.5 * (lo + total)) / w[d]
           for d, (m, (lo, hi)) in enumerate(zip(star, _neighbours(total, per, dim)))]
    vel = [m / rho for m in mom]
    energy = p / (GAMMA - 1.0) + 0.5 * rho * sum(v * v for v in vel)
    out = _outputs({"m": mom, "E": energy, "a": [], "ar": []}, {"rho": rho, "u": vel, "p": p})
    return dict(out, dt=dt, sigma=sigma)


def _exact_ensemble(case, seed):
    n, xi, pl, ra = _tubes(case, seed)
    k, top = len(n), int(n.max())
    host = {f: np.zeros((1, k, top)) for f in ENS_FIELDS}
    for t in range(k):
        st = _tube_state(int(n[t]), xi[t], pl[t], ra[t])
        for f in ENS_FIELDS:
            host[f][0, t, :n[t]] = st[f]
            host[f][0, t, n[t]:] = st[f][-1]
    q = {f: torch.from_numpy(a).cuda() for f, a in host.items()}
    lengths = torch.from_numpy(n.astype(np.int64)).cuda()
    # past a row's end the state is its last cell's, so the fluxes there vanish
    G = _Grid(1, [(1.0 / lengths.to(F64))[None, :, None]], "outflow", lengths)
    ar, a = [q[abi.F_ALPHARHO(i)] for i in range(2)], [q[abi.F_ALPHA(i)] for i in range(2)]
    U = {"rho": q[abi.F_RHO], "m": [q[abi.F_RHOU]], "E": q[abi.F_RHOE], "a": a, "ar": ar}
    W = {"rho": q[abi.F_RHO], "u": [q[abi.F_VELU]], "p": q[abi.F_PRES], "a": a, "ar": ar}
    keep = lambda v: torch.gather(v, 2, torch.minimum(torch.arange(top, device="cuda")[None, None, :],
                                                      lengths[None, :, None] - 1).expand(1, k, top))
    for _ in range(case["steps"]):
        U, W, _ = _explicit_steps(G, U, W, "hllc", 0.5, 1e-2, 1)
        U = {m: [keep(v) for v in x] if isinstance(x, list) else keep(x) for m, x in U.items()}
        W = {m: [keep(v) for v in x] if isinstance(x, list) else keep(x) for m, x in W.items()}
    out = {}
    for name, v in _outputs(U, W).items():
        # packed tube after tube, three ghost cells of the end cells on either side
        e = G.pad(v, 0, 3)[0]
        out[name] = torch.cat([e[t, :int(n[t]) + 6] for t in range(k)])
    # the ghosts of the state's momentum, energy and fractions stay as they were set
    for name in ("rhoU", "rhoE"):
        at = 0
        for t in range(k):
            out[name][at:at + 3] = 0.0
            out[name][at + 3 + int(n[t]):at + 6 + int(n[t])] = 0.0
            at += int(n[t]) + 6
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "ensemble":
        return _exact_ensemble(case, seed)
    if k == "semi":
        return _semi_step(case, seed)
    G, U, W, _ = _start(case, seed)
    if k == "explicit":
        U, W, t = _explicit_steps(G, U, W, case["riemann"], 0.5, 1e-2, case["steps"], case["mu"])
        return dict(_outputs(U, W), time=float(t))
    leaf = [q.clone().requires_grad_(True) for q in _stack(U)]
    U1, W1, t = _explicit_steps(G, _unstack(leaf, 2, 0), W, "hllc", 0.6, 1.0, case["steps"])
    J = sum((a * b).sum() for a, b in zip(_stack(U1), _adjoint_seed(case, seed)))
    J.backward()
    out = _outputs({m: [v.detach() for v in x] if isinstance(x, list) else x.detach() for m, x in U1.items()},
                   {m: [v.detach() for v in x] if isinstance(x, list) else x.detach() for m, x in W1.items()})
    for fid, q in zip((abi.F_RHO, abi.F_RHOU, abi.F_RHOV, abi.F_RHOE), leaf):
        out["grad_" + _name(fid)] = q.grad
    return dict(out, time=float(t))
