"""The fused stage kernel of the reference-ordered explicit step (1D / 2D, WENO5 / UPWIND5, at most two phases):
bit for bit against the C oracle at the sizes where its tiles can go wrong (one cell either side of a tile edge, the
smallest meshes), with viscosity, body force and every kind of face, and with operands outside the range of the
branch-free quotients (zeros of both signs, tiny and huge values).  The oracle evaluates the same expressions, so the
tolerance is zero.
"""
import numpy as np
import pytest

import backends
import cases
from semiimplicitfv_b200 import abi
from semiimplicitfv_b200.abi import F_PRES, F_RHO, F_RHOE, F_RHOU, F_RHOV, F_VELU, F_VELV

pytestmark = pytest.mark.gpu


def _compare(case, steps):
    cg, co = backends.make(backends.cuda(), case), backends.make(backends.oracle(), case)
    _, _, dg = cases.run_steps(cg, steps)
    _, _, do = cases.run_steps(co, steps)
    assert dg == do
    ca = backends.make(backends.cuda(), case)     # the device-resident loop folds the dt reduction into the stage
    if not any(case[0].bfA):
        t, n = ca.advance(0, 0.0, -1.0, steps)
        time = 0.0
        for dt in do:
            time += dt
        assert n == steps and t == time
    else:
        ca = None
    fids = list(case[2])
    for f in fids:
        a, b = cg.get_field(f), co.get_field(f)
        assert np.array_equal(a, b, equal_nan=True), f
        if ca is not None:
            assert np.array_equal(ca.get_field(f), b, equal_nan=True), f


def _box(nx, ny, bcs, seed=0, riemann=abi.HLLC, recon=abi.WENO5, rk=3, mu=0.0):
    case = cases.acoustic_box(nx, ny, semi=False, igr=False, rk=rk)
    cfg, mesh, fields = case
    cfg.riemannSolver, cfg.reconOrder, cfg.mu = riemann, recon, mu
    mesh.bc = list(bcs) + [abi.BC_OUTFLOW] * (6 - len(bcs))
    rng = np.random.default_rng(seed)
    sl = (slice(0, 1), slice(3, -3), slice(3, -3))
    shape = fields[F_RHO][sl].shape
    rho = 1.0 + 0.3 * rng.random(shape)
    u, v = rng.standard_normal(shape), rng.standard_normal(shape)
    p = 1.0 + rng.random(shape)
    fields[F_RHO][sl], fields[F_VELU][sl], fields[F_VELV][sl], fields[F_PRES][sl] = rho, u, v, p
    fields[F_RHOU][sl], fields[F_RHOV][sl] = rho * u, rho * v
    fields[F_RHOE][sl] = p / 0.4 + 0.5 * rho * (u * u + v * v)
    return case


O, P, S, N, Y = abi.BC_OUTFLOW, abi.BC_PERIODIC, abi.BC_SLIPWALL, abi.BC_NOSLIPWALL, abi.BC_SYMMETRY


@pytest.mark.parametrize("nx,ny", [(3, 3), (31, 7), (32, 8), (33, 9), (34, 16), (65, 17), (3, 40), (70, 3)])
@pytest.mark.parametrize("bcs", [(P, P, P, P), (O, S, N, Y)])
def test_tile_edges_2d(nx, ny, bcs):
    _compare(_box(nx, ny, bcs, seed=nx + ny), 3)


@pytest.mark.parametrize("riemann", [abi.RUSANOV, abi.LF])
@pytest.mark.parametrize("recon,rk", [(abi.WENO5, 2), (abi.UPWIND5, 3)])
def test_solvers_2d(riemann, recon, rk):
    _compare(_box(41, 19, (O, O, P, P), riemann=riemann, recon=recon, rk=rk), 3)


@pytest.mark.parametrize("n", [3, 29, 30, 31, 61, 200])
@pytest.mark.parametrize("riemann", [abi.HLLC, abi.LF])
def test_tile_edges_1d(n, riemann):
    _compare(cases.sod(n, riemann=riemann), 5)
    _compare(cases.water_air(n, riemann=riemann), 4)


@pytest.mark.parametrize("bcs", [(P, P, P, P), (N, N, S, O)])
def test_viscous_and_body_force(bcs):
    _compare(_box(35, 18, bcs, mu=0.02), 3)
    case = _box(35, 18, bcs, mu=0.02)
    case[0].bfA[0], case[0].bfB[1], case[0].bfC[1] = 0.3, 0.2, 1.5
    _compare(case, 3)


@pytest.mark.parametrize("n", [9, 33])
def test_two_phases_2d(n):
    _compare(cases.droplet(n, sigma=0.0), 3)
    case = cases.droplet(n, sigma=0.0, bc=abi.BC_SLIPWALL)
    case[0].nPhaseMu = 2
    case[0].phaseMu[0], case[0].phaseMu[1] = 1.0e-3, 1.8e-5
    case[0].mu = 1.0e-4
    _compare(case, 3)


@pytest.mark.parametrize("scale,eps", [(1e60, 1e-6), (1e-160, 1e-6), (1.0, 1e-120), (1.0, 1e110)])
def test_operands_outside_the_quotients_range(scale, eps):
    """Fields far from one (indicators above 2^256, products below 2^-450) and an eps outside [1e-100, 1e100] take
    the plain divisions; zeros of both signs and single huge cells among ordinary ones mix both in one warp."""
    case = _box(40, 12, (O, O, P, P))
    cfg, mesh, f = case
    cfg.wenoEps, cfg.constDt = eps, 1e-4
    sl = (slice(0, 1), slice(3, -3), slice(3, -3))
    rng = np.random.default_rng(5)
    pick = rng.random(f[F_RHO][sl].shape) < 0.2
    vel = np.where(pick, f[F_VELU][sl] * scale, f[F_VELU][sl])
    if scale > 1:        # keep the sound speeds finite: scale pressure and energy, not the velocity
        vel = f[F_VELU][sl]
        f[F_PRES][sl] = np.where(pick, f[F_PRES][sl] * scale, f[F_PRES][sl])
    vel[..., ::7] = 0.0
    vel[..., 3::7] = -0.0
    rho, p = f[F_RHO][sl], f[F_PRES][sl]
    f[F_VELU][sl], f[F_RHOU][sl] = vel, rho * vel
    f[F_RHOE][sl] = p / 0.4 + 0.5 * rho * (vel * vel + f[F_VELV][sl] ** 2)
    _compare(case, 2)
