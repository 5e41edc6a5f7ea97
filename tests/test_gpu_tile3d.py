"""The 3D fused stage (FP64-fast and mixed precision) at the edges of its plan: columns of 32 x 8 cells, segments of one
plane and more along z, meshes smaller than the stencil's reach, every kind of face, RK order and Riemann solver,
against the reference-ordered mode on noise.  FP64-fast to the relative 1e-10 of test_gpu_fast.py; mixed precision to
the error of a flux formed in FP32: a face value is within 2^-24 x (sum of |coefficients| < 4) x (weights, about 8) of
its exact one, and nine stages add dt / dx (< 0.3) x two faces x three directions of it, 16 x 2^-19 in all."""
import numpy as np
import pytest

import backends
import cases
from semiimplicitfv_b200 import abi
from test_gpu_fast import CONS, _max_rel

pytestmark = pytest.mark.gpu
O, P, S, N, Y = abi.BC_OUTFLOW, abi.BC_PERIODIC, abi.BC_SLIPWALL, abi.BC_NOSLIPWALL, abi.BC_SYMMETRY
BOUND = {abi.PREC_FP64_FAST: 1e-10, abi.PREC_MIXED: 16 * 2.0 ** -19}


def _noise(n, bcs, seed, rk=3, riemann=abi.HLLC):
    case = cases.acoustic_box(*n, semi=False, igr=False, rk=rk)
    cfg, mesh, fields = case
    cfg.riemannSolver = riemann
    mesh.bc = list(bcs)
    rng = np.random.default_rng(seed)
    sl = (slice(3, -3),) * 3
    shape = fields[abi.F_RHO][sl].shape
    rho, p = 1.0 + 0.3 * rng.random(shape), 1.0 + rng.random(shape)
    vel = [0.5 * rng.standard_normal(shape) for _ in range(3)]
    fields[abi.F_RHO][sl], fields[abi.F_PRES][sl] = rho, p
    for u, fv, fm in zip(vel, (abi.F_VELU, abi.F_VELV, abi.F_VELW), (abi.F_RHOU, abi.F_RHOV, abi.F_RHOW)):
        fields[fv][sl], fields[fm][sl] = u, rho * u
    fields[abi.F_RHOE][sl] = p / 0.4 + 0.5 * rho * sum(u * u for u in vel)
    return case


def _compare(precision, n, bcs, rk=3, riemann=abi.HLLC, steps=3):
    runs = []
    for prec in (precision, abi.PREC_FP64):
        case = _noise(n, bcs, sum(n), rk, riemann)
        case[0].precision = prec
        ctx = backends.make(backends.cuda(), case)
        cases.run_steps(ctx, steps)
        runs.append(ctx)
    assert all(np.all(np.isfinite(runs[0].get_field(f))) for f in CONS)
    assert _max_rel(runs[0], runs[1], runs[1].cfg) <= BOUND[precision]


@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("n", [(3, 3, 3), (4, 70, 5), (31, 7, 9), (32, 8, 16), (33, 9, 3), (65, 17, 40)])
@pytest.mark.parametrize("bcs", [(P,) * 6, (O, S, N, Y, S, O), (Y, O, P, P, N, S)])
def test_tile_edges(precision, n, bcs):
    _compare(precision, n, bcs)


@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("riemann", [abi.HLLC, abi.RUSANOV, abi.LF])
@pytest.mark.parametrize("rk", [1, 2])
def test_orders_and_solvers(precision, riemann, rk):
    _compare(precision, (35, 10, 12), (O, O, P, P, S, S), rk, riemann)
