"""The PCG + multigrid solver at the edges of its launch plan: one level only (at most 256 cells), every level in the
single-block tail (at most 4096 cells), one and two levels above it, odd and thin meshes.  The stopping rule
|A p - b| <= tol |b| is checked on the assembled system (factor 2: the recurrence's residual against the true one), and
a solve queued in batches as long as the one before it stops where a fresh one does, on the same bits."""
import numpy as np
import pytest

import backends
from semiimplicitfv_b200 import abi
from test_gpu_pcg_mg import _inputs, hypre_system

pytestmark = pytest.mark.gpu


def _setup(n, periodic):
    dim = len(n)
    cfg = abi.config_defaults(dim=dim, nGhost=3, reconOrder=abi.WENO5, semiImplicit=1)
    nodes = [abi.linspace_nodes(k, 0.0, 1.0 + 0.2 * a) for a, k in enumerate(n)]
    face = abi.BC_PERIODIC if periodic else abi.BC_SLIPWALL
    mesh = abi.MeshSpec(*nodes, bc=[face if a < dim else abi.BC_OUTFLOW for a in (0, 0, 1, 1, 2, 2)])
    return cfg, mesh, nodes


def _context(cfg, mesh):
    ctx = backends.cuda().create(cfg, mesh)
    ctx.set_pressure_solver(abi.PRESSURE_PCG_MG)
    return ctx


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("n", [(4,), (300,), (5000,), (3, 3), (16, 16), (17, 16), (64, 64), (65, 64), (1500, 3),
                               (131, 77), (16, 16, 16), (17, 16, 16), (3, 4, 70), (33, 29, 23)])
def test_pcg_mg_launch_plan(n, periodic):
    cfg, mesh, nodes = _setup(n, periodic)
    per = tuple(periodic and a < len(n) for a in range(3))
    ctx = _context(cfg, mesh)
    rho, rhoc2, rhs, p0 = _inputs(ctx, per, sum(n))
    dt, tol = 8.0 / max(n), 1e-9
    p, iters, st = ctx.pressure_solve(rho, rhoc2, rhs, p0, dt, tol, 500)
    assert st == abi.OK and 0 < iters < 500
    nodes = nodes + [np.array([0.0, 1.0])] * (3 - len(n))
    n3 = tuple(n) + (1,) * (3 - len(n))
    ng = tuple(ctx.ng if a < len(n) else 0 for a in range(3))
    widths = [hypre_system.ext_widths(nodes[a], ng[a]) for a in range(3)]
    A, b = hypre_system.assemble(len(n), n3, ng, widths, per, rho.ravel(), rhoc2.ravel(), rhs.ravel(), dt)
    x = ctx.interior(p).ravel()
    assert np.linalg.norm(A @ x - b) <= 2.0 * tol * np.linalg.norm(b)
    # a shorter solve queued in a batch of the last one's length
    p1, it1, _ = ctx.pressure_solve(rho, rhoc2, rhs, p0, dt, 1e-2, 500)
    p2, it2, _ = _context(cfg, mesh).pressure_solve(rho, rhoc2, rhs, p0, dt, 1e-2, 500)
    assert it1 == it2 <= iters and np.array_equal(p1, p2)
    # the iteration limit
    _, it3, _ = ctx.pressure_solve(rho, rhoc2, rhs, p0, dt, tol, 1)
    assert it3 == 1
