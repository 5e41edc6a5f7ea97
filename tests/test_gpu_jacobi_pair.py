"""Two Jacobi iterations per launch (3D) at the edges of its blocks (32 x 16 columns, segments of planes): meshes of one
cell either side of a block and smaller, every pair of scalar faces, per-face and per-cell coefficients, iteration
limits and tolerances that end inside a pair.  Iteration count and iterate are the oracle's bit for bit."""
import numpy as np
import pytest

import backends
import cases
from semiimplicitfv_b200 import abi

pytestmark = pytest.mark.gpu
P, O, S = abi.BC_PERIODIC, abi.BC_OUTFLOW, abi.BC_SLIPWALL


def _pair(n, bcs, uniform):
    cfg, mesh, fields = cases.acoustic_box(*n)
    rng = np.random.default_rng(sum(n))
    nodes = []
    for k in n:
        w = np.full(k, 1.0 / 64.0) if uniform else (0.5 + rng.random(k)) / 64.0
        nodes.append(np.concatenate([[0.0], np.cumsum(w)]))
    mesh.x, mesh.y, mesh.z = nodes
    mesh.bc = list(bcs)
    return [backends.make(b, (cfg, mesh, fields)) for b in (backends.cuda(), backends.oracle())], rng


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("bcs", [(P,) * 6, (O, S, P, P, S, O), (P, P, O, O, P, P)])
@pytest.mark.parametrize("n", [(3, 3, 3), (31, 15, 5), (32, 16, 33), (33, 17, 4), (70, 34, 9), (5, 50, 40)])
def test_jacobi_pair_edges(n, bcs, uniform):
    (cg, co), rng = _pair(n, bcs, uniform)
    m = cg.ncells
    args = (1.0 + 0.1 * rng.random(m), 1.4 + 0.2 * rng.random(m), rng.random(m), rng.random(m))
    for max_iter, tol in ((1, 1e-14), (2, 1e-14), (7, 1e-14), (12, 1e-14), (300, 1e-5), (300, 3e-6), (300, 1e-6), (300, 3e-7)):
        pg, ig, sg = cg.pressure_solve(*args, 5e-3, tol, max_iter)
        po, io, so = co.pressure_solve(*args, 5e-3, tol, max_iter)
        assert (ig, sg) == (io, so), (max_iter, tol)
        assert np.array_equal(cg.interior(pg), co.interior(po)), (max_iter, tol)


def test_jacobi_pair_plain_division():
    """Values outside the range of the corrected quotient (zeros, tiny and huge ones) divide plainly."""
    (cg, co), rng = _pair((36, 18, 7), (P, P, O, S, P, P), True)
    m = cg.ncells
    rhs, p0 = rng.random(m), rng.random(m)
    rhs[rng.choice(m, 400)] = 0.0
    rhs[rng.choice(m, 400)] = 1e-300
    p0[rng.choice(m, 400)] = 1e160
    p0[rng.choice(m, 400)] = -0.0
    rhoc2 = 1.4 + 0.2 * rng.random(m)
    rhoc2[rng.choice(m, 400)] = 1e140
    rhoc2[rng.choice(m, 400)] = 0.0
    args = (1.0 + 0.1 * rng.random(m), rhoc2, rhs, p0)
    for max_iter in (2, 5):
        pg, ig, _ = cg.pressure_solve(*args, 5e-3, 1e-14, max_iter)
        po, io, _ = co.pressure_solve(*args, 5e-3, 1e-14, max_iter)
        assert ig == io and np.array_equal(cg.interior(pg), co.interior(po))
