"""3D FP64-fast and mixed steps on the meshes that the tiles of 32 x 8 columns fit badly: they run as dimension sweeps, the
others as one kernel per stage, and long meshes of few columns take more segments.  Both against the reference-ordered
mode on noise, to the bounds of test_gpu_tile3d.py."""
import numpy as np
import pytest

import backends
import cases
from semiimplicitfv_b200 import abi
from test_gpu_fast import CONS
from test_gpu_tile3d import BOUND, N, O, P, S, Y, _compare, _noise

pytestmark = pytest.mark.gpu
SWEEPS = [(300, 9, 260), (9, 9, 12000), (12000, 9, 9)]
TILES = [(64, 9, 70), (4, 5, 1500), (300, 8, 40)]


def _families(n, precision):
    case = _noise(n, (P,) * 6, 1)
    case[0].precision = precision
    return set(backends.make(backends.cuda(), case).profile_step(0, 0.0))


@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("n", SWEEPS + TILES)
def test_route(n, precision):
    families = _families(n, precision)
    assert ("sweep_z" in families) == (n in SWEEPS) and ("tile3d" in families) == (n in TILES)


@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("n", SWEEPS + TILES)
@pytest.mark.parametrize("bcs", [(P,) * 6, (Y, O, S, N, S, O)])
def test_against_the_reference_order(n, precision, bcs):
    _compare(precision, n, bcs, steps=2)


@pytest.mark.parametrize("precision", sorted(BOUND))
@pytest.mark.parametrize("rk,riemann", [(1, abi.LF), (2, abi.RUSANOV)])
def test_orders_and_solvers(precision, rk, riemann):
    _compare(precision, (300, 9, 260), (O, O, P, P, S, S), rk, riemann, steps=2)


@pytest.mark.parametrize("precision", sorted(BOUND))
def test_time_step_of_the_resident_loop(precision):
    """The sweeps leave no limits for the next step: its dt is the reduction over the new state."""
    runs = []
    for resident in (True, False):
        case = _noise((300, 9, 260), (O, S, P, P, N, O), 2)
        case[0].precision = precision
        ctx = backends.make(backends.cuda(), case)
        if resident:
            t, n = ctx.advance(0, 0.0, -1.0, 3)
        else:
            t, n, _ = cases.run_steps(ctx, 3)
        runs.append((t, n, [ctx.get_field(f) for f in CONS]))
    assert runs[0][:2] == runs[1][:2]
    assert all(np.array_equal(a, b) for a, b in zip(runs[0][2], runs[1][2]))


def test_long_columns_fill_the_device():
    """4000 cells per column in 16 columns: three times the time of a cube of that many cells, where 64 segments at most
    made it nine times."""
    def ms(n):
        case = _noise(n, (P,) * 6, 1)
        case[0].precision = abi.PREC_FP64_FAST
        ctx = backends.make(backends.cuda(), case)
        best = 1e30
        for _ in range(3):
            ctx.advance(0, 0.0, -1.0, 5)
            best = min(best, ctx.last_step_stats()[0])
        return best
    assert ms((4, 4, 4000)) <= 5.0 * ms((40, 40, 40))
