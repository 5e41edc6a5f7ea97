"""Reference-ordered explicit steps on either side of the line between the fused stage kernel and the separate ones
(meshes of few columns, long 1D meshes): the oracle's bits on both, through sifv_step and the device-resident loop, and
no time for columns that are not there."""
import pytest

import backends
import cases
from semiimplicitfv_b200 import abi
from test_gpu_stage import N, O, P, S, Y, _box, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(4, 1000), (4, 9000), (9, 3000), (9, 8000), (40, 6100), (7000, 3), (60000, 3)])
@pytest.mark.parametrize("mu", [0.0, 1e-4])
def test_columns(nx, ny, mu):
    _compare(_box(nx, ny, (O, S, P, P), seed=nx, mu=mu), 2)


@pytest.mark.parametrize("bcs", [(P, P, N, Y), (Y, O, S, S)])
@pytest.mark.parametrize("rk,riemann", [(2, abi.LF), (3, abi.RUSANOV)])
def test_columns_faces(bcs, rk, riemann):
    _compare(_box(5, 8000, bcs, seed=rk, riemann=riemann, rk=rk), 2)


@pytest.mark.parametrize("n", [600000, 600001])
def test_long_1d(n):
    _compare(cases.sod(n), 1)


@pytest.mark.parametrize("n", [60000, 60001])
def test_long_1d_two_phases(n):
    _compare(cases.water_air(n, p_left=2e5), 2)


def _step_ms(nx, ny):
    ctx = backends.make(backends.cuda(), _box(nx, ny, (P, P, P, P), seed=1))
    best = 1e30
    for _ in range(3):
        ctx.advance(0, 0.0, -1.0, 10)
        best = min(best, ctx.last_step_stats()[0])
    return best


def test_few_columns_do_not_pay_for_a_tile():
    """As many cells in 4 columns: 1.6 times the time, where 28 idle lanes of 32 made it 6 times."""
    assert _step_ms(4, 50000) <= 3.5 * _step_ms(500, 400)
