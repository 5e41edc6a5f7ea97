"""The reverse kernel of the discrete adjoint at the edges of its tiles (58 positions of a grid line per block, the
three ghost layers of either end among them; four lines per block): the dot-product identity <lam, T v> = <T^T lam, v>
with the tangent, to round-off (the bound of test_gpu_adjoint.py), over sizes, faces and Riemann solvers, and the
upwind reconstruction, whose transpose has no weights.
"""
import pytest

import cases
from semiimplicitfv_b200 import abi
from test_gpu_adjoint import _dot_test
from test_gpu_stage import N, O, P, S, Y, _box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 4), (5, 3), (52, 5), (53, 6), (58, 3), (111, 7), (6, 53)])
@pytest.mark.parametrize("bcs", [(P, P, P, P), (O, S, N, Y)])
def test_dot_product_at_tile_edges(nx, ny, bcs):
    case = _box(nx, ny, bcs, seed=nx)
    case[0].constDt = 2e-4
    _dot_test(case, 6e-4, every=2)


@pytest.mark.parametrize("riemann", [abi.RUSANOV, abi.LF])
@pytest.mark.parametrize("recon", [abi.WENO5, abi.UPWIND5])
def test_dot_product_2d_solvers(riemann, recon):
    case = _box(54, 9, (S, O, P, P), riemann=riemann, recon=recon, rk=2)
    case[0].constDt = 2e-4
    _dot_test(case, 6e-4, every=3)


@pytest.mark.parametrize("n", [52, 53, 60])
def test_dot_product_1d_edges(n):
    _dot_test(cases.sod(n), 0.03, every=2)
