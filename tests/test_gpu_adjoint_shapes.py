"""The reverse kernel's blocks follow each direction's own count: elongated meshes keep the dot-product identity and cost
no more per cell than their short lines waste."""
import numpy as np
import pytest

import backends
from semiimplicitfv_b200 import abi
from adjoint_autograd import cons_fids
from test_gpu_adjoint import _dot_test
from test_gpu_stage import O, P, S, Y, _box
from test_gpu_tile3d import _noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(300, 3), (3, 300)])
def test_dot_product_on_elongated_meshes(nx, ny):
    case = _box(nx, ny, (O, S, P, P), seed=nx)
    case[0].constDt = 2e-5
    _dot_test(case, 6e-5, every=2)


@pytest.mark.parametrize("n", [(120, 3, 5), (3, 120, 4), (4, 3, 120)])
def test_dot_product_on_elongated_meshes_3d(n):
    case = _noise(n, (P, P, O, S, S, Y), 1)
    case[0].constDt = 2e-5
    _dot_test(case, 6e-5, every=2)


def _backward_ms(nx, ny):
    case = _box(nx, ny, (P, P, P, P), seed=1)
    ctx = backends.make(backends.cuda(), case)
    best = 1e30
    for _ in range(3):
        ctx.adjoint_forward(0, 0.0, 1.0, 4, 2)
        for f in cons_fids(2):
            ctx.adjoint_set_seed(f, np.ones(ctx.shape))
        best = min(best, ctx.adjoint_backward())
    return best


@pytest.mark.parametrize("nx,ny", [(8000, 4), (4, 8000)])
def test_elongated_meshes_cost_their_waste(nx, ny):
    """4 of the 58 positions that a block owns along a line: 15 times the blocks at most, where blocks of empty
    directions made it several hundred."""
    assert _backward_ms(nx, ny) <= 15.0 * _backward_ms(179, 179)
