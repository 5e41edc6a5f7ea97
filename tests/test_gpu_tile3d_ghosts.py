"""The 3D FP64-fast and mixed steps write interior cells of the conservative state only: the ghost layers of the momenta
and the energy keep what the caller put there, whatever the RK order."""
import numpy as np
import pytest

import backends
from semiimplicitfv_b200 import abi
from test_gpu_tile3d import O, P, S, _noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("rk", [1, 2, 3])
def test_conservative_ghost_layers_are_left_alone(precision, rk):
    case = _noise((9, 10, 11), (O, O, P, P, S, S), 3, rk)
    case[0].precision = precision
    ctx = backends.make(backends.cuda(), case)
    ghost = np.ones(ctx.shape, dtype=bool)
    ctx.interior(ghost)[...] = False
    before = {}
    for q, f in enumerate((abi.F_RHOU, abi.F_RHOV, abi.F_RHOW, abi.F_RHOE)):
        a = ctx.get_field(f)
        a[ghost] = 5.0 + q + np.arange(np.count_nonzero(ghost))
        ctx.set_field(f, a)
        before[f] = a
    ctx.advance(0, 0.0, 0.0, 2)
    for f, a in before.items():
        b = ctx.get_field(f)
        assert np.array_equal(a[ghost], b[ghost]), f
        assert not np.array_equal(a[~ghost], b[~ghost])
