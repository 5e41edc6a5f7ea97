"""1D fast and mixed modes on either side of the size where the fused stage kernel of the reference-ordered mode hands
over to the sweeps (240000 cells): below it the states are that mode's bit for bit, above it FP64-fast stays within the
relative 1e-10 of test_gpu_fast.py and mixed within the error of fluxes formed in FP32 (2^-24 x 4 x 8 per face value,
two faces and dt / dx < 1 over six stages)."""
import numpy as np
import pytest

import backends
import cases
from semiimplicitfv_b200 import abi
from test_gpu_fast import CONS, _max_rel

pytestmark = pytest.mark.gpu
LINE = 240000


@pytest.mark.parametrize("precision", [abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("rk", [1, 2, 3])
@pytest.mark.parametrize("n", [3, 31, 1000, LINE, LINE + 1])
def test_fast_1d_route(precision, rk, n):
    runs = []
    for prec in (precision, abi.PREC_FP64):
        case = cases.sod(n)
        case[0].precision, case[0].RKOrder = prec, rk
        ctx = backends.make(backends.cuda(), case)
        cases.run_steps(ctx, 2)
        runs.append(ctx)
    if rk > 1 and n <= LINE:
        assert all(np.array_equal(runs[0].get_field(f), runs[1].get_field(f)) for f in CONS)
    else:
        bound = 1e-10 if precision == abi.PREC_FP64_FAST else 6 * 2 * 2.0 ** -19
        assert _max_rel(runs[0], runs[1], runs[1].cfg) <= bound
