"""The default block size of an ensemble has no more warps than its longest instance has strips of 26 cells, whatever the
arithmetic and the number of phases: the run is the one of that block size, and short instances do not pay for idle
warps."""
import numpy as np
import pytest

import cases
from semiimplicitfv_b200 import abi
from test_gpu_ensemble import _ensemble

pytestmark = pytest.mark.gpu


def _tubes(sizes, phases):
    return [cases.water_air(n, p_left=2e5) if phases else cases.sod(n) for n in sizes]


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("phases", [0, 2])
@pytest.mark.parametrize("sizes", [[3, 20], [26, 27, 60], [500, 30], [4000, 40, 41]])
def test_default_run_is_the_run_of_any_block_size(precision, phases, sizes):
    runs = []
    for block in (0, 32, 256):
        ens = _ensemble(_tubes(sizes, phases), precision)
        t, s, _ = ens.run(1e9, 5, block)
        assert np.all(s == 5)
        runs.append([t] + [ens.get_field(f) for f in (abi.F_RHO, abi.F_RHOU, abi.F_RHOE, abi.F_PRES)])
    for a in runs[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(a, runs[0]))


def _ms(count, n, phases, precision):
    ens = _ensemble(_tubes([n] * count, phases), precision)
    return min(ens.run(1e9, 10 * (k + 1))[2] for k in range(4))


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("phases", [0, 2])
def test_short_tubes_do_not_pay_for_idle_warps(precision, phases):
    """Sixteen times the tubes of a sixteenth of the cells: no more than three times the time, as much work in shorter
    chains; a fixed block size would leave 15 of its 16 warps idle."""
    assert _ms(4096, 26, phases, precision) <= 3.0 * _ms(256, 416, phases, precision)
