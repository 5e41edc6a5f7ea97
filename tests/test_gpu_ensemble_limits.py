"""A non-finite wave speed ends an ensemble run with SIFV_ERR_NAN in either arithmetic: an infinite velocity or pressure
makes the time step 0, and the instances beside it must not carry the run on.  A cell whose limit is not a number is
passed over, as the reference's minimum passes over it."""
import numpy as np
import pytest

import cases
from semiimplicitfv_b200 import abi
from test_gpu_ensemble import _ensemble

pytestmark = pytest.mark.gpu


def _tubes(phases):
    return [cases.water_air(n, p_left=2e5) if phases else cases.sod(n) for n in (20, 60, 130)]


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
@pytest.mark.parametrize("phases,field", [(0, abi.F_VELU), (0, abi.F_PRES), (2, abi.F_VELU)])
@pytest.mark.parametrize("where", [0, 57, -1])
def test_infinite_wave_speed_is_an_error(precision, phases, field, where):
    inst = _tubes(phases)
    ens = _ensemble(inst, precision)
    g = inst[1][0].nGhost
    fields = [c[2][field].copy() for c in inst]
    fields[1][0, 0, g:-g][where] = np.inf
    ens.set_field(field, ens.pack(fields))
    with pytest.raises(abi.AbiError) as e:
        ens.run(1e-4)
    assert e.value.status == abi.ERR_NAN
    assert "instance 1" in str(e.value)


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
def test_nan_limit_is_passed_over(precision):
    inst = _tubes(0)
    ref, ens = _ensemble(inst, precision), _ensemble(inst, precision)
    g = inst[1][0].nGhost
    fields = [c[2][abi.F_VELU].copy() for c in inst]
    fields[1][0, 0, g:-g][5] = np.nan   # at rest: not the cell that sets the step
    ens.set_field(abi.F_VELU, ens.pack(fields))
    t1, s1, _ = ref.run(1e-2)
    t2, s2, _ = ens.run(1e-2)   # the stored velocity only enters the first limit
    assert np.array_equal(t1, t2) and np.array_equal(s1, s2)
    assert np.array_equal(ref.get_field(abi.F_RHOE), ens.get_field(abi.F_RHOE))
