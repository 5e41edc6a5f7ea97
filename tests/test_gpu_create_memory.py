"""What a context takes of the device: its arrays and little more, at sizes where several share an allocation and where
one does not fit twice into a shared one, and no more than that where the device is nearly full."""
import pytest
import torch

import backends
from semiimplicitfv_b200 import abi

pytestmark = pytest.mark.gpu
MB = 1 << 20
ARRAYS = 18   # 2D, explicit, single phase: 10 of the state and the solver, two scratch states of 4


def _create(n):
    nodes = abi.linspace_nodes(n, 0.0, 1.0)
    return backends.cuda().create(abi.config_defaults(dim=2, nGhost=3), abi.MeshSpec(nodes, nodes))


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("n", [500, 1018, 1500, 2100, 3000])
def test_context_memory(n):
    _create(32).close()   # loads the kernels
    array = 8 * (n + 6) ** 2
    before = _free()
    ctx = _create(n)
    used = before - _free()
    ctx.close()
    # a last chunk of up to seven spare arrays and 64 MB, and the driver's granularity
    assert used <= ARRAYS * array + min(7 * array, 64 * MB) + 16 * MB, used / MB
    assert used <= 1.5 * ARRAYS * array + 16 * MB, used / MB


def test_context_on_a_nearly_full_device():
    n = 1018
    array = 8 * (n + 6) ** 2   # eight to a chunk, so that 18 take three: 24
    _create(n).close()
    torch.cuda.empty_cache()
    spare = ARRAYS * array + 12 * MB
    filler = torch.empty(_free() - spare, dtype=torch.uint8, device="cuda")
    try:
        assert ARRAYS * array < _free() < 3 * 8 * array
        ctx = _create(n)
        ctx.close()
    finally:
        del filler
        torch.cuda.empty_cache()
