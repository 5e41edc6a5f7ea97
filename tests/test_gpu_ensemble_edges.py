"""Ensembles at the edges of the kernel's strips (26 cells per warp): FP64 instances bit for bit against the oracle run
alone, on sizes one cell either side of a strip and smaller than its halo, every RK order, periodic and outflow ends,
two phases, and blocks with fewer and more warps than strips."""
import pytest

import cases
from semiimplicitfv_b200 import abi
from test_gpu_ensemble import _check_bitwise, _ensemble, _tube

pytestmark = pytest.mark.gpu

EDGES = [3, 4, 25, 26, 27, 51, 52, 53, 79]


@pytest.mark.parametrize("bc", [abi.BC_OUTFLOW, abi.BC_PERIODIC, abi.BC_SLIPWALL])
@pytest.mark.parametrize("rk,block", [(1, 32), (2, 64), (3, 512)])
def test_strip_edges_match_the_oracle(bc, rk, block):
    cfg = abi.config_defaults(dim=1, nGhost=3, RKOrder=rk, reconOrder=abi.WENO5, cfl=0.5, maxDt=1.0)
    # on [0, 1], whose last node is the upper end exactly (the ensemble is given the ends, the oracle the nodes)
    inst = [_tube(cfg, n, 0.0, 1.0, (1.0 + 0.1 * k, 0.05 * (k % 3), 1.0 + 0.2 * k),
                  (0.125, -0.02 * (k % 2), 0.1), bc) for k, n in enumerate(EDGES)]
    ens = _ensemble(inst)
    t, s, _ = ens.run(0.02, 0, block)
    _check_bitwise(ens, inst, 0.02, t, s)


@pytest.mark.parametrize("block", [32, 128])
def test_two_phase_strip_edges_match_the_oracle(block):
    inst = [cases.water_air(n, p_left=2e5 + 1e4 * n) for n in (25, 26, 27, 53)]
    ens = _ensemble(inst)
    t, s, _ = ens.run(1e-4, 0, block)
    _check_bitwise(ens, inst, 1e-4, t, s)
