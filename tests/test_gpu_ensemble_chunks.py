"""FP64 ensembles whose blocks work through chunks of blockDim - 6 cells, at the edges of the chunks: every instance bit
for bit the oracle's run of it alone, over RK orders, faces, Riemann solvers, one, two and three phases, with short
instances among them whose warps idle."""
import numpy as np
import pytest

import cases
from semiimplicitfv_b200 import abi
from test_gpu_ensemble import _check_bitwise, _ensemble, _tube

pytestmark = pytest.mark.gpu
# per block size: sizes around its chunks whose strips take more rounds
SIZES = {64: [57, 58, 59, 116, 117, 3, 175], 256: [249, 250, 251, 27, 500, 501], 512: [505, 506, 507, 4, 33, 1012]}


@pytest.mark.parametrize("bc", [abi.BC_OUTFLOW, abi.BC_PERIODIC, abi.BC_SLIPWALL])
@pytest.mark.parametrize("rk,riemann,recon", [(1, abi.HLLC, abi.WENO5), (2, abi.LF, abi.UPWIND5), (3, abi.RUSANOV, abi.WENO5)])
@pytest.mark.parametrize("block", sorted(SIZES))
def test_chunk_edges_match_the_oracle(block, rk, riemann, recon, bc):
    cfg = abi.config_defaults(dim=1, nGhost=3, RKOrder=rk, reconOrder=recon, riemannSolver=riemann, cfl=0.5, maxDt=1.0)
    inst = [_tube(cfg, n, 0.0, 1.0, (1.0 + 0.1 * k, 0.05 * (k % 3), 1.0 + 0.2 * k), (0.125, -0.02 * (k % 2), 0.1), bc)
            for k, n in enumerate(SIZES[block])]
    ens = _ensemble(inst)
    t, s, _ = ens.run(1.0, 6, block)
    _check_bitwise(ens, inst, 1.0, t, s, 6)


def _third_phase(case):
    """A third phase of 2 % of the volume everywhere, as light as air."""
    cfg, mesh, f = case
    cfg.nPhases = 3
    cfg.phaseGamma[2], cfg.phasePInf[2] = 1.6, 0.0
    ng = cfg.nGhost
    sl = (slice(0, 1), slice(0, 1), slice(ng, -ng))
    share, p = 0.02, f[abi.F_PRES][sl]
    for q in (0, 1):
        f[abi.F_ALPHA(q)][sl] *= 1.0 - share
        f[abi.F_ALPHARHO(q)][sl] *= 1.0 - share
    f[abi.F_ALPHA(2)], f[abi.F_ALPHARHO(2)] = np.zeros_like(f[abi.F_RHO]), np.zeros_like(f[abi.F_RHO])
    f[abi.F_ALPHA(2)][sl], f[abi.F_ALPHARHO(2)][sl] = share, share * 1.1
    f[abi.F_RHO][sl] = sum(f[abi.F_ALPHARHO(q)][sl] for q in range(3))
    f[abi.F_RHOE][sl] = sum(f[abi.F_ALPHA(q)][sl] * (p + cfg.phaseGamma[q] * cfg.phasePInf[q]) / (cfg.phaseGamma[q] - 1.0)
                            for q in range(3))
    return case


@pytest.mark.parametrize("phases", [2, 3])
@pytest.mark.parametrize("block", sorted(SIZES))
def test_chunk_edges_with_phases_match_the_oracle(block, phases):
    inst = [cases.water_air(n, p_left=2e5 + 1e3 * n) for n in SIZES[block]]
    if phases == 3:
        inst = [_third_phase(c) for c in inst]
    ens = _ensemble(inst)
    t, s, _ = ens.run(1.0, 6, block)
    _check_bitwise(ens, inst, 1.0, t, s, 6)
