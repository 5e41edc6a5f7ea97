"""3D Jacobi solves on the meshes where single iterations beat the paired ones (many tiles of few planes; coefficients
per cell beyond the L2 cache): iteration count and iterate are the oracle's bit for bit, as on the paired side."""
import numpy as np
import pytest

from test_gpu_jacobi_pair import O, P, S, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("bcs", [(P,) * 6, (O, S, P, P, S, O)])
@pytest.mark.parametrize("n", [(5100, 3, 4), (5, 2600, 3), (40, 41, 2000), (106, 106, 106)])
def test_either_side_of_the_rule(n, bcs, uniform):
    (cg, co), rng = _pair(n, bcs, uniform)
    m = cg.ncells
    args = (1.0 + 0.1 * rng.random(m), 1.4 + 0.2 * rng.random(m), rng.random(m), rng.random(m))
    for max_iter, tol in ((1, 1e-14), (5, 1e-14), (300, 1e-3)):
        pg, ig, sg = cg.pressure_solve(*args, 5e-3, tol, max_iter)
        po, io, so = co.pressure_solve(*args, 5e-3, tol, max_iter)
        assert (ig, sg) == (io, so), (max_iter, tol)
        assert np.array_equal(cg.interior(pg), co.interior(po)), (max_iter, tol)
