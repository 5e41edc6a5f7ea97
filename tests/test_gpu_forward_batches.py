"""Forward runs of the adjoint and the tangent queue several steps per look of the host, and the steps queued past the
end time do nothing: not to the state, not to the tangent, and not to the calls that follow."""
import numpy as np
import pytest
import torch

import backends
import cases
from adjoint_autograd import cons_fids
from semiimplicitfv_b200 import abi

pytestmark = pytest.mark.gpu


def _stretching(slope, n=64, dim=1):
    """u = slope (x - 1/2): the gas thins out and slows down, dt grows."""
    cfg, mesh, fields = cases.sod(n) if dim == 1 else cases.riemann2d(n)
    cfg.maxDt = 1.0
    sl = cases._interior_slices(cfg)
    x = 0.5 * (mesh.x[:-1] + mesh.x[1:])
    one = np.ones(fields[abi.F_RHO][sl].shape)
    u = slope * (x - 0.5) * one
    args = (one, u, 0.0 * one if dim == 2 else None, None, one, 1.4)
    return cfg, mesh, cases._single_phase_fields(cfg, fields[abi.F_RHO].shape, *args)


def _const_dt(case, dt):
    case[0].constDt = dt
    return case


CASES = {
    # name: (case, end time, sign of the dt's change over the run)
    "constant": (lambda: _const_dt(cases.sod(64), 1e-3), 5e-3, 0),
    "constant_exact": (lambda: _const_dt(_stretching(0.5, 8), 2.0 ** -6), 2.0 ** -3, 0),
    "growing": (lambda: _stretching(3.0), 0.12, 1),
    "shrinking": (lambda: cases.sod(64), 0.04, -1),
    "growing_2d": (lambda: _stretching(3.0, 24, 2), 0.12, 1),
}


def _run(case, t_end, v, schedule):
    ctx = backends.make(backends.cuda(), case)
    for f, a in v.items():
        ctx.tangent_set_direction(f, a)
    t, n = ctx.tangent_forward(0, 0.0, t_end, 0, schedule)
    return t, n, {f: (ctx.get_field(f), ctx.tangent_get(f)) for f in v}


@pytest.mark.parametrize("rk", [1, 3])
@pytest.mark.parametrize("name", sorted(CASES))
def test_tangent_to_an_end_time_takes_the_recorded_steps(name, rk):
    make, t_end, change = CASES[name]
    case = make()
    case[0].RKOrder = rk
    ctx = backends.make(backends.cuda(), case)
    ctx.adjoint_forward(0, 0.0, t_end, 0, 1)   # one step per look at the host
    sched = ctx.adjoint_schedule()
    assert len(sched) >= 5 and np.sign(sched[-2] - sched[0]) == change
    rng = np.random.default_rng(len(sched))
    v = {f: rng.standard_normal(ctx.shape) for f in cons_fids(case[0].dim)}
    t1, n1, free = _run(case, t_end, v, None)
    t2, n2, fixed = _run(case, t_end, v, sched)
    assert (t1, n1) == (t2, n2) and n1 == len(sched)
    for f in v:
        for a, b in zip(free[f], fixed[f]):
            assert np.array_equal(a, b), f


@pytest.mark.parametrize("between", ["overwritten", "advanced"])
@pytest.mark.parametrize("name", ["constant", "growing", "growing_2d"])
def test_backward_restores_the_end_state_whatever_came_between(name, between):
    make, t_end, _ = CASES[name]
    case = make()
    dim = case[0].dim
    ctx = backends.make(backends.cuda(), case)
    t, n = ctx.adjoint_forward(0, 0.0, t_end, 0, 64)
    fids = cons_fids(dim) + [abi.F_VELU, abi.F_PRES] + ([abi.F_VELV] if dim == 2 else [])
    end = {f: ctx.get_field(f) for f in fids}
    if between == "overwritten":
        for f in fids:
            ctx.set_field(f, np.full(ctx.shape, 7.0))
    else:   # to an end time, with steps to spare
        assert ctx.advance(n, t, t + 2.5 * t / n, 6)[1] < 6
    for f in cons_fids(dim):
        ctx.adjoint_set_seed(f, np.ones(ctx.shape))
    ctx.adjoint_backward()
    for f in fids:
        assert np.array_equal(ctx.get_field(f), end[f]), f


def test_failed_forward_keeps_no_checkpoints():
    """A forward run that fails gives the memory of its checkpoints, and of the earlier run's, back."""
    ctx = backends.make(backends.cuda(), cases.vortex2d(1000))
    ctx.adjoint_forward(0, 0.0, 1.0, 8, 4)   # three checkpoints
    free = torch.cuda.mem_get_info()[0]
    u = ctx.get_field(abi.F_VELU)
    u[0, 500, 500] = np.inf   # the first time step is 0
    ctx.set_field(abi.F_VELU, u)
    with pytest.raises(abi.AbiError) as e:
        ctx.adjoint_forward(0, 0.0, 1.0, 8, 4)
    assert e.value.status == abi.ERR_NAN
    assert torch.cuda.mem_get_info()[0] - free >= 3 * 4 * 8 * ctx.ncells
