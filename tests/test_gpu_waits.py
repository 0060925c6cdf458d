"""Waits of the fused step kernel that run out: the barrier is told to expect arrivals that never
come, with a limit of a millisecond.  No result of such a launch passes for a value."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _integrator(form, precision):
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.vern7 import GpuVern7
    dtype = "c128" if precision == "double" else "c64"
    if form == "half":
        from qutip_gb300.superop import device_term_groups
        s = S.ising_chain(6)
        op = DeviceOperator.from_device_groups(device_term_groups(s.terms), dtype, fmt="dict")
        op.hermitian_dim = lambda: s.dim             # below the size from which it pays
    else:
        s = S.jaynes_cummings(7)
        op = DeviceOperator(s.terms, dtype=dtype, fmt=form)
    ig = GpuVern7(op, precision=precision)
    ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    assert ig._half() is (form == "half")
    return s, ig


def _no_arrivals(ig):
    ig._wait_mcycles = 1
    ig._barrier_base.value += 1 << 20


FORMS = [("csr", "double"), ("dict", "mixed"), ("half", "double"), ("half", "mixed")]


@pytest.mark.parametrize("form,precision", FORMS)
def test_a_trial_step_that_gives_up(form, precision):
    from qutip_gb300 import _lib
    from qutip_gb300.vern7 import IntegratorError
    s, ig = _integrator(form, precision)
    _no_arrivals(ig)
    with pytest.raises(IntegratorError, match="gave up"):
        ig.integrate(1.0)
    assert _lib.load().qg_device_fault() != 0        # read and cleared
    assert not ig.successful()
    ig.integrate(1.0)                                # no step to go on from
    with pytest.raises(IntegratorError, match="Not initialized"):
        ig.check()
    ig._wait_mcycles = 0
    again = _integrator(form, precision)[1]
    for g in (ig, again):
        g.set_initial_value(torch.from_numpy(s.state0), 0.0)
        g.integrate(1.0)
        g.check()
    assert torch.equal(ig.get_state(), again.get_state())


@pytest.mark.parametrize("form,precision", FORMS)
def test_a_dense_output_that_gives_up(form, precision):
    """One output, and the outputs of a run: what is read is NaN, and the next look or call
    raises."""
    from qutip_gb300 import _lib
    from qutip_gb300.solver import ExpectOps
    from qutip_gb300.vern7 import IntegratorError
    for whole_run in (False, True):
        s, ig = _integrator(form, precision)
        ig.integrate(100.0, step=True)               # one step, no dense output yet
        ig.check()
        t = 0.5 * (ig.t_prev + ig.t_front)
        _no_arrivals(ig)
        if whole_run:
            ex = ExpectOps(s.e_ops)
            out = torch.zeros(1, 2 * (ex.n + 1), dtype=torch.float64, device="cuda")
            assert ig.run_dm(np.array([t]), ex.dev, s.dim, out)
            assert bool(torch.isnan(out.cpu()[0, -2:]).any())          # the trace
        else:
            ig.integrate(t)
            state = ig.get_state().cpu()
            assert bool(torch.isnan(torch.view_as_real(state)).all())
        assert not ig.successful()
        with pytest.raises(IntegratorError, match="gave up"):
            ig.check()
        assert _lib.load().qg_device_fault() != 0    # read and cleared
        ig.integrate(t)
        with pytest.raises(IntegratorError, match="Not initialized"):
            ig.check()
        ig._wait_mcycles = 0
        ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
        ig.integrate(0.01)
        ig.check()
        assert bool(torch.isfinite(torch.view_as_real(ig.get_state())).all())


def test_a_new_state_after_a_give_up():
    """Set while the last state's dense output is known to have given up: a fresh start."""
    s, ig = _integrator("csr", "double")
    ig.integrate(100.0, step=True)
    _no_arrivals(ig)
    ig.integrate(0.5 * (ig.t_prev + ig.t_front))
    torch.cuda.synchronize()
    assert not ig.successful()
    ig._wait_mcycles = 0
    again = _integrator("csr", "double")[1]
    for g in (ig, again):
        g.set_initial_value(torch.from_numpy(s.state0), 0.0)
        g.integrate(1.0)
        g.check()
    assert torch.equal(ig.get_state(), again.get_state())
    from qutip_gb300 import _lib
    assert _lib.load().qg_device_fault() != 0        # read and cleared


@pytest.mark.parametrize("in_library", [False, True])
def test_a_give_up_seen_by_the_next_call(in_library):
    """A dense output that gave up ends the next call, before its trial step or, where it
    was still running then, after it."""
    from qutip_gb300.vern7 import IntegratorError
    _, ig = _integrator("csr", "double")
    ig.integrate(100.0, step=True)
    ig._words[1] = -1.0                              # as the launch leaves it
    if in_library:
        ig._check_waits = lambda: None
    with pytest.raises(IntegratorError, match="gave up"):
        ig.integrate(100.0, step=True)
