"""Long integrations return to the interpreter every so often: an interrupt ends them, and a call
that was taken up again any number of times does what one call does."""
import _thread
import threading
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _op(kind):
    from qutip_gb300.dense import DenseLindbladOperator
    from qutip_gb300.lindblad import LindbladOperator
    from qutip_gb300.operator import DeviceOperator
    if kind == "csr":
        s = S.jaynes_cummings(7)
        return s, DeviceOperator(s.terms), "double"
    s = S.ising_chain(5)
    if kind == "matrix":
        return s, LindbladOperator.from_hamiltonian(s.h_terms, s.c_ops, dtype="c64"), "mixed"
    return s, DenseLindbladOperator.from_hamiltonian(s.h_terms, s.c_ops[:3]), "mixed"


@pytest.mark.parametrize("whole_run", [False, True])
def test_an_interrupt_ends_a_long_solve(whole_run):
    """Some 300,000 steps (over ten seconds), interrupted after a third of a second."""
    from qutip_gb300.solver import solve_system
    from qutip_gb300.vern7 import GpuVern7
    s, op, _ = _op("csr")
    opt = {"max_step": 0.01, "nsteps": 10**9}
    ig = GpuVern7(op, **opt)
    ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    ig.integrate(0.1)
    timer = threading.Timer(0.3, _thread.interrupt_main)
    t0 = time.perf_counter()
    timer.start()
    with pytest.raises(KeyboardInterrupt):
        if whole_run:
            solve_system(s, np.linspace(0, 3000, 301), opt, op=op)
        else:
            ig.integrate(3000.0)
    assert time.perf_counter() - t0 < 3.0
    timer.cancel()


@pytest.mark.parametrize("opts", [{}, {"nsteps": 3}, {"interpolate": False}], ids=str)
@pytest.mark.parametrize("kind", ["csr", "matrix", "dense"])
def test_calls_taken_up_again(kind, opts):
    """Back in the interpreter after every step: the scalars, counts and state of one call,
    the limit of steps counted across the pieces."""
    from qutip_gb300.vern7 import GpuVern7
    s, op, precision = _op(kind)
    whole, pieces = (GpuVern7(op, precision=precision, **opts) for _ in range(2))
    whole._slice, pieces._slice = 0.0, 1e-12
    calls = []
    take = pieces._take
    pieces._take = lambda c: calls.append(c.paused) or take(c)
    for ig in (whole, pieces):
        ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    for t, step in [(0.01, False), (3.0, False), (3.1, True), (6.0, True), (9.0, False), (9.0, False)]:
        for ig in (whole, pieces):
            ig.integrate(t, step=step)
        assert whole.status == pieces.status and whole.stats == pieces.stats, t
        for name in ("t", "t_prev", "t_front", "dt_safe", "dt_int", "_out"):
            assert getattr(whole, name) == getattr(pieces, name), name
        assert torch.equal(whole.get_state(), pieces.get_state())
    assert 1 in calls
    assert (whole.status < 0) is ("nsteps" in opts)


@pytest.mark.parametrize("opts", [{}, {"nsteps": 3}], ids=str)
@pytest.mark.parametrize("kind", ["csr", "matrix", "dense"])
def test_runs_taken_up_again(kind, opts):
    """Outputs inside a step, between steps and repeated, bit for bit."""
    from qutip_gb300.solver import ExpectOps
    from qutip_gb300.vern7 import GpuVern7
    s, op, precision = _op(kind)
    ex = ExpectOps(s.e_ops)
    tl = np.concatenate([[0.0, 0.0], np.linspace(0.001, 0.002, 40), [0.5, 0.5, 0.4999, 4.0, 4.0]])
    whole, pieces = (GpuVern7(op, precision=precision, **opts) for _ in range(2))
    whole._slice, pieces._slice = 0.0, 1e-12
    calls = []
    take = pieces._take
    pieces._take = lambda c: calls.append(c.paused) or take(c)
    out = torch.zeros((2, len(tl), 2 * (ex.n + 1)), dtype=torch.float64, device="cuda")
    for ig, o in ((whole, out[0]), (pieces, out[1])):
        ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
        assert ig.run_dm(tl, ex.dev, s.dim, o)
    assert whole.status == pieces.status and whole.stats == pieces.stats
    assert (whole.t, whole.t_prev, whole.t_front) == (pieces.t, pieces.t_prev, pieces.t_front)
    assert torch.equal(out[0], out[1])
    assert {1, 2} <= set(calls)
    assert (whole.status < 0) is ("nsteps" in opts)
