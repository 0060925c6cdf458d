"""The library's integration loop (``qg_vern7_integrate``, ``qg_vern7_run_dm``) against the
same loop in Python on the same kernels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _op(kind, precision):
    from qutip_gb300.dense import DenseLindbladOperator
    from qutip_gb300.lindblad import LindbladOperator
    from qutip_gb300.operator import DeviceOperator
    dtype = "c128" if precision == "double" else "c64"
    if kind == "csr":
        s = S.jaynes_cummings(7)
        return s, DeviceOperator(s.terms, dtype=dtype)
    if kind == "csr16":                               # a launch shape the fused step has not
        s = S.jaynes_cummings(7)
        op = DeviceOperator(s.terms, dtype=dtype)
        op.set_launch(("direct", 0, 16))
        return s, op
    s = S.ising_chain(5)
    if kind == "dict":
        return s, DeviceOperator(s.terms, dtype=dtype, fmt="dict")
    if kind == "matrix":
        return s, LindbladOperator.from_hamiltonian(s.h_terms, s.c_ops, dtype=dtype)
    return s, DenseLindbladOperator.from_hamiltonian(s.h_terms, s.c_ops[:3])


OPTIONS = [{}, {"interpolate": False}, {"max_step": 0.05}, {"first_step": 2.0}, {"nsteps": 3},
           {"min_step": 0.3, "first_step": 0.9}]
KINDS = [("csr", "double"), ("csr16", "double"), ("dict", "mixed"), ("dict", "single"),
         ("matrix", "mixed"), ("dense", "mixed")]


@pytest.mark.parametrize("opts", OPTIONS, ids=[str(o) for o in OPTIONS])
@pytest.mark.parametrize("kind,precision", KINDS)
def test_integrate_follows_the_python_loop(kind, precision, opts):
    """Outputs inside one step, past several, twice the same, before the step, one step at a
    time, and the failures: the same scalars, counts, status and states after each call (the
    same IEEE operations on both sides; states to rounding)."""
    from qutip_gb300.vern7 import GpuVern7
    s, op = _op(kind, precision)
    lib, py = (GpuVern7(op, precision=precision, **opts) for _ in range(2))
    py._generator = lambda: None
    for ig in (lib, py):
        ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    assert lib._generator() is not None
    for t, step in [(0.0, False), (0.01, False), (0.02, False), (0.02, False), (0.4, False),
                    (0.41, False), (2.0, True), (2.0, True), (2.0, False), (2.2, False), (0.1, False),
                    (2.3, False)]:
        for ig in (lib, py):
            ig.integrate(t, step=step)
        assert lib.status == py.status and lib.stats == py.stats, (t, step)
        for name in ("t", "t_prev", "t_front", "dt_safe", "dt_int"):
            assert getattr(lib, name) == pytest.approx(getattr(py, name), rel=1e-14, abs=0), name
        if py.status < 0:
            continue
        assert lib._out[0] == py._out[0]
        a, b = lib.get_state(), py.get_state()
        assert float((a - b).abs().max()) <= 1e-13


@pytest.mark.parametrize("kind,precision", KINDS)
def test_outputs_of_a_run(kind, precision):
    """All outputs of a solve in one call: 0, 1 and 40 times in a step, repeated and
    descending ones, against a launch per output."""
    from qutip_gb300.solver import ExpectOps
    from qutip_gb300.vern7 import GpuVern7
    s, op = _op(kind, precision)
    ex = ExpectOps(s.e_ops)
    tl = np.concatenate([[0.0, 0.0], np.linspace(0.001, 0.002, 40), [0.5, 0.5, 0.4999, 1.5]])
    lib, py = (GpuVern7(op, precision=precision) for _ in range(2))
    out = torch.zeros((2, len(tl), 2 * (ex.n + 1)), dtype=torch.float64, device="cuda")
    for ig in (lib, py):
        ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    assert lib.run_dm(tl, ex.dev, s.dim, out[0])
    py._generator = lambda: None
    for i, t in enumerate(tl):
        py.integrate(t)
        py.check()
        ex.expect_dm(s.dim, py.state_view(), out[1, i])
    lib.check()
    assert lib.t == py.t == 1.5 and lib.stats == py.stats
    got = out.cpu().numpy()
    # up to 64 products of values below one in another order
    np.testing.assert_allclose(got[0], got[1], atol=1e-13, rtol=0)


def test_failures_reach_the_caller():
    from qutip_gb300 import _lib
    from qutip_gb300.solver import ExpectOps, solve_system
    from qutip_gb300.vern7 import GpuVern7, IntegratorError
    s, op = _op("csr", "double")
    with pytest.raises(IntegratorError, match="Too much work"):
        solve_system(s, np.linspace(0, 20, 3), {"nsteps": 2}, op=op)
    ig = GpuVern7(op)
    ig.integrate(1.0)                                 # not initialised
    assert not ig.successful()
    ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    with pytest.raises(ValueError):                   # an operator of another dimension
        ig.run_dm([0.0], ExpectOps([np.eye(3)]).dev, 3, torch.zeros(1, 4, device="cuda"))
    gen = _lib.Generator(7, 0, 1, 0)
    assert _lib.load().qg_vern7_integrate(gen, ig._rk(), _lib.Vern7Ctl(), 1.0, 0, None) == \
        _lib.QG_ERR_ARG


@pytest.mark.parametrize("hermitian", [False, True])
@pytest.mark.parametrize("n_cops", [1, 33])
def test_coefficients_evaluated_once_per_step(hermitian, n_cops):
    """Programs of the Hamiltonian's terms and of up to more collapse operators than a warp,
    constant and time-dependent in turn: as when each stage evaluates its own (to rounding)."""
    from qutip_gb300.coefficients import coefficient
    from qutip_gb300.lindblad import LindbladOperator
    from qutip_gb300.vern7 import GpuVern7
    s = S.ising_chain(5)
    f = [None, coefficient("0.5*exp(-t/3) + 0.2j*cos(t)"), coefficient("0.7*sin(2*t)")]
    c_ops = [(0.1 * s.c_ops[i % len(s.c_ops)], f[(i + 1) % 3]) for i in range(n_cops)]
    op = LindbladOperator.from_hamiltonian(s.h_terms, c_ops, dtype="c128")
    op.hermitian = hermitian
    lib, py = (GpuVern7(op) for _ in range(2))
    py._generator = lambda: None
    for ig in (lib, py):
        ig.set_initial_value(torch.from_numpy(s.state0), 0.3)
        for t in (0.35, 1.0):                          # dense output and whole steps
            ig.integrate(t)
        ig.check()
    assert lib.stats == py.stats
    # t_prev + c dt may be fused into one rounding on the host
    assert float((lib.get_state() - py.get_state()).abs().max()) <= 1e-13
