"""The half form in complex64 stages is no less exact than the full form."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["superoperator", "matrix"])
def test_mixed_half_form_against_complex128(form):
    """Largest error of the outputs against the complex128 solution, the mean of sixteen
    random Ising chains: an element and its mirror share their rounding errors in the half
    form, so it must make fewer."""
    from qutip_gb300.lindblad import LindbladOperator
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.solver import ExpectOps, solve_system
    tl = np.linspace(0, 10, 51)
    errors = {True: [], False: []}
    for seed in range(16):
        s = S.ising_chain(7, seed=seed)
        ex = ExpectOps(s.e_ops)
        want = solve_system(s, tl, op=DeviceOperator(s.terms, dtype="c128", fmt="dict"), ex=ex).expect
        if form == "matrix":
            op = LindbladOperator.from_hamiltonian(s.h_terms, s.c_ops, dtype="c64")
        else:
            op = DeviceOperator(s.terms, dtype="c64", fmt="dict")
        for half in (True, False):
            opt = {"precision": "mixed"}
            if form == "matrix":
                opt["hermitian_branch"] = half
            else:
                op.hermitian_dim = (lambda: s.dim) if half else (lambda: 0)
            got = solve_system(s, tl, opt, op=op, ex=ex).expect
            errors[half].append(max(np.abs(a - b).max() for a, b in zip(got, want)))
    half, full = np.mean(errors[True]), np.mean(errors[False])
    print(f"half {half:.3g}, full {full:.3g}")
    assert half <= full < 1e-6
