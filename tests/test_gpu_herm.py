"""The Hermitian half form of the Vern7 stages (``qg_vern7_stage_herm``): against the full
stages, and the test that decides whether it applies (``qg_hermitian_check``)."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402
from qutip_gb300 import vern7_tableau as T  # noqa: E402
from qutip_gb300.coefficients import coefficient  # noqa: E402

pytestmark = pytest.mark.gpu


def _operators(d, seed=0):
    """Sparse Hermitian H0, H1 with few distinct complex elements and two collapse operators."""
    rng = np.random.default_rng(seed)

    def herm():
        m = sp.diags(rng.choice([1.0, -0.5, 0.25], d))
        for o in (1, 3, d // 2):
            v = rng.choice([0.5, 0.25j, -0.5 + 0.25j], d - o)
            m = m + sp.diags(v, o, shape=(d, d)) + sp.diags(v.conj(), -o, shape=(d, d))
        return sp.csr_matrix(m)
    c = sp.diags(rng.choice([0.5, 0.25], d - 1), 1, shape=(d, d), format="csr")
    return herm(), herm(), [c, sp.diags(rng.choice([0.25, -0.25], d), format="csr")]


def _operator(h0, h1, c_ops, coef, dtype):
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.superop import device_term_groups
    terms = [(S.liouvillian(h0, c_ops), None),
             (-1j * (S.spre(h1) - S.spost(h1)), coefficient(coef))]
    return DeviceOperator.from_device_groups(device_term_groups(terms), dtype, fmt="dict")


def _rho(d, seed):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(d, 6)) + 1j * rng.normal(size=(d, 6))
    r = a @ a.conj().T
    r = (r + r.conj().T) / 2
    return torch.from_numpy((r / np.trace(r).real).reshape(-1, order="F").copy()).cuda()


@pytest.mark.parametrize("precision", ["double", "mixed", "single"])
@pytest.mark.parametrize("d", [32, 64, 96, 160])
def test_half_form_matches_the_full_stages(d, precision):
    """One to five 32-row blocks: every k_j, the new state, the error norm and the dense
    output.  A row has at most 20 entries below 4 in magnitude; the two forms sum mirrored
    rows in another order: within 100 eps of the largest k."""
    from qutip_gb300.vern7 import GpuVern7
    op = _operator(*_operators(d, d), "cos(1.3*t)", "c128" if precision == "double" else "c64")
    y0 = _rho(d, d)
    assert op.real_coefficients()
    half, full = (GpuVern7(op, precision=precision, first_step=0.01) for _ in range(2))
    errors = []
    op.hermitian_dim = lambda: d                      # below the size from which it pays
    for ig, h in ((half, True), (full, False)):
        ig._range = lambda *a: False
        ig.set_initial_value(y0, 0.2)
        assert ig._hermitian
        ig._hermitian = h
        ig.t_prev = 0.2
        errors.append([ig._compute_step(dt) for dt in (0.01, 0.03)])
        ig.dt_int = 0.03
        ig._prep_dense_out()
    eps = 2.3e-16 if precision == "double" else 1.2e-7
    for a, b in ((half.k, full.k), (half.y_front, full.y_front)):
        assert float((a - b).abs().max()) <= 100 * eps * float(b.abs().max())
    # a weighted norm of dt sum e_j k_j: it moves by at most dt sum |e_j| max|dk| / atol
    move = 0.03 * np.abs(T.E).sum() * 100 * eps * float(full.k.abs().max()) / full.atol
    np.testing.assert_allclose(errors[0], errors[1], rtol=0, atol=move)
    k = half.k.view(16, d, d)
    i = torch.arange(d, device="cuda") // 32
    off = (i[:, None] != i[None, :])
    assert torch.equal(k[:, off], k.transpose(1, 2).conj()[:, off])   # mirrored bit for bit


@pytest.mark.parametrize("precision", ["double", "mixed", "single"])
@pytest.mark.parametrize("d", [32, 96, 256, 352])
def test_fused_half_form_matches_the_full_stages(d, precision):
    """The half form inside the fused step: one block, several, one unit of 8 warps per SM and
    two.  Bounds as above."""
    from qutip_gb300.vern7 import GpuVern7
    op = _operator(*_operators(d, d), "cos(1.3*t)", "c128" if precision == "double" else "c64")
    y0 = _rho(d, d)
    half, full = (GpuVern7(op, precision=precision, first_step=0.01) for _ in range(2))
    op.hermitian_dim = lambda: d
    run, calls, errors = op.vern7_range_herm, [], []
    op.vern7_range_herm = lambda *a: calls.append(run(*a)) or calls[-1]
    full._range = lambda *a: False
    for ig, h in ((half, True), (full, False)):
        ig.set_initial_value(y0, 0.2)
        assert ig._hermitian
        ig._hermitian = h
        ig.t_prev = 0.2
        errors.append([ig._compute_step(dt) for dt in (0.01, 0.03)])
        ig.dt_int = 0.03
        ig._prep_dense_out()
    assert calls == [True] * 3
    eps = 2.3e-16 if precision == "double" else 1.2e-7
    for a, b in ((half.k, full.k), (half.y_front, full.y_front)):
        assert float((a - b).abs().max()) <= 100 * eps * float(b.abs().max())
    move = 0.03 * np.abs(T.E).sum() * 100 * eps * float(full.k.abs().max()) / full.atol
    np.testing.assert_allclose(errors[0], errors[1], rtol=0, atol=move)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("case", ["ok", "rho", "rho_nan", "h", "c_coef"])
def test_what_the_check_accepts(case, dtype):
    """A non-Hermitian state (one element, a NaN), a non-Hermitian generator (one element of
    H) and a complex coefficient keep the full form."""
    d = 64
    h0, h1, c_ops = _operators(d, 5)
    rho = _rho(d, 5)
    if case == "rho":
        rho[3 + 40 * d] += 1e-9
    if case == "rho_nan":
        rho[7] = float("nan")
    if case == "h":                                   # -i (H rho - rho H) with H not Hermitian
        h0 = h0.tolil()
        h0[50, 2] = 1e-3
        h0 = h0.tocsr()
    op = _operator(h0, h1, c_ops, "exp(1j*t)" if case == "c_coef" else "sin(t)", dtype)
    op.hermitian_dim = lambda: d
    if case == "c_coef":
        assert not op.real_coefficients()
        return
    assert op.check_hermitian(rho) is (case == "ok")


def test_large_solve_takes_the_half_form_and_a_new_coefficient_leaves_it():
    """d = 320 (102,400 rows): chosen by itself, and left when the coefficients become
    complex in mid-solve."""
    from qutip_gb300.vern7 import GpuVern7
    d = 320
    op = _operator(*_operators(d, 1), "cos(t)", "c128")
    ig = GpuVern7(op, first_step=0.01)
    ig.set_initial_value(_rho(d, 2), 0.0)
    assert ig._hermitian and ig._stage() == op.vern7_stage_herm
    op.set_coefficients([None, coefficient("exp(1j*t)")])
    assert ig._stage() == op.vern7_stage
    x = torch.randn(d * d, dtype=torch.complex128, device="cuda")
    op.set_coefficients([None, coefficient("cos(t)")])
    ig.set_initial_value(x, 0.0)
    assert not ig._hermitian
