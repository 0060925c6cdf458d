"""The library's integration loop on the half form (the fused step and the stages one by one): outputs
and states against the same loop on the full form."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402
from qutip_gb300.coefficients import coefficient  # noqa: E402

pytestmark = pytest.mark.gpu


def _operator(d, dtype):
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.superop import device_term_groups
    h0 = sp.diags([np.full(d - 1, 0.5), (np.arange(d) % 3) * 0.25, np.full(d - 1, 0.5)], [-1, 0, 1],
                  format="csr")
    h1 = sp.diags([np.full(d - 3, 0.5j), np.full(d - 3, -0.5j)], [3, -3], format="csr")
    c = sp.diags(np.full(d - 1, 0.5), 1, format="csr")
    terms = [(S.liouvillian(h0, [c]), None),
             (-1j * (S.spre(h1) - S.spost(h1)), coefficient("cos(1.3*t)"))]
    return DeviceOperator.from_device_groups(device_term_groups(terms), dtype, fmt="dict")


def _rho(d):
    rng = np.random.default_rng(d)
    a = rng.normal(size=(d, 6)) + 1j * rng.normal(size=(d, 6))
    r = a @ a.conj().T
    r = (r + r.conj().T) / 2
    return torch.from_numpy((r / np.trace(r).real).reshape(-1, order="F").copy()).cuda()


# launches of a trial step: one where the rows fit the GPU at once, else the coefficients' and ten
@pytest.mark.parametrize("d,per_step", [(32, 1), (96, 1), (288, 1), (384, 11)])
@pytest.mark.parametrize("precision", ["double", "mixed", "single"])
def test_half_form_in_the_library(d, per_step, precision):
    """Two outputs in one step and a whole run.  Rows of at most 12 entries of magnitude one at
    most summed in another order: a stage moves by 12 eps of the largest k (below 8), the state
    over 0.3 time units by that, the step control by less; tenfold."""
    from qutip_gb300 import _lib
    from qutip_gb300.solver import ExpectOps
    from qutip_gb300.vern7 import GpuVern7
    op = _operator(d, "c128" if precision == "double" else "c64")
    op.hermitian_dim = lambda: d                     # below the size from which it pays, too
    half, full = (GpuVern7(op, precision=precision, first_step=0.02) for _ in range(2))
    e = sp.diags(np.arange(d) / d, format="csr")
    ex = ExpectOps([sp.csr_matrix(e, dtype=np.complex128)])
    tl = np.array([0.0, 0.005, 0.01, 0.15, 0.3])
    eps = 2.3e-16 if precision == "double" else 1.2e-7
    tol = 10 * 12 * 8 * 0.3 * eps
    states, outs = [], []
    for ig, h in ((half, True), (full, False)):
        for run in (False, True):
            ig.set_initial_value(_rho(d), 0.0)
            assert ig._hermitian
            ig._hermitian = h
            gen = ig._generator()
            assert gen.hermitian_d == (d if h else 0)
            if not run:
                before = _lib.LAUNCHES[0]
                ig.integrate(1.0, step=True)
                ig.check()
                if h:
                    assert _lib.LAUNCHES[0] - before == per_step
                ig.set_initial_value(_rho(d), 0.0)
                ig._hermitian = h
                for t in (0.005, 0.01, 0.3):
                    ig.integrate(t)
                ig.check()
                states.append(ig.get_state().clone())
            else:
                out = torch.zeros(len(tl), 4, dtype=torch.float64, device="cuda")
                assert ig.run_dm(tl, ex.dev, d, out)
                out = out.cpu().numpy()
                ig.check()
                outs.append(out)
    assert float((states[0] - states[1]).abs().max()) <= tol
    np.testing.assert_allclose(outs[0], outs[1], rtol=0, atol=tol)
    # the mirrors of what was evaluated, in the 32 x 32 blocks off the diagonal: bit for bit
    r = states[0].view(d, d)
    i = torch.arange(d, device="cuda") // 32
    off = i[:, None] != i[None, :]
    assert torch.equal(r[off], r.t().conj()[off])
