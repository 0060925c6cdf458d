"""Stochastic steps of states from the shortest to past the row kernel's limits (640 entries,
one or two operators), against the numpy restatement of the reference's schemes."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from oracle.sde import euler_steps, platen_steps  # noqa: E402
from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _ops(d, m):
    a = S.destroy(d)
    h = a.conj().T @ a + 0.3 * (a + a.conj().T) + 0.1j * (a - a.conj().T)
    cs = [(0.4 + 0.1j * i) * a if i % 2 == 0 else 0.2 * sp.diags(np.cos(np.arange(d)))
          for i in range(m)]
    return sp.csr_matrix(h), [sp.csr_matrix(c, dtype=np.complex128) for c in cs]


def _check(op, L, C, M, x0, dW, dt, scheme, open_, pick):
    x = torch.from_numpy(x0).cuda()
    op.advance(x, torch.from_numpy(dW).cuda(), dW.shape[1], dt, scheme=scheme)
    got = x.cpu().numpy()
    steps = platen_steps if scheme == "platen" else euler_steps
    for k in pick:
        want = steps(L, C, M, x0[k], dW[k], dt, open_)
        # ~40 operations per entry and step on values below one: 1e-13 over 5 steps
        np.testing.assert_allclose(got[k], want, atol=1e-12, rtol=0)


@pytest.mark.parametrize("scheme", ["platen", "euler"])
@pytest.mark.parametrize("d,m,ntraj", [(2, 1, 1), (5, 1, 700), (5, 2, 333), (31, 2, 161),
                                       (32, 1, 5), (33, 1, 400), (64, 2, 700), (65, 1, 310),
                                       (213, 1, 460), (512, 2, 2), (513, 2, 2), (640, 1, 3),
                                       (641, 1, 2), (12, 3, 4)])
def test_kets(d, m, ntraj, scheme):
    """Short kets side by side in a CTA (the last CTA partly empty), the longest of either
    operator count, and one entry or one operator past it."""
    from qutip_gb300.stochastic import SdeOperator
    rng = np.random.default_rng(d + 10 * m)
    h, cs = _ops(d, m)
    psi = rng.normal(size=(ntraj, d)) + 1j * rng.normal(size=(ntraj, d))
    psi *= np.exp(-np.arange(d))[None, :]
    psi /= np.linalg.norm(psi, axis=1, keepdims=True)
    dt = 1e-3
    dW = rng.normal(size=(ntraj, 5, m)) * np.sqrt(dt)
    L = -1j * h - 0.5 * sum(c.conj().T @ c for c in cs)
    _check(SdeOperator.sse(h, cs), L, cs, [c + c.conj().T for c in cs], psi, dW, dt, scheme, False,
           sorted({0, ntraj // 2, ntraj - 1}))


@pytest.mark.parametrize("scheme", ["platen", "euler"])
@pytest.mark.parametrize("d,m,ntraj", [(2, 1, 500), (5, 2, 310), (9, 1, 400), (20, 1, 3),
                                       (22, 2, 2), (23, 2, 2), (25, 1, 2), (26, 1, 2), (4, 3, 3)])
def test_density_matrices(d, m, ntraj, scheme):
    from qutip_gb300.stochastic import SdeOperator
    rng = np.random.default_rng(d + 20 * m)
    h, cs = _ops(d, m)
    psi = rng.normal(size=(ntraj, d)) + 1j * rng.normal(size=(ntraj, d))
    psi *= np.exp(-np.arange(d))[None, :]
    psi /= np.linalg.norm(psi, axis=1, keepdims=True)
    x0 = (psi.conj()[:, :, None] * psi[:, None, :]).reshape(ntraj, -1)
    dt = 1e-3
    dW = rng.normal(size=(ntraj, 5, m)) * np.sqrt(dt)
    L = S.liouvillian(h, cs)
    C = [S.spre(c) + S.spost(c.conj().T) for c in cs]
    _check(SdeOperator(L, C, open=True, d=d), L, C, None, x0, dW, dt, scheme, True,
           sorted({0, ntraj // 2, ntraj - 1}))
