"""Expectation values at several output times inside one Vern7 step
(``qg_expect_dm_times``) against the dense output formed in numpy FP64."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import vern7_tableau as T  # noqa: E402

pytestmark = pytest.mark.gpu


def _factors(tau, dt):
    out = []
    for i in range(16):
        acc = 0.0
        for j in range(T.DENSEOUT_ORDER - 1, -1, -1):
            acc = (acc + T.BI[i][j]) * tau
        out.append(dt * acc)
    return np.array(out)


@pytest.mark.parametrize("stage_dtype", ["c128", "c64"])
@pytest.mark.parametrize("d,n_ops,n_times", [(1, 1, 1), (2, 2, 33), (15, 1, 2), (16, 3, 32),
                                             (33, 2, 65), (64, 31, 3), (130, 1, 1), (300, 11, 5)])
def test_expect_at_several_times(d, n_ops, n_times, stage_dtype):
    """Operators of every fill (empty rows, an empty operator, dense rows), one to many row
    chunks, and more times than one launch takes.  The entries are of order one, so a sum
    of m products differs between orders by less than 4 m eps (1 + sum |f|)."""
    from qutip_gb300.solver import ExpectOps
    rng = np.random.default_rng(7 * d + n_ops)
    n = d * d
    ops = [sp.random(d, d, density=[0.0, 1.0, 0.05][k % 3], random_state=k + d, format="csr")
           * (1 + 0.5j) for k in range(1, n_ops + 1)]
    kd = torch.complex128 if stage_dtype == "c128" else torch.complex64
    z = lambda m: rng.normal(size=m) + 1j * rng.normal(size=m)  # noqa: E731
    base = torch.from_numpy(z(n)).cuda()
    k = torch.from_numpy(z(16 * n)).cuda().to(kd)

    class Step:
        t_prev, dt_int = 0.3, 0.17
        scratch = torch.zeros(4096, dtype=torch.float64, device="cuda")
        counter = torch.zeros(4, dtype=torch.int32, device="cuda")

        @staticmethod
        def step_view():
            import ctypes as C
            from qutip_gb300 import _lib
            return _lib.StateView(n, 0, 0 if stage_dtype == "c128" else 1, base.data_ptr(),
                                  k.data_ptr(), 0, 0, (C.c_double * 16)())

    times = Step.t_prev + Step.dt_int * rng.uniform(0, 1, n_times)
    times[0] = Step.t_prev                       # every factor zero: the base itself
    out = torch.full((n_times, 2 * (n_ops + 1)), 7.0, dtype=torch.float64, device="cuda")
    ExpectOps(ops).expect_dm_step(d, Step, times, out)
    got = out.cpu().numpy()
    assert int(Step.counter[0]) == 0
    kk = k.cpu().numpy().astype(np.complex128).reshape(16, n)
    for i, t in enumerate(times):
        f = _factors((t - Step.t_prev) / Step.dt_int, Step.dt_int)
        rho = (base.cpu().numpy() + f @ kk).reshape(d, d, order="F")
        for g, op in enumerate(ops + [sp.identity(d, format="csr")]):
            want = (op @ rho).trace()
            tol = 4 * max(op.nnz, 1) * 2.3e-16 * 6 * (1 + np.abs(f).sum())
            assert abs(got[i, 2 * g] + 1j * got[i, 2 * g + 1] - want) <= tol, (i, g)
