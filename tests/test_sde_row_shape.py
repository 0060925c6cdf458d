"""The launch shapes of the stochastic row kernel (``qg_sde_row_shape``): every state length and
operator count that it takes fits the shared memory it asks for."""
import math

import numpy as np
import pytest
import scipy.sparse as sp

from qutip_gb300 import _lib

LIMIT = 227 * 1024 - 1024   # shared memory of a CTA, less what the kernel declares itself


@pytest.mark.parametrize("sms", [1, 148, 152])
@pytest.mark.parametrize("n_sc", [1, 2])
@pytest.mark.parametrize("open_", [False, True])
def test_vectors_and_operators_fit(open_, n_sc, sms):
    lib = _lib.load()
    shape = np.zeros(4, dtype=np.int32)
    lengths = [d * d for d in range(1, 26)] if open_ else range(1, 641)
    taken = 0
    for n in lengths:
        d = math.isqrt(n) if open_ else n
        for n_traj in (1, sms, 3 * sms + 1, 100 * sms, 392 * sms, 600 * sms, 2**31 - 1):
            rc = lib.qg_sde_row_shape(n, n_sc, int(open_), n_traj, sms, 0, shape.ctypes.data)
            assert rc == (1 if n > (640 if n_sc == 1 else 512) else 0)
            if rc:
                continue
            taken += 1
            T, threads, vecs, ops = (int(v) for v in shape)
            # X and VT, VP and VM of each operator; the terms of every sum, the sums and, of a
            # ket, what their squares scale
            sums = 2 * n_sc * n_sc + (0 if open_ else n_sc)
            need = 16 * T * ((2 + 2 * n_sc) * n + sums * (d + (1 if open_ else 2)))
            assert T >= 1 and vecs >= need and ops >= 0 and vecs + ops <= LIMIT, (n, n_traj)
            assert T * n <= threads <= (640 if n_sc == 1 else 512) and threads % 32 == 0
            most = ops
            for known in (16, 4096, 71 * 1024, 73 * 1024, 2**31 - 1):
                assert lib.qg_sde_row_shape(n, n_sc, int(open_), n_traj, sms, known,
                                            shape.ctypes.data) == 0
                assert list(shape) == [T, threads, vecs, min(most, known)]
    assert taken > 100
    assert lib.qg_sde_row_shape(4, 3, 0, 1, sms, 0, shape.ctypes.data) == 1
    assert lib.qg_sde_row_shape(0, 1, 0, 1, sms, 0, shape.ctypes.data) == _lib.QG_ERR_ARG
    assert lib.qg_sde_row_shape(4, 1, 0, 1, sms, 0, None) == _lib.QG_ERR_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", ["platen", "euler"])
def test_kets_of_one_entry_fill_a_cta(scheme):
    """Two operators and enough trajectories that the shared memory limits a CTA."""
    torch = pytest.importorskip("torch")
    from oracle.sde import euler_steps, platen_steps
    from qutip_gb300.stochastic import SdeOperator
    rng = np.random.default_rng(1)
    ntraj, dt = 512 * torch.cuda.get_device_properties(0).multi_processor_count, 1e-3
    h = sp.csr_matrix(np.array([[0.7 + 0j]]))
    cs = [sp.csr_matrix(np.array([[v]])) for v in (0.4 + 0.1j, -0.3j)]
    psi = np.exp(2j * np.pi * rng.uniform(size=(ntraj, 1)))
    dW = rng.normal(size=(ntraj, 5, 2)) * np.sqrt(dt)
    x = torch.from_numpy(psi).cuda()
    SdeOperator.sse(h, cs).advance(x, torch.from_numpy(dW).cuda(), 5, dt, scheme=scheme)
    got = x.cpu().numpy()
    L = -1j * h - 0.5 * sum(c.conj().T @ c for c in cs)
    steps = platen_steps if scheme == "platen" else euler_steps
    for k in (0, 390, 391, 392, 511, 512, ntraj // 2, ntraj - 1):
        want = steps(L, cs, [c + c.conj().T for c in cs], psi[k], dW[k], dt, False)
        # ~40 operations per entry and step on values of magnitude one: 1e-13 over 5 steps
        np.testing.assert_allclose(got[k], want, atol=1e-12, rtol=0)
