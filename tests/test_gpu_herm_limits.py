"""The Hermitian half form at its launch limits: every size of the dictionary's tables."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _operator(d, dtype, entries=None):
    """A driven chain's Liouvillian; its tables filled up with unused entries to ``entries``."""
    from qutip_gb300.coefficients import coefficient
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.superop import device_term_groups
    h0 = sp.diags([np.full(d - 1, 0.5), (np.arange(d) % 3) * 0.25, np.full(d - 1, 0.5)], [-1, 0, 1])
    h1 = sp.diags([np.full(d - 3, 0.5j), np.full(d - 3, -0.5j)], [3, -3])
    c = sp.diags(np.full(d - 1, 0.5), 1)
    terms = [(S.liouvillian(sp.csr_matrix(h0), [sp.csr_matrix(c)]), None),
             (-1j * (S.spre(sp.csr_matrix(h1)) - S.spost(sp.csr_matrix(h1))), coefficient("cos(t)"))]
    op = DeviceOperator.from_device_groups(device_term_groups(terms), dtype, fmt="dict")
    if entries is not None:
        more = entries - op.struct.lanes
        assert more >= 0
        val = torch.cat([op.val, torch.zeros(more, *op.val.shape[1:], dtype=op.val.dtype,
                                             device=op.val.device)])
        off = torch.cat([op.dict_off, torch.zeros(more, dtype=op.dict_off.dtype,
                                                  device=op.dict_off.device)])
        start = op.dict_start.clone()
        start[-1] = entries
        op.val, op.dict_off, op.dict_start = val, off, start
        op.struct.val, op.struct.dict_off, op.struct.dict_start = (
            t.data_ptr() for t in (val, off, start))
        op.struct.lanes = entries
    return op


def _rho(d, seed):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(d, 6)) + 1j * rng.normal(size=(d, 6))
    r = a @ a.conj().T
    r = (r + r.conj().T) / 2
    return torch.from_numpy((r / np.trace(r).real).reshape(-1, order="F").copy()).cuda()


# static shared memory and tables together pass the 48 KB default at 1,599 entries of 20 bytes
# (complex128) and 3,355 of 12 bytes (complex64)
@pytest.mark.parametrize("precision,entries", [
    ("double", 64), ("double", 1597), ("double", 1598), ("double", 1599), ("double", 1638),
    ("double", 1639), ("double", 4096), ("mixed", 2730), ("mixed", 2731), ("mixed", 3355), ("mixed", 4096)])
def test_every_size_of_the_tables_is_taken(precision, entries):
    """A trial step and the dense-output stages by half against the full form: rows of at most
    12 entries of magnitude one at most, summed in another order: 100 eps of the largest k."""
    from qutip_gb300.vern7 import GpuVern7
    d = 64
    op = _operator(d, "c128" if precision == "double" else "c64", entries)
    op.hermitian_dim = lambda: d                     # below the size from which it pays
    half, full = (GpuVern7(op, precision=precision, first_step=0.01) for _ in range(2))
    for ig, h in ((half, True), (full, False)):
        ig._range = lambda *a: False
        ig.set_initial_value(_rho(d, 3), 0.2)
        assert ig._hermitian
        ig._hermitian = h
        ig._compute_step(0.01)
        ig.dt_int = 0.01
        ig._prep_dense_out()
    eps = 2.3e-16 if precision == "double" else 1.2e-7
    assert float((half.k - full.k).abs().max()) <= 100 * eps * float(full.k.abs().max())
