"""The fused trial step and dense-output stages (``qg_vern7_range``) against the same stages
launched one by one (``qg_vern7_stage``, itself checked against the numpy oracle)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300.coefficients import coefficient  # noqa: E402

pytestmark = pytest.mark.gpu


def _terms(n, n_groups, seed, structured):
    """Square random terms; structured: a few diagonals of few values (dictionary codes)."""
    rng = np.random.default_rng(seed)
    coefs = [None, coefficient("cos(1.3*t)"), coefficient("exp(-1j*t)*0.5")]
    out = []
    for g in range(n_groups):
        if structured:
            offs = [o for o in (0, 1, -2, 5, 17) if abs(o) < n]
            m = sum(sp.diags(rng.choice([0.5, -1.0, 0.25j, 1 - 1j], n - abs(o)), o, shape=(n, n))
                    for o in offs)
        else:
            lens = rng.integers(0, min(n, 12) + 1, n)     # empty rows among them
            if n > 40:
                lens[n // 2] = 40                        # a row longer than a thread keeps
            rows = np.repeat(np.arange(n), lens)
            v = rng.uniform(-1, 1, (2, len(rows)))
            m = sp.coo_matrix((v[0] + 1j * v[1], (rows, rng.integers(0, n, len(rows)))), (n, n))
        out.append((sp.csr_matrix(m, dtype=np.complex128), coefs[g]))
    return out


CASES = [("csr", 2, 1, 1), ("csr", 2, 33, 2), ("csr", 4, 400, 1), ("csr", 8, 1023, 3),
         ("csr", 4, 9001, 2), ("csr", 2, 38912, 1), ("sliced", 1, 31, 1), ("sliced", 1, 1025, 3),
         ("dict", 1, 32, 2), ("dict", 1, 129, 1), ("dict", 1, 4099, 3), ("dict", 1, 77824, 2)]


@pytest.mark.parametrize("precision", ["double", "mixed", "single"])
@pytest.mark.parametrize("fmt,lanes,n,n_groups", CASES)
def test_range_matches_single_stages(fmt, lanes, n, n_groups, precision):
    """Every k_j, the new state, its error norm and the dense-output stages.  A row has at
    most 60 entries of magnitude below 2, so two orders or contractions of its sum differ by
    less than 200 eps of the largest k."""
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.vern7 import GpuVern7
    dtype = "c128" if precision == "double" else "c64"
    op = DeviceOperator(_terms(n, n_groups, n, fmt == "dict"), dtype=dtype, fmt=fmt)
    if fmt == "csr":
        op.set_launch(("direct", 0, lanes))
    rng = np.random.default_rng(n)
    y0 = torch.from_numpy(rng.normal(size=n) + 1j * rng.normal(size=n))
    got, want = (GpuVern7(op, precision=precision, first_step=0.01) for _ in range(2))
    want._range = lambda *a: False
    calls = []
    run = op.vern7_range
    op.vern7_range = lambda *a: calls.append(run(*a)) or calls[-1]
    errors = []
    for ig in (got, want):
        ig.set_initial_value(y0, 0.1)
        ig.t_prev = 0.1
        errors.append([])
        for dt in (0.01, 0.02):                          # two trial steps, then dense output
            errors[-1].append(ig._compute_step(dt))
        ig.dt_int = 0.02
        ig._prep_dense_out()
    assert calls and all(calls), "the fused kernel did not take this operator"
    eps = 2.3e-16 if precision == "double" else 1.2e-7
    for a, b in ((got.k, want.k), (got.y_front, want.y_front)):
        scale = float(b.abs().max())
        assert float((a - b).abs().max()) <= 200 * eps * scale
    np.testing.assert_allclose(errors[0], errors[1], rtol=1e-9 if precision == "double" else 1e-3)
    assert int(got.counter[0]) == 0


def test_too_many_rows_take_single_stages():
    """One row more than the GPU holds at once: no fused launch, the same integration."""
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.vern7 import GpuVern7
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 512 + 1
    op = DeviceOperator(_terms(n, 1, 3, True), dtype="c64", fmt="dict")
    ig = GpuVern7(op, precision="mixed", first_step=0.01)
    ig.set_initial_value(torch.ones(n, dtype=torch.complex128), 0.0)
    assert ig._range(ig._rk(), 0, 10, 0.01, 0) is False
    ig.integrate(0.05)
    ig.check()


def test_range_rejects_bad_calls():
    from qutip_gb300 import _lib
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.vern7 import GpuVern7
    ig = GpuVern7(DeviceOperator(_terms(40, 1, 3, False)))
    rk, base = ig._rk(), C.c_uint32(0)
    lib = _lib.load()
    args = lambda s0, s1, bar: (C.byref(ig.op.struct), C.byref(rk), s0, s1, 0.0, 0.1, 1e-8, 1e-6,  # noqa: E731
                                bar, C.byref(base), None)
    assert lib.qg_vern7_range(*args(0, 9, ig.counter.data_ptr())) == _lib.QG_ERR_ARG
    assert lib.qg_vern7_range(*args(3, 10, ig.counter.data_ptr())) == _lib.QG_ERR_ARG
    assert lib.qg_vern7_range(*args(0, 10, None)) == _lib.QG_ERR_ARG
