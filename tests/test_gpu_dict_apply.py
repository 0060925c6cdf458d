"""One application of a dictionary-coded operator: blocks with fewer slices than warps, one
and two rounds, and enough rows that the blocks stride; coefficients of every class."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300.coefficients import coefficient  # noqa: E402

pytestmark = pytest.mark.gpu

# slices of 32 rows over 152 blocks of 32 warps: one, one short of and over a block's 31
# workers, one round and one more, two rounds and one more, with ragged last slices
SIZES = [1, 31, 32, 33, 152 * 31 * 32, 152 * 31 * 32 + 5, 152 * 64 * 32, 152 * 64 * 32 + 1]
COEFS = [None, "cos(1.3*t)", "exp(1j*t)"]


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("order", [(0,), (1,), (0, 1, 2), (2, 0, 1)])
@pytest.mark.parametrize("n", SIZES)
def test_apply_matches_scipy(n, order, dtype):
    """A row has at most 5 entries per group, of magnitude below 1.5 with the coefficient:
    rounding stays within (5 groups + 6) eps of 5 x 1.5 x groups x max|x|; times two for the
    complex products."""
    from qutip_gb300.operator import DeviceOperator
    rng = np.random.default_rng(n % 1000 + len(order))
    terms, ref, t = [], 0, 0.4
    for i in order:
        m = sum(sp.diags(rng.choice([0.5, -1.0, 0.25j, 1 - 1j], max(n - abs(o), 0)), o, shape=(n, n))
                for o in (0, 1, -2, 5, 17) if abs(o) < n).tocsr()
        c = coefficient(COEFS[i]) if COEFS[i] else None
        terms.append((m.astype(np.complex128), c))
        ref = ref + (c(t) if c else 1.0) * m
    op = DeviceOperator(terms, dtype=dtype, fmt="dict")
    x = rng.normal(size=n) + 1j * rng.normal(size=n)
    xd = torch.from_numpy(x).cuda().to(torch.complex128 if dtype == "c128" else torch.complex64)
    y = torch.full_like(xd, float("nan"))
    op.matvec(t, xd, y)
    eps = 2.3e-16 if dtype == "c128" else 1.2e-7
    g = len(order)
    bound = 2 * (5 * g + 6) * eps * 5 * 1.5 * g * np.abs(x).max()
    assert np.abs(y.cpu().numpy() - ref @ xd.cpu().numpy().astype(complex)).max() <= bound
