"""What the check of the half form says of operators and states that are not finite: the half form
would not meet what stands above the diagonal, so they keep the full form."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _operator(d, dtype):
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.superop import device_term_groups
    h = sp.diags([np.full(d - 1, 0.5), (np.arange(d) % 3) * 0.25, np.full(d - 1, 0.5)], [-1, 0, 1],
                 format="csr")
    c = sp.diags(np.full(d - 1, 0.5), 1, format="csr")
    op = DeviceOperator.from_device_groups(device_term_groups([(S.liouvillian(h, [c]), None)]),
                                           dtype, fmt="dict")
    op.hermitian_dim = lambda: d
    return op


def _rho(d):
    return (torch.eye(d, dtype=torch.complex128, device="cuda") / d).reshape(-1)


# a complex128 table entry holds one real factor twice, a complex64 one a whole value
BOTH, ONE = [(INF, INF), (-INF, INF), (NAN, NAN)], [(INF, 0.0), (0.0, -INF), (NAN, 0.0), (0.0, NAN)]


@pytest.mark.parametrize("dtype,value", [("c128", v) for v in BOTH] + [("c64", v) for v in BOTH + ONE],
                         ids=str)
def test_operators(dtype, value):
    """Every table entry in turn, in both parts and in one."""
    d = 32
    op = _operator(d, dtype)
    assert op.check_hermitian(_rho(d))
    parts = torch.view_as_real(op.val)
    for k in range(1, op.struct.lanes):
        kept = parts[k].clone()
        parts[k] = torch.tensor(value, dtype=parts.dtype, device="cuda")
        assert not op.check_hermitian(_rho(d)), k
        parts[k] = kept
    assert op.check_hermitian(_rho(d))


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("value", [INF, -INF, NAN])
def test_states(value, dtype):
    """One component of an element on, below and above the diagonal, alone or with its mirror."""
    d = 32
    op = _operator(d, dtype)
    for r, c in ((5, 5), (20, 3), (3, 20)):
        for part in (0, 1):
            for mirror in (False, True):
                rho = _rho(d)
                parts = torch.view_as_real(rho)
                parts[r + c * d, part] = value
                if mirror:
                    parts[c + r * d, part] = value if part == 0 else -value
                assert not op.check_hermitian(rho), (r, c, part, mirror)
