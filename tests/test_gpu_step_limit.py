"""Step limits of any size: those past 64 bits are no limit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsteps", [1000, 1e19, 2**63 - 1, 2**63, 2**64, 2**64 + 1])
def test_large_limits(nsteps):
    from qutip_gb300.solver import solve_system
    s = S.jaynes_cummings(5)
    tl = np.linspace(0, 2, 5)
    want = solve_system(s, tl).expect
    got = solve_system(s, tl, {"nsteps": nsteps}).expect
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("nsteps", [0, -1, -2**64])
def test_no_steps_left(nsteps):
    from qutip_gb300.solver import solve_system
    from qutip_gb300.vern7 import IntegratorError
    with pytest.raises(IntegratorError, match="Too much work"):
        solve_system(S.jaynes_cummings(5), np.linspace(0, 20, 5), {"nsteps": nsteps})
