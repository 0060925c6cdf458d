"""Operators that replace ``vern7_stage``, by a subclass or on the object: every stage goes through
the replacement, whatever fused or half form the original would have taken."""
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _operator(cls, half):
    s = S.ising_chain(5) if half else S.jaynes_cummings(7)
    if not half:
        return s, cls(s.terms)
    from qutip_gb300.superop import device_term_groups
    op = cls.from_device_groups(device_term_groups(s.terms), "c128", fmt="dict")
    op.hermitian_dim = lambda: s.dim                  # below the size from which it pays
    return s, op


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("how", ["subclass", "object"])
def test_replaced_stages_are_called(how, half):
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.vern7 import GpuVern7
    calls = []

    class Counting(DeviceOperator):
        def vern7_stage(self, rk, stage, *args):
            calls.append(stage)
            return super().vern7_stage(rk, stage, *args)
    s, op = _operator(Counting if how == "subclass" else DeviceOperator, half)
    if how == "object":
        own = op.vern7_stage
        op.vern7_stage = lambda rk, stage, *args: calls.append(stage) or own(rk, stage, *args)
    plain = _operator(DeviceOperator, half)[1]
    got, want = GpuVern7(op), GpuVern7(plain)
    for ig in (got, want):
        ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
        ig.integrate(0.05)
        ig.check()
    assert want._generator() is not None
    trials = got.stats["steps"]
    assert calls == list(range(10)) * trials + list(range(10, 16))
    assert got.stats == want.stats
    # one trial step or a few of the same stages, summed in another order at most
    assert float((got.get_state() - want.get_state()).abs().max()) <= 1e-13


@pytest.mark.parametrize("kind", ["matrix", "dense"])
def test_replaced_stages_of_the_matrix_forms(kind):
    from qutip_gb300.dense import DenseLindbladOperator
    from qutip_gb300.lindblad import LindbladOperator
    from qutip_gb300.vern7 import GpuVern7
    s = S.ising_chain(5)
    op = (LindbladOperator.from_hamiltonian(s.h_terms, s.c_ops, dtype="c64") if kind == "matrix"
          else DenseLindbladOperator.from_hamiltonian(s.h_terms, s.c_ops[:3]))
    ig = GpuVern7(op, precision="mixed")
    assert ig._generator() is not None
    calls, own = [], op.vern7_stage
    op.vern7_stage = lambda rk, stage, *args: calls.append(stage) or own(rk, stage, *args)
    ig.set_initial_value(torch.from_numpy(s.state0), 0.0)
    ig.integrate(0.05)
    ig.check()
    assert calls == list(range(10)) * ig.stats["steps"] + list(range(10, 16))
