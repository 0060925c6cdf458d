"""Host threads that launch one kernel with different sizes of shared memory, each on a stream of
its own: no thread's launch depends on the limit another one set last."""
import threading

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


def _operator(d, entries):
    """A chain's Liouvillian with tables filled up with unused entries."""
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.superop import device_term_groups
    h = sp.diags([np.full(d - 1, 0.5), (np.arange(d) % 3) * 0.25, np.full(d - 1, 0.5)], [-1, 0, 1],
                 format="csr")
    c = sp.diags(np.full(d - 1, 0.5), 1, format="csr")
    op = DeviceOperator.from_device_groups(device_term_groups([(S.liouvillian(h, [c]), None)]),
                                           "c128", fmt="dict")
    more = entries - op.struct.lanes
    pad = lambda t: torch.cat([t, torch.zeros(more, dtype=t.dtype, device=t.device)])  # noqa: E731
    op.val, op.dict_off = pad(op.val), pad(op.dict_off)
    op.dict_start = op.dict_start.clone()
    op.dict_start[-1] = op.struct.lanes = entries
    op.struct.val, op.struct.dict_off, op.struct.dict_start = (
        t.data_ptr() for t in (op.val, op.dict_off, op.dict_start))
    return op


def test_solves_with_tables_of_different_sizes():
    """Two solves by half, 42 and 82 KB of tables, each some 3000 launches inside the library
    (without the interpreter's lock): both succeed and give the states of a solve alone, bit
    for bit."""
    from qutip_gb300.vern7 import GpuVern7
    d = 384                                           # stages of one launch each
    rho = torch.eye(d, dtype=torch.complex128).reshape(-1) / d
    got, failures = {}, []

    def solve(key, op):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                ig = GpuVern7(op, first_step=0.001, max_step=0.001)
                ig.set_initial_value(rho, 0.0)
                assert ig._hermitian
                ig.integrate(0.3)
                ig.check()
                got[key] = ig.get_state().cpu()
        except Exception as exc:  # noqa: BLE001
            failures.append(repr(exc))
    ops = {n: _operator(d, n) for n in (2100, 4096)}
    torch.cuda.synchronize()
    for n, op in ops.items():
        solve(("alone", n), op)
    threads = [threading.Thread(target=solve, args=((i, n), op)) for i in range(4)
               for n, op in ops.items()]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    for i in range(4):
        for n in ops:
            assert torch.equal(got[i, n], got["alone", n])
