"""A solve beside a long batch on another stream: the fused step asks for the shared memory that
its rows need, so its blocks find room on SMs that the batch holds in part."""
import time

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from qutip_gb300 import systems as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("fmt", ["csr", "sliced", "dict"])
def test_longest_rows(fmt, dtype):
    """The operator's own count against its stored layout, on both ways to build one."""
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.superop import device_term_groups
    s = S.jaynes_cummings(7)
    ops = [DeviceOperator(s.terms, dtype=dtype, fmt=fmt)]
    if fmt != "csr":
        ops.append(DeviceOperator.from_device_groups(device_term_groups(s.terms), dtype, fmt=fmt))
    for op in ops:
        G = op.n_groups
        if fmt == "csr":
            rp = op.row_ptr.cpu().numpy()[:op.n_rows * G + 1]
            want = np.diff(rp[::G]).max()
        else:
            w = op.slice_width.cpu().numpy().reshape(-1, G)
            want = (w if fmt == "sliced" else (w + 3) // 4).sum(axis=1).max()
        assert op.struct.row_words == want > 0


def test_a_solve_beside_a_batch():
    """One ket of 1,000 entries per SM for half a second, each with some 100 KB of shared
    memory; a solve of a few milliseconds ends long before they do, with its own result."""
    from qutip_gb300.batched import BatchProblem
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.solver import ExpectOps, solve_system
    d, sms = 1000, torch.cuda.get_device_properties(0).multi_processor_count
    h = sp.diags([np.full(d - 1, 1.0), np.full(d - 1, 1.0)], [-1, 1], format="csr")
    psi = np.zeros(d, dtype=np.complex128)
    psi[d // 2] = 1.0
    bp = BatchProblem("c128")
    k = bp.add_system([(-1j * h, None)], [sp.identity(d, format="csr")], [0.0, 1500.0], kind="mc",
                      nsteps=10**6)
    for i in range(sms):
        bp.add_item(k, psi, seed=i)
    bp.build(max_jumps=1, group="cta", n_slots=sms, stage_operator=True)
    s = S.jaynes_cummings(10)
    op, ex, tl = DeviceOperator(s.terms), ExpectOps(s.e_ops), np.linspace(0, 20, 201)
    batch, mine = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(mine):
        for _ in range(3):                            # memory of this stream, and the result alone
            want = solve_system(s, tl, op=op, ex=ex).expect
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    t0 = time.perf_counter()
    with torch.cuda.stream(batch):
        bp.launch()
        done.record()
    with torch.cuda.stream(mine):
        got = solve_system(s, tl, op=op, ex=ex).expect
    solved, running = time.perf_counter() - t0, not done.query()
    torch.cuda.synchronize()
    total = time.perf_counter() - t0
    print(f"batch {total:.3f} s, solve beside it {solved:.4f} s")
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert total > 0.2 and running and solved < 0.25 * total
