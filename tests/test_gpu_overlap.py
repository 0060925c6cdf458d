"""Solves and trajectories beside a long batch on another stream: a launch asks for the shared
memory that its operators need, so its blocks find room on SMs that the batch holds in part."""
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


def _beside_a_batch(d, work):
    """Run ``work`` on a stream while one ket of ``d`` entries per SM is integrated on another,
    for some half a second; the result, and that of ``work`` alone."""
    from qutip_gb300.batched import BatchProblem
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h = sp.diags([np.full(d - 1, 1.0), np.full(d - 1, 1.0)], [-1, 1], format="csr")
    psi = np.zeros(d, dtype=np.complex128)
    psi[d // 2] = 1.0
    bp = BatchProblem("c128")
    k = bp.add_system([(-1j * h, None)], [sp.identity(d, format="csr")], [0.0, 1.5e6 / d],
                      kind="mc", nsteps=10**6)
    for i in range(sms):
        bp.add_item(k, psi, seed=i)
    bp.build(max_jumps=1, group="cta", n_slots=sms, stage_operator=True)
    batch, mine = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(mine):
        for _ in range(3):                            # this stream's memory, and the result alone
            want = work()
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    t0 = time.perf_counter()
    with torch.cuda.stream(batch):
        bp.launch()
        done.record()
    with torch.cuda.stream(mine):
        got = work()
    took, running = time.perf_counter() - t0, not done.query()
    torch.cuda.synchronize()
    total = time.perf_counter() - t0
    print(f"batch {total:.3f} s, work beside it {took:.4f} s")
    assert total > 0.2 and running and took < 0.25 * total
    return got, want


def test_a_solve_beside_a_batch():
    """Some 100 KB of shared memory a block of the batch; the solve takes a few milliseconds."""
    from qutip_gb300.operator import DeviceOperator
    from qutip_gb300.solver import ExpectOps, solve_system
    s = S.jaynes_cummings(10)
    op, ex, tl = DeviceOperator(s.terms), ExpectOps(s.e_ops), np.linspace(0, 20, 201)
    got, want = _beside_a_batch(1000, lambda: solve_system(s, tl, op=op, ex=ex).expect)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("d,ntraj", [(40, 100), (5, 10)])
def test_trajectories_beside_a_batch(d, ntraj):
    """Some 30 KB of shared memory a block of the batch; a ket on a CTA of its own takes a few."""
    from qutip_gb300.stochastic import SdeOperator
    a = S.destroy(d)
    op = SdeOperator.sse(sp.csr_matrix(a.conj().T @ a), [sp.csr_matrix(0.3 * a)])
    rng = np.random.default_rng(d)
    psi = rng.normal(size=(ntraj, d)) + 1j * rng.normal(size=(ntraj, d))
    psi = torch.from_numpy(psi / np.linalg.norm(psi, axis=1, keepdims=True)).cuda()
    dW = torch.from_numpy(rng.normal(size=(ntraj, 20, 1)) * 1e-3**0.5).cuda()

    def work():
        x = psi.clone()
        op.advance(x, dW, 20, 1e-3)
        torch.cuda.current_stream().synchronize()
        return x
    got, want = _beside_a_batch(300, work)
    assert torch.equal(got, want)
