"""The dense generator's split over a cluster: none to more collapse operators than ranks, at
dimensions around the 16-column blocks and K chunks, against numpy complex128."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300.coefficients import coefficient  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [0, 1, 2, 6, 7, 8, 9, 17])
@pytest.mark.parametrize("d", [1, 9, 16, 33, 128])
def test_generator_split_over_ranks(d, m):
    """A chunk of 32 products accumulates with at most 32 units of 2^-23 of its absolute sum
    and the split of the operands leaves 2^-22: 40 units, twice for the pair of products of a
    collapse operator."""
    from qutip_gb300.dense import DenseLindbladOperator
    rng = np.random.default_rng(100 * d + m)

    def mat(scale=1.0):
        return scale * (rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    cos = coefficient("cos(0.7*t)")
    a_terms = [(mat(), None), (mat(), cos), (mat(), None), (mat(0.5), cos)]
    c_terms = [(mat(0.5), cos if i % 3 == 2 else None) for i in range(m)]
    op = DenseLindbladOperator(a_terms, c_terms)
    assert op.n_groups == 2
    X = mat()
    x = torch.from_numpy(X.reshape(-1, order="F").astype(np.complex64)).cuda()
    y = torch.zeros_like(x)
    t = 0.4
    op.matvec(t, x, y)
    k = np.cos(0.7 * t)
    a = sum(A * (1 if c is None else k) for A, c in a_terms)
    want = a @ X + X @ a.conj().T
    bound = abs(a) @ abs(X) + abs(X) @ abs(a).T
    for C, c in c_terms:
        w = 1 if c is None else k * k
        want += w * (C @ X @ C.conj().T)
        bound += 2 * w * (abs(C) @ abs(X) @ abs(C).T)
    got = y.cpu().numpy().reshape(d, d, order="F")
    assert np.all(abs(got - want) <= 40 * 2.0 ** -23 * bound)
