"""The dense generator's FP32 sums against numpy complex128, in the norm of the whole result."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from qutip_gb300.coefficients import coefficient  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [0, 2, 5, 17])
@pytest.mark.parametrize("d", [8, 17, 64, 128])
def test_error_of_the_fp32_sums(d, m):
    """With random entries: a half-warp adds its at most 16 (2 + m) real products one by one, a
    partial sum growing as the root of its terms, so n roundings of u / sqrt(3) leave
    sqrt(n / 6) u; the 16 partials, the rounded inputs and coefficients and the inner product
    of a collapse operator leave some 3 u more.  Twice that."""
    from qutip_gb300.dense import DenseLindbladOperator
    rng = np.random.default_rng(10 * d + m)

    def mat(scale=1.0):
        return scale * (rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    cos = coefficient("cos(0.7*t)")
    a_terms = [(mat(), None), (mat(), cos)]
    c_terms = [(mat(1.0 / d**0.5), cos if i % 2 else None) for i in range(m)]
    op = DenseLindbladOperator(a_terms, c_terms)
    X = mat()
    x = torch.from_numpy(X.reshape(-1, order="F").astype(np.complex64)).cuda()
    y = torch.zeros_like(x)
    op.matvec(0.4, x, y)
    k = np.cos(0.7 * 0.4)
    a = a_terms[0][0] + k * a_terms[1][0]
    want = a @ X + X @ a.conj().T
    for C, c in c_terms:
        want += (1 if c is None else k * k) * (C @ X @ C.conj().T)
    got = y.cpu().numpy().reshape(d, d, order="F")
    error = np.linalg.norm(got - want) / np.linalg.norm(want)
    print(f"d={d} m={m}: {error:.2e}")
    assert error <= 2 * (np.sqrt(16 * (2 + m) / 6) + 3) * 2.0 ** -24
