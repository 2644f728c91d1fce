"""The substitution products on the tensor cores hold FP32: every bit of an operand,
and every entry of a row or a column whatever the magnitudes beside it."""
import numpy as np
import pytest

from test_gpu_skinny import skinny

pytestmark = pytest.mark.gpu


def run(herm, A, B, M, chunk=128):
    """op(A) B for op(A) given."""
    A = np.ascontiguousarray(A.conj().T if herm else A, np.complex64)
    return skinny(herm, 0, A, np.ascontiguousarray(B, np.complex64), M, chunk)


@pytest.mark.parametrize("nc", [8, 16, 32])
@pytest.mark.parametrize("herm", [False, True])
@pytest.mark.parametrize("side", ["factor", "sources"])
def test_every_bit(nc, herm, side):
    """One product per result, of 24-bit parts and a power of two: exact in FP32."""
    M, K = 70, 150
    r = np.random.default_rng(nc)
    full = lambda *s: ((2 * r.integers(2**22, 2**23, s) + 1) * r.choice([-1, 1], s)).astype(float)
    power = lambda *s: np.ldexp(1.0, r.integers(-20, 20, s))
    if side == "factor":
        A = (full(M, K) + 1j * full(M, K)) * power(M, 1)
        B = np.zeros((K, nc), complex)
        B[r.integers(0, K, nc), np.arange(nc)] = power(nc)
    else:
        A = np.zeros((M, K), complex)
        A[np.arange(M), r.integers(0, K, M)] = power(M)
        B = (full(K, nc) + 1j * full(K, nc)) * power(1, nc)
    np.testing.assert_array_equal(run(herm, A, B, M), A @ B)


@pytest.mark.parametrize("nc", [8, 16, 32])
@pytest.mark.parametrize("herm", [False, True])
@pytest.mark.parametrize("kind", ["scatter", "opposed", "grading"])
@pytest.mark.parametrize("M,K", [(15, 64), (64, 160)])
def test_every_entry(nc, herm, kind, M, K):
    r = np.random.default_rng(M + K + nc)
    cn = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)
    if kind == "scatter":      # every entry its own magnitude
        A, B = cn(M, K) * 2.0 ** r.uniform(-60, 0, (M, K)), cn(K, nc) * 2.0 ** r.uniform(-60, 0, (K, nc))
    else:                      # large entries of A meet small ones of B: all products alike
        p = r.uniform(0, 60, K) if kind == "opposed" else np.linspace(0, 60, K)
        A, B = cn(M, K) * 2.0 ** -p, cn(K, nc) * 2.0 ** (p - 60)[:, None]
    A, B = A.astype(np.complex64), B.astype(np.complex64)
    # 2 K rounded terms, and 3 eps more for the products that a split leaves out
    bound = (2 * K + 3) * np.finfo(np.float32).eps * (abs(A.astype(complex)) @ abs(B.astype(complex)))
    assert (abs(run(herm, A, B, M) - A.astype(complex) @ B.astype(complex)) <= bound).all()
