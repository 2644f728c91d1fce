"""The substitution products on the tensor cores: rows and columns of very
different magnitudes keep the accuracy of FP32 products, entries that are not
finite stay in their row or column, and lengths off the 16-deep chunks."""
import numpy as np
import pytest

from test_gpu_skinny import skinny

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [8, 16, 32])
@pytest.mark.parametrize("herm", [False, True])
@pytest.mark.parametrize("M,K", [(15, 33), (17, 47), (33, 129), (64, 640)])
def test_scales(nc, herm, M, K):
    r = np.random.default_rng(M + K + nc)
    cn = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)
    # rows of op(A) over 40 decades, columns of B over 16, entries within a row over 4
    A = cn(M, K) * 10.0 ** r.uniform(-20, 20, (M, 1)) * 10.0 ** r.uniform(-4, 0, (M, K))
    B = (cn(K, nc) * 10.0 ** r.uniform(-8, 8, (1, nc))).astype(np.complex64)
    A = np.ascontiguousarray(A.conj().T if herm else A, np.complex64)
    out = skinny(herm, 0, A, B, M, 128)
    op = (A.conj().T if herm else A).astype(np.complex128)
    # 2 K rounded terms, and 3 eps more for a split product
    bound = (2 * K + 3) * np.finfo(np.float32).eps * (np.abs(op) @ np.abs(B).astype(np.float64))
    assert (np.abs(out - op @ B.astype(np.complex128)) <= bound).all()


@pytest.mark.parametrize("nc", [8, 16, 32])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite(nc, bad):
    M, K = 40, 200
    r = np.random.default_rng(nc)
    A = (r.standard_normal((M, K)) + 1j * r.standard_normal((M, K))).astype(np.complex64)
    B = (r.standard_normal((K, nc)) + 1j * r.standard_normal((K, nc))).astype(np.complex64)
    good = skinny(False, 0, A, B, M, 256)
    A[7, 150] = bad
    B[20, 3] = bad
    out = skinny(False, 0, A, B, M, 256)
    assert not np.isfinite(out[7]).any() and not np.isfinite(out[:, 3]).any()
    keep = np.ones((M, nc), bool)
    keep[7] = False
    keep[:, 3] = False
    assert (out[keep] == good[keep]).all()
