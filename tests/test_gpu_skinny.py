"""The products of the substitution passes against numpy: every width, rows and
columns off the tile sizes, cut along K, both triangles of a packed inverse,
stored and conjugate-transposed."""
import ctypes

import numpy as np
import pytest

import wtomo3d_gb300 as wt

pytestmark = pytest.mark.gpu


def skinny(herm, tri, A, B, M, chunk):
    K, nc = B.shape
    out = np.zeros((M, nc), np.complex64)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    rc = wt.lib().wt3d_debug_skinny(int(herm), tri, M, K, nc, chunk, p(A), A.shape[1], p(B), p(out))
    assert rc == 0, wt.lib().wt3d_last_error()
    return out


@pytest.mark.parametrize("nc", [1, 4, 8, 16, 32])
@pytest.mark.parametrize("herm", [False, True])
@pytest.mark.parametrize("tri,M,K,chunk", [(0, 1, 1, 32), (0, 63, 65, 64), (0, 130, 700, 256), (0, 64, 1024, 1024),
                                           (1, 189, 189, 64), (2, 189, 189, 64), (1, 64, 64, 64), (2, 65, 65, 1024)])
def test_skinny(nc, herm, tri, M, K, chunk):
    r = np.random.default_rng(M + 3 * K + nc)
    shape = (K, M) if herm else (M, K)
    A = (r.standard_normal(shape) + 1j * r.standard_normal(shape)).astype(np.complex64)
    lda = shape[1] + (3 if shape[1] % 2 == 0 else 0)     # rows off 16-byte boundaries
    Ab = np.full((shape[0], lda), np.nan, np.complex64)
    Ab[:, :shape[1]] = A
    B = (r.standard_normal((K, nc)) + 1j * r.standard_normal((K, nc))).astype(np.complex64)
    Ad = A.astype(np.complex128)
    if tri == 1:
        Ad = np.tril(Ad, -1) + np.eye(M)
    elif tri == 2:
        Ad = np.triu(Ad)
    op = Ad.conj().T if herm else Ad
    out = skinny(herm, tri, Ab, B, M, chunk)
    # 2 K rounded terms: 2 K eps of the sum of magnitudes bounds any order of summation,
    # and 3 eps more covers a split product
    bound = (2 * K + 3) * np.finfo(np.float32).eps * (np.abs(op) @ np.abs(B).astype(np.float64))
    assert (np.abs(out - op @ B.astype(np.complex128)) <= bound).all()
