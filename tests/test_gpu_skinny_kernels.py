"""Every kernel of the substitution products in both precisions, with the row maps and
the accumulation that the passes use them with."""
import ctypes

import numpy as np
import pytest

import wtomo3d_gb300 as wt

pytestmark = pytest.mark.gpu

# (precision, kernel, columns, conjugate-transposed): multiply-adds through shared memory,
# one column through registers (complex128: only the conjugate transpose), tensor cores
KERNELS = [(prec, kernel, nc, herm) for prec in (wt.PREC_FP64, wt.PREC_MIXED)
           for kernel, ncs in ((0, (1, 4, 8, 16, 32)), (1, (1,)), (2, (8, 16, 32))) for nc in ncs for herm in (False, True)
           if not (prec == wt.PREC_FP64 and (kernel == 2 or (kernel == 1 and not herm)))]


@pytest.mark.parametrize("prec,kernel,nc,herm", KERNELS)
@pytest.mark.parametrize("tri,M,K,chunk", [(0, 1, 1, 32), (0, 70, 31, 32), (0, 63, 200, 1024), (0, 130, 1500, 512),
                                           (0, 64, 1024, 1024), (1, 189, 189, 64), (2, 189, 189, 64),
                                           (1, 256, 256, 256), (2, 65, 65, 1024)])
def test_kernel(prec, kernel, nc, herm, tri, M, K, chunk):
    r = np.random.default_rng(M + 3 * K + nc + kernel)
    dt = np.complex128 if prec == wt.PREC_FP64 else np.complex64
    cn = lambda *s: (r.standard_normal(s) + 1j * r.standard_normal(s)).astype(dt)
    shape = (K, M) if herm else (M, K)
    A = cn(*shape)
    Ab = np.full((shape[0], shape[1] + 1), np.nan, dt)
    Ab[:, :-1] = A
    nin, nout = K + 9, M + 5
    B, C = cn(nin, nc), cn(nout, nc)
    for sub, maps in ((0, False), (1, True)):
        bm = r.permutation(nin)[:K].astype(np.int32) if maps else np.arange(K, dtype=np.int32)
        cm = r.permutation(nout)[:M].astype(np.int32) if maps else np.arange(M, dtype=np.int32)
        D = A.astype(np.complex128)
        D = np.tril(D, -1) + np.eye(M) if tri == 1 else np.triu(D) if tri == 2 else D
        op = D.conj().T if herm else D
        # products that are stored, not added, need a cleared output where units add up
        out = C.copy() if sub else np.zeros_like(C)
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        rc = wt.lib().wt3d_debug_skinny_kernel(prec, kernel, int(herm), tri, sub, M, K, nc, chunk, p(Ab), Ab.shape[1],
                                               p(B), p(bm) if maps else None, nin, p(out),
                                               p(cm) if maps else None, nout)
        assert rc == 0
        ref, mag = np.zeros((nout, nc), complex), np.zeros((nout, nc))
        ref[cm] = op @ B[bm].astype(np.complex128)
        mag[cm] = abs(op) @ abs(B[bm].astype(np.complex128))
        if sub:
            ref, mag = C - ref, abs(C) + mag
        # 2 K rounded terms in any order, the units' additions, and 3 eps for a split
        # product; the host's sum for complex128
        bound = (2 * K + 3 + K / 32) * np.finfo(dt).eps * mag * (2 if dt == np.complex128 else 1)
        assert (abs(out - ref) <= bound).all()


def test_refused():
    z = np.zeros(64, np.complex64)
    m = np.array([4], np.int32)
    p = ctypes.c_void_p(z.ctypes.data)
    f = wt.lib().wt3d_debug_skinny_kernel
    call = lambda prec=0, kernel=0, nc=1, chunk=32, im=None: f(prec, kernel, 0, 0, 0, 1, 1, nc, chunk, p, 1, p, im, 4, p,
                                                               None, 4)
    assert call() == 0
    for bad in (dict(kernel=1, nc=4), dict(kernel=2), dict(prec=1, kernel=2, nc=8), dict(nc=3), dict(chunk=48), dict(prec=1, kernel=1),
                dict(im=ctypes.c_void_p(m.ctypes.data))):
        assert call(**bad) == wt.WT3D_ERR_ARG
