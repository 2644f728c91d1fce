"""Products of the grid's operator, row by row: every row has the error of its own
FP64 sum whatever the magnitudes of X around it, at every width of a block of
columns, stored and conjugate-transposed."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

import wtomo3d_gb300 as wt
from wtomo3d_gb300 import Grid, model

pytestmark = pytest.mark.gpu

DIMS = (11, 9, 10)
EPS = np.finfo(float).eps


def matrix(g, mdl, om):
    ir, jc = wt.pattern(g.nx, g.ny, g.nz, base=0)
    return sp.csr_matrix((wt.assemble(g, *mdl, om), jc, ir), shape=(g.n, g.n))


def fields(kind, k, r):
    """n x k columns whose entries span up to 2^-80 .. 1 within a few nodes."""
    nx, ny, nz = DIMS
    at = np.stack(np.meshgrid(np.arange(ny), np.arange(nx), np.arange(nz), indexing="ij"), -1)
    shape = (k, ny, nx, nz, 3)
    x = r.standard_normal(shape) + 1j * r.standard_normal(shape)
    if kind == "spike":         # one node far above all others
        for j in range(k):
            x[j, ny // 2, nx // 2, j % nz] *= 2.0 ** (80 * (j + 1) / k)
    elif kind == "decay":       # up to 2^-20 from node to node
        d = np.abs(at - np.array([ny // 2, nx // 2, nz // 2])).sum(-1)
        x *= 2.0 ** -(20.0 * (np.arange(k) + 1)[:, None, None, None, None] / k * np.minimum(d, 30)[..., None])
    elif kind == "scatter":     # every entry its own
        x *= 2.0 ** r.uniform(-80, 0, shape)
    elif kind == "components":  # u, v, w
        x *= 2.0 ** np.array([0, -24, -60])
    elif kind == "zeros":       # mostly zeros, a few small entries next to a large one
        x *= 2.0 ** r.uniform(-40, 0, shape) * (r.random(shape) < 0.05)
    return np.asfortranarray(x.reshape(k, -1).T)


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("k", [4, 5, 16, 33])
@pytest.mark.parametrize("kind", ["spike", "decay", "scatter", "components", "zeros"])
def test_rows(kind, k, adjoint):
    g = Grid(*DIMS, 20.0, pmld=3 * 20.0, fst=1)
    mdl = model.layered_random(*DIMS, 20.0, seed=4)
    A = matrix(g, mdl, 2 * np.pi)
    A = A.conj().T.tocsr() if adjoint else A
    X = fields(kind, k, np.random.default_rng(k))
    with wt.Solver(g) as s:
        s.set_model(*mdl)
        s.factor(2 * np.pi)
        if adjoint:
            Y = np.empty_like(X)
            wt._check(wt.lib().wt3d_debug_product(s._h, 1, k, ctypes.c_void_p(X.ctypes.data),
                                                  ctypes.c_void_p(Y.ctypes.data)))
        else:
            Y = s.apply(X)
    # at most 162 rounded products and additions per part, here and on the host
    assert (abs(Y - A @ X) <= 400 * EPS * (abs(A) @ abs(X))).all()


def test_incident_field_rows():
    """(A_bg - A) u0 against the host's sum of the same entries, row by row."""
    dims, k = (13, 11, 18), 17
    g = Grid(*dims, 20.0, pmld=3 * 20.0, fst=1)
    mdl, bg = model.layered_random(*dims, 20.0, seed=5), model.layered(*dims)
    om = 2 * np.pi * 1.5
    D = matrix(g, bg, om) - matrix(g, mdl, om)
    with wt.Solver(g) as s:
        s.set_model(*mdl)
        s.set_background(*bg)
        s.factor(om)
        F, U = s.rhs_planewave(wt.Layered1D(*model.layered1d(dims[2], 20.0)), np.radians(np.linspace(1.0, 29.0, k)),
                               np.radians(np.linspace(0.0, 350.0, k)))
    assert (abs(F - D @ U) <= 400 * EPS * (abs(D) @ abs(U))).all()
