"""Substitution passes: block inverses and skinny products at every width of the
right-hand-side blocks, forward and conjugate-transpose, on fronts shorter and
longer than a diagonal block and with ragged last tiles."""
import numpy as np
import pytest

import wtomo3d_gb300 as wt
from wtomo3d_gb300 import Grid, model

pytestmark = pytest.mark.gpu

# top separators of 72, 630 (one full block of 512 and 118 more) and 1053
# unknowns (two full blocks and 29 more)
GRIDS = [(4, 6, 4), (16, 15, 14), (14, 27, 13)]


def point_forces(g, k, seed):
    r = np.random.default_rng(seed)
    B = np.zeros((g.n, k), complex)
    for j in range(k):
        iz, ix, iy = r.integers(0, g.nz - 1), r.integers(1, g.nx - 1), r.integers(1, g.ny - 1)
        B[3 * (iz + g.nz * (ix + g.nx * iy)) + j % 3, j] = r.standard_normal() + 1j * r.standard_normal()
    return B


@pytest.mark.parametrize("dims", GRIDS)
def test_widths(dims):
    g = Grid(*dims, 20.0, pmld=2 * 20.0, fst=1)
    B = point_forces(g, 33, sum(dims))
    with wt.Solver(g, wt.PREC_FP64) as s64, wt.Solver(g) as s32:
        for s in (s64, s32):
            s.set_model(*model.layered_random(*dims, 20.0, seed=3))
            s.factor(2 * np.pi * 1.5)
        for k in (1, 2, 5, 9, 17, 33):
            for name in ("solve", "solve_adjoint"):
                # complex128: one pass, no refinement.  The residual of a
                # backward-stable solve is eps |A| |x| / |b| <= eps * cond, and cond
                # is below 1e7 here: 1e-8 leaves a factor of five
                X64 = getattr(s64, name)(B[:, :k], tol=1e-8, maxit=0)
                # complex64 factors, refined to 1e-11: cond * tol bounds the difference
                X = getattr(s32, name)(B[:, :k], tol=1e-11, maxit=30)
                assert np.linalg.norm(X - X64) <= 1e-4 * np.linalg.norm(X64)


@pytest.mark.parametrize("k", [1, 3, 8, 11, 32, 35])
def test_products(k):
    """A X at every width: FP64 rounding of 81-term sums; an infinity reaches
    every row that stores an entry for it, zero entries included, as it does in
    the full product."""
    import scipy.sparse as sp
    g = Grid(9, 8, 7, 20.0, pmld=2 * 20.0, fst=1)
    vp, vs, rho = model.layered_random(9, 8, 7, 20.0, seed=4)
    ir, jc = wt.pattern(9, 8, 7, base=0)
    A = sp.csr_matrix((wt.assemble(g, vp, vs, rho, 2 * np.pi), jc, ir), shape=(g.n, g.n))
    r = np.random.default_rng(k)
    X = r.standard_normal((g.n, k)) + 1j * r.standard_normal((g.n, k))
    with wt.Solver(g) as s:
        s.set_model(vp, vs, rho)
        s.factor(2 * np.pi)
        Y = s.apply(X)
        # at most 162 rounded products and additions per part
        bound = 200 * np.finfo(float).eps * (abs(A) @ abs(X))
        assert (abs(Y - A @ X) <= bound).all()
        hit = 3 * (g.nnodes // 2) + 1
        X[hit, 0] = np.inf
        Y = s.apply(X)
        stored = np.zeros(g.n, bool)
        stored[np.repeat(np.arange(g.n), np.diff(ir))[jc == hit]] = True
        np.testing.assert_array_equal(~np.isfinite(Y[:, 0]), stored)
        assert np.isfinite(Y[:, 1:]).all()
