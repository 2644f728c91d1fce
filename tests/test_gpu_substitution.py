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


@pytest.mark.parametrize("k", [8, 17, 33])
def test_incident_field_sources(k):
    """(A_bg - A) u0 by digit products (8 and more sources) against the same
    sources one to three at a time, by the FP64 sum: 162-term sums in both, so
    200 eps of the largest entry of a column."""
    dims = (13, 11, 18)
    g = Grid(*dims, 20.0, pmld=3 * 20.0, fst=1)
    ain, baz = np.radians(np.linspace(1.0, 29.0, k)), np.radians(np.linspace(0.0, 350.0, k))
    lay = wt.Layered1D(*model.layered1d(dims[2], 20.0))
    with wt.Solver(g) as s:
        s.set_model(*model.layered_random(*dims, 20.0, seed=5))
        s.set_background(*model.layered(*dims))
        s.factor(2 * np.pi * 1.5)
        F, U = s.rhs_planewave(lay, ain, baz)
        for c in range(0, k, 3):
            f, u = s.rhs_planewave(lay, ain[c:c + 3], baz[c:c + 3])
            np.testing.assert_array_equal(U[:, c:c + 3], u)
            # the sums' terms: |A_bg - A| |u0| <= 81 * 4e8 * |u0|, F itself 1e5 times less
            scale = 81 * 4e8 * np.abs(u).max(axis=0)
            assert (np.abs(F[:, c:c + 3] - f) <= 200 * np.finfo(float).eps * scale).all()
