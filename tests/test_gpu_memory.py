"""Device memory that is short for part of a call: allocations made to fail on the
host."""
import numpy as np
import pytest

import wtomo3d_gb300 as wt
from test_gpu_substitution import point_forces
from wtomo3d_gb300 import Grid, model

pytestmark = pytest.mark.gpu

DIMS = (12, 11, 10)


@pytest.fixture
def solver():
    """Factors of one model, operator of one whose velocities are 1 % higher in places:
    solves need the Krylov solver."""
    g = Grid(*DIMS, 20.0, pmld=3 * 20.0, fst=1)
    with wt.Solver(g) as s:
        vp, vs, rho = model.layered_random(*DIMS, 20.0, seed=1)
        s.set_model(vp, vs, rho)
        s.factor(2 * np.pi * 1.5)
        f = (1 + 0.01 * np.random.default_rng(2).random(vp.shape)).astype(vp.dtype)
        s.set_model(vp * f, vs * f, rho)
        s.update_operator()
        yield s
        wt.lib().wt3d_debug_fail_alloc(0)


# allocations of a device call: digits 1, 2; Krylov bases 3, 4
@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_digits_give_way(solver, nth):
    """Without memory for the digits, or for the Krylov bases beside them, a solve uses
    the FP64 kernel and gives the same wavefields."""
    import torch
    s = solver
    F = torch.from_numpy(np.ascontiguousarray(point_forces(s.grid, 16, 0).T)).cuda()
    X, Y = torch.zeros_like(F), torch.zeros_like(F)
    s.solve_device(F.data_ptr(), X.data_ptr(), 16, tol=1e-10, maxit=60)
    wt.lib().wt3d_debug_fail_alloc(nth)
    s.solve_device(F.data_ptr(), Y.data_ptr(), 16, tol=1e-10, maxit=60)
    assert wt.lib().wt3d_debug_fail_alloc(0) == 0
    # both to 1e-10 of the sources; condition below 1e6
    assert torch.linalg.norm(X - Y) <= 1e-4 * torch.linalg.norm(X)


def test_without_memory_for_the_bases(solver):
    """Fewer columns have no digits to give way: an error, and the next call is right."""
    s = solver
    B = point_forces(s.grid, 3, 0)
    X = s.solve(B, tol=1e-10, maxit=60)
    wt.lib().wt3d_debug_fail_alloc(3)     # sources, solutions, basis
    with pytest.raises(wt.WT3DError):
        s.solve(B, tol=1e-10, maxit=60)
    assert wt.lib().wt3d_debug_fail_alloc(0) == 0
    Y = s.solve(B, tol=1e-10, maxit=60)
    assert np.linalg.norm(X - Y) <= 1e-4 * np.linalg.norm(X)
