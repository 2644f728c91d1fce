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


def test_nothing_runs_after_an_error():
    """A call that fails has finished with its caller's buffers: here before its first
    pass, with the columns' conversion queued behind the caller's own work."""
    import ctypes
    import torch
    dims = (24, 22, 20)
    g = Grid(*dims, 20.0, pmld=5 * 20.0, fst=1)
    L = wt.lib()
    with wt.Solver(g) as s:
        s.set_model(*model.layered_random(*dims, 20.0, seed=1))
        s.factor(2 * np.pi)
        F = torch.randn((32, s.n), dtype=torch.complex128, device="cuda")
        X = torch.zeros_like(F)
        work = torch.zeros(1 << 27, device="cuda")
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        torch.cuda.synchronize()
        for _ in range(400):      # 1 GB each: 60 ms and more
            work.mul_(1.0)
        L.wt3d_debug_fail_alloc(3)     # digits 1, 2; the pass's schedule
        rc = L.wt3d_solve_device(s._h, 32, p(F), p(X), 1e-10, 10, None, None, 0)
        idle = L.wt3d_debug_idle(s._h)
        assert L.wt3d_debug_fail_alloc(0) == 0
        assert rc == wt.WT3D_ERR_NOMEM and idle == 1


def test_pool_of_temporaries(solver):
    """What the pool keeps between calls is counted, and returned when asked for."""
    s = solver
    s.solve(point_forces(s.grid, 16, 0), tol=1e-10, maxit=60)
    held, used = wt.scratch_info()
    assert held > 0 and used == 0
    free, _ = wt.mem_info()
    wt.scratch_trim()
    assert wt.scratch_info() == (0.0, 0.0)
    assert wt.mem_info()[0] > free


def test_no_pool_without_handles():
    """A call without a handle leaves nothing behind in the pool."""
    g = Grid(*DIMS, 20.0, pmld=3 * 20.0, fst=1)
    wt.assemble(g, *model.layered_random(*DIMS, 20.0, seed=1), 2 * np.pi)
    assert wt.scratch_info() == (0.0, 0.0)
