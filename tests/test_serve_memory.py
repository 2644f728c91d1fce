"""Admission counts the memory that the pool of temporaries keeps as free, and the
temporaries of a solve as needed."""
import pytest

from wtomo3d_gb300 import serve

KEY = ((12, 11, 10), 0, 1.0)


@pytest.mark.parametrize("free,kept,fits", [(0, 0, False), (0, 1, True), (0.5, 0.5, True), (1, 0, True), (0.5, 0.4, False)])
def test_can_open(monkeypatch, free, kept, fits):
    be = serve.GpuBackend(dx=20.0, pml_nodes=3)
    n = be.grid(KEY[0]).n
    _, _, ws = be.wt.solver_bytes(be.grid(KEY[0]), be.precision)
    # the handle, its workspace, Krylov bases (32 columns, complex128), digits (16 bytes and
    # one for each of 88 entries per row, and 6 integers), a margin of 4 GB
    need = be.bytes_needed(KEY) + 1.25 * ws + n * (288 * 32 + 88 * 17 + 24) + 4e9
    monkeypatch.setattr(be.wt, "mem_info", lambda: (free * need, 280e9))
    # 1 GB of the pool is in use by a running call
    monkeypatch.setattr(be.wt, "scratch_info", lambda: (kept * need * 1.001 + 1e9, 1e9), raising=False)
    assert be.can_open(KEY, freeing=0.001 * need * (free > 0)) == fits
