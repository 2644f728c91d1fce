import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
TESTS = os.path.dirname(os.path.abspath(__file__))
for p in (TESTS, os.path.join(TESTS, "golden"), os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300, sm_103a)")


@pytest.fixture(autouse=True)
def shared_factorisations(request, monkeypatch):
    """test_gpu_serve asks that some of its requests share a batch.  The closest two
    for one key come 25.9 ms apart, which is longer than a request takes, so by
    default none meet.  There a key that would evict another waits for 0.2 s: the
    third key of the stream is the first to wait, the others queue behind it, and the
    two come while their key is waiting."""
    if request.module.__name__ == "test_gpu_serve":
        from wtomo3d_gb300 import serve
        monkeypatch.setattr(serve.Server, "HOLD_S", 0.2)
        monkeypatch.setattr(serve.Server, "THRASH_S", float("inf"))


@pytest.fixture(scope="session")
def oracle():
    import oracle_ctypes
    return oracle_ctypes.Oracle()
