"""The hold of a thrashing factorisation cache: requests for a key that would
evict a factorisation in use a moment ago wait for others of their key; without
pressure nothing waits."""
import pytest

from test_serve import FakeBackend, _req
from wtomo3d_gb300 import serve


@pytest.mark.parametrize("budget,hold,shared", [(10.0, 0.2, True), (10.0, 0.0, False), (100.0, 0.2, False)])
def test_hold(budget, hold, shared):
    be = FakeBackend(factor_s=0.01, solve_s=0.01, size=lambda dims: 10.0)
    srv = serve.Server(be, budget_bytes=budget, workers=2, hold_s=hold, thrash_s=0.5)
    A, B = ((4, 4, 4), 0, 1.0), ((4, 4, 4), 1, 1.0)
    # A is done by 0.1 and idle; B comes twice, the second time well inside the hold
    # and well after a factorisation and a solve that had not waited
    stream = [_req(0, 0.0, *A), _req(1, 0.15, *B), _req(2, 0.25, *B)]
    srv.run(stream, timeout_s=30)
    srv.close()
    assert (stream[1].batch_id == stream[2].batch_id) == shared
    # the hold is bounded: the first request of B is not answered later than its
    # hold, a factorisation, a solve and some scheduling after it came
    assert stream[1].t_done - stream[1].t_arrival < hold + 0.15
