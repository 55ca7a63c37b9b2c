"""The server's slot limit and its statistics: a job is active from its
admission (its slot and memory are taken) until it is retired."""
import time

import numpy as np
import pytest

from conftest import relerr
from test_gpu_server import TOL, _studies, _submit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1, 2, 3])
def test_no_more_jobs_than_slots(S, O, limit):
    """Four scheduler threads, eight jobs at once: no more than max_active are
    ever admitted together, at any time that the statistics are read."""
    st = _studies(O)[1]
    srv = S.Server(max_active=limit)
    tickets = [_submit(srv, st) for _ in range(8)]
    seen = []
    while not seen or seen[-1]["done"] + seen[-1]["failed"] < 8:
        seen.append(srv.stats())
        assert seen[-1]["active"] <= seen[-1]["max_active_seen"] <= limit, seen[-1]
        time.sleep(1e-4)
    res = [srv.wait(t)[0] for t in tickets]
    for r in res[1:]:
        assert relerr(r, res[0]) <= TOL
    end = srv.stats()
    assert end["active"] == end["pending"] == end["failed"] == 0 and 1 <= end["max_active_seen"] <= limit
    assert np.isfinite(res[0]).all()
    srv.close()
