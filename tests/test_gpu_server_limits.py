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


def test_budget_for_a_shear_rotation_job(S):
    """A :one job is admitted by a server whose budget is half above what its
    plan takes: no second set of adjoint planes is set aside for it."""
    nx, nz, nview, p = 64, 64, 64, 11
    rng = np.random.default_rng(5)
    mumap = np.zeros((nx, nx, nz), np.float32, order="F")
    psfs = np.asfortranarray(np.repeat(S.psf_gauss(ny=nx, px=p, fwhm_end=2)[:, :, :, None], nview, axis=3), np.float32)
    y = np.asfortranarray(rng.random((nx, nz, nview)), np.float32)
    bg = np.full_like(y, 0.1, order="F")
    plan = S.SPECTplan(mumap, psfs, 4.8, interpmeth="one")
    x0 = np.ones((nx, nx, nz), np.float32, order="F")
    ref = S.osem(x0, y, bg, S.Ablock(plan, 1), niter=1)
    need = plan.info()["device_bytes"]
    plan.close()
    srv = S.Server(budget_bytes=need + need // 2 + (16 << 20))
    img, _ = srv.wait(srv.submit(mumap, psfs, 4.8, y, bg, 1, 1, interpmeth="one"))
    assert relerr(img, ref) <= TOL
    srv.close()
