"""The autotuner measures what a plan runs: results are shared by plans of the
same kernels only, and candidates that do not differ are not timed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(S, plan, nv):
    L = S._native.lib()
    before = L.spect_kernel_launches()
    fwd, adj = plan.autotune(nv)
    assert fwd > 0 and adj > 0
    return L.spect_kernel_launches() - before


def _plan(S, nx, nz, p, nview, end, factors=True):
    psf = S.psf_gauss(ny=nx, px=p, pz=p, fwhm_start=1, fwhm_end=end)
    if not factors:
        i, j = np.meshgrid(np.arange(p) - p // 2, np.arange(p) - p // 2, indexing="ij")
        psf = psf * (1 + 0.5 * np.cos(i * j)).astype(np.float32)[:, :, None]
    psfs = np.asfortranarray(np.repeat((psf / psf.sum(axis=(0, 1)))[:, :, :, None], nview, axis=3), np.float32)
    return S.SPECTplan(np.zeros((nx, nx, nz), np.float32, order="F"), psfs, 4.8)


def test_gather_and_slice_plans_are_tuned_apart(S, monkeypatch):
    """Split plans with the gather rotation launch neither k_rot_fwd nor
    k_rot_adj, whose splits the others try; their choice is not handed on."""
    n = {}
    for gather in ("1", "0"):
        monkeypatch.setenv("SPECT_GADJ", gather)
        plan = _plan(S, 36, 11, 5, 9, 2.0, factors=False)
        assert plan.path == "split"
        n[gather] = _launches(S, plan, 7)
        assert _launches(S, plan, 7) == 0  # known by now
        plan.close()
    assert 0 < n["1"] < n["0"] / 2, n


def test_plans_of_other_kept_taps_are_measured(S):
    """Two fused plans of one PSF size whose planes keep few and many taps."""
    for end in (1.5, 9.0):
        plan = _plan(S, 44, 13, 21, 9, end)
        assert plan.path == "fused"
        assert _launches(S, plan, 7) > 0, end
        assert _launches(S, plan, 7) == 0
        plan.close()
