"""View groups of the split kernels with the gather rotation at their limits:
single slices of large matrices, where a group holds the most planes."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-4  # against the oracle, as in the other parity tests
SAME = 1e-5  # between two orders of a Float32 sum over a few hundred views (sqrt(720) 2^-24 = 1.6e-6)


def _study(S, nx, nview, seed, separable=False):
    rng = np.random.default_rng(seed)
    mumap = np.asfortranarray(0.01 * rng.random((nx, nx, 1)), np.float32)
    psf = S.psf_gauss(ny=nx, px=3, pz=3, fwhm_start=1, fwhm_end=1.5)
    if not separable:
        i, j = np.meshgrid(np.arange(3) - 1, np.arange(3) - 1, indexing="ij")
        psf = psf * (1 + 0.5 * np.cos(i * j)).astype(np.float32)[:, :, None]
    psf = psf / psf.sum(axis=(0, 1), keepdims=True)
    psfs = np.asfortranarray(np.repeat(psf[:, :, :, None], nview, axis=3), np.float32)
    y = np.asfortranarray(rng.random((nx, 1, nview)), np.float32)
    return mumap, psfs, y


def test_more_columns_than_a_list_word_holds(S, O):
    """720 views of 500x500x1 are 1.8e8 adjoint columns, above the 2^27 of one
    group: all views at once against two index lists that fit a group each, and
    against the oracle."""
    nx, nview = 500, 720
    mumap, psfs, y = _study(S, nx, nview, 1)
    plan = S.SPECTplan(mumap, psfs, 4.8)
    assert plan.path == "split"
    whole = S.backproject(y, plan)
    parts = [S.backproject(np.asfortranarray(y[:, :, i]), plan, index=i.astype(np.int32))
             for i in (np.arange(0, nview // 2), np.arange(nview // 2, nview))]
    plan.close()
    assert relerr(whole, parts[0] + parts[1]) <= SAME
    assert relerr(whole, O.Geometry(mumap, psfs, 4.8).backproject(y)) <= TOL


def test_more_planes_than_a_grid_holds(S, O, monkeypatch):
    """520 views of 128x128x1 are 66 560 adjoint planes, above the 65 535
    blocks of a grid's second dimension that the transpose of the direct
    convolution's planes has."""
    nx, nview = 128, 520
    monkeypatch.setenv("SPECT_ZPATH", "0")
    monkeypatch.setenv("SPECT_CONV", "direct")
    mumap, psfs, y = _study(S, nx, nview, 2, separable=True)
    plan = S.SPECTplan(mumap, psfs, 4.8)
    assert plan.path == "split" and plan.conv_kernels()["adjoint"] == "direct"
    out = S.backproject(y, plan)
    plan.close()
    assert relerr(out, O.Geometry(mumap, psfs, 4.8).backproject(y)) <= TOL


@pytest.mark.parametrize("interp", ["one", "two"])
def test_more_views_than_a_grid_holds(S, O, interp):
    """70 000 views of a 6x6x1 image on the fused pair: the attenuation of
    views past the 65 535 blocks of a grid's second dimension."""
    nx, nview = 6, 70000
    mumap, _, _ = _study(S, nx, 1, 3)
    psf = S.psf_gauss(ny=nx, px=3, pz=1, fwhm_start=1, fwhm_end=1.5)
    psfs = np.asfortranarray(np.repeat(psf[:, :, :, None], nview, axis=3), np.float32)
    plan = S.SPECTplan(mumap, psfs, 4.8, interpmeth=interp)
    assert plan.path == "fused"
    idx = np.array([69999, 0, 65535, 17501, 65534], np.int32)
    x = np.asfortranarray(np.random.default_rng(4).random((nx, nx, 1)), np.float32)
    out = S.project(x, plan, index=idx)
    plan.close()
    G = O.Geometry(mumap, psfs, 4.8, interp=interp)
    assert relerr(out, G.project(x, index=idx)) <= TOL


def test_padded_cache_too_large_for_the_fused_pair(S, O):
    """2200 views of 500x500x1: the fused pair's z-fastest attenuation (16 values
    a column) would take 35 GB, above the cache's bound; the 2.2 GB of the split
    kernels' cache still fit, and the plan keeps them."""
    nx, nview = 500, 2200
    mumap, _, _ = _study(S, nx, 1, 5)
    psf = S.psf_gauss(ny=nx, px=3, pz=1, fwhm_start=1, fwhm_end=1.5)
    psfs = np.asfortranarray(np.repeat(psf[:, :, :, None], nview, axis=3), np.float32)
    plan = S.SPECTplan(mumap, psfs, 4.8)
    assert plan.path == "split"
    assert plan.info()["device_bytes"] > 4 * nx * nx * nview
    idx = np.array([2199, 3, 1100], np.int32)
    x = np.asfortranarray(np.random.default_rng(6).random((nx, nx, 1)), np.float32)
    out = S.project(x, plan, index=idx)
    plan.close()
    assert relerr(out, O.Geometry(mumap, psfs, 4.8).project(x, index=idx)) <= TOL
