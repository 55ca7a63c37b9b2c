"""Every form of the adjoint convolution kernel: tasks of 8 and 16 outputs, one
and two row buffers, one and several row tiles (some shorter than the PSF's half
width, the last one partial)."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-4  # against the oracle, as in the other parity tests


@pytest.mark.parametrize("nx,nz,px,pz,nview,tiles", [
    (64, 40, 11, 11, 12, (1, 2, 5)),   # whole x tasks; five tiles of 8 rows
    (46, 37, 9, 33, 10, (1, 3, 5)),    # ragged; half width 16 against tiles of 8 rows, an odd last row
    (6, 1, 3, 1, 4, (1,)),             # one row
])
def test_adjoint_forms_agree(S, O, monkeypatch, nx, nz, px, pz, nview, tiles):
    """An output's taps run in the same order in every form, so the
    back-projections are the same bits; one of them meets the oracle."""
    rng = np.random.default_rng(nx + nz)
    mumap = np.asfortranarray(0.01 * rng.random((nx, nx, nz)), np.float32)
    psf = S.psf_gauss(ny=nx, px=px, pz=pz, fwhm_x=np.linspace(1, px / 2, nx), fwhm_z=np.linspace(1, max(1, pz / 2), nx))
    psfs = np.asfortranarray(np.repeat(psf[:, :, :, None], nview, axis=3), np.float32)
    y = np.asfortranarray(rng.random((nx, nz, nview)), np.float32)
    idx = np.array([nview - 1, 0, 2], np.int32)
    out = {}
    for w in ("8", "16"):
        for nxb in ("1", "2"):
            for nt in tiles:
                monkeypatch.setenv("SPECT_ZW", w)
                monkeypatch.setenv("SPECT_ZADJ_BUFFERS", nxb)
                monkeypatch.setenv("SPECT_ZADJ_TILES", str(nt))
                plan = S.SPECTplan(mumap, psfs, 4.8)
                assert plan.path == "fused"
                out[w, nxb, nt] = (S.backproject(y, plan),
                                   S.backproject(np.asfortranarray(y[:, :, idx]), plan, index=idx))
                plan.close()
    first = out["8", "1", 1]
    for k, o in out.items():
        for a, b in zip(o, first):
            np.testing.assert_array_equal(a, b, err_msg=str(k))
    G = O.Geometry(mumap, psfs, 4.8)
    assert relerr(first[0], G.backproject(y)) <= TOL
    assert relerr(first[1], G.backproject(np.asfortranarray(y[:, :, idx]), index=idx)) <= TOL
