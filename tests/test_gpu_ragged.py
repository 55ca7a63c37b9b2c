"""The fused projector pair on matrices that no task width divides (any even
nx, any nz, px != pz), against the split kernels (SPECT_ZPATH=0) of the same
plan and against the Float32 and Float64 oracles.

Tolerances: 1e-4 against the oracles, the bound of the other parity tests
(max|gpu - oracle| / max|oracle|); 1e-5 between the two GPU paths, which carry
~1e-6 each (Float32 FFT and direct sums of up to 65 taps).
"""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _plan_inputs(S, nx, nz, px, pz, nview, seed):
    rng = np.random.default_rng(seed)
    mumap = np.asfortranarray(0.01 * rng.random((nx, nx, nz)), np.float32)
    psf = S.psf_gauss(ny=nx, px=px, pz=pz, fwhm_start=1, fwhm_end=max(1.5, px / 5))
    psfs = np.asfortranarray(np.repeat(psf[:, :, :, None], nview, axis=3), np.float32)
    x = np.asfortranarray(rng.random((nx, nx, nz)), np.float32)
    y = np.asfortranarray(rng.random((nx, nz, nview)), np.float32)
    return mumap, psfs, x, y


@pytest.mark.parametrize("nx,nz,px,pz,nview,idx", [
    (90, 53, 21, 17, 12, [11, 0, 4]),  # a partial x task of two columns, an odd last row
    (46, 80, 7, 7, 10, None),          # six columns in the last x task
    (34, 9, 5, 3, 9, [8, 2]),          # one z task and a row
    (10, 3, 3, 3, 7, None),            # one x task and two columns
    (2, 1, 1, 1, 4, None),             # the smallest image, no blur
    (66, 1, 9, 1, 16, [3, 15]),        # one slice
    (122, 66, 25, 25, 5, [4, 1]),      # several warps of partial tasks
])
def test_ragged_fused_pair(S, O, monkeypatch, nx, nz, px, pz, nview, idx):
    mumap, psfs, x, y = _plan_inputs(S, nx, nz, px, pz, nview, 7 * nx + nz)
    ii = None if idx is None else np.array(idx, np.int32)
    ys = y if ii is None else np.asfortranarray(y[:, :, ii])
    out = {}
    for path in ("fused", "split"):
        monkeypatch.setenv("SPECT_ZPATH", "1" if path == "fused" else "0")
        plan = S.SPECTplan(mumap, psfs, 4.8)
        assert plan.path == path
        out[path] = (S.project(x, plan, index=ii), S.backproject(ys, plan, index=ii))
        plan.close()
    for a, b in zip(out["fused"], out["split"]):
        assert relerr(a, b) <= 1e-5
    for dtype in (np.float32, np.float64):
        G = O.Geometry(mumap, psfs, 4.8, dtype=dtype)
        assert relerr(out["fused"][0], G.project(x, index=ii)) <= TOL
        assert relerr(out["fused"][1], G.backproject(ys, index=ii)) <= TOL


def test_ragged_osem_and_view_dependent_psfs(S, O):
    """OS-EM with a PSF stack of its own for every view (a body-contouring
    orbit) on a matrix of 38 columns and 21 rows."""
    nx, nz, p, nview = 38, 21, 9, 8
    mumap, _, x, _ = _plan_inputs(S, nx, nz, p, p, nview, 3)
    psfs = np.stack([S.psf_gauss(ny=nx, px=p, fwhm_start=1, fwhm_end=1.5 + 0.1 * v) for v in range(nview)], axis=3)
    psfs = np.asfortranarray(psfs, np.float32)
    plan = S.SPECTplan(mumap, psfs, 4.8)
    assert plan.path == "fused" and plan.info()["nset"] == nview
    G = O.Geometry(mumap, psfs, 4.8)
    yn = np.asfortranarray(G.project(x) + 0.1, np.float32)
    bg = np.full(yn.shape, 0.05, np.float32, order="F")
    x0 = np.ones(x.shape, np.float32, order="F")
    assert relerr(S.osem(x0, yn, bg, S.Ablock(plan, 4), niter=2), G.osem(x0, yn, bg, 4, 2)) <= TOL


@pytest.mark.parametrize("nx,nz,px,pz,nview,idx", [
    (32, 20, 5, 3, 8, None),           # views at multiples of 45 and 90 degrees
    (46, 17, 7, 7, 11, [10, 0, 3]),    # a partial x task, an odd last row
    (2, 1, 1, 1, 5, None),
    (128, 80, 37, 37, 120, [0, 30, 44, 97]),
])
def test_shear_rotation_on_the_fused_pair(S, O, monkeypatch, nx, nz, px, pz, nview, idx):
    """:one (three shears) as one gather of eight taps and its transpose,
    against the line-by-line kernels of the split path and the oracles; image
    and views are dense up to the corners, where the shears reach the edge of
    the padded grid."""
    mumap, psfs, x, y = _plan_inputs(S, nx, nz, px, pz, nview, 5 * nx + nz)
    ii = None if idx is None else np.array(idx, np.int32)
    ys = y if ii is None else np.asfortranarray(y[:, :, ii])
    out = {}
    for path in ("fused", "split"):
        monkeypatch.setenv("SPECT_ZPATH", "1" if path == "fused" else "0")
        plan = S.SPECTplan(mumap, psfs, 4.8, interpmeth="one")
        assert plan.path == path
        out[path] = (S.project(x, plan, index=ii), S.backproject(ys, plan, index=ii))
        plan.close()
    for a, b in zip(out["fused"], out["split"]):
        assert relerr(a, b) <= 1e-5
    G = O.Geometry(mumap, psfs, 4.8, interp="one")
    assert relerr(out["fused"][0], G.project(x, index=ii)) <= TOL
    assert relerr(out["fused"][1], G.backproject(ys, index=ii)) <= TOL


@pytest.mark.parametrize("nx,nz,px,pz,nview,idx", [
    (90, 53, 21, 17, 12, [11, 0, 4]),  # three column tiles, the last of 26 columns; an odd last row
    (34, 9, 5, 3, 9, None),            # two tiles of 20 and 14 columns
    (10, 3, 3, 3, 7, None),
    (2, 1, 1, 1, 4, None),
])
def test_ragged_large_plane_kernels(S, O, monkeypatch, nx, nz, px, pz, nview, idx):
    """The large-plane forward kernels (forced) on ragged matrices equal the
    fused kernel bit for bit."""
    mumap, psfs, x, y = _plan_inputs(S, nx, nz, px, pz, nview, 11 * nx + nz)
    ii = None if idx is None else np.array(idx, np.int32)
    out = {}
    for strip in ("0", "1"):
        monkeypatch.setenv("SPECT_ZSTRIP", strip)
        plan = S.SPECTplan(mumap, psfs, 4.8)
        assert plan.path == ("strip" if strip == "1" else "fused")
        out[strip] = S.project(x, plan, index=ii)
        plan.close()
    assert np.array_equal(out["0"], out["1"])
    assert relerr(out["1"], O.Geometry(mumap, psfs, 4.8).project(x, index=ii)) <= TOL


def test_unsynchronised_chain_equals_synchronised(S):
    """Kernels of consecutive calls overlap at their ends (programmatic
    dependent launch): a chain of projections and back-projections in which
    every call reads what the call before it wrote gives the same bits as with
    a synchronisation after each, on the default and on another stream."""
    import torch

    nx, nz, nview = 48, 21, 12
    mumap, psfs, x, y = _plan_inputs(S, nx, nz, 7, 5, nview, 9)
    plan = S.SPECTplan(mumap, psfs, 4.8)
    idx = [np.array([3, 0, 7], np.int32), None, np.array([11, 2], np.int32)]
    x0 = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    ref = None
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        for sync in (True, False):
            with torch.cuda.stream(stream):
                stream.wait_stream(torch.cuda.default_stream())
                im = x0.clone()
                got = []
                for step in range(9):
                    ii = idx[step % 3]
                    n = nview if ii is None else len(ii)
                    v = torch.empty((n, nz, nx), device="cuda")
                    S.project_(v.permute(2, 1, 0), im.permute(2, 1, 0), plan, index=ii, stream=stream)
                    if sync:
                        torch.cuda.synchronize()
                    out = torch.empty_like(im)
                    S.backproject_(out.permute(2, 1, 0), v.permute(2, 1, 0), plan, index=ii, stream=stream)
                    if sync:
                        torch.cuda.synchronize()
                    im = out / out.abs().max()
                    got += [v, im]
                torch.cuda.synchronize()
            if ref is None:
                ref = got
            assert all(torch.equal(a, b) for a, b in zip(got, ref))


def test_device_array_checks(S):
    """Device arrays meet the same checks however they are read: shape, type,
    strides, gradients; arrays that only offer the interface still work, and
    an index list longer than a kernel's own list gives the same views."""
    import torch

    nx, nz, nview = 16, 5, 300
    mumap, psfs, x, _ = _plan_inputs(S, nx, nz, 3, 3, nview, 1)
    plan = S.SPECTplan(mumap, psfs, 4.8)
    im = torch.from_numpy(np.ascontiguousarray(x.T)).cuda().permute(2, 1, 0)
    out = torch.empty((nview, nz, nx), device="cuda").permute(2, 1, 0)
    S.project_(out, im, plan)
    with pytest.raises(S.SpectError):
        S.project_(out[:, :, :2], im, plan)
    with pytest.raises(TypeError):
        S.project_(out, im.double(), plan)
    with pytest.raises(ValueError):
        S.project_(out, im.permute(1, 0, 2), plan)
    with pytest.raises(RuntimeError):
        S.project_(out, im.clone().requires_grad_(True), plan)

    class Interface:
        def __init__(self, t):
            self.__cuda_array_interface__ = t.__cuda_array_interface__

    again = torch.empty_like(out)
    S.project_(Interface(again), Interface(im), plan, index=np.arange(nview, dtype=np.int32))
    torch.cuda.synchronize()
    assert relerr(again.cpu().numpy(), out.cpu().numpy()) <= 1e-6


@pytest.mark.parametrize("nx,nz,px,pz,nview,idx", [
    (90, 53, 21, 17, 12, [11, 0, 4]),  # rows of 90: unstaged planes, an odd last row, z groups past the end
    (128, 80, 37, 37, 8, None),        # staged planes, whole tiles of 32 columns
    (36, 9, 5, 3, 9, [8, 2]),          # staged, one tile and four columns
    (2, 1, 1, 1, 4, None),             # the smallest image
    (66, 1, 9, 1, 6, [3, 5]),          # one slice
    (32, 200, 7, 5, 5, None),          # many z groups of one column tile
])
@pytest.mark.parametrize("stage", ["1", "0"])
def test_split_rotation_by_gathers(S, O, monkeypatch, nx, nz, px, pz, nview, idx, stage):
    """PSFs that no two factors give: the rotation by gathers of z-fastest
    columns and the convolution's z-fastest store against the slice kernels
    (SPECT_GADJ=0), whose forward planes are the same bits, and the oracle."""
    mumap, psfs, x, y = _plan_inputs(S, nx, nz, px, pz, nview, 11 * nx + nz)
    i, j = np.meshgrid(np.arange(px) - px // 2, np.arange(pz) - pz // 2, indexing="ij")
    psfs = psfs * (1 + 0.5 * np.cos(i * j)).astype(np.float32)[:, :, None, None]
    psfs = np.asfortranarray(psfs / psfs.sum(axis=(0, 1), keepdims=True), np.float32)
    ii = None if idx is None else np.array(idx, np.int32)
    ys = y if ii is None else np.asfortranarray(y[:, :, ii])
    monkeypatch.setenv("SPECT_ZPATH", "0")
    monkeypatch.setenv("SPECT_NO_STAGE", "0" if stage == "1" else "1")
    out = {}
    for gather in ("1", "0"):
        monkeypatch.setenv("SPECT_GADJ", gather)
        plan = S.SPECTplan(mumap, psfs, 4.8)
        assert plan.path == "split"
        out[gather] = (S.project(x, plan, index=ii), S.backproject(ys, plan, index=ii))
        plan.close()
    np.testing.assert_array_equal(out["1"][0], out["0"][0])
    assert relerr(out["1"][1], out["0"][1]) <= 1e-5
    G = O.Geometry(mumap, psfs, 4.8)
    assert relerr(out["1"][0], G.project(x, index=ii)) <= TOL
    assert relerr(out["1"][1], G.backproject(ys, index=ii)) <= TOL
