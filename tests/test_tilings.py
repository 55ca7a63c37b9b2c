"""Launch shapes of the library's own tiling rules (spect_selftest_tiling runs
the functions of csrc/zpath_api.h that plan creation calls; no GPU needed)."""
import ctypes

import pytest

OPTIN, SMS = 232448, 148


@pytest.fixture(scope="module")
def tiling(S):
    def call(what, nx, nz, px=1, pz=1, nv=1, option=0, sms=SMS, optin=OPTIN):
        args = (ctypes.c_int * 8)(nx, nz, px, pz, nv, option, sms, optin)
        out = (ctypes.c_longlong * 12)()
        S._native.check(S._native.lib().spect_selftest_tiling(what.encode(), args, out))
        return list(out)

    return call


@pytest.mark.parametrize("nx,nz,nview", [(500, 1, 720), (440, 1, 700), (512, 1, 512), (512, 1, 10000), (512, 2, 900),
                                         (256, 1, 5000), (2, 1, 10 ** 8), (128, 80, 120), (512, 256, 720), (2, 1, 4)])
@pytest.mark.parametrize("option", [0, 1, 2])
def test_group_of_views(tiling, nx, nz, nview, option):
    """The gather adjoint packs a hit count above the 27 bits of a T column
    number: a group's columns and the zero column behind them have to fit.  The
    other bounds: the plan's views, one view at least, about 1 GiB of planes."""
    g = tiling("group", nx, nz, nv=nview, option=option)[0]
    assert 1 <= g <= nview
    slot = nx * nx * (nz if option < 2 else -(-nz // 16) * 16)
    assert g == 1 or g * slot * 4 <= 1 << 30
    if option:
        assert g * nx * nx <= (1 << 27) - 1
    # no smaller than those bounds ask for
    most = min(nview, max(1, (1 << 30) // (4 * slot)))
    if option:
        most = min(most, ((1 << 27) - 1) // (nx * nx))
    assert g == most
