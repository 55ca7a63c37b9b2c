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


# nx, nz, kept px, pz: whole and partial tasks, single slices, wide and flat planes
SIZES = [(128, 80, 37, 37), (64, 64, 11, 11), (64, 40, 19, 19), (96, 48, 21, 21), (128, 128, 37, 37), (16, 12, 5, 3),
         (64, 1, 11, 1), (128, 1, 11, 1), (256, 200, 65, 65), (64, 90, 21, 21), (40, 37, 9, 9), (8, 5, 5, 5),
         (512, 96, 21, 21), (256, 17, 63, 3), (24, 230, 7, 65), (90, 53, 21, 17), (46, 80, 7, 7), (82, 73, 17, 17),
         (34, 9, 5, 3), (2, 1, 1, 1), (6, 3, 3, 3), (170, 1, 7, 1), (122, 100, 25, 25), (222, 150, 41, 41),
         (512, 230, 65, 65), (32, 160, 5, 5), (512, 250, 5, 5), (4, 256, 1, 65), (46, 37, 9, 33)]
X, NTH = 8, 640  # outputs of an x task; threads an SM's registers allow the pair-pass kernels
GEO = ("nzp", "L", "pad", "hx", "hz", "R0", "C0", "zpw", "xpw", "hs", "ts", "trow")
TILE = ("w", "tz", "ntile", "vst", "bst", "nxb", "nth", "occ", "ystep", "nxt", "smem")


@pytest.fixture(scope="module")
def named(tiling):
    keys = {"geometry": GEO, "k_zadj": TILE, "k_zfwd": TILE,
            "k_zs": ("tx", "zvst", "fz_nth", "fz_occ", "tz", "xbst", "fx_nth", "fx_occ", "fz_smem", "fx_smem"),
            "k_zrot_adj": ("tx", "ty", "S", "vb", "nth", "grid", "smem")}
    return lambda what, *a, **k: dict(zip(keys[what], tiling(what, *a, **k)))


def walk(tid, nth, inner, outer):
    """The units of a thread that a kernel deals by constant steps: unit u =
    outer index * inner + inner index."""
    d_out, d_in = divmod(nth, inner)
    o, i = divmod(tid, inner)
    got = []
    while o < outer:
        got.append(o * inner + i)
        o, i = o + d_out, i + d_in
        if i >= inner:
            o, i = o + 1, i - inner
    return got


def check_adjoint_tile(nx, nz, g, t):
    """Indexes of k_zadj inside its buffers."""
    W, tz, vst, bst, hx, hz, R0, C0 = (*(t[k] for k in ("w", "tz", "vst", "bst")), *(g[k] for k in ("hx", "hz", "R0", "C0")))
    assert W in (8, 16) and 32 <= t["nth"] <= NTH and t["nth"] % 32 == 0 and 1 <= t["occ"] <= NTH // t["nth"]
    assert tz % 2 == 0 and tz * t["ntile"] >= nz > tz * (t["ntile"] - 1)
    assert (vst // 2) % 2 == 1 and (bst // 2) % 2 == 1 and vst % 2 == bst % 2 == 0
    floats = 2 * (nx // 2 * vst + t["nxb"] * (tz // 2) * bst) + 3 * g["trow"]
    assert t["nxb"] in (1, 2) and 4 * floats <= t["smem"] <= OPTIN
    vlen = W * ((tz + W - 1) // W) + g["zpw"]
    assert vlen <= vst and R0 >= hz and C0 >= hx
    for tile in range(t["ntile"]):
        Z0 = tile * tz
        rows = min(tz, nz - Z0)
        zb = (rows + W - 1) // W
        assert W * (zb - 1) + g["zpw"] + W <= vlen  # z windows
        if Z0 == 0 and hz:
            assert R0 + hz - 1 < vlen  # the fold of the first row
        last = nz - 1 - Z0
        if last < W * zb:  # the fold of the last row
            assert R0 + last - (hz - 1) >= 0 and R0 + last < vlen
        # row pairs that the z pass stores are those that the x pass reads, inside XB and the T column
        pairs = {z0 // 2 + m for z0 in range(0, W * zb, W) for m in range(W // 2) if z0 + 2 * m < rows}
        assert pairs == set(range((rows + 1) // 2)) and max(pairs) < tz // 2 and Z0 + 2 * max(pairs) + 1 < g["nzp"]
    nxw = (nx + X - 1) // X
    assert C0 % 2 == 0 and C0 + nx <= bst and X * (nxw - 1) + g["xpw"] + X <= bst
    assert C0 + hx - 1 < bst and C0 + nx - hx >= 0
    # zdiv is exact below 2^20
    assert vlen * (nx // 2) + 8 * t["nth"] < 1 << 20 and (tz // 2) * nxw < 1 << 20


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
def test_adjoint_tile(named, nx, nz, px, pz):
    g, t = named("geometry", nx, nz, px, pz), named("k_zadj", nx, nz, px, pz)
    assert g["trow"] % 4 == 0 and g["hs"] % 8 == 0 and g["nzp"] % 16 == 0
    check_adjoint_tile(nx, nz, g, t)


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
def test_adjoint_tile_forms(named, nx, nz, px, pz):
    """Every form that the switches can ask for stays inside its buffers, and
    one that fits nowhere falls back on the rule's own."""
    g, own = named("geometry", nx, nz, px, pz), named("k_zadj", nx, nz, px, pz)
    met = set()
    for w in (0, 8, 16):
        for nxb in (0, 1, 2):
            for ntile in range(0, (nz + 1) // 2 + 1):
                t = named("k_zadj", nx, nz, px, pz, option=w + 256 * nxb + 65536 * ntile)
                check_adjoint_tile(nx, nz, g, t)
                if (w or t["w"], nxb or t["nxb"], ntile or t["ntile"]) == (t["w"], t["nxb"], t["ntile"]):
                    met.add((t["w"], t["nxb"], t["ntile"]))
                else:
                    assert t == own
    assert (own["w"], own["nxb"], own["ntile"]) in met
    if nx * nz <= 64 * 64:
        ceil = lambda a, b: -(-a // b)  # noqa: E731
        tiles = {nt for nt in range(1, (nz + 1) // 2 + 1) if nt == 1 or ceil(nz, 8 * ceil(ceil(nz, nt), 8)) == nt}
        assert met == {(w, nxb, nt) for w in (8, 16) for nxb in (1, 2) for nt in tiles}


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
@pytest.mark.parametrize("interp", [1, 2])
def test_forward_tile(named, nx, nz, px, pz, interp):
    g, t = named("geometry", nx, nz, px, pz), named("k_zfwd", nx, nz, px, pz, option=interp)
    if t["w"] == 0:  # the large-plane kernels
        assert nx * nz > 5000
        return
    vst, bst, nth = t["vst"], t["bst"], t["nth"]
    nzb, nz4, nxp, nzp2, nxw = (nz + 7) // 8, (nz + 3) // 4, nx // 2, (nz + 1) // 2, (nx + X - 1) // X
    assert nth % 32 == 0 and 1 <= t["occ"] <= NTH // nth and t["nxt"] in (1, 2)
    assert (vst // 2) % 2 == 1 and (bst // 2) % 2 == 1 and g["R0"] % 2 == g["C0"] % 2 == 0
    geo = (4 * 4 + 4) * nx if interp == 1 else 2 * 4 * nx + -(-nx // 4) * 4
    assert 4 * (2 * g["trow"] + geo + 2 * (nxp * vst + nzp2 * bst)) <= t["smem"] <= OPTIN
    assert t["nxt"] * nth >= nzp2 * nxw  # every x task has a thread slot
    for tid in (0, 1, nth // 2, nth - 1):
        assert walk(tid, nth, nz4, nxp) == list(range(tid, nxp * nz4, nth))
        assert walk(tid, nth, nxp, nzb) == list(range(tid, nxp * nzb, nth))
    # gather stores, windows, rows that the z pass stores
    assert g["R0"] + 4 * nz4 <= vst and 8 * (nzb - 1) + g["zpw"] + 8 <= vst
    assert g["C0"] + nx <= bst and X * (nxw - 1) + g["xpw"] + X <= bst
    assert max(z0 // 2 + m for z0 in range(0, 8 * nzb, 8) for m in range(4) if z0 + 2 * m < nz) == nzp2 - 1
    # the depth step visits every depth
    assert sorted(j * t["ystep"] % nx for j in range(nx)) == list(range(nx))


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
def test_large_plane_tiles(named, nx, nz, px, pz):
    g, t = named("geometry", nx, nz, px, pz), named("k_zs", nx, nz, px, pz)
    assert t["fz_nth"] > 0
    tx, tzp = t["tx"], t["tz"] // 2
    nzb, nrp, nxw, n2 = (nz + 7) // 8, (nz + 1) // 2, (nx + X - 1) // X, nx // 2
    # k_zs_fz: whole warps a plane, even tiles, gather stores and windows, shared memory
    assert t["fz_nth"] % 64 == 0 and t["fz_nth"] <= 320 and 1 <= t["fz_occ"] <= 960 // t["fz_nth"]
    assert tx % 2 == 0 and (nx - (nx - 1) // tx * tx) % 2 == 0
    assert g["R0"] + 4 * ((nz + 3) // 4) <= t["zvst"] and 8 * (nzb - 1) + g["zpw"] + 8 <= t["zvst"]
    assert 4 * (4 * (g["trow"] + 8 * tx + -(-tx // 4) * 4) + 2 * 2 * (tx // 2) * t["zvst"]) <= t["fz_smem"] <= OPTIN
    # k_zs_fx: a thread for every task, data columns and windows, shared memory, copies dealt once
    assert t["fx_nth"] % 32 == 0 and tzp * nxw <= t["fx_nth"] <= NTH and 1 <= t["fx_occ"] <= NTH // t["fx_nth"]
    assert 1 <= tzp <= nrp and g["C0"] + nx <= t["xbst"] and X * (nxw - 1) + g["xpw"] + X <= t["xbst"]
    assert 4 * 2 * (2 * tzp * t["xbst"] + g["trow"]) <= t["fx_smem"] <= OPTIN
    for tid in (0, 1, t["fx_nth"] - 1):
        assert walk(tid, t["fx_nth"], n2, tzp) == list(range(tid, tzp * n2, t["fx_nth"]))
    # the exchange buffer's planes fit its allocation (nzp values a column)
    assert 2 * nrp <= g["nzp"]


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
@pytest.mark.parametrize("nv", [1, 2, 15, 128, 700])
def test_gather_tile(named, nx, nz, px, pz, nv):
    g, t = named("geometry", nx, nz, px, pz), named("k_zrot_adj", nx, nz, px, pz, nv=nv)
    C, n4, nth = t["tx"] * t["ty"], g["nzp"] // 4, t["nth"]
    assert 1 <= t["S"] <= nv and nth <= 512 and nth % t["S"] == 0 and (nth // t["S"]) % 32 == 0
    gth = nth // t["S"]
    assert 2 * gth >= C * n4 and 1 <= t["vb"] and t["vb"] * C <= nth  # units and pairs have threads
    assert 2 * nth * 9 * 8 <= t["smem"] <= 512 * 2 * 9 * 8  # the lists; the limit that the setup asks for
    assert (t["S"] - 1) * 2 * gth * 16 <= t["smem"]  # the group sums in their place
    assert t["grid"] == -(-nx // t["tx"]) * -(-nx // t["ty"])
    slots = [s0 + b for s0 in range(0, nv, t["vb"]) for grp in range(t["S"])
             for b in range(grp, min(t["vb"], nv - s0), t["S"])]
    assert sorted(slots) == list(range(nv))  # the groups take every slot once
