"""The pair-pass kernels (csrc/zpath.cuh) checked on the CPU: the index
arithmetic of their tiles stays inside their buffers, and their walk over
(slot, row tile, depth) planes covers every plane once.

Mirrors of zadj_tile and ztable_floats (csrc/zpath_api.h); the geometry is
zgeom of test_fused_math.
"""
import math

import pytest

from test_fused_math import zgeom, zround

OPTIN = 232448
NTH = 640
X = 8  # outputs of an x-pass task


def zstride2(v):
    r = zround(v, 2)
    return r if (r // 2) % 2 == 1 else r + 2


def zadj_tile(g, optin=OPTIN):
    nx, nz = g["nx"], g["nz"]
    trow = 2 * g["hs"] + g["ts"] + 4
    best, bc = None, 0.0
    for w in (16, 8):
        for nt in range(1, (nz + 1) // 2 + 1):
            t = dict(w=w, tz=zround((nz + nt - 1) // nt, 8 if nt > 1 else 2))
            t["ntile"] = (nz + t["tz"] - 1) // t["tz"]
            if t["ntile"] != nt:
                continue
            t["vst"] = zstride2(w * ((t["tz"] + w - 1) // w) + g["zpw"])
            t["bst"] = zstride2(X * ((nx + X - 1) // X) + g["xpw"])
            zt = nx // 2 * ((t["tz"] + w - 1) // w)
            xt = t["tz"] // 2 * ((nx + X - 1) // X)
            most = zt if w == 16 else max(zt, xt)
            rounds = (most + NTH - 1) // NTH
            t["nth"] = zround((most + rounds - 1) // rounds, 32)
            for nxb in (1, 2):
                smem = 4 * (2 * (nx // 2 * t["vst"] + nxb * (t["tz"] // 2) * t["bst"]) + 3 * trow)
                if smem > optin:
                    continue
                occ = min((optin + 1024) // (smem + 1024), NTH // t["nth"], 16)
                if nxb > 1 and occ > 1:
                    continue
                warps = occ * t["nth"] / 32
                rz, rx = math.ceil(zt / t["nth"]), math.ceil(xt / t["nth"])
                c = t["ntile"] * t["nth"] * (rz * w * (1.15 if w == 8 else 1.0) + rx * X * 1.15)
                c *= max(1.0, 16 / warps) * (1.0 if occ > 1 or nxb > 1 else 1.25)
                if best is None or c < bc:
                    best, bc = dict(t, nxb=nxb, smem=smem, occ=occ), c
    return best


SIZES = [(128, 80, 37, 37), (64, 64, 11, 11), (64, 40, 19, 19), (96, 48, 21, 21), (128, 128, 37, 37), (16, 12, 5, 3),
         (64, 1, 11, 1), (128, 1, 11, 1), (256, 200, 65, 65), (64, 90, 21, 21), (40, 37, 9, 9), (8, 5, 5, 5),
         (512, 96, 21, 21), (256, 17, 63, 3), (24, 230, 7, 65), (90, 53, 21, 17), (46, 80, 7, 7), (82, 73, 17, 17),
         (34, 9, 5, 3), (2, 1, 1, 1), (6, 3, 3, 3), (170, 1, 7, 1), (122, 100, 25, 25)]


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
def test_adjoint_tile_bounds(nx, nz, px, pz):
    g = zgeom(nx, nz, px, pz)
    t = zadj_tile(g)
    assert t is not None and t["smem"] <= OPTIN and 32 <= t["nth"] <= NTH and t["occ"] * t["nth"] <= NTH
    W, tz, vst, bst = t["w"], t["tz"], t["vst"], t["bst"]
    assert tz % 2 == 0 and tz * t["ntile"] >= nz > tz * (t["ntile"] - 1)
    assert vst % 2 == 0 and (vst // 2) % 2 == 1 and bst % 2 == 0 and (bst // 2) % 2 == 1
    R0, C0, hz, hx, nzp = g["R0"], g["C0"], g["hz"], g["hx"], zround(nz, 16)
    vlen = W * ((tz + W - 1) // W) + g["zpw"]
    assert vlen <= vst and R0 >= hz and C0 >= hx
    for tile in range(t["ntile"]):
        Z0 = tile * tz
        rows = min(tz, nz - Z0)
        zb = (rows + W - 1) // W
        # z windows and folds stay inside the loaded line
        assert W * (zb - 1) + g["zpw"] + W <= vlen
        if Z0 == 0 and hz:
            assert R0 + hz - 1 < vlen
        last = nz - 1 - Z0
        if last < W * zb:
            assert 0 <= R0 + last - (hz - 1) and R0 + last < vlen
        # row pairs stored by the z pass are those the x pass reads, inside XB and the T column
        pairs = {(z0 + 2 * m) // 2 for z0 in range(0, W * zb, W) for m in range(W // 2) if z0 + 2 * m < rows}
        assert pairs == set(range((rows + 1) // 2)) and max(pairs) < tz // 2
        assert Z0 + 2 * max(pairs) + 1 < nzp
    # x windows, data columns and folds stay inside a row
    nxw = (nx + X - 1) // X
    assert C0 % 2 == 0 and C0 + nx <= bst and X * (nxw - 1) + g["xpw"] + X <= bst
    assert C0 + hx - 1 < bst and C0 + nx - 1 - (hx - 1) >= 0
    assert g["hs"] % 8 == 0 and (2 * g["hs"] + g["ts"] + 4) % 4 == 0


@pytest.mark.parametrize("n,grid", [(1920, 296), (80 * 128, 740), (7, 7), (5, 148), (1, 1), (8 * 5 * 256, 148)])
def test_plane_walk_covers_once(n, grid):
    spans = [(b * n // grid, (b + 1) * n // grid) for b in range(grid)]
    assert [q for a, b in spans for q in range(a, b)] == list(range(n))
    assert max(b - a for a, b in spans) - min(b - a for a, b in spans) <= 1


@pytest.mark.parametrize("ny", [2, 4, 8, 40, 64, 96, 128, 256, 512, 90, 46])
def test_depth_step_visits_every_depth(ny):
    s = max(1, int(0.618 * ny))
    while math.gcd(s, ny) != 1:
        s += 1
    assert s < ny or ny == 2 and s == 1
    y, seen = 0, []
    for _ in range(ny):
        seen.append(y)
        y += s
        if y >= ny:
            y -= ny
    assert sorted(seen) == list(range(ny))


def zfwd_tile(g, optin=OPTIN):
    """Mirror of zfwd_tile (csrc/zpath_api.h): None where the plane does not fit."""
    nx, nz = g["nx"], g["nz"]
    nxw, nzb = (nx + 7) // 8, (nz + 7) // 8
    xt = (nz + 1) // 2 * nxw
    if xt > 2 * NTH:
        return None
    t = dict(vst=zstride2(8 * nzb + g["zpw"]), bst=zstride2(8 * nxw + g["xpw"]))
    trow = 2 * g["hs"] + g["ts"] + 4
    t["smem"] = 4 * (2 * trow + 8 * nx + zround(nx, 4) + 2 * (nx // 2 * t["vst"] + (nz + 1) // 2 * t["bst"]))
    if t["smem"] > optin:
        return None
    t["nxt"] = 1 if xt <= NTH else 2
    zh, gq = (nx // 2 * nzb + 1) // 2, (nx // 2 * ((nz + 3) // 4) + 3) // 4
    t["nth"] = min(NTH, zround(max((xt + t["nxt"] - 1) // t["nxt"], zh, gq), 32))
    return t


@pytest.mark.parametrize("nx,nz,px,pz", SIZES)
def test_forward_tile_bounds(nx, nz, px, pz):
    g = zgeom(nx, nz, px, pz)
    t = zfwd_tile(g)
    if t is None:  # the large-plane kernels
        assert nx * nz > 8000
        return
    R0, C0, hz, hx, vst, bst, nth = g["R0"], g["C0"], g["hz"], g["hx"], t["vst"], t["bst"], t["nth"]
    nzb, nz4, nxp, nzp2, nxw = (nz + 7) // 8, (nz + 3) // 4, nx // 2, (nz + 1) // 2, (nx + 7) // 8
    assert (vst // 2) % 2 == 1 and (bst // 2) % 2 == 1 and R0 % 2 == 0 and C0 % 2 == 0
    # every x task has a thread slot; the z tasks and gather units are walked by constant steps
    assert t["nxt"] * nth >= nzp2 * nxw
    for tid in (0, 1, nth // 2, nth - 1):
        dq, dr = divmod(nth, nz4)
        xp, z4 = divmod(tid, nz4)
        got = []
        while xp < nxp:
            got.append(xp * nz4 + z4)
            xp, z4 = xp + dq, z4 + dr
            if z4 >= nz4:
                xp, z4 = xp + 1, z4 - nz4
        assert got == list(range(tid, nxp * nz4, nth))
        dq, dr = divmod(nth, nxp)
        zb, xp = divmod(tid, nxp)
        got = []
        while zb < nzb:
            got.append(zb * nxp + xp)
            zb, xp = zb + dq, xp + dr
            if xp >= nxp:
                zb, xp = zb + 1, xp - nxp
        assert got == list(range(tid, nxp * nzb, nth))
    # lines: gather stores, windows, clamped edges; rows stored by the z pass
    assert R0 + 4 * nz4 <= vst and 8 * (nzb - 1) + g["zpw"] + 8 <= vst
    assert C0 + nx <= bst and 8 * (nxw - 1) + g["xpw"] + 8 <= bst
    assert max(z0 // 2 + m for z0 in range(0, 8 * nzb, 8) for m in range(4) if z0 + 2 * m < nz) == nzp2 - 1


@pytest.mark.parametrize("nv,ny,grid", [(15, 128, 148), (8, 256, 296), (3, 40, 60), (1, 64, 31), (120, 128, 148),
                                        (2, 8, 8), (1, 2, 1)])
def test_partial_views_of_the_forward_walk(nv, ny, grid):
    """Partial view block + slot is unique, a slot's partials are consecutive
    (zblock_of), and they cover its planes once, in order."""
    n = nv * ny

    def block_of(q):
        return ((q + 1) * grid - 1) // n

    seen = {}
    for b in range(grid):
        for q in range(b * n // grid, (b + 1) * n // grid):
            assert block_of(q) == b
            seen.setdefault((b, q // ny), []).append(q % ny)
    ids = [b + s for b, s in seen]
    assert len(set(ids)) == len(ids) and max(ids) < grid + nv
    for s in range(nv):
        b0, b1 = block_of(s * ny), block_of((s + 1) * ny - 1)
        assert sum((seen[(b, s)] for b in range(b0, b1 + 1)), []) == list(range(ny))


def zrot_tile(g, nv, sms=148):
    """Mirror of zrot_tile (csrc/zpath_api.h)."""
    n4 = zround(g["nz"], 16) // 4
    C = 16 if n4 <= 40 else 8
    tx, ty = 4, C // 4
    grid = -(-g["nx"] // tx) * -(-g["nx"] // ty)
    gth = zround((C * n4 + 1) // 2, 32)
    S = min((s for s in range(1, min(nv, 512 // gth) + 1)),
            key=lambda s: -(-grid // (sms * (1024 // (s * gth)))) / s * (1 + 0.15 * (s - 1)))
    return dict(C=C, tx=tx, ty=ty, grid=grid, gth=gth, S=S, nth=S * gth, vb=S * gth // C, n4=n4)


@pytest.mark.parametrize("nx,nz,px,pz", SIZES + [(90, 53, 5, 5), (32, 160, 5, 5), (512, 250, 5, 5)])
@pytest.mark.parametrize("nv", [1, 2, 15, 128])
def test_gather_adjoint_tile(nx, nz, px, pz, nv):
    g = zgeom(nx, nz, px, pz)
    t = zrot_tile(g, nv)
    assert t["nth"] <= 512 and t["vb"] >= 1 and t["vb"] * t["C"] <= t["nth"]
    # every unit of a tile has a thread, the group sums fit in the lists' memory
    assert 2 * t["gth"] >= t["C"] * t["n4"]
    assert (t["S"] - 1) * 2 * t["gth"] * 16 <= t["nth"] * 2 * 9 * 8
    # the groups take every slot of a batch once
    slots = []
    for s0 in range(0, nv, t["vb"]):
        nb = min(t["vb"], nv - s0)
        for grp in range(t["S"]):
            slots += [s0 + b for b in range(grp, nb, t["S"])]
    assert sorted(slots) == list(range(nv))
    # tiles cover the image
    assert -(-nx // t["tx"]) * t["tx"] >= nx and -(-nx // t["ty"]) * t["ty"] >= nx


@pytest.mark.parametrize("nx,nz,px,pz", SIZES + [(222, 150, 41, 41), (254, 199, 65, 65), (512, 230, 65, 65)])
def test_large_plane_forward_tiles(nx, nz, px, pz):
    """Mirror of zs_tiles (csrc/zpath_api.h): the indexes of k_zs_fz and
    k_zs_fx stay inside their buffers, and every task has a thread."""
    g = zgeom(nx, nz, px, pz)
    trow = 2 * g["hs"] + g["ts"] + 4
    nzb, nrp, nxw = (nz + 7) // 8, (nz + 1) // 2, (nx + 7) // 8
    tmax = min(32, 2 * (320 // nzb))
    ntile = -(-nx // tmax)
    tx = min(nx, zround(-(-nx // ntile), 4))
    zvst, xbst = zstride2(8 * nzb + g["zpw"]), zstride2(8 * nxw + g["xpw"])
    tzp = min(max(1, 320 // nxw), nrp)
    fz, fx = 4 * (4 * (trow + 8 * tx + zround(tx, 4)) + 2 * tx * zvst), 4 * 2 * (2 * tzp * xbst + trow)
    assert fz <= OPTIN and fx <= OPTIN and zround(tzp * nxw, 32) <= NTH
    assert min(320, 2 * zround((tx // 2 * nzb + 1) // 2, 32)) % 64 == 0  # whole warps a plane
    # k_zs_fz: gather stores, windows; the last tile has an even number of columns
    assert tx % 2 == 0 and (nx - (nx - 1) // tx * tx) % 2 == 0
    assert g["R0"] + 4 * ((nz + 3) // 4) <= zvst and 8 * (nzb - 1) + g["zpw"] + 8 <= zvst
    # rows it stores are the row pairs k_zs_fx reads
    assert {(z0 + 2 * m) // 2 for z0 in range(0, 8 * nzb, 8) for m in range(4) if z0 + 2 * m < nz} == set(range(nrp))
    # k_zs_fx: data columns and windows
    assert g["C0"] + nx <= xbst and 8 * (nxw - 1) + g["xpw"] + 8 <= xbst
    # planes of the exchange buffer fit its allocation (nzp values a column)
    assert 2 * nrp * nx <= zround(nz, 16) * nx
    n2, nth = nx // 2, zround(tzp * nxw, 32)
    for tid in (0, 1, nth - 1):
        dr, dc = divmod(nth, n2)
        r, c = divmod(tid, n2)
        got = []
        while r < tzp:
            got.append(r * n2 + c)
            r, c = r + dr, c + dc
            if c >= n2:
                r, c = r + 1, c - n2
        assert got == list(range(tid, tzp * n2, nth))
