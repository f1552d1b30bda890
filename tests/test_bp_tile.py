"""The back projector's staged views stay inside their shared-memory slots (CPU).

A CTA of `gf_bp_tile.cu` owns a block of columns (warp tiles of 4x8, two in y and
half its warps in x) and a run of slices.  Per view it copies the rows of the
radial bins that the block touches and the run can reach into a slot sized by
`tile_shape` (gf_plan.cpp), with the bin and row ranges taken from the block's
corner columns, and every lane with a voxel in the segment's range reads
ZR + 2 rows of two bins (and 64 mask bits) from its run's first row on.
Checked here with the kernel's float32 coordinates for every column: copies and
reads inside the slot, and rows that are used inside what was copied.
"""
import math

import numpy as np
import pytest

F = np.float32
TX, TY = 4, 8


def segments(geo):
    res, nzs, nrad, nang, span, nseg, pitch, diam, fov = geo
    vx = F(F(fov) / F(res))
    out, acc = [], 0
    for s in range(nseg):
        k = (s + 1) // 2
        zmin = 0 if s == 0 else (k - 1) * span + span // 2 + 1
        sgn = 0 if s == 0 else 1 - 2 * (s % 2)
        fz = F(float(F(vx * F(sgn * zmin))) / (float(F(diam)) / 2.0))
        out.append((zmin, nzs - 2 * zmin, acc + 2 * s, fz))
        acc += nzs - 2 * zmin
    return out


def tile_shape(geo, warps, zr, eb):
    """tile_shape's numbers for a given run length."""
    res, nzs, nrad, nang, span, nseg, pitch, diam, fov = geo
    vx = float(F(F(fov) / F(res)))
    fx = vx / (float(F(pitch)) / 2.0)
    diag = math.hypot(TX * (warps // 2) - 1, TY * 2 - 1)
    fzmax = max(abs(float(s[3])) for s in segments(geo))
    ve = 16 // eb
    nb = min(nrad, int(math.floor(diag * fx + 1e-3)) + 3)
    spread = int(math.floor(diag * fzmax + 1e-3)) + 1
    rows = min(nzs + 2, zr + spread + 2)
    words = ((rows + 2 * (ve - 1)) * eb + 3) // 4
    words += (12 - words % 8) % 8
    rs = words * 4 // eb
    mw = (rows + 62) // 32 + 2
    padf = (zr + ve - 1) // ve * ve
    return dict(nb=nb, rows=rows, rs=rs, mw=mw, ve=ve, padf=padf, elems=padf + nb * rs + zr + 2)


GEOS = [(128, 159, 128, 160, 3, 53, 1.6, 165.7758, 100.0), (128, 159, 147, 168, 11, 15, 1.63, 165.7758, 100.0),
        (64, 32, 64, 64, 3, 11, 1.6, 84.8772096, 51.2), (16, 15, 17, 8, 3, 5, 1.6, 20.7219750, 12.5),
        (20, 18, 24, 12, 5, 3, 1.63, 24.86637, 15.0), (16, 256, 16, 12, 3, 7, 1.6, 20.7219750, 12.5),
        (96, 96, 96, 96, 3, 31, 1.6, 127.3158, 76.8), (64, 100, 40, 32, 1, 41, 2.0, 60.0, 51.2),
        (32, 200, 20, 16, 2, 61, 2.0, 30.0, 25.6), (33, 47, 61, 20, 1, 21, 0.5, 40.0, 25.0)]


@pytest.mark.parametrize("geo", GEOS, ids=lambda g: f"{g[0]}x{g[1]}_{g[2]}x{g[3]}")
@pytest.mark.parametrize("warps,zr,eb", [(8, 12, 4), (8, 12, 2), (4, 12, 4), (4, 12, 2), (8, 8, 4), (8, 8, 2), (4, 8, 4), (4, 8, 2)])
def test_staged_views_fit_their_slots(geo, warps, zr, eb):
    res, nzs, nrad, nang, span, nseg, pitch, diam, fov = geo
    sh = tile_shape(geo, warps, zr, eb)
    ve, rs, padf = sh["ve"], sh["rs"], sh["padf"]
    resm, radm = F(F(res - 1) * F(0.5)), F(F(nrad - 1) * F(0.5))
    vx = F(F(fov) / F(res))
    fx = F(vx / F(float(F(pitch)) / 2.0))
    cx, cy = TX * (warps // 2), TY * 2
    gx = np.minimum(np.arange(-(-res // cx) * cx), res - 1).reshape(-1, cx)
    gy = np.minimum(np.arange(-(-res // cy) * cy), res - 1).reshape(-1, cy)
    # [block, column]
    ix = np.broadcast_to(gx[None, :, None, :], (gy.shape[0], gx.shape[0], cy, cx)).reshape(-1, cx * cy)
    iy = np.broadcast_to(gy[:, None, :, None], (gy.shape[0], gx.shape[0], cy, cx)).reshape(-1, cx * cy)
    xv, yv = ix.astype(F) - resm, iy.astype(F) - resm
    corners = [0, cx - 1, cx * (cy - 1), cx * cy - 1]
    for th in np.unique(np.linspace(0, nang - 1, 9).astype(int)):
        a = F(F(F(-F(th)) / F(nang)) * F(3.1415926)) + F(3.1415926)
        sn, cs = F(np.sin(float(a))), F(np.cos(float(a)))
        xrot = (xv * cs).astype(F) + (yv * sn).astype(F)
        yrot = (-xv * sn).astype(F) + (yv * cs).astype(F)
        x = (radm + (xrot * fx).astype(F)).astype(F) + F(0.5)
        i = np.floor(x - F(0.5)).astype(np.int64)
        i0, i1 = np.clip(i, 0, nrad - 1), np.clip(i + 1, 0, nrad - 1)
        bmin = i0[:, corners].min(1, keepdims=True)
        nb = i1[:, corners].max(1, keepdims=True) - bmin + 1
        assert (i0 >= bmin).all() and (i1 <= bmin + nb - 1).all()  # the corners bound every column
        assert nb.max() <= sh["nb"]
        for zmin, npl, blk, fz in segments(geo):
            nrow = npl + 2
            k = np.floor((yrot * fz).astype(F)).astype(np.int64) - (zmin - 1)
            kmin, kmax = k[:, corners].min(1, keepdims=True), k[:, corners].max(1, keepdims=True)
            assert (k >= kmin).all() and (k <= kmax).all()
            for z0 in range(0, nzs, zr):
                nv = min(zr, nzs - z0)
                active = ((z0 + kmax + nv - 1 >= 0) & (z0 + kmin <= nrow - 2))[:, 0]
                j0 = z0 + k
                has = np.minimum(nv, nrow - 1 - j0) > np.maximum(0, -j0)
                assert not (has & ~active[:, None]).any()
                if not active.any():
                    continue
                ra = np.maximum(0, z0 + kmin)
                rb = np.minimum(nrow - 1, z0 + zr + kmax + 1)
                assert (rb >= ra)[active].all()
                base = (blk + ra) // ve * ve
                nvec = (blk + rb - base) // ve + 1
                assert (nvec[active] * ve <= rs).all()
                off = blk - base + padf
                wb = (blk + ra) // 32 - 1
                words = (blk + rb) // 32 - wb
                assert (words[active] + 2 <= sh["mw"]).all()
                if not has.any():
                    continue
                for b in (i0, i1):
                    at = ((b - bmin) * rs + off + j0)[has]
                    assert at.min() >= 0 and at.max() + zr + 1 < sh["elems"]
                # the rows of voxels in the range, and one more, were copied
                lo = np.maximum(j0, 0)
                hi = np.minimum(j0 + nv + 1, nrow - 1)
                assert (lo >= ra)[has].all() and (hi <= rb)[has].all()
                q = (blk - 32 * wb + j0)[has]
                assert q.min() >= 0 and (q // 32).max() + 1 < sh["mw"]


@pytest.mark.parametrize("zr", [8, 12, 20])
def test_run_fraction_is_every_voxels(zr):
    """Where a run's n = iz + floor(t) stays in one power-of-two interval (and
    n + zr too), the per-voxel form's fraction is that of its first voxel."""
    rs = np.random.RandomState(zr)
    t = (rs.uniform(-60, 60, 500000) * 10.0 ** rs.uniform(-7, 0, 500000)).astype(F)
    t[:1000] = 0
    z0 = rs.randint(0, 500, t.size)
    ft = np.floor(t)
    n0 = z0 + ft.astype(np.int64)
    one = (n0 > 0) & (np.frexp(np.maximum(n0, 1))[1] == np.frexp(np.maximum(n0 + zr, 1))[1])
    one &= ~((t - ft).astype(F) > F(0.9999))  # such lanes go voxel by voxel

    def fraction(i):
        fiz = (z0 + i).astype(F)
        return ((fiz + t + F(0.5)) - F(0.5)) - (fiz + ft)

    first = fraction(0)
    assert first.dtype == F and one.sum() > 100000
    for i in range(1, zr):
        assert np.array_equal(fraction(i)[one], first[one])
