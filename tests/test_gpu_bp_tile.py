"""GPU parity of the column-tile back projector (gf_bp_tile.cu), through the C-ABI.

Geometries large enough to take it (bp_uses_tiles in gf_plan.cpp), with sizes
off its blocks of 16x16 columns and runs of 12 slices, few views (the oracle
runs on the CPU).  Per-voxel form: the oracle's sums bit for bit, masked bins,
infinities and NaN included.  Per-view form: its own definition in float32
(the oracle has the per-voxel form only, and where a ratio of 0 meets a gap the
two count different samples), to 1e-6: the sums of at most 300 samples, each
rounded once more than here where a fused multiply-add rounds through float64.
"""
import ctypes

import numpy as np
import pytest

import gfo
from test_gpu_parity import IMG_TOL, gf, rel  # noqa: F401

pytestmark = pytest.mark.gpu

GEOS = [
    (73, 75, 70, 7, 3, 9, 1.6, 95.8, 58.4),    # 25 blocks x 7 runs, remainders in x, y and z
    (80, 72, 81, 6, 1, 21, 1.5, 60.0, 64.0),   # whole blocks and runs; steep segments
    (131, 27, 90, 5, 5, 3, 2.1, 150.0, 101.0),  # wide and flat: 81 blocks, 3 runs, the last of 3 slices
    (66, 256, 61, 4, 7, 35, 1.6, 90.0, 54.0),  # the deepest image, segments past the 32nd
    (66, 160, 61, 3, 1, 71, 1.6, 90.0, 54.0),  # segments past the 64th
    (130, 61, 90, 5, 3, 11, 1.8, 150.0, 101.0),  # runs of 12, remainders in x, y and z
    (102, 66, 81, 6, 1, 21, 1.6, 100.0, 72.0),   # runs of 8, remainders in x, y and z
]


def ratio_and_mask(o, geo, seed, gaps):
    rs = np.random.RandomState(seed)
    corr = rs.uniform(0.0, 3.0, o.ndata).astype(np.float32)
    corr[rs.uniform(size=o.ndata) < 0.01] = -1000.0
    corr[rs.uniform(size=o.ndata) < 0.3] = 0.0
    calib = np.where(rs.uniform(size=o.ndata) < gaps, -1000.0, 1.0).astype(np.float32)
    calib.reshape(-1, geo[2])[:, [0, -1]] = -1000.0  # the outermost bins
    return corr, calib


def per_view(o, geo, corr, calib, nsub, subset):
    """GF_BP_PER_VIEW of one subset: one axial fraction per (column, view)."""
    F, m = np.float32, ctypes.CDLL("libm.so.6")
    m.sinf.restype = m.cosf.restype = ctypes.c_float
    m.sinf.argtypes = m.cosf.argtypes = [ctypes.c_float]
    res, nzs, nrad, nang, span, nseg, pitch, diam, fov = geo
    corr, calib = corr.reshape(-1, nang, nrad), calib.reshape(-1, nang, nrad)
    vx = F(F(fov) / F(res))
    fx = F(vx / F(float(F(pitch)) / 2.0))
    resm, radm = F(F(res - 1) * F(0.5)), F(F(nrad - 1) * F(0.5))
    xv = np.tile(np.arange(res, dtype=F) - resm, res)
    yv = np.repeat(np.arange(res, dtype=F) - resm, res)

    def lerp(a, b, w):
        return (w.astype(np.float64) * (b - a).astype(F) + a).astype(F)

    num, den = np.zeros((nzs, res * res), F), np.zeros((nzs, res * res), F)
    acc = 0
    for s in range(nseg):
        zmin = 0 if s == 0 else ((s + 1) // 2 - 1) * span + span // 2 + 1
        fz = F(float(F(vx * F((0 if s == 0 else 1 - 2 * (s % 2)) * zmin))) / (float(F(diam)) / 2.0))
        n = nzs - 2 * zmin
        for t in range(subset, nang, nsub):
            ang = F(F(-F(t) / F(nang)) * F(3.1415926)) + F(3.1415926)
            sn, cs = F(m.sinf(ang)), F(m.cosf(ang))
            xrot, yrot = xv * cs + yv * sn, -xv * sn + yv * cs
            xb = ((radm + xrot * fx) + F(0.5)) - F(0.5)
            fl = np.floor(xb)
            i0 = np.clip(fl.astype(int), 0, nrad - 1)
            i1 = np.clip(fl.astype(int) + 1, 0, nrad - 1)
            tt = yrot * fz
            be = (tt - np.floor(tt))[None, :]
            rows = []
            for a in (corr, calib):
                v = np.full((n + 2, nrad), F(-1000.0))
                v[1:-1] = a[acc:acc + n, t]
                if s == 0:
                    v[0], v[-1] = v[1], v[-2]
                rows.append(lerp(v[:, i0], v[:, i1], (xb - fl)[None, :]))
            j = np.arange(nzs)[:, None] + np.floor(tt).astype(int)[None, :] - (zmin - 1)
            inside = (j >= 0) & (j <= n)
            j = np.clip(j, 0, n)
            c = np.arange(res * res)[None, :]
            vr, vc = (lerp(r[j, c], r[j + 1, c], be) for r in rows)
            ok = inside & ~((vc < 0) | (vr < 0))
            num += np.where(ok, vr, F(0))
            den += np.where(ok, vc, F(0))
        acc += n
    return num.ravel(), den.ravel()


def project_back(gf_, ctx, corr, calib, subset, form):
    ctx.set_bp_form(form)
    n, d = ctx.array(ctx.nvox), ctx.array(ctx.nvox)
    ctx.back_project(ctx.put(corr), ctx.put(calib), subset, n, d)
    return n.download(), d.download()


@pytest.mark.parametrize("geo", GEOS, ids=lambda g: f"{g[0]}x{g[1]}")
@pytest.mark.parametrize("gaps", [0.0, 0.03])
def test_tiles_match_oracle(gf, geo, gaps):  # noqa: F811
    o = gfo.Oracle(geo)
    ctx = gf.Context(gf.Geometry(*geo), nsub=2)
    corr, calib = ratio_and_mask(o, geo, 5, gaps)
    wn, wd = o.bp(corr, calib, 2, 1)
    vn, vd = per_view(o, geo, corr, calib, 2, 1)
    for warps in (8, 4):
        ctx.set_tile_shapes(33, 16, warps)
        n, d = project_back(gf, ctx, corr, calib, 1, "voxel")
        assert np.array_equal(n, wn) and np.array_equal(d, wd)
        n, d = project_back(gf, ctx, corr, calib, 1, "view")
        assert rel(n, vn) < 1e-6 and rel(d, vd) < 1e-6


def test_masks_of_other_values_match_oracle(gf):  # noqa: F811
    geo = GEOS[-1]
    o = gfo.Oracle(geo)
    ctx = gf.Context(gf.Geometry(*geo), nsub=2)
    corr, calib = ratio_and_mask(o, geo, 6, 0.02)
    rs = np.random.RandomState(7)
    calib = np.where(calib > 0, rs.uniform(0.0, 2.0, o.ndata), calib).astype(np.float32)
    wn, wd = o.bp(corr, calib, 2, 0)
    n, d = project_back(gf, ctx, corr, calib, 0, "voxel")
    assert np.array_equal(n, wn) and np.array_equal(d, wd)
    # and a mask of 1 and -1000 after it on the same context
    corr, calib = ratio_and_mask(o, geo, 8, 0.02)
    wn, wd = o.bp(corr, calib, 2, 0)
    n, d = project_back(gf, ctx, corr, calib, 0, "voxel")
    assert np.array_equal(n, wn) and np.array_equal(d, wd)


def test_infinities_and_nan_match_oracle(gf):  # noqa: F811
    geo = GEOS[-1]
    o = gfo.Oracle(geo)
    ctx = gf.Context(gf.Geometry(*geo), nsub=2)
    corr, calib = ratio_and_mask(o, geo, 9, 0.02)
    rs = np.random.RandomState(10)
    for v in (np.inf, -np.inf, np.nan):
        corr[rs.randint(0, o.ndata, 40)] = v
    wn, wd = o.bp(corr, calib, 2, 1)
    assert np.isnan(wn).any()
    n, d = project_back(gf, ctx, corr, calib, 1, "voxel")
    assert np.array_equal(n, wn, equal_nan=True) and np.array_equal(d, wd)


@pytest.mark.parametrize("mode,storage,tol", [(1, "f32", IMG_TOL), (3, "f32", IMG_TOL), (1, "f16", IMG_TOL),
                                              (1, "bf16", 10 * IMG_TOL)])
@pytest.mark.parametrize("geo", [(72, 72, 72, 8, 3, 5, 1.6, 95.48, 57.6), GEOS[-1]], ids=["72", "102"])
def test_reconstruction_over_tiles_matches_oracle(gf, geo, mode, storage, tol):  # noqa: F811
    """16-bit ratios round by 2^-11 (2^-8 in BF16) per sample, 2 subsets of one iteration."""
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(11)
    nd = o.ndata
    dsino = np.concatenate([rs.poisson(30.0, nd), rs.uniform(0, 0.2, nd)]).astype(np.float32)
    tsino = np.concatenate([rs.poisson(3.0, nd), np.zeros(nd)]).astype(np.float32)
    norm = rs.uniform(0.8, 1.2, nd).astype(np.float32)
    norm[rs.uniform(size=nd) < 0.01] = 0.0
    ev = rs.randint(1, nd + 1, size=(nd // 4, 2)).astype(np.int32)
    kw = dict(dsino=dsino, norm=norm) if mode == 1 else dict(dsino=dsino, tsino=tsino, norm=norm, ev=ev)
    want = o.recon(mode, nsub=2, niter=1, **kw)
    ctx = gf.Context(gf.Geometry(*geo), nsub=2)
    r = gf.Recon(ctx, mode, niter=1, storage=storage)
    if mode == 3:
        kw["events"] = kw.pop("ev")
    r.load(**kw)
    r.iterate(1)
    assert rel(r.image(0), want["img_d"]) < tol
    if mode == 3:
        assert rel(r.image(1), want["img_t"]) < tol
