"""GPU checks of the back projector's routes, each with its route asserted.

Column tiles in runs of 8 and of 12 slices, at sizes off their 16x16 columns and
their runs, at whole ones, steep and flat: the per-voxel form against the oracle
bit for bit, and both forms against one warp per column bit for bit (a mask value
that is neither 1 nor -1000, in a bin that no column touches, sends the same call
there).  Reconstructions over 12-slice runs against the oracle; frames whose runs
are 8 slices alone and 12 in a group, and pairs of deep columns, against frames
alone bit for bit.
"""
import numpy as np
import pytest

import gfo
from test_gpu_bp_tile import project_back, ratio_and_mask
from test_gpu_parity import IMG_TOL, gf, rel  # noqa: F401

pytestmark = pytest.mark.gpu

TILES = [  # slices of a run, geometry
    (12, (109, 83, 159, 5, 1, 21, 1.6, 140.0, 87.2)),   # remainders in x, y and z
    (12, (112, 84, 163, 4, 3, 11, 1.6, 150.0, 89.6)),   # whole blocks and runs
    (12, (112, 72, 163, 4, 1, 21, 1.6, 40.0, 89.6)),    # steep: a block spans many rows
    (12, (200, 27, 289, 5, 1, 9, 1.6, 260.0, 160.0)),   # flat: three runs, the last of 3 slices
    (8, (93, 83, 137, 4, 1, 31, 1.6, 120.0, 74.4)),     # remainders in x, y and z
    (8, (80, 112, 117, 4, 1, 35, 1.6, 100.0, 64.0)),    # whole blocks and runs
    (8, (80, 109, 117, 4, 1, 43, 1.6, 30.0, 64.0)),     # steep
]


@pytest.mark.parametrize("slices,geo", TILES, ids=lambda g: f"{g[0]}x{g[1]}" if isinstance(g, tuple) else f"run{g}")
@pytest.mark.parametrize("gaps", [0.0, 0.03])
def test_tiles_match_oracle_and_columns(gf, slices, geo, gaps):  # noqa: F811
    g = gf.Geometry(*geo)
    assert gf.bp_run(g, 2) == slices
    assert (g.nrad - 1) / 2 - (g.res - 1) / 2 * 2 ** 0.5 * (g.fov / g.res) / (g.pitch / 2) > 1.5  # spare outermost bins
    o = gfo.Oracle(geo)
    ctx = gf.Context(g, nsub=2)
    corr, calib = ratio_and_mask(o, geo, 15, gaps)
    other = calib.reshape(-1, g.nang, g.nrad).copy()
    other[:, :, 0] = 0.5
    wn, wd = o.bp(corr, calib, 2, 1)
    for form in ("voxel", "view"):
        tn, td = project_back(gf, ctx, corr, calib, 1, form)
        if form == "voxel":
            assert np.array_equal(tn, wn) and np.array_equal(td, wd)
        cn, cd = project_back(gf, ctx, corr, other.ravel(), 1, form)
        assert np.array_equal(tn, cn) and np.array_equal(td, cd)


def counts(rs, nd):
    dsino = np.concatenate([rs.poisson(30.0, nd), rs.uniform(0, 0.2, nd)]).astype(np.float32)
    norm = rs.uniform(0.8, 1.2, nd).astype(np.float32)
    norm[rs.uniform(size=nd) < 0.01] = 0.0
    return dsino, norm


@pytest.mark.parametrize("mode,storage,tol", [(1, "f32", IMG_TOL), (3, "f32", IMG_TOL), (1, "f16", IMG_TOL),
                                              (1, "bf16", 10 * IMG_TOL)])
def test_reconstruction_over_twelve_slice_runs_matches_oracle(gf, mode, storage, tol):  # noqa: F811
    """16-bit ratios round by 2^-11 (2^-8 in BF16) per sample, 2 subsets of one iteration."""
    geo = (104, 104, 80, 6, 3, 9, 1.6, 130.0, 83.2)
    assert gf.bp_run(gf.Geometry(*geo), 2) == 12
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(11)
    nd = o.ndata
    dsino, norm = counts(rs, nd)
    kw = dict(dsino=dsino, norm=norm)
    ev = rs.randint(1, nd + 1, size=(nd // 4, 2)).astype(np.int32)
    if mode == 3:
        kw["tsino"] = np.concatenate([rs.poisson(3.0, nd), np.zeros(nd)]).astype(np.float32)
    want = o.recon(mode, nsub=2, niter=1, **kw, **({"ev": ev} if mode == 3 else {}))
    r = gf.Recon(gf.Context(gf.Geometry(*geo), nsub=2), mode, niter=1, storage=storage)
    r.load(**kw, **({"events": ev} if mode == 3 else {}))
    r.iterate(1)
    assert rel(r.image(0), want["img_d"]) < tol
    if mode == 3:
        assert rel(r.image(1), want["img_t"]) < tol


def frames(gf, geo, n, storage, nsub=2):  # noqa: F811
    recs = [gf.Recon(gf.Context(gf.Geometry(*geo), nsub=nsub), 1, niter=1, storage=storage) for _ in range(n)]
    norm = counts(np.random.RandomState(0), recs[0].ctx.ndata)[1]
    for k, r in enumerate(recs):
        r.load(dsino=counts(np.random.RandomState(k), r.ctx.ndata)[0], norm=norm)
    return recs


def fused_equal_alone(gf, geo, n, storage):  # noqa: F811
    recs = frames(gf, geo, n, storage)
    b = gf.Batch(recs)
    b.set_fused(True)
    groups = b.groups()
    b.iterate(1)
    b.sync()
    for r, a in zip(recs, frames(gf, geo, n, storage)):
        a.iterate(1)
        assert np.array_equal(r.image(0), a.image(0))
    return groups


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_fused_frames_of_other_run_length_equal_frames_alone(gf, storage):  # noqa: F811
    geo = (80, 110, 80, 6, 1, 35, 1.6, 116.7, 70.4)
    g = gf.Geometry(*geo)
    assert (gf.bp_run(g, 2), gf.bp_run(g, 2, images=3)) == (8, 12)
    assert fused_equal_alone(gf, geo, 3, storage)[:2] == (1, 3)


@pytest.mark.parametrize("nzs", [70, 160, 256])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
def test_pairs_of_deep_columns_equal_frames_alone(gf, nzs, storage):  # noqa: F811
    geo = (24, nzs, 26, 6, 3, 11, 1.6, 40.0, 19.2)
    assert gf.bp_run(gf.Geometry(*geo), 2, images=3) == 0  # one warp per column: a pair and one frame alone
    assert fused_equal_alone(gf, geo, 3, storage) == (1, 3, 1)


def test_filter_without_a_scale_on_the_device_matches_oracle(gf):  # noqa: F811
    """An empty doubles image: the joint filter's scale, found on the device, is no number."""
    geo = (17, 40, 19, 8, 3, 5, 1.6, 24.0, 13.6)
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(3)
    nd = o.ndata
    tsino = np.concatenate([rs.poisson(9.0, nd), np.zeros(nd)]).astype(np.float32)
    kw = dict(dsino=np.zeros(2 * nd, np.float32), tsino=tsino, norm=np.ones(nd, np.float32))
    want = o.recon(2, nsub=2, niter=2, **kw)
    r = gf.Recon(gf.Context(gf.Geometry(*geo), nsub=2), 2, niter=2)
    r.load(**kw)
    r.iterate(2)
    assert not r.image(0).any() and want["img_t"].any()
    assert rel(r.image(1), want["img_t"]) < IMG_TOL
