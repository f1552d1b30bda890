"""GPU parity of the forward projector's one-bin and four-bin CTAs, with the route asserted.

One geometry on each side of every line of the rule (threads of a CTA, threads of
the grid, runs of planes a segment), with bin counts that leave each remainder of
the four, axial sizes off the vector width of the resampling and steep segments
whose columns are padded by more than the image is deep, against the oracle
(projection bound 1e-4); and the ratio path, which takes one bin at any size, for
row counts that leave each remainder of the four rows a thread loads together.
"""
import numpy as np
import pytest

import gfo
from test_gpu_parity import FP_TOL, IMG_TOL, gf, rel  # noqa: F401

pytestmark = pytest.mark.gpu

GEOS = [  # bins a CTA, geometry
    (4, (24, 58, 149, 40, 1, 5, 0.4, 32.0, 19.2)),    # two warps a CTA, the last CTA one bin
    (4, (24, 61, 150, 40, 1, 5, 0.4, 2.0, 19.2)),     # steep, two bins
    (4, (24, 64, 151, 40, 1, 5, 0.4, 32.0, 19.2)),    # three bins
    (1, (24, 58, 49, 40, 1, 5, 0.4, 32.0, 19.2)),     # too few threads
    (4, (20, 100, 66, 30, 1, 9, 0.4, 32.0, 16.0)),    # four warps, long runs
    (1, (20, 46, 110, 30, 1, 19, 0.4, 32.0, 16.0)),   # three warps, short segments
    (4, (16, 112, 47, 44, 1, 21, 0.4, 32.0, 12.8)),   # eight warps
    (1, (16, 112, 47, 18, 1, 21, 0.4, 32.0, 12.8)),   # eight warps, too few threads
    (1, (16, 118, 47, 60, 1, 25, 0.4, 32.0, 12.8)),   # ten warps
    (4, (16, 150, 46, 30, 1, 31, 0.4, 32.0, 12.8)),   # fifteen warps
    (1, (16, 150, 46, 26, 1, 31, 0.4, 32.0, 12.8)),   # fifteen warps, too few threads
]


@pytest.mark.parametrize("bins,geo", GEOS, ids=lambda g: f"{g[0]}x{g[1]}_{g[2]}x{g[3]}" if isinstance(g, tuple) else str(g))
def test_projection_matches_oracle(gf, bins, geo):  # noqa: F811
    g = gf.Geometry(*geo)
    assert gf.fp_run(g) == bins
    o = gfo.Oracle(geo)
    ctx = gf.Context(g, nsub=1)
    img = np.random.RandomState(3).uniform(-1.0, 3.0, o.nvox).astype(np.float32)
    proj = ctx.array(o.ndata).upload(np.full(o.ndata, -7.0, np.float32))
    ctx.forward_project(ctx.put(img), 0, proj)
    got, want = proj.download(), o.fp(img, 1, 0)
    assert rel(got, want) < FP_TOL and np.abs(got - want).max() <= 1e-4 * np.abs(want).max()


# planes of 3 segments with nzs slices: nzs + 2 (nzs - 2), in one warp: 4 rows of a thread hold 128
@pytest.mark.parametrize("nzs", [11, 43, 44, 45, 86, 87])
def test_ratio_rows_match_oracle(gf, nzs):  # noqa: F811
    geo = (16, nzs, 17, 9, 1, 3, 1.6, 32.0, 12.8)
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(6)
    nd = o.ndata
    dsino = np.concatenate([rs.poisson(20.0, nd), rs.uniform(0, 0.3, nd)]).astype(np.float32)
    norm = rs.uniform(0.9, 1.1, nd).astype(np.float32)
    norm[rs.uniform(size=nd) < 0.05] = 0.0
    want = o.recon(1, nsub=2, niter=1, dsino=dsino, norm=norm)
    ctx = gf.Context(gf.Geometry(*geo), nsub=2)
    r = gf.Recon(ctx, 1, niter=1)
    r.load(dsino=dsino, norm=norm)
    r.iterate(1)
    assert rel(r.image(0), want["img_d"]) < IMG_TOL
