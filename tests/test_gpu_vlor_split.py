"""GPU parity of the VLOR split and of the triples ratio it feeds.

The split (vlor_ends_kernel, vlor_split_sorted_kernel in gf_sino.cu) at the edges
of its blocks, with long runs of one bin and rejected events, bit for bit; the
ratio's 32x32 tiles (ratio_gather_kernel) through mode-3 images at sizes that
leave remainders in both directions, as ratios and as (ratio, mask) pairs.
"""
import numpy as np
import pytest

import gfo
from test_gpu_parity import IMG_TOL, gf, rel  # noqa: F401

pytestmark = pytest.mark.gpu

SMALL = (40, 33, 37, 9, 3, 7, 1.6, 53.0, 32.0)    # (ratio, mask) pairs
TILES = (73, 75, 70, 7, 3, 9, 1.6, 95.8, 58.4)
BITS = (102, 66, 81, 6, 1, 21, 1.6, 100.0, 72.0)  # ratios and mask bits


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 4097])
def test_split_matches_oracle(gf, n):  # noqa: F811
    o = gfo.Oracle(SMALL)
    rs = np.random.RandomState(n)
    ev = rs.randint(2, 2 + max(3, n // 8), (n, 2)).astype(np.int32)
    if n > 2:
        ev[-1, 0] = ev[n // 2, 1] = 0  # rejected
    proj, bl = rs.uniform(0, 1, o.ndata).astype(np.float32), rs.uniform(0, 2, o.ndata).astype(np.float32)
    proj[::3] = 0
    ctx = gf.Context(gf.Geometry(*SMALL))
    out = ctx.array(o.ndata).zero()
    ctx.vlor_split(ctx.put(ev, np.int32), n, ctx.put(proj), ctx.put(bl), out)
    assert np.array_equal(out.download(), o.vlor_split(ev, proj, bl))


@pytest.mark.parametrize("geo", [SMALL, TILES, BITS], ids=["pairs", "wide", "bits"])
def test_triples_match_oracle(gf, geo):  # noqa: F811
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(8)
    nd = o.ndata
    dsino = np.concatenate([rs.poisson(20.0, nd), rs.uniform(0, 0.3, nd)]).astype(np.float32)
    tsino = np.concatenate([rs.poisson(4.0, nd), rs.uniform(0, 0.1, nd)]).astype(np.float32)
    norm = rs.uniform(0.9, 1.1, nd).astype(np.float32)
    ev = rs.randint(1, nd, (nd, 2)).astype(np.int32)
    want = o.recon(3, nsub=2, niter=1, dsino=dsino, tsino=tsino, norm=norm, ev=ev)
    r = gf.Recon(gf.Context(gf.Geometry(*geo), nsub=2), 3, niter=1)
    r.load(dsino=dsino, tsino=tsino, norm=norm, events=ev)
    r.iterate(1)
    assert rel(r.image(0), want["img_d"]) < IMG_TOL and rel(r.image(1), want["img_t"]) < IMG_TOL
