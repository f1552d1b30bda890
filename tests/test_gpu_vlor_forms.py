"""GPU parity of the VLOR split's two forms, bit for bit, through the C-ABI.

By event where projection and weight lie in L2 (up to 10 M bins, every geometry
of the other tests), by end above: the same events on geometries of either side,
rejected events and long runs of one bin included, as an operator and through a
mode-3 reconstruction that is loaded again with fewer and with more events.
"""
import numpy as np
import pytest

import gfo
from test_gpu_parity import IMG_TOL, gf, rel  # noqa: F401

pytestmark = pytest.mark.gpu

BY_EVENT = (40, 33, 37, 9, 3, 7, 1.6, 53.0, 32.0)
BY_END = (16, 60, 120, 90, 1, 31, 1.6, 120.0, 12.8)  # 1.4 K planes


def events(rs, nd, n):
    ev = rs.randint(2, 2 + max(3, min(nd - 2, n // 8)), (n, 2)).astype(np.int32)
    ev[rs.uniform(size=n) < 0.5, 1] = rs.randint(1, nd + 1)
    ev[n // 2, 0] = 0  # rejected
    ev[-1, 1] = nd + 1
    return ev


@pytest.mark.parametrize("geo,above", [(BY_EVENT, False), (BY_END, True)], ids=["event", "end"])
@pytest.mark.parametrize("n", [2, 129, 5000])
def test_split_matches_oracle(gf, geo, above, n):  # noqa: F811
    o = gfo.Oracle(geo)
    assert (o.ndata > 10 << 20) == above
    rs = np.random.RandomState(n)
    ev = events(rs, o.ndata, n)
    proj, bl = rs.uniform(0, 1, o.ndata).astype(np.float32), rs.uniform(0, 2, o.ndata).astype(np.float32)
    proj[::3] = 0
    ctx = gf.Context(gf.Geometry(*geo))
    out = ctx.array(o.ndata).zero()
    ctx.vlor_split(ctx.put(ev, np.int32), n, ctx.put(proj), ctx.put(bl), out)
    assert np.array_equal(out.download(), o.vlor_split(ev, proj, bl))


@pytest.mark.parametrize("geo", [BY_EVENT, BY_END], ids=["event", "end"])
def test_reloaded_reconstruction_matches_oracle(gf, geo):  # noqa: F811
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(5)
    nd = o.ndata
    kw = dict(dsino=np.concatenate([rs.poisson(20.0, nd), np.zeros(nd)]).astype(np.float32),
              tsino=np.concatenate([rs.poisson(4.0, nd), np.zeros(nd)]).astype(np.float32), norm=np.ones(nd, np.float32))
    r = gf.Recon(gf.Context(gf.Geometry(*geo), nsub=3), 3, niter=1)
    for n in (4000, 300, 9000):
        ev = events(rs, nd, n)
        r.load(**kw, events=ev)
        r.iterate(1)
        want = o.recon(3, nsub=3, niter=1, ev=ev, **kw)
        assert rel(r.image(0), want["img_d"]) < IMG_TOL and rel(r.image(1), want["img_t"]) < IMG_TOL
