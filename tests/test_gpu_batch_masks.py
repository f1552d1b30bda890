"""Fused frames that back-project two per warp follow their masks.

Where the back projector runs one warp per column, a batch's frames of equal
normalization masks share it two by two, and the captured graph holds the pairs:
a frame loaded with another mask afterwards must not keep its partner's.
"""
import numpy as np
import pytest

from test_gpu_parity import gf  # noqa: F401

pytestmark = pytest.mark.gpu

GEO = (40, 33, 37, 9, 3, 7, 1.6, 53.0, 32.0)


def data(gf, ctx, seed, masked):  # noqa: F811
    rs = np.random.RandomState(seed)
    nd = ctx.ndata
    dsino = np.concatenate([rs.poisson(20.0, nd), rs.uniform(0, 0.3, nd)]).astype(np.float32)
    norm = np.ones(nd, np.float32)
    norm[::masked] = 0.0
    return dict(dsino=dsino, norm=norm)


@pytest.mark.parametrize("graph", [False, True])
def test_pairs_follow_a_later_load(gf, graph):  # noqa: F811
    def frame():
        return gf.Recon(gf.Context(gf.Geometry(*GEO), nsub=2), 1, niter=1)

    recs = [frame() for _ in range(3)]
    for k, r in enumerate(recs):
        r.load(**data(gf, r.ctx, k, 7))
    b = gf.Batch(recs)
    b.set_fused(True)
    for masks in ((7, 7, 7), (7, 5, 7), (5, 5, 7), (7, 7, 5)):
        for k, r in enumerate(recs):
            r.load(**data(gf, r.ctx, k, masks[k]))
        b.iterate(1, graph=graph)
        b.sync()
        for k, r in enumerate(recs):
            a = frame()
            a.load(**data(gf, a.ctx, k, masks[k]))
            a.iterate(1)
            assert np.array_equal(r.image(0), a.image(0))
