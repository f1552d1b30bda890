"""Frames of several normalizations and subset counts in one fused group, on columns.

Every frame equals itself alone, bit for bit, and the pairs counted are those of
equal mask and subset count: classes that interleave, classes of one, and a group
of the most frames a launch takes.
"""
import numpy as np
import pytest

from test_gpu_batch_masks import GEO, data
from test_gpu_parity import gf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masks,nsubs", [
    ((7, 5, 7, 5, 3, 7), (2, 2, 2, 2, 2, 2)),
    ((7, 7, 7, 5, 7, 5), (2, 3, 2, 3, 3, 3)),
    ((7, 5, 3, 11), (2, 2, 2, 2)),
    ((7, 5) * 8, (2, 2, 2, 3) * 4),
], ids=["interleaved", "subsets", "alone", "sixteen"])
def test_classes_match_frames_alone(gf, masks, nsubs):  # noqa: F811
    assert gf.bp_run(gf.Geometry(*GEO), 2) == 0  # one warp per column: pairs run

    def frames():
        recs = [gf.Recon(gf.Context(gf.Geometry(*GEO), nsub=n), 1, niter=1) for n in nsubs]
        for k, (r, m) in enumerate(zip(recs, masks)):
            r.load(**data(gf, r.ctx, k, m))
        return recs

    recs = frames()
    b = gf.Batch(recs)
    b.set_fused(True)
    pairs = sum(sum(z == c for z in zip(masks, nsubs)) // 2 for c in set(zip(masks, nsubs)))
    assert b.groups() == (1, len(masks), pairs)
    b.iterate(1)
    b.sync()
    for r, a in zip(recs, frames()):
        a.iterate(1)
        assert np.array_equal(r.image(0), a.image(0))
