"""GPU parity of the joint bilateral filter without a range term, through the C-ABI.

An infinite sigmai or max_ref, or a pair whose scale 1 / (max_ref sigmai) under- or
overflows although each factor is an ordinary number: the far-side voxels, whose
window is cut by the image, included.  Against the oracle, whose exponentials are
double; a weight is one FP32 exponential with an argument rounded at most four
times (relative 1e-6 where the weight matters), the result a weighted mean: 1e-5
of the largest value.
"""
import numpy as np
import pytest

import gfo
from test_gpu_bilateral import run
from test_gpu_parity import gf  # noqa: F401

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("res,nzs", [(9, 6), (19, 33), (24, 64)])
@pytest.mark.parametrize("r", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("sigmai,max_ref,scale", [
    (INF, 1.0, 1.0), (0.025, INF, 1.0), (INF, INF, 1.0), (1e30, 1e17, 1.0), (3e38, 3e38, 1.0),
    (0.025, 2.3e-38, 2e-38),  # the scale overflows
    (0.5, 3e38, 1.0),         # and is subnormal
])
def test_range_term_off_or_extreme_matches_oracle(gf, res, nzs, r, sigmai, max_ref, scale):  # noqa: F811
    geo = (res, nzs, 9, 4, 1, 1, 1.6, 20.0, 12.0)
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(res + r)
    img = rs.uniform(0.5, 2.0, o.nvox).astype(np.float32)
    ref = (scale * (1.0 + 0.05 * rs.randn(o.nvox))).astype(np.float32)
    want = o.bilateral(img, ref, max_ref, r, 0.75, sigmai)
    assert (want.reshape(nzs, res, res)[r:, r:, r:] > 0.4).all()
    got = run(gf, geo, img, ref, max_ref, r, 0.75, sigmai)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(img).max()


@pytest.mark.parametrize("sigmai,max_ref", [(INF, 1.0), (0.025, INF), (0.025, 1.0)])
def test_infinite_reference_values_match_oracle(gf, sigmai, max_ref):  # noqa: F811
    geo = (19, 40, 9, 4, 1, 1, 1.6, 20.0, 12.0)
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(4)
    img = rs.uniform(0.5, 2.0, o.nvox).astype(np.float32)
    ref = (1.0 + 0.05 * rs.randn(o.nvox)).astype(np.float32)
    ref[rs.randint(0, o.nvox, 5)] = np.inf
    want = o.bilateral(img, ref, max_ref, 2, 0.75, sigmai)
    got = run(gf, geo, img, ref, max_ref, 2, 0.75, sigmai)
    assert np.isfinite(want).all() and np.abs(got - want).max() <= 1e-5 * np.abs(img).max()
