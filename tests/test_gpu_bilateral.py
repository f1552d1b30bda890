"""GPU parity of the joint bilateral filter at its tiles' edges, through the C-ABI.

Sizes off the 8x8-column, 32-slice tiles and below one, every window radius,
against the oracle, whose exponentials are double.  Tolerance: a weight is one
FP32 exponential with an argument rounded three times (relative 1e-6 where the
weight matters), the result a weighted mean: 1e-5 of the largest value.
"""
import numpy as np
import pytest

import gfo
from test_gpu_parity import gf  # noqa: F401

pytestmark = pytest.mark.gpu


def run(gf_, geo, img, ref, max_ref, r, sigma3d=0.75, sigmai=0.025):
    ctx = gf_.Context(gf_.Geometry(*geo))
    out = ctx.array(ctx.nvox)
    ctx.bilateral(ctx.put(img), ctx.put(ref), max_ref, out, r, sigma3d, sigmai)
    return out.download()


@pytest.mark.parametrize("res,nzs", [(8, 5), (16, 32), (19, 33), (25, 70)])
@pytest.mark.parametrize("r", [0, 1, 2, 3, 4])
def test_window_radii_match_oracle(gf, res, nzs, r):  # noqa: F811
    geo = (res, nzs, 9, 4, 1, 1, 1.6, 20.0, 12.0)
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(res + r)
    img = rs.uniform(0.0, 2.0, o.nvox).astype(np.float32)
    ref = (1.0 + 0.05 * rs.randn(o.nvox)).astype(np.float32)
    for sigma3d, sigmai in ((0.75, 0.025), (2.0, 0.5)):
        want = o.bilateral(img, ref, float(ref.max()), r, sigma3d, sigmai)
        got = run(gf, geo, img, ref, float(ref.max()), r, sigma3d, sigmai)
        assert np.abs(got - want).max() <= 1e-5 * np.abs(img).max()


def test_narrowest_spatial_weight_is_the_voxel_itself(gf):  # noqa: F811
    geo = (17, 34, 9, 4, 1, 1, 1.6, 20.0, 12.0)
    rs = np.random.RandomState(1)
    n = 17 * 17 * 34
    img, ref = rs.uniform(0.5, 2.0, n).astype(np.float32), rs.uniform(0.5, 1.0, n).astype(np.float32)
    got = run(gf, geo, img, ref, 1.0, 4, sigma3d=1e-20).reshape(34, 17, 17)
    want = img.reshape(34, 17, 17).copy()
    want[:4], want[:, :4], want[:, :, :4] = 0.0, 0.0, 0.0
    assert np.array_equal(got, want)


def test_zero_range_gives_zero(gf):  # noqa: F811
    geo = (16, 33, 9, 4, 1, 1, 1.6, 20.0, 12.0)
    n = 16 * 16 * 33
    got = run(gf, geo, np.ones(n, np.float32), np.zeros(n, np.float32), 0.0, 4)
    assert not got.any()
