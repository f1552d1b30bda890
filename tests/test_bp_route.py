"""Which kernel a geometry's back projections take (CPU).

Geometries measured with both kernels, without masked bins and with 2 % of them:
those that column tiles slow down by more than 8 % take one warp per column, and
the configurations keep the tiles, in runs of 12 slices where these make enough
CTAs.
"""
import pytest

import gfirst_gb300 as gf


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__

    __graft_entry__.build()


def geometry(res, nzs, nseg, span=1):
    return gf.Geometry(res, nzs, res, 64, span, nseg, 1.6, 1.3 * res, 0.8 * res)


@pytest.mark.parametrize("res,nzs,span,nseg", [
    (97, 117, 3, 5), (97, 124, 3, 5), (117, 102, 3, 3), (114, 93, 3, 3), (98, 86, 1, 31), (69, 147, 3, 25),
    (68, 150, 3, 25)])
def test_geometries_that_tiles_slow_down_take_columns(res, nzs, span, nseg):
    assert gf.bp_run(geometry(res, nzs, nseg, span), 4) == 0


@pytest.mark.parametrize("g,alone,two", [
    (gf.Geometry.preclinical(), 12, 12), (gf.Geometry.reference(), 12, 12), (gf.Geometry.small(), 0, 0),
    (gf.Geometry(64, 64, 64, 64, 3, 21, 1.6, 84.8772096, 51.2), 0, 0),
    (gf.Geometry(96, 96, 96, 96, 3, 31, 1.6, 127.3158, 76.8), 12, 12),
    (geometry(91, 90, 53), 8, 12), (geometry(80, 110, 35), 8, 12), (geometry(105, 114, 5, 3), 12, 12)])
def test_run_lengths(g, alone, two):
    assert (gf.bp_run(g, 4), gf.bp_run(g, 4, images=2)) == (alone, two)


def test_query_checks_its_arguments():
    with pytest.raises(gf.GfError):
        gf.bp_run(gf.Geometry.small(), 4, images=0)
    with pytest.raises(gf.GfError):
        gf.bp_run(gf.Geometry.small(), 0)
