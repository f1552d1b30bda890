"""GPU parity of the forward projector's one-bin and four-bin CTAs, through the C-ABI.

Geometries on both sides of the line between them (launch_fp_t in gf_fp.cu),
with bin counts that leave a remainder of the four, axial sizes off the vector
width of the resampling and segments whose columns need padding on both sides,
against the oracle (projection bound 1e-4); and the ratio path's rows, pad rows
included, through the images of a reconstruction (bound 1e-3).
"""
import numpy as np
import pytest

import gfo
from test_gpu_parity import FP_TOL, IMG_TOL, gf, rel  # noqa: F401

pytestmark = pytest.mark.gpu

GEOS = [
    (40, 33, 37, 9, 3, 7, 1.6, 53.0, 32.0),     # one bin a CTA, every size odd
    (24, 58, 149, 48, 1, 23, 0.4, 32.0, 19.2),  # four bins a CTA, the last CTA one bin
    (24, 61, 150, 45, 1, 29, 0.4, 20.0, 19.2),  # steep: columns padded by more than the image is deep
    (24, 64, 148, 45, 3, 9, 0.4, 32.0, 19.2),   # whole vectors and whole CTAs
]


@pytest.mark.parametrize("geo", GEOS, ids=lambda g: f"{g[0]}x{g[1]}_{g[2]}")
def test_projection_matches_oracle(gf, geo):  # noqa: F811
    o = gfo.Oracle(geo)
    ctx = gf.Context(gf.Geometry(*geo), nsub=1)
    img = np.random.RandomState(3).uniform(-1.0, 3.0, o.nvox).astype(np.float32)
    proj = ctx.array(o.ndata).upload(np.full(o.ndata, -7.0, np.float32))
    ctx.forward_project(ctx.put(img), 0, proj)
    got, want = proj.download(), o.fp(img, 1, 0)
    assert rel(got, want) < FP_TOL and np.abs(got - want).max() <= 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("nrad", [290, 291])
def test_reconstruction_with_four_bins_matches_oracle(gf, nrad):  # noqa: F811
    geo = (24, 40, nrad, 80, 1, 23, 0.2, 32.0, 19.2)
    o = gfo.Oracle(geo)
    rs = np.random.RandomState(6)
    nd = o.ndata
    dsino = np.concatenate([rs.poisson(20.0, nd), rs.uniform(0, 0.3, nd)]).astype(np.float32)
    norm = rs.uniform(0.9, 1.1, nd).astype(np.float32)
    want = o.recon(1, nsub=1, niter=1, dsino=dsino, norm=norm)
    ctx = gf.Context(gf.Geometry(*geo), nsub=1)
    r = gf.Recon(ctx, 1, niter=1)
    r.load(dsino=dsino, norm=norm)
    r.iterate(1)
    assert rel(r.image(0), want["img_d"]) < IMG_TOL
