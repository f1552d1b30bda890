"""A batch's graph is captured again whenever its pairs no longer share a mask.

The captured graph holds the pairs of the masks it was captured with.  What
happens between a load and the next replay must not hide the change: iterations
without the graph, or a comparison that ended in an error (here a frame's stream
that is being captured, where the library may not wait).
"""
import ctypes
import ctypes.util

import numpy as np
import pytest

from test_gpu_batch_masks import GEO, data
from test_gpu_parity import gf  # noqa: F401

pytestmark = pytest.mark.gpu


def frames(gf, masks):  # noqa: F811
    recs = [gf.Recon(gf.Context(gf.Geometry(*GEO), nsub=2), 1, niter=1) for _ in masks]
    load(gf, recs, masks)
    return recs


def load(gf, recs, masks, which=None):  # noqa: F811
    for k, r in enumerate(recs):
        if which is None or k in which:
            r.load(**data(gf, r.ctx, k, masks[k]))


def alone(gf, masks, its):  # noqa: F811
    recs = frames(gf, masks)
    for r, n in zip(recs, its):
        r.iterate(n)
    return [r.image(0) for r in recs]


def test_iterations_without_the_graph_between_load_and_replay(gf):  # noqa: F811
    recs = frames(gf, (7, 7, 5))
    b = gf.Batch(recs)
    b.set_fused(True)
    b.iterate(1)
    load(gf, recs, (7, 3, 5), which=(1,))
    b.iterate(1, graph=False)
    b.iterate(1)
    b.sync()
    for r, want in zip(recs, alone(gf, (7, 3, 5), (3, 2, 3))):
        assert np.array_equal(r.image(0), want)


def test_failed_comparison_between_load_and_replay(gf):  # noqa: F811
    name = ctypes.util.find_library("cudart") or "libcudart.so"
    try:
        rt = ctypes.CDLL(name)
    except OSError:
        rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
    stream = ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    recs = frames(gf, (7, 7, 5))
    assert gf.lib().gf_set_stream(recs[2].ctx.h, stream) == 0
    b = gf.Batch(recs)
    b.set_fused(True)
    b.iterate(1)
    load(gf, recs, (7, 3, 5), which=(1,))
    b.sync()
    assert rt.cudaStreamBeginCapture(stream, 2) == 0
    graph = ctypes.c_void_p()
    with pytest.raises(gf.GfError):
        b.iterate(1)
    rt.cudaStreamEndCapture(stream, ctypes.byref(graph))  # the wait above ended the capture
    gf.Context(gf.Geometry(*GEO)).close()  # reads the error that the runtime still holds for the next launch
    b.iterate(1)
    b.sync()
    for r, want in zip(recs, alone(gf, (7, 3, 5), (2, 1, 2))):
        assert np.array_equal(r.image(0), want)
    b.close()
    assert gf.lib().gf_set_stream(recs[2].ctx.h, None) == 0
    assert rt.cudaStreamDestroy(stream) == 0
