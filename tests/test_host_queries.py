"""Host geometry queries cost a table of the segments, whatever the ring's width (CPU).

The back projector's staged-row buffer takes a loop whose length follows 1 /
diameter; only a context needs it.  A 0.01 mm ring makes that loop take more
than a second.
"""
import time

import pytest

import gfirst_gb300 as gf

RING = gf.Geometry(128, 159, 129, 160, 3, 53, 1.6, 0.01, 100.0)


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__

    __graft_entry__.build()


@pytest.mark.parametrize("query", [lambda: gf.sizes(RING), lambda: gf.segment_table(RING),
                                   lambda: gf.lor_index(RING, 0, 0, 0, 0), lambda: gf.bin_endpoints(RING, 64),
                                   lambda: gf.recon_bytes(RING, 4)],
                         ids=["sizes", "segments", "lor_index", "bin_endpoints", "recon_bytes"])
def test_queries_do_not_size_the_staged_rows(query):
    query()
    t = time.perf_counter()
    for _ in range(20):
        query()
    assert time.perf_counter() - t < 2.0


def test_an_event_costs_its_sorted_ends_and_their_values():
    """2 ends a VLOR event: 8 bytes of key, 8 of projection and weight each."""
    import ctypes

    def total(events):
        p, b = gf.recon_defaults(3), ctypes.c_int64()
        g = gf.Geometry.small()
        assert gf.lib().gf_recon_bytes(ctypes.byref(g.c()), 4, ctypes.byref(p), ctypes.c_int64(events), ctypes.byref(b)) == 0
        return b.value

    assert total(1000) - total(0) == 1000 * 32
