"""A queued query that gives up waiting reports GS_ERR_TIMEOUT where it is collected, and nothing else: errors of
calls before and behind it are reported by the calls that report them after any other query."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200 import _native

pytestmark = pytest.mark.gpu

V = 1 << 16


def _status(call):
    try:
        call()
    except gs.GpuSketchError as e:
        return e.status
    return _native.GS_OK


@pytest.mark.parametrize("synchronize_first", [False, True])
def test_errors_around_a_query_that_gives_up(restatement, synchronize_first):
    pairs, bad = gs.rmat_stream(16, 100_000, 0x5EED5400), np.array([[V, 1], [2, 3]], np.uint32)
    with gs.GraphSketch(V, 11) as g:
        g.ingest_pairs(pairs)
        for _ in range(3):
            g.set_device_wait_limit(1)
            g.connected_components_async()
            if synchronize_first:
                assert _status(g.synchronize) == _native.GS_OK
            g.ingest_pairs_async(bad)
            if synchronize_first:
                assert _status(g.synchronize) == _native.GS_ERR_BAD_ARG
            assert _status(g.query_wait) == _native.GS_ERR_TIMEOUT
            assert _status(g.synchronize) == (_native.GS_OK if synchronize_first else _native.GS_ERR_BAD_ARG)
            assert _status(g.synchronize) == _native.GS_OK
            g.ingest_pairs(bad)                            # before the query: reported with it, and first
            g.connected_components_async()
            assert _status(g.query_wait) == _native.GS_ERR_BAD_ARG
            assert _status(g.synchronize) == _native.GS_OK
        g.set_device_wait_limit(0)
        labels, ncc, _ = g.connected_components()
        n, exact = restatement.exact_cc(V, pairs)
        assert ncc == n and np.array_equal(labels, exact)
