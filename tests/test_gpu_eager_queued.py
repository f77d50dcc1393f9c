"""The eager DSU switched on while a query is queued: the query's partition becomes the DSU's only when nothing
changed the sketches in between."""
import numpy as np
import pytest

import gpusketch_b200 as gs

pytestmark = pytest.mark.gpu

V = 400


def _path(lo, hi):
    v = np.arange(lo, hi - 1, dtype=np.uint32)
    return np.stack([v, v + 1], 1)


def _check(restatement, g, *parts):
    labels, ncc, _ = g.connected_components()
    n, exact = restatement.exact_cc(V, np.concatenate(parts))
    assert ncc == n and np.array_equal(labels, exact)


@pytest.mark.parametrize("between", ["nothing", "ingest", "async", "clear"])
def test_switched_on_between_a_query_and_its_answer(restatement, between):
    a, b = _path(0, 100), _path(150, 300)
    with gs.GraphSketch(V, 9) as g:
        g.ingest_pairs(a)
        g.connected_components_async()
        g.set_eager_dsu(True)
        parts = [a]
        if between == "clear":
            g.clear()
            parts = []
        if between in ("ingest", "clear"):
            g.ingest_pairs(b)
        elif between == "async":
            g.ingest_pairs_async(b)
        if between != "nothing":
            parts.append(b)
        labels, ncc, _ = g.query_wait()
        n, exact = restatement.exact_cc(V, a)
        assert ncc == n and np.array_equal(labels, exact)
        _check(restatement, g, *parts)
        half = parts[-1][::2].copy()
        g.ingest_pairs(half)                   # forest edges go
        _check(restatement, g, *parts, half)
        g.ingest_pairs(half)
        _check(restatement, g, *parts)


@pytest.mark.parametrize("how", ["uploaded", "profiled", "read", "batches"])
def test_switched_on_over_sketches_that_are_there(restatement, tmp_path, how):
    """A handle whose record count says zero is not an empty graph when its sketches were uploaded or read from a
    file, or when the profile was reset after the ingest."""
    a = _path(0, 100)
    with gs.GraphSketch(V, 9) as g:
        g.ingest_pairs(a)
        if how == "profiled":
            g.synchronize()
            g.profile_enable(False)
            g.set_eager_dsu(True)
            assert not g.has_cached_query()
            _check(restatement, g, a)
            return
        g.write_binary(str(tmp_path / "g"))
        sketches = g.download()
    if how == "read":
        h = gs.GraphSketch.read_binary(str(tmp_path / "g"))
    else:
        h = gs.GraphSketch(V, 9)
        if how == "uploaded":
            h.upload(sketches)
        else:
            src, dst = np.concatenate([a[:, 0], a[:, 1]]), np.concatenate([a[:, 1], a[:, 0]])
            h.ingest_vertex_batches(src, np.arange(len(src), dtype=np.uint64), np.ones(len(src), np.uint64), dst)
            h.synchronize()
            h.profile_enable(False)
    with h:
        h.set_eager_dsu(True)
        assert not h.has_cached_query()
        _check(restatement, h, a)
