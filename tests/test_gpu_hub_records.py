"""Small batches whose records meet at one or a few vertices: the direct update holds a repeated vertex's buckets
until another one repeats.  Every sketch byte equals the restatement's."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu


def _hubs(V, n, hubs, share, seed):
    """A share of the records has a hub at either end; the others, self-loops and repeats among them, are random."""
    r = np.random.default_rng(seed)
    p = r.integers(0, V, size=(n, 2), dtype=np.uint32)
    at = r.random(n) < share
    p[at, 0] = r.integers(0, min(hubs, V), int(at.sum()))
    flip = r.random(n) < 0.5
    p[flip] = p[flip][:, ::-1]
    return p


def _want(restatement, V, seed, pairs, factor=1.0):
    sk = restatement.new_sketches(V, factor)
    restatement.ingest(sk, V, seed, pairs, factor)
    return sk.tobytes()


@pytest.mark.parametrize("factor,columns", [(1.0, 18), (2.2, 31), (2.25, 32), (2.3, 33), (4.45, 63), (4.5, 64)])
@pytest.mark.parametrize("n", [2, 31, 9473, 20_000, 65536])
def test_hubs_at_every_width(restatement, factor, columns, n):
    V, seed = 1300, 0x5EED5600
    assert gs.geometry_for(V, factor).num_columns == columns
    for hubs, share in ((1, 1.0), (1, 0.6), (2, 1.0), (5, 0.9)):
        pairs = _hubs(V, n, hubs, share, n + hubs)
        with gs.GraphSketch(V, seed, sketches_factor=factor) as g:
            g.ingest_pairs(pairs)
            g.synchronize()
            assert g.download().tobytes() == _want(restatement, V, seed, pairs, factor), (hubs, share)


@pytest.mark.parametrize("V", [2, 3, 5, 23])
def test_tiny_graphs(restatement, V):
    pairs = _hubs(V, 40_000, 1, 0.5, V)
    with gs.GraphSketch(V, 1) as g:
        g.ingest_pairs(pairs)
        g.synchronize()
        assert g.download().tobytes() == _want(restatement, V, 1, pairs)


def test_records_out_of_range_between_a_hubs(restatement):
    V = 1000
    pairs = _hubs(V, 50_000, 1, 1.0, 3)
    bad = pairs.copy()
    bad[::3, 1] = V + 7                                       # skipped; a hub's records stand on both sides
    with gs.GraphSketch(V, 1) as g:
        g.ingest_pairs(bad)
        with pytest.raises(gs.GpuSketchError):
            g.synchronize()
        got = g.download().tobytes()
    keep = np.delete(pairs, np.s_[::3], axis=0)
    assert got == _want(restatement, V, 1, keep)


def test_hubs_of_tenants_and_levels(restatement):
    sizes = [2, 900, 5, 1400, 24]
    with SketchEngine(sum(tenant_bytes(V) for V in sizes), len(sizes), sum(sizes), max(sizes)) as e:
        ids = [e.add_tenant(V, 9 + i) for i, V in enumerate(sizes)]
        recs = [_hubs(V, 12_000 + i, 1, 0.9, 31 + i) for i, V in enumerate(sizes)]
        e.ingest_batches(list(zip(ids, recs)))
        e.synchronize()
        for i, V in enumerate(sizes):
            assert e.download(ids[i]).tobytes() == _want(restatement, V, 9 + i, recs[i])
    V, levels, L, seed = 400, 3, 9, 0xABC
    for hubs in (1, 3):
        pairs = _hubs(V, 60_000, hubs, 0.95, hubs)
        with gs.GraphSketch(V, seed, num_levels=levels, num_subgraphs=L) as g:
            g.ingest_pairs(pairs)
            g.synchronize()
            got = b"".join(g.download(level=l).tobytes() for l in range(levels))
        sk = restatement.new_sketches(V, 1.0, levels)
        restatement.ingest_levels(sk, V, levels, L, seed, pairs)
        assert got == sk.tobytes()
