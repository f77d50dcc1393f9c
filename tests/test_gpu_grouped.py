"""The grouped update (bucketing, work lists, k_ingest_packed and k_ingest) over every column count, every tuning,
hubs, tenants of all sizes and two-word records, in batches large enough to be grouped; each test checks that its
batches were.  Every sketch byte equals the restatement's."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200 import autotune as tune
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu

N = 65536 + 4000


def _hub(V, n, hub_records, seed):
    r = np.random.default_rng(seed)
    p = r.integers(0, V, size=(n, 2), dtype=np.uint32)
    hub = np.stack([np.full(hub_records, 7, np.uint32), r.integers(0, V, hub_records, dtype=np.uint32)], axis=1)
    p = np.concatenate([p, hub])
    return p[r.permutation(len(p))]


def _want(restatement, V, seed, pairs, factor=1.0):
    sk = restatement.new_sketches(V, factor)
    restatement.ingest(sk, V, seed, pairs, factor)
    return sk.tobytes()


def _grouped(g, call):
    """The call's records went through the bucketing kernels, of which a grouped pass has at least six."""
    g.profile_enable(True)
    call()
    p = g.profile_read()
    g.profile_enable(False)
    return p["bucket_launches"] >= 6


FACTORS = [1.38, 1.45, 1.5, 1.6, 1.66, 1.75, 1.8, 1.9, 1.95, 2.0, 2.1, 2.2, 2.25, 2.3, 2.4]


def test_factors_name_every_column_count():
    assert [gs.geometry_for(1024, f).num_columns for f in FACTORS] == list(range(19, 34))


@pytest.mark.parametrize("factor", FACTORS)
def test_every_column_count(restatement, factor):
    V, seed = 1024, 0x5EED3000
    pairs = _hub(V, N, 9000, int(factor * 100))          # 140 records a vertex, a hub of many chunks
    with gs.GraphSketch(V, seed, sketches_factor=factor) as g:
        assert _grouped(g, lambda: g.ingest_pairs(pairs))
        assert g.download().tobytes() == _want(restatement, V, seed, pairs, factor)


@pytest.mark.parametrize("V", [700, 5000])                # many records a vertex, few
@pytest.mark.parametrize("tuning", [(32, 1, 1), (1024, 4, 2), (4096, 8, 3), (100000, 16, 1), (777, 3, 2), (64, 2, 0),
                                    (5000, 16, 0)])
def test_every_tuning(restatement, V, tuning):
    pairs = _hub(V, N, 3000, V)
    with gs.GraphSketch(V, 41) as g:
        tune.set_tuning(g, *tuning)
        assert _grouped(g, lambda: g.ingest_pairs(pairs))
        assert g.download().tobytes() == _want(restatement, V, 41, pairs)


def test_hub_of_many_chunks(restatement):
    V, seed = 20000, 99
    r = np.random.default_rng(4)
    star = np.stack([np.zeros(V - 1, np.uint32), np.arange(1, V, dtype=np.uint32)], 1)
    pairs = np.concatenate([star, r.integers(0, V, size=(N, 2), dtype=np.uint32), star[:5000]])
    with gs.GraphSketch(V, seed) as g:
        assert _grouped(g, lambda: g.ingest_pairs(pairs))
        assert g.download().tobytes() == _want(restatement, V, seed, pairs)
        labels, ncc, _ = g.connected_components()
    n, exact = restatement.exact_cc(V, pairs)
    assert ncc == n and np.array_equal(labels, exact)


@pytest.mark.parametrize("max_vertices", [1 << 14, 1 << 22])     # one-word records, two-word records
def test_tenants_of_all_sizes(restatement, max_vertices):
    """Fewer buckets per column than rows, more, few records a vertex and many, and several widths, in one launch."""
    sizes = [(3, 1.0, 900), (12, 1.0, 3000), (23, 1.0, 4000), (24, 1.0, 5000), (4096, 1.0, 60_000), (300, 1.0, 30_000),
             (777, 1.5, 2000), (2000, 2.3, 5000)]
    budget = sum(tenant_bytes(V, f) for V, f, _ in sizes)
    with SketchEngine(budget, len(sizes), max_vertices, max_vertices // 2 if max_vertices > 1 << 14 else 4096,
                      max_batch_edges=1 << 20) as e:
        ids = [e.add_tenant(V, 50 + i, f) for i, (V, f, _) in enumerate(sizes)]
        recs = [_hub(V, n, n // 10, i) % np.uint32(V) for i, (V, _, n) in enumerate(sizes)]
        assert sum(len(p) for p in recs) > N
        assert _grouped(e, lambda: e.ingest_batches(list(zip(ids, recs))))
        res = e.connected_components(ids)
        for i, (V, f, _) in enumerate(sizes):
            assert e.download(ids[i]).tobytes() == _want(restatement, V, 50 + i, recs[i], f)
            assert np.array_equal(res[ids[i]].labels, restatement.exact_cc(V, recs[i])[1])
