"""Tenants that fill the engine's arena to its last bucket: vertices of few records of a large tenant and of small
ones behind it are updated by the same warps, and nothing is read or asked for past the arena."""
import numpy as np
import pytest

from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[30_000, 2], [30_000, 24, 5, 3, 2], [2, 3, 30_000, 40], [12_000, 700, 11_000, 2, 2]])
def test_small_tenants_at_the_end_of_the_arena(restatement, sizes):
    with SketchEngine(sum(tenant_bytes(V) for V in sizes), len(sizes), sum(sizes), max(sizes)) as e:
        ids = [e.add_tenant(V, 7 + i) for i, V in enumerate(sizes)]
        assert e.memory()[0] == e.memory()[1]
        r = np.random.default_rng(sum(sizes))
        recs = [r.integers(0, V, size=(80_000 if V == max(sizes) else 3 * V, 2), dtype=np.uint32) for V in sizes]
        for _ in range(3):
            e.ingest_batches(list(zip(ids, recs)))
        e.synchronize()
        for i, V in enumerate(sizes):
            sk = restatement.new_sketches(V)
            restatement.ingest(sk, V, 7 + i, recs[i])
            assert e.download(ids[i]).tobytes() == sk.tobytes()
