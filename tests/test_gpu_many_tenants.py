"""Queries of very many small tenants share one launch over the whole GPU; fewer run on a cluster each.  Partitions
are exact, round counts those of a graph of its own, in every mix and in recorded phases."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [[], [17_000], [17_000, 20_001]])
@pytest.mark.parametrize("count", [300, 1500])
def test_many_small_tenants(restatement, count, extra):
    import torch
    r = np.random.default_rng(count)
    sizes = [int(x) for x in r.integers(2, 90, count)] + extra
    recs = [r.integers(0, V, size=(max(1, int(V * r.uniform(0.2, 2.5))), 2), dtype=np.uint32) for V in sizes]
    exact = [restatement.exact_cc(V, p) for V, p in zip(sizes, recs)]
    with SketchEngine(sum(tenant_bytes(V) for V in sizes), len(sizes), sum(sizes), max(sizes),
                      max_batch_edges=1 << 18) as e:
        ids = [e.add_tenant(V, 7 + i) for i, V in enumerate(sizes)]
        e.ingest_batches(list(zip(ids, recs)))
        rounds = {}
        for part in (ids, ids[::-1], ids[::2], ids[-1:], ids):
            res = e.connected_components(part)
            assert set(res) == set(part)
            for t in part:
                i = t if ids[t] == t else ids.index(t)
                assert res[t].num_cc == exact[i][0] and np.array_equal(res[t].labels, exact[i][1])
                assert rounds.setdefault(t, res[t].rounds) == res[t].rounds
        for i in list(range(0, count, max(1, count // 25))) + list(range(count, len(sizes))):
            with gs.GraphSketch(sizes[i], 7 + i) as g:
                g.ingest_pairs(recs[i])
                assert g.connected_components()[2] == rounds[ids[i]]
        # phases, recorded and not: the same records again, and once more
        offs = np.cumsum([0] + [len(p) for p in recs]).astype(np.uint64)
        d = torch.from_numpy(np.concatenate(recs).view(np.int32)).cuda()
        for step in range(4):
            got = e.phase(ids, offs, d, ids, cuda_graph=step % 2 == 0)
            for i, t in enumerate(ids):
                assert got[t] == ((sizes[i], 0) if step % 2 == 0 else (exact[i][0], rounds[t]))
