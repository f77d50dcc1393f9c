"""The Boruvka kernel's scopes at the sizes where they meet and at the edges of its pieces: one graph on a
cluster (up to 8192 vertices) and on the whole GPU, with the complement and (one-sided batches) without it,
and several tenants in narrow, wide and whole-GPU scopes.  Partitions and round counts are exact."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu


def _two_sided_batches(pairs):
    src = np.concatenate([pairs[:, 0], pairs[:, 1]])
    order = np.argsort(src, kind="stable")
    src, dst = src[order], np.concatenate([pairs[:, 1], pairs[:, 0]])[order]
    first = np.flatnonzero(np.concatenate([[True], src[1:] != src[:-1]]))
    sizes = np.diff(np.append(first, len(src)))
    return src[first].astype(np.uint32), first.astype(np.uint64), sizes.astype(np.uint64), dst.astype(np.uint32)


def _stream(kind, V, seed):
    if kind == "path":          # long chains: many rounds of small components
        ids = np.random.default_rng(seed).permutation(V).astype(np.uint32)
        return np.stack([ids[:-1], ids[1:]], 1)
    if kind == "blocks":        # components of 17 vertices: one more than a piece
        v = np.arange(V - 1, dtype=np.uint32)
        return np.stack([v, v + 1], 1)[(v + 1) % 17 != 0]
    return gs.er_stream(V, min(1.0, 3.0 / V), seed, 0.1, 0.5)


@pytest.mark.parametrize("one_sided", [False, True])
@pytest.mark.parametrize("kind", ["er", "path", "blocks"])
@pytest.mark.parametrize("V", [2, 3, 33, 1025, 8192, 8193, 20011])
def test_single_graph_scopes(restatement, V, kind, one_sided):
    pairs = _stream(kind, V, V)
    with gs.GraphSketch(V, 0xC0FFEE + V) as g:
        if len(pairs):
            if one_sided:
                g.ingest_vertex_batches(*_two_sided_batches(pairs))
            else:
                g.ingest_pairs(pairs)
        labels, ncc, rounds = g.connected_components()
        n, exact = restatement.exact_cc(V, pairs)
        assert ncc == n and np.array_equal(labels, exact)
        if V <= 8193:
            st, olabels, orounds, _ = restatement.boruvka(g.download().view(np.uint64).reshape(-1).copy(), V, 0xC0FFEE + V)
            assert st == 0 and rounds == orounds and np.array_equal(olabels, exact)
        forest = g.spanning_forest()
        assert len(forest) == V - n and np.all(forest[:, 0] < forest[:, 1])
        assert np.array_equal(restatement.exact_cc(V, forest)[1], exact)


@pytest.mark.parametrize("sizes", [[9001], [300, 70001, 65537], [70001, 70002, 70003, 5], [5000] * 12 + [40000],
                                   [700] * 19, list(range(2, 42))])
def test_tenant_scopes(restatement, sizes):
    with SketchEngine(sum(tenant_bytes(V) for V in sizes) + (1 << 20), len(sizes), sum(sizes), max(max(sizes), 2),
                      max_batch_edges=1 << 18) as e:
        ids = [e.add_tenant(V, 77 + i) for i, V in enumerate(sizes)]
        recs = [_stream("er", V, 5 + i) for i, V in enumerate(sizes)]
        e.ingest_batches(list(zip(ids, recs)))
        res = e.connected_components(ids)
        for t, V, r, i in zip(ids, sizes, recs, range(len(sizes))):
            n, exact = restatement.exact_cc(V, r)
            assert res[t].num_cc == n and np.array_equal(res[t].labels, exact)
            with gs.GraphSketch(V, 77 + i) as g:
                if len(r):
                    g.ingest_pairs(r)
                assert g.connected_components()[2] == res[t].rounds
