"""The sketch update's paths at the sizes where they meet: batches of up to 65536 records are XORed in
directly, larger ones are grouped by vertex, vertices of up to 64 records and work chunks of the others take
different kernels.  Every sketch byte equals the restatement's."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu

DIRECT = 65536


def _random(V, n, seed):
    r = np.random.default_rng(seed)
    return r.integers(0, V, size=(n, 2), dtype=np.uint32)      # self-loops among them: skipped


def _stars(V, counts, n, seed):
    """Vertex i has counts[i] records (towards the high ids); filled up to n records with self-loops, which
    are skipped."""
    r = np.random.default_rng(seed)
    parts = [np.stack([np.full(c, i), r.integers(len(counts), V, c)], 1) for i, c in enumerate(counts)]
    p = np.concatenate(parts).astype(np.uint32)
    loops = np.full((n - len(p), 2), V - 1, np.uint32)
    p = np.concatenate([p, loops])
    flip = r.random(len(p)) < 0.5
    p[flip] = p[flip][:, ::-1]
    return p[r.permutation(len(p))]


def _check(restatement, V, pairs, factor=1.0, seed=0xC0FFEE):
    with gs.GraphSketch(V, seed, sketches_factor=factor) as g:
        g.ingest_pairs(pairs)
        g.synchronize()
        got = g.download()
    sk = restatement.new_sketches(V, factor)
    restatement.ingest(sk, V, seed, pairs, factor)
    assert got.tobytes() == sk.tobytes()


@pytest.mark.parametrize("V,factor", [(2, 1.0), (3, 1.0), (23, 1.0), (24, 1.0), (1500, 1.0), (1500, 1.65), (1500, 1.7),
                                      (1500, 2.2), (1500, 2.3), (1500, 4.3), (300, 1.65)])
@pytest.mark.parametrize("n", [1, 33, DIRECT, DIRECT + 1])
def test_direct_and_grouped(restatement, V, factor, n):
    _check(restatement, V, _random(V, n, V + n), factor)


@pytest.mark.parametrize("factor", [1.0, 1.7, 2.3])
def test_vertices_around_the_few_limit(restatement, factor):
    counts = [1, 2, 31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 1023, 1024, 1025, 2049]
    _check(restatement, 1500, _stars(1500, counts, DIRECT + 7, 3), factor)


def test_many_vertices_of_few_records(restatement):
    _check(restatement, 40009, _random(40009, DIRECT + 4097, 5))


@pytest.mark.parametrize("n", [5, DIRECT // 2, DIRECT + 100])
def test_tenants(restatement, n):
    sizes = [2, 5, 23, 24, 700, 1500]
    with SketchEngine(sum(tenant_bytes(V) for V in sizes) + (1 << 20), len(sizes), sum(sizes), 1500) as e:
        ids = [e.add_tenant(V, 9 + i) for i, V in enumerate(sizes)]
        recs = [_random(V, n // 6 + i, 31 + i) for i, V in enumerate(sizes)]
        e.ingest_batches(list(zip(ids, recs)))
        e.synchronize()
        for i, V in enumerate(sizes):
            sk = restatement.new_sketches(V)
            restatement.ingest(sk, V, 9 + i, recs[i])
            assert e.download(ids[i]).tobytes() == sk.tobytes()


@pytest.mark.parametrize("n", [999, DIRECT + 1])
def test_tagged_levels(restatement, n):
    V, levels, L, seed = 400, 3, 9, 0xABC
    pairs = _random(V, n, 8)
    with gs.GraphSketch(V, seed, num_levels=levels, num_subgraphs=L) as g:
        g.ingest_pairs(pairs)
        g.synchronize()
        got = [g.download(level=l).tobytes() for l in range(levels)]
    sk = restatement.new_sketches(V, 1.0, levels)
    restatement.ingest_levels(sk, V, levels, L, seed, pairs)
    flat = sk.tobytes()
    step = len(flat) // levels
    assert got == [flat[l * step:(l + 1) * step] for l in range(levels)]


def _repeated(V, hubs, n, seed, share=0.5):
    """n records of which `share` repeat an earlier one: vertex i < len(hubs) has about hubs[i] records."""
    r = np.random.default_rng(seed)
    parts = [np.stack([np.full(c, i), r.integers(len(hubs), V, c)], 1) for i, c in enumerate(hubs)]
    fresh = np.concatenate(parts + [r.integers(0, V, size=(max(0, int(n * (1 - share)) - sum(hubs)), 2))]).astype(np.uint32)
    again = fresh[r.integers(0, len(fresh), max(0, n - len(fresh)))][:, ::-1]
    p = np.concatenate([fresh, again])
    return np.ascontiguousarray(p[r.permutation(len(p))])


@pytest.mark.parametrize("V,hubs,n", [
    (50, [], 2_000_000),                              # every vertex several items
    (100, [], 300_000),                               # bitmap listed by words
    (5000, [1023, 1024, 1025, 2048, 2049, 4000], DIRECT + 5000),   # limits of the pass, of a tile
    (200_003, [9000, 12000, 30000, 70000], 400_000),  # several tiles, by words, two items of one vertex
    (1 << 18, [5000], DIRECT + 3), ((1 << 18) + 1, [5000], DIRECT + 3)])   # largest bitmap; none
def test_toggles_that_cancel(restatement, V, hubs, n):
    pairs = _repeated(V, hubs, n, V + n)
    with gs.GraphSketch(V, 0xC0FFEE) as g:
        for _ in range(2 if V <= 5000 else 1):        # a second pass starts from what the first one left
            g.clear()
            g.ingest_pairs(pairs)
            g.synchronize()
            if V <= 5000:
                sk = restatement.new_sketches(V)
                restatement.ingest(sk, V, 0xC0FFEE, pairs)
                assert g.download().tobytes() == sk.tobytes()
            else:
                # by linearity: the same records in batches that are not grouped give the same sketches
                with gs.GraphSketch(V, 0xC0FFEE) as h:
                    for i in range(0, len(pairs), DIRECT):
                        h.ingest_pairs(pairs[i:i + DIRECT])
                    h.synchronize()
                    for lo in range(0, V, 60000):
                        c = min(60000, V - lo)
                        assert g.download(first=lo, count=c).tobytes() == h.download(first=lo, count=c).tobytes()


def test_toggles_that_cancel_in_tenants_and_levels(restatement):
    sizes = [40, 3000, 700]
    with SketchEngine(sum(tenant_bytes(V) for V in sizes) + (1 << 20), 3, sum(sizes), 3700) as e:
        ids = [e.add_tenant(V, 9 + i) for i, V in enumerate(sizes)]
        recs = [_repeated(V, [2500] if V == 3000 else [], 90_000, 31 + i, 0.6) for i, V in enumerate(sizes)]
        e.ingest_batches(list(zip(ids, recs)))
        e.synchronize()
        for i, V in enumerate(sizes):
            sk = restatement.new_sketches(V)
            restatement.ingest(sk, V, 9 + i, recs[i])
            assert e.download(ids[i]).tobytes() == sk.tobytes()
    V, levels, L, seed = 60, 3, 9, 0xABC
    pairs = _repeated(V, [], 200_000, 8)
    with gs.GraphSketch(V, seed, num_levels=levels, num_subgraphs=L) as g:
        g.ingest_pairs(pairs)
        g.synchronize()
        got = b"".join(g.download(level=l).tobytes() for l in range(levels))
    sk = restatement.new_sketches(V, 1.0, levels)
    restatement.ingest_levels(sk, V, levels, L, seed, pairs)
    assert got == sk.tobytes()


@pytest.mark.parametrize("n", [1024, 1025, (1 << 22) - 1, 1 << 22, (1 << 22) + 1, 3 * (1 << 22) + 5])
def test_host_slices(n):
    """Host batches: read in place up to 1024 records, else in slices (of 2^22 records at this V) through the
    two slots; ordinary and page-locked memory, into a fresh handle and one whose slots are in use."""
    torch = pytest.importorskip("torch")
    V, seed = 1500, 0xC0FFEE
    pairs = torch.from_numpy(_random(V, n, n).view(np.int32))
    with gs.GraphSketch(V, seed) as g:
        g.ingest_pairs(pairs.cuda())
        g.synchronize()
        want = g.download().tobytes()
    for first in (pairs.pin_memory(), pairs):
        with gs.GraphSketch(V, seed) as g:
            g.ingest_pairs(first.numpy().view(np.uint32))
            g.synchronize()
            assert g.download().tobytes() == want
            g.ingest_pairs(pairs.numpy().view(np.uint32))      # the same records again: all cancel
            g.ingest_pairs(first.numpy().view(np.uint32))
            g.synchronize()
            assert g.download().tobytes() == want
