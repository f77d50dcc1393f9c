"""Handles of different sizes on different host threads: a launch on one thread does not take away what a launch on
another needs."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import gpusketch_b200 as gs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small", [((20_011, 1.0), (9001, 1.0)),       # rows of the query, buckets of the sort
                                         ((100_003, 1.0), (70_001, 1.0)),
                                         ((2000, 1.6), (1800, 1.0)),         # columns of the update
                                         ((2000, 2.6), (300, 2.6))])         # the wide update
def test_small_launches_between_large_ones(restatement, large, small):
    with ThreadPoolExecutor(1) as a, ThreadPoolExecutor(1) as b:
        def make(V, factor):
            r = np.random.default_rng(V)
            p = r.integers(0, V, size=(70_000, 2), dtype=np.uint32)
            return gs.GraphSketch(V, 3, sketches_factor=factor), p, restatement.exact_cc(V, p)

        def use(g, p, exact):
            g.clear()
            g.ingest_pairs(p)
            labels, ncc, _ = g.connected_components()
            assert ncc == exact[0] and np.array_equal(labels, exact[1])

        x, y = a.submit(make, *large).result(), b.submit(make, *small).result()
        for _ in range(3):
            a.submit(use, *x).result()
            b.submit(use, *y).result()
        x[0].close()
        y[0].close()
