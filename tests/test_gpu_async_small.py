"""gs_ingest_pairs_async with page-locked input returns at once, however few the records and however far behind
the device is."""
import numpy as np
import pytest

import gpusketch_b200 as gs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 100, 1024, 1025])
def test_small_page_locked_batches_wait_for_nothing(restatement, n):
    import torch
    V, seed = 4096, 0x5EED5500
    r = np.random.default_rng(n)
    pairs = r.integers(0, V, size=(20 * n, 2), dtype=np.uint32)
    host = torch.from_numpy(pairs.view(np.int32)).pin_memory()
    side, big = torch.cuda.Stream(), torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()
    with gs.GraphSketch(V, seed) as g:
        g.set_stream(side)
        for _ in range(4):
            g.ingest_pairs_async(host[:n])
        g.synchronize()
        g.clear()
        with torch.cuda.stream(side):
            for _ in range(60):                     # 2 GB each: the device is at least ten milliseconds behind
                big.add_(1)
        behind = torch.cuda.Event()
        behind.record(side)
        for i in range(20):
            g.ingest_pairs_async(host[i * n:(i + 1) * n])
        assert not behind.query()                   # every call returned before the first batch was looked at
        g.synchronize()
        got = g.download().tobytes()
    sk = restatement.new_sketches(V)
    restatement.ingest(sk, V, seed, pairs)
    assert got == sk.tobytes()
