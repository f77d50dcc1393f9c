"""A caller's device buffer that is written while the library reads it (no stream named, so nothing orders the
two): the records are counted and placed from different contents.  The answer of such a call is undefined, but it
ends with GS_OK or a reported consistency error, and the handle is exact again after a clear."""
import ctypes as C

import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,levels", [(2048, 1), (1500, 1), (100_003, 1), (700, 3)])
def test_records_that_change_while_they_are_read(restatement, V, levels):
    import torch
    n, seed, L = (1 << 17) + 77, 0x5EED5100, 9
    r = np.random.default_rng(V)
    hub = np.stack([r.integers(0, 3, n), r.integers(3, V, n)], 1).astype(np.uint32)        # one bucket, toggles cancel
    high = np.stack([np.full(n, V - 1), r.integers(0, V - 1, n)], 1).astype(np.uint32)     # the last one
    even = r.integers(0, V, size=(n, 2), dtype=np.uint32)
    kinds = [torch.from_numpy(p.view(np.int32)).cuda() for p in (hub, even, high, even)]
    buf = kinds[0].clone()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with gs.GraphSketch(V, seed, num_levels=levels, num_subgraphs=L if levels > 1 else 0) as g:
        seen = set()
        for it in range(40):
            with torch.cuda.stream(side):
                for k in range(12):
                    buf.copy_(kinds[(it + k) % 4])
            _native.check(g._lib.gs_ingest_pairs(g._h, C.c_void_p(buf.data_ptr()), n, 1, None), "gs_ingest_pairs")
            seen.add(g._lib.gs_synchronize(g._h))
            side.synchronize()
        assert seen <= {_native.GS_OK, _native.GS_ERR_INTERNAL}
        g.clear()
        g.ingest_pairs(kinds[1])
        g.synchronize()
        got = b"".join(g.download(level=l).tobytes() for l in range(levels))
    sk = restatement.new_sketches(V, 1.0, levels)
    if levels > 1:
        restatement.ingest_levels(sk, V, levels, L, seed, even)
    else:
        restatement.ingest(sk, V, seed, even)
    assert got == sk.tobytes()
