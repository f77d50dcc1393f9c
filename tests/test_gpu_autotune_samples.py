"""The autotuner on samples that the tuned kernels see, and on samples that they do not."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200 import autotune as tune
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu

N = 65536 + 4000


def _records(V, n, seed):
    return np.random.default_rng(seed).integers(0, V, size=(n, 2), dtype=np.uint32)


def test_autotune_leaves_the_tuning_to_samples_that_it_shows_in():
    import torch
    V = 2048
    with gs.GraphSketch(V, 9) as g, gs.GraphSketch(V, 9, max_batch_edges=50_000) as small:
        for handle, n in ((g, 65536), (g, 300), (small, 200_000)):
            d = torch.from_numpy(_records(V, n, n).view(np.int32)).cuda()
            before = tune.get_tuning(handle)
            tune.set_tuning(handle, 640, 5, 0)
            rows = []
            assert tune.autotune(handle, d, chunks=(32, 4096), warps=(1,), reg_depths=(1, 3), table=rows) == {
                "chunk": 640, "warps_per_block": 5, "reg_depth": 0}
            assert rows == [] and tune.get_tuning(handle)["chunk"] == 640
            tune.set_tuning(handle, **before)
        d = torch.from_numpy(_records(V, N, 1).view(np.int32)).cuda()
        assert tune.autotune(g, d, chunks=(32, 4096), warps=(2,), reg_depths=(1, 3))["chunk"] in (32, 4096)
        g.synchronize()
        assert not g.download().view(np.uint64).any()
    with SketchEngine(tenant_bytes(V), 1, V, V, max_batch_edges=1 << 18) as e:
        t = e.add_tenant(V, 3)
        tune.set_tuning(e, 640, 5, 0)
        d = torch.from_numpy(_records(V, 60_000, 2).view(np.int32)).cuda()
        assert tune.autotune_engine(e, [t], [0, 60_000], d, chunks=(32,), warps=(1,))["chunk"] == 640
        d = torch.from_numpy(_records(V, N, 2).view(np.int32)).cuda()
        assert tune.autotune_engine(e, [t], [0, N], d, chunks=(32,), warps=(1,))["chunk"] == 32
