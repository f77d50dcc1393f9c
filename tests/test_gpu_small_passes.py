"""A handle whose internal ingest passes are small (max_batch_edges): every host path fits its staging slots."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200.engine import SketchEngine, tenant_bytes
from stream_file import write_stream_file

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [1, 6, 7, 100, 1023])
def test_host_input_of_a_handle_with_small_passes(restatement, tmp_path, most):
    torch = pytest.importorskip("torch")
    V, seed = 300, 0x5EED5200
    r = np.random.default_rng(most)
    small, large = r.integers(0, V, size=(1024, 2), dtype=np.uint32), r.integers(0, V, size=(1500, 2), dtype=np.uint32)
    src = np.arange(40, dtype=np.uint32)
    dst = r.integers(0, V, 40 * 30).astype(np.uint32)
    path = str(tmp_path / "s.data")
    write_stream_file(path, V, small, np.zeros(len(small), np.uint8))
    with gs.GraphSketch(V, seed, max_batch_edges=most) as g:
        for p in (small, large, torch.from_numpy(large.view(np.int32)).pin_memory(), small):
            g.ingest_pairs(p)
        for p in (small, large):
            g.ingest_pairs_async(p)
        g.ingest_stream_file(path)
        g.synchronize()
        sk = restatement.new_sketches(V)
        restatement.ingest(sk, V, seed, large)       # three times; `small` four times
        assert g.download().tobytes() == sk.tobytes()
        g.ingest_vertex_batches(src, np.arange(40, dtype=np.uint64) * 30, np.full(40, 30, np.uint64), dst)
        g.ingest_vertex_batches(src, np.arange(40, dtype=np.uint64) * 30, np.full(40, 30, np.uint64), dst)
        g.synchronize()
        assert g.download().tobytes() == sk.tobytes()
    with SketchEngine(tenant_bytes(V) + (1 << 20), 1, V, V, max_batch_edges=most) as e:
        t = e.add_tenant(V, seed)
        e.ingest_batches([(t, large)])
        e.ingest_slices([(t, small), (t, small)])
        e.synchronize()
        assert e.download(t).tobytes() == sk.tobytes()
        with pytest.raises(gs.GpuSketchError):       # a phase is one pass
            e.phase([t], [0, most + 1], torch.zeros((most + 1, 2), dtype=torch.int32, device="cuda"), [t])
