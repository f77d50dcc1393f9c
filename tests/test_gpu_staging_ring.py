"""The page-locked ring is shared by all host input: a call writes a slot only once the copy that an earlier call
queued from it, of whatever kind, has been made."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from stream_file import write_stream_file

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("second", ["pairs", "small", "file", "batches"])
@pytest.mark.parametrize("first", ["pairs", "small", "file", "batches"])
def test_a_queued_copy_is_made_before_its_slot_is_written(restatement, tmp_path, first, second):
    import torch
    V, seed = 4096, 0x5EED5300
    side, big = torch.cuda.Stream(), torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()
    r = np.random.default_rng(53)
    data = []
    for i in range(2):
        n = 1000 if (first, second)[i] == "small" else 50_000
        data.append(r.integers(0, V, size=(n, 2), dtype=np.uint32))
        write_stream_file(str(tmp_path / f"{i}.data"), V, data[i], np.zeros(n, np.uint8))
    # the vertex batches of both endpoints, as worker threads hand them over
    def batches(p):
        src, dst = np.concatenate([p[:, 0], p[:, 1]]), np.concatenate([p[:, 1], p[:, 0]])
        keep = src != dst
        order = np.argsort(src[keep], kind="stable")
        src, dst = src[keep][order], dst[keep][order]
        at = np.flatnonzero(np.concatenate([[True], src[1:] != src[:-1]]))
        return src[at], at.astype(np.uint64), np.diff(np.append(at, len(src))).astype(np.uint64), dst

    made = [batches(p) for p in data]
    with gs.GraphSketch(V, seed) as g:
        g.set_stream(side)

        def put(i):
            kind = (first, second)[i]
            if kind == "file":
                g.ingest_stream_file(str(tmp_path / f"{i}.data"))
            elif kind == "batches":
                g.ingest_vertex_batches(*made[i])
            else:
                g.ingest_pairs_async(data[i])

        for i in (0, 1, 0, 1):                # everything is allocated; all of it cancels
            put(i)
        g.synchronize()
        with torch.cuda.stream(side):
            for _ in range(60):               # 2 GB each: the device is at least ten milliseconds behind
                big.add_(1)
        g.connected_components_async()
        put(0)
        put(1)
        g.query_wait()
        g.synchronize()
        got = g.download().tobytes()
    sk = restatement.new_sketches(V)
    for p in data:
        restatement.ingest(sk, V, seed, p)
    assert got == sk.tobytes()
