"""Device records are read in the order of the stream that wrote them, and their memory may be used again in
that order: torch's default stream, side streams and explicitly named ones.  Every batch is small enough to be
read once, so a record that came late or was overwritten shows as different sketch bytes and nothing else."""
import numpy as np
import pytest

import gpusketch_b200 as gs
from gpusketch_b200.engine import SketchEngine, tenant_bytes

pytestmark = pytest.mark.gpu

V, SEED, N = 4096, 0x5EED5000, 40_000


def _records(seed):
    return np.random.default_rng(seed).integers(0, V, size=(N, 2), dtype=np.uint32)


def _want(restatement, *parts):
    sk = restatement.new_sketches(V)
    for p in parts:
        restatement.ingest(sk, V, SEED, p)
    return sk.tobytes()


def _ingest(kind, g, recs, stream=None):
    if kind == "pairs":
        g.ingest_pairs(recs, stream=stream)
    elif kind == "async":
        g.ingest_pairs_async(recs, stream=stream)
    elif kind == "edges":
        g.ingest_edges(recs[:, 0], recs[:, 1], stream=stream)     # strided: copies are made on the way
    else:
        g.ingest([0], [0, recs.shape[0]], recs, stream=stream)


class _Handle:
    """A graph, or an engine with one tenant, with the same sketches."""

    def __init__(self, kind):
        self.engine = kind == "engine"
        if self.engine:
            self.h = SketchEngine(tenant_bytes(V) + (1 << 20), 1, V, V, max_batch_edges=1 << 16)
            assert self.h.add_tenant(V, SEED) == 0
        else:
            self.h = gs.GraphSketch(V, SEED)

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.h.close()

    def warm(self, kind, recs):
        """Everything is loaded and allocated, so that the calls after this only queue."""
        import torch
        for _ in range(2):
            _ingest(kind, self.h, recs)
        self.clear()
        self.h.synchronize()
        torch.cuda.synchronize()

    def clear(self):
        self.h.clear_tenant(0) if self.engine else self.h.clear()

    def bytes(self):
        self.h.synchronize()
        return (self.h.download(0) if self.engine else self.h.download()).tobytes()


def _device(torch, a):
    d = torch.from_numpy(a.view(np.int32)).cuda()
    torch.cuda.synchronize()
    return d


def _busy(torch, big):
    for _ in range(40):          # some milliseconds of work on the current stream
        big.add_(1)


KINDS = ["pairs", "async", "edges", "engine"]


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_records_written_just_before_the_call(restatement, kind, side):
    import torch
    a = _records(1)
    src, recs, big = _device(torch, a), torch.zeros((N, 2), dtype=torch.int32, device="cuda"), torch.zeros(1 << 28, device="cuda")
    stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
    with _Handle(kind) as g:
        g.warm(kind, src)
        with torch.cuda.stream(stream):
            _busy(torch, big)
            recs.copy_(src)
            _ingest(kind, g.h, recs)
        assert g.bytes() == _want(restatement, a)


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_memory_used_again_after_the_call(restatement, kind, side):
    import torch
    a, b = _records(2), _records(3)
    src = [_device(torch, x) for x in (a, b)]
    stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
    with _Handle(kind) as g:
        g.warm(kind, src[0])
        with torch.cuda.stream(stream):
            for s in src:
                recs = s.clone()
                stream.synchronize()
                if s is src[0]:
                    for _ in range(200):      # the handle's stream is some milliseconds behind
                        g.clear()
                _ingest(kind, g.h, recs)
                recs.fill_(5)                 # self-loops: skipped
                del recs
        assert g.bytes() == _want(restatement, a, b)


@pytest.mark.parametrize("kind", KINDS)
def test_clear_before_an_ingest_on_a_side_stream(restatement, kind):
    import torch
    a = _records(4)
    recs, side = _device(torch, a), torch.cuda.Stream()
    with _Handle(kind) as g:
        g.warm(kind, recs)
        for _ in range(200):
            g.clear()
        with torch.cuda.stream(side):
            _ingest(kind, g.h, recs)
        assert g.bytes() == _want(restatement, a)


@pytest.mark.parametrize("kind", KINDS)
def test_named_streams(restatement, kind):
    """A stream named in the call orders it, whatever torch's current stream is; strided operands are copied in
    its order too, and torch's default stream may be named."""
    import torch
    a, b = _records(5), _records(6)
    wide = [_device(torch, np.concatenate([x, x], 1)) for x in (a, b)]
    big = torch.zeros(1 << 28, device="cuda")
    side = torch.cuda.Stream()
    with _Handle(kind) as g:
        g.warm(kind, wide[0][:, :2])
        for w, stream, other in zip(wide, (side, torch.cuda.default_stream()), (torch.cuda.default_stream(), side)):
            with torch.cuda.stream(stream):
                recs = torch.zeros_like(w)
                _busy(torch, big)
                recs.copy_(w)
            with torch.cuda.stream(other):
                _ingest(kind, g.h, recs[:, 1:3] if kind != "edges" else recs[:, :2], stream=stream)
            torch.cuda.synchronize()
        want = _want(restatement, a if kind == "edges" else a[:, ::-1].copy(), b if kind == "edges" else b[:, ::-1].copy())
        assert g.bytes() == want
