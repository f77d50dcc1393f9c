"""The work this framework is used for, as measured cases.

A case is a dict of plain values.  `kind` names the entry points it goes through:

  phase    one graph: clear (or a sliding window, see `window`), ingest a batch of edge records,
           connected_components().  `source` says where the records are: device-resident (a tensor),
           page-locked host memory, or an ordinary host array.
  noalloc  gs_ingest_pairs_noalloc into the caller's own sketch buffer.
  workers  per-vertex batches from the host, as worker threads hand them over, then a query.
  batched  many independent graphs in one engine: clear, then phases of ingest + query of all of them.
  served   resident tenants of an engine: a coalesced ingest of several clients' page-locked batches, a
           query of some tenants, and the expiry (deletion) of the same batches.
  mincut   a min-cut graph: subgraph-tagged ingest and the k-forest min-cut driver.
  query    connected_components() alone, over sketches that are already there.

Streams: `rmat` is R-MAT(0.57, 0.19, 0.19, 0.05) with 12% of the records re-emitting (deleting) an earlier
record's edge, which is the large-ingest benchmark's stream; `er` is a simple random graph's edges in
random order with a tenth of them deleted and half of those inserted again, which is the plain and the
batched workloads' stream.  Both are made on the GPU with torch, from the seed alone.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import gpusketch_b200 as gs
from gpusketch_b200 import _native
from gpusketch_b200.engine import SketchEngine, tenant_bytes

SKETCH_SEED = 0xC0FFEE
NOALLOC_EDGES = 65536      # most records of one allocation-free call


def listed():
    return [
        # a handful of toggles on a small live graph and the answer after them, then the toggles undone:
        # the smallest calls, where launches and waits are everything
        dict(name="few_toggles", kind="phase", V=1000, n=100, stream="er", source="host", window=20000),
        # the plain connected-components workload: G(1024, 0.05) with churn, one batch and one query
        dict(name="plain_1k", kind="phase", V=1024, n=30160, stream="er", source="device", window=0),
        # a caller that owns its device memory and may not allocate: one full-sized call
        dict(name="noalloc_8k", kind="noalloc", V=8191, n=65536),
        # worker batches (one source vertex, up to a batch of destinations) from host memory
        dict(name="workers_8k", kind="workers", V=8192, n=1 << 20),
        # an ordinary skewed stream: a few hundred records per vertex
        dict(name="rmat_16k", kind="phase", V=1 << 14, n=1 << 22, stream="rmat", source="device", window=0),
        # a uniform stream of a ragged size
        dict(name="er_100k", kind="phase", V=100003, n=12345677, stream="er", source="device", window=0),
        # the large-ingest benchmark's phase: 2^27 records, then the query
        dict(name="rmat_128k", kind="phase", V=1 << 17, n=1 << 27, stream="rmat", source="device", window=0),
        # the same graph fed from page-locked host memory
        dict(name="host_128k", kind="phase", V=1 << 17, n=1 << 25, stream="rmat", source="pinned", window=0),
        # many vertices, few records each: a window of updates over a large sparse graph
        dict(name="sparse_1m", kind="phase", V=1000003, n=1 << 22, stream="er", source="device", window=1 << 24),
        # 256 independent streams in four phases
        dict(name="batched_256", kind="batched", tenants=256, lo=8.0, hi=14.0, phases=4),
        # 64 resident tenants, one serving iteration
        dict(name="served_64", kind="served", tenants=64, lo=10.0, hi=16.0, batches=24, blo=10.0, bhi=20.0, queries=8),
        # two dense blocks joined by three edges: the level-by-level min cut
        dict(name="mincut_4k", kind="mincut", block=2048, p=0.3, k=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["phase", "phase", "phase", "phase", "query", "noalloc", "workers", "batched", "served", "mincut"])
    if kind in ("phase", "query"):
        V = _log(rng, 500, 1000003)
        # from a few records to 2^27 in all, at most 2^10 per vertex, and a simple graph's worth for `er`
        stream = rng.choice(["rmat", "er"])
        most = min(1 << 27, V << 10)
        if stream == "er":
            most = min(most, V * (V - 1) // 8, 1 << 24)
        n = _log(rng, 64, most)
        if kind == "query":
            return dict(kind=kind, V=V, n=max(n, min(most, V)), stream=stream)
        if stream == "er" and rng.random() < 0.4:
            n = min(n, 1 << 22)
            return dict(kind=kind, V=V, n=n, stream=stream, source=rng.choice(["device", "host"]),
                        window=min(most, max(n, 16 * V)))
        source = rng.choice(["device", "device", "pinned", "host"])
        if source != "device":
            n = min(n, 1 << 25 if source == "pinned" else 1 << 22)
        return dict(kind=kind, V=V, n=n, stream=stream, source=source, window=0)
    if kind == "noalloc":
        return dict(kind=kind, V=_log(rng, 500, 65536), n=_log(rng, 64, NOALLOC_EDGES))
    if kind == "workers":
        V = _log(rng, 1000, 32768)
        return dict(kind=kind, V=V, n=_log(rng, 4096, min(1 << 21, V * (V - 1) // 8)))
    if kind == "batched":
        return dict(kind=kind, tenants=_log(rng, 4, 256), lo=8.0, hi=round(rng.uniform(10.0, 14.0), 2),
                    phases=rng.randint(1, 4))
    if kind == "served":
        t = _log(rng, 8, 64)
        return dict(kind=kind, tenants=t, lo=10.0, hi=round(rng.uniform(12.0, 16.0), 2), batches=_log(rng, 1, 32),
                    blo=10.0, bhi=round(rng.uniform(12.0, 20.0), 2), queries=rng.randint(1, t))
    return dict(kind=kind, block=_log(rng, 200, 2048), p=round(rng.uniform(0.2, 0.4), 3), k=4)


# ---- streams ----

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed & (2**62 - 1))
    return g


def _rmat(V, n, seed):
    """(n, 2) int32: R-MAT records over ceil(log2 V) bits, ids taken modulo V, 12% re-emissions."""
    bits = max(1, (V - 1).bit_length())
    out = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    g = _gen(seed)
    step = 1 << 24
    for lo in range(0, n, step):
        m = min(step, n - lo)
        u = torch.zeros(m, dtype=torch.int32, device="cuda")
        v = torch.zeros(m, dtype=torch.int32, device="cuda")
        for _ in range(bits):
            q = torch.rand(m, device="cuda", generator=g)
            qu = q >= 0.76
            qv = ((q >= 0.57) & ~qu) | (q >= 0.95)
            u = u * 2 + qu
            v = v * 2 + qv
        u %= V
        v %= V
        v = torch.where(u == v, (v + 1) % V, v)
        out[lo:lo + m, 0] = u
        out[lo:lo + m, 1] = v
    for lo in range(0, n, step):
        m = min(step, n - lo)
        i = torch.arange(lo, lo + m, device="cuda", dtype=torch.int64)
        pick = torch.rand(m, device="cuda", generator=g) < 0.12
        pick &= i > 0
        i = i[pick]
        j = (torch.rand(i.numel(), device="cuda", generator=g, dtype=torch.float64) * i).long()
        out[i] = out[j]
    return out


def _er(V, n, seed):
    """(n, 2) int32: n / 1.15 distinct random edges in random order, a tenth of them then deleted, half of
    those inserted again."""
    g = _gen(seed)
    m = max(1, min(int(n / 1.15), V * (V - 1) // 2))
    want = m
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while keys.numel() < m:
        k = max(64, int(1.1 * want))
        a = torch.randint(V, (k,), device="cuda", generator=g)
        b = torch.randint(V - 1, (k,), device="cuda", generator=g)
        b += b >= a
        keys = torch.unique(torch.cat([keys, torch.minimum(a, b) * V + torch.maximum(a, b)]))
        want = m - keys.numel() if keys.numel() < m else 0
    keys = keys[torch.randperm(keys.numel(), device="cuda", generator=g)[:m]]
    rest = n - m
    again = max(0, min(m, rest - rest // 3))
    stream = torch.cat([keys, keys[:again], keys[:max(0, min(again, rest - again))]])[:n]
    out = torch.stack([stream // V, stream % V], 1).to(torch.int32)
    flip = torch.rand(out.shape[0], device="cuda", generator=g) < 0.5
    return torch.where(flip[:, None], out.flip(1), out).contiguous()


def _stream(kind, V, n, seed):
    return _rmat(V, n, seed) if kind == "rmat" else _er(V, n, seed)


def _planted(case, seed):
    """Records, vertex count and one side's vertices of two G(block, p) joined by three edges, with 5% churn;
    the vertices are numbered at random."""
    b, g = case["block"], _gen(seed)
    parts = []
    for off in (0, b):
        hit = torch.rand((b, b), device="cuda", generator=g) < case["p"]
        e = torch.triu(hit, 1).nonzero()
        parts.append(e + off)
    a = torch.randperm(b, device="cuda", generator=g)[:3]
    c = torch.randperm(b, device="cuda", generator=g)[:3] + b
    e = torch.cat(parts + [torch.stack([a, c], 1)])
    e = e[torch.randperm(e.shape[0], device="cuda", generator=g)]
    churn = e[torch.randperm(e.shape[0], device="cuda", generator=g)[:e.shape[0] // 20]]
    ids = torch.randperm(2 * b, device="cuda", generator=g)
    return ids[torch.cat([e, churn, churn])].to(torch.int32).contiguous(), 2 * b, ids[b:]


def _placed(pairs, source):
    if source == "device":
        return pairs
    if source == "pinned":
        host = torch.empty(pairs.shape, dtype=pairs.dtype, pin_memory=True)
        host.copy_(pairs)
        return host
    return pairs.cpu().numpy().astype(np.uint32)


def _tenants(case, seed):
    """Vertex counts of the tenants (the case's own), and a numpy generator of the seed for the rest."""
    sizes = np.random.default_rng(0x5EED2000)
    return ([int(round(2.0 ** sizes.uniform(case["lo"], case["hi"]))) for _ in range(case["tenants"])],
            np.random.default_rng(seed))


def _batched_streams(case, seed):
    """Per tenant its V and records, all tenants' records of each phase back to back, and the offsets."""
    Vs, r = _tenants(case, seed)
    recs = []
    for i, V in enumerate(Vs):
        d = float(r.uniform(4.0, 64.0))
        recs.append(_er(V, max(8, int(1.15 * min(d, (V - 1) / 2) * V / 2)), seed * 1009 + i))
    P = case["phases"]
    phases = []
    for p in range(P):
        cut = [x[len(x) * p // P: len(x) * (p + 1) // P] for x in recs]
        offs = np.cumsum([0] + [len(x) for x in cut]).astype(np.uint64)
        phases.append((offs, torch.cat(cut).contiguous()))
    return Vs, phases


def _served_batches(case, seed):
    Vs, r = _tenants(case, seed)
    out = []
    for i in range(case["batches"]):
        t = int(r.integers(len(Vs)))
        n = int(round(2.0 ** r.uniform(case["blo"], case["bhi"])))
        out.append((t, _rmat(Vs[t], n, seed * 1009 + i)))
    # the queried tenants are the case's own too
    asked = sorted(np.random.default_rng(7).choice(len(Vs), size=min(case["queries"], len(Vs)), replace=False).tolist())
    return Vs, out, asked


# ---- the cases ----

def prepare(case, seed):
    kind = case["kind"]
    if kind == "phase":
        V = case["V"]
        g = gs.GraphSketch(V, SKETCH_SEED)
        pairs = _stream(case["stream"], V, case["n"], seed)
        if case["window"]:
            g.ingest_pairs(_stream(case["stream"], V, case["window"], seed + 77777))
            g.synchronize()
        return dict(kind=kind, g=g, pairs=_placed(pairs, case["source"]), window=bool(case["window"]))
    if kind == "query":
        g = gs.GraphSketch(case["V"], SKETCH_SEED)
        g.ingest_pairs(_stream(case["stream"], case["V"], case["n"], seed))
        g.synchronize()
        return dict(kind=kind, g=g)
    if kind == "noalloc":
        V = case["V"]
        sk = torch.zeros((V, gs.geometry_for(V).num_buckets, 2), dtype=torch.int64, device="cuda")
        pairs = _er(V, case["n"], seed)
        return dict(kind=kind, V=V, sk=sk, pairs=pairs)
    if kind == "workers":
        V = case["V"]
        g = gs.GraphSketch(V, SKETCH_SEED)
        p = _er(V, case["n"], seed).long()
        src = torch.cat([p[:, 0], p[:, 1]])
        order = torch.argsort(src, stable=True)
        src, dst = src[order].cpu().numpy(), torch.cat([p[:, 1], p[:, 0]])[order].cpu().numpy().astype(np.uint32)
        most = int(g.geometry.num_buckets * 4)     # destinations of one worker batch
        first = np.flatnonzero(np.concatenate([[True], src[1:] != src[:-1]]))
        size = np.diff(np.append(first, len(src)))
        srcs, starts, sizes = [], [], []
        for f, s in zip(first.tolist(), size.tolist()):
            for o in range(0, s, most):
                srcs.append(int(src[f]))
                starts.append(f + o)
                sizes.append(min(most, s - o))
        return dict(kind=kind, g=g, batches=(np.array(srcs, np.uint32), np.array(starts, np.uint64),
                                             np.array(sizes, np.uint64), dst))
    if kind == "batched":
        Vs, phases = _batched_streams(case, seed)
        e = SketchEngine(sum(tenant_bytes(V) for V in Vs) + (1 << 20), len(Vs), sum(Vs), max(Vs),
                         max_batch_edges=max(1 << 16, max(int(o[-1]) for o, _ in phases)))
        ids = [e.add_tenant(V, SKETCH_SEED + i) for i, V in enumerate(Vs)]
        return dict(kind=kind, e=e, ids=ids, phases=phases)
    if kind == "served":
        Vs, batches, asked = _served_batches(case, seed)
        e = SketchEngine(sum(tenant_bytes(V) for V in Vs) + (1 << 20), len(Vs), sum(Vs), max(Vs), max_batch_edges=1 << 23)
        ids = [e.add_tenant(V, SKETCH_SEED + i) for i, V in enumerate(Vs)]
        for i, V in enumerate(Vs):
            base = _rmat(V, 8 * V, seed * 2003 + i)
            e.ingest([ids[i]], [0, base.shape[0]], base)
        e.synchronize()
        return dict(kind=kind, e=e, asked=[ids[t] for t in asked],
                    batches=[(ids[t], _placed(p, "pinned")) for t, p in batches])
    pairs, V, _ = _planted(case, seed)
    log2 = math.log2(V)
    factor = math.ceil(log2 / 0.75 ** 2) / log2 * 1.5      # the min-cut tool's sketch size
    g = gs.GraphSketch(V, SKETCH_SEED, sketches_factor=factor, num_levels=4, num_subgraphs=14)
    return dict(kind=kind, g=g, pairs=pairs, k=case["k"])


def run(state):
    kind = state["kind"]
    if kind == "phase":
        g, pairs = state["g"], state["pairs"]
        if not state["window"]:
            g.clear()
        g.ingest_pairs(pairs)
        out = g.connected_components()
        if state["window"]:
            g.ingest_pairs(pairs)          # the window's records expire: toggled back out
        return out
    if kind == "query":
        return state["g"].connected_components()
    if kind == "noalloc":
        sk, pairs = state["sk"], state["pairs"]
        sk.zero_()
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _native.check(_native.lib().gs_ingest_pairs_noalloc(
            state["V"], SKETCH_SEED, 1.0, ctypes.c_void_p(pairs.data_ptr()), pairs.shape[0],
            ctypes.c_void_p(sk.data_ptr()), stream), "gs_ingest_pairs_noalloc")
        return sk
    if kind == "workers":
        g = state["g"]
        g.clear()
        g.ingest_vertex_batches(*state["batches"])
        return g.connected_components()
    if kind == "batched":
        e, ids = state["e"], state["ids"]
        for t in ids:
            e.clear_tenant(t)
        got = [e.phase(ids, offs, pairs, ids) for offs, pairs in state["phases"]]
        return np.array([[r[t] for t in ids] for r in got], np.int64)
    if kind == "served":
        e = state["e"]
        e.ingest_slices(state["batches"])
        res = e.connected_components(state["asked"])
        e.ingest_slices(state["batches"])
        return (np.concatenate([res[t].labels for t in state["asked"]]),
                np.array([[res[t].num_cc, res[t].rounds] for t in state["asked"]], np.int64))
    g = state["g"]
    g.clear()
    g.ingest_pairs(state["pairs"])
    value, level, cut, side = g.min_cut(state["k"])
    return value, level, cut, side ^ side[0]      # which side is called 1 is not part of the answer


# ---- what a pass cannot do without ----

def _sketch_bytes(V, factor=1.0):
    return V * gs.geometry_for(V, factor).num_buckets * 16


def work(case):
    """Records read once, the sketches written once (all of them after a clear, else the buckets that the
    records reach, read and written), labels written once.  The path is integer work: no flops."""
    kind = case["kind"]

    def reached(V, n):
        # buckets that 2 n endpoint records over V vertices reach: per column the depths that some record of
        # the vertex has, depth d with probability 2^-(d+1), and the deterministic bucket
        geo, m = gs.geometry_for(V), 2 * n / V
        depths = sum(1 - (1 - 0.5 ** (d + 1)) ** m for d in range(geo.bkt_per_col))
        return int(V * 16 * (geo.num_columns * depths + min(1.0, m)))

    if kind == "phase":
        V, n = case["V"], case["n"]
        if case["window"]:
            return {"bytes": 2 * (8 * n + 2 * reached(V, n)) + 4 * V, "flops": 0}
        return {"bytes": 8 * n + _sketch_bytes(V) + 4 * V, "flops": 0}
    if kind == "query":
        geo = gs.geometry_for(case["V"])
        return {"bytes": case["V"] * (geo.bkt_per_col + 1) * 16 + 4 * case["V"], "flops": 0}
    if kind == "noalloc":
        return {"bytes": 8 * case["n"] + _sketch_bytes(case["V"]), "flops": 0}
    if kind == "workers":
        return {"bytes": 8 * case["n"] + _sketch_bytes(case["V"]) + 4 * case["V"], "flops": 0}
    if kind == "batched":
        # mean over the draw of V and of the degree
        V = sum(2.0 ** (case["lo"] + (case["hi"] - case["lo"]) * (i + 0.5) / 64) for i in range(64)) / 64
        n = 1.15 * 17 * V
        return {"bytes": case["tenants"] * (8 * n + _sketch_bytes(int(V)) + case["phases"] * 4 * V), "flops": 0}
    if kind == "served":
        n = sum(2.0 ** (case["blo"] + (case["bhi"] - case["blo"]) * (i + 0.5) / 64) for i in range(64)) / 64 * case["batches"]
        return {"bytes": 2 * 8 * n, "flops": 0}
    V = 2 * case["block"]
    n = 1.1 * case["p"] * case["block"] ** 2
    return {"bytes": 8 * n + 2 * _sketch_bytes(V, 2.7), "flops": 0}


# ---- exact answers ----

def _components(pairs, V):
    """Smallest vertex id of every vertex's component, of the edges that occur an odd number of times."""
    p = pairs.long()
    keys, count = torch.unique(torch.minimum(p[:, 0], p[:, 1]) * V + torch.maximum(p[:, 0], p[:, 1]),
                               return_counts=True)
    keys = keys[count % 2 == 1]
    a, b = keys // V, keys % V
    lab = torch.arange(V, device=p.device)
    while True:
        low = torch.minimum(lab[a], lab[b])
        new = lab.clone()
        new.scatter_reduce_(0, lab[a], low, "amin")
        new.scatter_reduce_(0, lab[b], low, "amin")
        while True:
            up = new[new]
            if torch.equal(up, new):
                break
            new = up
        if torch.equal(new, lab):
            return lab
        lab = new


def _answer(lab):
    lab = lab.cpu().numpy()
    return lab.astype(np.uint32), int((lab == np.arange(len(lab))).sum()), None


def exact(case, seed):
    """Component labels and counts by plain label propagation, and the planted cut.  How many Boruvka rounds
    an answer took, and sketch bytes, have no such value."""
    kind = case["kind"]
    if kind in ("phase", "query"):
        pairs = _stream(case["stream"], case["V"], case["n"], seed)
        if case.get("window"):
            pairs = torch.cat([pairs, _stream(case["stream"], case["V"], case["window"], seed + 77777)])
        return _answer(_components(pairs, case["V"]))
    if kind == "workers":
        return _answer(_components(_er(case["V"], case["n"], seed), case["V"]))
    if kind == "mincut":
        _, V, half = _planted(case, seed)
        side = np.zeros(V, np.uint8)
        side[half.cpu().numpy()] = 1
        return 3, 0, 3, side ^ side[0]
    return None
