"""Workloads of the streaming repair engine, as a program that uses it runs them.

One case is one kind of pass through the public entry points at one size:

  stream   one engine (SSSP / BFS / CC / PageRank), fed snapshot after snapshot of
           edge deletions and insertions; a pass applies `snapshots` of them one
           call each (Engine.apply_batch) and reads the results once, as the
           hybrid_* sample drivers do (they apply their batches and gather).
  batched  many SSSP / BFS sources on one graph; a pass replays `snapshots`
           snapshots of uneven size in one call (Engine.apply_batches) and reads
           the results of eight of the sources.
  infer    the admission network over every cache page (mlp_infer).
  grad     loss and gradient of the network over a batch of traced pages
           (mlp_loss_grad), one training step's forward and backward.
  group    an update batch grouped by (u, v) with multiplicities and per-segment
           counts, on device buffers (dycg_group_updates).

A stream's snapshots are all different: the program walks through `STREAM` of them
and then back, each undone by its mirror image (what was inserted is deleted, what
was deleted is inserted again), so that a pass can be repeated without end and the
graph keeps its size. Graphs are R-MAT (a=.57 b=.19 c=.19, self-loops and
duplicates removed) or road-like grids (4 neighbours both ways, 1% shortcuts
within radius 8); deletions are live edges drawn uniformly, insertions R-MAT
draws (new shortcuts on the grid), half of each. The weight of (u, v) is a hash
of its endpoints, so parallel occurrences agree.
"""
import ctypes

import numpy as np
import torch

import dycgraph_b200 as dg

STREAM_RECORDS = 1_500_000  # records a state's stream holds at most
MAX_STREAM = 64             # snapshots a state's stream holds at most
READ = 8                    # sources whose results a batched pass reads


def listed():
    return [
        # a handful of edges at a time on a small graph without a page cache:
        # the latency of one call
        {"name": "sssp tiny updates", "kind": "stream", "algo": "sssp", "weights": "stored",
         "n": 65536, "edge_factor": 16, "updates": 32, "budget_kb": 0, "snapshots": 1},
        # the small configuration of the workload table (R-MAT 16, 1,000 inserts +
        # 1,000 deletes, cache 0)
        {"name": "sssp r16 2k", "kind": "stream", "algo": "sssp", "weights": "stored",
         "n": 65536, "edge_factor": 16, "updates": 2000, "budget_kb": 0, "snapshots": 4},
        # ordinary snapshots on a graph several times its HBM budget, the
        # reference's weight rules (values and parents are both determined)
        {"name": "bfs r20 10k", "kind": "stream", "algo": "bfs", "weights": "hash128",
         "n": 1 << 20, "edge_factor": 16, "updates": 10_000, "budget_kb": 65_536, "snapshots": 4},
        # the large snapshots of the out-of-memory configuration (100K updates,
        # weights 1..64 in every slot), budget about an eighth of the graph
        {"name": "sssp r21 100k", "kind": "stream", "algo": "sssp", "weights": "stored",
         "n": 1 << 21, "edge_factor": 16, "updates": 100_000, "budget_kb": 196_608, "snapshots": 8},
        # connected components: symmetrised graph and batches, a vertex count that
        # is no power of two
        {"name": "cc 500k 20k", "kind": "stream", "algo": "cc", "weights": "hash128",
         "n": 500_003, "edge_factor": 8, "updates": 20_000, "budget_kb": 16_384, "snapshots": 4},
        # PageRank, epsilon 1e-4
        {"name": "pagerank r18 10k", "kind": "stream", "algo": "pr", "weights": "hash128",
         "n": 1 << 18, "edge_factor": 16, "updates": 10_000, "budget_kb": 8_192, "snapshots": 2},
        # high-diameter graph, ordered closure (the road-like configuration, 1/16 of
        # its vertices and budget)
        {"name": "grid sssp 1024", "kind": "stream", "algo": "sssp", "weights": "stored",
         "n": 1024 * 1024, "edge_factor": 0, "updates": 1000, "budget_kb": 24_576,
         "snapshots": 1},
        # few sources, small graph: the replayed graphs' launches and barriers count
        {"name": "batched bfs q40", "kind": "batched", "algo": "bfs", "weights": "hash128",
         "n": 65536, "edge_factor": 16, "queries": 40, "least": 100, "most": 4000,
         "budget_kb": 0, "policy": "none", "snapshots": 8},
        # the headline configuration's form (256 sources, uneven snapshots, learned
        # admission), on a smaller graph
        {"name": "batched sssp q256", "kind": "batched", "algo": "sssp", "weights": "stored",
         "n": 1 << 18, "edge_factor": 16, "queries": 256, "least": 1000, "most": 100_000,
         "budget_kb": 32_768, "policy": "learned", "snapshots": 8},
        # network over the pages of the R-MAT 27 workload
        {"name": "mlp infer 1.85M pages", "kind": "infer", "pages": 1_850_000},
        # one minibatch of the training the benchmark does
        {"name": "mlp grad 8192", "kind": "grad", "samples": 8192},
        # the largest update batch of the workload table
        {"name": "group 1M records", "kind": "group", "records": 1_000_000, "n": 1 << 24,
         "segments": 512},
    ]


def _log(rng, lo, hi):
    """An integer whose logarithm is uniform over [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the same ranges: any vertex count, batch size, budget, source
    count and buffer size between the smallest and the largest in use."""
    kind = rng.choice(["stream", "stream", "stream", "grid", "batched", "batched", "infer", "grad",
                       "group"])
    if kind == "stream":
        algo, weights = rng.choice([("sssp", "stored"), ("sssp", "hash128"), ("bfs", "hash128"),
                                    ("cc", "hash128"), ("pr", "hash128")])
        n = _log(rng, 2000, 400_000 if algo == "pr" else 1_000_000)
        ef = rng.choice([4, 8, 16])
        updates = _log(rng, 2, max(4, min(60_000, n * ef // 16)))
        graph_kb = n * ef * (8 if weights == "stored" else 4) // 1024
        return {"kind": "stream", "algo": algo, "weights": weights, "n": n, "edge_factor": ef,
                "updates": updates, "budget_kb": int(graph_kb * rng.choice([0, 0.25, 0.5, 2])),
                "snapshots": rng.choice([1, 2, 4])}
    if kind == "grid":
        algo, weights = rng.choice([("sssp", "stored"), ("bfs", "hash128")])
        side = _log(rng, 40, 700)
        return {"kind": "stream", "algo": algo, "weights": weights, "n": side * side,
                "edge_factor": 0, "updates": _log(rng, 4, max(8, side * side // 1000)),
                "budget_kb": int(side * side // 32 * rng.choice([0, 0.5, 2])), "snapshots": 1}
    if kind == "batched":
        algo, weights = rng.choice([("sssp", "stored"), ("sssp", "hash128"), ("bfs", "hash128")])
        n = _log(rng, 2000, 130_000)
        policy = rng.choice(["none", "hotness", "learned"])
        least = _log(rng, 4, 1000)
        return {"kind": "batched", "algo": algo, "weights": weights, "n": n,
                "edge_factor": rng.choice([8, 16]), "queries": _log(rng, 1, 256), "least": least,
                "most": _log(rng, least, max(least, n // 4)),
                "budget_kb": 0 if policy == "none" else max(2048, n // 8), "policy": policy,
                "snapshots": rng.choice([1, 3, 8])}
    if kind == "infer":
        return {"kind": "infer", "pages": _log(rng, 1, 1_850_000)}
    if kind == "grad":
        return {"kind": "grad", "samples": _log(rng, 1, 200_000)}
    return {"kind": "group", "records": _log(rng, 1, 1_000_000), "n": _log(rng, 1000, 1 << 27),
            "segments": rng.choice([0, 1, 37, 512])}


# ---- inputs ----------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 2654435761 % (1 << 62))
    return g


def _rmat(n, count, gen):
    """`count` R-MAT draws over n vertices, no self-loops."""
    scale = max(1, (n - 1).bit_length())
    u = torch.zeros(count, dtype=torch.int64, device="cuda")
    v = torch.zeros(count, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(count, device="cuda", generator=gen)
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    u, v = u % n, v % n
    return u, torch.where(u == v, (v + 1) % n, v)


def _weights(u, v, most):
    x = (u * 0x9E3779B1 + v * 0x85EBCA77) & 0xFFFFFFFF
    x = ((x ^ (x >> 15)) * 0x2C1B3C6D) & 0xFFFFFFFF
    return 1 + (x ^ (x >> 12)) % most


def _shortcuts(side, count, gen):
    """Vertex pairs within radius 8 of each other on a side x side grid."""
    n = side * side
    u = torch.randint(0, n, (count,), device="cuda", generator=gen)
    dr = torch.randint(-8, 9, (count,), device="cuda", generator=gen)
    dc = torch.randint(-8, 9, (count,), device="cuda", generator=gen)
    v = (u // side + dr).clamp(0, side - 1) * side + (u % side + dc).clamp(0, side - 1)
    return u, torch.where(u == v, (u + 1) % n, v)


def _edges(case, gen):
    """Distinct directed edges (u * n + v) of the initial graph, ascending."""
    n, ef = case["n"], case["edge_factor"]
    if ef:
        u, v = _rmat(n, n * ef, gen)
        key = u * n + v
        if case["algo"] == "cc":
            key = torch.cat([key, v * n + u])
        return torch.unique(key)
    side = int(round(n ** 0.5))
    i = torch.arange(n, device="cuda")
    right, down = i[i % side < side - 1], i[i < n - side]
    a, b = _shortcuts(side, n // 100, gen)
    u = torch.cat([right, right + 1, down, down + side, a, b])
    v = torch.cat([right + 1, right, down + side, down, b, a])
    return torch.unique(u * n + v)


def _records(case, key):
    """Update records (u, v, w) of edges given as u * n + v."""
    n = case["n"]
    u, v = key // n, key % n
    w = _weights(u, v, 64 if case["edge_factor"] else 1000)
    return torch.stack([u, v, w], 1).cpu().numpy().astype(np.uint32)


def _mirrored(key, n):
    return torch.stack([key, key % n * n + key // n], 1).reshape(-1)


def _graph(case, seed):
    """(edge keys, weights per edge): the initial graph."""
    gen = _generator(seed)
    key = _edges(case, gen)
    n = case["n"]
    return gen, key, _weights(key // n, key % n, 64 if case["edge_factor"] else 1000)


def _stream(case, gen, key, sizes):
    """Snapshots [(deletion keys, insertion keys)] of the given sizes: deletions are
    distinct live edges of the initial graph, insertions draws of its generator; CC
    snapshots carry both directions of every edge."""
    n, cc = case["n"], case["algo"] == "cc"
    pool = key[key // n < key % n] if cc else key
    halves = [max(1, s // (4 if cc else 2)) for s in sizes]
    pick = pool[torch.randperm(len(pool), device="cuda", generator=gen)[:sum(halves)]]
    if case["edge_factor"]:
        u, v = _rmat(n, sum(halves), gen)
    else:
        u, v = _shortcuts(int(round(n ** 0.5)), sum(halves), gen)
    new = u * n + v
    out, at = [], 0
    for h in halves:
        d, a = pick[at:at + h], new[at:at + h]
        out.append((_mirrored(d, n), _mirrored(a, n)) if cc else (d, a))
        at += h
    return out


def _csr(case, key, w):
    n = case["n"]
    off = np.zeros(n + 1, np.uint64)
    off[1:] = torch.bincount(key // n, minlength=n).cumsum(0).cpu().numpy()
    dst = (key % n).cpu().numpy().astype(np.uint32)
    return off, dst, w.cpu().numpy().astype(np.uint32) if case["weights"] == "stored" else None


def _length(case, largest, edges):
    """Snapshots in a state's stream: at most MAX_STREAM, an eighth of the edges."""
    return max(2 * case["snapshots"],
               min(MAX_STREAM, STREAM_RECORDS // largest, edges // (4 * largest)))


class Walk:
    """Snapshots of a stream forward, then their mirror images backward, and so on."""

    def __init__(self, snapshots):
        self.snapshots, self.at, self.back = snapshots, 0, False

    def next(self):
        if self.back:
            self.at -= 1
            adds, dels = self.snapshots[self.at]
            self.back = self.at > 0
        else:
            dels, adds = self.snapshots[self.at]
            self.at += 1
            self.back = self.at == len(self.snapshots)
        return dels, adds


def _engine(case, key, w):
    policy = case.get("policy") or ("hotness" if case["budget_kb"] else "none")
    grid = not case["edge_factor"]
    # a stream that goes on: room for the rows' growth
    e = dg.Engine(case["algo"], weight_mode=case["weights"], cache_policy=policy,
                  hbm_graph_budget_bytes=case["budget_kb"] * 1024, symmetric=case["algo"] == "cc",
                  epsilon=1e-4, arena_headroom_permille=1000,
                  ordered_delta=(2048 if case["algo"] == "sssp" else 1) if grid else 0)
    off, dst, ww = _csr(case, key, w)
    e.load_csr(case["n"], off, dst, ww)
    return e, off


def _prepare_stream(case, seed):
    gen, key, w = _graph(case, seed)
    count = _length(case, case["updates"], len(key))
    keys = _stream(case, gen, key, [case["updates"]] * count)
    e, _ = _engine(case, key, w)
    e.start()
    e.reserve_batch(case["updates"])
    return {"case": case, "engine": e,
            "walk": Walk([(_records(case, d), _records(case, a)) for d, a in keys])}


def _sizes(case, count, seed):
    """Snapshot sizes, uniform in their logarithm over [least, most]."""
    r = np.random.default_rng(seed).random(count)
    return [int(round(case["least"] * (case["most"] / case["least"]) ** x)) for x in r]


def _prepare_batched(case, seed):
    gen, key, w = _graph(case, seed)
    count = _length(case, case["most"], len(key))
    sizes = _sizes(case, count, seed)
    keys = _stream(case, gen, key, sizes)
    e, off = _engine(case, key, w)
    rows = np.nonzero(np.diff(off.astype(np.int64)) > 0)[0]
    pick = np.random.default_rng(seed + 1).choice(rows, size=min(case["queries"], len(rows)),
                                                  replace=False)
    e.set_queries(pick.astype(np.uint32), "batched")
    e.start()
    walk = Walk([(_records(case, d), _records(case, a)) for d, a in keys])
    # what a program does once: tune the work mapping on one snapshot, record and
    # train the admission network, capture the replay graphs
    e.tune_query_mapping(*walk.next())
    if case["policy"] == "learned":
        e.policy_trace(3)
        for _ in range(5):
            e.apply_batch(*walk.next())
        e.policy_train(1, 2e-3, 2048, 1)
    e.reserve_batch(max(sizes))
    return {"case": case, "engine": e, "walk": walk, "queries": len(pick)}


def _pages(count, gen):
    """Feature rows with the ranges of the engine's page features (log counts, ages)."""
    x = torch.rand((count, 8), device="cuda", generator=gen)
    x = x * torch.tensor([8., 8., 8., 9., 6., 1., .8, .7], device="cuda")
    x = torch.where(torch.rand((count, 8), device="cuda", generator=gen) < 0.3,
                    torch.zeros_like(x), x)
    return x.to(torch.bfloat16)


def _params(gen):
    """Network parameters W1[8x64] b1[64] W2[64x64] b2[64] W3[64] b3."""
    p = []
    for i, o in ((8, 64), (64, 64), (64, 1)):
        a = (6.0 / (i + o)) ** 0.5
        p.append((torch.rand(i * o, device="cuda", generator=gen) * 2 - 1) * a)
        p.append((torch.rand(o, device="cuda", generator=gen) - 0.5) * 0.2)
    return torch.cat(p).float()


def _prepare_network(case, seed):
    gen = _generator(seed)
    if case["kind"] == "infer":
        return {"case": case, "x": _pages(case["pages"], gen), "p": _params(gen),
                "out": torch.zeros(case["pages"], device="cuda")}
    k = case["samples"]
    return {"case": case, "x": _pages(k, gen), "p": _params(gen),
            "y": torch.rand(k, device="cuda", generator=gen) * 9,
            "grad": torch.zeros(dg.POLICY_PARAMS, device="cuda"),
            "loss": torch.zeros(1, device="cuda")}


def _prepare_group(case, seed):
    gen = _generator(seed)
    k, n, s = case["records"], case["n"], case["segments"]
    u, v = _rmat(n, k, gen)
    # a few repeated records and a few with an endpoint that does not exist
    back = torch.randint(0, 50, (k,), device="cuda", generator=gen)
    at = (torch.arange(k, device="cuda") - torch.where(back < 3, back, 0)).clamp(min=0)
    u, v = u[at], v[at]
    v = torch.where(torch.rand(k, device="cuda", generator=gen) < 0.001, v + n, v)
    rec = torch.stack([u, v, torch.ones_like(u)], 1).to(torch.int32).contiguous()
    ends = torch.tensor([(n * (i + 1)) // s for i in range(s)] or [n], device="cuda")
    z = lambda m: torch.zeros(m, dtype=torch.int32, device="cuda")  # noqa: E731
    return {"case": case, "rec": rec, "ends": ends.to(torch.int32), "uv": z(2 * k), "mult": z(k),
            "seg": z(max(1, s)), "counts": z(2)}


def prepare(case, seed):
    if case["kind"] == "stream":
        return _prepare_stream(case, seed)
    if case["kind"] == "batched":
        return _prepare_batched(case, seed)
    if case["kind"] == "group":
        return _prepare_group(case, seed)
    return _prepare_network(case, seed)


# ---- passes ----------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "stream":
        e, walk = state["engine"], state["walk"]
        for _ in range(case["snapshots"]):
            e.apply_batch(*walk.next())
        if case["algo"] == "pr":
            return e.gather_ranks()[0]
        values, parents = e.gather()
        # with stored weights and for CC any tight parent may be recorded
        return (values, parents) if case["weights"] == "hash128" and case["algo"] != "cc" \
            else values
    if kind == "batched":
        e, walk, q = state["engine"], state["walk"], state["queries"]
        e.apply_batches([walk.next() for _ in range(case["snapshots"])])
        return [e.gather_query(i * q // READ)[0] for i in range(READ) if i < q]
    if kind == "infer":
        dg.mlp_infer(state["x"].data_ptr(), case["pages"], state["p"].data_ptr(),
                     state["out"].data_ptr())
        return state["out"]
    if kind == "grad":
        state["grad"].zero_()
        state["loss"].zero_()
        dg.mlp_loss_grad(state["x"].data_ptr(), state["y"].data_ptr(), case["samples"],
                         state["p"].data_ptr(), state["grad"].data_ptr(),
                         state["loss"].data_ptr())
        return state["grad"], state["loss"]
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rc = dg.lib().dycg_group_updates(ptr(state["rec"]), case["records"], case["n"],
                                     ptr(state["ends"]), case["segments"], ptr(state["uv"]),
                                     ptr(state["mult"]), ptr(state["seg"]), ptr(state["counts"]),
                                     None)
    if rc:
        raise dg.DycgError(rc, "dycg_group_updates")
    return state["uv"], state["mult"], state["seg"], state["counts"]


def work(case):
    """Bytes and operations a pass cannot do without. Stream and batched passes: every
    record read once and stored in its row(s), the results written once; what the
    repair itself has to read depends on the graph and is not counted."""
    kind = case["kind"]
    if kind == "infer":
        return {"bytes": case["pages"] * 20.0, "flops": case["pages"] * 2.0 * (8 * 64 + 64 * 64 + 64)}
    if kind == "grad":
        return {"bytes": case["samples"] * 20.0 + 2 * 4 * 4801,
                "flops": case["samples"] * 6.0 * (8 * 64 + 64 * 64 + 64)}
    if kind == "group":
        return {"bytes": case["records"] * 24.0, "flops": 0}
    rows = 1 if case["algo"] in ("pr", "cc") else 2
    slot = 8 if case["weights"] == "stored" else 4
    if kind == "stream":
        records = case["updates"] * case["snapshots"]
        return {"bytes": records * (12.0 + rows * slot) + case["n"] * 4.0, "flops": 0}
    mean = (case["most"] - case["least"]) / max(1e-9, np.log(case["most"] / case["least"])) \
        if case["most"] > case["least"] else case["most"]
    return {"bytes": mean * case["snapshots"] * (12.0 + rows * slot)
            + min(READ, case["queries"]) * case["n"] * 4.0, "flops": 0}


# ---- the same results in 64 bits ----------------------------------------------------


def _ranks(case, seed):
    """Fixed point of x = 0.15 + 0.85 P^T x on the graph after the first pass."""
    gen, key, _ = _graph(case, seed)
    n = case["n"]
    walk = Walk(_stream(case, gen, key, [case["updates"]] * _length(case, case["updates"], len(key))))
    for _ in range(case["snapshots"]):
        dels, adds = walk.next()
        alive = torch.cat([key, adds])
        kinds, count = torch.unique(alive, return_counts=True)
        gone, times = torch.unique(dels, return_counts=True)
        count[torch.searchsorted(kinds, gone)] -= times
        key = torch.repeat_interleave(kinds, count)
    u, v = key // n, key % n
    share = 0.85 / torch.bincount(u, minlength=n).clamp(min=1).double()
    x = torch.full((n,), 0.15, dtype=torch.float64, device="cuda")
    for _ in range(250):
        x = torch.full_like(x, 0.15).index_add_(0, v, (x * share)[u])
    return x


def _network(p):
    p = p.to(torch.bfloat16).double()
    at, out = 0, []
    for shape in ((8, 64), (64,), (64, 64), (64,), (64, 1), (1,)):
        size = int(np.prod(shape))
        out.append(p[at:at + size].reshape(shape))
        at += size
    return out


def exact(case, seed):
    if case["kind"] == "stream" and case["algo"] == "pr":
        return _ranks(case, seed)
    if case["kind"] not in ("infer", "grad"):
        return None  # whole numbers
    s = _prepare_network(case, seed)
    layers = [t.requires_grad_() for t in _network(s["p"])]
    w1, b1, w2, b2, w3, b3 = layers
    x = s["x"].double()
    if case["kind"] == "infer":
        with torch.no_grad():
            return ((x @ w1 + b1).relu() @ w2 + b2).relu().matmul(w3).add(b3)[:, 0]
    y = ((x @ w1 + b1).relu() @ w2 + b2).relu().matmul(w3).add(b3)[:, 0]
    loss = (y - s["y"].double()).square().sum()
    grads = torch.autograd.grad(loss, layers)
    return torch.cat([g.reshape(-1) for g in grads]), loss.detach().reshape(1)
