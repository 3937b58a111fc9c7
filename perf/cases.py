"""The work that users of the engine have it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what a user's program holds before the call
(resident graphs with their trees, change records and read buffers in pinned host memory, a pool
or a server), `run` makes one pass through the public entry points and returns its outputs.

Batches come as a stream: a pass applies a batch B and then its inverse (B's insertions deleted,
its deletions inserted again, a valid batch of the same size), and reads the whole updated tree
after each, so a pass can be repeated on the same resident graph and the rows see the churn that a
program in service sees: tombstones, unsorted row tails, rows that run out of slack.  All weights
are positive, which makes parents as well as distances a function of the graph alone (the least
tight neighbour).  Inputs are drawn on the GPU from the seed.
"""
import math
import random

import numpy as np
import torch

import dynamicssspv2_gb300 as D
from dynamicssspv2_gb300.pool import GraphPool
from dynamicssspv2_gb300.serve import Request, Server, Tenant

RMAT = (0.57, 0.19, 0.19)


def listed():
    return [
        # a monitoring loop over a small network: a handful of changes per call, all launch and latency
        dict(name="er_tiny", kind="update", graph="er", n=2003, m=8009, k=17, ins=0.5, whi=100, records="host"),
        # the plain method on the small configuration: 10,000 vertices, 1,000 changes
        dict(name="er_10k", kind="update", graph="er", n=10_000, m=50_000, k=1000, ins=0.5, whi=100, records="host"),
        # one tenant-sized graph with odd sizes, its records produced on the device
        dict(name="er_300k", kind="update", graph="er", n=300_007, m=1_200_041, k=12_345, ins=0.5, whi=100,
             records="device"),
        # a growing social graph: only insertions, then only deletions (the inverse)
        dict(name="rmat_20_grow", kind="update", graph="rmat", n=1 << 20, m=8_388_608, k=100_003, ins=1.0, whi=100,
             records="host"),
        # the plain method on the large skewed configuration: a stream of 10^6-change batches
        dict(name="rmat_22", kind="update", graph="rmat", n=1 << 22, m=33_554_432, k=1_000_000, ins=0.5, whi=100,
             records="host"),
        # a city's road network, ragged sides, closures more than openings
        dict(name="grid_1021", kind="update", graph="grid", n=1021 * 1543, cols=1543, k=9_001, ins=0.25, whi=1000,
             records="host"),
        # the high-diameter configuration: deep cut-off subtrees, thousands of relaxation rounds
        dict(name="grid_4096", kind="update", graph="grid", n=4096 * 4096, cols=4096, k=100_000, ins=0.25, whi=1000,
             records="host"),
        # many uneven graphs, each with its own batch, in one launch sequence
        dict(name="pool_64", kind="pool", count=64, nlo=3.0, nhi=5.5, flo=-3.0, fhi=-1.0),
        # a saturated server: every tenant with requests of mixed sizes waiting
        dict(name="serve_9", kind="serve", scale=20, m=8_388_608, tenants=8, nlo=4.5, nhi=5.5, requests=96, blo=1.0,
             bhi=4.0),
        # the initial tree of a large skewed graph
        dict(name="compute_rmat_22", kind="compute", graph="rmat", n=1 << 22, m=33_554_432, whi=100),
        # the initial tree of a road network
        dict(name="compute_grid_2048", kind="compute", graph="grid", n=2048 * 2048, cols=2048, whi=1000),
        # a plugin's call on its own CSR arrays, no device allocation
        dict(name="noalloc_30k", kind="noalloc", n=30_000, m=150_000, whi=100),
    ]


def _odd(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(int(lo), min(int(hi), int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["update", "update", "update", "update", "pool", "serve", "compute", "noalloc"])
    graph = rng.choice(["er", "rmat", "grid"])
    if kind in ("update", "compute"):
        if graph == "er":
            n = _odd(rng, 1000, 1_000_000)
            c = dict(kind=kind, graph=graph, n=n, m=int(n * rng.uniform(3.0, 8.0)), whi=100)
        elif graph == "rmat":
            n = 1 << rng.randint(12, 21)
            c = dict(kind=kind, graph=graph, n=n, m=int(n * rng.uniform(4.0, 8.0)), whi=100)
        else:
            cols = _odd(rng, 64, 2000)
            rows = _odd(rng, 64, 2000)
            c = dict(kind=kind, graph=graph, n=rows * cols, cols=cols, m=2 * rows * cols, whi=1000)
        if kind == "update":
            frac = 10.0 ** rng.uniform(-3.5, -1.3 if graph != "grid" else -2.0)
            c.update(k=max(10, int(frac * c["m"])), ins=rng.choice([0.0, 0.25, 0.5, 0.5, 1.0]),
                     records=rng.choice(["host", "device"]))
        if graph == "grid":
            del c["m"]
        return c
    if kind == "pool":
        return dict(kind=kind, count=rng.randint(8, 64), nlo=3.0, nhi=rng.uniform(4.0, 5.5), flo=-3.0, fhi=-1.0)
    if kind == "serve":
        scale = rng.randint(14, 19)
        return dict(kind=kind, scale=scale, m=rng.randint(4, 8) << scale, tenants=rng.randint(2, 8),
                    nlo=4.0, nhi=rng.uniform(4.5, 5.5), requests=rng.randint(16, 96), blo=1.0, bhi=rng.uniform(2.5, 4.0))
    n = _odd(rng, 1000, 60_000)
    return dict(kind=kind, n=n, m=int(n * rng.uniform(2.0, 8.0)), whi=100)


# ---- inputs ------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(lo, hi, k, g):
    return torch.randint(lo, hi, (k,), generator=g, device="cuda", dtype=torch.int64)


def _pairs(graph, n, cols, k, g):
    """k random vertex pairs of the graph's own distribution, as keys u * n + v with u < v (some invalid: -1)."""
    if graph == "rmat":
        u = torch.zeros(k, dtype=torch.int64, device="cuda")
        v = torch.zeros(k, dtype=torch.int64, device="cuda")
        a, b, c = RMAT
        for _ in range(n.bit_length() - 1):
            r = torch.rand(k, generator=g, device="cuda")
            u = 2 * u + (r >= a + b)
            v = 2 * v + (((r >= a) & (r < a + b)) | (r >= a + b + c))
    elif graph == "grid":  # short links: up to two rows and columns away
        u = _ints(0, n, k, g)
        y, x = u // cols + _ints(-2, 3, k, g), u % cols + _ints(-2, 3, k, g)
        v = torch.where((x >= 0) & (x < cols) & (y >= 0) & (y < n // cols), y * cols + x, u)
    else:
        u, v = _ints(0, n, k, g), _ints(0, n, k, g)
    return torch.where(u == v, -1, torch.minimum(u, v) * n + torch.maximum(u, v))


def _choose(keys, k, g):
    return keys[torch.randperm(len(keys), generator=g, device="cuda")[:k]]


def _new_pairs(graph, n, cols, k, have, g):
    """k distinct pairs, none of them in the sorted keys `have`."""
    got = torch.empty(0, dtype=torch.int64, device="cuda")
    while len(got) < k:
        c = torch.unique(torch.cat([got, _pairs(graph, n, cols, int(1.3 * (k - len(got))) + 64, g)]))
        c = c[c >= 0]
        if len(have):
            at = torch.searchsorted(have, c).clamp(max=len(have) - 1)
            c = c[have[at] != c]
        got = c
    return _choose(got, k, g)


def _edges(c, g):
    """The case's edge list: sorted pair keys and a weight each."""
    n, whi = c["n"], c["whi"]
    if c["graph"] == "grid":
        cols = c["cols"]
        at = torch.arange(n, dtype=torch.int64, device="cuda")
        right, down = at[at % cols < cols - 1], at[: n - cols]
        keys = torch.cat([right * n + right + 1, down * n + down + cols])
        keys = torch.sort(keys[torch.rand(len(keys), generator=g, device="cuda") >= 0.05])[0]
        diag = _new_pairs("grid", n, cols, n // 100, keys, g)
        keys = torch.sort(torch.cat([keys, diag]))[0]
    else:
        none = torch.empty(0, dtype=torch.int64, device="cuda")
        keys = torch.sort(_new_pairs(c["graph"], n, 0, c["m"], none, g))[0]
    return keys, _ints(1, whi + 1, len(keys), g)


def _records(u, v, w, op):
    """Change records as a 16-byte row each, on the GPU."""
    return torch.stack([u, v, w, op], dim=1).to(torch.int32).contiguous()


def _changes(c, keys, w, k, n_ins, g):
    """k change records in random order (new pairs inserted, existing edges deleted), and the inverse batch."""
    n = c["n"]
    at = torch.randperm(len(keys), generator=g, device="cuda")[: k - n_ins]
    new = _new_pairs(c["graph"], n, c.get("cols", 0), n_ins, keys, g)
    key = torch.cat([new, keys[at]])
    wt = torch.cat([_ints(1, c["whi"] + 1, n_ins, g), w[at]])
    op = torch.cat([torch.ones_like(new), torch.zeros_like(at)])
    order = torch.randperm(k, generator=g, device="cuda")
    key, wt, op = key[order], wt[order], op[order]
    back = torch.randperm(k, generator=g, device="cuda")
    return _records(key // n, key % n, wt, op), _records(key // n, key % n, wt, 1 - op)[back]


def _host(t):
    return t.to(torch.int32).cpu().numpy()


def _pinned_records(r):
    return r.cpu().pin_memory().numpy().view(D.CHANGE_DTYPE).reshape(-1)


def _pinned_tree(n):
    return [torch.empty(n, dtype=torch.int32).pin_memory().numpy() for _ in range(2)]


def _source(c, keys):
    if c["graph"] != "rmat":
        return 0
    n = c["n"]
    return int(torch.argmax(torch.bincount(torch.cat([keys // n, keys % n]), minlength=n)))


def _sizes(lo, hi, count):
    """count vertex counts spread evenly over the logarithm of [10^lo, 10^hi], large and small mixed."""
    sizes = [int(10.0 ** (lo + (hi - lo) * (i + 0.5) / count)) | 1 for i in range(count)]
    random.Random(count).shuffle(sizes)
    return sizes


def _tenant_case(n, m):
    return dict(graph="er", n=n, m=m, whi=100)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "pool":
        r = random.Random(seed)
        graphs, batches, inverse = [], [], []
        for i, n in enumerate(_sizes(case["nlo"], case["nhi"], case["count"])):
            c = _tenant_case(n, 4 * n)
            keys, w = _edges(c, g)
            k = max(2, int(10.0 ** r.uniform(case["flo"], case["fhi"]) * len(keys)))
            b, inv = _changes(c, keys, w, k, k // 2, g)
            graphs.append((n, _host(keys // n), _host(keys % n), _host(w)))
            batches.append((i, _pinned_records(b)))
            inverse.append((i, _pinned_records(inv)))
        pool = GraphPool(graphs, slack_pct=50, slack_min=16)
        pool.tree_compute([0] * len(graphs))
        return dict(kind=kind, pool=pool, batches=[batches, inverse], trees=[_pinned_tree(pool.n) for _ in range(2)])
    if kind == "serve":
        r = random.Random(seed)
        cs = [dict(graph="rmat", n=1 << case["scale"], m=case["m"], whi=100)]
        cs += [_tenant_case(n, 4 * n) for n in _sizes(case["nlo"], case["nhi"], case["tenants"])]
        share = [[_odd(r, 10 ** case["blo"], 10 ** case["bhi"]) for _ in range(i, case["requests"], len(cs))]
                 for i in range(len(cs))]
        tenants, first, second = [], [], []
        for t, (c, sizes) in enumerate(zip(cs, share)):
            keys, w = _edges(c, g)
            n, k = c["n"], sum(sizes)
            b, inv = _changes(c, keys, w, k, k // 2, g)
            tenants.append(Tenant(f"t{t}", n, _host(keys // n), _host(keys % n), _host(w), _source(c, keys)))
            cuts = np.cumsum(sizes)[:-1]
            for i, (x, y) in enumerate(zip(np.split(_pinned_records(b), cuts), np.split(_pinned_records(inv), cuts))):
                first.append((i, t, x))
                second.append((i, t, y))
        first.sort(key=lambda x: x[:2])  # the tenants' requests arrive in turn
        second.sort(key=lambda x: x[:2])
        return dict(kind=kind, server=Server(tenants), requests=[[(t, ch) for _, t, ch in rs] for rs in (first, second)])
    if kind == "noalloc":
        c = dict(case, graph="er")
        n = c["n"]
        keys, w = _edges(c, g)
        u, v = torch.cat([keys // n, keys % n]), torch.cat([keys % n, keys // n])
        order = torch.argsort(u * n + v)
        off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        off[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
        adj = torch.stack([v[order], torch.cat([w, w])[order]], dim=1).to(torch.int32).contiguous()
        return dict(kind=kind, n=n, off=off, adj=adj, src=n // 2, stream=torch.cuda.current_stream().cuda_stream,
                    parent=torch.empty(n, dtype=torch.int32, device="cuda"),
                    dist=torch.empty(n, dtype=torch.int64, device="cuda"))
    n = case["n"]
    keys, w = _edges(case, g)
    src = _source(case, keys)
    graph = D.Graph(n, _host(keys // n), _host(keys % n), _host(w))
    if kind == "compute":
        return dict(kind=kind, graph=graph, src=src, tree=_pinned_tree(n))
    k = case["k"]
    pair = _changes(case, keys, w, k, int(round(k * case["ins"])), g)
    graph.tree_compute(src)
    host = case["records"] == "host"
    return dict(kind=kind, graph=graph, host=host, batches=[_pinned_records(b) if host else b for b in pair],
                trees=[_pinned_tree(n) for _ in range(2)])


# ---- passes ------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "update":
        graph, out = state["graph"], []
        for batch, (parent, dist) in zip(state["batches"], state["trees"]):
            if state["host"]:
                graph.apply_batch(batch)
            else:
                graph.apply_batch_async(batch.data_ptr(), len(batch))
                graph.batch_finish()
            graph.tree_read32(parent, dist)
            out += [parent, dist]
        return out
    if kind == "pool":
        out = []
        for batches, (parent, dist) in zip(state["batches"], state["trees"]):
            state["pool"].apply(batches)
            state["pool"].graph.tree_read32(parent, dist)
            out += [parent, dist]
        return out
    if kind == "serve":
        srv, out = state["server"], []
        for requests in state["requests"]:
            srv.serve([Request(t, 0.0, ch) for t, ch in requests], realtime=False)
            for t in range(len(srv.tenants)):
                out += srv.tree(t)
        return out
    if kind == "compute":
        state["graph"].tree_compute(state["src"])
        state["graph"].tree_read32(*state["tree"])
        return state["tree"]
    D.sssp_noalloc(state["n"], len(state["adj"]), state["off"].data_ptr(), state["adj"].data_ptr(), state["src"],
                   state["parent"].data_ptr(), state["dist"].data_ptr(), state["stream"])
    return [state["parent"], state["dist"]]


def work(case):
    """Bytes that a pass cannot do without: records read, matching entries found and marked or placed at
    both ends, and the tree read from the state and written to its buffers; for a tree from scratch (and a
    road network's batch, which cuts off almost every vertex) the whole adjacency and state once."""
    kind = case["kind"]
    if kind == "noalloc":
        return dict(bytes=8 * (case["n"] + 1) + 16 * case["m"] + 12 * case["n"], flops=0)
    if kind == "pool":
        span = math.log(10.0) * (case["nhi"] - case["nlo"])
        n = case["count"] * (10.0 ** case["nhi"] - 10.0 ** case["nlo"]) / span
        frac = (10.0 ** case["fhi"] - 10.0 ** case["flo"]) / (math.log(10.0) * (case["fhi"] - case["flo"]))
        return dict(bytes=2 * (48 * frac * 4 * n + 16 * n), flops=0)
    if kind == "serve":
        mean = lambda lo, hi: (10.0 ** hi - 10.0 ** lo) / (math.log(10.0) * (hi - lo))  # noqa: E731
        n = (1 << case["scale"]) + case["tenants"] * mean(case["nlo"], case["nhi"])
        return dict(bytes=2 * (48 * case["requests"] * mean(case["blo"], case["bhi"]) + 20 * n), flops=0)
    n = case["n"]
    m = case.get("m", 1.91 * n)
    whole = 16 * m + 8 * n
    if kind == "compute":
        return dict(bytes=whole + 16 * n, flops=0)
    return dict(bytes=2 * (48 * case["k"] + 16 * n + (whole if case["graph"] == "grid" else 0)), flops=0)


# ---- the same results by plain tensor operations --------------------------------------------------

def _tree64(n, keys, w, src):
    """(parent, dist) by sweeps over all edges in 64 bits: dist -1 and parent -1 where unreachable."""
    far = 1 << 60
    u, v = torch.cat([keys // n, keys % n]), torch.cat([keys % n, keys // n])
    w = torch.cat([w, w])
    dist = torch.full((n,), far, dtype=torch.int64, device="cuda")
    dist[src] = 0
    while True:
        new = dist.scatter_reduce(0, v, dist[u] + w, "amin")
        if torch.equal(new, dist):
            break
        dist = new
    tight = (dist[u] + w == dist[v]) & (dist[u] < far)
    parent = torch.full((n,), n, dtype=torch.int64, device="cuda").scatter_reduce(0, v[tight], u[tight], "amin")
    parent[src] = src
    gone = dist >= far
    return torch.where(gone, -1, parent), torch.where(gone, -1, dist)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pool", "serve") or (case.get("graph") == "grid" and case["n"] > 300_000):
        return None  # many graphs, or thousands of sweeps: too long here
    g = _gen(seed)
    n = case["n"]
    c = case if kind != "noalloc" else dict(case, graph="er")
    keys, w = _edges(c, g)
    if kind == "noalloc":
        return list(_tree64(n, keys, w, n // 2))
    src = _source(c, keys)
    before = list(_tree64(n, keys, w, src))
    if kind == "compute":
        return before
    k = case["k"]
    batch = _changes(c, keys, w, k, int(round(k * case["ins"])), g)[0].to(torch.int64)
    ins, gone = batch[batch[:, 3] == 1], batch[batch[:, 3] == 0]
    kept = ~torch.isin(keys, gone[:, 0] * n + gone[:, 1])
    keys = torch.cat([keys[kept], ins[:, 0] * n + ins[:, 1]])
    return list(_tree64(n, keys, torch.cat([w[kept], ins[:, 2]]), src)) + before
