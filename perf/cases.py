"""Workloads for timing this framework through its public calls.

A case is one piece of work a user's program gives a resident graph: BFS or SSSP queries, the
layer builds, an update batch, or a batch followed by queries. Graphs are the two shapes the
benchmark uses, drawn here on the GPU from a seed:

  rmat     R-MAT (a, b, c = .57, .19, .19), ids permuted: a power-law graph with one giant SCC
  lattice  side x side 4-neighbour lattice, 5% of its edges removed, 0.1% long-range edges with
           Pareto(1.5) lengths, weights 100 x length + U[0, 50]: a high-diameter, road-like graph

Update cases apply a batch and then the batch that undoes it, so a pass leaves the graph as it
found it and can be run again.
"""
import importlib
import math

import numpy as np
import torch

gir = importlib.import_module("graph-intermedia-representation_b200")
native = gir.native

_LABELS = (native.LABEL_WCC, native.LABEL_SCC, native.LABEL_SCC_RANK, native.LABEL_BLOCK, native.LABEL_BCNT)
INF = -1  # an unreachable distance (UINT64_MAX) in an int64 tensor


def _rmat(name, kind, V, E, **kw):
    return {"name": name, "kind": kind, "graph": "rmat", "V": V, "E": E, **kw}


def _lattice(name, kind, side, **kw):
    return {"name": name, "kind": kind, "graph": "lattice", "V": side * side, "E": _lattice_edges(side), **kw}


def _lattice_edges(side):
    """About how many directed edges a lattice of this side gets (drawn with chance)."""
    return 2 * int(0.951 * 2 * side * (side - 1))


def listed():
    return [
        # An interactive single-source query on a small graph, result as a host array: latency.
        _rmat("bfs_one_small", "bfs", 4096, 65_000, lanes=1, host=True),
        # The benchmark's BFS half: 64 sources on the LiveJournal-shaped graph, rows kept on the device.
        _rmat("bfs_64_large", "bfs", 4_800_000, 69_000_000, lanes=64, host=False),
        # Multi-source queries of uneven sizes (log-uniform in [1, 4096]), an odd number of them.
        _rmat("bfs_sets", "bfs", 777_777, 12_300_001, lanes=37, sets=4096, host=False),
        # Road-like graph: thousands of small levels.
        _lattice("bfs_lattice", "bfs", 701, lanes=8, host=False),
        # An interactive shortest-path query with the graph's own weights, result on the host.
        _rmat("sssp_one_medium", "sssp", 65_536, 1_000_000, lanes=1, delta=16, stored=True, learned=False, host=True),
        # The benchmark's SSSP half: 64 sources, hash weights, the default bucket width.
        _rmat("sssp_64_large", "sssp", 4_800_000, 69_000_000, lanes=64, delta=16, stored=False, learned=False,
              host=False),
        # Route lengths on a road-like graph, bucket width from the schedule network.
        _lattice("sssp_lattice", "sssp", 901, lanes=16, delta=0, stored=True, learned=True, host=False),
        # Every layer of the large power-law graph from scratch.
        _rmat("build_large", "build", 4_800_000, 69_000_000),
        # The same of a road-like graph: deep spanning forest, many blocks.
        _lattice("build_lattice", "build", 803),
        # A large update batch, half inserts and half deletions, every layer kept exact.
        _rmat("update_large", "update", 4_800_000, 69_000_000, ops=100_000),
        # A small batch on a medium graph: mostly launches and host work.
        _rmat("update_medium", "update", 65_536, 1_000_000, ops=1_000),
        # Streaming: an update batch, then BFS and SSSP queries on the changed graph.
        _rmat("stream", "stream", 1_048_576, 16_000_000, ops=200_000, lanes=32, delta=16, stored=False, learned=False),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["bfs", "bfs", "sssp", "sssp", "build", "update", "stream"])
    if rng.random() < 0.3 and kind != "stream":
        c = _lattice("", kind, logint(40, 700))
    else:
        V = logint(2_000, 3_000_000)
        c = _rmat("", kind, V, int(V * rng.uniform(4.0, 16.0)))
    del c["name"]
    small = c["V"] < 300_000
    if kind in ("bfs", "sssp", "stream"):
        c["lanes"] = logint(1, 64)
        if c["V"] < 30_000 and rng.random() < 0.3:
            c["lanes"] += 64  # a second lane group
        if kind != "stream":
            c["host"] = small and c["lanes"] <= 4
        if kind == "bfs" and rng.random() < 0.3:
            c["sets"] = logint(2, min(4096, c["V"]))
    if kind in ("sssp", "stream"):
        lattice = c["graph"] == "lattice"
        c["stored"] = kind == "sssp" and rng.random() < 0.5
        c["learned"] = lattice and rng.random() < 0.5
        c["delta"] = 0 if c["learned"] else rng.choice([2048, 8192] if lattice and c["stored"] else [16, 64, 256])
    if kind in ("update", "stream"):
        c["ops"] = logint(1, min(1_000_000, c["E"] // 16))
    return c


# ---- inputs ------------------------------------------------------------------------------------


def _rand(n, g):
    return torch.rand(n, device="cuda", generator=g)


def _rmat_keys(V, E, g):
    """E distinct directed edges without self-loops, as sorted keys u << 32 | v."""
    scale = max(1, (V - 1).bit_length())
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    want = int(E * 1.25) + 1024
    for _ in range(12):
        u = torch.zeros(want, dtype=torch.int64, device="cuda")
        v = torch.zeros(want, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = _rand(want, g)
            u = (u << 1) | (r >= 0.76).long()
            v = (v << 1) | (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long()
        ok = (u != v) & (u < V) & (v < V)
        keys = torch.unique(torch.cat([keys, (u[ok] << 32) | v[ok]]))
        if len(keys) >= E:
            break
        want = 2 * (E - len(keys)) + 4096
    if len(keys) > E:
        keys = keys[torch.argsort(_rand(len(keys), g))[:E]]
    perm = torch.randperm(V, device="cuda", generator=g)
    return torch.sort((perm[keys >> 32] << 32) | perm[keys & 0xFFFFFFFF])[0]


def _lattice_keys(V, g):
    """Both directions of every kept lattice and long-range edge, as sorted keys, with weights."""
    side = math.isqrt(V)
    at = torch.arange(V, device="cuda").view(side, side)
    a = torch.cat([at[:, :-1].reshape(-1), at[:-1, :].reshape(-1)])
    b = torch.cat([at[:, 1:].reshape(-1), at[1:, :].reshape(-1)])
    keep = _rand(len(a), g) >= 0.05
    a, b = a[keep], b[keep]
    n = max(1, len(a) // 1000)
    length = ((1.0 - _rand(n, g)) ** (-1.0 / 1.5)).clamp(max=float(side))
    angle = _rand(n, g) * (2.0 * math.pi)
    x, y = (_rand(n, g) * side).long().clamp(max=side - 1), (_rand(n, g) * side).long().clamp(max=side - 1)
    x2 = (x + (length * angle.cos()).round().long()).clamp(0, side - 1)
    y2 = (y + (length * angle.sin()).round().long()).clamp(0, side - 1)
    a, b = torch.cat([a, x * side + y]), torch.cat([b, x2 * side + y2])
    pairs = torch.unique((torch.minimum(a, b) << 32) | torch.maximum(a, b))
    a, b = pairs >> 32, pairs & 0xFFFFFFFF
    a, b = a[a != b], b[a != b]
    dist = torch.hypot((a // side - b // side).double(), (a % side - b % side).double())
    w = (100.0 * dist).long() + (_rand(len(a), g) * 51.0).long().clamp(max=50)
    keys, order = torch.sort(torch.cat([(a << 32) | b, (b << 32) | a]))
    return keys, torch.cat([w, w])[order]


def _hash_weight(u, v):
    """GIR.edgeWeight of every edge: a 64-bit mix of u << 32 | v, into [1, 100]."""

    def shift33(x):  # logical shift of an int64 tensor
        return (x >> 33) & ((1 << 31) - 1)

    x = (u << 32) | v
    x = x ^ shift33(x)
    x = x * (0xFF51AFD7ED558CCD - (1 << 64))
    x = x ^ shift33(x)
    x = x * (0xC4CEB9FE1A85EC53 - (1 << 64))
    x = x ^ shift33(x)
    # unsigned x mod 100 of a signed tensor: 2^64 mod 100 = 16
    return 1 + (torch.remainder(x, 100) + torch.where(x < 0, 16, 0)) % 100


def _inputs(case, seed):
    """Everything a case is made of, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1_000_003 + 17)
    V = case["V"]
    if case["graph"] == "rmat":
        keys = _rmat_keys(V, case["E"], g)
        w = torch.randint(1, 256, (len(keys),), device="cuda", generator=g)
    else:
        keys, w = _lattice_keys(V, g)
    x = {"keys": keys, "w": w}
    if "lanes" in case:  # sources with out-edges, as a benchmark's search keys
        n = case["lanes"]
        sizes = [1] * n
        if "sets" in case:
            r = _rand(n, g).double().tolist()
            sizes = [int(math.exp(t * math.log(case["sets"]))) for t in r]
        pick = torch.randint(0, len(keys), (sum(sizes),), device="cuda", generator=g)
        src = (keys[pick] >> 32).int().cpu().numpy()
        x["sets"] = np.split(src, np.cumsum(sizes)[:-1])
        x["src"] = src
    if "ops" in case:  # half deletions of present edges, half inserts of absent ones
        n_del = case["ops"] // 2
        n_ins = case["ops"] - n_del
        dele = keys[torch.randperm(len(keys), device="cuda", generator=g)[:n_del]]
        u = torch.randint(0, V, (2 * n_ins + 64,), device="cuda", generator=g)
        v = torch.randint(0, V, (2 * n_ins + 64,), device="cuda", generator=g)
        new = torch.unique(((u << 32) | v)[u != v])
        at = torch.searchsorted(keys, new).clamp(max=len(keys) - 1)
        new = new[keys[at] != new]
        new = new[torch.randperm(len(new), device="cuda", generator=g)[:n_ins]]
        ops = torch.cat([dele, new])
        order = torch.randperm(len(ops), device="cuda", generator=g)
        x["ops"] = ops[order]
        x["ins"] = (torch.arange(len(ops), device="cuda") >= len(dele))[order]
    return x


def _create(case, x):
    V, keys = case["V"], x["keys"]

    def beg(rows):
        b = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
        b[1:] = torch.cumsum(torch.bincount(rows, minlength=V), 0)
        return b.int()

    back = torch.sort(((keys & 0xFFFFFFFF) << 32) | (keys >> 32))[0]
    args = (beg(keys >> 32), (keys & 0xFFFFFFFF).int(), beg(back >> 32), (back & 0xFFFFFFFF).int())
    w = x["w"].int() if case.get("stored") else None
    torch.cuda.synchronize()
    return gir.DeviceGraph.create(*args, V, w)


def prepare(case, seed):
    x = _inputs(case, seed)
    d = _create(case, x)
    V, lanes = case["V"], case.get("lanes", 0)
    s = {"case": case, "d": d}
    if case.get("learned"):
        d.use_learned_schedule()
    if lanes:
        s["src"], s["sets"] = x["src"], x["sets"]
        if not case.get("host"):
            if case["kind"] in ("bfs", "stream"):
                s["level"] = torch.empty((lanes, V), dtype=torch.int32, device="cuda")
            if case["kind"] in ("sssp", "stream"):
                s["dist"] = torch.empty((lanes, V), dtype=torch.int64, device="cuda")
    if "ops" in case:
        d.build()
        s["u"] = (x["ops"] >> 32).int().cpu().numpy()
        s["v"] = (x["ops"] & 0xFFFFFFFF).int().cpu().numpy()
        s["ins"] = x["ins"].cpu().numpy().astype(np.uint8)
        s["undo"] = 1 - s["ins"]
        s["restored"] = _layer_buffers(V)
    if case["kind"] in ("build", "update"):
        s["layers"] = _layer_buffers(V)
    room = case["E"] + case["E"] // 10 + case.get("ops", 0) + 64  # (a lattice's edge count varies with the seed)
    if case["kind"] == "build":
        s["dag"] = torch.full((2, room), -1, dtype=torch.int32, device="cuda")
    if case["kind"] == "update":
        s["edges"] = [torch.zeros(V + 1, dtype=torch.int64, device="cuda"),
                      torch.full((room,), -1, dtype=torch.int32, device="cuda")]
    torch.cuda.synchronize()
    return s


# ---- passes ------------------------------------------------------------------------------------


def _check(d, rc):
    if rc != native.GIR_OK:
        raise native.GirError(rc, native.dev_lib().gir_dev_last_error(d.handle).decode())


def _layer_buffers(V):
    return [torch.full((len(_LABELS), V), -1, dtype=torch.int32, device="cuda"),
            torch.full((V,), -1, dtype=torch.int32, device="cuda")]


def _layers(d, bufs):
    """Labels of every layer and the blocks' heads (at most one block per vertex; the rest of the
    buffer stays -1), copied on the device through the C ABI."""
    lib = native.dev_lib()
    labels, head = bufs
    for row, which in zip(labels, _LABELS):
        _check(d, lib.gir_dev_get_labels(d.handle, which, native.ptr(row)))
    _check(d, lib.gir_dev_get_blocks(d.handle, native.ptr(head), len(head), native._I64()))
    return bufs


def _dag(d, pair):
    src, dst = pair
    _check(d, native.dev_lib().gir_dev_get_dag(d.handle, native.ptr(src), native.ptr(dst), len(src), native._I64()))
    return [pair]


def _edges(d, bufs):
    beg, adj = bufs
    _check(d, native.dev_lib().gir_dev_get_csr(d.handle, 0, native.ptr(beg), native.ptr(adj), len(adj), native._I64()))
    return bufs


def _bfs(s):
    if "sets" in s["case"]:
        return s["d"].bfs_sets(s["sets"], out=s.get("level"))
    return s["d"].bfs(s["src"], out=s.get("level"))


def _sssp(s):
    c = s["case"]
    weights = native.WEIGHT_STORED if c["stored"] else native.WEIGHT_HASH
    return s["d"].sssp(s["src"], delta=c["delta"], weights=weights, out=s.get("dist"))


def run(state):
    c, d = state["case"], state["d"]
    if c["kind"] == "bfs":
        return _bfs(state)
    if c["kind"] == "sssp":
        return _sssp(state)
    if c["kind"] == "build":
        d.build()
        return _layers(d, state["layers"]) + _dag(d, state["dag"])
    d.apply_batch(state["u"], state["v"], state["ins"])
    if c["kind"] == "stream":
        out = [_bfs(state), _sssp(state)]
    else:
        out = _layers(d, state["layers"]) + _edges(d, state["edges"])
    d.apply_batch(state["u"], state["v"], state["undo"])
    return out + _layers(d, state["restored"])


# ---- what a pass cannot do without, and its exact outputs ----------------------------------------


def work(case):
    V, E, lanes = case["V"], case["E"], case.get("lanes", 0)
    csr = 8 * V + 4 * E
    kind = case["kind"]
    layers = 4 * V * (len(_LABELS) + 1)
    if kind == "bfs":
        return {"bytes": csr + 4 * V * lanes, "flops": E * lanes}
    if kind == "sssp":
        return {"bytes": csr + (4 * E if case["stored"] else 0) + 8 * V * lanes, "flops": E * lanes}
    if kind == "build":
        return {"bytes": 2 * csr + layers, "flops": 2 * E}
    one_batch = 9 * case["ops"] + 2 * csr + layers
    if kind == "update":
        return {"bytes": 2 * one_batch + csr, "flops": 4 * E}
    return {"bytes": 2 * one_batch + 2 * csr + 12 * V * lanes, "flops": 2 * E * lanes}


def _relax(V, src, dst, w, sets):
    """Shortest distances from every source set, int64[len(sets)][V], -1 where there is no path."""
    far = 1 << 60
    out = []
    for k in range(0, len(sets), 8):
        part = sets[k:k + 8]
        dist = torch.full((V, len(part)), far, dtype=torch.int64, device=src.device)
        for j, x in enumerate(part):
            dist[torch.as_tensor(x, dtype=torch.int64, device=src.device), j] = 0
        to = dst[:, None].expand(-1, len(part))
        while True:
            new = dist.scatter_reduce(0, to, dist[src] + w[:, None], "amin")
            if torch.equal(new, dist):
                break
            dist = new
        out.append(torch.where(dist >= far, INF, dist).t().contiguous())
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("bfs", "sssp"):
        return None  # labels, DAGs and edge sets: whole numbers without a short restatement
    rounds = 3 * math.isqrt(case["V"]) if case["graph"] == "lattice" else (12 if kind == "bfs" else 40)
    if case["E"] * case["lanes"] * rounds > 10_000_000_000:
        return None
    x = _inputs(case, seed)
    src, dst = x["keys"] >> 32, x["keys"] & 0xFFFFFFFF
    if kind == "bfs":
        w = torch.ones_like(src)
    else:
        w = x["w"] if case["stored"] else _hash_weight(src, dst)
    r = _relax(case["V"], src, dst, w, x["sets"])
    if case.get("host"):
        r = r.cpu().numpy()
        return r if kind == "bfs" else r.view(np.uint64)
    return r
