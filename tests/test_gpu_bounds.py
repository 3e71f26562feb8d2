"""Values and batches at the edges of what a call takes: the largest stored weights, weights through
batches of many ops, backward rows that do not match the forward ones, memory that runs out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _weighted(pkg, V, u, v, w):
    key, first = np.unique(np.asarray(u, np.int64) * V + np.asarray(v, np.int64), return_index=True)
    return pkg.graphs.from_edges(V, key // V, key % V, np.asarray(w, np.uint32)[first])


@pytest.mark.parametrize("lanes", [2, 8, 64])
@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("all_wrap", [False, True])
def test_sssp_weights_up_to_the_largest_word(pkg, orc, lanes, alike, all_wrap):
    """Stored weights within a 16-bit distance of 2^32: narrow lanes cannot hold the sum with a source's
    distance, and 32 bits of it wrap to a small one. `all_wrap`: every sum that does not fit wraps, so nothing
    else has the group run again; `alike`: all lanes alike, so an edge is relaxed by eight threads."""
    n = 600
    rng = np.random.default_rng(lanes)
    step = rng.integers(60, 100, n - 1)
    at = np.r_[0, np.cumsum(step)]  # below 65,534
    chain = np.arange(n)
    src = (np.zeros(lanes, np.int64) if alike else rng.integers(0, 8, lanes)).astype(np.int32)
    # from every vertex of the chain's rest an edge of nearly 2^32 leads out, to a leaf of its own
    far = chain[20:]
    big = (1 << 32) - rng.integers(1, at[far] - at[8] + 1)
    big[::50] = (1 << 32) - (at[far] - at[8])[::50]
    if not all_wrap:
        big[::7] = rng.choice([0xFFFF, 0x10000, 0xFFFF0000, 0xFFFE], len(big[::7]))
    V = n + len(far)
    g = _weighted(pkg, V, np.r_[chain[:-1], chain[1:], far], np.r_[chain[1:], chain[:-1], n + np.arange(len(far))],
                  np.r_[step, step, big])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    exp = np.stack([orc.sssp(V, fb, fa, [int(s)], w=g.w) for s in src])
    assert exp[:, :n].max() < 0xFFFF and exp[:, n:].max() > 0xFFFFFFFF
    for bits in (16, 32, 64, 0):
        for delta in (1, 64, 1 << 20, 1 << 40):
            d = pkg.DeviceGraph.from_graph(g)  # (a handle remembers that 16 bits did not do)
            d.set_param(pkg.native.PARAM_LANE_BITS, bits)
            got = d.sssp(src, delta=delta, weights=pkg.native.WEIGHT_STORED)
            np.testing.assert_array_equal(got, exp, err_msg=f"{bits} bits, delta {delta}")
            d.close()


@pytest.mark.parametrize("insert", [True, False])
@pytest.mark.parametrize("n", [2, 40])
def test_backward_rows_that_do_not_match(pkg, insert, n):
    """A backward CSR with as many edges as the forward one, but one of them elsewhere: a batch that inserts the
    edge it holds already, or deletes the one it lacks, is malformed, and no backward row changes."""
    V = 50
    a = np.arange(V - 1)
    g = pkg.graphs.from_edges(V, a, a + 1)
    src, dst = a.copy(), a + 1
    src[7], dst[7] = 7, 30  # (the forward rows have 7 -> 8)
    b = pkg.graphs.from_edges(V, src, dst)
    d = pkg.DeviceGraph.create(g.fw_beg, g.fw_adj, b.bw_beg, b.bw_adj, V)
    before = [x.copy() for x in d.csr(1)]
    u = np.r_[7, np.arange(9, 8 + n)].astype(np.int32)
    v = np.r_[30 if insert else 8, np.zeros(n - 1, int)].astype(np.int32)  # (edges to vertex 0: new)
    ins = np.r_[1 if insert else 0, np.ones(n - 1, int)].astype(np.uint8)
    with pytest.raises(pkg.GirError, match="not the transpose") as e:
        d.apply_batch(u, v, ins)
    assert e.value.code == 5
    for x, y in zip(d.csr(1), before):
        np.testing.assert_array_equal(x, y)
    d.close()


@pytest.mark.parametrize("lanes", [64, 65, 130])
def test_bfs_without_memory_for_the_bit_planes(pkg, orc, monkeypatch, capfd, lanes):
    """The planes' 32 bytes a vertex cannot be had: the levels are written straight to the output, the call leaves
    no error text, and it asks for the memory once, not once a group of 64 lanes."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("GIR_TRACE", "2")  # (failed allocations on stderr; read when a handle is made)
    V = 140_000
    rng = np.random.default_rng(lanes)
    tail = np.arange(V - 40, V)  # more levels than the planes hold
    u, v = np.r_[rng.integers(0, V - 60, 3 * V), 5, tail[:-1]], np.r_[rng.integers(0, V - 60, 3 * V), tail[0], tail[1:]]
    key = np.unique(u[u != v] * V + v[u != v])
    g = pkg.graphs.from_edges(V, key // V, key % V)
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    src = rng.integers(0, V - 60, lanes).astype(np.int32)
    src[3] = -1
    out = [torch.full((lanes, V), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    failed = []
    for limit, res in zip((0, 31 * V), out):
        d = pkg.DeviceGraph.from_graph(g, weights=False)
        d.set_param(pkg.native.PARAM_ALLOC_LIMIT, limit)
        capfd.readouterr()
        d.bfs(src, out=res)
        failed.append(capfd.readouterr().err.count("pool exhausted"))
        assert pkg.native.dev_lib().gir_dev_last_error(d.handle) == b""
        d.close()
    assert failed == [0, 1]
    got = out[0].cpu().numpy()
    np.testing.assert_array_equal(out[1].cpu().numpy(), got)
    for i in (0, 3, lanes - 1):
        np.testing.assert_array_equal(got[i], orc.bfs(V, fb, fa, [int(src[i])]) if src[i] >= 0 else np.full(V, -1))


def test_allocation_limit_is_an_error_where_memory_is_needed(pkg):
    g = pkg.graphs.rmat(12, seed=4)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    with pytest.raises(pkg.GirError):
        d.set_param(pkg.native.PARAM_ALLOC_LIMIT, -1)
    d.set_param(pkg.native.PARAM_ALLOC_LIMIT, 4096)
    with pytest.raises(pkg.GirError) as e:
        d.bfs(np.zeros(1, np.int32))
    assert e.value.code == 3
    d.set_param(pkg.native.PARAM_ALLOC_LIMIT, 0)
    assert d.bfs(np.zeros(1, np.int32))[0, 0] == 0
    d.close()


def _host_level_graphs(pkg):
    """Power-law, deep (past the builds' level limits), a deep DAG, one-way streets, nothing at all."""
    from test_gpu_kernel_edges import _deep_shapes
    rng = np.random.default_rng(6)
    yield "rmat", pkg.graphs.rmat(13, seed=5)
    for name, V, u, v in _deep_shapes():
        if name in ("path 66", "path 700", "one-way, long range, loops", "joined paths"):
            keep = (u != v) | ("loops" in name)
            yield name, _weighted(pkg, V, u[keep], v[keep], rng.integers(1, 90, int(keep.sum())))
    u = np.arange(5999)
    far = rng.integers(0, 6000, (2, 4000))
    far = far[:, far[0] != far[1]]
    yield "dag", _weighted(pkg, 6000, np.r_[u[::2], np.minimum(*far)], np.r_[u[::2] + 1, np.maximum(*far)],
                           rng.integers(1, 90, len(u[::2]) + far.shape[1]))
    yield "empty", _weighted(pkg, 300, np.zeros(0, np.int64), np.zeros(0, np.int64), np.zeros(0))


@pytest.mark.parametrize("learned", [False, True])
def test_levels_and_phases_launched_from_the_host(pkg, orc, learned):
    """Where a device takes no cooperative launches every BFS level, SSSP phase, build level and round of the DAG's
    levels is a launch of its own: the same results, before and after a batch."""
    from test_gpu_layers import _oracle_match
    for name, g in _host_level_graphs(pkg):
        V = g.V
        fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
        d = pkg.DeviceGraph.from_graph(g)
        d.set_param(pkg.native.PARAM_COOPERATIVE, 0)
        if learned:
            d.use_learned_schedule()
        rng = np.random.default_rng(V)
        weights = g.w
        for step in range(2):
            d.build()
            _oracle_match(pkg, orc, d, V, fb, fa, f"{name}, step {step}")
            for lanes in (1, 9, 65):
                src = rng.integers(0, V, lanes).astype(np.int32)
                src[-1] = -1 if lanes > 1 else src[0]
                exp = np.stack([orc.bfs(V, fb, fa, [int(s)]) if s >= 0 else np.full(V, -1) for s in src])
                np.testing.assert_array_equal(d.bfs(src), exp, err_msg=name)
                st = d.query_stats()
                assert st["persistent_levels"] == 0 and st["reached"] == (exp >= 0).sum()
                for mode, w in ((pkg.native.WEIGHT_HASH, None), (pkg.native.WEIGHT_STORED, weights)):
                    if w is None and mode == pkg.native.WEIGHT_STORED:
                        continue
                    got = d.sssp(src, delta=20, weights=mode)
                    for i in {0, lanes // 2, lanes - 1}:
                        e = orc.sssp(V, fb, fa, [int(src[i])], w=w) if src[i] >= 0 else np.full(V, 2**64 - 1, np.uint64)
                        np.testing.assert_array_equal(got[i], e, err_msg=name)
            if step == 0 and V > 1000:
                a, b = rng.integers(0, V, 60).astype(np.int32), rng.integers(0, V, 60).astype(np.int32)
                rows = np.repeat(np.arange(V), np.diff(fb))
                at = rng.integers(0, len(fa), 30)
                a[:30], b[:30] = rows[at], fa[at]
                ins = (np.arange(60) >= 30).astype(np.uint8)
                d.apply_batch(a, b, ins)
                fb, fa, _, _ = orc.apply_batch(V, fb, fa, a, b, ins)
                weights = None
        d.close()


def test_large_levels_without_cooperative_launches(pkg):
    """Levels of over 2^22 row entries and passes of over 2^18 edges, which leave the loops where there are any: the
    results of the loops."""
    g = pkg.graphs.rmat(18, n_draws=24 << 18, seed=9)
    src = np.flatnonzero(np.diff(g.fw_beg))[:: 3000][:40].astype(np.int32)
    got = []
    for coop in (1, 0):
        d = pkg.DeviceGraph.from_graph(g)
        d.set_param(pkg.native.PARAM_COOPERATIVE, coop)
        d.build()
        got.append([d.labels(k) for k in range(5)] + list(d.blocks()) + list(d.dag()) + [d.bfs(src), d.sssp(src)])
        assert (d.query_stats()["launches"] > 0) and d.get_param(pkg.native.PARAM_COOPERATIVE) == coop
        d.close()
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


def _batch_weights(pkg, V, n, step, rng, fb, fa):
    """Ops of a batch: a hub's row, present edges, both directions of pairs, repeated keys."""
    a, b = rng.integers(0, V, n), rng.integers(0, V, n)
    a[: n // 4] = rng.integers(0, 1 + V // 20)  # one hub
    rows, at = np.repeat(np.arange(V), np.diff(fb)), rng.integers(0, max(len(fa), 1), n)
    if len(fa):
        a[::3], b[::3] = rows[at[::3]], fa[at[::3]]
    k = np.arange(n) % 5 == 1
    a[k], b[k] = np.roll(b, 1)[k], np.roll(a, 1)[k]
    ins = (rng.random(n) < (0.5, 0.0, 1.0, 0.3)[step]).astype(np.uint8)
    return a.astype(np.int32), b.astype(np.int32), ins


@pytest.mark.parametrize("rule", ["hash", "uniform"])
@pytest.mark.parametrize("V,n", [(40, 2), (40, 33), (40, 600), (300, 4096), (300, 20_000)])
def test_stored_weights_through_batches(pkg, orc, V, n, rule):
    """Every edge's stored weight after batches of many ops: survivors keep theirs (in rows with inserts and
    deletions, in rows that outgrow their slack and the layout that follows), inserted edges, among them those
    deleted a batch before, get the rule's. No path of two edges is shorter than one (uniform rule) or the
    oracle's distances say what is (hash rule), so the distances from every vertex hold every weight."""
    rng = np.random.default_rng(V + n)
    lo = 1 << 20
    hi = lo + (1 << 19)
    u, v = rng.integers(0, V, 4 * V), rng.integers(0, V, 4 * V)
    u, v = np.r_[u, v[::3], 0], np.r_[v, u[::3], 1]
    keep = u != v
    w = rng.permutation(len(u)).astype(np.uint32) + (lo if rule == "uniform" else 1)
    g = _weighted(pkg, V, u[keep], v[keep], w[keep])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    weight = {(int(x), int(y)): int(z) for x, y, z in zip(np.repeat(np.arange(V), np.diff(fb)), fa, g.w)}
    d = pkg.DeviceGraph.from_graph(g)
    if rule == "uniform":
        d.set_weight_rule(7, lo, hi)
    d.build()
    grown = False
    for step in (0, 2, 1, 2, 3):
        a, b, ins = _batch_weights(pkg, V, n, step, rng, fb, fa)
        d.apply_batch(a, b, ins)
        fb, fa, _, _ = orc.apply_batch(V, fb, fa, a, b, ins)
        rows = np.repeat(np.arange(V), np.diff(fb))
        gb, ga = d.csr(0)
        np.testing.assert_array_equal(gb, fb)
        np.testing.assert_array_equal(ga, fa)
        if rule == "uniform":
            new = pkg.graphs.uniform_weights(pkg.graphs.Graph(V, fb.astype(np.int32), fa, None, None), lo, hi, 7)
        else:
            new = [orc.edge_weight(int(x), int(y)) for x, y in zip(rows, fa)]
        weight = {(int(x), int(y)): weight.get((int(x), int(y)), int(z)) for x, y, z in zip(rows, fa, new)}
        now = np.array([weight[int(x), int(y)] for x, y in zip(rows, fa)], np.uint32)
        src = np.arange(V, dtype=np.int32)
        got = d.sssp(src, delta=1 << 21 if rule == "uniform" else 64, weights=pkg.native.WEIGHT_STORED)
        if rule == "uniform":
            np.testing.assert_array_equal(got[rows, fa], now)
        for s in range(0, V, 1 if rule == "hash" else 37):
            np.testing.assert_array_equal(got[s], orc.sssp(V, fb, fa, [s], w=now))
        grown |= int(np.diff(fb).max()) > 2 * int(np.diff(g.fw_beg).max())
    assert grown or n < 600  # (a row outgrew its slack: a new layout)
    d.close()


def test_handles_on_several_threads(pkg):
    """Builds and queries of three graphs at once, a thread and a handle each: their cooperative launches share the GPU."""
    import threading
    graphs = [pkg.graphs.rmat(14, seed=3), pkg.graphs.lattice(side=120, seed=4), pkg.graphs.rmat(16, seed=5)]
    handles = [pkg.DeviceGraph.from_graph(g) for g in graphs]

    def results(d, g):
        src = np.flatnonzero(np.diff(g.fw_beg))[:70].astype(np.int32)
        d.build()
        return [d.labels(k) for k in range(5)] + [d.bfs(src[:9]), d.sssp(src[:9]), d.sssp(src[:1])]

    alone = [results(d, g) for d, g in zip(handles, graphs)]
    wrong = []

    def loop(i):
        try:
            for _ in range(10):
                if not all((x == y).all() for x, y in zip(results(handles[i], graphs[i]), alone[i])):
                    wrong.append(i)
        except Exception as e:  # (a failure in a thread would pass unseen)
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for d in handles:
        d.close()
