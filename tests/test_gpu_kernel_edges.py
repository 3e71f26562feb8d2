"""Sizes at which the query and layer kernels change path (edges of tiles, of launches, of the rules
that pick a variant), each against the oracle. Integer work: bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(pkg, V, u, v):
    key = np.unique(np.asarray(u, np.int64) * V + np.asarray(v, np.int64))
    return pkg.graphs.from_edges(V, key // V, key % V)


def _brooms(pkg, V, hub):
    """Hubs with rows of `hub` entries (longer than one warp's run of edge positions), hanging on a
    directed ring through every vertex (as many levels as vertices), and a few random edges."""
    rng = np.random.default_rng(V + hub)
    ring = np.arange(V, dtype=np.int64)
    u, v = [ring, np.zeros(hub, np.int64), np.full(hub, V // 2)], [(ring + 1) % V, 1 + ring[:hub] % (V - 1), ring[-hub:]]
    u.append(rng.integers(0, V, V // 50))
    v.append(rng.integers(0, V, V // 50))
    u, v = np.concatenate(u), np.concatenate(v)
    return _graph(pkg, V, u[u != v], v[u != v])


@pytest.mark.parametrize("V,hub,alpha", [(33, 3, 15), (4095, 700, 15), (4096, 513, 15), (4097, 512, 1e-6), (9000, 8999, 15),
                                         (9000, 4000, 1e9)])
def test_bfs_levels_across_launch_rules(pkg, orc, V, hub, alpha):
    """The device-resident level loop: below and above 4,096 vertices (where directions are chosen),
    thousands of levels (more decisions than are read with the counters), hub rows longer than a run,
    both directions forced, 1 to 65 lanes with repeated and out-of-range sources."""
    g = _brooms(pkg, V, hub)
    fb, fa = orc.normalize(g.V, g.fw_beg, g.fw_adj)
    deg = np.diff(fb)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.set_param(pkg.native.PARAM_ALPHA, alpha)
    if alpha > 1e6:
        d.set_param(pkg.native.PARAM_BETA, 1e9)
    rng = np.random.default_rng(1)
    for lanes in (1, 2, 33, 65):
        src = rng.integers(0, V, lanes).astype(np.int32)
        src[-1] = src[0]
        if lanes > 2:
            src[1] = -1
            src[2] = V
        exp = np.stack([orc.bfs(g.V, fb, fa, [int(s)]) for s in src])
        np.testing.assert_array_equal(d.bfs(src), exp)
        st = d.query_stats()
        assert st["reached"] == (exp >= 0).sum() and st["edges"] == ((exp >= 0) * deg).sum()
        if V >= 4096 and lanes < 65:
            assert len(d.sched_trace()[1]) >= st["iterations"]
    sets = [rng.integers(0, V, n).astype(np.int32) for n in (1, 5, 0, 40)]
    got = d.bfs_sets(sets)
    for row, s in zip(got, sets):
        np.testing.assert_array_equal(row, orc.bfs(g.V, fb, fa, [int(x) for x in s]) if len(s) else np.full(V, -1))
    d.close()


def test_bfs_of_a_graph_whose_bottom_up_levels_leave_the_launch(pkg, orc):
    """More than 2^20 vertices: bottom-up levels, and frontiers of over 2^22 out-edges, run as their own
    launches between two device-resident stretches."""
    V = (1 << 20) + 77
    rng = np.random.default_rng(5)
    tail = np.arange(V - 300, V - 1)
    u = np.concatenate([rng.integers(0, V - 300, 6 * V), tail, [0]])
    v = np.concatenate([rng.integers(0, V - 300, 6 * V), tail + 1, [V - 300]])
    g = _graph(pkg, V, u[u != v], v[u != v])
    fb, fa = orc.normalize(g.V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    src = np.array([0, V - 300, 17, V - 1], np.int32)
    exp = np.stack([orc.bfs(g.V, fb, fa, [int(s)]) for s in src])
    for alpha in (15, 1e-6):
        d.set_param(pkg.native.PARAM_ALPHA, alpha)
        np.testing.assert_array_equal(d.bfs(src), exp)
        st = d.query_stats()
        assert 0 < st["persistent_levels"] < st["iterations"]
        assert (st["bottom_up"] > 0) == (alpha > 1)
    d.close()


def _deep_shapes():
    """(name, V, u, v): graphs whose searches run past the level counts at which the builds change to the
    reciprocal classes (SCC) and to the forest without levels (blocks), and just below them."""
    rng = np.random.default_rng(3)
    for n in (24, 25, 26, 64, 65, 66, 129, 700):  # paths: eccentricity n - 1 from the smallest vertex
        a = np.arange(n - 1)
        yield f"path {n}", n, np.r_[a, a + 1], np.r_[a + 1, a]
    side = 90
    at = np.arange(side * side).reshape(side, side)
    a = np.r_[at[:, :-1].ravel(), at[:-1, :].ravel()]
    b = np.r_[at[:, 1:].ravel(), at[1:, :].ravel()]
    keep = rng.random(len(a)) > 0.25  # holes: bridges, small components, many blocks
    a, b = a[keep], b[keep]
    V = side * side
    perm = rng.permutation(V)
    yield "lattice", V, perm[np.r_[a, b]], perm[np.r_[b, a]]
    # one-way streets: classes joined into one SCC by one-way cycles, others left one-way between SCCs
    one = rng.random(len(a)) < 0.3
    yield "one-way", V, perm[np.r_[a, b[~one]]], perm[np.r_[b, a[~one]]]
    extra = rng.integers(0, V, (2, 60))
    loops = rng.integers(0, V, 50)
    yield "one-way, long range, loops", V, np.r_[perm[np.r_[a, b[~one]]], extra[0], loops], np.r_[
        perm[np.r_[b, a[~one]]], extra[1], loops]
    n = 2000  # two long reciprocal paths joined by one-way edges both ways (one SCC), a third only one way
    p = np.arange(n - 1)
    parts = [(p + k * n, p + 1 + k * n) for k in range(3)]
    u = np.concatenate([np.r_[x, y] for x, y in parts] + [[5, n + 900, 2 * n + 7]])
    v = np.concatenate([np.r_[y, x] for x, y in parts] + [[n + 3, 1500, 12]])
    yield "joined paths", 3 * n, u, v
    c = np.arange(1500)  # directed rings sharing single vertices, a hub with every tenth vertex
    yield "rings", 4500, np.r_[c, c + 1500, 1500 * 2 + c, c[::10], np.full(150, 7)], np.r_[
        (c + 1) % 1500, np.where(c == 1499, 0, c + 1501), 3000 + (c + 1) % 1500, np.full(150, 7), c[::10]]


def test_layers_of_deep_graphs(pkg, orc):
    from test_gpu_layers import _oracle_match
    for name, V, u, v in _deep_shapes():
        keep = (u != v) | ("loops" in name)
        g = _graph(pkg, V, u[keep], v[keep])
        fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
        d = pkg.DeviceGraph.from_graph(g, weights=False)
        d.build()
        _oracle_match(pkg, orc, d, V, fb, fa, name)
        if V > 1000:  # one-way inserts and deletions: fewer vertices with reciprocal edges only
            for step in range(2):
                cb, ca = d.csr(0)
                bu, bv, ins = pkg.graphs.updates(pkg.graphs.Graph(V, cb.astype(np.int32), ca, None, None), 40, 40, 9 + step)
                d.apply_batch(bu, bv, ins)
                fb, fa, _, _ = orc.apply_batch(V, fb, fa, bu, bv, ins)
                _oracle_match(pkg, orc, d, V, fb, fa, f"{name}, batch {step}")
        d.close()


def _weighted(pkg, V, u, v, w):
    key, first = np.unique(np.asarray(u, np.int64) * V + np.asarray(v, np.int64), return_index=True)
    return pkg.graphs.from_edges(V, key // V, key % V, np.asarray(w, np.uint32)[first])


@pytest.mark.parametrize("lanes", [1, 2, 3, 5, 8, 17, 33, 63, 64, 65])
def test_sssp_lane_counts_widths_and_buckets(pkg, orc, lanes):
    """Rows of every padding, lane widths of 16, 32 and 64 bits, bucket widths from one (every edge heavy)
    to wider than any path (every edge light), weights of zero, sources repeated and out of range; hubs
    whose rows are cut into runs, and long stretches of settled vertices without a heavy edge."""
    rng = np.random.default_rng(lanes)
    V = 3000
    u = np.concatenate([rng.integers(0, V, 3 * V), np.zeros(2500, np.int64), np.full(900, 7), np.arange(V - 1)])
    v = np.concatenate([rng.integers(0, V, 3 * V), 1 + np.arange(2500), V - 1 - np.arange(900), 1 + np.arange(V - 1)])
    w = rng.integers(0, 60, len(u))
    w[rng.random(len(u)) < 0.002] = 5000
    w[-(V - 1):] = 3
    keep = u != v
    g = _weighted(pkg, V, u[keep], v[keep], w[keep])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g)
    src = rng.integers(0, V, lanes).astype(np.int32)
    src[-1] = src[0]
    if lanes > 4:
        src[2], src[3] = -1, V
    exp = np.stack([orc.sssp(V, fb, fa, [int(s)], w=g.w) for s in src])
    exp_hash = np.stack([orc.sssp(V, fb, fa, [int(s)]) for s in src[:4]])
    for bits in (0, 16, 32, 64):
        d.set_param(pkg.native.PARAM_LANE_BITS, bits)
        for delta in (1, 16, 61, 1000, 1 << 40):
            got = d.sssp(src, delta=delta, weights=pkg.native.WEIGHT_STORED)
            np.testing.assert_array_equal(got, exp, err_msg=f"{bits} bits, delta {delta}")
            st = d.query_stats()
            fin = exp != np.uint64(2**64 - 1)
            assert st["reached"] == fin.sum() and st["edges"] == (fin * np.diff(fb)).sum()
    np.testing.assert_array_equal(d.sssp(src, delta=16)[:4], exp_hash)
    sets = [rng.integers(0, V, n).astype(np.int32) for n in (1, 700, 0, 3)]
    got = d.sssp_sets(sets, delta=20, weights=pkg.native.WEIGHT_STORED)
    for row, s in zip(got, sets):
        np.testing.assert_array_equal(row, orc.sssp(V, fb, fa, [int(x) for x in s], w=g.w) if len(s)
                                      else np.full(V, 2**64 - 1, np.uint64))
    d.close()


def test_sssp_phases_inside_and_outside_the_bucket_loop(pkg, orc):
    """Passes of over 2^18 edges and far queues of over 2^18 entries leave the device-resident loop for
    launches of their own, and the loop takes over again for a long tail; 32- and 64-bit lanes."""
    V = 400_000
    rng = np.random.default_rng(8)
    tail = np.arange(V - 400, V - 1)
    u = np.concatenate([rng.integers(0, V - 400, 8 * V), tail, [11], np.zeros(9000, np.int64)])
    v = np.concatenate([rng.integers(0, V - 400, 8 * V), tail + 1, [V - 400], rng.integers(0, V - 400, 9000)])
    w = rng.integers(1, 200, len(u))
    keep = u != v
    for scale in (1, 300):  # the larger weights do not fit 32-bit lanes
        g = _weighted(pkg, V, u[keep], v[keep], w[keep] * scale)
        fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
        d = pkg.DeviceGraph.from_graph(g)
        src = np.concatenate([rng.integers(0, V, 38), [0, V - 1]]).astype(np.int32)
        got = d.sssp(src, delta=40 * scale, weights=pkg.native.WEIGHT_STORED)
        for i in (0, 5, 38, 39):
            np.testing.assert_array_equal(got[i], orc.sssp(V, fb, fa, [int(src[i])], w=g.w))
        one = d.sssp(src[:1], delta=7 * scale, weights=pkg.native.WEIGHT_STORED)
        np.testing.assert_array_equal(one[0], got[0])
        d.close()


@pytest.mark.parametrize("lanes", [7, 8, 9, 64])
def test_bfs_levels_kept_in_bit_planes(pkg, orc, lanes):
    """Eight lanes or more over at least 2^23 (lane, vertex) pairs: levels below 15 go through bit planes,
    the deeper ones of a tail straight to the output, unreached vertices and lanes without a source are -1."""
    V = (1 << 20) + 77
    rng = np.random.default_rng(lanes)
    u, v = rng.integers(0, V - 200, 3 * V), rng.integers(0, V - 200, 3 * V)
    tail = np.arange(V - 150, V)  # 50 vertices before it have no edge
    u, v = np.r_[u, 5, tail[:-1]], np.r_[v, tail[0], tail[1:]]
    g = _graph(pkg, V, u[u != v], v[u != v])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    src = rng.integers(0, V - 200, lanes).astype(np.int32)
    src[1], src[2], src[3], src[-1] = V - 1, -1, V - 180, tail[0]
    got = d.bfs(src)
    for row, s in zip(got, src):
        np.testing.assert_array_equal(row, orc.bfs(V, fb, fa, [int(s)]) if s >= 0 else np.full(V, -1))
    d.close()


def test_builds_with_levels_taken_bottom_up(pkg, orc):
    """Levels of more than 2^22 row entries and a class that holds nearly every row: the rows of the giant
    component, SCC and block are left out of the passes that look for the others."""
    from test_gpu_layers import _oracle_match
    core, V = 300_000, 360_000
    rng = np.random.default_rng(3)
    u, v = rng.integers(0, core, 20 * core), rng.integers(0, core, 20 * core)
    w = np.arange(core, core + 30_000)  # hanging in or out by one edge, or by a small ring
    x = np.arange(core + 30_000, V, 3)
    u = np.r_[u, w[::2], rng.integers(0, core, 15_000), x, x + 1, x + 2, x[::2], rng.integers(0, core, 2_500)]
    v = np.r_[v, rng.integers(0, core, 15_000), w[1::2], x + 1, x + 2, x, rng.integers(0, core, 5_000), x[1::4]]
    g = _graph(pkg, V, u[u != v], v[u != v])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.build()
    _oracle_match(pkg, orc, d, V, fb, fa, "bottom-up levels")
    d.close()


@pytest.mark.parametrize("V,n", [(2, 2), (40, 2), (40, 33), (40, 600), (700, 1), (700, 4096), (3000, 20_000)])
def test_batches_that_change_both_directions_of_pairs(pkg, orc, V, n):
    """Every way a batch can change a pair (one edge, both alike, one each way, one of two), several ops of
    a key, rows with both inserts and deletions, rows with more ops than a warp, rows that outgrow their
    slack: the three CSRs and the layers, with and without anything to insert or to delete."""
    from test_gpu_layers import _oracle_match
    rng = np.random.default_rng(V + n)
    u, v = rng.integers(0, V, 4 * V), rng.integers(0, V, 4 * V)
    u, v = np.r_[u, v[::3], 0], np.r_[v, u[::3], 1]
    g = _graph(pkg, V, u[u != v], v[u != v])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g)
    d.build()
    for step in range(4):
        a, b = rng.integers(0, V, n), rng.integers(0, V, n)
        a[: n // 4] = rng.integers(0, 1 + V // 20)  # one hub
        rows, at = np.repeat(np.arange(V), np.diff(fb)), rng.integers(0, max(len(fa), 1), n)
        if len(fa):
            a[::3], b[::3] = rows[at[::3]], fa[at[::3]]
        k = np.arange(n) % 5 == 1
        a[k], b[k] = np.roll(b, 1)[k], np.roll(a, 1)[k]
        a, b = a.astype(np.int32), b.astype(np.int32)
        ins = (rng.random(n) < (0.5, 0.0, 1.0, 0.3)[step]).astype(np.uint8)
        d.apply_batch(a, b, ins)
        fb, fa, n_ins, n_del = orc.apply_batch(V, fb, fa, a, b, ins)
        st = d.batch_stats()
        assert (st["inserted"], st["deleted"]) == (n_ins, n_del)
        tb, ta = orc.transpose(V, fb, fa)
        for which, (eb, ea) in enumerate(((fb, fa), (tb, ta), orc.sym(V, fb, fa, tb, ta))):
            gb, ga = d.csr(which)
            np.testing.assert_array_equal(gb, eb)
            np.testing.assert_array_equal(ga, ea)
        _oracle_match(pkg, orc, d, V, fb, fa, f"step {step}")
    d.close()


@pytest.mark.parametrize("where", ["first", "middle", "last", "none"])
def test_bottom_up_rows_to_their_last_entry(pkg, orc, where):
    """Bottom-up levels of rows of every remainder of the warp's and the CTA's rounds, found by one entry of
    the row: the first, one in between, the last, or none (lanes of the other sources find them)."""
    deg = np.r_[31:35, 125:130, 157:166, 285:292, 4093:4102, 5117:5124, 8190:8196]
    L, n = 8200, len(deg)  # leaves, then the hubs, then a vertex that reaches one leaf of every hub
    V = L + n + 2
    u = np.concatenate([np.arange(L - d, L) for d in deg])
    v = np.repeat(L + np.arange(n), deg)
    at = {"first": L - deg, "middle": L - deg // 2 - 1, "last": np.full(n, L - 1), "none": np.zeros(0, np.int64)}[where]
    tail = np.arange(0, L, 50)
    g = _graph(pkg, V, np.r_[u, np.full(len(at), V - 2), np.full(len(tail), V - 1)], np.r_[v, at, tail])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.set_param(pkg.native.PARAM_ALPHA, 1e9)
    d.set_param(pkg.native.PARAM_BETA, 1e9)
    for src in ([V - 2], [V - 2, V - 1, 0, L - 1, L + 3]):
        got = d.bfs(np.array(src, np.int32))
        for row, s in zip(got, src):
            np.testing.assert_array_equal(row, orc.bfs(V, fb, fa, [s]))
        if len(src) > 1 or where != "none":  # (a lone source without edges has no level to take)
            assert d.query_stats()["bottom_up"] > 0
    d.close()
