"""Graphs whose rows or chains are long: layers against the oracle where it is quick, and no build that one warp
or one thread holds up for a whole row or chain (times of the same graph under another numbering, in one process)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(pkg, V, u, v):
    key = np.unique(np.asarray(u, np.int64) * V + np.asarray(v, np.int64))
    return pkg.graphs.from_edges(V, key // V, key % V)


def _both(pkg, V, u, v):
    return _graph(pkg, V, np.r_[u, v], np.r_[v, u])


def _star(pkg, V, hub):
    leaf = np.delete(np.arange(V), hub)
    return _both(pkg, V, np.full(V - 1, hub), leaf)


def _build_ms(pkg, g, layer, reps=5):
    """Least wall time of a build of one layer (the others are there)."""
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.build()
    best = 1e9
    for _ in range(reps):
        t = time.perf_counter()
        d.build(layer)
        best = min(best, time.perf_counter() - t)
    d.close()
    return 1e3 * best


@pytest.mark.parametrize("outside,inside", [(0, 1), (0, 31), (0, 33), (31, 2), (33, 700), (5000, 1), (5000, 3000), (40, 9000)])
def test_blocks_of_a_root_with_a_long_row(pkg, orc, outside, inside):
    """The SCC's smallest vertex is a hub: the first neighbours of its row in other SCCs, the rest in its own (as
    leaves, in triangles and on a ring), so that the row's least entry of its own SCC is at any place in it."""
    from test_gpu_layers import _oracle_match
    V = 1 + outside + inside
    rng = np.random.default_rng(outside + inside)
    out, mine = 1 + np.arange(outside), 1 + outside + np.arange(inside)
    u, v = [np.zeros(outside, np.int64), np.zeros(inside, np.int64), mine], [out, mine, np.zeros(inside, np.int64)]
    for k in (2, 3):
        a = mine[: len(mine) // (2 * k) * k].reshape(-1, k)
        u.append(a.ravel())
        v.append(np.roll(a, 1, 1).ravel())
    perm = np.r_[0, 1 + rng.permutation(outside), 1 + outside + rng.permutation(inside)]
    u, v = perm[np.concatenate(u)], perm[np.concatenate(v)]
    keep = u != v
    g = _graph(pkg, V, u[keep], v[keep])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.build()
    _oracle_match(pkg, orc, d, V, fb, fa, f"{outside} outside, {inside} inside")
    d.close()


def test_blocks_of_a_star_whose_hub_is_the_root(pkg):
    V = 400_000
    first, last = (_build_ms(pkg, _star(pkg, V, hub), pkg.native.LAYER_BCT) for hub in (0, V - 1))
    assert first < 3 * last, (first, last)


@pytest.mark.parametrize("layer", ["WCC", "BCT"])
def test_builds_of_a_chain_in_the_order_of_its_ids(pkg, layer):
    """A path for the components; for the blocks a ring whose vertices all hang on one hub, so that every edge of
    the ring puts a tree edge under the one before it. The ids run along the chain, or in any order."""
    V = 600_000
    a = np.arange(1, V)
    if layer == "WCC":
        u, v = a - 1, a
    else:
        hub, rest = V // 2, np.delete(np.arange(V), V // 2)
        u, v = np.r_[rest, np.full(V - 1, hub)], np.r_[np.roll(rest, 1), rest]
    perm = np.random.default_rng(1).permutation(V)
    which = getattr(pkg.native, f"LAYER_{layer}")
    if layer == "WCC":
        ms = []
        for p in (np.arange(V), perm):
            d = pkg.DeviceGraph.from_graph(_both(pkg, V, p[u], p[v]), weights=False)
            best = 1e9
            for _ in range(5):
                t = time.perf_counter()
                d.build(which)
                best = min(best, 1e3 * (time.perf_counter() - t))
            ms.append(best)
            assert (d.labels(pkg.native.LABEL_WCC) == 0).all()
            d.close()
    else:
        ms = [_build_ms(pkg, _both(pkg, V, p[u], p[v]), which) for p in (np.arange(V), perm)]
    assert ms[0] < 3 * ms[1] + 1, ms


def test_components_of_chains_of_every_length(pkg, orc):
    """Paths in the order of their ids, side by side, with lengths about those of warps, CTAs and waves."""
    length = np.array([1, 2, 31, 32, 33, 255, 256, 257, 4095, 4097, 70_000, 303_103, 303_105, 606_209])
    V = int(length.sum())
    end = np.cumsum(length)
    a = np.delete(np.arange(V), end - 1)
    g = _both(pkg, V, a, a + 1)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.build(pkg.native.LAYER_WCC)
    np.testing.assert_array_equal(d.labels(pkg.native.LABEL_WCC), np.repeat(end - length, length))
    assert d.counts()["n_wcc"] == len(length)
    d.close()


def _kite(pkg, V, path, p):
    """A hub with leaves, and a path hanging on it: deep, with one row that holds nearly every entry."""
    leaf, tail = np.arange(1, V - path), np.arange(V - path, V)
    return _both(pkg, V, p[np.r_[np.zeros(len(leaf), np.int64), 0, tail[:-1]]], p[np.r_[leaf, tail[0], tail[1:]]])


@pytest.mark.parametrize("hub", ["root", "anywhere"])
@pytest.mark.parametrize("layer", ["SCC", "BCT"])
def test_builds_of_a_deep_graph_with_a_long_row(pkg, layer, hub):
    """The ways for deep graphs (reciprocal classes, the forest by union-find) on a hub's row: no more than a few
    times what the hub costs without the path."""
    V = 600_000
    p = np.arange(V) if hub == "root" else np.random.default_rng(3).permutation(V)
    which = getattr(pkg.native, f"LAYER_{layer}")
    deep, flat = (_build_ms(pkg, _kite(pkg, V, path, p), which) for path in (300, 2))
    assert deep < 4 * flat + 2, (deep, flat)


@pytest.mark.parametrize("one_way", [0.0, 0.02, 0.3])
def test_layers_of_deep_graphs_with_hubs(pkg, orc, one_way):
    """A long path with hubs on it (rows beyond a warp's run), whose leaves are tied to one another here and there;
    some edges only one way, so that classes, quotient and forest all take part."""
    from test_gpu_layers import _oracle_match
    n, leaves = 400, 3000
    rng = np.random.default_rng(int(100 * one_way))
    a = np.arange(n - 1)
    u, v = [a], [a + 1]
    at = n
    for hub in (0, 1, 150, n - 1):
        mine = np.arange(at, at + leaves)
        at += leaves
        u += [np.full(leaves, hub), mine[:600:3]]
        v += [mine, mine[1:600:3]]
    u, v = np.concatenate(u), np.concatenate(v)
    one = rng.random(len(u)) < one_way
    perm = rng.permutation(at)
    for p in (np.arange(at), perm):
        g = _graph(pkg, at, p[np.r_[u, v[~one]]], p[np.r_[v, u[~one]]])
        fb, fa = orc.normalize(at, g.fw_beg, g.fw_adj)
        d = pkg.DeviceGraph.from_graph(g, weights=False)
        d.build()
        _oracle_match(pkg, orc, d, at, fb, fa, f"one way {one_way}")
        d.close()


def _ladder(n):
    a, b = np.arange(n - 1), np.arange(n)
    return 2 * n, np.r_[a, a + n, b], np.r_[a + 1, a + n + 1, b + n]


def _grid3(s):
    at = np.arange(s**3).reshape(s, s, s)
    return s**3, np.r_[at[1:].ravel(), at[:, 1:].ravel(), at[:, :, 1:].ravel()], np.r_[
        at[:-1].ravel(), at[:, :-1].ravel(), at[:, :, :-1].ravel()]


@pytest.mark.parametrize("shape", [lambda: _ladder(300_000), lambda: _grid3(80)], ids=["ladder", "grid"])
def test_components_of_short_rows_in_any_order(pkg, shape):
    """Rows of three and of six entries, ids in order (one tree after the first links) and permuted (many): the
    exact links that are left must not meet at a few roots."""
    V, u, v = shape()
    perm = np.random.default_rng(2).permutation(V)
    order, mixed = (_build_ms(pkg, _both(pkg, V, p[u], p[v]), pkg.native.LAYER_WCC, 9) for p in (np.arange(V), perm))
    assert mixed < 4 * order + 0.1, (mixed, order)


@pytest.mark.parametrize("V,entries", [(5, 1), (300, 1), (300, 3), (20_000, 1), (20_000, 2), (20_000, 3.4), (20_000, 3.6),
                                       (20_000, 5), (20_000, 7.9), (20_000, 8.1), (20_000, 14), (200_000, 2.2), (200_000, 6)])
def test_components_at_every_row_length(pkg, orc, V, entries):
    """About the average row lengths at which the sampling changes, with equal halves, isolated vertices and small
    components beside: the smallest vertex of every component, against the oracle."""
    rng = np.random.default_rng(int(10 * entries) + V)
    m = int(V * entries / 2)
    u, v = rng.integers(0, V, m), rng.integers(0, V, m)
    for part in (False, True):
        if part:  # two halves and a rest of small pieces
            piece = np.minimum(u * 5 // (2 * V), 2)
            v = np.where(piece < 2, piece * (2 * V // 5) + v % (2 * V // 5), np.minimum(u + v % 3, V - 1))
        g = _graph(pkg, V, u[u != v], v[u != v])
        fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
        d = pkg.DeviceGraph.from_graph(g, weights=False)
        d.build(pkg.native.LAYER_WCC)
        exp = orc.canon_labels(orc.wcc(V, fb, fa))
        np.testing.assert_array_equal(d.labels(pkg.native.LABEL_WCC), exp)
        assert d.counts()["n_wcc"] == len(np.unique(exp))
        d.close()


def _beside_a_core(pkg, core, deg, pages, flip, hubs=1):
    """A dense core, and beside it pages in rings of three that all link to a hub (one after another where there are
    several), which links back to one: with `flip`, all edges the other way."""
    rng = np.random.default_rng(core + deg)
    u, v = rng.integers(0, core, (2, core * deg))
    first = core + hubs
    p = np.arange(first, first + pages // 3 * 3)
    ring = p + np.where((p - first) % 3 == 2, -2, 1)
    hub = core + (p - first) // 3 % hubs
    e = [np.r_[u, p, p, core + np.arange(hubs)], np.r_[v, ring, hub, first + 3 * np.arange(hubs)]]
    keep = e[0] != e[1]
    e = [x[keep] for x in e]
    return first + len(p), e[flip], e[1 - flip]


def test_components_of_a_hub_beside_the_largest(pkg):
    """The hub's rows are outside the component that holds most row entries."""
    V, u, v = _beside_a_core(pkg, 8000, 600, 600_000, 0)
    hub, spread = (_build_ms(pkg, _graph(pkg, *a), pkg.native.LAYER_WCC)
                   for a in ((V, u, v), _beside_a_core(pkg, 8000, 600, 600_000, 0, hubs=3000)))
    assert hub < 4 * spread + 1, (hub, spread)


@pytest.mark.parametrize("hubs,pages", [(1, 4000), (1, 4090), (1, 4100), (1, 5121), (2, 12_000), (3, 60_000), (300, 1_500_000)])
def test_components_with_rows_about_the_long_one(pkg, orc, hubs, pages):
    V, u, v = _beside_a_core(pkg, 3000, 600 if pages < 100_000 else 2500, pages, 0, hubs)
    g = _graph(pkg, V, u, v)
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    d = pkg.DeviceGraph.from_graph(g, weights=False)
    d.build(pkg.native.LAYER_WCC)
    np.testing.assert_array_equal(d.labels(pkg.native.LABEL_WCC), orc.canon_labels(orc.wcc(V, fb, fa)))
    d.close()


def test_levels_that_look_through_a_long_row_in_vain(pkg):
    """A core of over 2^22 row entries in a level, whose search reaches a hub only some levels later; pages that no
    edge leads to are the rest of the hub's row. One hub, or as many entries on three thousand."""
    core, deg, pages, tail = 8000, 500, 400_000, 6
    rng = np.random.default_rng(1)
    u, v = rng.integers(0, core, (2, core * deg))
    ms = []
    for hubs in (1, 3000):
        chain = core + np.arange(tail)
        hub = core + tail + np.arange(hubs)
        page = core + tail + hubs + np.arange(pages)
        V = core + tail + hubs + pages
        a = np.r_[u, 0, chain[:-1], np.full(hubs, chain[-1]), hub, page]
        b = np.r_[v, chain[0], chain[1:], hub, np.zeros(hubs, np.int64), hub[np.arange(pages) % hubs]]
        ms.append(_build_ms(pkg, _graph(pkg, V, a[a != b], b[a != b]), pkg.native.LAYER_SCC))
    assert ms[0] < 3 * ms[1] + 1, ms


@pytest.mark.parametrize("where", ["before the line", "at the line", "last", "none"])
def test_bottom_up_levels_and_long_rows(pkg, orc, where):
    """A core of over 2^22 row entries in a level, and hubs whose only neighbours in the frontier come early in a
    long row, about where the warp leaves off, last, or not at all: SCCs, DAG and blocks against the oracle."""
    from test_gpu_layers import _oracle_match
    core, pages, hubs = 3000, 9000, 6
    rng = np.random.default_rng(len(where))
    u, v = rng.integers(0, core, (2, core * 2200))
    V = pages + core + 2 * hubs  # pages first, so that the core's entries come last in a hub's row (or the other way)
    at = {"before the line": 4000, "at the line": 4096, "last": pages, "none": pages}[where]
    page = np.r_[np.arange(at), np.arange(at + core, pages + core)]  # the core's ids lie from `at` on
    u, v = u + at, v + at
    into, out = V - 2 * hubs + np.arange(hubs), V - hubs + np.arange(hubs)
    parts_u, parts_v = [u], [v]
    for k in range(hubs):
        mine = page[rng.random(len(page)) < (1.0, 0.9)[k % 2]]
        parts_u += [mine, np.full(len(mine), out[k])]
        parts_v += [np.full(len(mine), into[k]), mine]
        if where != "none":  # a core vertex at one end of the row, both ways for half of the hubs
            c = at + rng.integers(0, core, 3)
            parts_u += [c, np.full(3, out[k])] + ([np.full(3, into[k]), c] if k % 2 else [])
            parts_v += [np.full(3, into[k]), c] + ([c, np.full(3, out[k])] if k % 2 else [])
    ring = page[: len(page) // 3 * 3].reshape(-1, 3)[::5]
    parts_u.append(ring.ravel())
    parts_v.append(np.roll(ring, 1, 1).ravel())
    u, v = np.concatenate(parts_u), np.concatenate(parts_v)
    g = _graph(pkg, V, u[u != v], v[u != v])
    fb, fa = orc.normalize(V, g.fw_beg, g.fw_adj)
    for pivot in (-1, 1, 2):
        d = pkg.DeviceGraph.from_graph(g, weights=False)
        d.set_param(pkg.native.PARAM_PIVOT, pivot)
        d.build()
        _oracle_match(pkg, orc, d, V, fb, fa, f"{where}, pivot {pivot}")
        d.close()
