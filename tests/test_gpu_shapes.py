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
