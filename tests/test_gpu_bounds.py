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
