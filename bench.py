#!/usr/bin/env python
"""GIR-B200 benchmark: BFS / SSSP GTEPS and update throughput on one B200 (or N replicas).

One step = 64 BFS queries + 64 SSSP queries (Delta-stepping, Delta = 16, the reference's
GIR::edgeWeight weights in [1, 100], so the reference computes the identical result) on the
4.8M-vertex / 69M-edge power-law R-MAT graph (ids permuted, seed 3; a seeded synthetic stand-in
for soc-LiveJournal1). GTEPS = traversed edges (out-edges of the reached vertices, summed over the
queries) / time. The graph (~1.6 GB in HBM) is larger than L2, so no L2 flush is needed.

  value      device-resident run: sources and result buffers already in HBM
  e2e        the same calls through the C ABI with pinned HOST buffers: the sources are copied in
             and the 64 level rows + 64 distance rows copied out inside every step
  roofline   the dominant kernel's algorithmic bytes / its CUDA-event time (live), against the
             measured HBM copy bandwidth of this pool (MEASURED_PEAKS.json)
  cpu_baseline  the reference GIR compiled from its own sources (oracle/_ref), timed on this
             host's cores on a bounded sample of the same queries

Also reported (not part of `value`): SSSP with the stored U[1,255] weights, the layer builds and
update batches of 10K / 100K / 1M edges at 50/50 with every layer kept exact.

Multi-GPU (torchrun): replicas -- every rank holds the whole graph and runs its own 64 + 64
queries (weak scaling); the time is the max over ranks.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
import argparse
import importlib
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "BFS/SSSP GTEPS, updates/s on 1 B200; learned vs fixed schedule, bit-exact"
N_BFS = 64
N_SSSP = 64
DELTA = 16


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--workload", default="rmat_lj", choices=["rmat_lj", "rmat_s20", "rmat_s16", "lattice_2000"])
    p.add_argument("--no-updates", action="store_true")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--no-schedule", action="store_true", help="skip the learned-vs-fixed schedule comparison")
    p.add_argument("--no-batched", action="store_true", help="skip the batched queries + uneven batches section")
    p.add_argument("--no-incremental", action="store_true", help="skip the incremental BFS / SSSP section")
    p.add_argument("--no-single", action="store_true", help="skip the single-edge update latency section")
    p.add_argument("--stream", type=int, default=0, metavar="ROUNDS",
                   help="instead of the bench: the 41.6M-vertex / 1.47B-edge R-MAT (seed 5, weights U[1,1023]), "
                        "WCC + SCC build, then ROUNDS x (1M-edge batch 60/40 + 32 BFS + 32 SSSP), checked by "
                        "the size-independent certificates; one JSON line")
    p.add_argument("--only", choices=["bfs", "sssp", "build", "reach", "bc", "incr", "single"], default=None,
                   help="profiling runs: one call of one query kind (or the three layer builds and one 10K "
                        "update batch; 64K reachability pairs; betweenness over 64 sources; a 10K-op batch "
                        "and the incremental BFS / SSSP updates after it; 20 single-edge updates), no timing")
    return p.parse_args()


def workload(pkg, name):
    if name == "rmat_lj":
        return pkg.graphs.rmat_lj()
    if name == "rmat_s20":  # 1M vertices, 2^24 draws: a profiling case larger than L2
        return pkg.graphs.rmat(20, seed=3, permute=True, name="rmat_s20")
    if name == "lattice_2000":  # 4M vertices, the lattice procedure at side 2000: a profiling case
        return pkg.graphs.lattice(side=2000)
    return pkg.graphs.rmat_s16()


def run_only(args):
    """One call of one query kind (64 queries) on cuda:0, for ncu captures."""
    import torch
    pkg = importlib.import_module("graph-intermedia-representation_b200")
    g = workload(pkg, args.workload)
    d = pkg.DeviceGraph.from_graph(g)
    src = torch.from_numpy(pkg.graphs.sources_with_edges(g, 64, 11)).to("cuda:0")
    if args.only == "build":
        d.build(pkg.native.LAYER_ALL)
        u, v, ins = pkg.graphs.updates(g, 5000, 5000, 5)
        d.apply_batch(u, v, ins)
        torch.cuda.synchronize()
        print(json.dumps({"only": "build", "workload": args.workload, **d.counts()}))
        d.close()
        return
    if args.only in ("reach", "bc", "incr", "single"):
        import numpy as np
        d.build(pkg.native.LAYER_ALL)
        if args.only == "reach":
            rng = np.random.default_rng(77)
            n = 1 << 16
            ru = torch.from_numpy(rng.integers(0, g.V, n).astype(np.int32)).to("cuda:0")
            rv = torch.from_numpy(rng.integers(0, g.V, n).astype(np.int32)).to("cuda:0")
            d.reachable(ru, rv, out=torch.empty(n, dtype=torch.uint8, device="cuda:0"))
        elif args.only == "bc":
            d.bc(src, out=torch.empty(g.V, dtype=torch.float64, device="cuda:0"))
        elif args.only == "incr":
            s0 = int(src[0].item())
            d.inc_track(s0, False)
            d.inc_track(s0, True)
            u, v, ins = pkg.graphs.updates(g, 5000, 5000, 6)
            d.apply_batch(u, v, ins)
            d.inc_update(False)
            d.inc_update(True)
        else:
            rng = np.random.default_rng(5)
            cb, ca = d.csr(0)
            for i in range(20):
                a = int(rng.integers(g.V))
                while cb[a + 1] == cb[a]:
                    a = int(rng.integers(g.V))
                b = int(ca[cb[a] + rng.integers(cb[a + 1] - cb[a])]) if i % 2 == 0 else int(rng.integers(g.V))
                if a != b:
                    d.apply_batch(np.array([a], np.int32), np.array([b], np.int32), np.array([i % 2], np.uint8))
        torch.cuda.synchronize()
        print(json.dumps({"only": args.only, "workload": args.workload, **d.counts()}))
        d.close()
        return
    if args.only == "bfs":
        out = torch.empty((64, g.V), dtype=torch.int32, device="cuda:0")
        d.bfs(src, out=out)
    else:
        out = torch.empty((64, g.V), dtype=torch.int64, device="cuda:0")
        d.sssp(src, delta=DELTA, weights=pkg.native.WEIGHT_HASH, out=out)
    torch.cuda.synchronize()
    print(json.dumps({"only": args.only, "workload": args.workload, **d.query_stats()}))
    d.close()


def config(name, g):
    return {"workload": f"{name}: R-MAT a,b,c=.57/.19/.19, V={g.V}, E={g.E}"
                        + (", ids permuted, seed 3" if name == "rmat_lj" else ", seed 1"),
            "queries_per_step": {"bfs": N_BFS, "sssp": N_SSSP},
            "sssp_weights": "GIR::edgeWeight hash in [1,100] (the reference's), delta 16",
            "l2": "inputs larger than L2 (graph ~1.6 GB resident)",
            "parallelism": "replicas (one full graph per GPU, queries split by rank)"}


class Clocks:
    """nvidia-smi sampling during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        rows = []
        for line in open(self.path):
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


def measured_peak():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6650.0, "fallback"


def traffic_ratio(kernel):
    """DRAM bytes over algorithmic bytes of the dominant kernel, measured by ncu on a smaller case of
    the same kernel (the committed summary under profiles/), or None."""
    path = os.path.join(ROOT, "profiles", "traffic.json")
    try:
        with open(path) as f:
            r = json.load(f).get(kernel)
            return r.get("dram_over_algorithmic") if isinstance(r, dict) else None
    except (OSError, ValueError):
        return None


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def cpu_reference_sample(pkg, g, n_bfs, n_sssp, seed, budget_s=0.0):
    """The reference GIR (compiled from its sources) on this host's cores: bfs / sssp per source.
    With budget_s > 0, BFS and SSSP sources alternate until that much query time is sampled
    (n_bfs / n_sssp then only bound the counts)."""
    import numpy as np
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    kind = "reference" if oracle.ref_available() else "port"
    src = pkg.graphs.sources_with_edges(g, max(n_bfs, n_sssp), seed)
    outdeg = np.diff(g.fw_beg).astype(np.int64)
    counts = {"bfs": 0, "sssp": 0, "edges": 0, "t": 0.0}
    if kind == "reference":
        r = oracle.RefGIR(g.V, g.fw_beg, g.fw_adj, g.bw_beg, g.bw_adj)
        r.bfs(int(src[0]))  # warm (page faults of the query arrays)
        run_bfs = lambda s: r.bfs(int(s))
        run_sssp = lambda s: r.sssp(int(s), DELTA)
    else:
        fb = g.fw_beg.astype(np.int64)
        run_bfs = lambda s: oracle.bfs(g.V, fb, g.fw_adj, [s])
        run_sssp = lambda s: oracle.sssp(g.V, fb, g.fw_adj, [s])

    def one(kind_, s):
        t = time.perf_counter()
        out = run_bfs(s) if kind_ == "bfs" else run_sssp(s)
        counts["t"] += time.perf_counter() - t
        reached = out >= 0 if kind_ == "bfs" else out != np.iinfo(np.uint64).max
        counts["edges"] += int(outdeg[reached].sum())
        counts[kind_] += 1

    if budget_s > 0:
        i = 0
        while counts["t"] < budget_s and (counts["bfs"] < n_bfs or counts["sssp"] < n_sssp):
            if counts["bfs"] < n_bfs:
                one("bfs", src[i % len(src)])
            if counts["sssp"] < n_sssp and counts["t"] < budget_s:
                one("sssp", src[i % len(src)])
            i += 1
    else:
        for s in src[:n_bfs]:
            one("bfs", s)
        for s in src[:n_sssp]:
            one("sssp", s)
    if kind == "reference":
        r.close()
    return counts["edges"], counts["t"], kind, counts["bfs"], counts["sssp"]


def run_reference(args):
    world, rank, local = dist_setup()
    if rank != 0:
        return
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    if not oracle.ref_available():  # (the oracle is this repository's code, not the reference's)
        print(json.dumps({"impl": "reference", "unavailable": "the reference compiled from its sources "
                          "(oracle/_ref/libgirref.so) is not here, and its sources are not either"}), flush=True)
        return
    os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count()))
    os.environ.setdefault("OMP_PROC_BIND", "close")
    pkg = importlib.import_module("graph-intermedia-representation_b200")
    g = workload(pkg, args.workload)
    n_bfs, n_sssp = 4, 4  # (the step's 1:1 mix of BFS and SSSP queries)
    for w in range(args.warmup):
        cpu_reference_sample(pkg, g, 1, 0, 100 + w)
    edges = 0
    t = 0.0
    kind = "reference"
    for s in range(args.steps):
        e, dt, kind, _, _ = cpu_reference_sample(pkg, g, n_bfs, n_sssp, 7 + s)
        edges += e
        t += dt
    gteps = edges / t / 1e9
    cores = int(os.environ["OMP_NUM_THREADS"])
    sample = f"{n_bfs} bfs + {n_sssp} sssp(delta={DELTA}) sources per step of the same graph"
    line = {"impl": "reference", "metric": METRIC, "value": gteps, "unit": "GTEPS", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * t / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32 levels, uint64 sums",
            "data": "synthetic", "config": config(args.workload, g),
            "cpu_baseline": {"value": gteps, "unit": "GTEPS", "cores": cores, "kind": kind, "sample": sample},
            "e2e": {"value": gteps, "unit": "GTEPS", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def reference_instance(pkg, d):
    """The reference GIR (compiled from its sources) holding the device graph's current edges,
    and the host seconds its construction took; None when the reference is not compiled here.
    The device's create is timed on the same int32 arrays (sorted rows) beside it."""
    import numpy as np
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    if not oracle.ref_available():
        return None, {}
    cb, ca = d.csr(0)
    bb, ba = d.csr(1)
    arrs = (cb.astype(np.int32), ca, bb.astype(np.int32), ba)
    t = time.perf_counter()
    ref = oracle.RefGIR(d.V, *arrs)
    t_ref = time.perf_counter() - t
    t = time.perf_counter()
    d2 = pkg.DeviceGraph.create(*arrs, d.V)
    t_dev = time.perf_counter() - t
    d2.close()
    return ref, {"device_s": t_dev, "reference_s": t_ref,
                 "input": f"int32 four-array CSR of the current graph (V={d.V}, E={len(ca)}), host memory"}


def stream_protocol_section(pkg, with_reference, scale=18, batch=10000, batches=10):
    """The reference's streaming protocol (experiments/baselines/gir/gir_stream.cpp): one exported
    protocol (R-MAT scale `scale`, half its edges loaded, insert / delete / mixed streams), run by
    this package's gir_stream on the GPU and by the reference's own driver on the host cores, in
    the applyBatch, lazy (ingestBatch + sync) and incremental modes. Rows: mutation MEPS per
    stream, BFS and SSSP end-to-end ms per batch, the lazy mode's sync ms, incremental mismatches."""
    import tempfile
    st = importlib.import_module("graph-intermedia-representation_b200.stream")
    ref_driver = os.path.join(ROOT, "oracle", "_ref", "gir_stream_ref")
    g = pkg.graphs.rmat(scale, seed=8, permute=True, weights=None)
    keep = ("mutation_MEPS", "endtoend_ms", "sync_", "inc_mismatch")
    out = {"graph": f"R-MAT scale {scale}, V={g.V}", "batch": batch, "batches": batches}
    with tempfile.TemporaryDirectory() as d:
        out["protocol"] = st.export_protocol(g, d, ops_per_stream=batch * batches)
        out["protocol"].pop("sources", None)
        systems = [("device", st.DRIVER)] + ([("reference", ref_driver)] if with_reference and os.path.exists(ref_driver) else [])
        for name, binary in systems:
            res = {}
            for mode in ("", "lazy", "inc"):
                rows = st.run_driver(binary, d, f"rmat_s{scale}", os.path.join(d, f"{name}.csv"), batch, batches, mode)
                res[mode or "fmu"] = {r["metric"]: round(r["value"], 4) for r in rows if any(k in r["metric"] for k in keep)}
            out[name] = res
    return out


def two_level_section(pkg, d, ref, native, n_src=4):
    """The reference's two-level queries (GIR::bfsTwoLevel / ssspTwoLevel, gir_query.cpp:604-722: a
    wavefront over the condensation DAG with block tasks in the source SCC) beside its flat bfs /
    sssp and the device's flat single-source query, from the same sources on the same graph
    (host wall clock per source; delta 16, hash weights); every result must agree."""
    import numpy as np
    fb, fa = d.csr(0)
    src = pkg.graphs.sources_with_edges(pkg.graphs.Graph(d.V, fb.astype(np.int32), fa, None, None), n_src, 23)
    t = {"ref_bfs": 0.0, "ref_bfs_two_level": 0.0, "ref_sssp": 0.0, "ref_sssp_two_level": 0.0,
         "device_bfs": 0.0, "device_sssp": 0.0}
    same = True
    d.bfs(src[:1])
    d.sssp(src[:1], delta=DELTA)
    for s in src.tolist():
        t0 = time.perf_counter(); a = ref.bfs(s); t1 = time.perf_counter(); b = ref.bfs_two_level(s)
        t2 = time.perf_counter(); c = ref.sssp(s, DELTA); t3 = time.perf_counter(); e = ref.sssp_two_level(s, DELTA)
        t4 = time.perf_counter(); x = d.bfs([s])[0]; t5 = time.perf_counter(); y = d.sssp([s], delta=DELTA)[0]
        t6 = time.perf_counter()
        for k, dt in zip(t, (t1 - t0, t2 - t1, t3 - t2, t4 - t3, t5 - t4, t6 - t5)):
            t[k] += dt * 1e3 / len(src)
        same &= bool(np.array_equal(a, b) and np.array_equal(a, x) and np.array_equal(c, e) and np.array_equal(c, y))
    return {"ms_per_source": {k: round(v, 3) for k, v in t.items()}, "identical": same, "sources": len(src),
            "note": "host wall clock per single-source call; device calls include the copy of the V-entry result row"}


def cpu_model():
    """The host CPU's model name and logical core count."""
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    return f"{line.split(':', 1)[1].strip()} ({os.cpu_count()} logical cores)"
    except OSError:
        pass
    return f"unknown ({os.cpu_count()} logical cores)"


def parity_vs_reference(pkg, d, ref, native, n_src=4):
    """Bit-exactness of the device's layers and queries against the reference on the same graph
    (canonical forms): WCC, SCC, condensation-DAG key set, blocks, articulation points, BFS levels
    and SSSP distances (delta 16, hash weights) from n_src sources each."""
    import numpy as np
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    t0 = time.perf_counter()
    res = {"wcc": bool(np.array_equal(d.labels(native.LABEL_WCC), ref.wcc())),
           "scc": bool(np.array_equal(d.labels(native.LABEL_SCC), ref.scc()))}
    s, t = d.dag()
    res["dag"] = bool(np.array_equal(np.unique((s.astype(np.int64) << 32) | t.astype(np.int64)), ref.dag()))
    label, head = d.blocks()
    res["blocks"] = bool(np.array_equal(oracle.canon_blocks_from_device(label, head), ref.blocks()))
    res["articulation_points"] = bool(np.array_equal(d.labels(native.LABEL_BCNT) >= 2, ref.ap()))
    fb, fa = d.csr(0)
    src = pkg.graphs.sources_with_edges(pkg.graphs.Graph(d.V, fb.astype(np.int32), fa, None, None), n_src, 17)
    lv = d.bfs(src)
    ds = d.sssp(src, delta=DELTA, weights=native.WEIGHT_HASH)
    res["bfs_rows"] = bool(all(np.array_equal(lv[i], ref.bfs(int(x))) for i, x in enumerate(src)))
    res["sssp_rows"] = bool(all(np.array_equal(ds[i], ref.sssp(int(x), DELTA)) for i, x in enumerate(src)))
    res["state"] = "after the build and the 10K, 100K and 1M-edge batches of updates_per_s"
    res["check_s"] = time.perf_counter() - t0
    return res


def single_edge_section(pkg, d, ref, ref_builds, n_ops=100):
    """Single-edge updates (insertEdge / deleteEdge, gir.cpp:3043-3134) on the current graph with
    every layer kept exact: n_ops ops alternating between deleting an existing edge and inserting
    a random pair, one call each, host wall clock per call (the call returns after the device is
    done). With ref the reference (its three layers built on the host cores first) takes the same
    ops through updateEdgeDirected, and afterwards both WCC and SCC partitions must agree."""
    import numpy as np
    rng = np.random.default_rng(321)
    V = d.V
    cb, ca = d.csr(0)
    ops = []
    for i in range(n_ops):
        if i % 2 == 0:
            a = int(rng.integers(V))
            while cb[a + 1] == cb[a]:
                a = int(rng.integers(V))
            ops.append((a, int(ca[cb[a] + rng.integers(cb[a + 1] - cb[a])]), 0))
        else:
            a, b = int(rng.integers(V)), int(rng.integers(V))
            ops.append((a, b if b != a else (a + 1) % V, 1))
    res = {"ops": n_ops}
    if ref is not None:
        res.update(ref_builds)  # the reference's layers were built before the update batches
        res["ref_threads"] = int(os.environ.get("OMP_NUM_THREADS", os.cpu_count()))
    st0 = d.single_stats()
    dev_ms, plans, phases, per_op = [], {"wcc": {}, "scc": {}, "bct": {}}, {0: [], 1: []}, []
    for a, b, i in ops:
        t = time.perf_counter()
        d.apply_batch(np.array([a], np.int32), np.array([b], np.int32), np.array([i], np.uint8))
        dev_ms.append((time.perf_counter() - t) * 1e3)
        ph = d.batch_times()
        ph["checks"] = dev_ms[-1] - sum(ph.values())  # (the searches run between the phases)
        phases[i].append(ph)
        plan = d.batch_plan()
        for k, x in plan.items():
            plans[k][x] = plans[k].get(x, 0) + 1
        # (kind, ms, search ms, decisions as three letters: k kept, p patched, r rebuilt)
        per_op.append(["di"[i], round(dev_ms[-1], 2), round(ph["checks"], 2), "".join(x[0] for x in plan.values())])
    st1 = d.single_stats()
    by_kind = {}
    for i, name in ((0, "delete"), (1, "insert")):
        ms = [sum(p.values()) for p in phases[i]]
        by_kind[name] = {"median_ms": float(np.median(ms)),
                         "phase_median_ms": {k: round(float(np.median([p[k] for p in phases[i]])), 3)
                                             for k in phases[i][0]}}
    res.update(device_median_ms=float(np.median(dev_ms)), device_mean_ms=float(np.mean(dev_ms)),
               device_p90_ms=float(np.percentile(dev_ms, 90)), by_kind=by_kind, layer_decisions=plans,
               per_op=per_op,
               checked=st1["checked"] - st0["checked"], rebuilds_avoided=st1["kept"] - st0["kept"])
    if ref is not None:
        ref_ms = []
        for a, b, i in ops:
            t = time.perf_counter()
            ref.update_edge(a, b, bool(i))
            ref_ms.append((time.perf_counter() - t) * 1e3)
        res.update(ref_median_ms=float(np.median(ref_ms)), ref_mean_ms=float(np.mean(ref_ms)),
                   ref_p90_ms=float(np.percentile(ref_ms, 90)))
        res["scc_identical_to_reference"] = bool(np.array_equal(d.labels(pkg.native.LABEL_SCC), ref.scc()))
        res["wcc_identical_to_reference"] = bool(np.array_equal(d.labels(pkg.native.LABEL_WCC), ref.wcc()))
    return res


def incremental_section(pkg, d, stream, dev, src, ref):
    """Incremental single-source BFS / SSSP (GIR::trackIncremental / updateIncremental) on the
    current graph: batches of 1K / 10K / 100K ops (two thirds deletions of existing edges, one third
    random insertions), each applied (untimed here) and followed by the update of both tracked
    results, timed against a from-scratch query of the same source; after every update both results
    must equal the from-scratch ones. With with_ref the reference (compiled from its sources) tracks
    the same source and takes the same batches (ingestBatch); its updateIncremental is timed on the
    host cores beside the device's and its results must equal the device's (ref: the instance
    from reference_instance, or None)."""
    import numpy as np
    import torch
    V = d.V
    rng = np.random.default_rng(123)
    s_d = torch.tensor([src], dtype=torch.int32, device=dev)
    ds1 = torch.empty((1, V), dtype=torch.int64, device=dev)
    lv1 = torch.empty((1, V), dtype=torch.int32, device=dev)
    inc = torch.empty(V, dtype=torch.int64, device=dev)
    d.sssp(s_d, delta=DELTA, out=ds1)  # warm
    res = {"source": src, "scratch_ms": {"sssp": ev_time(stream, lambda: d.sssp(s_d, delta=DELTA, out=ds1)),
                                         "bfs": ev_time(stream, lambda: d.bfs(s_d, out=lv1))},
           "track_ms": {"sssp": ev_time(stream, lambda: d.inc_track(src, True)),
                        "bfs": ev_time(stream, lambda: d.inc_track(src, False))}, "batches": {}}
    cb, ca = d.csr(0)
    if ref is not None:
        t = time.perf_counter()
        ref.inc_track(src, True)
        ref.inc_track(src, False)
        res["ref_track_s"] = time.perf_counter() - t
        res["ref_threads"] = int(os.environ.get("OMP_NUM_THREADS", os.cpu_count()))
    none = np.iinfo(np.uint64).max
    for k in (1_000, 10_000, 100_000):
        a = rng.integers(0, V, 2 * k // 3)
        a = a[cb[a + 1] > cb[a]]
        b = ca[cb[a] + rng.integers(0, 1 << 30, len(a)) % (cb[a + 1] - cb[a])]
        n_ins = k - len(a)
        u = np.concatenate([a, rng.integers(0, V, n_ins)]).astype(np.int32)
        v = np.concatenate([b, rng.integers(0, V, n_ins)]).astype(np.int32)
        ins = np.concatenate([np.zeros(len(a)), np.ones(n_ins)]).astype(np.uint8)
        d.apply_batch(u, v, ins)
        row = {"ops": k, "sssp_update_ms": ev_time(stream, lambda: d.inc_update(True))}
        st = d.query_stats()
        row.update(cut_vertices=st["reached"], rounds=st["iterations"], relaxed_entries=st["edges"])
        row["bfs_update_ms"] = ev_time(stream, lambda: d.inc_update(False))
        d.sssp(s_d, delta=DELTA, out=ds1)
        d.inc_dist(True, out=inc)
        ok_w = bool(torch.equal(inc, ds1[0]))
        d.bfs(s_d, out=lv1)
        d.inc_dist(False, out=inc)
        lv = lv1[0].to(torch.int64)
        ok_b = bool(torch.equal(inc, torch.where(lv < 0, torch.full_like(lv, -1), lv)))
        row["identical_to_scratch"] = ok_w and ok_b
        if ref is not None:
            ref.ingest_batch(u, v, ins)
            t = time.perf_counter()
            ref.inc_update(True)
            row["ref_sssp_update_ms"] = (time.perf_counter() - t) * 1e3
            t = time.perf_counter()
            ref.inc_update(False)
            row["ref_bfs_update_ms"] = (time.perf_counter() - t) * 1e3
            dw = d.inc_dist(True)
            db = d.inc_dist(False)
            row["identical_to_reference"] = bool(np.array_equal(dw, ref.inc_dist(True)) and
                                                 np.array_equal(db, ref.inc_dist(False)))
            assert dw[src] == 0 and db[src] == 0 and (dw != none).sum() == (db != none).sum()
        res["batches"][str(k)] = row
        cb, ca = d.csr(0)
    return res


def ev_time(stream, fn):
    """Device ms of fn() between CUDA events on the handle's stream."""
    import torch
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(stream)
    fn()
    e1.record(stream)
    e1.synchronize()
    return e0.elapsed_time(e1)


def compare_schedules(pkg, d, stream, sb, ss, lv, ds, weights, delta_fixed, reps, mean_weight=None):
    """The same BFS and SSSP sources under the fixed heuristics (the reference's alpha/beta switch
    and delta) and under the trained schedule network; results must be identical. With
    mean_weight, SSSP also runs with a one-line weight rule (delta = the candidate nearest, in log
    scale, to the mean edge weight) as a second baseline for the network's delta."""
    import torch
    native = pkg.native
    out = {}
    lv2, ds2 = torch.empty_like(lv), torch.empty_like(ds)
    d.set_schedule(native.SCHEDULE_FIXED)
    d.bfs(sb, out=lv)
    # (builds the weight-sorted rows and the cached lane order of the 64 sources, so neither arm
    # pays that one-time setup inside its timing)
    d.sssp(ss, delta=2048, weights=weights, out=ds)
    t_bf = min(ev_time(stream, lambda: d.bfs(sb, out=lv)) for _ in range(reps))
    t_sf = min(ev_time(stream, lambda: d.sssp(ss, delta=delta_fixed, weights=weights, out=ds)) for _ in range(reps))
    d.use_learned_schedule()
    d.bfs(sb, out=lv2)
    t_bl = min(ev_time(stream, lambda: d.bfs(sb, out=lv2)) for _ in range(reps))
    _, y_bfs = d.sched_trace()
    t_sl = min(ev_time(stream, lambda: d.sssp(ss, delta=0, weights=weights, out=ds2)) for _ in range(reps))
    _, y_sssp = d.sched_trace()
    d.set_schedule(native.SCHEDULE_FIXED)
    choices = pkg.DeviceGraph.delta_choices()
    out["bfs"] = {"fixed_ms": t_bf, "learned_ms": t_bl, "speedup": t_bf / t_bl, "identical": bool(torch.equal(lv, lv2)),
                  "learned_bottom_up_levels": int((y_bfs == 1).sum()), "levels": int(len(y_bfs))}
    out["sssp"] = {"fixed_ms": t_sf, "learned_ms": t_sl, "speedup": t_sf / t_sl, "identical": bool(torch.equal(ds, ds2)),
                   "fixed_delta": delta_fixed,
                   "learned_delta": [int(choices[c - 2]) for c in y_sssp.tolist() if c >= 2]}
    out["both_speedup"] = (t_bf + t_sf) / (t_bl + t_sl)
    if mean_weight:
        import math
        rule = int(min(choices, key=lambda c: abs(math.log2(c) - math.log2(mean_weight))))
        ds3 = torch.empty_like(ds)
        d.sssp(ss, delta=rule, weights=weights, out=ds3)
        t_sr = min(ev_time(stream, lambda: d.sssp(ss, delta=rule, weights=weights, out=ds3)) for _ in range(reps))
        out["sssp"]["weight_rule"] = {"delta": rule, "ms": t_sr, "speedup_vs_fixed": t_sf / t_sr,
                                      "learned_vs_rule": t_sr / t_sl, "identical": bool(torch.equal(ds, ds3)),
                                      "mean_weight": mean_weight}
    return out


def batched_section(pkg, d, g, stream, dev, rounds=64, seed=90):
    """Source sets of log-uniform size in [1, 4096] (16 BFS + 4 SSSP sets per round) interleaved
    with update batches of log-uniform size in [1, 1M] (half inserts; 70% of the deletions drawn
    from edges inside an SCC, the rest from all edges), after autotuning the launch parameters."""
    import numpy as np
    import torch
    native = pkg.native
    rng = np.random.default_rng(seed)
    V = g.V
    tune = d.autotune(pkg.graphs.sources_with_edges(g, 64, seed), reps=1)
    scc = d.labels(native.LABEL_SCC)
    rows = np.repeat(np.arange(V, dtype=np.int32), np.diff(g.fw_beg))
    intra = np.nonzero(scc[rows] == scc[g.fw_adj])[0]

    def log_uniform(hi, n):
        return np.exp(rng.uniform(0, np.log(hi), n)).astype(np.int64).clip(1, hi)

    plan = []
    for r in range(rounds):
        k = int(log_uniform(1_000_000, 1)[0])
        ni, nd = (k + 1) // 2, k // 2
        n_in = int(round(0.7 * nd))
        e = np.concatenate([rng.choice(intra, n_in), rng.integers(0, len(rows), nd - n_in)])
        u = np.concatenate([rng.integers(0, V, ni).astype(np.int32), rows[e]])
        v = np.concatenate([rng.integers(0, V, ni).astype(np.int32), g.fw_adj[e]])
        ins = np.concatenate([np.ones(ni, np.uint8), np.zeros(nd, np.uint8)])
        bsets = [rng.integers(0, V, int(m)).astype(np.int32) for m in log_uniform(4096, 16)]
        ssets = [rng.integers(0, V, int(m)).astype(np.int32) for m in log_uniform(4096, 4)]
        plan.append((u, v, ins, bsets, ssets))
    lv = torch.empty((16, V), dtype=torch.int32, device=dev)
    ds = torch.empty((4, V), dtype=torch.int64, device=dev)
    edges = {"bfs": 0, "sssp": 0}
    n_upd = 0
    plans = {"wcc": {}, "scc": {}, "bct": {}}

    def run():
        nonlocal n_upd
        for u, v, ins, bsets, ssets in plan:
            d.apply_batch(u, v, ins)
            n_upd += len(u)
            for k2, x in d.batch_plan().items():
                plans[k2][x] = plans[k2].get(x, 0) + 1
            d.bfs_sets(bsets, out=lv)
            edges["bfs"] += d.query_stats()["edges"]
            d.sssp_sets(ssets, out=ds)
            edges["sssp"] += d.query_stats()["edges"]

    ms = ev_time(stream, run)
    return {"rounds": rounds, "ms": ms, "updates": n_upd, "updates_per_s": n_upd / (ms * 1e-3),
            "bfs_sets": 16 * rounds, "sssp_sets": 4 * rounds,
            "query_gteps": (edges["bfs"] + edges["sssp"]) / (ms * 1e-3) / 1e9, "autotuned": tune,
            "repair_plans": plans,
            "note": "one timed region: batches, then the round's BFS and SSSP source sets (delta 16, hash "
                    "weights), every layer kept exact after every batch"}


def run_stream(args):
    """The large power-law configuration as a stream (see --stream)."""
    import numpy as np
    import torch
    pkg = importlib.import_module("graph-intermedia-representation_b200")
    vf = importlib.import_module("graph-intermedia-representation_b200.verify")
    native = pkg.native
    t0 = time.time()
    g = pkg.graphs.rmat_tw()
    t_gen = time.time() - t0
    d = pkg.DeviceGraph.from_graph(g)
    stream = torch.cuda.ExternalStream(d.stream(), device="cuda:0")
    t_create = time.time() - t0 - t_gen
    builds = {"wcc_ms": ev_time(stream, lambda: d.build(native.LAYER_WCC)),
              "scc_dag_ms": ev_time(stream, lambda: d.build(native.LAYER_SCC))}
    lv = torch.empty((32, g.V), dtype=torch.int32, device="cuda:0")
    ds = torch.empty((32, g.V), dtype=torch.int64, device="cuda:0")
    rows = []
    for r in range(args.stream):
        u, v, ins = pkg.graphs.updates(g, 600_000, 400_000, 500 + r)
        t_b = ev_time(stream, lambda: d.apply_batch(u, v, ins))
        src = torch.from_numpy(pkg.graphs.sources_with_edges(g, 32, 600 + r)).to("cuda:0")
        t_q = ev_time(stream, lambda: d.bfs(src, out=lv))
        e_b = d.query_stats()["edges"]
        t_s = ev_time(stream, lambda: d.sssp(src, delta=0 if r % 2 else 16, weights=native.WEIGHT_STORED, out=ds))
        e_s = d.query_stats()["edges"]
        rows.append({"batch_ms": t_b, "bfs_ms": t_q, "bfs_gteps": e_b / (t_q * 1e-3) / 1e9, "sssp_ms": t_s,
                     "sssp_gteps": e_s / (t_s * 1e-3) / 1e9, "sssp_schedule": "learned" if r % 2 else "fixed",
                     "plan": d.batch_plan()})
        if r == 0:
            d.use_learned_schedule()
    fb, fa = d.csr(0)
    s_last = src.cpu().numpy()
    cert = {"bfs": vf.bfs_levels(fb, fa, [s_last[0]], lv[0]), "wcc": vf.wcc_labels(fb, fa, d.labels(native.LABEL_WCC))}
    s_d, t_d = d.dag()
    cert["scc_dag"] = vf.scc_dag(fb, fa, d.labels(native.LABEL_SCC), d.labels(native.LABEL_SCC_RANK), s_d, t_d)
    d.sssp(src[:1], delta=0, weights=native.WEIGHT_HASH, out=ds[:1])
    cert["sssp_hash"] = vf.sssp_dists(fb, fa, [s_last[0]], ds[0])
    c = d.counts()
    print(json.dumps({"stream": "rmat_tw", "V": c["V"], "E": c["E"], "n_scc": c["n_scc"], "n_wcc": c["n_wcc"],
                      "generate_s": t_gen, "create_s": t_create, "build": builds, "rounds": rows,
                      "updates_per_s": 1e6 * len(rows) / (1e-3 * sum(x["batch_ms"] for x in rows)),
                      "certificate_violations": cert}), flush=True)
    d.close()


def run_ours(args):
    import numpy as np
    import torch
    world, rank, local = dist_setup()
    torch.cuda.set_device(local)
    pg = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
        pg = dist
    pkg = importlib.import_module("graph-intermedia-representation_b200")
    native = pkg.native
    g = workload(pkg, args.workload)
    d = pkg.DeviceGraph.from_graph(g)
    stream = torch.cuda.ExternalStream(d.stream(), device=f"cuda:{local}")
    V = g.V
    src_bfs = pkg.graphs.sources_with_edges(g, N_BFS, 11 + 1000 * rank)
    src_sssp = pkg.graphs.sources_with_edges(g, N_SSSP, 12 + 1000 * rank)
    dev = f"cuda:{local}"
    lv_d = torch.empty((N_BFS, V), dtype=torch.int32, device=dev)
    ds_d = torch.empty((N_SSSP, V), dtype=torch.int64, device=dev)
    sb_d = torch.from_numpy(src_bfs).to(dev)
    ss_d = torch.from_numpy(src_sssp).to(dev)

    def step(lv, ds, sb, ss):
        d.bfs(sb, out=lv)
        qb = d.query_stats()
        d.sssp(ss, delta=DELTA, weights=native.WEIGHT_HASH, out=ds)
        qs = d.query_stats()
        return qb, qs

    def barrier():
        torch.cuda.synchronize()
        if pg is not None:
            pg.barrier()

    def timed(fn, steps):
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        barrier()
        ev0.record(stream)
        stats = [fn() for _ in range(steps)]
        ev1.record(stream)
        ev1.synchronize()
        barrier()
        ms = ev0.elapsed_time(ev1)
        if pg is not None:
            t = torch.tensor([ms], device=dev)
            pg.all_reduce(t, op=pg.ReduceOp.MAX)
            ms = float(t.item())
        return ms, stats

    # launch parameters picked by the library's autotuner on this step's BFS sources (setup, untimed)
    tuned = d.autotune(sb_d, reps=1)
    for _ in range(args.warmup):
        step(lv_d, ds_d, sb_d, ss_d)
    clocks = Clocks(local)
    clocks.start()
    ms, stats = timed(lambda: step(lv_d, ds_d, sb_d, ss_d), args.steps)
    clk = clocks.stop()
    edges_step = stats[0][0]["edges"] + stats[0][1]["edges"]
    bfs_ms = sum(s[0]["total_ms"] for s in stats) / args.steps
    sssp_ms = sum(s[1]["total_ms"] for s in stats) / args.steps
    launches = sum(s[0]["launches"] + s[1]["launches"] for s in stats)
    total_edges = edges_step * args.steps * world
    value = total_edges / (ms * 1e-3) / 1e9

    # e2e: pinned host buffers through the same C-ABI calls
    lv_h = torch.empty((N_BFS, V), dtype=torch.int32, pin_memory=True)
    ds_h = torch.empty((N_SSSP, V), dtype=torch.int64, pin_memory=True)
    sb_h = torch.from_numpy(src_bfs).pin_memory()
    ss_h = torch.from_numpy(src_sssp).pin_memory()
    step(lv_h, ds_h, sb_h, ss_h)
    ms_e2e, _ = timed(lambda: step(lv_h, ds_h, sb_h, ss_h), args.steps)
    e2e = {"value": total_edges / (ms_e2e * 1e-3) / 1e9, "unit": "GTEPS",
           "h2d_bytes_per_step": int(sb_h.numel() * 4 + ss_h.numel() * 4),
           "d2h_bytes_per_step": int(lv_h.numel() * 4 + ds_h.numel() * 8), "ms_per_step": ms_e2e / args.steps}
    # parity spot check of the e2e results against the device-resident run
    assert torch.equal(lv_h, lv_d.cpu()) and torch.equal(ds_h, ds_d.cpu()), "host and device runs disagree"

    # roofline of the dominant kernel (live CUDA events around its launches)
    d.set_param(native.PARAM_PROFILE, 1)
    qb, qs = step(lv_d, ds_d, sb_d, ss_d)
    d.set_param(native.PARAM_PROFILE, 0)
    bfs_bytes = 4 * qb["edges"] + 12 * qb["reached"] + 4 * V * N_BFS
    sssp_bytes = 8 * qs["edges"] + 16 * qs["reached"] + 8 * V * N_SSSP
    if qs["main_ms"] >= qb["main_ms"]:
        kern, kb, kms, kl = "k_relax (SSSP)", sssp_bytes, qs["main_ms"], qs["main_launches"]
    else:
        kern, kb, kms, kl = "BFS level kernels", bfs_bytes, qb["main_ms"], qb["main_launches"]
    peak, peak_src = measured_peak()
    achieved = kb / (kms * 1e-3) / 1e9
    ratio = traffic_ratio(kern)
    tr = ratio * kb / max(kl, 1) if ratio else None
    roofline = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "traffic": tr, "kernel": kern, "launches": kl, "kernel_ms": kms,
                "algorithmic_bytes": kb, "algorithmic_bytes_per_launch": kb / max(kl, 1),
                "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of every launch of one 64-source "
                                  "call on the 1M-vertex R-MAT (rmat_s20), as a ratio to that call's algorithmic "
                                  "bytes, times this call's algorithmic bytes per launch" if tr else None,
                "peak_source": f"{peak_src} (MEASURED_PEAKS.json hbm_gbs)"}

    # SSSP with the stored U[1,255] weights (the configuration's weights), reported beside
    d.sssp(ss_d, delta=DELTA, weights=native.WEIGHT_STORED, out=ds_d)
    qst = d.query_stats()
    extra = {"autotuned": tuned, "bfs_gteps": stats[0][0]["edges"] / (bfs_ms * 1e-3) / 1e9,
             "bfs_roofline": {"kernels": "BFS level kernels (top-down expand, bottom-up bins)",
                              "algorithmic_bytes": bfs_bytes, "kernel_ms": qb["main_ms"],
                              "achieved": bfs_bytes / (qb["main_ms"] * 1e-3) / 1e9 if qb["main_ms"] else None,
                              "frac": bfs_bytes / (qb["main_ms"] * 1e-3) / 1e9 / peak if qb["main_ms"] else None},
             "sssp_gteps": stats[0][1]["edges"] / (sssp_ms * 1e-3) / 1e9,
             "sssp_stored_u255_gteps": qst["edges"] / (qst["total_ms"] * 1e-3) / 1e9,
             "bfs_ms_per_64": bfs_ms, "sssp_ms_per_64": sssp_ms}

    # learned vs fixed schedule on this graph (same sources, identical results required)
    if not args.no_schedule:
        sch = {args.workload: compare_schedules(pkg, d, stream, sb_d, ss_d, lv_d, ds_d, native.WEIGHT_HASH, DELTA, 2,
                                                mean_weight=50.5)}  # (GIR::edgeWeight is uniform on [1, 100])

    # layer builds and update batches (every layer kept exact)
    upd = {}
    if not args.no_updates:
        # each build twice: the first call also grows the handle's memory pool to the build's
        # working set; the repeat is the steady state (what a rebuild after a batch costs)
        builds = {}
        for name, layer in (("wcc", native.LAYER_WCC), ("scc_dag", native.LAYER_SCC), ("bct", native.LAYER_BCT)):
            builds[f"{name}_ms"] = ev_time(stream, lambda: d.build(layer))
            builds[f"{name}_repeat_ms"] = ev_time(stream, lambda: d.build(layer))
        extra["build"] = builds
        u, v, ins = pkg.graphs.updates(g, 5000, 5000, 49)  # untimed warm-up batch
        d.apply_batch(u, v, ins)
        rep = None
        if world > 1:  # replicas: rank 0's batch is broadcast, so every replica stays identical
            rep = importlib.import_module("graph-intermedia-representation_b200.replicas").Replicas(d)
        # the reference on the host cores, holding the same graph (create timed beside the
        # device's), its three layers built; it takes the same batches, timed beside the device's
        ref, ref_builds = None, {}
        if rank == 0 and world == 1 and not args.no_cpu:
            os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count()))
            ref, extra["create_from_csr"] = reference_instance(pkg, d)
            if ref is not None:
                for mask, name in ((1, "wcc"), (2, "scc_dag"), (4, "bct")):
                    t0 = time.perf_counter()
                    ref.build(mask)
                    ref_builds[f"ref_build_{name}_s"] = time.perf_counter() - t0
        upd_ref = {}
        for n in (10_000, 100_000, 1_000_000):
            if rep is not None:
                u, v, ins = rep.broadcast_batch(*(pkg.graphs.updates(g, n // 2, n // 2, 50 + n) if rank == 0 else ()))
            else:
                u, v, ins = pkg.graphs.updates(g, n // 2, n // 2, 50 + n)
            ub, vb, ib = (torch.from_numpy(x).pin_memory() for x in (u, v, ins))
            t = ev_time(stream, lambda: d.apply_batch(ub.numpy(), vb.numpy(), ib.numpy()))
            upd[str(n)] = n / (t * 1e-3)
            extra.setdefault("update_phases_ms", {})[str(n)] = {k: round(x, 2) for k, x in d.batch_times().items()}
            extra.setdefault("update_plans", {})[str(n)] = d.batch_plan()
            if ref is not None:
                t0 = time.perf_counter()
                ref.apply_batch(u, v, ins)
                upd_ref[str(n)] = n / (time.perf_counter() - t0)
        extra["updates_per_s"] = upd
        if ref is not None:
            extra["updates_per_s_reference"] = {
                "value": upd_ref, "cores": int(os.environ.get("OMP_NUM_THREADS", os.cpu_count())),
                "cpu": cpu_model(), "note": "GIR::applyBatch of the reference compiled from its sources, the same "
                                            "batches on the same graph, host wall clock"}
            extra["full_size_parity"] = parity_vs_reference(pkg, d, ref, native)
            extra["two_level"] = two_level_section(pkg, d, ref, native)
        # reachability (GIR::reachable) for 64K random pairs on the current graph, device arrays
        n_r = 1 << 16
        rng = np.random.default_rng(77)
        ru = torch.from_numpy(rng.integers(0, V, n_r).astype(np.int32)).to(dev)
        rv = torch.from_numpy(rng.integers(0, V, n_r).astype(np.int32)).to(dev)
        rout = torch.empty(n_r, dtype=torch.uint8, device=dev)
        d.reachable(ru[:64], rv[:64], out=rout[:64])
        t_r = ev_time(stream, lambda: d.reachable(ru, rv, out=rout))
        # betweenness (GIR::bc) over the step's 64 BFS sources
        bc_out = torch.empty(V, dtype=torch.float64, device=dev)
        d.bc(sb_d, out=bc_out)  # (warm-up: the first call grows the memory pool by its 7 GB of lanes)
        t_bc = ev_time(stream, lambda: d.bc(sb_d, out=bc_out))
        extra["bc_64_sources_ms"] = t_bc
        # single-edge update latency (every layer kept exact), beside the reference's; first, since
        # the reference's single-edge entry points sync the batches ingestBatch leaves pending
        if not args.no_single:
            extra["single_edge_updates"] = single_edge_section(pkg, d, ref, ref_builds)
        # incremental BFS / SSSP of one source under 1K / 10K / 100K-op batches
        if not args.no_incremental:
            extra["incremental"] = incremental_section(pkg, d, stream, dev, int(sb_d[0].item()), ref)
        if ref is not None:
            ref.close()
        extra["reachable"] = {"pairs": n_r, "ms": t_r, "pairs_per_s": n_r / (t_r * 1e-3),
                              "true_fraction": float(rout.float().mean().item())}
        if rep is not None:
            extra["replicas_agree_checksum"] = rep.check_agree()

    # the reference's streaming protocol, both drivers on the same protocol files
    if not args.no_updates and rank == 0:
        extra["stream_protocol"] = stream_protocol_section(pkg, with_reference=world == 1 and not args.no_cpu)

    # batched source sets interleaved with uneven update batches (on the updated graph)
    if not args.no_batched and not args.no_updates:
        extra["batched"] = batched_section(pkg, d, g, stream, dev)

    # the high-diameter lattice (4,900 x 4,900, stored Euclidean weights): where the fixed delta
    # and alpha/beta are far from the best schedule
    if not args.no_schedule:
        d.close()
        del lv_d, ds_d, lv_h, ds_h
        torch.cuda.empty_cache()
        gl = pkg.graphs.lattice()
        d = pkg.DeviceGraph.from_graph(gl)
        stream = torch.cuda.ExternalStream(d.stream(), device=dev)
        sl_b = torch.from_numpy(pkg.graphs.sources_with_edges(gl, N_BFS, 21 + 1000 * rank)).to(dev)
        sl_s = torch.from_numpy(pkg.graphs.sources_with_edges(gl, N_SSSP, 22 + 1000 * rank)).to(dev)
        lv_l = torch.empty((N_BFS, gl.V), dtype=torch.int32, device=dev)
        ds_l = torch.empty((N_SSSP, gl.V), dtype=torch.int64, device=dev)
        res = compare_schedules(pkg, d, stream, sl_b, sl_s, lv_l, ds_l, native.WEIGHT_STORED, DELTA, 1,
                                mean_weight=float(np.mean(gl.w)))
        res["build_wcc_scc_bct_ms"] = ev_time(stream, lambda: d.build(native.LAYER_ALL))
        res["graph"] = f"lattice 4900 x 4900, 5% removed, 0.1% Pareto(1.5) long-range, V={gl.V}, E={gl.E}"
        sch["lattice"] = res
        del lv_l, ds_l
    if not args.no_schedule:
        extra["schedule"] = sch

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count()))
        e, t, kind, nb, ns = cpu_reference_sample(pkg, g, 256, 256, 7, budget_s=12.0)
        cpu = {"value": e / t / 1e9, "unit": "GTEPS", "cores": int(os.environ.get("OMP_NUM_THREADS", os.cpu_count())),
               "kind": kind, "sample": f"{nb} bfs + {ns} sssp(delta={DELTA}) sources of the same graph, alternating "
                                       f"until 12 s of query time (sources with out-edges): {t:.1f} s on the host cores"}
    line = {"metric": METRIC, "value": value, "unit": "GTEPS", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int32 levels, uint64 distance sums", "data": "synthetic",
            "config": config(args.workload, g), "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e,
            "clocks": clk, "gpu_launches": int(launches), **extra}
    if rank == 0:
        print(json.dumps(line), flush=True)
    d.close()
    if pg is not None:
        pg.barrier()
        pg.destroy_process_group()


def main():
    args = parse()
    if args.only:
        run_only(args)
    elif args.stream:
        run_stream(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
