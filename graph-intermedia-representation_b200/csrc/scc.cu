// Strongly connected components and the condensation DAG (buildSCC_DAG, gir.cpp:798-839).
//
// The reference runs one sequential iterative Tarjan over all vertices (gir.cpp:494-537) and
// counts cross-SCC edges into per-SCC hash maps (gir.cpp:825-831). The partition is unique,
// so any exact algorithm gives the same SCCs; here it is the data-parallel decomposition
// (as in iSpan / Multistep, gir_constructor/includes/scc_cpu):
//  1. trim-1 as a worklist: a vertex without an in- or out-neighbour among the unassigned
//     vertices (self-loops ignored) is a singleton SCC; removing it lowers its neighbours'
//     counts, which may trim them in turn; then trim-2: two vertices that are each other's only
//     unassigned in- (or out-) neighbour form an SCC of two;
//  2. forward-backward from a pivot of maximal out-degree x in-degree (the giant SCC of a
//     power-law graph): SCC(pivot) = forward reach ∩ backward reach over unassigned vertices;
//     (a reach that is still growing after deep_levels(V) levels gives way to the reciprocal classes
//     of a mostly undirected graph and the SCCs of their small quotient, where it has them);
//  3. colour propagation for the rest, repeated until every vertex is assigned: every
//     unassigned vertex starts with its own id as colour, colours spread along forward edges
//     by max until stable, so colour(v) = largest id that reaches v; a vertex r with
//     colour(r) = r is a root, and SCC(r) = the vertices of colour r that reach r (a backward
//     search restricted to colour r);
//  4. labels are made canonical (smallest member id) and the condensation edges are the
//     distinct (scc(u), scc(v)) keys of all cross edges: radix sort + unique;
//  5. topological ranks: Kahn levels over the condensation DAG, rank = position in
//     (level, label) order, so rank(a) < rank(b) for every DAG edge a -> b (the invariant of
//     scc_rank, gir.h:54-57).
#include "common.cuh"
#include "frontier.cuh"
#include "unionfind.cuh"

namespace gir {

namespace {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

enum { C_Q = 0, C_ACT = 1, C_ROOTS = 2, C_PIV = 3, C_ACT_E = 4, C_N = 8 };

// Active in/out degree counts (self-loops excluded) and the first trim frontier.
__global__ void k_trim_init(int64_t V, CSRView fw, CSRView bw, int32_t* label, int32_t* indeg, int32_t* outdeg,
                            Queue q, unsigned long long* cnt) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    auto deg = [&](int32_t v) { return (int64_t)fw.deg[v] + bw.deg[v]; };
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        bool trim = false;
        if (v < V) {
            int32_t o = fw.deg[v], in = bw.deg[v];
            // self-loop: rows are sorted, binary search for v
            const int64_t fb = fw.beg[v];
            const int64_t p = lower_bound_dev(fw.adj, fb, fb + o, (int32_t)v);
            if (p < fb + o && fw.adj[p] == (int32_t)v) { --o; --in; }
            outdeg[v] = o;
            indeg[v] = in;
            trim = (o == 0 || in == 0);
            label[v] = trim ? (int32_t)v : -1;
        }
        queue_push(trim, (int32_t)v, s_st[threadIdx.x >> 5], n_st, q, deg, cnt);
    }
    queue_flush(s_st[threadIdx.x >> 5], n_st, q, deg, cnt);
}

// One trim round over the removed vertices of the last round (frontier.cuh): lower the counts of their
// neighbours; a neighbour whose count reaches 0 is removed (claimed once by CAS). A removed vertex's row
// here is its forward row with its backward row behind it; pay holds the vertex, its forward length from
// bit 32 on, and bit 63 for an entry of the backward row.
struct Trim {
    CSRView fw, bw;
    int32_t *label, *indeg, *outdeg;
    __device__ __forceinline__ int64_t deg(int32_t v) const { return (int64_t)fw.deg[v] + bw.deg[v]; }
    __device__ __forceinline__ void row(int32_t v, int64_t& beg, unsigned long long& pay) const {
        beg = 0;
        pay = ((unsigned long long)(uint32_t)fw.deg[v] << 32) | (uint32_t)v;
    }
    __device__ __forceinline__ int32_t adj(int64_t i, unsigned long long& pay) const {
        const int32_t v = (int32_t)(uint32_t)pay;
        const int64_t n = (int64_t)(pay >> 32);
        if (i < n) return fw.adj[fw.beg[v] + i];
        pay |= 1ull << 63;
        return bw.adj[bw.beg[v] + i - n];
    }
    __device__ __forceinline__ unsigned long long want(int32_t w, unsigned long long pay) const {
        return w != (int32_t)(uint32_t)pay;
    }
    __device__ __forceinline__ bool apply(int32_t w, unsigned long long pay, unsigned long long, int32_t& e) {
        e = w;
        if (atomicSub((pay >> 63 ? outdeg : indeg) + w, 1) != 1) return false;
        return atomicCAS(&label[w], -1, w) == -1;
    }
};

// Trim-2 (iSpan's trim_2_from_fq, gir_constructor/includes/scc_cpu/trim_2_3.h:161, as an
// algorithm source): u and v form an SCC of two when each is the other's only unassigned in-
// neighbour (or, in the second pass, only unassigned out-neighbour): no other unassigned vertex
// reaches either, and the two edges close the cycle. Two launches per direction, so labels are
// never read while they change: k_trim2_pair records each vertex's only unassigned neighbour in
// rows `c` when its count (`deg_act`, exact or an over-count of the unassigned neighbours) is 1,
// then k_trim2_apply labels the mutual pairs with the smaller id.
__global__ void k_trim2_pair(int64_t V, CSRView c, const int32_t* label, const int32_t* deg_act, int32_t* partner) {
    GRID_STRIDE(u, V) {
        int32_t p = -1;
        if (label[u] == -1 && deg_act[u] == 1) {
            const int64_t b = c.beg[u], e = b + c.deg[u];
            for (int64_t k = b; k < e; ++k) {
                const int32_t w = c.adj[k];
                if (w != (int32_t)u && label[w] == -1) {
                    p = w;
                    break;
                }
            }
        }
        partner[u] = p;
    }
}

__global__ void k_trim2_apply(int64_t V, const int32_t* partner, int32_t* label, unsigned long long* n_pairs) {
    unsigned long long c = 0;
    GRID_STRIDE(u, V) {
        const int32_t p = partner[u];
        if (p >= 0 && partner[p] == (int32_t)u) {
            label[u] = p < (int32_t)u ? p : (int32_t)u;
            c += p > (int32_t)u;
        }
    }
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane_id() == 0 && c) atomicAdd(n_pairs, c);
}

// Pivot: the unassigned vertex with the largest score (ties: larger id). Rules: 0 out x in
// degree (iSpan's pivot_selection_from_fq, gir_constructor/includes/scc_cpu/scc_common.h:98-146,
// the fixed schedule), 1 out + in, 2 in-degree. Also counts the unassigned vertices (C_ACT) and
// their edges (C_ROOTS + 1: out-degrees summed), the schedule's features.
__global__ void k_pivot(int64_t V, const int32_t* label, const int32_t* indeg, const int32_t* outdeg, int rule,
                        unsigned long long* cnt) {
    unsigned long long best = 0;
    unsigned long long act = 0, act_e = 0;
    GRID_STRIDE(v, V) {
        if (label[v] != -1) continue;
        ++act;
        act_e += (uint32_t)outdeg[v];
        const unsigned long long o = (uint32_t)outdeg[v], i = (uint32_t)indeg[v];
        const unsigned long long s = rule == 1 ? o + i : (rule == 2 ? i : o * i);
        const unsigned long long k = ((s < (1ull << 31) ? s : (1ull << 31)) << 32) | (unsigned long long)v;
        if (k + 1 > best) best = k + 1;
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
        best = t > best ? t : best;
        act += __shfl_xor_sync(0xffffffffu, act, o);
        act_e += __shfl_xor_sync(0xffffffffu, act_e, o);
    }
    if (lane_id() == 0) {
        if (best) atomicMax(&cnt[C_PIV], best);
        if (act) atomicAdd(&cnt[C_ACT], act);
        if (act_e) atomicAdd(&cnt[C_ACT_E], act_e);
    }
}

// Reach from the pivot, both directions in one level-synchronous traversal (frontier.cuh): a queue
// entry e >= 0 is vertex e searched forward (out-rows), e < 0 is vertex ~e searched backward
// (in-rows). An unassigned w joins a direction once (mark bit 1 forward, 2 backward; an assigned
// vertex starts with both, so one load tells both apart); afterwards the unassigned vertices with
// both bits are SCC(pivot). Paths inside the pivot's SCC never pass through trimmed (already labelled)
// vertices, so restricting both searches to unassigned vertices keeps FW and BW exact.
// Bound by the latency of the marks' random accesses; a level was a degree pass, a scan and a launch
// whose warps took 512 edges each, so on a lattice four warps worked: 46 us a level, now about 8.
struct ReachBoth {
    CSRView fw, bw;
    int32_t* mark;
    __device__ __forceinline__ int32_t deg(int32_t e) const { return e >= 0 ? fw.deg[e] : bw.deg[~e]; }
    __device__ __forceinline__ void row(int32_t e, int64_t& beg, unsigned long long& back) const {
        back = e < 0;
        beg = back ? bw.beg[~e] : fw.beg[e];
    }
    __device__ __forceinline__ int32_t adj(int64_t i, unsigned long long back) const {
        return back ? bw.adj[i] : fw.adj[i];
    }
    __device__ __forceinline__ unsigned long long want(int32_t w, unsigned long long back) const {
        const int bit = back ? 2 : 1;
        return __ldcg(mark + w) & bit ? 0ull : bit;
    }
    __device__ __forceinline__ bool apply(int32_t w, unsigned long long back, unsigned long long bit, int32_t& e) {
        touch_l1((back ? bw.deg : fw.deg) + w);  // (read at the level's end)
        e = back ? ~w : w;
        return (atomicOr(&mark[w], (int)bit) & (int)bit) == 0;
    }
};

// The same level bottom-up, on rows that start on 16-byte boundaries (the handle's graph): a vertex
// without the forward mark looks for an in-neighbour in the forward frontier, one without the backward
// mark for an out-neighbour in the backward frontier.
__global__ void __launch_bounds__(kBlock) k_reach_up(int64_t V, CSRView fw, CSRView bw, const uint32_t* fwd,
                                                     const uint32_t* bwd, int32_t* mark, Queue out,
                                                     unsigned long long* cnt, LongRows rest) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    auto deg = [&](int32_t e) { return e >= 0 ? fw.deg[e] : bw.deg[~e]; };
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        const int32_t m = v < V ? mark[v] : 3;
        const bool wf = !(m & 1), wb = !(m & 2);
        const bool f = first_hit(bw.adj, wf ? bw.beg[v] : 0, wf ? bw.deg[v] : 0, wf, 0,
                                 [&](int32_t w, int32_t) { return (fwd[w >> 5] >> (w & 31)) & 1u; }) >= 0;
        const bool b = first_hit(fw.adj, wb ? fw.beg[v] : 0, wb ? fw.deg[v] : 0, wb, 0,
                                 [&](int32_t w, int32_t) { return (bwd[w >> 5] >> (w & 31)) & 1u; }) >= 0;
        if (f || b) mark[v] = m | (f ? 1 : 0) | (b ? 2 : 0);
        if (wf && !f && bw.deg[v] > kLongRow) rest.add((int32_t)v);
        if (wb && !b && fw.deg[v] > kLongRow) rest.add(~(int32_t)v);
        queue_push(f, (int32_t)v, s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
        queue_push(b, ~(int32_t)v, s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
    }
    queue_flush(s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
}

__global__ void __launch_bounds__(kBlock) k_reach_up_long(CSRView fw, CSRView bw, const uint32_t* fwd, const uint32_t* bwd,
                                                          int32_t* mark, Queue out, unsigned long long* cnt, LongRows rest) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    auto deg = [&](int32_t e) { return e >= 0 ? fw.deg[e] : bw.deg[~e]; };
    walk_long_rows(rest.item, (int64_t)*rest.n, kLongRow, [&](int32_t e) { return e >= 0 ? bw.deg[e] : fw.deg[~e]; },
                   [&](int32_t e, int32_t k, bool on) {
                       const int32_t v = e >= 0 ? e : ~e, bit = e >= 0 ? 1 : 2;
                       bool hit = false;
                       if (on && !(__ldcg(mark + v) & bit)) {
                           const int32_t w = e >= 0 ? bw.adj[bw.beg[v] + k] : fw.adj[fw.beg[v] + k];
                           hit = ((e >= 0 ? fwd : bwd)[w >> 5] >> (w & 31)) & 1u;
                       }
                       const bool join = hit && !(atomicOr(&mark[v], bit) & bit);
                       queue_push(join, e, s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
                   });
    queue_flush(s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
}

// Bottom-up where the frontier's rows hold over four times as many entries as there are (vertex,
// direction) pairs left (4.8M-vertex R-MAT: both levels of over 2^22 entries, 0.62 ms each top-down).
struct ReachUp {
    CSRView fw, bw;
    int32_t* mark;
    uint32_t* bits;  // two bitmaps, the number of long rows, room for those of both CSRs
    int64_t V;
    bool aligned;
    bool wants(int64_t total, int64_t queued) const { return aligned && total > 4 * (2 * V - queued); }
    static int64_t words(int64_t V, int64_t E) { return 2 * (V / 32 + 1) + 1 + 2 * (E / kLongRow + 1); }
    int launch(gir_dev* g, const Queue& in, int64_t nq, const Queue& out, unsigned long long* cnt) const {
        uint32_t* bwd = bits + V / 32 + 1;
        const LongRows rest{reinterpret_cast<int32_t*>(bwd + V / 32 + 2), bwd + V / 32 + 1};
        GIR_CUDA(g, cudaMemsetAsync(bits, 0, sizeof(uint32_t) * (2 * (V / 32 + 1) + 1), g->stream));
        k_frontier_bits<<<grid_for(g, nq, kBlock), kBlock, 0, g->stream>>>(in.v, nq, bits, bwd);
        GIR_LAUNCH(g, "k_frontier_bits");
        k_reach_up<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, fw, bw, bits, bwd, mark, out, cnt, rest);
        GIR_LAUNCH(g, "k_reach_up");
        k_reach_up_long<<<g->num_sms * 4, kBlock, 0, g->stream>>>(fw, bw, bits, bwd, mark, out, cnt, rest);
        GIR_LAUNCH(g, "k_reach_up_long");
        return GIR_OK;
    }
};

// Marks of the assigned vertices, and the pivot in both directions as the first frontier.
__global__ void k_reach_init(int64_t V, const int32_t* label, int32_t pivot, CSRView fw, CSRView bw, int32_t* mark,
                             Queue q, unsigned long long* ctl) {
    GRID_STRIDE(v, V) mark[v] = label[v] != -1 || v == pivot ? 3 : 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        q.v[0] = pivot;
        q.v[1] = ~pivot;
        q.off[0] = 0;
        q.off[1] = (uint64_t)fw.deg[pivot];
        ctl[W_Q] = (2ull << kQShift) | (unsigned long long)((int64_t)fw.deg[pivot] + bw.deg[pivot]);
    }
}

// SCC(pivot): the unassigned vertices reached both ways.
__global__ void k_reach_label(int64_t V, const int32_t* mark, int32_t pivot, int32_t* label) {
    GRID_STRIDE(v, V) if (mark[v] == 3 && label[v] == -1) label[v] = pivot;
}

// Colour propagation: colour(w) = max(colour(w), colour(u)) along forward edges between
// unassigned vertices. `inq` de-duplicates the next queue per round.
__global__ void k_color_init(int64_t V, const int32_t* label, int32_t* color, int32_t* q, unsigned long long* cnt) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        const bool on = v < V && label[v] == -1;
        if (v < V) color[v] = (int32_t)v;
        stage_append(on, (int32_t)v, s_st[threadIdx.x >> 5], n_st, q, &cnt[C_Q]);
    }
    stage_flush(s_st[threadIdx.x >> 5], n_st, q, &cnt[C_Q]);
}

__global__ void __launch_bounds__(kBlock) k_color_prop(const int32_t* q, const unsigned long long* qlen, CSRView fw,
                                                       const int32_t* label, int32_t* color, int32_t* inq,
                                                       int32_t round, int32_t* nq, unsigned long long* cnt) {
    warp_expand(q, (int64_t)*qlen, fw, nq, &cnt[C_Q], [&](int32_t u, int32_t w) {
        if (label[w] != -1) return false;
        const int32_t cu = color[u];
        if (cu <= color[w]) return false;
        if (atomicMax(&color[w], cu) >= cu) return false;
        return atomicExch(&inq[w], round) != round;
    });
}

__global__ void k_color_roots(int64_t V, int32_t* label, const int32_t* color, int32_t* q, unsigned long long* cnt) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        bool root = false;
        if (v < V && label[v] == -1 && color[v] == (int32_t)v) {
            label[v] = (int32_t)v;
            root = true;
        }
        stage_append(root, (int32_t)v, s_st[threadIdx.x >> 5], n_st, q, &cnt[C_Q]);
    }
    stage_flush(s_st[threadIdx.x >> 5], n_st, q, &cnt[C_Q]);
}

// Backward search inside each colour class from its root.
__global__ void __launch_bounds__(kBlock) k_color_bw(const int32_t* q, const unsigned long long* qlen, CSRView bw,
                                                     int32_t* label, const int32_t* color, int32_t* nq,
                                                     unsigned long long* cnt) {
    warp_expand(q, (int64_t)*qlen, bw, nq, &cnt[C_Q], [&](int32_t u, int32_t w) {
        const int32_t c = color[u];
        if (label[w] != -1 || color[w] != c) return false;
        return atomicCAS(&label[w], -1, c) == -1;
    });
}

// Canonical labels: smallest member of every class.
__global__ void k_fill(int32_t* p, int64_t n, int32_t v) { GRID_STRIDE(i, n) p[i] = v; }

// Smallest member of every class. The lanes of a warp that share a label (consecutive vertices
// of the giant SCC mostly do) send one atomicMin, from their smallest vertex, and only when a
// plain read says it can still lower the minimum: otherwise the millions of members of one
// class would serialize on one address.
__global__ void k_class_min(int64_t V, const int32_t* label, int32_t* mn) {
    GRID_STRIDE(v, V) {
        const int32_t l = label[v];
        const unsigned grp = __match_any_sync(__activemask(), l);
        const bool leader = (int)(__ffs(grp) - 1) == lane_id();  // the group's smallest vertex
        if (leader && *(volatile int32_t*)&mn[l] > (int32_t)v) atomicMin(&mn[l], (int32_t)v);
    }
}

__global__ void k_apply_min(int64_t V, int32_t* label, const int32_t* mn, unsigned long long* n_classes) {
    unsigned long long c = 0;
    GRID_STRIDE(v, V) {
        const int32_t m = mn[label[v]];
        label[v] = m;
        c += (m == (int32_t)v);
    }
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane_id() == 0 && c) atomicAdd(n_classes, c);
}

// Rows whose entries hold every cross edge. Where one SCC G holds most edges, its rows are left out: an
// edge with its tail outside G is in that vertex's forward row, and one from G to a vertex outside in
// that vertex's backward row. Without such an SCC (*giant = -1) all forward rows and no backward ones.
__global__ void k_cross_len(int64_t V, const int32_t* deg, const int32_t* label, const int32_t* giant, int back,
                            int32_t* len) {
    const int32_t g = *giant;
    GRID_STRIDE(v, V) len[v] = g >= 0 ? (label[v] != g ? deg[v] : 0) : (back ? 0 : deg[v]);
}

// Cross-SCC edge keys (label(u) << 32 | label(w)), appended to `keys` in any order (they are sorted next)
// through a per-warp buffer; a run of equal keys within a step (a singleton's edges into the giant SCC)
// is appended once. Rows are cut into even runs whatever their length (off: scan of the row lengths); with
// `back` the rows are backward ones and only edges from G count. 69M edges of the 4.8M-vertex R-MAT: keys
// and flags at every edge's slot and a compaction took 1.1 ms, all rows this way 0.41 ms, without
// the giant SCC's rows 0.25 ms.
constexpr int kKeyStage = 128;
__global__ void __launch_bounds__(kBlock) k_cross_keys(int64_t V, const int64_t* off, CSRView c, const int32_t* label,
                                                       const int32_t* giant, int back, uint64_t* keys,
                                                       unsigned long long* n) {
    __shared__ uint64_t s_keys[kWarps][kKeyStage];
    uint64_t* buf = s_keys[threadIdx.x >> 5];
    int held = 0;
    const int ln = lane_id();
    auto flush = [&]() {
        unsigned long long at = 0;
        if (ln == 0) at = atomicAdd(n, (unsigned long long)held);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int i = ln; i < held; i += 32) keys[at + i] = buf[i];
        __syncwarp();
        held = 0;
    };
    const uint32_t from = (uint32_t)*giant;
    auto load = [&](int32_t u, int32_t w) {
        return ((uint64_t)(uint32_t)label[back ? w : u] << 32) | (uint32_t)label[back ? u : w];
    };
    walk_rows_of<4>(off, V, c.beg, c.adj, load, [&](bool on, int32_t, int32_t, int, uint64_t key) {
        const bool cross = on && (key >> 32) != (key & 0xffffffffULL) && (!back || (uint32_t)(key >> 32) == from);
        const uint64_t before = __shfl_up_sync(0xffffffffu, key, 1);
        const bool put = cross && (ln == 0 || before != key);
        const unsigned m = __ballot_sync(0xffffffffu, put);
        if (!m) return;
        if (held + __popc(m) > kKeyStage) flush();
        if (put) buf[held + __popc(m & ((1u << ln) - 1))] = key;
        __syncwarp();
        held += __popc(m);
    });
    if (held) flush();
}

__global__ void k_distinct_u64(const uint64_t* keys, int64_t n, uint8_t* flag) {
    GRID_STRIDE(i, n) flag[i] = (i == 0 || keys[i] != keys[i - 1]);
}

// Longest-path levels over the condensation edges: level(b) >= level(a) + 1 for every edge a -> b, in
// rounds until nothing changes, all of them in one cooperative launch with a grid barrier a round (a
// launch, two copies and a host read a round had been 22 us). Edge-parallel with a plain pre-check, so
// only raises take an atomic (no hot counter: a node with many in-edges, like the giant SCC, is raised a
// few times, not decremented once per edge as in Kahn's algorithm).
// ctl: [0..2] raises of a round (in turn), [3] error, [5] raises of the last round, [6] the largest level
// raised to (a round may carry a level far); the barrier's counter from word 16 on. Without kLoop one round,
// for an ordinary launch: its raises are in [0].
constexpr int kDagWords = 32;
template <bool kLoop>
__global__ void __launch_bounds__(kLoopThreads, 2) k_dag_levels(const uint64_t* keys, int64_t n, int32_t* level,
                                                                unsigned long long* ctl, int max_rounds) {
    unsigned int* bar = reinterpret_cast<unsigned int*>(ctl + 16);
    unsigned long long raised = 0;
    int32_t top = 0;
    int round = 0;
    unsigned met = 0;
    while (round < max_rounds) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl[(round + 1) % 3] = 0;
        unsigned long long c = 0;
        GRID_STRIDE(i, n) {
            const uint64_t k = keys[i];
            const int32_t a = (int32_t)(k >> 32), b = (int32_t)(k & 0xffffffffULL);
            const int32_t cand = __ldcg(level + a) + 1;
            if (cand > __ldcg(level + b) && atomicMax(&level[b], cand) < cand) {
                ++c;
                top = cand > top ? cand : top;
            }
        }
        c = warp_sum_u64(c);
        if (lane_id() == 0 && c) atomicAdd(&ctl[round % 3], c);
        if (!kLoop) break;
        if (!grid_barrier(bar, ctl + 3, met)) return;
        raised = __ldcg(ctl + round % 3);
        ++round;
        if (raised == 0) break;
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane_id() == 0 && top) atomicMax(&ctl[6], (unsigned long long)top);
    if (kLoop && blockIdx.x == 0 && threadIdx.x == 0) ctl[5] = raised;
}

// Keys (level << vb | label) of the SCCs, vb the bits of a vertex id.
__global__ void __launch_bounds__(kBlock) k_rank_keys(int64_t V, const int32_t* label, const int32_t* level, int vb,
                                                      uint64_t* keys, unsigned long long* n) {
    __shared__ int s_w[kWarps];
    __shared__ unsigned long long s_base;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        const bool on = v < V && label[v] == (int32_t)v;
        const unsigned long long at = block_slot(on, n, s_w, &s_base);
        if (on) keys[at] = ((uint64_t)(uint32_t)level[v] << vb) | (uint64_t)v;
    }
}

__global__ void k_rank_scatter(const uint64_t* keys, int64_t n, int vb, int32_t* rank_of) {
    GRID_STRIDE(i, n) rank_of[(int64_t)(keys[i] & ((1ull << vb) - 1))] = (int32_t)i;
}

__global__ void k_rank_gather(int64_t V, const int32_t* label, const int32_t* rank_of, int32_t* rank) {
    GRID_STRIDE(v, V) rank[v] = rank_of[label[v]];
}

// ---- Reciprocal classes ------------------------------------------------------------------------
// The ends of a reciprocal pair of edges (u -> v and v -> u) share an SCC. A vertex whose in- and
// out-rows (without a self-loop) are as long as its symmetrized row has reciprocal edges only, so
// that test per vertex finds them without a search per edge. Joining every such vertex with its
// neighbours by union-find leaves, on a graph that is undirected or nearly so (a road network), a few
// classes and only the edges between the other vertices; the SCCs of that small quotient graph are
// the SCCs of the graph.
__global__ void k_reciprocal(int64_t V, CSRView fw, CSRView bw, CSRView sym, uint8_t* full,
                             unsigned long long* n_full) {
    unsigned long long c = 0;
    GRID_STRIDE(v, V) {
        const int32_t o = fw.deg[v];
        const int64_t fb = fw.beg[v];
        const int64_t p = lower_bound_dev(fw.adj, fb, fb + o, (int32_t)v);
        const int32_t self = p < fb + o && fw.adj[p] == (int32_t)v;
        const bool f = o - self == sym.deg[v] && bw.deg[v] - self == sym.deg[v];
        full[v] = f;
        c += f;
    }
    c = warp_sum_u64(c);
    if (lane_id() == 0 && c) atomicAdd(n_full, c);
}

// Row lengths of the vertices with full[v] == want, 0 for the others.
__global__ void k_mask_deg(int64_t V, const int32_t* deg, const uint8_t* full, int want, int32_t* out) {
    GRID_STRIDE(v, V) out[v] = (full[v] != 0) == (want != 0) ? deg[v] : 0;
}

// (off: scan of the row lengths, so that a hub's row is shared by many warps.)
__global__ void __launch_bounds__(kBlock) k_class_link(int64_t V, const int64_t* off, CSRView sym, int32_t* cls,
                                                       unsigned long long* err) {
    walk_segments(off, V, [&](int64_t u, int64_t j) { uf_union(cls, (int32_t)u, sym.adj[sym.beg[u] + j], err); });
}

// Keys (class(u) << 32 | class(w)) of the edges between classes; counted only while keys is null.
__global__ void __launch_bounds__(kBlock) k_quotient_keys(int64_t V, const int64_t* off, CSRView fw, const int32_t* cls,
                                                          uint64_t* keys, unsigned long long* n) {
    walk_segments(off, V, [&](int64_t u, int64_t j) {
        const int32_t a = cls[u], b = cls[fw.adj[fw.beg[u] + j]];
        if (a == b) return;
        const unsigned m = __activemask();  // (one atomic for the threads that are here together)
        const int leader = __ffs(m) - 1;
        unsigned long long at = 0;
        if (lane_id() == leader) at = atomicAdd(n, (unsigned long long)__popc(m));
        at = __shfl_sync(m, at, leader) + __popc(m & ((1u << lane_id()) - 1));
        if (keys) keys[at] = ((uint64_t)(uint32_t)a << 32) | (uint32_t)b;
    });
}

__global__ void k_flip_keys(const uint64_t* in, int64_t n, uint64_t* out) {
    GRID_STRIDE(i, n) out[i] = (in[i] << 32) | (in[i] >> 32);
}

// Compact CSR of sorted keys.
__global__ void k_keys_csr(const uint64_t* keys, int64_t n, int64_t V, int64_t* beg, int32_t* deg, int32_t* adj) {
    GRID_STRIDE(v, V) {
        const int64_t a = lower_bound_dev(keys, (int64_t)0, n, (uint64_t)v << 32);
        beg[v] = a;
        deg[v] = (int32_t)(lower_bound_dev(keys, a, n, ((uint64_t)v + 1) << 32) - a);
    }
    GRID_STRIDE(i, n) adj[i] = (int32_t)(keys[i] & 0xffffffffULL);
}

__global__ void k_quotient_labels(int64_t V, const int32_t* cls, const int32_t* qlabel, int32_t* label,
                                  unsigned long long* n_classes) {
    unsigned long long c = 0;
    GRID_STRIDE(v, V) {
        const int32_t l = qlabel ? qlabel[cls[v]] : cls[v];
        label[v] = l;
        c += l == (int32_t)v;
    }
    c = warp_sum_u64(c);
    if (lane_id() == 0 && c) atomicAdd(n_classes, c);
}

struct Loop {
    gir_dev* g;
    unsigned long long* cnt;
    unsigned long long* hc;
    int read(int64_t* out) {
        GIR_CUDA(g, cudaMemcpyAsync(hc, cnt, sizeof(unsigned long long) * C_N, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        *out = (int64_t)hc[C_Q];
        return GIR_OK;
    }
};

}  // namespace

static int scc_labels(gir_dev* g, const CSRView fw, const CSRView bw, bool whole, int32_t* label, int64_t* n_scc);

// SCC labels of the handle's graph through its reciprocal classes (above), where at least half of the
// vertices have reciprocal edges only; *used says whether it was done.
static int scc_by_quotient(gir_dev* g, int32_t* label, int64_t* n_scc, bool* used) {
    const int64_t V = g->V;
    *used = false;
    Temps t{g, {}};
    uint8_t* full = nullptr;
    int32_t *cls = nullptr, *mdeg = nullptr;
    int64_t* off = nullptr;
    unsigned long long* cnt = nullptr;  // [0] full vertices, [1] union-find errors, [2] keys, [3] keys, [4] classes
    GIR_TRY(t.get(&full, V));
    GIR_TRY(t.get(&cls, V));
    GIR_TRY(t.get(&mdeg, V));
    GIR_TRY(t.get(&off, V + 1));
    GIR_TRY(t.get(&cnt, 8));
    void* hp = nullptr;
    GIR_TRY(pinned(g, 256, &hp));
    unsigned long long* hc = static_cast<unsigned long long*>(hp);
    auto read = [&]() -> int {
        GIR_CUDA(g, cudaMemcpyAsync(hc, cnt, sizeof(unsigned long long) * 8, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        return GIR_OK;
    };
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * 8, g->stream));
    k_reciprocal<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, view(g->fw), view(g->bw), view(g->sym), full, cnt);
    GIR_LAUNCH(g, "k_reciprocal");
    GIR_TRY(read());
    if ((int64_t)hc[0] * 2 < V) return GIR_OK;
    CSRView sym = view(g->sym), fw = view(g->fw);
    sym.deg = mdeg;
    k_mask_deg<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, g->sym.deg, full, 1, mdeg);
    GIR_LAUNCH(g, "k_mask_deg");
    k_uf_first<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(sym, V, cls);
    GIR_LAUNCH(g, "k_uf_first");
    GIR_TRY(uf_flatten(g, cls, V));
    GIR_TRY(scan_degrees(g, mdeg, V, off));
    k_class_link<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, off, sym, cls, cnt + 1);
    GIR_LAUNCH(g, "k_class_link");
    GIR_TRY(uf_flatten(g, cls, V));
    // (an edge between classes has two ends that are not full)
    fw.deg = mdeg;
    k_mask_deg<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, g->fw.deg, full, 0, mdeg);
    GIR_LAUNCH(g, "k_mask_deg");
    GIR_TRY(scan_degrees(g, mdeg, V, off));
    k_quotient_keys<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, off, fw, cls, nullptr, cnt + 2);
    GIR_LAUNCH(g, "k_quotient_keys");
    GIR_TRY(read());
    if (hc[1]) return fail(g, GIR_ERR_TIMEOUT, "scc: union-find exceeded its retry bound");
    const int64_t n = (int64_t)hc[2];
    int32_t* qlabel = nullptr;
    if (n > 0) {
        uint64_t *keys = nullptr, *flip = nullptr, *tmp = nullptr;
        uint8_t* flag = nullptr;
        GIR_TRY(t.get(&keys, n));
        GIR_TRY(t.get(&flip, n));
        GIR_TRY(t.get(&tmp, n));
        GIR_TRY(t.get(&flag, n));
        k_quotient_keys<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, off, fw, cls, keys, cnt + 3);
        GIR_LAUNCH(g, "k_quotient_keys");
        GIR_TRY(sort_keys_u64(g, keys, tmp, n, edge_key_bits(g->V)));
        k_distinct_u64<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(keys, n, flag);
        GIR_LAUNCH(g, "k_distinct_u64");
        int64_t m = 0;
        GIR_TRY(select_flagged_u64(g, keys, flag, tmp, n, &m));
        k_flip_keys<<<grid_for(g, m, kBlock), kBlock, 0, g->stream>>>(tmp, m, flip);
        GIR_LAUNCH(g, "k_flip_keys");
        GIR_TRY(sort_keys_u64(g, flip, keys, m, edge_key_bits(g->V)));
        int64_t* beg[2];
        int32_t *deg[2], *adj[2];
        for (int i = 0; i < 2; ++i) {
            GIR_TRY(t.get(&beg[i], V));
            GIR_TRY(t.get(&deg[i], V));
            GIR_TRY(t.get(&adj[i], m));
            k_keys_csr<<<grid_for(g, V > m ? V : m, kBlock), kBlock, 0, g->stream>>>(i ? flip : tmp, m, V, beg[i], deg[i],
                                                                                   adj[i]);
            GIR_LAUNCH(g, "k_keys_csr");
        }
        GIR_TRY(t.get(&qlabel, V));
        int64_t n_q = 0;
        GIR_TRY(scc_labels(g, CSRView{beg[0], deg[0], adj[0], nullptr}, CSRView{beg[1], deg[1], adj[1], nullptr}, false,
                           qlabel, &n_q));
    }
    // (class roots and SCC labels are smallest members: the composition is canonical)
    k_quotient_labels<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, cls, qlabel, label, cnt + 4);
    GIR_LAUNCH(g, "k_quotient_labels");
    GIR_TRY(read());
    *n_scc = (int64_t)hc[4];
    *used = true;
    return GIR_OK;
}

// SCC labels of the graph with rows fw / bw; `whole`: it is the handle's graph.
static int scc_labels(gir_dev* g, const CSRView fw, const CSRView bw, bool whole, int32_t* label, int64_t* n_scc) {
    const int64_t V = g->V;
    int32_t *indeg = nullptr, *outdeg = nullptr, *qa = nullptr, *qb = nullptr, *mark = nullptr, *color = nullptr;
    unsigned long long* cnt = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[0], V + 1, &indeg));
    GIR_TRY(ensure_n(g, g->scratch[1], V + 1, &outdeg));
    // (the queues hold up to 2V entries in the two-way reach from the pivot)
    GIR_TRY(ensure_n(g, g->scratch[2], 2 * V + 2, &qa));
    GIR_TRY(ensure_n(g, g->scratch[3], 2 * V + 2, &qb));
    GIR_TRY(ensure_n(g, g->scratch[4], V + 1, &mark));
    GIR_TRY(ensure_n(g, g->scratch[5], V + 1, &color));
    GIR_TRY(ensure_n(g, g->scratch[6], 2 * C_N, &cnt));
    unsigned long long* qlen = cnt + C_N;
    void* hp = nullptr;
    GIR_TRY(pinned(g, 256, &hp));
    Loop lp{g, cnt, static_cast<unsigned long long*>(hp)};
    *n_scc = 0;
    if (V == 0) return GIR_OK;
    const int grid = g->num_sms * (int)g->params[GIR_PARAM_CTAS_PER_SM];
    auto blocks_for_queue = [&](int64_t n) {
        const int64_t b = (n + 32 * kWarps - 1) / (32 * kWarps);
        return (int)(b < 1 ? 1 : (b < grid ? b : grid));
    };
    // One level-synchronous pass: `launch(in, inlen, out)` for each round until the queue empties.
    auto run_queue = [&](int32_t*& in, int32_t*& out, int64_t n, auto&& launch) -> int {
        while (n > 0) {
            GIR_CUDA(g, cudaMemcpyAsync(qlen, &cnt[C_Q], sizeof(unsigned long long), cudaMemcpyDeviceToDevice, g->stream));
            GIR_CUDA(g, cudaMemsetAsync(&cnt[C_Q], 0, sizeof(unsigned long long), g->stream));
            GIR_TRY(launch(in, out, n));
            std::swap(in, out);
            GIR_TRY(lp.read(&n));
        }
        return GIR_OK;
    };

    trace_mark(g, "scc: start");
    // 1. trim-1
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * 2 * C_N, g->stream));
    Queue q{qa, nullptr};
    unsigned long long* ctl = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[7], 2 * V + 2, &q.off));
    GIR_TRY(ensure_n(g, g->scratch[10], kLoopWords, &ctl));
    GIR_CUDA(g, cudaMemsetAsync(ctl, 0, sizeof(unsigned long long) * kLoopWords, g->stream));
    k_trim_init<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, fw, bw, label, indeg, outdeg, q, ctl + W_Q);
    GIR_LAUNCH(g, "k_trim_init");
    int64_t n = 0;
    {
        FrontierRun run;
        GIR_TRY(run_frontier(g, Trim{fw, bw, label, indeg, outdeg}, TopDownOnly{}, q, ctl, run, INT64_MAX));
    }

    // trim-2: SCCs of two vertices, through in-neighbours, then through out-neighbours
    {
        int32_t* partner = color;  // (colours are set up later)
        GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
        for (int dir = 0; dir < 2; ++dir) {
            k_trim2_pair<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, dir ? fw : bw, label, dir ? outdeg : indeg,
                                                                           partner);
            GIR_LAUNCH(g, "k_trim2_pair");
            k_trim2_apply<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, partner, label, &cnt[C_ROOTS]);
            GIR_LAUNCH(g, "k_trim2_apply");
        }
        if (g->trace_marks) {
            GIR_CUDA(g, cudaMemcpyAsync(lp.hc, cnt, sizeof(unsigned long long) * C_N, cudaMemcpyDeviceToHost, g->stream));
            GIR_CUDA(g, cudaStreamSynchronize(g->stream));
            std::fprintf(stderr, "[gir] scc: trim-2 pairs %llu\n", (unsigned long long)lp.hc[C_ROOTS]);
        }
    }

    trace_mark(g, "scc: trim");
    // 2. forward-backward from the max-degree pivot
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
    k_pivot<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, indeg, outdeg, 0, cnt);
    GIR_LAUNCH(g, "k_pivot");
    GIR_CUDA(g, cudaMemcpyAsync(lp.hc, cnt, sizeof(unsigned long long) * C_N, cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    // The pivot rule: forced by GIR_PARAM_PIVOT, else the fixed max out x in degree or the
    // schedule network (rule 3: no forward-backward pass, colour propagation does everything).
    // Any rule gives the same SCCs; only the time differs.
    int rule = (int)g->params[GIR_PARAM_PIVOT];
    {
        float feat[GIR_SCHED_IN];
        sched_scc_features(g, (double)lp.hc[C_ACT], (double)lp.hc[C_ACT_E],
                           lp.hc[C_PIV] ? (double)((lp.hc[C_PIV] - 1) >> 32) : 0.0, feat);
        if (rule < 0) {
            rule = 0;
            if (g->schedule == GIR_SCHEDULE_LEARNED && g->sched_loaded) GIR_TRY(sched_choose_pivot(g, feat, &rule));
        }
        if (whole) {
            g->trace_x.clear();
            g->trace_y.clear();
            sched_trace(g, feat, 8 + rule);
        }
    }
    if (rule == 1 || rule == 2) {
        GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
        k_pivot<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, indeg, outdeg, rule, cnt);
        GIR_LAUNCH(g, "k_pivot");
        GIR_CUDA(g, cudaMemcpyAsync(lp.hc, cnt, sizeof(unsigned long long) * C_N, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    }
    if (rule != 3 && lp.hc[C_PIV] != 0) {
        const int32_t pivot = (int32_t)((lp.hc[C_PIV] - 1) & 0xffffffffULL);
        // both searches start from the pivot (marked both ways)
        GIR_CUDA(g, cudaMemsetAsync(ctl, 0, sizeof(unsigned long long) * kLoopWords, g->stream));
        k_reach_init<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, pivot, fw, bw, mark, q, ctl);
        GIR_LAUNCH(g, "k_reach_init");
        const ReachBoth op{fw, bw, mark};
        uint32_t* bits = nullptr;
        if (whole) GIR_TRY(ensure_n(g, g->scratch[11], ReachUp::words(V, g->fw.E), &bits));
        const ReachUp up{fw, bw, mark, bits, V, whole};
        FrontierRun run;
        GIR_TRY(run_frontier(g, op, up, q, ctl, run, whole ? deep_levels(V) : INT64_MAX));
        if (!run.done()) {
            bool used = false;
            GIR_TRY(scc_by_quotient(g, label, n_scc, &used));
            trace_mark(g, "scc: reciprocal classes");
            if (used) return GIR_OK;
            GIR_TRY(run_frontier(g, op, up, q, ctl, run, INT64_MAX));
        }
        k_reach_label<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, mark, pivot, label);
        GIR_LAUNCH(g, "k_reach_label");
    }

    trace_mark(g, "scc: fw-bw");
    // 3. colour propagation rounds until every vertex is assigned
    int32_t* inq = mark;
    int32_t round = 1;
    GIR_CUDA(g, cudaMemsetAsync(inq, 0, sizeof(int32_t) * V, g->stream));
    for (int outer = 0; outer < (1 << 30); ++outer) {
        GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
        k_color_init<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, color, qa, cnt);
        GIR_LAUNCH(g, "k_color_init");
        GIR_TRY(lp.read(&n));
        if (n == 0) break;
        GIR_TRY(run_queue(qa, qb, n, [&](int32_t* in, int32_t* out, int64_t m) -> int {
            ++round;
            k_color_prop<<<blocks_for_queue(m), kBlock, 0, g->stream>>>(in, qlen, fw, label, color, inq, round, out, cnt);
            GIR_LAUNCH(g, "k_color_prop");
            return GIR_OK;
        }));
        GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
        k_color_roots<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, color, qa, cnt);
        GIR_LAUNCH(g, "k_color_roots");
        GIR_TRY(lp.read(&n));
        GIR_TRY(run_queue(qa, qb, n, [&](int32_t* in, int32_t* out, int64_t m) -> int {
            k_color_bw<<<blocks_for_queue(m), kBlock, 0, g->stream>>>(in, qlen, bw, label, color, out, cnt);
            GIR_LAUNCH(g, "k_color_bw");
            return GIR_OK;
        }));
    }

    if (g->trace_marks) std::fprintf(stderr, "[gir] scc: colour rounds %d\n", (int)round);
    trace_mark(g, "scc: colour");
    // 4. canonical labels
    int32_t* mn = color;
    k_fill<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(mn, V, INT32_MAX);
    GIR_LAUNCH(g, "k_fill");
    k_class_min<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, mn);
    GIR_LAUNCH(g, "k_class_min");
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
    k_apply_min<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, mn, &cnt[C_Q]);
    GIR_LAUNCH(g, "k_apply_min");
    GIR_TRY(lp.read(n_scc));
    return GIR_OK;
}

int scc_build(gir_dev* g) {
    const int64_t V = g->V;
    int32_t* label = nullptr;
    GIR_TRY(ensure_n(g, g->scc, V + 1, &label));
    GIR_TRY(scc_labels(g, view(g->fw), view(g->bw), true, label, &g->n_scc));
    trace_mark(g, "scc: labels");
    return scc_build_dag(g);
}

// One edge u -> v between two SCCs (u's SCC before v's in rank order), inserted or just deleted:
// out[0] = position of its condensation key in the sorted keys (lower bound), out[1] = the key is
// there; out[2] bit 0 = another edge joins the two SCCs from u's forward row or v's backward
// row, bit 1 = u has an out-neighbour in its own SCC, bit 2 = v has an in-neighbour in its own
// SCC (a vertex of a non-trivial SCC always has both, so without them both SCCs are singletons
// and the two rows are every edge between them).
__global__ void k_dag_probe(const uint64_t* dag, int64_t n, uint64_t key, CSRView fw, CSRView bw,
                            const int32_t* label, int32_t u, int32_t v, unsigned long long* out) {
    const int32_t cu = label[u], cv = label[v];
    unsigned long long bits = 0;
    for (int64_t k = fw.beg[u] + threadIdx.x; k < fw.beg[u] + fw.deg[u]; k += blockDim.x) {
        const int32_t y = label[fw.adj[k]];
        if (y == cv) bits |= 1;
        if (y == cu) bits |= 2;
    }
    for (int64_t k = bw.beg[v] + threadIdx.x; k < bw.beg[v] + bw.deg[v]; k += blockDim.x) {
        const int32_t x = label[bw.adj[k]];
        if (x == cu) bits |= 1;
        if (x == cv) bits |= 4;
    }
    if (bits) atomicOr(&out[2], bits);
    if (threadIdx.x == 0) {
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t m = (lo + hi) >> 1;
            if (dag[m] < key) lo = m + 1; else hi = m;
        }
        out[0] = (unsigned long long)lo;
        out[1] = lo < n && dag[lo] == key;
    }
}

__global__ void k_dag_put(uint64_t* dag, int64_t p, uint64_t key) { dag[p] = key; }

int scc_dag_patch_one(gir_dev* g, int32_t u, int32_t v, bool insert, bool* patched) {
    *patched = false;
    const int32_t* label = static_cast<const int32_t*>(g->scc.p);
    const int64_t n = g->n_dag;
    if (n < 0 || !g->dag.p || u < 0 || v < 0 || u >= g->V || v >= g->V) return scc_build_dag(g);
    unsigned long long* cnt = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[6], 2 * C_N, &cnt));
    void* hp = nullptr;
    GIR_TRY(pinned(g, 256, &hp));
    unsigned long long* hc = static_cast<unsigned long long*>(hp);
    int32_t lab[2];
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * 3, g->stream));
    GIR_CUDA(g, cudaMemcpyAsync(&lab[0], label + u, sizeof(int32_t), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaMemcpyAsync(&lab[1], label + v, sizeof(int32_t), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    const uint64_t key = ((uint64_t)(uint32_t)lab[0] << 32) | (uint32_t)lab[1];
    k_dag_probe<<<1, kBlock, 0, g->stream>>>(static_cast<const uint64_t*>(g->dag.p), n, key, view(g->fw), view(g->bw),
                                             label, u, v, cnt);
    GIR_LAUNCH(g, "k_dag_probe");
    GIR_CUDA(g, cudaMemcpyAsync(hc, cnt, sizeof(unsigned long long) * 3, cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    const int64_t p = (int64_t)hc[0];
    const bool present = hc[1] != 0;
    const unsigned long long bits = hc[2];
    uint64_t* dag = static_cast<uint64_t*>(g->dag.p);
    if (insert) {
        if (present) {
            *patched = true;  // the SCCs were joined already
            return GIR_OK;
        }
        if (g->dag.bytes < sizeof(uint64_t) * (size_t)(n + 2)) return scc_build_dag(g);
        uint64_t* tmp = nullptr;
        GIR_TRY(ensure_n(g, g->scratch[8], n - p + 1, &tmp));
        if (n > p) {
            GIR_CUDA(g, cudaMemcpyAsync(tmp, dag + p, sizeof(uint64_t) * (n - p), cudaMemcpyDeviceToDevice, g->stream));
            GIR_CUDA(g, cudaMemcpyAsync(dag + p + 1, tmp, sizeof(uint64_t) * (n - p), cudaMemcpyDeviceToDevice, g->stream));
        }
        k_dag_put<<<1, 1, 0, g->stream>>>(dag, p, key);
        GIR_LAUNCH(g, "k_dag_put");
        g->n_dag = n + 1;
    } else {
        if (!present || (bits & 1)) {
            *patched = true;  // another edge still joins the two SCCs (or none was recorded)
            return GIR_OK;
        }
        if (bits & 6) return scc_build_dag(g);  // a non-trivial SCC: its other members' rows count too
        if (n - p - 1 > 0) {
            uint64_t* tmp = nullptr;
            GIR_TRY(ensure_n(g, g->scratch[8], n - p, &tmp));
            GIR_CUDA(g, cudaMemcpyAsync(tmp, dag + p + 1, sizeof(uint64_t) * (n - p - 1), cudaMemcpyDeviceToDevice,
                                        g->stream));
            GIR_CUDA(g, cudaMemcpyAsync(dag + p, tmp, sizeof(uint64_t) * (n - p - 1), cudaMemcpyDeviceToDevice,
                                        g->stream));
        }
        g->n_dag = n - 1;
    }
    // the ranks stay a topological order (the edge respects them); reachability changed
    g->dag_rows_valid = false;
    g->reach_hub_valid = false;
    *patched = true;
    return GIR_OK;
}

int scc_build_dag(gir_dev* g) {
    const int64_t V = g->V;
    int32_t* label = static_cast<int32_t*>(g->scc.p);
    // condensation edges: cross keys, radix sort, unique
    const int64_t E = g->fw.E;
    uint64_t *keys = nullptr, *tmp = nullptr;
    uint8_t* flag = nullptr;
    int64_t* off = nullptr;
    unsigned long long* cnt = nullptr;
    // (the rank keys share keys / tmp: up to one per vertex)
    const int64_t room = E > V ? E : V;
    GIR_TRY(ensure_n(g, g->scratch[7], room + 1, &keys));
    GIR_TRY(ensure_n(g, g->scratch[8], room + 1, &tmp));
    GIR_TRY(ensure_n(g, g->scratch[9], room + 1, &flag));
    GIR_TRY(ensure_n(g, g->scratch[10], V + 1, &off));
    GIR_TRY(ensure_n(g, g->scratch[6], 2 * C_N, &cnt));
    void* hp = nullptr;
    GIR_TRY(pinned(g, 256, &hp));
    unsigned long long* hc = static_cast<unsigned long long*>(hp);
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
    if (E > 0) {
        int32_t *len = nullptr, *giant = reinterpret_cast<int32_t*>(cnt + C_N);
        GIR_TRY(ensure_n(g, g->scratch[11], V + 1, &len));
        GIR_TRY(sample_mode(g, g->fw, label, kModeSamples / 2, giant));
        for (int back = 0; back < 2; ++back) {
            const DevCSR& c = back ? g->bw : g->fw;
            k_cross_len<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, c.deg, label, giant, back, len);
            GIR_LAUNCH(g, "k_cross_len");
            GIR_TRY(scan_degrees(g, len, V, off));
            k_cross_keys<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, off, view(c), label, giant, back, keys, &cnt[C_Q]);
            GIR_LAUNCH(g, "k_cross_keys");
        }
    }
    GIR_CUDA(g, cudaMemcpyAsync(hc, cnt, sizeof(unsigned long long), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    const int64_t n_cross = (int64_t)hc[C_Q];
    GIR_TRY(sort_keys_u64(g, keys, tmp, n_cross, edge_key_bits(g->V)));
    int64_t n_dag = 0;
    uint64_t* dag = nullptr;
    GIR_TRY(ensure_n(g, g->dag, n_cross + 1, &dag));
    if (n_cross > 0) {
        k_distinct_u64<<<grid_for(g, n_cross, kBlock), kBlock, 0, g->stream>>>(keys, n_cross, flag);
        GIR_LAUNCH(g, "k_distinct_u64");
        GIR_TRY(select_flagged_u64(g, keys, flag, dag, n_cross, &n_dag));
    }
    g->n_dag = n_dag;
    g->dag_rows_valid = false;
    g->reach_hub_valid = false;
    trace_mark(g, "scc: dag edges");

    // topological ranks: longest-path levels over the condensation edges, rounds until stable
    // (at most the DAG's depth + 1 rounds)
    int32_t *level = nullptr, *rank_of = nullptr, *rank = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[1], V + 1, &level));
    GIR_TRY(ensure_n(g, g->scratch[5], V + 1, &rank_of));
    GIR_TRY(ensure_n(g, g->scc_rank, V + 1, &rank));
    GIR_CUDA(g, cudaMemsetAsync(level, 0, sizeof(int32_t) * V, g->stream));
    int64_t top = 0;  // the largest level
    if (n_dag > 0) {
        unsigned long long* ctl = nullptr;
        GIR_TRY(ensure_n(g, g->scratch[10], kDagWords, &ctl));
        int per_sm = 0;
        GIR_TRY(cooperative_ctas(g, (const void*)k_dag_levels<true>, kLoopThreads, &per_sm));
        while (true) {
            GIR_CUDA(g, cudaMemsetAsync(ctl, 0, sizeof(unsigned long long) * kDagWords, g->stream));
            int max_rounds = 1 << 22;  // (the barrier's counter is 32 bits wide)
            const uint64_t* dag_c = dag;
            int64_t n_c = n_dag;
            void* args[] = {&dag_c, &n_c, &level, &ctl, &max_rounds};
            if (per_sm > 0) {
                GIR_CUDA(g, cudaLaunchCooperativeKernel((const void*)k_dag_levels<true>, g->num_sms * (per_sm > 1 ? 2 : 1),
                                                        kLoopThreads, args, 0, g->stream));
            } else {
                k_dag_levels<false><<<grid_for(g, n_dag, kLoopThreads), kLoopThreads, 0, g->stream>>>(dag_c, n_c, level, ctl, 1);
                GIR_LAUNCH(g, "k_dag_levels");
            }
            GIR_CUDA(g, cudaMemcpyAsync(hc, ctl, sizeof(unsigned long long) * 7, cudaMemcpyDeviceToHost, g->stream));
            GIR_CUDA(g, cudaStreamSynchronize(g->stream));
            if (hc[3]) return fail(g, GIR_ERR_TIMEOUT, "scc: a grid barrier of the DAG levels ran out its bound");
            top = (int64_t)hc[6] > top ? (int64_t)hc[6] : top;
            if (hc[per_sm > 0 ? 5 : 0] == 0) break;
        }
    }
    trace_mark(g, "scc: levels");
    // rank = position in (level, label) order (no more key bits than the largest of either)
    const int vb = edge_key_bits(V) - 32;
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
    if (V > 0) {
        k_rank_keys<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, level, vb, keys, &cnt[C_Q]);
        GIR_LAUNCH(g, "k_rank_keys");
    }
    const int64_t ns = g->n_scc;
    GIR_TRY(sort_keys_u64(g, keys, tmp, ns, vb + edge_key_bits(top) - 32));
    if (ns > 0) {
        k_rank_scatter<<<grid_for(g, ns, kBlock), kBlock, 0, g->stream>>>(keys, ns, vb, rank_of);
        GIR_LAUNCH(g, "k_rank_scatter");
        k_rank_gather<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, label, rank_of, rank);
        GIR_LAUNCH(g, "k_rank_gather");
    }
    trace_mark(g, "scc: ranks");
    g->scc_built = true;
    return GIR_OK;
}

}  // namespace gir
