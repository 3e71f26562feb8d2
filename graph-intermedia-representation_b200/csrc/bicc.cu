// Per-SCC biconnected blocks and the block-cut forest (buildBCT, gir.cpp:2063-2089).
//
// The layer is defined on H, the undirected graph of the symmetrized edges whose endpoints lie
// in the same SCC (gir.h:45-46): its connected components are the SCCs, and its biconnected
// components are the blocks the reference computes SCC by SCC (sequential Hopcroft-Tarjan for
// small SCCs, gir.cpp:541-587; Tarjan-Vishkin over a BFS tree for large ones, gir.cpp:1804-2022).
// An SCC of one vertex is a singleton block (gir.cpp:584). Here Tarjan-Vishkin runs on every
// SCC at once:
//  1. BFS spanning forest of H from every SCC's smallest vertex (level-synchronous), or on a deep H a
//     forest from union-find, rooted by Euler tours, with 2. and 3. to match (see "Deep graphs");
//  2. subtree sizes nd (levels bottom-up, which also gives every vertex its offset among its siblings)
//     and preorder numbers pre (levels top-down);
//  3. low / high: min / max pre over each subtree and its non-tree neighbours;
//  4. union-find over tree edges (edge (p(v), v) is named by v): rule 1 joins the edges of
//     v and w for a non-tree edge {v, w} between unrelated vertices; rule 2 joins (p(v), v)
//     with (p(p(v)), p(v)) when v's subtree reaches outside p(v)'s subtree;
//  5. every class is a block: its vertices are the child ends of its tree edges plus the
//     parent of the topmost one (the block's head). Output in the reference's representation
//     (gir.h:58-64): every vertex has one parent block (label_block), every block one head
//     articulation point (-1 for the block a tree root belongs to first), bcnt = number of
//     blocks containing the vertex (AP iff >= 2).
#include "common.cuh"
#include "frontier.cuh"
#include "unionfind.cuh"

namespace gir {

namespace {

constexpr int kBlock = 256;

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

enum { C_Q = 0, C_ERR = 1, C_N = 4 };

// H row filter: neighbour w of u is in H iff same SCC (sym rows never contain u itself).
struct HView {
    CSRView sym;
    const int32_t* scc;
};

// SCCs with more than one vertex: every non-smallest member marks its SCC's smallest vertex
// (plain stores behind a read, so a giant SCC costs a few writes, not one per member).
__global__ void k_mark_nontrivial(int64_t V, const int32_t* scc, uint8_t* nontrivial) {
    GRID_STRIDE(v, V) {
        const int32_t r = scc[v];
        if (r != (int32_t)v && !nontrivial[r]) nontrivial[r] = 1;
    }
}

// Row lengths of H for the sweeps: 0 for the vertices of singleton SCCs (isolated in H).
__global__ void k_h_deg(int64_t V, const int32_t* scc, const uint8_t* nontrivial, const int32_t* sym_deg,
                        int32_t* hdeg) {
    GRID_STRIDE(v, V) hdeg[v] = nontrivial[scc[v]] ? sym_deg[v] : 0;
}

// Forest roots: every SCC's smallest vertex; only those of non-singleton SCCs start the BFS.
__global__ void k_roots(int64_t V, const int32_t* scc, const uint8_t* nontrivial, const int32_t* hdeg, int32_t* parent,
                        Queue q, unsigned long long* cnt) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    auto deg = [&](int32_t x) { return hdeg[x]; };
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        bool root = false;
        if (v < V) {
            const bool r = scc[v] == (int32_t)v;
            root = r && nontrivial[v];
            parent[v] = r ? (int32_t)v : -1;
        }
        queue_push(root, (int32_t)v, s_st[threadIdx.x >> 5], n_st, q, deg, cnt);
    }
    queue_flush(s_st[threadIdx.x >> 5], n_st, q, deg, cnt);
}

// One BFS level of the spanning forest over H (frontier.cuh): the atomicCAS on parent[w] gives w its
// parent and queues it. The levels end up back to back in the queue array.
// Bound by the latency of the parents' and SCC labels' random accesses. A level was a degree pass, a
// scan and a launch whose warps took 512 row entries each: 42 us a level of an 803 x 803 lattice.
struct ForestLevel {
    CSRView sym;  // (row lengths: H's)
    const int32_t* scc;
    int32_t* parent;
    __device__ __forceinline__ int32_t deg(int32_t u) const { return sym.deg[u]; }
    __device__ __forceinline__ void row(int32_t u, int64_t& beg, unsigned long long& who) const {
        beg = sym.beg[u];
        who = ((unsigned long long)(uint32_t)scc[u] << 32) | (uint32_t)u;
    }
    __device__ __forceinline__ int32_t adj(int64_t i, unsigned long long) const { return sym.adj[i]; }
    __device__ __forceinline__ unsigned long long want(int32_t w, unsigned long long who) const {
        return __ldcg(parent + w) == -1 && scc[w] == (int32_t)(who >> 32);
    }
    __device__ __forceinline__ bool apply(int32_t w, unsigned long long who, unsigned long long, int32_t& e) {
        touch_l1(sym.deg + w);  // (read at the level's end)
        e = w;
        return atomicCAS(&parent[w], -1, (int32_t)(uint32_t)who) == -1;
    }
};

// The same level bottom-up: every vertex without a parent takes the first entry of its row that is in
// the frontier (bits) and in its SCC.
__global__ void __launch_bounds__(kBlock) k_forest_up(int64_t V, CSRView sym, const int32_t* scc, const uint32_t* bits,
                                                      int32_t* parent, Queue out, unsigned long long* cnt, LongRows rest) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    auto deg = [&](int32_t x) { return sym.deg[x]; };
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < V; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = base + threadIdx.x;
        const bool want = v < V && parent[v] == -1;
        const int32_t mine = want ? scc[v] : -1;
        const int32_t p = first_hit(sym.adj, want ? sym.beg[v] : 0, want ? sym.deg[v] : 0, want, mine,
                                    [&](int32_t w, int32_t c) { return ((bits[w >> 5] >> (w & 31)) & 1u) && scc[w] == c; });
        if (p >= 0) parent[v] = p;
        if (want && p < 0 && sym.deg[v] > kLongRow) rest.add((int32_t)v);
        queue_push(p >= 0, (int32_t)v, s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
    }
    queue_flush(s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
}

__global__ void __launch_bounds__(kBlock) k_forest_up_long(CSRView sym, const int32_t* scc, const uint32_t* bits,
                                                           int32_t* parent, Queue out, unsigned long long* cnt,
                                                           LongRows rest) {
    __shared__ int32_t s_st[kBlock / 32][kStage];
    int n_st = 0;
    auto deg = [&](int32_t x) { return sym.deg[x]; };
    walk_long_rows(rest.item, (int64_t)*rest.n, kLongRow, deg, [&](int32_t v, int32_t k, bool on) {
        bool join = false;
        if (on && __ldcg(parent + v) == -1) {
            const int32_t w = sym.adj[sym.beg[v] + k];
            if (((bits[w >> 5] >> (w & 31)) & 1u) && scc[w] == scc[v]) join = atomicCAS(&parent[v], -1, w) == -1;
        }
        queue_push(join, v, s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
    });
    queue_flush(s_st[threadIdx.x >> 5], n_st, out, deg, cnt);
}

// Bottom-up where the frontier's rows hold over four times as many entries as there are vertices left
// (a vertex left reads a few entries to its first hit; 4.8M-vertex R-MAT: both levels of over 2^22
// entries, 0.6 ms each top-down).
struct ForestUp {
    CSRView sym;
    const int32_t* scc;
    int32_t* parent;
    uint32_t* bits;  // the bitmap, the number of long rows, room for them
    int64_t V;
    bool wants(int64_t total, int64_t queued) const { return total > 4 * (V - queued); }
    int launch(gir_dev* g, const Queue& in, int64_t nq, const Queue& out, unsigned long long* cnt) const {
        const LongRows rest{reinterpret_cast<int32_t*>(bits + V / 32 + 2), bits + V / 32 + 1};
        GIR_CUDA(g, cudaMemsetAsync(bits, 0, sizeof(uint32_t) * (V / 32 + 2), g->stream));
        k_frontier_bits<<<grid_for(g, nq, kBlock), kBlock, 0, g->stream>>>(in.v, nq, bits, bits);
        GIR_LAUNCH(g, "k_frontier_bits");
        k_forest_up<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, sym, scc, bits, parent, out, cnt, rest);
        GIR_LAUNCH(g, "k_forest_up");
        k_forest_up_long<<<g->num_sms * 4, kBlock, 0, g->stream>>>(sym, scc, bits, parent, out, cnt, rest);
        GIR_LAUNCH(g, "k_forest_up_long");
        return GIR_OK;
    }
};

// ---- Deep graphs: a spanning forest without levels ---------------------------------------------
// Tarjan-Vishkin takes any rooted spanning forest. Where the BFS forest is still growing after
// deep_levels(V) levels (a road network has thousands), the forest comes from union-find over H
// instead: every hook of one root under another is a tree edge. Each tree is rooted at its SCC's
// smallest vertex by its Euler tour: the two arcs of every tree edge, sorted, give each vertex its
// arcs; the arc after x -> y is the one after y -> x in y's list, cyclically, and the tour starts at
// the root's first arc. Pointer doubling over the arcs gives each its distance to the tour's end; the
// arc of a tree edge that comes first points down, the arcs between the two are twice the subtree,
// and the number of down arcs so far is the preorder. A subtree is then an interval of preorder
// positions, and low / high over it the minimum / maximum of an interval (doubling windows).
// 803 x 803 lattice, blocks only: about 1,300 levels of four launches each (94 ms) against some
// sixty launches in all (about 1.5 ms). The arcs' indices are 32 bits wide: below 2^30 vertices.
constexpr int64_t kEulerMaxV = 1ll << 30;

// Tree edges: the slot of the hooked root holds (u << 32 | w); ~0 elsewhere. (off: scan of H's row lengths.)
__global__ void __launch_bounds__(kBlock) k_tree_link(int64_t V, const int64_t* off, CSRView h, const int32_t* scc,
                                                      int32_t* uf, uint64_t* edge, unsigned long long* err) {
    walk_segments(off, V, [&](int64_t v, int64_t j) {
        const int32_t u = (int32_t)v, w = h.adj[h.beg[v] + j];
        if (u > w || scc[u] != scc[w]) return;  // (every pair is in both rows)
        const int32_t hooked = uf_union(uf, u, w, err);
        if (hooked >= 0) edge[hooked] = ((uint64_t)(uint32_t)u << 32) | (uint32_t)w;
    });
}

__global__ void k_tree_flags(int64_t V, const uint64_t* edge, uint8_t* flag) {
    GRID_STRIDE(v, V) flag[v] = edge[v] != ~0ull;
}

__global__ void k_tree_arcs(const uint64_t* edge, int64_t n, uint64_t* arcs) {
    GRID_STRIDE(i, n) {
        arcs[2 * i] = edge[i];
        arcs[2 * i + 1] = (edge[i] << 32) | (edge[i] >> 32);
    }
}

// Twins and successors of the sorted arcs: twin[i], and jump[i] = (next arc, 1); the arc that would
// enter its root's first arc again ends the tour: (n, 0) with slot n a fixed point.
__global__ void k_euler_next(const uint64_t* arcs, int64_t n, const int32_t* scc, int32_t* twin, int2* jump) {
    GRID_STRIDE(i, n) {
        const uint64_t a = arcs[i];
        const int32_t y = (int32_t)(a & 0xffffffffULL);
        const int64_t t = lower_bound_dev(arcs, (int64_t)0, n, (a << 32) | (a >> 32));
        twin[i] = (int32_t)t;
        int64_t nx = t + 1;
        bool end = false;
        if (nx == n || (int32_t)(arcs[nx] >> 32) != y) {  // the twin is y's last arc: on to its first
            nx = lower_bound_dev(arcs, (int64_t)0, n, (uint64_t)(uint32_t)y << 32);
            end = scc[y] == y;
        }
        jump[i] = end ? make_int2((int32_t)n, 0) : make_int2((int32_t)nx, 1);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) jump[n] = make_int2((int32_t)n, 0);
}

__global__ void k_euler_double(const int2* in, int64_t n, int2* out) {
    GRID_STRIDE(i, n + 1) {
        const int2 a = in[i], b = in[a.x];
        out[i] = make_int2(b.x, a.y + b.y);
    }
}

// Arcs of every tree's tour, at its root (0 elsewhere): its first arc is the root's first.
__global__ void k_tour_size(const uint64_t* arcs, int64_t n, const int32_t* scc, const int2* rank, int64_t* size) {
    GRID_STRIDE(i, n) {
        const int32_t x = (int32_t)(arcs[i] >> 32);
        if (scc[x] == x && (i == 0 || (int32_t)(arcs[i - 1] >> 32) != x)) size[x] = (int64_t)rank[i].y + 1;
    }
}

// Tour positions (trees back to back): the down arcs' flags, and every child's parent and subtree.
__global__ void k_tour_down(const uint64_t* arcs, int64_t n, const int32_t* scc, const int32_t* twin, const int2* rank,
                            const int64_t* tour, int64_t* down, int32_t* parent, int32_t* nd) {
    GRID_STRIDE(i, n) {
        const int32_t x = (int32_t)(arcs[i] >> 32), y = (int32_t)(arcs[i] & 0xffffffffULL);
        const int32_t r = scc[x];
        const int32_t d = rank[i].y, dt = rank[twin[i]].y;
        down[tour[r + 1] - 1 - d] = d > dt;
        if (d > dt) {
            parent[y] = x;
            nd[y] = (d - dt + 1) / 2;
        }
    }
}

// Preorder numbers (within the tree; roots have 0), all non-root vertices in preorder, and the roots'
// subtree sizes. downs: exclusive scan of the down flags.
__global__ void k_tour_pre(const uint64_t* arcs, int64_t n, const int32_t* scc, const int32_t* twin, const int2* rank,
                           const int64_t* tour, const int64_t* downs, int32_t* pre, int32_t* at, int32_t* nd) {
    GRID_STRIDE(i, n) {
        const int32_t x = (int32_t)(arcs[i] >> 32), y = (int32_t)(arcs[i] & 0xffffffffULL);
        const int32_t r = scc[x];
        const int32_t d = rank[i].y, dt = rank[twin[i]].y;
        if (d <= dt) continue;
        const int64_t k = downs[tour[r + 1] - 1 - d];
        pre[y] = (int32_t)(k - downs[tour[r]]) + 1;
        at[k] = y;
        if (x == r) nd[r] = (int32_t)((tour[r + 1] - tour[r]) / 2) + 1;
    }
}

// Doubling windows over the preorder positions: win[k] = (min low, max high) of [k, k + len). A vertex
// whose subtree is at least len and below 2 len long takes its interval from two of them.
__global__ void k_win_first(const int32_t* at, int64_t n, const int32_t* low, const int32_t* high, int2* win) {
    GRID_STRIDE(k, n) win[k] = make_int2(low[at[k]], high[at[k]]);
}
__global__ void k_win_step(const int32_t* at, int64_t n, int64_t len, const int32_t* nd, const int2* win, int2* next,
                           int32_t* low, int32_t* high) {
    GRID_STRIDE(k, n) {
        const int2 a = win[k];
        const int32_t v = at[k];
        const int64_t s = nd[v];
        if (s >= len && s < 2 * len) {
            const int2 b = win[k + s - len];
            low[v] = a.x < b.x ? a.x : b.x;
            high[v] = a.y > b.y ? a.y : b.y;
        }
        const int2 b = k + len < n ? win[k + len] : a;
        next[k] = make_int2(a.x < b.x ? a.x : b.x, a.y > b.y ? a.y : b.y);
    }
}

// The smallest H neighbour of every tree root: it decides which of its blocks is the root's parent block. In a
// BFS forest a root's neighbours are its children (no rows to read); consecutive children send one atomicMin.
__global__ void k_root_child_least(int64_t V, const int32_t* parent, int32_t* least) {
    GRID_STRIDE(v, V) {
        const int32_t p = parent[v];
        const bool child = p != (int32_t)v && parent[p] == p;
        const unsigned grp = __match_any_sync(__activemask(), child ? p : -1);
        if (child && __ffs(grp) - 1 == lane_id() && *(volatile int32_t*)&least[p] > (int32_t)v)
            atomicMin(&least[p], (int32_t)v);
    }
}
// In the forest of a deep graph they need not be: the roots' rows.
__global__ void k_root_rows(int64_t V, const int32_t* scc, const int32_t* hdeg, int32_t* deg) {
    GRID_STRIDE(v, V) deg[v] = scc[v] == (int32_t)v ? hdeg[v] : 0;
}
// Rows are cut into even runs whatever their length (off: scan of the row lengths): a root may be the hub that
// holds every row entry, and one warp for its whole row took 6.1 of 6.7 ms of the blocks of a star of 300,000
// vertices. Rows are sorted, so a row's first hit among the warp's lanes is its least there.
__global__ void __launch_bounds__(kBlock) k_root_least(int64_t V, const int64_t* off, CSRView h, const int32_t* scc,
                                                       int32_t* least) {
    const unsigned below = (1u << lane_id()) - 1;
    walk_rows_of<4>(off, V, h.beg, h.adj, [&](int32_t, int32_t w) { return scc[w]; },
                    [&](bool on, int32_t u, int32_t w, int x, int32_t c) {
                        const bool hit = on && c == u;
                        const unsigned before = __ballot_sync(0xffffffffu, hit) & below;
                        const int px = __shfl_sync(0xffffffffu, x, before ? 31 - __clz(before) : 0);
                        if (hit && (before == 0 || px != x) && w < least[u]) atomicMin(&least[u], w);
                    });
}
__global__ void k_root_block_least(int64_t V, const int32_t* least, const int32_t* uf, const int32_t* id_of_rep,
                                   int32_t* label) {
    GRID_STRIDE(v, V) if (least[v] != INT32_MAX) label[v] = id_of_rep[uf[least[v]]];
}

__global__ void k_fill_i32(int32_t* p, int64_t n, int32_t v) { GRID_STRIDE(i, n) p[i] = v; }

// nd[parent] += nd[v] for the vertices of one level (deepest level first). What the sum held before, less
// the parent itself, is the subtrees of the siblings that came earlier: the vertex's offset among them in
// a preorder (any order of siblings makes one). Grouping the children by a sort and scanning their sizes
// took another 0.3 ms of 4.5 ms on the 4.8M-vertex R-MAT, and fifteen launches on a small graph.
__global__ void k_nd_level(const int32_t* q, int64_t n, const int32_t* parent, int32_t* nd, int32_t* off) {
    GRID_STRIDE(i, n) {
        const int32_t v = q[i];
        off[v] = atomicAdd(&nd[parent[v]], nd[v]) - 1;
    }
}

__global__ void k_pre_level(const int32_t* q, int64_t n, const int32_t* parent, const int32_t* off, int32_t* pre) {
    GRID_STRIDE(i, n) {
        const int32_t v = q[i];
        pre[v] = pre[parent[v]] + 1 + off[v];
    }
}

__global__ void k_pre_roots(const int32_t* q, int64_t n, int32_t* pre) { GRID_STRIDE(i, n) pre[q[i]] = 0; }

// Per-vertex tree data packed for the sweeps over H: one 8-byte gather per neighbour. x = pre, y = scc.
__global__ void k_pack_keys(int64_t V, const int32_t* pre, const int32_t* scc, int2* key) {
    GRID_STRIDE(v, V) key[v] = make_int2(pre[v], scc[v]);
}

// Before the full sweep, a sample: every vertex of H takes the first kSample entries of its row for rule 1
// and for its low and high. After the unions, and rule 2 with low and high of the sample carried up the
// levels (both are facts, if not all of them), nearly every tree edge of a power-law graph is in its final
// class: a pair already joined costs the sweep one test, and most rows nothing at all (k_sweep_len).
// Unions are idempotent, so the sample changes no class.
constexpr int kSample = 4;

// The first pass takes low and high and, without atomics, puts every tree edge under the first of the
// smaller ones it is joined to; after a flatten the second joins loosely (uf_hook: the sweep below does not
// depend on it).
__global__ void k_nontree_first(int64_t V, HView h, const int2* key, const int32_t* nd, int32_t* low, int32_t* high,
                                int32_t* uf) {
    GRID_STRIDE(u, V) {
        const int32_t d = h.sym.deg[u];
        const int2 ku = key[u];
        const int64_t b = h.sym.beg[u];
        int32_t lo = ku.x, hi = ku.x, under = (int32_t)u;
        for (int j = 0; j < kSample && j < d; ++j) {
            const int32_t w = h.sym.adj[b + j];
            const int2 kw = key[w];
            if (ku.y != kw.y) continue;  // other SCC
            lo = kw.x < lo ? kw.x : lo;
            hi = kw.x > hi ? kw.x : hi;
            if (under == (int32_t)u && w < under && (kw.x > ku.x ? kw.x >= ku.x + nd[u] : ku.x >= kw.x + nd[w])) under = w;
        }
        low[u] = lo;
        high[u] = hi;
        uf[u] = under;
    }
}

__global__ void k_nontree_sample(int64_t V, HView h, const int2* key, const int32_t* nd, int32_t* uf) {
    GRID_STRIDE(u, V) {
        const int32_t d = h.sym.deg[u];
        const int64_t b = h.sym.beg[u];
        const int32_t ru = uf[u];
        for (int j = 0; j < kSample && j < d; ++j) {
            const int32_t w = h.sym.adj[b + j], rw = uf[w];
            if (ru == rw) continue;
            const int2 ku = key[u], kw = key[w];
            if (ku.y != kw.y) continue;
            const bool apart = kw.x > ku.x ? kw.x >= ku.x + nd[u] : ku.x >= kw.x + nd[w];
            if (apart) uf_hook(uf, ru, rw);
        }
    }
}

// Which rows the sweep below can leave out. After the sample nearly all tree edges are in one class G. Rule 2
// has nothing left to say about a vertex whose tree edge is in its parent's class already ("decided", and
// a root's child always), and low / high of a vertex matter only to itself and its ancestors: they are
// needed under undecided vertices only. A row of class G whose vertex and ancestors are all decided is
// left out: an edge from it to another vertex of G joins nothing, one to a vertex outside G is in that
// vertex's row, which is swept and takes rule 1 in both directions.
__global__ void k_need_level(const int32_t* q, int64_t n, const int32_t* parent, const int32_t* uf, uint8_t* need) {
    GRID_STRIDE(i, n) {
        const int32_t v = q[i], p = parent[v];
        need[v] = need[p] || (parent[p] != p && uf[v] != uf[p]);
    }
}
__global__ void k_sweep_len(int64_t V, const int32_t* hdeg, const int32_t* uf, const uint8_t* need, const int32_t* giant,
                            int32_t* len) {
    const int32_t g = *giant;
    GRID_STRIDE(v, V) len[v] = uf[v] == g && !need[v] ? 0 : hdeg[v];
}

// One sweep over the entries of H: low / high of every vertex from its neighbours, and rule 1 for edges
// between unrelated endpoints. Tree edges need no test: a parent's pre never lies below the parent's own
// subtree nor a child's beyond it, so neither changes what rule 2 reads off low and high, and an edge
// between related ends is no rule-1 edge. Per entry one 8-byte gather, (pre, scc) of the neighbour; the
// row's own values are the same for neighbouring lanes. A warp's lanes of one row reduce their minimum
// and maximum by shuffles, so a row costs an atomic per 32 entries at most. Rows are cut into even runs
// whatever their length. Bound by the L2's random gathers: 138M entries of the 4.8M-vertex R-MAT took
// 2.1 ms (a warp per 32 rows, 16-byte gathers), 1.46 ms so, 0.11 ms with the rows above left out.
__global__ void __launch_bounds__(kBlock) k_nontree(int64_t V, const int64_t* off, HView h, const int2* key,
                                                    const int32_t* nd, int32_t* low, int32_t* high, int32_t* uf,
                                                    unsigned long long* err) {
    const int ln = lane_id();
    struct Got {
        int2 kw, ku;
        int32_t end;
    };
    walk_rows_of<4>(
        off, V, h.sym.beg, h.sym.adj,
        [&](int32_t u, int32_t w) {
            Got g;
            g.kw = key[w];
            g.ku = key[u];
            g.end = g.ku.x + nd[u];
            return g;
        },
        [&](bool on, int32_t u, int32_t w, int x, const Got& g) {
            int32_t lo = INT32_MAX, hi = -1;
            if (on && g.kw.y == g.ku.y) {
                lo = hi = g.kw.x;
                const int32_t ru = uf[u], rw = uf[w];
                if (ru != rw && (g.kw.x > g.ku.x ? g.kw.x >= g.end : g.ku.x >= g.kw.x + nd[w])) uf_union(uf, u, w, err);
            }
            __syncwarp();
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {  // the row's first lane ends up with its minimum and maximum
                const int ox = __shfl_down_sync(0xffffffffu, x, o);
                const int32_t ol = __shfl_down_sync(0xffffffffu, lo, o), oh = __shfl_down_sync(0xffffffffu, hi, o);
                if (ln + o < 32 && ox == x) {
                    lo = ol < lo ? ol : lo;
                    hi = oh > hi ? oh : hi;
                }
            }
            const int before = __shfl_up_sync(0xffffffffu, x, 1);
            if (on && (ln == 0 || before != x)) {
                if (lo < low[u]) atomicMin(&low[u], lo);
                if (hi > high[u]) atomicMax(&high[u], hi);
            }
        });
}

// low / high of one level's vertices into their parents (need: only of the vertices that need them).
__global__ void k_lowhigh_level(const int32_t* q, int64_t n, const int32_t* parent, const uint8_t* need, int32_t* low,
                                int32_t* high) {
    GRID_STRIDE(i, n) {
        const int32_t v = q[i];
        if (need && !need[v]) continue;
        const int32_t p = parent[v], lo = low[v], hi = high[v];
        if (lo < low[p]) atomicMin(&low[p], lo);  // (plain pre-checks: a hub has a million children)
        if (hi > high[p]) atomicMax(&high[p], hi);
    }
}

// rule 2 for every non-root v whose parent u is not a root.
__global__ void k_rule2(int64_t V, const int32_t* parent, const int32_t* pre, const int32_t* nd, const int32_t* low,
                        const int32_t* high, int32_t* uf, unsigned long long* err) {
    GRID_STRIDE(v, V) {
        const int32_t u = parent[v];
        if (u < 0 || u == (int32_t)v) continue;  // unreached (cannot happen) or root
        if (parent[u] == u) continue;            // u is a root
        if (low[v] < pre[u] || high[v] >= pre[u] + nd[u]) uf_union(uf, (int32_t)v, u, err);
    }
}

__global__ void k_uf_init(int32_t* uf, int64_t V) { GRID_STRIDE(v, V) uf[v] = (int32_t)v; }

// Block representatives: non-root vertices that are their class root, and isolated tree roots.
// (Read-only root walk: path-halving writes of other threads could otherwise replace a root
// just stored in uf[v] by an intermediate ancestor; here the only writes are final roots.)
__global__ void k_block_flags(int64_t V, const int32_t* parent, const int32_t* nd, int32_t* uf, uint8_t* flag) {
    GRID_STRIDE(v, V) {
        const int32_t p = parent[v];
        const bool root = p == (int32_t)v;
        int32_t r = (int32_t)v;
        while (uf[r] != r) r = uf[r];
        uf[v] = r;
        flag[v] = root ? (nd[v] == 1) : (r == (int32_t)v);
    }
}

__global__ void k_block_ids(const int32_t* reps, int64_t nb, int32_t* id_of_rep) {
    GRID_STRIDE(b, nb) id_of_rep[reps[b]] = (int32_t)b;
}

// label_block and heads. Pass 1 (k_root_block_least): the block of every tree root's smallest H neighbour
// becomes the root's parent block (head -1); its other blocks hang from it.
// Pass 2: parent blocks of the other vertices, and heads: a block's head is the parent p of its
// topmost child ends (p is a tree root, or p's own parent edge is in another block); the root's
// parent block has head -1.
__global__ void k_block_assign(int64_t V, const int32_t* parent, const int32_t* nd, const int32_t* uf,
                               const int32_t* id_of_rep, int32_t* label, int32_t* head) {
    GRID_STRIDE(v, V) {
        const int32_t p = parent[v];
        if (p == (int32_t)v) {
            if (nd[v] == 1) {  // isolated: singleton block
                const int32_t b = id_of_rep[v];
                label[v] = b;
                head[b] = -1;
            }
            continue;
        }
        const int32_t b = id_of_rep[uf[v]];
        label[v] = b;
        const bool p_root = parent[p] == p;
        if (p_root || uf[p] != uf[v]) head[b] = (p_root && label[p] == b) ? -1 : p;
    }
}

__global__ void k_bcnt(int64_t V, const int32_t* head, int64_t nb, int32_t* bcnt) {
    GRID_STRIDE(v, V) bcnt[v] = 1;
}

__global__ void k_bcnt_heads(const int32_t* head, int64_t nb, int32_t* bcnt) {
    GRID_STRIDE(b, nb) {
        const int32_t h = head[b];
        if (h >= 0) atomicAdd(&bcnt[h], 1);
    }
}

}  // namespace

// The rooted spanning forest of a deep H by union-find and Euler tours: parent, nd and pre of every
// vertex of a non-singleton SCC (the callers' values stay elsewhere: parent = itself, nd = 1), and its
// n_tree non-root vertices in preorder, tree after tree.
static int euler_forest(gir_dev* g, const CSRView& h, const int32_t* scc, int32_t* parent, int32_t* nd, int32_t* pre,
                        int32_t* at, int64_t* n_tree, unsigned long long* err) {
    const int64_t V = g->V;
    Temps t{g, {}};
    uint64_t *edge = nullptr, *picked = nullptr;
    int32_t* uf = nullptr;
    uint8_t* flag = nullptr;
    int64_t *tour = nullptr, *down = nullptr;
    GIR_TRY(t.get(&tour, V + 1));
    GIR_TRY(t.get(&edge, V));
    GIR_TRY(t.get(&picked, V));
    GIR_TRY(t.get(&uf, V));
    GIR_TRY(t.get(&flag, V));
    GIR_CUDA(g, cudaMemsetAsync(edge, 0xff, sizeof(uint64_t) * V, g->stream));
    GIR_CUDA(g, cudaMemsetAsync(pre, 0, sizeof(int32_t) * V, g->stream));
    k_uf_init<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(uf, V);
    GIR_LAUNCH(g, "k_uf_init");
    int64_t* off = tour;  // (the tours' offsets come later)
    GIR_TRY(scan_degrees(g, h.deg, V, off));
    k_tree_link<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, off, h, scc, uf, edge, err);
    GIR_LAUNCH(g, "k_tree_link");
    k_tree_flags<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, edge, flag);
    GIR_LAUNCH(g, "k_tree_flags");
    int64_t m = 0;
    GIR_TRY(select_flagged_u64(g, edge, flag, picked, V, &m));
    *n_tree = m;
    const int64_t n = 2 * m;  // arcs
    uint64_t *arcs = nullptr, *atmp = nullptr;
    int32_t* twin = nullptr;
    int2 *ja = nullptr, *jb = nullptr;
    GIR_TRY(t.get(&arcs, n + 1));
    GIR_TRY(t.get(&atmp, n + 1));
    GIR_TRY(t.get(&twin, n + 1));
    GIR_TRY(t.get(&ja, n + 1));
    GIR_TRY(t.get(&jb, n + 1));
    GIR_TRY(t.get(&down, n + 1));
    if (m == 0) return GIR_OK;
    const int gn = grid_for(g, n + 1, kBlock);
    k_tree_arcs<<<gn, kBlock, 0, g->stream>>>(picked, m, arcs);
    GIR_LAUNCH(g, "k_tree_arcs");
    GIR_TRY(sort_keys_u64(g, arcs, atmp, n, edge_key_bits(g->V)));
    k_euler_next<<<gn, kBlock, 0, g->stream>>>(arcs, n, scc, twin, ja);
    GIR_LAUNCH(g, "k_euler_next");
    for (int64_t reach = 1; reach < n; reach *= 2) {
        k_euler_double<<<gn, kBlock, 0, g->stream>>>(ja, n, jb);
        GIR_LAUNCH(g, "k_euler_double");
        std::swap(ja, jb);
    }
    GIR_CUDA(g, cudaMemsetAsync(tour, 0, sizeof(int64_t) * (V + 1), g->stream));
    k_tour_size<<<gn, kBlock, 0, g->stream>>>(arcs, n, scc, ja, tour);
    GIR_LAUNCH(g, "k_tour_size");
    GIR_TRY(exclusive_scan_i64(g, tour, tour, V + 1));
    GIR_CUDA(g, cudaMemsetAsync(down + n, 0, sizeof(int64_t), g->stream));
    k_tour_down<<<gn, kBlock, 0, g->stream>>>(arcs, n, scc, twin, ja, tour, down, parent, nd);
    GIR_LAUNCH(g, "k_tour_down");
    GIR_TRY(exclusive_scan_i64(g, down, down, n + 1));
    k_tour_pre<<<gn, kBlock, 0, g->stream>>>(arcs, n, scc, twin, ja, tour, down, pre, at, nd);
    GIR_LAUNCH(g, "k_tour_pre");
    return GIR_OK;
}

// low / high of every non-root vertex over its subtree (at: the n non-root vertices in preorder).
static int subtree_windows(gir_dev* g, const int32_t* at, int64_t n, const int32_t* nd, int32_t* low, int32_t* high) {
    if (n == 0) return GIR_OK;
    Temps t{g, {}};
    int2 *wa = nullptr, *wb = nullptr;
    GIR_TRY(t.get(&wa, n));
    GIR_TRY(t.get(&wb, n));
    const int gn = grid_for(g, n, kBlock);
    k_win_first<<<gn, kBlock, 0, g->stream>>>(at, n, low, high, wa);
    GIR_LAUNCH(g, "k_win_first");
    for (int64_t len = 1; len <= n; len *= 2) {
        k_win_step<<<gn, kBlock, 0, g->stream>>>(at, n, len, nd, wa, wb, low, high);
        GIR_LAUNCH(g, "k_win_step");
        std::swap(wa, wb);
    }
    return GIR_OK;
}

int bct_build(gir_dev* g) {
    if (!g->scc_built) return fail(g, GIR_ERR_STATE, "buildBCT needs buildSCC_DAG first");
    const int64_t V = g->V;
    const int32_t* scc = static_cast<const int32_t*>(g->scc.p);
    HView h{view(g->sym), scc};  // (row lengths replaced by the H lengths below)
    int32_t *parent = nullptr, *order = nullptr, *nd = nullptr, *pre = nullptr, *off = nullptr;
    int32_t *low = nullptr, *high = nullptr, *uf = nullptr, *reps = nullptr, *id_of_rep = nullptr;
    uint8_t* flag = nullptr;
    int64_t* scan = nullptr;
    unsigned long long* cnt = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[0], V + 1, &parent));
    GIR_TRY(ensure_n(g, g->scratch[2], V + 1, &order));
    GIR_TRY(ensure_n(g, g->scratch[3], V + 1, &nd));
    GIR_TRY(ensure_n(g, g->scratch[4], V + 1, &pre));
    GIR_TRY(ensure_n(g, g->scratch[5], V + 1, &off));
    GIR_TRY(ensure_n(g, g->scratch[6], V + 1, &low));
    GIR_TRY(ensure_n(g, g->scratch[7], V + 1, &high));
    GIR_TRY(ensure_n(g, g->scratch[8], V + 1, &uf));
    GIR_TRY(ensure_n(g, g->scratch[11], V + 1, &flag));
    GIR_TRY(ensure_n(g, g->scratch[12], V + 2, &scan));
    GIR_TRY(ensure_n(g, g->scratch[14], 2 * C_N, &cnt));
    void* hp = nullptr;
    GIR_TRY(pinned(g, 256, &hp));
    unsigned long long* hc = static_cast<unsigned long long*>(hp);
    int32_t *label = nullptr, *head = nullptr, *bcnt = nullptr;
    GIR_TRY(ensure_n(g, g->blk_label, V + 1, &label));
    GIR_TRY(ensure_n(g, g->bcnt, V + 1, &bcnt));
    if (V == 0) {
        g->n_blocks = 0;
        g->bct_built = true;
        return GIR_OK;
    }
    auto read = [&]() -> int {
        GIR_CUDA(g, cudaMemcpyAsync(hc, cnt, sizeof(unsigned long long) * C_N, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        return GIR_OK;
    };
    trace_mark(g, "bct: start");
    // 1. BFS forest; order[] holds the levels back to back, lvl_off their boundaries
    GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * 2 * C_N, g->stream));
    uint8_t* nontrivial = nullptr;
    int32_t* hdeg = nullptr;
    GIR_TRY(ensure_n(g, g->work[6], V + 1, &nontrivial));
    GIR_TRY(ensure_n(g, g->work[7], V + 1, &hdeg));
    GIR_CUDA(g, cudaMemsetAsync(nontrivial, 0, V, g->stream));
    k_mark_nontrivial<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, scc, nontrivial);
    GIR_LAUNCH(g, "k_mark_nontrivial");
    k_h_deg<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, scc, nontrivial, g->sym.deg, hdeg);
    GIR_LAUNCH(g, "k_h_deg");
    h.sym.deg = hdeg;
    Queue fq{order, nullptr};
    unsigned long long* ctl = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[1], V + 1, &fq.off));
    GIR_TRY(ensure_n(g, g->scratch[15], kLoopWords, &ctl));
    GIR_CUDA(g, cudaMemsetAsync(ctl, 0, sizeof(unsigned long long) * kLoopWords, g->stream));
    k_roots<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, scc, nontrivial, hdeg, parent, fq, ctl + W_Q);
    GIR_LAUNCH(g, "k_roots");
    uint32_t* bits = nullptr;
    GIR_TRY(ensure_n(g, g->work[5], V / 32 + 3 + g->sym.E / kLongRow, &bits));
    FrontierRun run;
    GIR_TRY(run_frontier(g, ForestLevel{h.sym, scc, parent}, ForestUp{h.sym, scc, parent, bits, V}, fq, ctl, run, V < kEulerMaxV ? deep_levels(V) : INT64_MAX));
    const bool deep = !run.done();
    trace_mark(g, deep ? "bct: forest levels (given up)" : "bct: forest");
    std::vector<int64_t> lvl_off{0};
    for (int64_t n : run.levels) lvl_off.push_back(lvl_off.back() + n);
    const int D = deep ? 0 : (int)lvl_off.size() - 1;  // levels 0..D-1 (the last one may be empty)
    int64_t n_tree = 0;
    // 2. subtree sizes
    k_fill_i32<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(nd, V, 1);
    GIR_LAUNCH(g, "k_fill_i32");
    if (deep) {
        GIR_TRY(euler_forest(g, h.sym, scc, parent, nd, pre, order, &n_tree, &cnt[C_ERR]));
    } else {
        //    levels bottom-up
        for (int L = D - 1; L >= 1; --L) {
            const int64_t n = lvl_off[L + 1] - lvl_off[L];
            if (n == 0) continue;
            k_nd_level<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(order + lvl_off[L], n, parent, nd, off);
            GIR_LAUNCH(g, "k_nd_level");
        }
        //    preorder: levels top-down
        k_pre_roots<<<grid_for(g, lvl_off[1], kBlock), kBlock, 0, g->stream>>>(order, lvl_off[1], pre);
        GIR_LAUNCH(g, "k_pre_roots");
        for (int L = 1; L < D; ++L) {
            const int64_t n = lvl_off[L + 1] - lvl_off[L];
            if (n == 0) continue;
            k_pre_level<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(order + lvl_off[L], n, parent, off, pre);
            GIR_LAUNCH(g, "k_pre_level");
        }
    }
    trace_mark(g, "bct: subtree sizes + preorder");
    // 3. low / high and rule 1
    int2* key = nullptr;
    GIR_TRY(ensure_n(g, g->work[5], V + 1, &key));
    k_pack_keys<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, pre, scc, key);
    GIR_LAUNCH(g, "k_pack_keys");
    k_nontree_first<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, h, key, nd, low, high, uf);
    GIR_LAUNCH(g, "k_nontree_first");
    GIR_TRY(uf_flatten(g, uf, V));
    for (int r = 0; r < 2; ++r) {
        k_nontree_sample<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, h, key, nd, uf);
        GIR_LAUNCH(g, "k_nontree_sample");
        GIR_TRY(uf_flatten(g, uf, V));
    }
    auto carry_up = [&](const uint8_t* only) -> int {
        for (int L = D - 1; L >= 1; --L) {
            const int64_t n = lvl_off[L + 1] - lvl_off[L];
            if (n == 0) continue;
            k_lowhigh_level<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(order + lvl_off[L], n, parent, only, low,
                                                                             high);
            GIR_LAUNCH(g, "k_lowhigh_level");
        }
        return GIR_OK;
    };
    int32_t* len = hdeg;
    uint8_t* need = nullptr;
    if (!deep) {
        GIR_TRY(carry_up(nullptr));
        k_rule2<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, parent, pre, nd, low, high, uf, &cnt[C_ERR]);
        GIR_LAUNCH(g, "k_rule2");
    }
    GIR_TRY(uf_flatten(g, uf, V));
    if (!deep) {
        int32_t* giant = reinterpret_cast<int32_t*>(cnt + C_N);
        need = flag;
        len = off;  // (sibling offsets are no longer needed)
        GIR_CUDA(g, cudaMemsetAsync(need, 0, V, g->stream));
        for (int L = 1; L < D; ++L) {
            const int64_t n = lvl_off[L + 1] - lvl_off[L];
            if (n == 0) continue;
            k_need_level<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(order + lvl_off[L], n, parent, uf, need);
            GIR_LAUNCH(g, "k_need_level");
        }
        GIR_TRY(sample_mode(g, g->sym, uf, kModeSamples / 2, giant));
        k_sweep_len<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, hdeg, uf, need, giant, len);
        GIR_LAUNCH(g, "k_sweep_len");
    }
    GIR_TRY(scan_degrees(g, len, V, scan));
    k_nontree<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, scan, h, key, nd, low, high, uf, &cnt[C_ERR]);
    GIR_LAUNCH(g, "k_nontree");
    if (deep) GIR_TRY(subtree_windows(g, order, n_tree, nd, low, high));
    else GIR_TRY(carry_up(need));
    trace_mark(g, "bct: low/high + rule 1");
    // 4. rule 2
    k_rule2<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, parent, pre, nd, low, high, uf, &cnt[C_ERR]);
    GIR_LAUNCH(g, "k_rule2");
    trace_mark(g, "bct: rule 2");
    // 5. blocks
    k_block_flags<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, parent, nd, uf, flag);
    GIR_LAUNCH(g, "k_block_flags");
    reps = off;  // (sibling offsets are no longer needed)
    int64_t nb = 0;
    GIR_TRY(select_flagged_iota(g, flag, reps, V, &nb));
    id_of_rep = low;
    k_block_ids<<<grid_for(g, nb, kBlock), kBlock, 0, g->stream>>>(reps, nb, id_of_rep);
    GIR_LAUNCH(g, "k_block_ids");
    GIR_TRY(ensure_n(g, g->blk_head, nb + 1, &head));
    int32_t *rdeg = pre, *least = high;  // (neither is read any more)
    k_fill_i32<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(least, V, INT32_MAX);
    GIR_LAUNCH(g, "k_fill_i32");
    if (deep) {
        k_root_rows<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, scc, hdeg, rdeg);
        GIR_LAUNCH(g, "k_root_rows");
        GIR_TRY(scan_degrees(g, rdeg, V, scan));
        k_root_least<<<g->num_sms * 8, kBlock, 0, g->stream>>>(V, scan, h.sym, scc, least);
        GIR_LAUNCH(g, "k_root_least");
    } else {
        k_root_child_least<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, parent, least);
        GIR_LAUNCH(g, "k_root_child_least");
    }
    k_root_block_least<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, least, uf, id_of_rep, label);
    GIR_LAUNCH(g, "k_root_block_least");
    k_block_assign<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, parent, nd, uf, id_of_rep, label, head);
    GIR_LAUNCH(g, "k_block_assign");
    k_bcnt<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, head, nb, bcnt);
    GIR_LAUNCH(g, "k_bcnt");
    k_bcnt_heads<<<grid_for(g, nb, kBlock), kBlock, 0, g->stream>>>(head, nb, bcnt);
    GIR_LAUNCH(g, "k_bcnt_heads");
    GIR_TRY(read());
    if (hc[C_ERR]) return fail(g, GIR_ERR_TIMEOUT, "bct: union-find exceeded its retry bound");
    g->n_blocks = nb;
    g->bct_built = true;
    trace_mark(g, "bct: blocks");
    return GIR_OK;
}

}  // namespace gir
