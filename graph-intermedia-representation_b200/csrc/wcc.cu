// Weakly connected components (buildWCC, gir_constructor/gir.cpp:593-655).
//
// The reference runs a sequential union-find over the forward edges (gir.cpp:635-653). Here
// edges are linked concurrently into a lock-free union-find forest: link(u, w) finds both roots
// (with path halving) and hooks the larger root under the smaller one by compare-and-swap,
// retrying when another thread moved the root first. A root is therefore always the smallest
// vertex of its tree, and after a final pointer-jumping pass every vertex points at the smallest
// vertex id of its component -- the canonical label. The build samples the giant component first
// and links only the rows outside it (wcc_labels_sym, over the symmetric view).
#include <algorithm>

#include "common.cuh"
#include "unionfind.cuh"

namespace gir {

namespace {

constexpr int kBlock = 256;

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// Links the endpoints of every pair key (u << 32 | v) into the existing forest.
__global__ void k_uf_link_keys(const uint64_t* keys, int64_t n, int32_t* parent, unsigned long long* err) {
    GRID_STRIDE(i, n) uf_union(parent, (int32_t)(keys[i] >> 32), (int32_t)(keys[i] & 0xffffffffULL), err);
}

// Final pointer jumping. The walk only reads: with path halving, another thread could replace
// a root just stored in parent[v] by an intermediate ancestor; here every write is a final root.
__global__ void k_uf_compress(int32_t* parent, int64_t V, unsigned long long* roots) {
    unsigned long long r = 0;
    GRID_STRIDE(v, V) {
        int32_t x = (int32_t)v;
        while (parent[x] != x) x = parent[x];
        parent[v] = x;
        r += (x == (int32_t)v);
    }
    for (int o = 16; o; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0 && r) atomicAdd(roots, r);
}

// Afforest-style sampling over the symmetric view (every pair in both rows): every vertex goes under its
// first neighbour (k_uf_first), then in a few rounds the roots of every vertex and its first two neighbours are
// joined loosely (uf_hook) and the forest flattened; the most frequent root among sampled row slots is
// taken as the giant component's, and only the rows of vertices outside it are linked exactly. An edge
// between a giant vertex and any other is in the other vertex's row too, so skipping the giant's rows
// loses no link (whatever share of the graph that root has). A larger root always goes under a smaller one, so
// every root stays its component's smallest vertex.
// (Exact unions of the second neighbours, whose compare-and-swaps meet at few roots, took 120 us on
// 65,536 vertices and 230 us on 4.8M; two loose rounds with their flattens 20 and 165 us.)
// The shorter the rows, the fewer trees a round joins, and the exact links that follow are the slower the fewer
// roots they meet at. Below eight row entries a vertex on average four rounds (a 80^3 grid with its ids permuted
// 0.50 -> 0.13 ms; random graphs of 4 to 7 entries are done after two and pay 0.03); below 3.5 a round leaves a
// third of the trees, and exact unions of the first two neighbours come first (ladder, permuted ids 0.69 -> 0.15
// ms, random graph of two entries a vertex 0.45 -> 0.21, where two rounds had made the build 1.5 to 6 times
// slower than these).
inline int hook_rounds(int64_t V, int64_t E) { return 2 * E < 7 * V ? 0 : (E < 8 * V ? 4 : 2); }

__global__ void k_uf_link_first_two(CSRView c, int64_t V, int32_t* parent, unsigned long long* err) {
    GRID_STRIDE(v, V) {
        const int32_t d = c.deg[v];
        if (d == 0) continue;
        const int64_t b = c.beg[v];
        uf_union(parent, (int32_t)v, c.adj[b], err);
        if (d > 1) uf_union(parent, (int32_t)v, c.adj[b + 1], err);
    }
}

// A round: sets *hooked where it found trees to join; `before`, the word of the round before, says whether there
// is anything left to do (a lattice in the order of its ids is one tree after the first links).
__global__ void k_uf_hook_first_two(CSRView c, int64_t V, int32_t* parent, const int32_t* before, int32_t* hooked) {
    if (before && *before == 0) return;
    bool any = false;
    GRID_STRIDE(v, V) {
        const int32_t d = c.deg[v];
        if (d == 0) continue;
        const int64_t b = c.beg[v];
        const int32_t r = parent[v];
        any |= uf_hook(parent, r, parent[c.adj[b]]);
        if (d > 1) any |= uf_hook(parent, r, parent[c.adj[b + 1]]);
    }
    if (__syncthreads_or(any) && threadIdx.x == 0 && __ldcg(hooked) == 0) *hooked = 1;
}

// Rows of the vertices outside the sampled giant root: a warp takes 32 vertices, scans their row lengths and
// walks the rows laid end to end, 32 entries at a time. Long rows go to `list` (k_uf_link_long): one warp for a
// hub of 1.5M entries outside the giant took 39 ms.
__global__ void __launch_bounds__(kBlock) k_uf_link_rest(CSRView c, int64_t V, const int32_t* giant_p,
                                                         int32_t* parent, unsigned long long* err, int32_t* list,
                                                         unsigned int* n_list) {
    const int32_t giant = *giant_p;
    __shared__ int64_t s_excl[kBlock / 32][33];
    __shared__ int32_t s_u[kBlock / 32][32];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp * 32; base < V; base += nwarps * 32) {
        const int64_t v = base + lane;
        int64_t cnt = 0;
        if (v < V && parent[v] != giant) cnt = c.deg[v];
        if (cnt > kLongRow) {
            list[atomicAdd(n_list, 1u)] = (int32_t)v;
            cnt = 0;
        }
        int64_t incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        s_excl[wib][lane] = incl - cnt;
        if (lane == 31) s_excl[wib][32] = incl;
        s_u[wib][lane] = (int32_t)v;
        __syncwarp();
        const int64_t total = s_excl[wib][32];
        for (int64_t p0 = 0; p0 < total; p0 += 32) {
            const int64_t p = p0 + lane;
            if (p < total) {
                int lo = 0, hi = 31;
                while (lo < hi) {
                    const int m = (lo + hi + 1) >> 1;
                    if (s_excl[wib][m] <= p) lo = m; else hi = m - 1;
                }
                const int32_t u = s_u[wib][lo];
                uf_union(parent, u, c.adj[c.beg[u] + (p - s_excl[wib][lo])], err);
            }
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kBlock) k_uf_link_long(CSRView c, const int32_t* list, const unsigned int* n_list,
                                                         int32_t* parent, unsigned long long* err) {
    walk_long_rows(list, (int64_t)*n_list, 0, [&](int32_t v) { return c.deg[v]; }, [&](int32_t v, int32_t k, bool on) {
        if (on) uf_union(parent, v, c.adj[c.beg[v] + k], err);
    });
}

}  // namespace

// Components of the symmetric view by the sampled union-find above; labels = smallest vertex id.
static int wcc_labels_sym(gir_dev* g, int32_t* label, int64_t* n_comp) {
    const int64_t V = g->V;
    unsigned long long *roots = nullptr, *err = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[14], 6, &roots));
    int32_t* list = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[13], g->sym.E / kLongRow + 1, &list));
    unsigned int* n_list = reinterpret_cast<unsigned int*>(roots + 5);
    err = roots + 1;
    int32_t* giant = reinterpret_cast<int32_t*>(roots + 2);
    int32_t* hooked = giant + 1;  // a word per round
    GIR_CUDA(g, cudaMemsetAsync(roots, 0, 6 * sizeof(unsigned long long), g->stream));
    if (V == 0) { *n_comp = 0; return GIR_OK; }
    const CSRView s = view(g->sym);
    k_uf_first<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(s, V, label);
    GIR_LAUNCH(g, "k_uf_first");
    GIR_TRY(uf_flatten(g, label, V));
    const int rounds = hook_rounds(V, g->sym.E);
    if (rounds == 0) {
        k_uf_link_first_two<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(s, V, label, err);
        GIR_LAUNCH(g, "k_uf_link_first_two");
        GIR_TRY(uf_flatten(g, label, V));
    }
    for (int r = 0; r < rounds; ++r) {
        k_uf_hook_first_two<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(s, V, label, r > 0 ? hooked + r - 1 : nullptr,
                                                                             hooked + r);
        GIR_LAUNCH(g, "k_uf_hook_first_two");
        GIR_TRY(uf_flatten(g, label, V, hooked + r));
    }
    GIR_TRY(sample_mode(g, g->sym, label, 1, giant));
    trace_mark(g, "wcc: neighbour rounds + sample");
    k_uf_link_rest<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(s, V, giant, label, err, list, n_list);
    GIR_LAUNCH(g, "k_uf_link_rest");
    k_uf_link_long<<<g->num_sms * 8, kBlock, 0, g->stream>>>(s, list, n_list, label, err);
    GIR_LAUNCH(g, "k_uf_link_long");
    k_uf_compress<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(label, V, roots);
    GIR_LAUNCH(g, "k_uf_compress");
    unsigned long long h[2] = {0, 0};
    GIR_CUDA(g, cudaMemcpyAsync(h, roots, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    if (h[1]) return fail(g, GIR_ERR_TIMEOUT, "wcc: union-find link exceeded its retry bound");
    *n_comp = (int64_t)h[0];
    trace_mark(g, "wcc: rest + compress");
    return GIR_OK;
}


// Inserted undirected pairs only (no pair disappeared): the current labels (smallest member,
// so every label is its own root) are a union-find forest already; linking the new pairs into
// it and flattening gives the labels a rebuild would give.
int wcc_union_pairs(gir_dev* g, const uint64_t* keys, int64_t n) {
    const int64_t V = g->V;
    int32_t* label = static_cast<int32_t*>(g->wcc.p);
    unsigned long long* roots = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[14], 4, &roots));
    unsigned long long* err = roots + 1;
    GIR_CUDA(g, cudaMemsetAsync(roots, 0, 2 * sizeof(unsigned long long), g->stream));
    if (V == 0 || n == 0) return GIR_OK;
    k_uf_link_keys<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(keys, n, label, err);
    GIR_LAUNCH(g, "k_uf_link_keys");
    k_uf_compress<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(label, V, roots);
    GIR_LAUNCH(g, "k_uf_compress");
    unsigned long long h[2] = {0, 0};
    GIR_CUDA(g, cudaMemcpyAsync(h, roots, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    if (h[1]) return fail(g, GIR_ERR_TIMEOUT, "wcc: union-find link exceeded its retry bound");
    g->n_wcc = (int64_t)h[0];
    return GIR_OK;
}

int wcc_build(gir_dev* g) {
    int32_t* label = nullptr;
    GIR_TRY(ensure_n(g, g->wcc, g->V + 1, &label));
    GIR_TRY(wcc_labels_sym(g, label, &g->n_wcc));
    g->wcc_built = true;
    return GIR_OK;
}

}  // namespace gir
