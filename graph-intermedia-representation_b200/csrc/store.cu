// The edge store in HBM: forward, backward and symmetrized slack CSRs, their construction from
// sorted edge keys, and batched in-place row updates.
//
// Reference counterpart: the edge store of gir_constructor/gir.h:248-313 (immutable sorted base
// CSR + tombstone bitmaps + sorted per-vertex delta lists, with a symmetrized int64-offset
// view). Here one slack CSR per direction replaces base + tombstones + deltas: rows stay
// sorted and exact, so traversals need no per-edge tombstone test or delta-list walk.
#include "common.cuh"

namespace gir {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ int64_t row_capacity(int64_t d) {
    // Free room per row for later inserts: an eighth of the row, at least 4 entries; the
    // capacity is rounded up to a multiple of 4 so every row starts 16-byte aligned.
    const int64_t c = d + ((d >> 3) > 4 ? (d >> 3) : 4);
    return (c + 3) & ~(int64_t)3;
}

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// Stored weight of a newly inserted edge u -> x: the hash weight of GIR::edgeWeight when
// wlo > whi, else w(u,v) = lo + hash3(seed,u,v) mod span, the generator's rule (csrc/gen.cpp).
__device__ __forceinline__ uint32_t new_edge_weight(int32_t r, int32_t x, uint64_t wseed, uint32_t wlo, uint32_t whi) {
    if (wlo > whi) return hash_weight(r, x);
    uint64_t z = wseed ^ 0x5851f42d4c957f2dULL;
    auto mix = [](uint64_t s) {
        s += 0x9e3779b97f4a7c15ULL;
        s = (s ^ (s >> 30)) * 0xbf58476d1ce4e5b9ULL;
        s = (s ^ (s >> 27)) * 0x94d049bb133111ebULL;
        return s ^ (s >> 31);
    };
    const uint64_t h = mix(mix(z) ^ mix((uint64_t)(uint32_t)r * 0x2545f4914f6cdd1dULL + (uint64_t)(uint32_t)x));
    return wlo + (uint32_t)(h % ((uint64_t)whi - wlo + 1));
}

// Head and tail positions of every row's run in a sorted key array.
__global__ void k_row_runs(const uint64_t* keys, int64_t n, int64_t* first, int64_t* end) {
    GRID_STRIDE(i, n) {
        const int64_t r = (int64_t)(keys[i] >> 32);
        if (i == 0 || (int64_t)(keys[i - 1] >> 32) != r) first[r] = i;
        if (i == n - 1 || (int64_t)(keys[i + 1] >> 32) != r) end[r] = i + 1;
    }
}

__global__ void k_caps(int64_t V, const int64_t* first, const int64_t* end, int32_t* deg, int64_t* capv) {
    GRID_STRIDE(v, V) {
        const int64_t d = end[v] - first[v];
        deg[v] = (int32_t)d;
        capv[v] = row_capacity(d);
    }
}

__global__ void k_scatter_keys(const uint64_t* keys, const uint32_t* kw, int64_t n, const int64_t* first,
                               const int64_t* beg, int32_t* adj, uint32_t* w) {
    GRID_STRIDE(i, n) {
        const int64_t r = (int64_t)(keys[i] >> 32);
        const int64_t p = beg[r] + (i - first[r]);
        adj[p] = (int32_t)(keys[i] & 0xffffffffULL);
        if (w) w[p] = kw ? kw[i] : 0u;
    }
}

__global__ void k_sym_keys(int64_t V, const int64_t* cb, CSRView c, uint64_t* keys, uint8_t* keep) {
    walk_segments(cb, V, [&](int64_t u, int64_t j) {
        const int64_t i = cb[u] + j;
        const int32_t v = c.adj[c.beg[u] + j];
        keys[2 * i] = ((uint64_t)u << 32) | (uint32_t)v;
        keys[2 * i + 1] = ((uint64_t)(uint32_t)v << 32) | (uint64_t)u;
        keep[2 * i] = keep[2 * i + 1] = (v != (int32_t)u);
    });
}

__global__ void k_distinct_flags(const uint64_t* keys, int64_t n, uint8_t* flag) {
    GRID_STRIDE(i, n) flag[i] = (i == 0 || keys[i] != keys[i - 1]);
}

__global__ void k_compact_copy(int64_t V, const int64_t* cb, CSRView c, int32_t* adj_out, int64_t cap) {
    walk_segments(cb, V, [&](int64_t u, int64_t j) {
        const int64_t i = cb[u] + j;
        if (i < cap) adj_out[i] = c.adj[c.beg[u] + j];
    });
}

__global__ void k_has_edges(CSRView c, int64_t V, const int32_t* u, const int32_t* v, int64_t n, uint8_t* out) {
    GRID_STRIDE(i, n) {
        const int32_t a = u[i], b = v[i];
        bool hit = false;
        if (a >= 0 && b >= 0 && a < V && b < V) {
            const int64_t lo = c.beg[a], hi = lo + c.deg[a];
            const int64_t p = lower_bound_dev(c.adj, lo, hi, b);
            hit = p < hi && c.adj[p] == b;
        }
        out[i] = hit;
    }
}

// ---- batched row updates -------------------------------------------------------------------
// Ops are sorted, distinct keys (row << 32 | col): `ins` are absent edges to add, `del` present
// edges to remove. Between two ops of a row its old entries keep their order and all move by the same
// distance, so every op stands for a run: the entry it inserts, if it does, and the old entries after it as
// far as the row's next op. The runs go through `tmp` and back to their new places; a row's entries before
// its first op are not touched. When a row outgrows its capacity the whole CSR is re-laid-out with fresh
// slack.

// An op's run: `src` the first old entry of the run, `slot` where the run starts in the new row, `col` the
// inserted column or -1, newdeg the row's new length in its first op and -1 in the others.
struct OpRun {
    int64_t src;
    int32_t row, slot, col, newdeg;
};

// len = entries of the op's run. Bound by its chains of binary searches: about ten dependent accesses for
// each of the op's own place in the other list, in the row, and the next op's.
__global__ void k_op_runs(const uint64_t* ins, int64_t n_ins, const uint64_t* del, int64_t n_del, CSRView c, OpRun* runs,
                          int64_t* len, int32_t* overflow, int32_t* bad) {
    const int64_t n_ops = n_ins + n_del;
    GRID_STRIDE(k, n_ops) {
        const bool is_ins = k < n_ins;
        const int64_t own = is_ins ? k : k - n_ins;
        const uint64_t key = is_ins ? ins[own] : del[own];
        const uint64_t r = key >> 32, row_key = r << 32;
        const int32_t col = (int32_t)(key & 0xffffffffULL);
        // the row's first ops, and this op's place in both lists
        const int64_t ib = lower_bound_dev(ins, (int64_t)0, is_ins ? own : n_ins, row_key);
        const int64_t db = lower_bound_dev(del, (int64_t)0, is_ins ? n_del : own, row_key);
        const int64_t i = is_ins ? own : lower_bound_dev(ins, ib, n_ins, key);
        const int64_t d = is_ins ? lower_bound_dev(del, db, n_del, key) : own;
        const int64_t in = i + is_ins, dn = d + !is_ins;
        uint64_t next = ~0ull;  // the row's next op
        if (in < n_ins && ins[in] >> 32 == r) next = ins[in];
        if (dn < n_del && del[dn] >> 32 == r && del[dn] < next) next = del[dn];
        const int64_t beg = c.beg[r], end = beg + c.deg[r];
        const int64_t p = lower_bound_dev(c.adj, beg, end, col);
        const int64_t pn = next == ~0ull ? end : lower_bound_dev(c.adj, p, end, (int32_t)(next & 0xffffffffULL));
        // an insert that is there already or a deletion that is not: the ops do not match this CSR
        if (is_ins == (p < end && c.adj[p] == col)) atomicExch(bad, 1);
        OpRun t;
        t.src = p + !is_ins;
        t.row = (int32_t)r;
        t.slot = (int32_t)(p - beg - (d - db) + (i - ib));
        t.col = is_ins ? col : -1;
        t.newdeg = -1;
        if (i == ib && d == db) {
            const int64_t ie = lower_bound_dev(ins, in, n_ins, (r + 1) << 32);
            const int64_t de = lower_bound_dev(del, dn, n_del, (r + 1) << 32);
            const int64_t nd = end - beg - (de - db) + (ie - ib);
            if (beg + nd > c.beg[r + 1]) atomicExch(overflow, 1);
            t.newdeg = nd > 0 ? (int32_t)nd : 0;
        }
        runs[k] = t;
        len[k] = (pn > t.src ? pn - t.src : 0) + is_ins;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) len[n_ops] = 0;
}

// The runs, end to end, into tmp (off: exclusive scan of their lengths): one read and one write an entry, and
// the search for its run by shuffles, which bounds it (four entries a lane in flight: 0.73 -> 1.0 ms). 100K
// ops on the 4.8M-vertex R-MAT, two batches of three CSRs: 0.73 ms; 1.34 ms where every entry of a touched
// row's rest looked itself up among the row's inserts and deletions, and 2.8 ms each batch before that.
__global__ void k_take_runs(const OpRun* runs, const int64_t* off, int64_t n, CSRView c, int32_t* tmp, uint32_t* tmpw,
                            bool weights, uint64_t wseed, uint32_t wlo, uint32_t whi) {
    walk_segments(off, n, [&](int64_t k, int64_t j) {
        const OpRun t = runs[k];
        const int64_t to = off[k] + j, from = t.src + j - (t.col >= 0);
        const bool added = t.col >= 0 && j == 0;
        tmp[to] = added ? t.col : c.adj[from];
        if (weights) tmpw[to] = added ? new_edge_weight(t.row, t.col, wseed, wlo, whi) : c.w[from];
    });
}

// The sizes the host needs, in one place to read: entries to move, a row outgrew its slack (the flag is
// cleared for the next merge), the batch's bad flag.
__global__ void k_merge_sizes(const int64_t* off, int64_t n, int32_t* overflow, const int32_t* bad, int64_t* out) {
    out[0] = off[n];
    out[1] = *overflow;
    *overflow = 0;
    out[2] = *bad;
}

// The runs from tmp into their rows (which start at beg), and, where asked for, the rows' new lengths.
__global__ void k_put_runs(const OpRun* runs, const int64_t* off, int64_t n, const int64_t* beg, const int32_t* tmp,
                           const uint32_t* tmpw, int32_t* adj, uint32_t* w, int32_t* deg) {
    walk_segments(off, n, [&](int64_t k, int64_t j) {
        const OpRun t = runs[k];
        const int64_t to = beg[t.row] + t.slot + j;
        adj[to] = tmp[off[k] + j];
        if (w) w[to] = tmpw[off[k] + j];
    });
    if (deg) GRID_STRIDE(k, n) if (runs[k].newdeg >= 0) deg[runs[k].row] = runs[k].newdeg;
}

// Full re-layout: the new lengths and how far a row keeps its old entries (keep: all of them where it
// has no op), new capacities, every row's kept entries copied, then the runs.
__global__ void k_set_deg(const OpRun* runs, int64_t n, int32_t* deg, int32_t* keep) {
    GRID_STRIDE(k, n)
        if (runs[k].newdeg >= 0) {
            deg[runs[k].row] = runs[k].newdeg;
            keep[runs[k].row] = runs[k].slot;
        }
}

__global__ void k_new_caps(int64_t V, const int32_t* deg, int64_t* capv) {
    GRID_STRIDE(v, V) capv[v] = row_capacity(deg[v]);
    if (blockIdx.x == 0 && threadIdx.x == 0) capv[V] = 0;
}

__global__ void k_relayout_rows(int64_t V, const int64_t* old_beg, const int32_t* old_adj, const uint32_t* old_w,
                                const int32_t* deg, const int32_t* keep, const int64_t* new_beg, int32_t* new_adj,
                                uint32_t* new_w) {
    walk_segments(new_beg, V, [&](int64_t v, int64_t j) {
        if (j >= deg[v] || j >= keep[v]) return;  // (slack, or a run's)
        const int64_t to = new_beg[v] + j, from = old_beg[v] + j;
        new_adj[to] = old_adj[from];
        if (new_w) new_w[to] = old_w[from];
    });
}

__global__ void k_fill_i32(int32_t* p, int64_t n, int32_t v) { GRID_STRIDE(i, n) p[i] = v; }

__global__ void k_bin_flags(int64_t V, const int32_t* deg, int32_t small, int32_t large, uint8_t* f0, uint8_t* f1,
                            uint8_t* f2, int32_t* ids) {
    GRID_STRIDE(v, V) {
        const int32_t d = deg[v];
        f0[v] = d < small;
        f1[v] = d >= small && d < large;
        f2[v] = d >= large;
        ids[v] = (int32_t)v;
    }
}

// ---- one edge, edited in place (the single-edge latency path) -------------------------------
// Block-cooperative shifts of one row's entries (and weights): all reads of a chunk happen before
// its writes, and chunks move away from the gap, so nothing is overwritten before it is read.
__device__ void row_insert_at(int32_t* adj, uint32_t* w, int64_t p, int64_t end, int32_t x, uint32_t wx) {
    for (int64_t hi = end; hi > p; hi -= blockDim.x) {
        const int64_t lo = hi - (int64_t)blockDim.x > p ? hi - (int64_t)blockDim.x : p;
        const int64_t i = lo + threadIdx.x;
        const bool act = i < hi;
        int32_t a = 0;
        uint32_t b = 0;
        if (act) { a = adj[i]; if (w) b = w[i]; }
        __syncthreads();
        if (act) { adj[i + 1] = a; if (w) w[i + 1] = b; }
        __syncthreads();
    }
    if (threadIdx.x == 0) { adj[p] = x; if (w) w[p] = wx; }
    __syncthreads();
}

__device__ void row_erase_at(int32_t* adj, uint32_t* w, int64_t p, int64_t end) {
    for (int64_t lo = p + 1; lo < end; lo += blockDim.x) {
        const int64_t i = lo + threadIdx.x;
        const bool act = i < end;
        int32_t a = 0;
        uint32_t b = 0;
        if (act) { a = adj[i]; if (w) b = w[i]; }
        __syncthreads();
        if (act) { adj[i - 1] = a; if (w) w[i - 1] = b; }
        __syncthreads();
    }
}

struct MutCSR {
    const int64_t* beg;
    int32_t* deg;
    int32_t* adj;
    uint32_t* w;
};

// One directed change u -> v on the three slack CSRs, in one CTA. out[0]: 0 no-op (the edge is
// already present / absent), 1 applied, 2 a row lacks room (nothing changed: the batch merge
// runs instead). out[1]: 1 when the undirected pair {u, v} appeared, 2 when it disappeared.
// out[2]: layer flags judged with the current labels, as the batch classification does (bit 0
// an edge inside an SCC deleted, bit 1 an inserted cross edge against the rank order, bit 2 a
// cross edge changed, bit 3 the blocks may change, bit 4 an undirected pair appeared between two
// vertices that already share a weakly connected component, so the WCC labels stand). keys:
// u << 32 | v, then the two orientations of the pair.
__global__ void __launch_bounds__(1024) k_single_edit(MutCSR fw, MutCSR bw, MutCSR sym, int32_t u, int32_t v, int insert,
                                                      int weights, uint64_t wseed, uint32_t wlo, uint32_t whi,
                                                      const int32_t* scc, const int32_t* rank, const int32_t* blk,
                                                      const int32_t* head, const int32_t* wcc, unsigned long long* out,
                                                      uint64_t* keys) {
    __shared__ int64_t s_pos[4];
    __shared__ int s_st, s_sym;
    if (threadIdx.x == 0) {
        const int64_t fb = fw.beg[u], fd = fw.deg[u];
        const int64_t pf = lower_bound_dev(fw.adj, fb, fb + fd, v);
        const bool has_uv = pf < fb + fd && fw.adj[pf] == v;
        const int64_t rb = fw.beg[v], rd = fw.deg[v];
        const int64_t pr = lower_bound_dev(fw.adj, rb, rb + rd, u);
        const bool has_vu = pr < rb + rd && fw.adj[pr] == u;
        const int64_t bb = bw.beg[v], bd = bw.deg[v];
        const int64_t pb = lower_bound_dev(bw.adj, bb, bb + bd, u);
        const int64_t su = sym.beg[u], sdu = sym.deg[u], sv = sym.beg[v], sdv = sym.deg[v];
        const int64_t psu = lower_bound_dev(sym.adj, su, su + sdu, v);
        const int64_t psv = lower_bound_dev(sym.adj, sv, sv + sdv, u);
        int st = 1, symc = 0;
        if ((insert != 0) == has_uv) {
            st = 0;
        } else if (insert) {
            symc = has_vu ? 0 : 1;
            const bool room = fb + fd + 1 <= fw.beg[u + 1] && bb + bd + 1 <= bw.beg[v + 1] &&
                              (!symc || (su + sdu + 1 <= sym.beg[u + 1] && sv + sdv + 1 <= sym.beg[v + 1]));
            if (!room) st = 2;
        } else {
            symc = has_vu ? 0 : 2;
        }
        unsigned long long fl = 0;
        if (st == 1 && scc) {
            const bool same = scc[u] == scc[v];
            if (!insert && same) fl |= 1;
            if (!same) fl |= 4;
            if (insert && !same && rank[u] >= rank[v]) fl |= 2;
            if (symc && same && blk) {
                if (symc == 2) fl |= 8;
                else {
                    const int32_t bu = blk[u], bv = blk[v];
                    if (!(bu == bv || head[bv] == u || head[bu] == v)) fl |= 8;
                }
            }
        }
        if (st == 1 && symc == 1 && wcc && wcc[u] == wcc[v]) fl |= 16;
        s_pos[0] = pf; s_pos[1] = pb; s_pos[2] = psu; s_pos[3] = psv;
        s_st = st;
        s_sym = symc;
        out[0] = (unsigned long long)st;
        out[1] = (unsigned long long)symc;
        out[2] = fl;
        keys[0] = ((uint64_t)(uint32_t)u << 32) | (uint32_t)v;
        keys[1] = keys[0];
        keys[2] = ((uint64_t)(uint32_t)v << 32) | (uint32_t)u;
    }
    __syncthreads();
    if (s_st != 1) return;
    const int64_t fend = fw.beg[u] + fw.deg[u], bend = bw.beg[v] + bw.deg[v];
    const int64_t suend = sym.beg[u] + sym.deg[u], svend = sym.beg[v] + sym.deg[v];
    if (insert) {
        row_insert_at(fw.adj, weights ? fw.w : nullptr, s_pos[0], fend, v,
                      weights ? new_edge_weight(u, v, wseed, wlo, whi) : 0u);
        row_insert_at(bw.adj, nullptr, s_pos[1], bend, u, 0u);
        if (s_sym == 1) {
            row_insert_at(sym.adj, nullptr, s_pos[2], suend, v, 0u);
            row_insert_at(sym.adj, nullptr, s_pos[3], svend, u, 0u);
        }
    } else {
        row_erase_at(fw.adj, weights ? fw.w : nullptr, s_pos[0], fend);
        row_erase_at(bw.adj, nullptr, s_pos[1], bend);
        if (s_sym == 2) {
            row_erase_at(sym.adj, nullptr, s_pos[2], suend);
            row_erase_at(sym.adj, nullptr, s_pos[3], svend);
        }
    }
    if (threadIdx.x == 0) {
        const int d = insert ? 1 : -1;
        fw.deg[u] += d;
        bw.deg[v] += d;
        if (s_sym) {
            sym.deg[u] += d;
            sym.deg[v] += d;
        }
    }
}

}  // namespace

// The single-edge latency path: u -> v inserted (insert != 0) or deleted in place (see
// k_single_edit); the result words and keys are device arrays (3 and 3 entries) the caller reads.
int store_single_edit(gir_dev* g, int32_t u, int32_t v, int insert, unsigned long long* out, uint64_t* keys) {
    auto mut = [](DevCSR& c) { return MutCSR{c.beg, c.deg, c.adj, c.w}; };
    const int32_t* scc = g->scc_built ? static_cast<const int32_t*>(g->scc.p) : nullptr;
    const int32_t* rank = g->scc_built ? static_cast<const int32_t*>(g->scc_rank.p) : nullptr;
    const int32_t* blk = g->bct_built ? static_cast<const int32_t*>(g->blk_label.p) : nullptr;
    const int32_t* head = g->bct_built ? static_cast<const int32_t*>(g->blk_head.p) : nullptr;
    const int32_t* wcc = g->wcc_built ? static_cast<const int32_t*>(g->wcc.p) : nullptr;
    k_single_edit<<<1, 1024, 0, g->stream>>>(mut(g->fw), mut(g->bw), mut(g->sym), u, v, insert,
                                             g->has_weights && g->fw.w ? 1 : 0, g->wrule_seed, g->wrule_lo, g->wrule_hi,
                                             scc, rank, blk, head, wcc, out, keys);
    GIR_LAUNCH(g, "k_single_edit");
    return GIR_OK;
}

int store_free(gir_dev* g, DevCSR& c) {
    dev_free(g, c.beg);
    dev_free(g, c.deg);
    dev_free(g, c.adj);
    dev_free(g, c.w);
    c = DevCSR{};
    return GIR_OK;
}

int store_build_csr_from_keys(gir_dev* g, DevCSR& c, const uint64_t* keys, int64_t n, const uint32_t* kw) {
    // keys: sorted, distinct (row << 32 | col). kw (nullable): weight per key.
    const int64_t V = g->V;
    store_free(g, c);
    int64_t *first = nullptr, *endp = nullptr, *capv = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[10], V + 1, &first));
    GIR_TRY(ensure_n(g, g->scratch[11], V + 1, &endp));
    GIR_TRY(ensure_n(g, g->scratch[12], V + 1, &capv));
    GIR_CUDA(g, cudaMemsetAsync(first, 0, sizeof(int64_t) * (V + 1), g->stream));
    GIR_CUDA(g, cudaMemsetAsync(endp, 0, sizeof(int64_t) * (V + 1), g->stream));
    GIR_TRY(dev_alloc_n(g, &c.beg, V + 1));
    GIR_TRY(dev_alloc_n(g, &c.deg, V > 0 ? V : 1));
    if (n > 0) {
        k_row_runs<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(keys, n, first, endp);
        GIR_LAUNCH(g, "k_row_runs");
    }
    k_caps<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, first, endp, c.deg, capv);
    GIR_LAUNCH(g, "k_caps");
    GIR_CUDA(g, cudaMemsetAsync(capv + V, 0, sizeof(int64_t), g->stream));
    GIR_TRY(exclusive_scan_i64(g, capv, c.beg, V + 1));
    int64_t total = 0;
    GIR_CUDA(g, cudaMemcpyAsync(&total, c.beg + V, sizeof(int64_t), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    GIR_TRY(dev_alloc_n(g, &c.adj, total > 0 ? total : 4));
    if (kw) GIR_TRY(dev_alloc_n(g, &c.w, total > 0 ? total : 4));
    c.cap = total;
    c.E = n;
    if (n > 0) {
        k_scatter_keys<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(keys, kw, n, first, c.beg, c.adj, c.w);
        GIR_LAUNCH(g, "k_scatter_keys");
    }
    return GIR_OK;
}

int store_build_sym(gir_dev* g) {
    // Symmetrized view (buildWCC, gir.cpp:599-625): {u,v} for every u -> v with u != v, both
    // directions, sorted and distinct.
    const int64_t V = g->V, E = g->fw.E;
    int64_t* cb = nullptr;
    uint64_t *keys = nullptr, *tmp = nullptr, *out = nullptr;
    uint8_t* keep = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[0], V + 1, &cb));
    GIR_TRY(ensure_n(g, g->scratch[1], 2 * E + 1, &keys));
    GIR_TRY(ensure_n(g, g->scratch[2], 2 * E + 1, &tmp));
    GIR_TRY(ensure_n(g, g->scratch[3], 2 * E + 1, &keep));
    GIR_TRY(scan_degrees(g, g->fw.deg, V, cb));
    if (E > 0) {
        k_sym_keys<<<grid_for(g, E, kBlock), kBlock, 0, g->stream>>>(V, cb, view(g->fw), keys, keep);
        GIR_LAUNCH(g, "k_sym_keys");
    }
    int64_t n = 0;
    GIR_TRY(select_flagged_u64(g, keys, keep, tmp, 2 * E, &n));
    GIR_TRY(sort_keys_u64(g, tmp, keys, n, edge_key_bits(g->V)));
    if (n > 0) {
        k_distinct_flags<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(tmp, n, keep);
        GIR_LAUNCH(g, "k_distinct_flags");
    }
    out = keys;
    int64_t m = 0;
    GIR_TRY(select_flagged_u64(g, tmp, keep, out, n, &m));
    return store_build_csr_from_keys(g, g->sym, out, m, nullptr);
}

int store_compact_csr(gir_dev* g, const DevCSR& c, int64_t* beg_out, int32_t* adj_out, int64_t cap) {
    // beg_out / adj_out: device pointers (V+1 / cap entries)
    GIR_TRY(scan_degrees(g, c.deg, g->V, beg_out));
    if (c.E > 0 && adj_out && cap > 0) {
        k_compact_copy<<<grid_for(g, c.E, kBlock), kBlock, 0, g->stream>>>(g->V, beg_out, view(c), adj_out, cap);
        GIR_LAUNCH(g, "k_compact_copy");
    }
    return GIR_OK;
}

int store_has_edges(gir_dev* g, const DevCSR& c, const int32_t* u, const int32_t* v, int64_t n, uint8_t* out) {
    if (n <= 0) return GIR_OK;
    k_has_edges<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(view(c), g->V, u, v, n, out);
    GIR_LAUNCH(g, "k_has_edges");
    return GIR_OK;
}

int store_apply_ops(gir_dev* g, DevCSR& c, const uint64_t* ins, int64_t n_ins, const uint64_t* del, int64_t n_del,
                    bool weights, int32_t* bad, int32_t* overflow) {
    if (n_ins + n_del == 0) return GIR_OK;
    const int64_t V = g->V;
    const int64_t n = n_ins + n_del;
    int32_t* tmp = nullptr;
    int64_t *off = nullptr, *words = nullptr;  // (words: the sizes the host reads)
    OpRun* runs = nullptr;
    uint32_t* tmpw = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[9], n, &runs));
    GIR_TRY(ensure_n(g, g->scratch[10], n + 1, &off));
    GIR_TRY(ensure_n(g, g->scratch[12], 4, &words));
    k_op_runs<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(ins, n_ins, del, n_del, view(c), runs, off, overflow, bad);
    GIR_LAUNCH(g, "k_op_runs");
    GIR_TRY(exclusive_scan_i64(g, off, off, n + 1));
    k_merge_sizes<<<1, 1, 0, g->stream>>>(off, n, overflow, bad, words);
    GIR_LAUNCH(g, "k_merge_sizes");
    void* hp = nullptr;
    GIR_TRY(pinned(g, kPinnedBytes, &hp));
    int64_t* h = static_cast<int64_t*>(hp);
    GIR_CUDA(g, cudaMemcpyAsync(h, words, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    const int64_t n_moved = h[0];
    const bool ovf = h[1] != 0;
    if (h[2]) return fail(g, GIR_ERR_MALFORMED, "edge update: the backward CSR is not the transpose of the forward CSR");
    const bool wts = weights && c.w;
    GIR_TRY(ensure_n(g, g->stage_out, n_moved + 4, &tmp));
    if (wts) GIR_TRY(ensure_n(g, g->scratch[3], n_moved + 4, &tmpw));
    if (n_moved > 0) {
        k_take_runs<<<grid_for(g, n_moved, kBlock), kBlock, 0, g->stream>>>(runs, off, n, view(c), tmp, tmpw, wts,
                                                                            g->wrule_seed, g->wrule_lo, g->wrule_hi);
        GIR_LAUNCH(g, "k_take_runs");
    }
    const int put_grid = grid_for(g, n_moved > n ? n_moved : n, kBlock);
    if (!ovf) {
        k_put_runs<<<put_grid, kBlock, 0, g->stream>>>(runs, off, n, c.beg, tmp, tmpw, c.adj, wts ? c.w : nullptr, c.deg);
        GIR_LAUNCH(g, "k_put_runs");
    } else {
        // Some row outgrew its slack: new layout for the whole CSR.
        trace_mark(g, "store: merge before relayout");
        int32_t* keep = nullptr;
        int64_t* capv = nullptr;
        GIR_TRY(ensure_n(g, g->scratch[0], V + 1, &keep));
        GIR_TRY(ensure_n(g, g->scratch[1], V + 1, &capv));
        k_fill_i32<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(keep, V, INT32_MAX);
        GIR_LAUNCH(g, "k_fill_i32");
        k_set_deg<<<grid_for(g, n, kBlock), kBlock, 0, g->stream>>>(runs, n, c.deg, keep);
        GIR_LAUNCH(g, "k_set_deg");
        k_new_caps<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, c.deg, capv);
        GIR_LAUNCH(g, "k_new_caps");
        int64_t* nbeg = nullptr;
        GIR_TRY(dev_alloc_n(g, &nbeg, V + 1));
        GIR_TRY(exclusive_scan_i64(g, capv, nbeg, V + 1));
        int64_t total = 0;
        GIR_CUDA(g, cudaMemcpyAsync(&total, nbeg + V, sizeof(int64_t), cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        int32_t* nadj = nullptr;
        uint32_t* nw = nullptr;
        GIR_TRY(dev_alloc_n(g, &nadj, total > 0 ? total : 4));
        if (c.w) GIR_TRY(dev_alloc_n(g, &nw, total > 0 ? total : 4));
        k_relayout_rows<<<grid_for(g, total, kBlock), kBlock, 0, g->stream>>>(V, c.beg, c.adj, c.w, c.deg, keep, nbeg, nadj,
                                                                              nw);
        GIR_LAUNCH(g, "k_relayout_rows");
        k_put_runs<<<put_grid, kBlock, 0, g->stream>>>(runs, off, n, nbeg, tmp, tmpw, nadj, wts ? nw : nullptr, nullptr);
        GIR_LAUNCH(g, "k_put_runs");
        dev_free(g, c.beg);
        dev_free(g, c.adj);
        dev_free(g, c.w);
        c.beg = nbeg; c.adj = nadj; c.w = nw; c.cap = total;
        trace_mark(g, "store: relayout");
    }
    c.E += n_ins - n_del;
    return GIR_OK;
}

int store_build_bins(gir_dev* g) {
    // Vertices by in-degree class for the bottom-up kernels: [0, small) thread per vertex,
    // [small, large) warp per vertex, [large, inf) CTA per vertex.
    const int64_t V = g->V;
    int32_t *bins = nullptr, *ids = nullptr;
    uint8_t *f0 = nullptr, *f1 = nullptr, *f2 = nullptr;
    GIR_TRY(ensure_n(g, g->bins, V + 1, &bins));
    GIR_TRY(ensure_n(g, g->scratch[4], V + 1, &ids));
    GIR_TRY(ensure_n(g, g->scratch[5], V + 1, &f0));
    GIR_TRY(ensure_n(g, g->scratch[6], V + 1, &f1));
    GIR_TRY(ensure_n(g, g->scratch[7], V + 1, &f2));
    k_bin_flags<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, g->bw.deg, (int32_t)g->params[GIR_PARAM_SMALL_DEG],
                                                                   (int32_t)g->params[GIR_PARAM_LARGE_DEG], f0, f1, f2, ids);
    GIR_LAUNCH(g, "k_bin_flags");
    int64_t n0 = 0, n1 = 0, n2 = 0;
    GIR_TRY(select_flagged_i32(g, ids, f0, bins, V, &n0));
    GIR_TRY(select_flagged_i32(g, ids, f1, bins + n0, V, &n1));
    GIR_TRY(select_flagged_i32(g, ids, f2, bins + n0 + n1, V, &n2));
    g->bin_n[0] = n0; g->bin_n[1] = n1; g->bin_n[2] = n2;
    g->bins_valid = true;
    return GIR_OK;
}

}  // namespace gir
