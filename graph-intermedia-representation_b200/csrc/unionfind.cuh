// Lock-free union-find over vertex ids (roots are the smallest member of their class), used by the
// block build's edge classes and spanning forest and by the SCC build's reciprocal classes.
#pragma once

#include "common.cuh"

namespace gir {

#ifdef __CUDACC__

__device__ __forceinline__ int32_t uf_find(int32_t* uf, int32_t x) {
    int32_t p = uf[x];
    while (p != x) {
        const int32_t gp = uf[p];
        if (gp != p) uf[x] = gp;  // path halving (benign race: always an ancestor)
        x = p;
        p = uf[x];
    }
    return x;
}

// Joins the classes of a and b; returns the root that this call hooked under the other (each root is
// hooked once, by one caller), or -1 where they were joined already. A failed CAS means another union
// moved the root first, so the retries are bounded by the concurrent unions; the cap only turns a
// broken invariant into an error status. (Reading past the L1 after a failed CAS was slower: every
// search ends at the same few roots, whose lines the L2 then serves one at a time.)
__device__ __forceinline__ int32_t uf_union(int32_t* uf, int32_t a, int32_t b, unsigned long long* err) {
    for (int iter = 0; iter < (1 << 22); ++iter) {
        int32_t ra = uf_find(uf, a), rb = uf_find(uf, b);
        if (ra == rb) return -1;
        if (ra > rb) { const int32_t t = ra; ra = rb; rb = t; }
        if (atomicCAS(&uf[rb], rb, ra) == rb) return rb;
    }
    atomicAdd(err, 1ull);
    return -1;
}

// A loose join for sampling rounds over a flattened forest: the larger of the two entries (a root) goes
// under the smaller unless it is under a still smaller one. No search and no retry, but where one root
// meets several the least wins and the other joins are lost, so exactness must not depend on it. Returns
// whether the two differed.
__device__ __forceinline__ bool uf_hook(int32_t* uf, int32_t ra, int32_t rb) {
    const int32_t lo = ra < rb ? ra : rb, hi = ra < rb ? rb : ra;
    if (lo != hi && uf[hi] > lo) atomicMin(&uf[hi], lo);
    return lo != hi;
}

// Every entry to its root, run as a kernel of its own with no union meanwhile (uf_flatten). A thread writes
// its own entry only, at every step, so that the walks of all threads shorten one another's: a chain of n takes
// about log2 n steps (a lattice's first links form chains as long as its side). Long walks read past the
// L1, which would hide the others' steps; short ones do not, since most end at one root, whose line the
// L2 would serve one warp at a time (4.8M vertices: 106 us, 24 us so).
// Every CTA is resident: an entry points at a smaller one, so whatever a walk meets is done or about to be
// taken up. With more CTAs than fit, those of the first wave went on to their second vertices through entries
// that no thread had started with, one step after another: 56 ms for a path of a million vertices in the order
// of their ids (0.1 ms for the whole component build so). go (if given): nothing to do where it is zero.
__global__ static void __launch_bounds__(256, 8) k_uf_flatten(int32_t* uf, int64_t V, const int32_t* go) {
    if (go && *go == 0) return;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
        int32_t x = uf[v];
        int steps = 0;
        for (int32_t p = uf[x]; p != x; p = ++steps < 4 ? uf[x] : __ldcg(uf + x)) {
            uf[v] = p;
            x = p;
        }
    }
}
inline int uf_flatten(gir_dev* g, int32_t* uf, int64_t V, const int32_t* go = nullptr) {
    constexpr int kThreads = 256;
    if (V <= 0) return GIR_OK;
    const int64_t want = (V + kThreads - 1) / kThreads, fit = (int64_t)g->num_sms * 8;
    k_uf_flatten<<<(int)(want < fit ? want : fit), kThreads, 0, g->stream>>>(uf, V, go);
    GIR_LAUNCH(g, "k_uf_flatten");
    return GIR_OK;
}

// First links without atomics: every vertex with a smaller entry at the head of its (sorted) row goes
// under it, else it is a root. A kernel of its own, before any union.
__global__ static void k_uf_first(CSRView c, int64_t V, int32_t* uf) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t w = c.deg[v] > 0 ? c.adj[c.beg[v]] : (int32_t)v;
        uf[v] = w < (int32_t)v ? w : (int32_t)v;
    }
}

#endif

}  // namespace gir
