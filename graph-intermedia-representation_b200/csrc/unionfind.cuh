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
// broken invariant into an error status.
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

#endif

}  // namespace gir
