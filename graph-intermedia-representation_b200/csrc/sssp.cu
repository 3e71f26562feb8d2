// Delta-stepping shortest paths on the device (GIR::sssp / deltaStepping, gir_query.cpp:629-703):
// uint64 distances, UINT64_MAX = unreachable.
//
// Up to 64 queries run as one traversal (lanes), like the BFS: every vertex carries 64-bit lane
// masks for the work of the current bucket (near), for relaxations beyond it (far) and for the
// lanes settled in the bucket; distances are stored lane-interleaved (dist[v * ld + s]) so a
// relaxation of one edge for many lanes touches one contiguous row. All lanes step through the
// buckets together, each lane running exact Delta-stepping:
//  - bucket k = [k*Delta, (k+1)*Delta): the near vertices relax their light edges
//    (weight < Delta) round after round until no lane re-enters the bucket;
//  - then every (vertex, lane) settled in the bucket relaxes its heavy edges (weight >= Delta)
//    once -- those land in later buckets only. (The reference relaxes all edges every round and
//    has no light/heavy split, gir_query.cpp:674-688; the split changes the work, not the result.)
//  - the next bucket is the smallest live far distance; the far entries inside it become near.
// Rows are read from a weight-sorted copy of the forward CSR, so a row's light edges are its
// prefix. Shortest distances are unique, so the result is the same for every Delta, every
// schedule and every lane grouping.
#include <algorithm>

#include "common.cuh"
#include "frontier.cuh"

namespace gir {

namespace {

constexpr int kBlock = 256;
constexpr uint64_t kInf = ~0ull;

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// Device words of a call. Counters that one phase reads and a later one fills come in threes, used in
// turn (a slot is cleared while no phase can touch it): the near queues (entries << 33 | their light
// edges), the far queue's entries, the smallest distance a far split kept.
// X_SET: the settled queue (entries << 33 | their heavy edges); X_OVF: set when a 16-bit lane distance
// could not hold a tentative distance; X_PHASE .. X_PASSES: where the buckets stand (Bucket);
// X_REACHED, X_EDGES: accumulated over the call, reached (vertex, lane) pairs and their out-edges;
// X_TMP: scratch of the lane order; X_BAR: the loop's grid barrier (its own 128-byte line).
enum { X_NEAR = 0, X_SET = 3, X_FAR = 4, X_MIN = 7, X_OVF = 10, X_ERR = 11, X_PHASE = 12, X_LO, X_ROT, X_SPL, X_FQ,
       X_NCLEAR, X_NSETCLEAR, X_PASSES, X_GROUP = 24, X_REACHED = 24, X_EDGES = 25, X_TMP = 26, X_BAR = 32, X_N = 64 };

// Columns and weights of every entry of the compact copy of `c`, in row order, and the weights' sum and
// maximum (st[0], st[1]). For the forward CSR the weight of entry (u, v) is that of edge u -> v. With
// `reverse` the rows are those of the backward CSR: row v holds the u of every edge u -> v, whose
// weight is the hash weight of (u, v) or the stored weight found in the forward row of u (`f`).
__global__ void k_ws_gather(int64_t V, const int64_t* cb, CSRView c, int hash, int reverse, CSRView f, uint32_t* cols,
                            uint32_t* weights, unsigned long long* st) {
    unsigned long long s = 0, m = 0;
    walk_segments(cb, V, [&](int64_t u, int64_t j) {
        const int64_t i = cb[u] + j, p = c.beg[u] + j;
        const int32_t v = c.adj[p];
        uint32_t w;
        if (!reverse) {
            w = hash ? hash_weight((int32_t)u, v) : c.w[p];
        } else if (hash) {
            w = hash_weight(v, (int32_t)u);
        } else {
            const int64_t b = f.beg[v];
            w = f.w[lower_bound_dev(f.adj, b, b + f.deg[v], (int32_t)u)];
        }
        cols[i] = (uint32_t)v;
        weights[i] = w;
        s += w;
        m = w > m ? w : m;
    });
    s = warp_sum_u64(s);
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if (lane_id() == 0 && (s | m)) {
        atomicAdd(&st[0], s);
        atomicMax(&st[1], m);
    }
}

// Sort keys: row << wbits | weight.
template <class K>
__global__ void k_ws_keys(int64_t V, const int64_t* cb, const uint32_t* weights, int wbits, K* keys) {
    walk_segments(cb, V, [&](int64_t u, int64_t j) { keys[cb[u] + j] = ((K)u << wbits) | (K)weights[cb[u] + j]; });
}

template <class K>
__global__ void k_ws_split(int64_t E, const K* keys, const uint32_t* cols, int wbits, int32_t* adj, uint32_t* w) {
    GRID_STRIDE(i, E) {
        adj[i] = (int32_t)cols[i];
        w[i] = (uint32_t)(keys[i] & (((K)1 << wbits) - 1));
    }
}

// Distances inside a lane group are uint32 when every finite distance fits ((V - 1) * max weight
// < 2^32 - 1): half the bytes, eight lanes per 32-byte sector, 32-bit atomics. Output is uint64.
template <class D>
struct DistT;
template <>
struct DistT<uint64_t> {
    static constexpr uint64_t inf = ~0ull;
    using acc = uint64_t;  // what tentative distances are added up in
    __device__ static void atomic_min(uint64_t* p, uint64_t v) { atomicMin((unsigned long long*)p, (unsigned long long)v); }
};
template <>
struct DistT<uint32_t> {
    static constexpr uint32_t inf = ~0u;
    using acc = uint32_t;
    __device__ static void atomic_min(uint32_t* p, uint32_t v) { atomicMin((unsigned int*)p, v); }
};
// 16-bit lane distances (64 lanes in one 128-byte line) when the distances are small: the
// minimum is taken by compare-and-swap on the aligned 32-bit word holding the lane. Every failed
// swap means the word changed, and both halves only ever decrease, so the loop ends.
template <>
struct DistT<uint16_t> {
    static constexpr uint16_t inf = 0xffffu;
    using acc = uint32_t;  // (holds the sum of a distance and a weight below inf; see judge() in relax_edges)
    __device__ static void atomic_min(uint16_t* p, uint16_t v) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        unsigned int* wp = reinterpret_cast<unsigned int*>(a & ~(uintptr_t)3);
        const int sh = (a & 2) ? 16 : 0;
        unsigned int old = *(volatile unsigned int*)wp;
        while (true) {
            const uint16_t cur = (uint16_t)(old >> sh);
            if (cur <= v) return;
            const unsigned int nw = (old & ~(0xffffu << sh)) | ((unsigned int)v << sh);
            const unsigned int prev = atomicCAS(wp, old, nw);
            if (prev == old) return;
            old = prev;
        }
    }
    // Both halves of an aligned word at once (0xffff: leave it).
    __device__ static void atomic_min_pair(unsigned int* wp, unsigned int v) {
        unsigned int old = *(volatile unsigned int*)wp;
        for (unsigned int nw; (nw = __vminu2(old, v)) != old;) {
            const unsigned int prev = atomicCAS(wp, old, nw);
            if (prev == old) return;
            old = prev;
        }
    }
};

// Sixteen bytes of a distance row: n neighbouring lanes. Rows are padded to a multiple of it (`ld`;
// a single lane is not), so they can be read this way. Eight bytes of 16-bit lanes: with sixteen, 17 lanes kept
// three of the eight threads of a row group at work (4.6 ms a call on a 1M-vertex R-MAT, 3.4 so).
template <class D>
struct alignas(sizeof(D) == 2 ? 8 : 16) Vec {
    static constexpr int n = sizeof(D) == 2 ? 4 : 16 / sizeof(D);
    D v[n];
};
// Past the L1 (kCg) or through it.
template <bool kCg, class D>
__device__ __forceinline__ Vec<D> load_vec(const D* p) {
    if constexpr (sizeof(D) == 2) {
        const uint2 r = kCg ? __ldcg(reinterpret_cast<const uint2*>(p)) : *reinterpret_cast<const uint2*>(p);
        return *reinterpret_cast<const Vec<D>*>(&r);
    } else {
        const uint4 r = kCg ? __ldcg(reinterpret_cast<const uint4*>(p)) : *reinterpret_cast<const uint4*>(p);
        return *reinterpret_cast<const Vec<D>*>(&r);
    }
}

// OR over the eight threads of a row group.
__device__ __forceinline__ unsigned long long or8(unsigned long long x) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) x |= __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Staged append to a far queue (warp-uniform call).
template <int kSlots>
__device__ __forceinline__ void far_push(bool pred, int32_t v, int32_t* s_buf, int& s_n, int32_t* q,
                                         unsigned long long* cnt) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    const int k = __popc(m);
    if (s_n + k > kSlots) stage_flush(s_buf, s_n, q, cnt);
    if (pred) s_buf[s_n + __popc(m & ((1u << lane_id()) - 1))] = v;
    __syncwarp();
    s_n += k;
}

// One 16-byte record per vertex for every queue entry a pass handles: the start of its weight-sorted
// row (two halves), its length and its light edges (weight < delta), which are the row's prefix. Once
// per query group.
__global__ void k_light_split(int64_t V, const int64_t* wb, const int32_t* wdeg, const uint32_t* ww, uint64_t delta,
                              int4* rows) {
    GRID_STRIDE(v, V) {
        const int64_t b = wb[v];
        const int32_t d = wdeg[v];
        int64_t lo = b, hi = b + d;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((uint64_t)ww[mid] < delta) lo = mid + 1; else hi = mid;
        }
        rows[v] = make_int4((int32_t)(uint32_t)b, (int32_t)(b >> 32), d, (int32_t)(lo - b));
    }
}

__device__ __forceinline__ int64_t row_start(const int4& r) {
    return (int64_t)(((uint64_t)(uint32_t)r.y << 32) | (uint32_t)r.x);
}

// Light / heavy edges of a queued vertex (the lengths the queues' offsets add up).
struct LightLen {
    const int4* rows;
    __device__ __forceinline__ int32_t operator()(int32_t v) const { return rows[v].w; }
};
struct HeavyLen {
    const int4* rows;
    __device__ __forceinline__ int32_t operator()(int32_t v) const {
        const int4 r = rows[v];
        return r.z - r.w;
    }
};

// The lane at position p of the group starts at every vertex of srcs[lane_rng[2p] .. lane_rng[2p + 1])
// (one CTA row per lane: blockIdx.y = p).
template <class D>
__global__ void k_sssp_init(const int64_t* lane_rng, const int32_t* srcs, int64_t V, int ld, D* dist,
                            unsigned long long* mask, Queue q, const int4* rows, unsigned long long* cnt) {
    __shared__ int32_t s_stage[kBlock / 32][kStage];
    int32_t* s_buf = s_stage[threadIdx.x >> 5];
    int n_st = 0;
    const LightLen light{rows};
    const int p = blockIdx.y;
    const int64_t lo = lane_rng[2 * p], hi = lane_rng[2 * p + 1];
    for (int64_t base = lo + blockIdx.x * (int64_t)blockDim.x; base < hi; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = base + threadIdx.x;
        const int32_t v = e < hi ? srcs[e] : -1;
        bool on = false;
        if (v >= 0 && v < V) {
            dist[(int64_t)v * ld + p] = 0;
            on = atomicOr(&mask[v], 1ull << p) == 0ull;
        }
        queue_push(on, v, s_buf, n_st, q, light, cnt);
    }
    queue_flush(s_buf, n_st, q, light, cnt);
}

// What a group's passes work on. The near masks and queues rotate: a light pass reads one pair, fills
// the next and clears the masks of the one before, so a queued vertex's mask can be read by every
// warp that holds a piece of its row.
struct Group {
    const int4* rows;
    const int32_t* wadj;          // weight-sorted rows
    const uint32_t* ww;
    uint64_t delta;
    int nl, ld;                   // lanes, row stride of dist
    void* dist;                   // lane distances (see DistT)
    unsigned long long* mask[3];  // near lanes
    Queue q[3];
    unsigned long long* farmask;
    int32_t* farq[2];             // filled by the passes, rewritten into the other one by a far split
    unsigned long long* setmask;  // lanes settled in this bucket
    Queue setq;
    // Lanes whose distance is final: those settled in buckets whose light phase is over (their heavy
    // pass ORs them in). A relaxation drops such lanes of its target without reading their distances,
    // and so does the far split.
    unsigned long long* done;
    unsigned long long* ctl;
};

// Where the buckets stand: the phase to run next and the start of its bucket, which near queue (rot),
// far counter (spl) and far queue (fq) it uses, and the entries of the last near queue and of the
// settled queue whose masks are still to be cleared.
enum { PH_LIGHT = 0, PH_HEAVY = 1, PH_SPLIT = 2, PH_DONE = 3 };
struct Bucket {
    int phase, rot, spl, fq;
    uint64_t lo;
    int64_t n_clear, n_setclear;
    int64_t passes;  // light passes so far
};

// End of the bucket that holds `lo` (saturating).
__host__ __device__ inline uint64_t bucket_end(uint64_t lo, uint64_t delta) {
    const uint64_t b = lo / delta * delta;
    return b + delta < b ? ~0ull : b + delta;
}

// The phase that follows, from the counters the phase left in ctl (rd reads a word).
template <class Read>
__host__ __device__ inline void next_phase(Bucket& s, uint64_t delta, int64_t entries, Read&& rd) {
    if (s.phase == PH_LIGHT) {
        s.n_clear = entries;
        s.rot = (s.rot + 1) % 3;
        ++s.passes;
        if ((rd(X_NEAR + s.rot) >> kQShift) == 0) s.phase = PH_HEAVY;
    } else if (s.phase == PH_HEAVY) {
        s.n_clear = 0;
        s.n_setclear = entries;
        s.lo = bucket_end(s.lo, delta);
        s.phase = rd(X_FAR + s.spl) != 0 ? PH_SPLIT : PH_DONE;
    } else {
        s.n_setclear = 0;
        s.fq ^= 1;
        s.rot = (s.rot + 1) % 3;
        const unsigned long long least = rd(X_MIN + s.spl);
        s.spl = (s.spl + 1) % 3;
        if ((rd(X_NEAR + s.rot) >> kQShift) != 0) {
            s.phase = PH_LIGHT;
        } else if (least == kInf) {
            s.phase = PH_DONE;
        } else {
            s.lo = least;  // an empty bucket: on to the one of the smallest distance still far
        }
    }
}

// A warp's staged appends: near (or settled-next) entries, settled entries, far entries.
struct Stage {
    int32_t *near, *set, *far;
    unsigned char* map;  // 64 slots: the threads that hold the live edges of a step (relax_edges)
    int n_near, n_set, n_far;
};

// Lane distances are read past the L1 where other CTAs may have written them during this launch (kCg:
// the bucket loop; a pass of its own starts with a clean L1).
template <bool kCg, class D>
__device__ __forceinline__ D load_dist(const D* p) {
    return kCg ? __ldcg(p) : *p;
}

// Relaxes one edge per thread, u -> w of weight wt, in the lanes `need` (0: no edge), and queues what
// improved. A warp takes the cheaper of two ways, by the work in front of it:
//  - every thread steps through the lanes of its own edge (few lanes an edge);
//  - eight threads take an edge, so four edges at once, each thread a Vec of the two distance rows at
//    a time (many lanes an edge: the passes of a power-law graph, whose vertices are reached in most
//    lanes at once). The rows come from L2 and HBM; two such steps in flight (64 registers) measured as one
//    (40, and more warps).
// The minimum is taken without waiting for its result: a lane counts as improved by the plain read
// before it. Where another thread lowered the lane in between, that thread queued it as well, and a far
// entry that is no longer far is dropped by the far split, so the queues stay supersets of the lanes
// whose distance changed. Either way an edge's improved lanes go out with one atomicOr per mask.
constexpr int kThreadShare = 4;
template <class D, bool kCg, bool kHeavy, int kSlots>
__device__ __forceinline__ void relax_edges(const Group& a, uint64_t kend, int32_t u, int32_t w, uint32_t wt,
                                            unsigned long long need, unsigned long long* next, const Queue& outq,
                                            unsigned long long* near_cnt, int32_t* farq, unsigned long long* far_cnt,
                                            Stage& st) {
    using A = typename DistT<D>::acc;
    const unsigned any = __ballot_sync(0xffffffffu, need != 0ull);
    if (!any) return;
    D* const dist = static_cast<D*>(a.dist);
    const A kend_a = kend < (uint64_t)(A)~(A)0 ? (A)kend : (A)~(A)0;
    const int ln = lane_id();
    unsigned long long near = 0, far = 0;
    // judges one lane of a target by its tentative distance: 0 no gain, 1 near, 2 far
    auto judge = [&](A du, A dw, uint32_t weight, A& nd) -> int {
        nd = du + weight;
        // (the weight by itself first: the sum of 32 bits could wrap)
        if (sizeof(D) == 2 && (weight >= (A)DistT<D>::inf || nd >= (A)DistT<D>::inf)) {
            // a 16-bit lane cannot hold it: the group is run again with wider lanes
            if (dw == (A)DistT<D>::inf) a.ctl[X_OVF] = 1ull;
            return 0;
        }
        if (nd >= dw) return 0;  // (most relaxations lose)
        return !kHeavy && nd < kend_a ? 1 : 2;
    };
    // and takes it
    auto take = [&](D* at, A du, A dw, uint32_t weight) -> int {
        A nd;
        const int t = judge(du, dw, weight, nd);
        if (t) DistT<D>::atomic_min(at, (D)nd);
        return t;
    };
    const int lanes_max = __reduce_max_sync(0xffffffffu, __popcll(need)), live = __popc(any);
    if (a.ld == 1 || kThreadShare * lanes_max <= live) {
        const D* du_row = dist + (int64_t)u * a.ld;
        D* dw_row = dist + (int64_t)w * a.ld;
        while (need) {
            const int b0 = __ffsll((long long)need) - 1;
            need &= need - 1;
            const int b1 = need ? __ffsll((long long)need) - 1 : b0;
            const bool two = need != 0ull;
            need &= need - 1;
            const A du0 = load_dist<kCg>(du_row + b0), dw0 = __ldcg(dw_row + b0);
            A du1 = 0, dw1 = 0;
            if (two) {
                du1 = load_dist<kCg>(du_row + b1);
                dw1 = __ldcg(dw_row + b1);
            }
            const int t0 = take(dw_row + b0, du0, dw0, wt), t1 = two ? take(dw_row + b1, du1, dw1, wt) : 0;
            if (t0 == 1) near |= 1ull << b0;
            if (t0 == 2) far |= 1ull << b0;
            if (t1 == 1) near |= 1ull << b1;
            if (t1 == 2) far |= 1ull << b1;
        }
    } else {
        constexpr int kV = Vec<D>::n;
        const int sub = ln >> 3, k = ln & 7;
        const int rank = __popc(any & ((1u << ln) - 1));  // this thread's edge among the live ones
        st.map[rank | (need ? 0 : 32)] = (unsigned char)ln;  // (dead edges write past the live ones)
        __syncwarp();
        for (int r0 = 0; r0 < live; r0 += 4) {
            const bool on = r0 + sub < live;
            const int src = on ? st.map[r0 + sub] : 0;
            unsigned long long nj = __shfl_sync(0xffffffffu, need, src);
            nj = on ? nj : 0ull;
            const D* du_row = dist + (int64_t)__shfl_sync(0xffffffffu, u, src) * a.ld;
            D* dw_row = dist + (int64_t)__shfl_sync(0xffffffffu, w, src) * a.ld;
            const uint32_t weight = __shfl_sync(0xffffffffu, wt, src);
            unsigned long long n = 0, f = 0;
            for (int at = k * kV; at < a.ld; at += 8 * kV) {
                const unsigned m = (unsigned)(nj >> at) & ((1u << kV) - 1);
                if (!m) continue;
                const Vec<D> du = load_vec<kCg>(du_row + at), dw = load_vec<true>(dw_row + at);
                unsigned mn = 0, mf = 0;
                if constexpr (sizeof(D) == 2) {
                    // (two lanes share a word, and a swap of one had the other's fail: a swap for both)
#pragma unroll
                    for (int e = 0; e < kV; e += 2) {
                        unsigned pair = 0xffffffffu;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            A nd = 0;
                            const int t = (m >> (e + h)) & 1u ? judge(du.v[e + h], dw.v[e + h], weight, nd) : 0;
                            if (t) pair = h ? (pair & 0xffffu) | (nd << 16) : (pair & 0xffff0000u) | nd;
                            mn |= (unsigned)(t & 1) << (e + h);
                            mf |= (unsigned)(t >> 1) << (e + h);
                        }
                        if (pair != 0xffffffffu)
                            DistT<uint16_t>::atomic_min_pair(reinterpret_cast<unsigned int*>(dw_row + at + e), pair);
                    }
                }
                else
#pragma unroll
                for (int e = 0; e < kV; ++e) {
                    if ((m >> e) & 1u) {
                        const int t = take(dw_row + at + e, du.v[e], dw.v[e], weight);
                        mn |= (unsigned)(t & 1) << e;
                        mf |= (unsigned)(t >> 1) << e;
                    }
                }
                n |= (unsigned long long)mn << at;
                f |= (unsigned long long)mf << at;
            }
            if (!__any_sync(0xffffffffu, (n | f) != 0ull)) continue;
            // every edge's masks go to the thread that holds it
            const int from = 8 * (rank & 3);
            if (!kHeavy) n = __shfl_sync(0xffffffffu, or8(n), from);
            f = __shfl_sync(0xffffffffu, or8(f), from);
            if (need != 0ull && (rank & ~3) == r0) {
                near = n;
                far = f;
            }
        }
        __syncwarp();  // (the map is rewritten by the next edges)
    }
    if (!__any_sync(0xffffffffu, (near | far) != 0ull)) return;
    if (!kHeavy) {
        if (kCg && near) touch_l1(reinterpret_cast<const int32_t*>(a.rows + w) + 3);  // (read at the queue write)
        const bool to_near = near != 0ull && atomicOr(&next[w], near) == 0ull;
        queue_push<kSlots>(to_near, w, st.near, st.n_near, outq, LightLen{a.rows}, near_cnt);
    }
    const bool to_far = far != 0ull && atomicOr(&a.farmask[w], far) == 0ull;
    far_push<kSlots>(to_far, w, st.far, st.n_far, farq, far_cnt);
}

// A warp's share of a pass over the queue's rows (light prefixes or heavy rests), cut into equal runs of
// edges by the queue's offsets; `mask` holds every entry's lanes. The search for a run's first entry and
// the shuffles that find an edge's entry are per edge, not per (edge, lane) pair.
// The runs are dealt round-robin, about kDeal per warp and at most 512 edges long, so every warp gets a
// mix of cheap edges (targets already final) and costly ones; a pass of fewer edges than threads is cut
// finer than a warp's width, since an edge of many lanes is a chain of its own.
constexpr int kDeal = 8;
template <class D, bool kCg, bool kHeavy, int kSlots>
__device__ __forceinline__ void relax_rows(const Group& a, const Bucket& b, const Queue& q, const unsigned long long* mask,
                                           unsigned long long packed, int64_t warp, int64_t nwarps, Stage& st) {
    const int64_t nq = (int64_t)(packed >> kQShift), total = (int64_t)(packed & kQEdges);
    const uint64_t kend = bucket_end(b.lo, a.delta);
    const int nx = (b.rot + 1) % 3;
    const int ln = lane_id();
    int64_t run = (total + nwarps - 1) / nwarps;
    if (run > 32) run = ((total + nwarps * kDeal - 1) / (nwarps * kDeal) + 31) & ~(int64_t)31;
    run = run < kRun ? run : kRun;
    for (int64_t c0 = warp * run; c0 < total; c0 += nwarps * run) {
        const int64_t c1 = c0 + run < total ? c0 + run : total;
        int64_t i0 = kCg ? queue_guess(q.off, nq, total, c0) : queue_find(q.off, 0, nq, (uint64_t)c0);
        int64_t p = c0;
        while (p < c1) {
            // 32 queue entries, one per thread: where its edges start in the run, its row, its lanes
            const int64_t ij = i0 + ln;
            uint32_t relj = 0xffffffffu;
            int64_t begj = 0;
            unsigned long long mj = 0;
            int32_t uj = 0;
            if (ij < nq) {
                uj = __ldcg(q.v + ij);
                const int64_t off = (int64_t)__ldcg((const unsigned long long*)q.off + ij) - c0;
                relj = off <= 0 ? 0u : (off < 0x7fffffff ? (uint32_t)off : 0x7fffffffu);
                const int4 r = a.rows[uj];
                begj = row_start(r) + (kHeavy ? r.w : 0) - off;
                mj = __ldcg(mask + uj);
            }
            const int64_t wnext = i0 + 32 < nq ? (int64_t)__ldcg((const unsigned long long*)q.off + i0 + 32) : total;
            const int64_t wend = wnext < c1 ? wnext : c1;
            for (; p < wend; p += 32) {
                const int64_t pos = p + ln;
                const uint32_t rel = (uint32_t)(pos - c0);
                int x = 0;
#pragma unroll
                for (int s = 16; s; s >>= 1)
                    if (__shfl_sync(0xffffffffu, relj, x + s) <= rel) x += s;
                const int64_t bx = __shfl_sync(0xffffffffu, begj, x);
                unsigned long long need = __shfl_sync(0xffffffffu, mj, x);
                const int32_t u = __shfl_sync(0xffffffffu, uj, x);
                int32_t w = 0;
                uint32_t wt = 0;
                if (pos < wend) {
                    w = __ldcs(a.wadj + bx + rel);
                    wt = __ldcs(a.ww + bx + rel);
                    // (in the loop a single lane is not worth a load that stands before its distance's own)
                    if (a.nl > 1 && (!kCg || (need & (need - 1)))) need &= ~__ldcg(a.done + w);
                } else {
                    need = 0;
                }
                relax_edges<D, kCg, kHeavy, kSlots>(a, kend, u, w, wt, need, a.mask[nx], a.q[nx], a.ctl + X_NEAR + nx,
                                                    a.farq[b.fq], a.ctl + X_FAR + b.spl, st);
            }
            p = wend;
            if (p >= c1) break;
            i0 += 32;
            // Entries without edges keep their slots (a road network's settled queue holds a heavy edge
            // in every thousandth): where the next window has none, jump past the run of such entries.
            if (i0 + 32 < nq && (int64_t)__ldcg((const unsigned long long*)q.off + i0 + 32) <= p)
                i0 = queue_find(q.off, i0 + 32, nq, (uint64_t)p);
        }
    }
}

// A light pass: the near lanes relax their light edges; lanes entering the bucket are settled.
template <class D, bool kCg, int kSlots>
__device__ __forceinline__ void phase_light(const Group& a, const Bucket& b, unsigned long long packed, int64_t tid,
                                            int64_t nthreads, int64_t warp, int64_t nwarps, Stage& st) {
    const int64_t nq = (int64_t)(packed >> kQShift);
    const Queue& q = a.q[b.rot];
    const unsigned long long* mask = a.mask[b.rot];
    const int old = (b.rot + 2) % 3;
    if (tid == 0) a.ctl[X_NEAR + old] = 0ull;
    for (int64_t i = tid; i < b.n_clear; i += nthreads) a.mask[old][__ldcg(a.q[old].v + i)] = 0ull;
    // A short pass is a chain of dependent accesses: the second half of every CTA's warps settles while the
    // first half relaxes; in a long one every warp does both.
    const bool halves = kCg && (int64_t)(packed & kQEdges) <= nwarps * 16 && nq <= nthreads / 2;
    const int64_t half = nwarps / 2;
    if (halves && warp < half) {
        relax_rows<D, kCg, false, kSlots>(a, b, q, mask, packed, warp, half, st);
        return;
    }
    const int64_t first = halves ? (tid & ~(int64_t)31) - half * 32 : tid & ~(int64_t)31;
    for (int64_t base = first; base < nq; base += halves ? nthreads - half * 32 : nthreads) {
        const int64_t i = base + lane_id();
        int32_t u = 0;
        bool settles = false;
        if (i < nq) {  // (a vertex is queued once per pass: its settled mask is this thread's)
            u = __ldcg(q.v + i);
            const unsigned long long m = __ldcg(mask + u), s = __ldcg(a.setmask + u);
            if (m & ~s) a.setmask[u] = s | m;
            settles = m != 0ull && s == 0ull;
        }
        queue_push<kSlots>(settles, u, st.set, st.n_set, a.setq, HeavyLen{a.rows}, a.ctl + X_SET);
    }
    if (!halves) relax_rows<D, kCg, false, kSlots>(a, b, q, mask, packed, warp, nwarps, st);
}

// The heavy pass of a bucket: its settled lanes are final and relax their heavy edges once, into later
// buckets only. (A target lane that becomes final while this runs was settled in this bucket too, so no
// heavy edge improves it: it does not matter whether the relaxation sees its bit.)
template <class D, bool kCg, int kSlots>
__device__ __forceinline__ void phase_heavy(const Group& a, const Bucket& b, unsigned long long packed, int64_t tid,
                                            int64_t nthreads, int64_t warp, int64_t nwarps, Stage& st) {
    const int64_t nset = (int64_t)(packed >> kQShift);
    const int old = (b.rot + 2) % 3;
    for (int64_t i = tid; i < b.n_clear; i += nthreads) a.mask[old][__ldcg(a.q[old].v + i)] = 0ull;
    for (int64_t i = tid; i < nset; i += nthreads) {
        const int32_t u = __ldcg(a.setq.v + i);
        a.done[u] = __ldcg(a.done + u) | __ldcg(a.setmask + u);
    }
    relax_rows<D, kCg, true, kSlots>(a, b, a.setq, a.setmask, packed, warp, nwarps, st);
}

// Splits the far entries at the bucket of b.lo: lanes inside it become near work, later lanes stay far
// (queued in the other far queue) and their smallest distance goes to X_MIN (the bucket to jump to when
// this one turns out empty); settled lanes are dropped. n: the far entries.
template <class D, bool kCg, int kSlots>
__device__ __forceinline__ void phase_split(const Group& a, const Bucket& b, int64_t n, int64_t tid, int64_t nthreads,
                                            Stage& st) {
    const D* dist = static_cast<const D*>(a.dist);
    const uint64_t lo = b.lo / a.delta * a.delta, hi = bucket_end(b.lo, a.delta);
    const int nx = (b.rot + 1) % 3, ln = lane_id();
    if (tid == 0) {
        a.ctl[X_NEAR + (b.rot + 2) % 3] = 0ull;
        a.ctl[X_FAR + (b.spl + 2) % 3] = 0ull;
        a.ctl[X_MIN + (b.spl + 1) % 3] = kInf;
        a.ctl[X_SET] = 0ull;
    }
    for (int64_t i = tid; i < b.n_setclear; i += nthreads) a.setmask[__ldcg(a.setq.v + i)] = 0ull;
    unsigned long long mn = kInf;
    for (int64_t base = tid & ~(int64_t)31; base < n; base += nthreads) {
        const int64_t i = base + ln;
        int32_t w = 0;
        unsigned long long m = 0;
        if (i < n) {
            w = __ldcg(a.farq[b.fq] + i);
            // (lanes already final were reached by a shorter path since: dropped unread)
            m = __ldcg(a.farmask + w) & ~__ldcg(a.done + w);
        }
        // Eight threads take an entry, so four at once, a Vec of its distance row per thread.
        unsigned long long my_near = 0, my_keep = 0;
        constexpr int kV = Vec<D>::n;
        const int sub = ln >> 3, k = ln & 7;
#pragma unroll 2
        for (int j0 = 0; j0 < 32; j0 += 4) {
            const unsigned long long mj = __shfl_sync(0xffffffffu, m, j0 + sub);
            if (!__any_sync(0xffffffffu, mj != 0ull)) continue;
            const D* row = dist + (int64_t)__shfl_sync(0xffffffffu, w, j0 + sub) * a.ld;
            unsigned long long nm = 0, kp = 0;
            for (int at = k * kV; at < a.ld; at += 8 * kV) {
                const unsigned mk = (unsigned)(mj >> at) & ((1u << kV) - 1);
                if (!mk) continue;
                Vec<D> d;
                if (a.ld == 1) d.v[0] = load_dist<kCg>(row);
                else d = load_vec<kCg>(row + at);
#pragma unroll
                for (int e = 0; e < kV; ++e) {
                    const uint64_t x = d.v[e];
                    if (!((mk >> e) & 1u) || x < lo) continue;
                    if (x < hi) {
                        nm |= 1ull << (at + e);
                    } else {
                        kp |= 1ull << (at + e);
                        mn = x < mn ? x : mn;
                    }
                }
            }
            nm = __shfl_sync(0xffffffffu, or8(nm), 8 * (ln & 3));
            kp = __shfl_sync(0xffffffffu, or8(kp), 8 * (ln & 3));
            if ((ln & ~3) == j0) {
                my_near = nm;
                my_keep = kp;
            }
        }
        if (i < n) {
            a.farmask[w] = my_keep;
            if (my_near) a.mask[nx][w] = my_near;
        }
        queue_push<kSlots>(my_near != 0ull, w, st.near, st.n_near, a.q[nx], LightLen{a.rows}, a.ctl + X_NEAR + nx);
        far_push<kSlots>(my_keep != 0ull, w, st.far, st.n_far, a.farq[b.fq ^ 1], a.ctl + X_FAR + (b.spl + 1) % 3);
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, mn, o);
        mn = t < mn ? t : mn;
    }
    if (ln == 0 && mn != kInf) atomicMin(&a.ctl[X_MIN + b.spl], mn);
}

// ---- A phase launched from the host ------------------------------------------------------------
// Bound by the latency of the distance rows' accesses, so occupancy counts: six CTAs an SM (40 registers)
// 16.1 ms a call of 64 sources on the 4.8M-vertex R-MAT, four CTAs (64 registers) 16.6. At 40 registers the light
// phase of 32-bit lanes spills 248 bytes of stores and 372 of loads a thread, the heavy one 120 and 188 (the bucket
// loop, at 64, 128 and 256); five CTAs, about 48 registers, are not measured. Pairs of edge and
// lane dealt one to a thread, numbered by a scan, had taken 26.4 of 35 ms: about 140 instructions a pair
// to find it, and every pair's distance read; now final lanes are dropped by one mask per edge (8 of 10
// edges of the heavy passes have none left) and a row of 64 lanes costs about 20 instructions.
constexpr int kPassThreads = 256;

template <class D, int kPhase>
__global__ void __launch_bounds__(kPassThreads, 6) k_relax(Group a, Bucket b) {
    constexpr int kWarpsPer = kPassThreads / 32;
    __shared__ int32_t s_near[kWarpsPer][kStage], s_set[kWarpsPer][kStage], s_far[kWarpsPer][kStage];
    const int wib = threadIdx.x >> 5;
    __shared__ unsigned char s_map[kWarpsPer][64];
    Stage st{s_near[wib], s_set[wib], s_far[wib], s_map[wib], 0, 0, 0};
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nthreads = (int64_t)gridDim.x * blockDim.x;
    const int nx = (b.rot + 1) % 3;
    if (kPhase == PH_LIGHT) phase_light<D, false, kStage>(a, b, a.ctl[X_NEAR + b.rot], tid, nthreads, tid >> 5, nthreads >> 5, st);
    if (kPhase == PH_HEAVY) phase_heavy<D, false, kStage>(a, b, a.ctl[X_SET], tid, nthreads, tid >> 5, nthreads >> 5, st);
    if (kPhase == PH_SPLIT) phase_split<D, false, kStage>(a, b, (int64_t)a.ctl[X_FAR + b.spl], tid, nthreads, st);
    if (kPhase != PH_HEAVY) queue_flush(st.near, st.n_near, a.q[nx], LightLen{a.rows}, a.ctl + X_NEAR + nx);
    if (kPhase == PH_LIGHT) queue_flush(st.set, st.n_set, a.setq, HeavyLen{a.rows}, a.ctl + X_SET);
    const int fq = kPhase == PH_SPLIT ? b.fq ^ 1 : b.fq, spl = kPhase == PH_SPLIT ? (b.spl + 1) % 3 : b.spl;
    stage_flush(st.far, st.n_far, a.farq[fq], a.ctl + X_FAR + spl);
}

// ---- The bucket loop ---------------------------------------------------------------------------
// Phase after phase in one cooperative launch (a CTA of 1,024 threads per SM, one grid barrier a phase)
// while the phases are small: on a road network, or for a single source, a pass has a few thousand
// edges and was four launches and a host read. It hands back when a pass has more than max_edges edges
// or the far queue more than max_far entries; the host launches such a phase at full occupancy and
// comes back. Bound by latency, about 12 us a pass (a chain of dependent L2 accesses and the barrier): 16
// sources on a 901 x 901 lattice (1,600 passes) 71 -> 18.7 ms, one source on 65,536 vertices 4.4 -> 1.3 ms.
// Of that the first look by interpolation, prefetched row lengths, settling and relaxing on different
// warps, no `done` load for a single lane and the barrier's one-way arrival gave 23.5 -> 18.7 ms; in the
// host-launched phases, which have warps enough to hide the chain, the same cost 21.4 -> 23.2 ms a call of
// 64 sources on the 4.8M-vertex R-MAT (more loads, more targets read), so they are for the loop alone.
constexpr int kLoopSlots = 64;
constexpr int kMaxPhases = 1 << 23;  // of one launch (its barrier's counter is 32 bits wide)

template <class D>
__global__ void __launch_bounds__(kLoopThreads, 1) k_bucket_loop(Group a, int64_t max_edges, int64_t max_far) {
    __shared__ int32_t s_near[32][kLoopSlots], s_set[32][kLoopSlots], s_far[32][kLoopSlots];
    __shared__ unsigned char s_map[32][64];
    __shared__ uint32_t s_n[3][32];
    __shared__ uint64_t s_e[2][32];
    __shared__ unsigned long long s_base[3];
    unsigned int* bar = reinterpret_cast<unsigned int*>(a.ctl + X_BAR);
    const int wib = threadIdx.x >> 5, ln = lane_id();
    // (warps and threads numbered across the CTAs first, so that a short queue spreads over the SMs)
    const int64_t warp = (int64_t)wib * gridDim.x + blockIdx.x, nwarps = (int64_t)gridDim.x * 32;
    const int64_t tid = warp * 32 + ln, nthreads = nwarps * 32;
    auto rd = [&](int i) { return __ldcg(a.ctl + i); };
    Bucket b{(int)rd(X_PHASE), (int)rd(X_ROT), (int)rd(X_SPL), (int)rd(X_FQ), rd(X_LO), (int64_t)rd(X_NCLEAR),
             (int64_t)rd(X_NSETCLEAR), (int64_t)rd(X_PASSES)};
    unsigned met = 0;
    for (int ph = 0; ph < kMaxPhases && b.phase != PH_DONE; ++ph) {
        Stage st{s_near[wib], s_set[wib], s_far[wib], s_map[wib], 0, 0, 0};
        const int nx = (b.rot + 1) % 3;
        int64_t entries = 0;
        int fq = b.fq, spl = b.spl;
        if (b.phase == PH_LIGHT) {
            const unsigned long long packed = rd(X_NEAR + b.rot);
            if ((int64_t)(packed & kQEdges) > max_edges) break;
            entries = (int64_t)(packed >> kQShift);
            phase_light<D, true, kLoopSlots>(a, b, packed, tid, nthreads, warp, nwarps, st);
        } else if (b.phase == PH_HEAVY) {
            const unsigned long long packed = rd(X_SET);
            if ((int64_t)(packed & kQEdges) > max_edges) break;
            entries = (int64_t)(packed >> kQShift);
            phase_heavy<D, true, kLoopSlots>(a, b, packed, tid, nthreads, warp, nwarps, st);
        } else {
            entries = (int64_t)rd(X_FAR + b.spl);
            if (entries > max_far) break;
            fq ^= 1;
            spl = (spl + 1) % 3;
            phase_split<D, true, kLoopSlots>(a, b, entries, tid, nthreads, st);
        }
        // the CTA's staged entries go out with one reservation per queue
        const uint64_t e_near = staged_edges(st.near, st.n_near, LightLen{a.rows});
        const uint64_t e_set = staged_edges(st.set, st.n_set, HeavyLen{a.rows});
        if (ln == 0) {
            s_n[0][wib] = (uint32_t)st.n_near;
            s_n[1][wib] = (uint32_t)st.n_set;
            s_n[2][wib] = (uint32_t)st.n_far;
            s_e[0][wib] = e_near;
            s_e[1][wib] = e_set;
        }
        __syncthreads();
        if (wib < 3) {  // warp 0 near, warp 1 settled, warp 2 far
            const uint32_t n = s_n[wib][ln];
            const uint64_t e = wib < 2 ? s_e[wib][ln] : 0ull;
            const uint64_t n_in = warp_incl_u64(n), e_in = warp_incl_u64(e);
            s_n[wib][ln] = (uint32_t)n_in - n;
            if (wib < 2) s_e[wib][ln] = e_in - e;
            if (ln == 31) {
                unsigned long long* c = a.ctl + (wib == 0 ? X_NEAR + nx : wib == 1 ? X_SET : X_FAR + spl);
                s_base[wib] = n_in ? atomicAdd(c, wib < 2 ? ((unsigned long long)n_in << kQShift) | e_in : n_in) : 0ull;
            }
        }
        __syncthreads();
        if (st.n_near)
            queue_write(st.near, st.n_near, a.q[nx], LightLen{a.rows}, (s_base[0] >> kQShift) + s_n[0][wib],
                        (s_base[0] & kQEdges) + s_e[0][wib]);
        if (st.n_set)
            queue_write(st.set, st.n_set, a.setq, HeavyLen{a.rows}, (s_base[1] >> kQShift) + s_n[1][wib],
                        (s_base[1] & kQEdges) + s_e[1][wib]);
        for (int i = ln; i < st.n_far; i += 32) a.farq[fq][s_base[2] + s_n[2][wib] + i] = st.far[i];
        if (!grid_barrier(bar, a.ctl + X_ERR, met)) return;
        next_phase(b, a.delta, entries, rd);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.ctl[X_PHASE] = (unsigned long long)b.phase;
        a.ctl[X_ROT] = (unsigned long long)b.rot;
        a.ctl[X_SPL] = (unsigned long long)b.spl;
        a.ctl[X_FQ] = (unsigned long long)b.fq;
        a.ctl[X_LO] = b.lo;
        a.ctl[X_NCLEAR] = (unsigned long long)b.n_clear;
        a.ctl[X_NSETCLEAR] = (unsigned long long)b.n_setclear;
        a.ctl[X_PASSES] = (unsigned long long)b.passes;
    }
}

// Reached (vertex, lane) pairs and their out-degrees (the traversed edges of the GTEPS figure).
template <class D>
__global__ void k_sssp_reached(const D* dist, int64_t V, int nl, const int32_t* outdeg,
                               unsigned long long* cnt) {
    unsigned long long r = 0, e = 0;
    GRID_STRIDE(v, V) {
        unsigned c = 0;
        for (int s = 0; s < nl; ++s) c += dist[v * nl + s] != DistT<D>::inf;
        r += c;
        e += (unsigned long long)c * (unsigned long long)outdeg[v];
    }
    for (int o = 16; o; o >>= 1) {
        r += __shfl_xor_sync(0xffffffffu, r, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if (lane_id() == 0) {
        if (r) atomicAdd(&cnt[X_REACHED], r);
        if (e) atomicAdd(&cnt[X_EDGES], e);
    }
}

// dist[v * ld + s] -> out[row[s] * V + v], through 32 x 32 shared-memory tiles, a warp and a tile of its
// own at a time (no CTA barrier), all 32 row loads in flight. On the way it counts what k_sssp_reached
// counts (reached (vertex, lane) pairs and their out-edges), with one atomicAdd per CTA. Bound by DRAM: 64
// lanes of 32 bits on 4.8M vertices move 3.7 GB; a CTA a tile with eight loads in two barriers, and the
// out-degree loaded for every pair instead of once a tile and vertex, took 1.14 ms, this 0.76 (4.9 TB/s).
constexpr int kTransposeWarps = 4;  // (the tiles of 64-bit distances fit the 48 KB of static shared memory)
template <class D>
__global__ void __launch_bounds__(kTransposeWarps * 32) k_transpose(const D* dist, int64_t V, int nl, int ld,
                                                                    const int64_t* row, const int32_t* outdeg,
                                                                    uint64_t* out, unsigned long long* cnt) {
    __shared__ D tiles[kTransposeWarps][32][33];
    __shared__ unsigned long long s_r[kTransposeWarps], s_e[kTransposeWarps];
    const int tx = lane_id(), ty = threadIdx.x >> 5;
    D(*tile)[33] = tiles[ty];
    const int64_t tiles_v = (V + 31) / 32, tiles_s = (nl + 31) / 32;
    unsigned long long r_cnt = 0, e_cnt = 0;
    for (int64_t t = blockIdx.x * (int64_t)kTransposeWarps + ty; t < tiles_v * tiles_s;
         t += (int64_t)gridDim.x * kTransposeWarps) {
        const int64_t v0 = (t % tiles_v) * 32, v = v0 + tx;
        const int s0 = (int)(t / tiles_v) * 32, s = s0 + tx;
        const int nv = V - v0 < 32 ? (int)(V - v0) : 32, ns = nl - s0 < 32 ? nl - s0 : 32;
        const unsigned deg = tx < nv ? (unsigned)outdeg[v] : 0u;
#pragma unroll
        for (int r = 0; r < 32; ++r)
            if (r < nv && tx < ns) tile[r][tx] = __ldcs(dist + (v0 + r) * ld + s);
        __syncwarp();
        unsigned reached = 0;
        if (tx < nv)
            for (int r = 0; r < ns; ++r) {
                const D d = tile[tx][r];
                const bool fin = d != DistT<D>::inf;
                reached += fin;
                __stcs(out + row[s0 + r] * V + v, fin ? (uint64_t)d : kInf);
            }
        r_cnt += reached;
        e_cnt += (unsigned long long)reached * deg;
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) {
        r_cnt += __shfl_xor_sync(0xffffffffu, r_cnt, o);
        e_cnt += __shfl_xor_sync(0xffffffffu, e_cnt, o);
    }
    if (tx == 0) {
        s_r[ty] = r_cnt;
        s_e[ty] = e_cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long rr = 0, ee = 0;
        for (int k = 0; k < kTransposeWarps; ++k) {
            rr += s_r[k];
            ee += s_e[k];
        }
        if (rr) atomicAdd(&cnt[X_REACHED], rr);
        if (ee) atomicAdd(&cnt[X_EDGES], ee);
    }
}

// Lane-order key of every query set: the smallest distance to the hub over the set's sources
// (UINT64_MAX when none reaches it or none is in range).
__global__ void k_set_keys(const int64_t* set_beg, int64_t n_sets, const int32_t* srcs, int64_t V,
                           const uint64_t* hub_dist, uint64_t* key) {
    GRID_STRIDE(i, n_sets) {
        uint64_t k = kInf;
        for (int64_t e = set_beg[i]; e < set_beg[i + 1]; ++e) {
            const int32_t v = srcs[e];
            if (v >= 0 && v < V) k = hub_dist[v] < k ? hub_dist[v] : k;
        }
        key[i] = k;
    }
}

// The vertex of largest in-degree (smallest id among ties) as in-degree << 32 | ~id, and the
// largest finite value of a distance array: st[0], st[1] (atomicMax).
__global__ void k_argmax_deg(int64_t V, const int32_t* deg, unsigned long long* st) {
    unsigned long long best = 0;
    GRID_STRIDE(v, V) {
        const unsigned long long k = ((unsigned long long)(uint32_t)deg[v] << 32) | (uint32_t)~(uint32_t)v;
        best = k > best ? k : best;
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
        best = t > best ? t : best;
    }
    if (lane_id() == 0) atomicMax(&st[0], best);
}
__global__ void k_max_finite(int64_t V, const uint64_t* d, unsigned long long* st) {
    unsigned long long m = 0;
    GRID_STRIDE(v, V) if (d[v] != kInf && d[v] > m) m = d[v];
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if (lane_id() == 0) atomicMax(&st[1], m);
}

}  // namespace

// Weight-sorted compact copy of the forward CSR for one weight mode; with `reverse`, of the
// backward CSR, each entry (v <- u) carrying the weight of the forward edge u -> v.
static int build_weight_sorted(gir_dev* g, int hash, int reverse, DevCSR& ws) {
    const DevCSR& c = reverse ? g->bw : g->fw;
    const int64_t V = g->V, E = c.E;
    store_free(g, ws);
    GIR_TRY(dev_alloc_n(g, &ws.beg, V + 1));
    GIR_TRY(dev_alloc_n(g, &ws.deg, V > 0 ? V : 1));
    GIR_TRY(dev_alloc_n(g, &ws.adj, E > 0 ? E : 1));
    GIR_TRY(dev_alloc_n(g, &ws.w, E > 0 ? E : 1));
    ws.cap = ws.E = E;
    int64_t* cb = ws.beg;
    GIR_TRY(scan_degrees(g, c.deg, V, cb));
    GIR_CUDA(g, cudaMemcpyAsync(ws.deg, c.deg, sizeof(int32_t) * V, cudaMemcpyDeviceToDevice, g->stream));
    if (E == 0) return GIR_OK;
    uint32_t *cols = nullptr, *ctmp = nullptr;
    unsigned long long* st = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[10], E, &cols));
    GIR_TRY(ensure_n(g, g->scratch[11], E, &ctmp));
    GIR_TRY(ensure_n(g, g->sssp_ctl, X_N, &st));
    GIR_CUDA(g, cudaMemsetAsync(st, 0, 2 * sizeof(unsigned long long), g->stream));
    k_ws_gather<<<grid_for(g, E, kBlock), kBlock, 0, g->stream>>>(V, cb, view(c), hash, reverse, view(g->fw), cols, ws.w, st);
    GIR_LAUNCH(g, "k_ws_gather");
    // The sort key holds no more bits than rows and weights have (4.8M vertices, hash weights: 30, so
    // 32-bit keys and four radix passes instead of eight over 64-bit ones).
    unsigned long long h[2] = {0, 100};
    if (!hash || !reverse) {
        GIR_CUDA(g, cudaMemcpyAsync(h, st, sizeof(h), cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
    }
    auto bits_of = [](uint64_t x) {
        int n = 0;
        while (x >> n) ++n;
        return n;
    };
    const int wbits = bits_of(h[1]), bits = std::max(1, wbits + bits_of((uint64_t)(V - 1)));
    if (bits <= 32 && wbits < 32) {
        uint32_t *keys = nullptr, *ktmp = nullptr;
        GIR_TRY(ensure_n(g, g->scratch[8], E, &keys));
        GIR_TRY(ensure_n(g, g->scratch[9], E, &ktmp));
        k_ws_keys<uint32_t><<<grid_for(g, E, kBlock), kBlock, 0, g->stream>>>(V, cb, ws.w, wbits, keys);
        GIR_LAUNCH(g, "k_ws_keys");
        GIR_TRY(sort_pairs_u32(g, keys, ktmp, cols, ctmp, E, bits));
        k_ws_split<uint32_t><<<grid_for(g, E, kBlock), kBlock, 0, g->stream>>>(E, keys, cols, wbits, ws.adj, ws.w);
    } else {
        uint64_t *keys = nullptr, *ktmp = nullptr;
        GIR_TRY(ensure_n(g, g->scratch[8], E, &keys));
        GIR_TRY(ensure_n(g, g->scratch[9], E, &ktmp));
        k_ws_keys<uint64_t><<<grid_for(g, E, kBlock), kBlock, 0, g->stream>>>(V, cb, ws.w, wbits, keys);
        GIR_LAUNCH(g, "k_ws_keys");
        GIR_TRY(sort_pairs_u64(g, keys, ktmp, cols, ctmp, E, bits));
        k_ws_split<uint64_t><<<grid_for(g, E, kBlock), kBlock, 0, g->stream>>>(E, keys, cols, wbits, ws.adj, ws.w);
    }
    GIR_LAUNCH(g, "k_ws_split");
    if (reverse) return GIR_OK;
    // weight statistics for the schedule's features
    g->wstat[hash ? 0 : 1][0] = (double)h[0] / (double)E;
    g->wstat[hash ? 0 : 1][1] = (double)h[1];
    return GIR_OK;
}

namespace {

// Working arrays of one SSSP call, sized for V vertices and up to 64 lanes.
struct Work {
    Group a;
    int4* rows;
    unsigned long long *ctl, *hc;  // device words (X_*), their pinned host copy
};

int sssp_work(gir_dev* g, Work& w) {
    const int64_t V = g->V;
    Group& a = w.a;
    const int mask_slots[3] = {5, 6, 13}, q_slots[3] = {0, 1, 14};
    for (int i = 0; i < 3; ++i) {
        GIR_TRY(ensure_n(g, g->scratch[mask_slots[i]], V + 1, &a.mask[i]));
        GIR_TRY(ensure_n(g, g->scratch[q_slots[i]], V + 1, &a.q[i].v));
        GIR_TRY(ensure_n(g, g->qitems[i], V + 1, &a.q[i].off));
    }
    GIR_TRY(ensure_n(g, g->scratch[2], V + 1, &a.farq[0]));
    GIR_TRY(ensure_n(g, g->scratch[3], V + 1, &a.farq[1]));
    GIR_TRY(ensure_n(g, g->scratch[4], V + 1, &a.setq.v));
    GIR_TRY(ensure_n(g, g->qitems[4], V + 1, &a.setq.off));
    GIR_TRY(ensure_n(g, g->scratch[7], V + 1, &a.farmask));
    GIR_TRY(ensure_n(g, g->scratch[12], V + 1, &a.setmask));
    GIR_TRY(ensure_n(g, g->sssp_done, V + 1, &a.done));
    GIR_TRY(ensure_n(g, g->qitems[3], V + 1, &w.rows));
    GIR_TRY(ensure_n(g, g->sssp_ctl, X_N, &w.ctl));
    a.rows = w.rows;
    a.ctl = w.ctl;
    void* h = nullptr;
    GIR_TRY(pinned(g, kPinnedBytes, &h));
    w.hc = static_cast<unsigned long long*>(h);
    return GIR_OK;
}

// Phases of more edges (far entries) than these run as launches of their own at full occupancy.
constexpr int64_t kLoopMaxRelax = 1ll << 18;
constexpr int64_t kLoopMaxFar = 1ll << 18;

template <class D>
int launch_phase(gir_dev* g, const Group& a, const Bucket& b, int64_t edges, int64_t entries) {
    auto grid = [&](const void* f, int64_t threads) -> int {
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kPassThreads, 0);
        const int64_t cap = (int64_t)g->num_sms * (per_sm > 0 ? per_sm : 1), want = (threads + kPassThreads - 1) / kPassThreads;
        return (int)(want < 1 ? 1 : (want < cap ? want : cap));
    };
    const int64_t threads = edges > entries ? edges : entries;
    if (b.phase == PH_LIGHT)
        k_relax<D, PH_LIGHT><<<grid((const void*)k_relax<D, PH_LIGHT>, threads), kPassThreads, 0, g->stream>>>(a, b);
    else if (b.phase == PH_HEAVY)
        k_relax<D, PH_HEAVY><<<grid((const void*)k_relax<D, PH_HEAVY>, threads), kPassThreads, 0, g->stream>>>(a, b);
    else
        k_relax<D, PH_SPLIT><<<grid((const void*)k_relax<D, PH_SPLIT>, threads), kPassThreads, 0, g->stream>>>(a, b);
    GIR_LAUNCH(g, "k_relax");
    return GIR_OK;
}

// One group of nl lanes (1..64) over the weight-sorted rows `ws`: the lane at
// position p starts from srcs[lane_rng[2p] .. lane_rng[2p + 1]) (device arrays, n_entries sources in all). Lane
// distances have the type D. With nl == 1 and 64-bit lanes the result is written straight into
// `out` (V entries); otherwise position p ends in row lane_row[p] of `out` (rows of V). A 16-bit run
// that met a distance it cannot hold sets *overflow and writes nothing.
template <class D>
int sssp_group(gir_dev* g, Work& wk, const DevCSR& ws, int nl, const int64_t* lane_rng_d, const int32_t* srcs_d,
               int64_t n_entries, const int64_t* lane_row_d, uint64_t* out, uint64_t Dw, bool* overflow) {
    const int64_t V = g->V;
    QueryStats& st = g->qstats;
    *overflow = false;
    Group& a = wk.a;
    unsigned long long *ctl = wk.ctl, *hc = wk.hc;
    const bool direct = nl == 1 && sizeof(D) == sizeof(uint64_t);
    const int ld = nl == 1 ? 1 : (nl + Vec<D>::n - 1) / Vec<D>::n * Vec<D>::n;
    D* dist = nullptr;
    if (direct) {
        dist = reinterpret_cast<D*>(out);
    } else {
        GIR_TRY(ensure_n(g, g->lane_dist, (size_t)V * ld * sizeof(D) / sizeof(uint64_t) + 1,
                         reinterpret_cast<uint64_t**>(&dist)));
    }
    a.wadj = ws.adj; a.ww = ws.w; a.delta = Dw; a.nl = nl; a.ld = ld; a.dist = dist;
    MainTimer timer{g, g->params[GIR_PARAM_PROFILE] != 0.0};
    // (a group that ends on settled-only far entries leaves their lane bits behind)
    for (unsigned long long* m : {a.mask[0], a.mask[1], a.mask[2], a.farmask, a.setmask, a.done})
        GIR_CUDA(g, cudaMemsetAsync(m, 0, sizeof(unsigned long long) * V, g->stream));
    GIR_CUDA(g, cudaMemsetAsync(dist, 0xff, sizeof(D) * V * ld, g->stream));
    GIR_CUDA(g, cudaMemsetAsync(ctl, 0, sizeof(unsigned long long) * X_GROUP, g->stream));
    GIR_CUDA(g, cudaMemsetAsync(ctl + X_MIN, 0xff, sizeof(unsigned long long), g->stream));
    k_light_split<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, ws.beg, ws.deg, ws.w, Dw, wk.rows);
    GIR_LAUNCH(g, "k_light_split");
    if (n_entries > 0) {
        const int gx = (int)((n_entries / nl + kBlock - 1) / kBlock > 0 ? (n_entries / nl + kBlock - 1) / kBlock : 1);
        k_sssp_init<D><<<dim3(gx < 1024 ? gx : 1024, nl), kBlock, 0, g->stream>>>(lane_rng_d, srcs_d, V, ld, dist,
                                                                                  a.mask[0], a.q[0], wk.rows, ctl + X_NEAR);
        GIR_LAUNCH(g, "k_sssp_init");
    }
    // (bucket 0 starts with a light pass, of no entries where no source is in range)
    Bucket b{PH_LIGHT, 0, 0, 0, 0, 0, 0, 0};
    auto rd = [&](int i) { return hc[i]; };
    auto read = [&]() -> int {
        GIR_CUDA(g, cudaMemcpyAsync(hc, ctl, sizeof(unsigned long long) * X_GROUP, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        return GIR_OK;
    };
    int loop_ctas = 0;  // (0: every phase is launched from here)
    GIR_TRY(cooperative_ctas(g, (const void*)k_bucket_loop<D>, kLoopThreads, &loop_ctas));
    bool fresh = loop_ctas > 0;  // the first phase's size was not read: the loop looks at it
    if (!fresh) GIR_TRY(read());
    while (b.phase != PH_DONE) {
        int64_t edges = 0, entries = 0;
        if (!fresh) {
            const unsigned long long packed = b.phase == PH_LIGHT ? hc[X_NEAR + b.rot]
                                              : b.phase == PH_HEAVY ? hc[X_SET] : hc[X_FAR + b.spl] << kQShift;
            edges = (int64_t)(packed & kQEdges);
            entries = b.phase == PH_SPLIT ? (int64_t)hc[X_FAR + b.spl] : (int64_t)(packed >> kQShift);
        }
        if (fresh || (loop_ctas > 0 && edges <= kLoopMaxRelax && (b.phase != PH_SPLIT || entries <= kLoopMaxFar))) {
            if (!fresh) {
                hc[X_PHASE] = (unsigned long long)b.phase;
                hc[X_ROT] = (unsigned long long)b.rot;
                hc[X_SPL] = (unsigned long long)b.spl;
                hc[X_FQ] = (unsigned long long)b.fq;
                hc[X_LO] = b.lo;
                hc[X_NCLEAR] = (unsigned long long)b.n_clear;
                hc[X_NSETCLEAR] = (unsigned long long)b.n_setclear;
                hc[X_PASSES] = (unsigned long long)b.passes;
                GIR_CUDA(g, cudaMemcpyAsync(ctl + X_PHASE, hc + X_PHASE, sizeof(unsigned long long) * (X_PASSES + 1 - X_PHASE),
                                            cudaMemcpyHostToDevice, g->stream));
            }
            GIR_CUDA(g, cudaMemsetAsync(ctl + X_BAR, 0, sizeof(unsigned long long), g->stream));
            int64_t max_edges = kLoopMaxRelax, max_far = kLoopMaxFar;
            void* args[] = {&a, &max_edges, &max_far};
            GIR_TRY(timer.run([&]() -> int {
                GIR_CUDA(g, cudaLaunchCooperativeKernel((const void*)k_bucket_loop<D>, g->num_sms, kLoopThreads, args, 0,
                                                        g->stream));
                return GIR_OK;
            }));
            GIR_TRY(read());
            if (hc[X_ERR]) return fail(g, GIR_ERR_TIMEOUT, "sssp: the bucket loop ran out its barrier bound");
            b = Bucket{(int)hc[X_PHASE], (int)hc[X_ROT], (int)hc[X_SPL], (int)hc[X_FQ], hc[X_LO], (int64_t)hc[X_NCLEAR],
                       (int64_t)hc[X_NSETCLEAR], (int64_t)hc[X_PASSES]};
            fresh = false;
        } else {
            GIR_TRY(timer.run([&]() -> int { return launch_phase<D>(g, a, b, edges, entries); }));
            GIR_TRY(read());
            next_phase(b, a.delta, entries, rd);
        }
        st.launches++;
    }
    st.iterations += b.passes;
    if (g->trace_marks)
        std::fprintf(stderr, "[gir] sssp group of %d lanes, %d-bit distances, delta %llu: %lld light passes\n", nl,
                     (int)(8 * sizeof(D)), (unsigned long long)Dw, (long long)b.passes);
    if (sizeof(D) == sizeof(uint16_t) && hc[X_OVF]) {
        *overflow = true;
        return GIR_OK;
    }
    if (!direct) {  // (the transpose also counts the reached pairs and their edges)
        k_transpose<D><<<g->num_sms * 12, kTransposeWarps * 32, 0, g->stream>>>(dist, V, nl, ld, lane_row_d, g->fw.deg, out, ctl);
        GIR_LAUNCH(g, "k_transpose");
    } else {
        k_sssp_reached<D><<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(dist, V, nl, g->fw.deg, ctl);
        GIR_LAUNCH(g, "k_sssp_reached");
    }
    return GIR_OK;
}

}  // namespace

// The lane order of a weight mode (hub_dist, hub_max): one backward single-lane run from the
// vertex of largest in-degree over a temporary weight-sorted copy of the backward CSR.
static int hub_order(gir_dev* g, int hash) {
    const int mi = hash ? 0 : 1;
    if (g->hub_valid[mi]) return GIR_OK;
    const int64_t V = g->V;
    const double t0 = now_ms();
    const QueryStats saved = g->qstats;
    uint64_t* hd = nullptr;
    GIR_TRY(ensure_n(g, g->hub_dist[mi], V, &hd));
    DevCSR wsb;
    int rc = build_weight_sorted(g, hash, 1, wsb);
    Work wk;
    if (!rc) rc = sssp_work(g, wk);
    int64_t* lanes = nullptr;
    if (!rc) rc = ensure_n(g, g->sssp_lanes, 4, &lanes);
    unsigned long long st[2] = {0, 0};
    if (!rc) rc = cuda_check(g, cudaMemsetAsync(wk.ctl + X_TMP, 0, 2 * sizeof(unsigned long long), g->stream), "memset");
    if (!rc) {
        k_argmax_deg<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, g->bw.deg, wk.ctl + X_TMP);
        rc = cuda_check(g, cudaGetLastError(), "k_argmax_deg");
    }
    if (!rc) rc = cuda_check(g, cudaMemcpyAsync(st, wk.ctl + X_TMP, sizeof(st), cudaMemcpyDeviceToHost, g->stream), "copy");
    if (!rc) rc = cuda_check(g, cudaStreamSynchronize(g->stream), "sync");
    if (!rc) {
        const int32_t hub = (int32_t)~(uint32_t)(st[0] & 0xffffffffull);
        const int64_t h_lane[2] = {0, 1};
        int32_t* src_d = reinterpret_cast<int32_t*>(lanes + 2);
        rc = cuda_check(g, cudaMemcpyAsync(lanes, h_lane, sizeof(h_lane), cudaMemcpyHostToDevice, g->stream), "copy");
        if (!rc) rc = cuda_check(g, cudaMemcpyAsync(src_d, &hub, sizeof(hub), cudaMemcpyHostToDevice, g->stream), "copy");
        // One lane's passes are short, so wide buckets win (fewer phases): 32 mean weights took a 901 x 901
        // lattice's run from 280 ms (a width of 16, 27,000 phases) to 15.
        const uint64_t width = 16 + (uint64_t)(32.0 * g->wstat[mi][0]);
        bool ovf = false;
        if (!rc) rc = sssp_group<uint64_t>(g, wk, wsb, 1, lanes, src_d, 1, nullptr, hd, width, &ovf);
        if (!rc) rc = cuda_check(g, cudaMemsetAsync(wk.ctl + X_TMP + 1, 0, sizeof(unsigned long long), g->stream), "memset");
        if (!rc) {
            k_max_finite<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(V, hd, wk.ctl + X_TMP);
            rc = cuda_check(g, cudaGetLastError(), "k_max_finite");
        }
        if (!rc) rc = cuda_check(g, cudaMemcpyAsync(st, wk.ctl + X_TMP, sizeof(st), cudaMemcpyDeviceToHost, g->stream), "copy");
        if (!rc) rc = cuda_check(g, cudaStreamSynchronize(g->stream), "sync");
        if (!rc) {
            g->hub_max[mi] = st[1];
            g->hub_valid[mi] = true;
        }
    }
    store_free(g, wsb);
    g->qstats = saved;
    if (g->trace_on)
        std::fprintf(stderr, "[gir] sssp lane order (backward run from the hub, %s weights): %.3f ms, max %llu\n",
                     hash ? "hash" : "stored", now_ms() - t0, (unsigned long long)g->hub_max[mi]);
    return rc;
}

int sssp_run(gir_dev* g, const int64_t* set_beg_h, const int32_t* srcs_d, int64_t n_sets, uint64_t delta,
             int weight_mode, uint64_t* dist_d) {
    const int64_t V = g->V;
    QueryStats& st = g->qstats;
    st = QueryStats{};
    g->trace_x.clear();
    g->trace_y.clear();
    if (n_sets <= 0 || V == 0) return GIR_OK;  // (every row of dist_d is written whole by its group)
    const int hash = weight_mode == GIR_WEIGHT_HASH;
    const int mi = hash ? 0 : 1;
    if (!hash && !g->has_weights) return fail(g, GIR_ERR_STATE, "sssp: the graph has no stored weights");
    DevCSR& ws = g->ws[mi];
    if (!g->ws_valid[mi]) {
        GIR_TRY(build_weight_sorted(g, hash, 0, ws));
        g->ws_valid[mi] = true;
    }
    // Lane order: sets sorted by their distance to the hub, so that neighbouring lanes (which
    // share the 32-byte sectors of a distance row) tend to be active in the same buckets. Only
    // the placement of the queries changes, never their results.
    std::vector<int64_t> order((size_t)n_sets);
    for (int64_t i = 0; i < n_sets; ++i) order[i] = i;
    if (n_sets > 1 && g->params[GIR_PARAM_LANE_ORDER] != 0.0) {
        GIR_TRY(hub_order(g, hash));
        int64_t* sb = nullptr;
        GIR_TRY(ensure_n(g, g->sssp_sets, 2 * n_sets + 1, &sb));
        uint64_t* key_d = reinterpret_cast<uint64_t*>(sb + n_sets + 1);
        GIR_CUDA(g, cudaMemcpyAsync(sb, set_beg_h, sizeof(int64_t) * (n_sets + 1), cudaMemcpyHostToDevice, g->stream));
        k_set_keys<<<grid_for(g, n_sets, kBlock), kBlock, 0, g->stream>>>(
            sb, n_sets, srcs_d, V, static_cast<const uint64_t*>(g->hub_dist[mi].p), key_d);
        GIR_LAUNCH(g, "k_set_keys");
        std::vector<uint64_t> key((size_t)n_sets);
        GIR_CUDA(g, cudaMemcpyAsync(key.data(), key_d, sizeof(uint64_t) * n_sets, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        std::stable_sort(order.begin(), order.end(), [&](int64_t x, int64_t y) { return key[x] < key[y]; });
    }
    Work wk;
    GIR_TRY(sssp_work(g, wk));
    int64_t* lanes = nullptr;  // lane ranges (2 per lane), then output rows (1 per lane)
    GIR_TRY(ensure_n(g, g->sssp_lanes, 3 * 64, &lanes));
    // Lane distance width (GIR_PARAM_LANE_BITS): by default 32 bits when every finite distance
    // fits ((V - 1) x max weight), else 64. 16 bits are taken only when asked for, and only while
    // no 16-bit run of this handle has overflowed (an overflow reruns the group wider, so the
    // width never changes a result): their minimum is a compare-and-swap on the 32-bit word the
    // lane shares with its neighbour, and neighbouring lanes active together make those swaps
    // retry (measured slower than 32-bit atomicMin on the LJ-shape graph).
    const double wmax = g->wstat[mi][1] > 0 ? g->wstat[mi][1] : 4294967295.0;
    const int bits = (int)g->params[GIR_PARAM_LANE_BITS];
    const bool fits32 = bits != 64 && (double)V * wmax < 4294967295.0;
    const bool try16 = bits == 16 && !g->narrow16_failed[mi];
    GIR_CUDA(g, cudaEventRecord(g->ev0, g->stream));
    GIR_CUDA(g, cudaMemsetAsync(wk.ctl, 0, sizeof(unsigned long long) * X_N, g->stream));
    std::vector<int64_t> lh(3 * 64);
    for (int64_t g0 = 0; g0 < n_sets; g0 += 64) {
        const int nl = (int)((n_sets - g0) < 64 ? (n_sets - g0) : 64);
        int64_t n_entries = 0;
        for (int j = 0; j < nl; ++j) {
            const int64_t q = order[g0 + j];
            lh[2 * j] = set_beg_h[q];
            lh[2 * j + 1] = set_beg_h[q + 1];
            lh[2 * nl + j] = q;
            n_entries += set_beg_h[q + 1] - set_beg_h[q];
        }
        GIR_CUDA(g, cudaMemcpyAsync(lanes, lh.data(), sizeof(int64_t) * 3 * nl, cudaMemcpyHostToDevice, g->stream));
        uint64_t D = delta;
        float feat[GIR_SCHED_IN];
        sched_sssp_features(g, weight_mode, nl, feat);
        if (D == 0) {
            if (g->schedule == GIR_SCHEDULE_LEARNED && g->sched_loaded) {
                GIR_TRY(sched_choose_delta(g, feat, &D));
            } else {
                D = (uint64_t)g->params[GIR_PARAM_DELTA];
            }
            if (D == 0) D = 16;
        }
        sched_trace(g, feat, sched_delta_class(D));
        bool ovf = false;
        if (nl == 1) {
            GIR_TRY(sssp_group<uint64_t>(g, wk, ws, 1, lanes, srcs_d, n_entries, nullptr, dist_d + order[g0] * V, D, &ovf));
            continue;
        }
        const int64_t* rows_d = lanes + 2 * nl;
        if (try16 && !g->narrow16_failed[mi]) {
            GIR_TRY(sssp_group<uint16_t>(g, wk, ws, nl, lanes, srcs_d, n_entries, rows_d, dist_d, D, &ovf));
            if (!ovf) continue;
            g->narrow16_failed[mi] = true;
            if (g->trace_on) std::fprintf(stderr, "[gir] sssp: 16-bit lane distances overflowed, group rerun\n");
        }
        if (fits32)
            GIR_TRY(sssp_group<uint32_t>(g, wk, ws, nl, lanes, srcs_d, n_entries, rows_d, dist_d, D, &ovf));
        else
            GIR_TRY(sssp_group<uint64_t>(g, wk, ws, nl, lanes, srcs_d, n_entries, rows_d, dist_d, D, &ovf));
    }
    unsigned long long* hc = wk.hc;
    GIR_CUDA(g, cudaMemcpyAsync(hc, wk.ctl, sizeof(unsigned long long) * X_N, cudaMemcpyDeviceToHost, g->stream));
    GIR_CUDA(g, cudaEventRecord(g->ev1, g->stream));
    GIR_CUDA(g, cudaEventSynchronize(g->ev1));
    st.reached = (int64_t)hc[X_REACHED];
    st.edges = (int64_t)hc[X_EDGES];
    float ms = 0;
    GIR_CUDA(g, cudaEventElapsedTime(&ms, g->ev0, g->ev1));
    st.kernel_ms = ms;
    return GIR_OK;
}

}  // namespace gir
