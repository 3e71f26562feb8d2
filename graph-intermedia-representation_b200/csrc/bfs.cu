// Direction-optimizing breadth-first search on the device (GIR::bfs, gir_query.cpp:108-294).
//
// Up to 64 queries run as one traversal: every vertex carries 64-bit lane masks (seen, current
// frontier, next frontier), bit i standing for query i. A query's level of v is the iteration in
// which its bit first reaches v, so every query gets exactly the levels a single-source BFS
// gives it. One source per lane is GIR::bfs; several sources in a lane are the multi-source
// query (all start at level 0).
//
// Each iteration runs in one of two directions, chosen per iteration by the schedule:
//  - top-down: the frontier queue's out-edges are cut into equal runs (edge-balanced, as the
//    reference's 2048-edge chunks, gir_query.cpp:182-219); a lane bit newly set in seen[w] is
//    OR-ed into next[w] and w is queued once (the atomicOr that turns next[w] non-zero queues it);
//  - bottom-up: every vertex that some lane has not reached ORs its in-neighbours' frontier
//    masks and stops once every missing lane is found (gir_query.cpp:232-279), with vertices
//    binned by in-degree: a thread, a warp or a CTA per vertex.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "frontier.cuh"
#include "sched_net.cuh"

namespace gir {

namespace {

constexpr int kBlock = 256;

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// counters: [0] the queue: entries << 33 | their out-edges, [1] (vertex, lane) pairs reached this
// iteration, [2] out-edges of those pairs,
// [4] the device-decided direction of the next level and [5..8] its features (learned schedule)
enum { C_Q = 0, C_PAIRS = 1, C_MEDGES = 2, C_DIR = 4, C_FEAT = 5, C_N = 9 };

// Where levels go. Written straight into the output's rows, every (vertex, lane) pair is a 4-byte write
// into another 32-byte sector; with many lanes the levels below kPlaneLevels are kept in four bit planes
// per vertex instead (one sector: bit s of plane b is bit b of lane s's code, 15 - level, 0 for none), and
// k_expand_levels writes every row of the output once, coalesced, after the search. (The minus-one fill
// of the output goes with it.)
constexpr int kPlaneLevels = 15;
struct Levels {
    int32_t* out;
    int64_t V;
    unsigned long long* plane;  // 4 per vertex, zeroed; null: every level goes straight to the output
};
// The planes cost a sector per vertex and pass, the straight writes a sector per pair. 64 lanes, 4.8M
// vertices: 5.1 ms a call with straight writes, 2.7 ms so; small calls keep those and save the launch.
constexpr int kPlaneMinLanes = 8;
constexpr int64_t kPlaneMinPairs = 1ll << 23;

// Level L of the lanes nb of vertex v. Several threads may write lanes of one vertex.
__device__ __forceinline__ void write_levels(const Levels& l, int32_t v, uint64_t nb, int32_t L) {
    if (l.plane && L < kPlaneLevels) {
        const int code = kPlaneLevels - L;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if ((code >> b) & 1) atomicOr(l.plane + 4 * (int64_t)v + b, (unsigned long long)nb);
        return;
    }
    while (nb) {
        const int s = __ffsll((long long)nb) - 1;
        nb &= nb - 1;
        l.out[(int64_t)s * l.V + v] = L;
    }
}
// The same by a warp whose lanes all hold v and nb.
__device__ __forceinline__ void write_levels_warp(const Levels& l, int32_t v, uint64_t nb, int32_t L) {
    const int ln = lane_id();
    if (l.plane && L < kPlaneLevels) {
        if (nb && ln < 4 && (((kPlaneLevels - L) >> ln) & 1)) atomicOr(l.plane + 4 * (int64_t)v + ln, (unsigned long long)nb);
        return;
    }
    if ((nb >> ln) & 1ull) l.out[(int64_t)ln * l.V + v] = L;
    if ((nb >> 32 >> ln) & 1ull) l.out[(int64_t)(ln + 32) * l.V + v] = L;
}

// The output rows from the planes: a thread per vertex, so a warp writes 128 bytes of each row. Lanes that
// were seen without a code have their level in the output already. Bound by the output's writes.
__global__ void __launch_bounds__(kBlock) k_expand_levels(Levels l, const uint64_t* seen, int nl) {
    GRID_STRIDE(v, l.V) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(l.plane + 4 * v);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(l.plane + 4 * v + 2);
        const uint64_t done = seen[v] & ~(a.x | a.y | b.x | b.y);
        for (int s = 0; s < nl; ++s) {
            const int code = (int)((a.x >> s) & 1) | (int)((a.y >> s) & 1) << 1 | (int)((b.x >> s) & 1) << 2 |
                             (int)((b.y >> s) & 1) << 3;
            if (!((done >> s) & 1)) __stcs(l.out + (int64_t)s * l.V + v, code ? kPlaneLevels - code : -1);
        }
    }
}

__device__ __forceinline__ void warp_add_u64(unsigned long long* p, unsigned long long x) {
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane_id() == 0 && x) atomicAdd(p, x);
}

// Row lengths of queue entries.
struct RowLen {
    const int32_t* deg;
    __device__ __forceinline__ int32_t operator()(int32_t v) const { return deg[v]; }
};

// Sources: lane s of the group starts at every vertex of set s (set_beg is device memory). Counts
// the sources' (vertex, lane) pairs and out-edges with the queue.
__global__ void k_init_sources(const int64_t* set_beg, int n_lanes, const int32_t* srcs, int64_t V, uint64_t* seen,
                               uint64_t* front, Queue q, unsigned long long* cnt, Levels level, const int32_t* deg) {
    __shared__ int32_t s_stage[kBlock / 32][kStage];
    int n_st = 0;
    const int64_t lo = set_beg[0], hi = set_beg[n_lanes];
    unsigned long long pairs = 0, medges = 0;
    for (int64_t base = lo + blockIdx.x * (int64_t)blockDim.x; base < hi; base += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = base + threadIdx.x;
        const int32_t v = e < hi ? srcs[e] : -1;
        bool on = false;
        if (v >= 0 && v < V) {
            int s = 0, t = n_lanes - 1;  // lane of entry e: the last set starting at or before it
            while (s < t) {
                const int m = (s + t + 1) >> 1;
                if (set_beg[m] <= e) s = m; else t = m - 1;
            }
            const unsigned long long bit = 1ull << s;
            if (!(atomicOr((unsigned long long*)&seen[v], bit) & bit)) {
                on = atomicOr((unsigned long long*)&front[v], bit) == 0ull;
                write_levels(level, v, bit, 0);
                ++pairs;
                medges += (unsigned long long)deg[v];
            }
        }
        queue_push(on, v, s_stage[threadIdx.x >> 5], n_st, q, RowLen{deg}, &cnt[C_Q]);
    }
    queue_flush(s_stage[threadIdx.x >> 5], n_st, q, RowLen{deg}, &cnt[C_Q]);
    warp_add_u64(&cnt[C_PAIRS], pairs);
    warp_add_u64(&cnt[C_MEDGES], medges);
}

// What a warp carries through a level: its staging buffer and the level's sums.
struct LevelAcc {
    int32_t* s_buf;
    int n = 0;
    unsigned long long pairs = 0, medges = 0;
};

// Masks a level works on: the frontier's lanes, the lanes seen so far, and the next frontier's
// lanes (zero wherever this level has not written).
struct LevelMasks {
    const uint64_t* front;
    uint64_t* seen;
    uint64_t* next;
    Levels level;
};

// A top-down level (walk_rows). One pass does the whole level: the atomicOr on seen[w] hands every
// newly reached (w, lane) pair to exactly one thread, which writes its level and adds it to the next
// frontier; the pair's bit is for the next level, so no thread of this level reads what another
// writes, beyond the pre-check of seen[w] that only saves atomics.
struct TopDown {
    CSRView fw;
    LevelMasks k;
    int32_t L;
    unsigned long long pairs, medges;  // this thread's sums
    __device__ __forceinline__ int32_t deg(int32_t u) const { return fw.deg[u]; }
    __device__ __forceinline__ void row(int32_t u, int64_t& beg, unsigned long long& lanes) const {
        beg = fw.beg[u];
        lanes = __ldcg((const unsigned long long*)k.front + u);
    }
    __device__ __forceinline__ int32_t adj(int64_t i, unsigned long long) const { return fw.adj[i]; }
    __device__ __forceinline__ unsigned long long want(int32_t w, unsigned long long lanes) const {
        return lanes & ~__ldcg((const unsigned long long*)k.seen + w);
    }
    __device__ __forceinline__ bool apply(int32_t w, unsigned long long, unsigned long long bits, int32_t& e) {
        const unsigned d = (unsigned)fw.deg[w];
        const unsigned long long nb = bits & ~atomicOr((unsigned long long*)k.seen + w, bits);
        if (!nb) return false;
        const bool fresh = atomicOr((unsigned long long*)k.next + w, nb) == 0ull;
        write_levels(k.level, w, nb, L);
        const unsigned c = __popcll(nb);
        pairs += c;
        medges += (unsigned long long)c * d;
        e = w;
        return fresh;
    }
};

__device__ __forceinline__ uint64_t warp_or_u64(uint64_t x) {
    const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)(x & 0xffffffffu));
    const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(x >> 32));
    return ((uint64_t)hi << 32) | lo;
}

// The frontier masks of the row entries [j, j + 4) below e: one 16-byte load (rows start 16-byte aligned
// and their slots are a multiple of four), four gathers in flight.
__device__ __forceinline__ uint64_t four_fronts(const unsigned long long* front, const int32_t* adj, int64_t j, int64_t e) {
    if (j >= e) return 0;
    const int4 a = *reinterpret_cast<const int4*>(adj + j);
    uint64_t got = __ldcg(front + a.x);
    if (j + 1 < e) got |= __ldcg(front + a.y);
    if (j + 2 < e) got |= __ldcg(front + a.z);
    if (j + 3 < e) got |= __ldcg(front + a.w);
    return got;
}

// Bottom-up, thread per vertex (small in-degree bin), over ids[i] for i = first, first + stride, ..
// (first and stride are multiples of 32 threads apart, so a warp stays together). A vertex is its
// thread's alone, so its masks need no atomics.
__device__ __forceinline__ void bu_threads(const int32_t* ids, int64_t n, int64_t first, int64_t stride,
                                           const CSRView& bw, const LevelMasks& k, uint64_t all, const int32_t* outdeg,
                                           int32_t L, const Queue& out, unsigned long long* cnt, LevelAcc& acc) {
    const unsigned long long* front = (const unsigned long long*)k.front;
    for (int64_t base = first; base < n; base += stride) {
        const int64_t i = base + lane_id();
        bool on = false;
        int32_t v = 0;
        if (i < n) {
            v = ids[i];
            const uint64_t s = __ldcg((const unsigned long long*)k.seen + v);
            const uint64_t want = all & ~s;
            if (want) {
                // four row entries per step (rows start 16-byte aligned), their frontier masks
                // loaded together; entries read past the point where every missing lane is found
                // are in-neighbours all the same, so the lanes they add are found lanes too
                uint64_t got = 0;
                const int64_t b = bw.beg[v], e = b + bw.deg[v];
                int64_t j = b;
                for (; j + 4 <= e; j += 4) {
                    const int4 a4 = *reinterpret_cast<const int4*>(bw.adj + j);
                    got |= __ldcg(front + a4.x) | __ldcg(front + a4.y) | __ldcg(front + a4.z) | __ldcg(front + a4.w);
                    if ((got & want) == want) break;
                }
                if ((got & want) != want)
                    for (; j < e; ++j) {
                        got |= __ldcg(front + bw.adj[j]);
                        if ((got & want) == want) break;
                    }
                const uint64_t nb = got & want;
                if (nb) {
                    k.next[v] = nb;
                    k.seen[v] = s | nb;
                    write_levels(k.level, v, nb, L);
                    const unsigned c = __popcll(nb);
                    acc.pairs += c;
                    acc.medges += (unsigned long long)c * (unsigned long long)outdeg[v];
                    on = true;
                }
            }
        }
        queue_push(on, v, acc.s_buf, acc.n, out, RowLen{outdeg}, cnt);
    }
}

// Bottom-up, warp per vertex (medium bin): 32 in-neighbours first, since most vertices of a large level
// find their lanes among them, then 128 a round. Bound by the rounds' two dependent accesses (row, masks): with
// one entry a lane throughout and 32 a round, 64 sources on the 4.8M-vertex R-MAT of the benchmark took 1.64 ms
// here and 1.27 ms in bu_ctas of 4.4 ms a call; with four a lane the call takes 3.35 ms.
__device__ __forceinline__ void bu_warps(const int32_t* ids, int64_t n, int64_t warp, int64_t nwarps, const CSRView& bw,
                                         const LevelMasks& k, uint64_t all, const int32_t* outdeg, int32_t L,
                                         const Queue& out, unsigned long long* cnt, LevelAcc& acc) {
    const int lane = lane_id();
    const unsigned long long* front = (const unsigned long long*)k.front;
    for (int64_t i = warp; i < n; i += nwarps) {
        const int32_t v = ids[i];
        const uint64_t s = __ldcg((const unsigned long long*)k.seen + v);
        const uint64_t want = all & ~s;
        uint64_t nb = 0;
        if (want) {
            uint64_t got = 0;
            const int64_t b = bw.beg[v], e = b + bw.deg[v];
            got = warp_or_u64(b + lane < e ? __ldcg(front + bw.adj[b + lane]) : 0ull);
            for (int64_t j0 = b + 32; j0 < e && (got & want) != want; j0 += 128)
                got |= warp_or_u64(four_fronts(front, bw.adj, j0 + 4 * lane, e));
            nb = got & want;
        }
        if (lane == 0 && nb) {
            k.next[v] = nb;
            k.seen[v] = s | nb;
            const unsigned c = __popcll(nb);
            acc.pairs += c;
            acc.medges += (unsigned long long)c * (unsigned long long)outdeg[v];
        }
        queue_push(lane == 0 && nb != 0, v, acc.s_buf, acc.n, out, RowLen{outdeg}, cnt);
        write_levels_warp(k.level, v, nb, L);
    }
}

// Bottom-up, CTA per vertex (large bin; block-uniform call), four entries a thread and round.
__device__ __forceinline__ void bu_ctas(const int32_t* ids, int64_t n, const CSRView& bw, const LevelMasks& k,
                                        uint64_t all, const int32_t* outdeg, int32_t L, const Queue& out,
                                        unsigned long long* cnt, LevelAcc& acc, unsigned long long* s_acc) {
    const unsigned long long* front = (const unsigned long long*)k.front;
    for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
        const int32_t v = ids[i];
        const uint64_t s = __ldcg((const unsigned long long*)k.seen + v);
        const uint64_t want = all & ~s;
        if (threadIdx.x == 0) *s_acc = 0;
        __syncthreads();
        if (want) {
            const int64_t b = bw.beg[v], e = b + bw.deg[v];
            for (int64_t j0 = b; j0 < e; j0 += 4 * (int64_t)blockDim.x) {
                const uint64_t a = warp_or_u64(four_fronts(front, bw.adj, j0 + 4 * threadIdx.x, e));
                if (lane_id() == 0 && (a & want)) atomicOr(s_acc, (unsigned long long)(a & want));
                __syncthreads();
                const bool done = (*s_acc & want) == want;
                __syncthreads();
                if (done) break;
            }
        }
        const uint64_t nb = *s_acc & want;
        if (threadIdx.x == 0 && nb) {
            k.next[v] = nb;
            k.seen[v] = s | nb;
            const unsigned c = __popcll(nb);
            acc.pairs += c;
            acc.medges += (unsigned long long)c * (unsigned long long)outdeg[v];
        }
        if (threadIdx.x < 32) {
            queue_push(threadIdx.x == 0 && nb != 0, v, acc.s_buf, acc.n, out, RowLen{outdeg}, cnt);
            write_levels_warp(k.level, v, nb, L);
        }
        __syncthreads();
    }
}

// ---- Persistent levels -------------------------------------------------------------------------
// Driven from the host, every level costs launches and a synchronization. One cooperative launch
// (a CTA of 1,024 threads per SM) runs level after level instead, its CTAs meeting at one grid
// barrier per level: the frontier's masks rotate over three arrays and its queues over three, so a
// level reads one, fills the second and clears the third (the level before last), and no CTA touches
// what another still reads. It takes the direction itself (the fixed switch or the network, every
// CTA from the same counters) and hands back to the host when the frontier outgrows it: above
// kPersistMaxEdges out-edges, or bottom-up on a graph of more than kPersistBuMaxV vertices, the
// host's launches (full occupancy) take the level. Data that other CTAs write during the launch is
// read with ld.cg, past the SMs' incoherent L1; every barrier wait is bounded and sets an error flag
// when it runs out.
// Bound by latency: a level is a chain of about eight dependent L2 accesses and the barrier, about
// 10 us on a lattice. (64 registers a thread, the most that 1,024 threads have: 56 bytes of stores and 144 of loads
// spill.) Before, a level was two phases (expand, commit) with a barrier of eight CTAs
// per SM after each and a warp took 32 frontier vertices whatever the frontier's size: 64 sources on
// a 4.8M-vertex R-MAT 11.4 ms a call, now 5.1 ms; 37 sets on 0.78M vertices 3.0 -> 0.89 ms; 8 sources
// on a 701 x 701 lattice 29.3 -> 10.4 ms (11.4 before the barrier's one-way arrival, the first look
// by interpolation and the degree loaded beside the claim); one source on 4,096 vertices 317 -> 145 us.
constexpr int kPersistThreads = 1024;
constexpr int kPersistWarps = kPersistThreads / 32;
constexpr int64_t kPersistMaxEdges = 1ll << 22;   // a frontier's out-edges
constexpr int64_t kPersistBuMaxV = 1ll << 20;     // vertices of a graph whose bottom-up levels stay inside
constexpr int kPersistMaxLevels = 1 << 23;        // of one launch (its barrier's counter is 32 bits wide)
constexpr int kPersistTrace = 8192;               // schedule decisions recorded per launch
constexpr int kPersistTraceEager = 64;            // ... of which this many are read with the counters

// Device words of one call: the host levels' counters (C_*), the launch's control words, its counter
// slots (one per level, reused every third level), the barrier's counter on its own 128-byte line,
// then the trace (per decision: frontier vertices, out-edges, unexplored out-edges, direction bits).
enum { P_LEVELS = 16, P_REASON, P_DIR, P_EDGES, P_REACHED, P_MF, P_NF, P_MU, P_ROT, P_ERR, P_BU, P_SLOTS = 32 };
enum { S_Q = 0, S_PAIRS, S_MEDGES, S_W = 4 };
enum { R_DONE = 0, R_BOTTOM_UP = 1, R_BIG = 2, R_LIMIT = 3 };
constexpr int kCtlBarrier = 48;
constexpr int kCtlTrace = 96;
constexpr int kTraceW = 4;

struct PersistArgs {
    CSRView fw, bw;
    uint64_t* seen;
    uint64_t* front[3];       // the frontier's masks, the next frontier's (zero) and the last one's (zero)
    Queue q[3];               // frontier, next frontier, last frontier (empty)
    Levels level;
    const int32_t* bins;
    int64_t bin_n[3];
    int64_t V;
    uint64_t all;
    double E, mu0, alpha, beta;  // mu0: unexplored out-edges per lane before this frontier's
    int lanes, L0, max_levels, dir0;
    int fixed_dir;            // 0: the schedule decides; 1: top-down throughout (graphs below 4,096 vertices)
    int count_first;          // the first frontier (the sources) belongs in the sums
    int dir_given;            // the first level's direction is already decided (dir0)
    int bu_inside;            // bottom-up levels run inside the launch
    const float* net;         // schedule network parameters, or null for the fixed switch
    unsigned long long* ctl;
};

__device__ __forceinline__ unsigned long long ldcg_u64(const unsigned long long* p) { return __ldcg(p); }

__global__ void __launch_bounds__(kPersistThreads, 1) k_bfs_persistent(PersistArgs a) {
    __shared__ int32_t s_stage[kPersistWarps][kStage];
    __shared__ LevelShared<kPersistWarps> sh;
    __shared__ unsigned long long s_acc;
    __shared__ int s_dir;
    unsigned long long* err = a.ctl + P_ERR;
    unsigned int* bar = reinterpret_cast<unsigned int*>(a.ctl + kCtlBarrier);
    double* trace = reinterpret_cast<double*>(a.ctl + kCtlTrace);
    const int wib = threadIdx.x >> 5;
    // (warps numbered across the CTAs first, so that a short frontier spreads over the SMs)
    const int64_t warp = (int64_t)wib * gridDim.x + blockIdx.x, nwarps = (int64_t)gridDim.x * kPersistWarps;
    const int64_t tid = blockIdx.x * (int64_t)kPersistThreads + threadIdx.x, nthreads = (int64_t)gridDim.x * kPersistThreads;
    int reason = R_LIMIT, dir = a.dir0, lev = 0, rot = 0, n_bu = 0;
    unsigned long long packed = ldcg_u64(a.ctl + C_Q);
    int64_t n_last = 0;
    const unsigned long long pairs0 = ldcg_u64(a.ctl + C_PAIRS), medges0 = ldcg_u64(a.ctl + C_MEDGES);
    double nf = (double)pairs0 / a.lanes, mf = (double)medges0 / a.lanes, mu = a.mu0 - mf;
    unsigned long long edges = a.count_first ? medges0 : 0, reached = a.count_first ? pairs0 : 0;
    unsigned long long pr = pairs0, me = medges0;
    unsigned met = 0;
    for (lev = 0; lev < a.max_levels; ++lev) {
        const int64_t nq = (int64_t)(packed >> kQShift), vedges = (int64_t)(packed & kQEdges);
        if (nq == 0) { reason = R_DONE; break; }
        if (!a.fixed_dir && !(lev == 0 && a.dir_given)) {
            const int before = dir;
            if (a.net) {
                if (threadIdx.x < 32) {  // (every CTA computes the same decision from the same counters)
                    const int d = sched_net::decide_direction_warp(a.net, (double)a.V, a.E, nf, mf, mu, dir, a.lanes,
                                                                   a.alpha, a.beta);
                    if (threadIdx.x == 0) s_dir = d;
                }
                __syncthreads();
                dir = s_dir;
            } else {
                dir = sched_net::fixed_direction((double)a.V, nf, mf, mu, dir, a.alpha, a.beta);
            }
            if (tid == 0 && lev < kPersistTrace) {
                double* t = trace + kTraceW * lev;
                t[0] = nf;
                t[1] = mf;
                t[2] = mu;
                t[3] = (double)(dir | before << 1);
            }
        }
        if (dir && !a.bu_inside) { reason = R_BOTTOM_UP; break; }
        if (!dir && vedges > kPersistMaxEdges) { reason = R_BIG; break; }
        unsigned long long* sl = a.ctl + P_SLOTS + S_W * (lev % 3);
        const Queue &qa = a.q[rot], &qb = a.q[(rot + 1) % 3], &qc = a.q[(rot + 2) % 3];
        LevelMasks k{a.front[rot], a.seen, a.front[(rot + 1) % 3], a.level};
        uint64_t* old = a.front[(rot + 2) % 3];
        // (the slot after this level's was last read before the barrier of the level before)
        if (blockIdx.x == 0 && threadIdx.x < S_W) a.ctl[P_SLOTS + S_W * ((lev + 1) % 3) + threadIdx.x] = 0;
        for (int64_t i = tid; i < n_last; i += nthreads) old[__ldcg(qc.v + i)] = 0;
        LevelAcc acc;
        acc.s_buf = s_stage[wib];
        const int32_t L = a.L0 + lev + 1;
        if (!dir) {
            TopDown op{a.fw, k, L, 0, 0};
            walk_level(qa, nq, vedges, warp, nwarps, op, qb, &sl[S_Q], acc.s_buf, acc.n);
            acc.pairs = op.pairs;
            acc.medges = op.medges;
        } else {
            bu_ctas(a.bins + a.bin_n[0] + a.bin_n[1], a.bin_n[2], a.bw, k, a.all, a.fw.deg, L, qb, &sl[S_Q], acc, &s_acc);
            bu_warps(a.bins + a.bin_n[0], a.bin_n[1], warp, nwarps, a.bw, k, a.all, a.fw.deg, L, qb, &sl[S_Q], acc);
            bu_threads(a.bins, a.bin_n[0], warp * 32, nwarps * 32, a.bw, k, a.all, a.fw.deg, L, qb, &sl[S_Q], acc);
            ++n_bu;
        }
        block_publish<kPersistWarps>(sh, acc.s_buf, acc.n, qb, RowLen{a.fw.deg}, &sl[S_Q], acc.pairs, acc.medges,
                                     &sl[S_PAIRS]);
        if (!grid_barrier(bar, err, met)) break;
        n_last = nq;
        packed = ldcg_u64(&sl[S_Q]);
        pr = ldcg_u64(&sl[S_PAIRS]);
        me = ldcg_u64(&sl[S_MEDGES]);
        nf = (double)pr / a.lanes;
        mf = (double)me / a.lanes;
        mu -= mf;
        edges += me;
        reached += pr;
        rot = (rot + 1) % 3;
    }
    // the last frontier's masks are cleared for the host's levels
    for (int64_t i = tid; i < n_last; i += nthreads) a.front[(rot + 2) % 3][__ldcg(a.q[(rot + 2) % 3].v + i)] = 0;
    if (tid == 0) {
        a.ctl[P_LEVELS] = (unsigned long long)lev;
        a.ctl[C_Q] = packed;  // (where a following launch starts from)
        a.ctl[C_PAIRS] = pr;
        a.ctl[C_MEDGES] = me;
        a.ctl[P_REASON] = (unsigned long long)reason;
        a.ctl[P_DIR] = (unsigned long long)dir;
        a.ctl[P_EDGES] = edges;
        a.ctl[P_REACHED] = reached;
        a.ctl[P_MF] = (unsigned long long)__double_as_longlong(mf);
        a.ctl[P_NF] = (unsigned long long)__double_as_longlong(nf);
        a.ctl[P_MU] = (unsigned long long)__double_as_longlong(mu);
        a.ctl[P_ROT] = (unsigned long long)rot;
        a.ctl[P_BU] = (unsigned long long)n_bu;
    }
}

// ---- Levels launched from the host -------------------------------------------------------------

__device__ __forceinline__ void level_end(LevelAcc& acc, const Queue& out, const int32_t* outdeg,
                                          unsigned long long* cnt) {
    queue_flush(acc.s_buf, acc.n, out, RowLen{outdeg}, &cnt[C_Q]);
    warp_add_u64(&cnt[C_PAIRS], acc.pairs);
    warp_add_u64(&cnt[C_MEDGES], acc.medges);
}

__global__ void __launch_bounds__(kBlock) k_td_level(Queue q, int64_t nq, int64_t total, CSRView fw, LevelMasks k, int32_t L,
                                                     Queue out, unsigned long long* cnt) {
    __shared__ int32_t s_stage[kBlock / 32][kStage];
    LevelAcc acc;
    acc.s_buf = s_stage[threadIdx.x >> 5];
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    TopDown op{fw, k, L, 0, 0};
    walk_level(q, nq, total, warp, ((int64_t)gridDim.x * blockDim.x) >> 5, op, out, &cnt[C_Q], acc.s_buf, acc.n);
    acc.pairs = op.pairs;
    acc.medges = op.medges;
    level_end(acc, out, fw.deg, cnt);
}

__global__ void k_clear_front(const int32_t* q, int64_t nq, uint64_t* front) {
    GRID_STRIDE(i, nq) front[q[i]] = 0;
}

__global__ void k_bu_thread(const int32_t* ids, int64_t n, CSRView bw, LevelMasks k, uint64_t all, const int32_t* outdeg,
                            int32_t L, Queue out, unsigned long long* cnt) {
    __shared__ int32_t s_stage[kBlock / 32][kStage];
    LevelAcc acc;
    acc.s_buf = s_stage[threadIdx.x >> 5];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    bu_threads(ids, n, (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~(int64_t)31, stride, bw, k, all, outdeg, L, out,
               &cnt[C_Q], acc);
    level_end(acc, out, outdeg, cnt);
}

__global__ void k_bu_warp(const int32_t* ids, int64_t n, CSRView bw, LevelMasks k, uint64_t all, const int32_t* outdeg,
                          int32_t L, Queue out, unsigned long long* cnt) {
    __shared__ int32_t s_stage[kBlock / 32][kStage];
    LevelAcc acc;
    acc.s_buf = s_stage[threadIdx.x >> 5];
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    bu_warps(ids, n, warp, ((int64_t)gridDim.x * blockDim.x) >> 5, bw, k, all, outdeg, L, out, &cnt[C_Q], acc);
    level_end(acc, out, outdeg, cnt);
}

__global__ void k_bu_cta(const int32_t* ids, int64_t n, CSRView bw, LevelMasks k, uint64_t all, const int32_t* outdeg,
                         int32_t L, Queue out, unsigned long long* cnt) {
    __shared__ int32_t s_stage[kBlock / 32][kStage];
    __shared__ unsigned long long s_acc;
    LevelAcc acc;
    acc.s_buf = s_stage[threadIdx.x >> 5];
    bu_ctas(ids, n, bw, k, all, outdeg, L, out, &cnt[C_Q], acc, &s_acc);
    level_end(acc, out, outdeg, cnt);
}

}  // namespace

int bfs_run(gir_dev* g, const int64_t* set_beg_h, const int32_t* srcs_d, int64_t n_sets, int32_t* level_d) {
    const int64_t V = g->V;
    QueryStats& st = g->qstats;
    st = QueryStats{};
    g->trace_x.clear();
    g->trace_y.clear();
    if (n_sets <= 0 || V == 0) return GIR_OK;
    if (!g->bins_valid) GIR_TRY(store_build_bins(g));

    uint64_t *seen = nullptr, *front[3] = {nullptr, nullptr, nullptr};
    Queue q[3];
    int64_t* sbeg = nullptr;
    unsigned long long* ctl = nullptr;
    GIR_TRY(ensure_n(g, g->scratch[0], V, &seen));
    GIR_TRY(ensure_n(g, g->scratch[1], V, &front[0]));
    GIR_TRY(ensure_n(g, g->scratch[2], V, &front[1]));
    GIR_TRY(ensure_n(g, g->scratch[8], V, &front[2]));
    const int q_slots[3] = {3, 4, 9}, off_slots[3] = {5, 7, 11};
    for (int i = 0; i < 3; ++i) {
        GIR_TRY(ensure_n(g, g->scratch[q_slots[i]], V + 1, &q[i].v));
        GIR_TRY(ensure_n(g, g->scratch[off_slots[i]], V + 1, &q[i].off));
    }
    GIR_TRY(ensure_n(g, g->scratch[6], 65, &sbeg));
    GIR_TRY(ensure_n(g, g->scratch[10], kCtlTrace + kTraceW * kPersistTrace, &ctl));
    unsigned long long* cnt = ctl;
    constexpr size_t kRead = sizeof(unsigned long long) * (kCtlTrace + kTraceW * kPersistTraceEager);
    static_assert(kRead <= kPinnedBytes, "the handle's pinned buffer holds the counters and the eager trace");
    unsigned long long* hc = nullptr;
    {
        void* h = nullptr;
        GIR_TRY(pinned(g, kPinnedBytes, &h));
        hc = static_cast<unsigned long long*>(h);
    }
    const double alpha = g->params[GIR_PARAM_ALPHA], beta = g->params[GIR_PARAM_BETA];
    const int64_t E = g->fw.E;
    const int grid = g->num_sms * (int)g->params[GIR_PARAM_CTAS_PER_SM];
    // persistent levels (the device must take cooperative launches)
    int persist_grid = 0;
    {
        int per_sm = 0;
        GIR_TRY(cooperative_ctas(g, (const void*)k_bfs_persistent, kPersistThreads, &per_sm));
        if (per_sm > 0) persist_grid = g->num_sms;
    }
    const bool learned = g->schedule == GIR_SCHEDULE_LEARNED && g->sched_loaded && V >= 4096;
    // Bit planes, for the groups of lanes that want them (the first group is the widest). Decided once a call:
    // an allocation that fails has synchronized the stream and trimmed the pool by then.
    auto wants_planes = [&](int64_t lanes) { return lanes >= kPlaneMinLanes && lanes * V >= kPlaneMinPairs; };
    unsigned long long* plane = nullptr;
    if (wants_planes(std::min<int64_t>(n_sets, 64)) && set_beg_h[n_sets] > set_beg_h[0]) {
        const std::string err = g->err;
        const int rc = ensure_n(g, g->scratch[12], 4 * V, &plane);
        if (rc == GIR_ERR_OOM) g->err = err;  // (the straight writes need no memory: not this call's error)
        else GIR_TRY(rc);
    }
    std::vector<double> trace_rows;
    MainTimer timer{g, g->params[GIR_PARAM_PROFILE] != 0.0};
    GIR_CUDA(g, cudaEventRecord(g->ev0, g->stream));

    for (int64_t g0 = 0; g0 < n_sets; g0 += 64) {
        const int nl = (int)((n_sets - g0) < 64 ? (n_sets - g0) : 64);
        const uint64_t all = nl == 64 ? ~0ull : ((1ull << nl) - 1);
        Levels level{level_d + g0 * V, V, nullptr};
        GIR_CUDA(g, cudaMemsetAsync(seen, 0, sizeof(uint64_t) * V, g->stream));
        for (uint64_t* f : front) GIR_CUDA(g, cudaMemsetAsync(f, 0, sizeof(uint64_t) * V, g->stream));
        GIR_CUDA(g, cudaMemsetAsync(ctl, 0, sizeof(unsigned long long) * kCtlTrace, g->stream));
        GIR_CUDA(g, cudaMemcpyAsync(sbeg, set_beg_h + g0, sizeof(int64_t) * (nl + 1), cudaMemcpyHostToDevice, g->stream));
        const int64_t n_entries = set_beg_h[g0 + nl] - set_beg_h[g0];
        if (n_entries > 0 && wants_planes(nl)) level.plane = plane;
        if (level.plane) {
            GIR_CUDA(g, cudaMemsetAsync(level.plane, 0, sizeof(uint64_t) * 4 * V, g->stream));
        } else {
            GIR_CUDA(g, cudaMemsetAsync(level.out, 0xff, sizeof(int32_t) * V * nl, g->stream));
        }
        if (n_entries == 0) continue;
        k_init_sources<<<grid_for(g, n_entries, kBlock), kBlock, 0, g->stream>>>(sbeg, nl, srcs_d, V, seen, front[0], q[0],
                                                                                cnt, level, g->fw.deg);
        GIR_LAUNCH(g, "k_init_sources");
        st.launches++;
        auto read = [&]() -> int {
            GIR_CUDA(g, cudaMemcpyAsync(hc, ctl, kRead, cudaMemcpyDeviceToHost, g->stream));
            GIR_CUDA(g, cudaStreamSynchronize(g->stream));
            return GIR_OK;
        };
        int64_t nq = 0, vedges = 0;                // the frontier: vertices and their out-edges
        double mf = 0, nf = 0, mu = (double)E;     // per lane: its out-edges, vertices, and out-edges left
        auto take_counters = [&]() {
            nq = (int64_t)(hc[C_Q] >> kQShift);
            vedges = (int64_t)(hc[C_Q] & kQEdges);
            mf = (double)hc[C_MEDGES] / nl;
            nf = (double)hc[C_PAIRS] / nl;
            mu -= mf;
            st.edges += (int64_t)hc[C_MEDGES];
            st.reached += (int64_t)hc[C_PAIRS];
        };
        bool bottom_up = false, handed_back = false, fresh = true;  // fresh: the counters were not read yet
        int pending = -1;  // a direction already decided for this level
        int32_t L = 0;
        if (persist_grid == 0) {
            if (learned)
                GIR_TRY(sched_bfs_decide_async(g, cnt, C_PAIRS, C_MEDGES, C_DIR, C_FEAT, nl, mu, false, alpha, beta));
            GIR_TRY(read());
            take_counters();
            fresh = false;
        }
        while (fresh || nq > 0) {
            // direction (the reference's switch, gir_query.cpp:159-169, or the schedule network)
            if (fresh) {
                // (the sources' level: the launch decides from the counters on the device)
            } else if (pending >= 0) {
                bottom_up = pending != 0;
                pending = -1;
            } else if (learned) {  // decided on the device with the counters just read
                bottom_up = hc[C_DIR] != 0;
                sched_trace(g, reinterpret_cast<const float*>(&hc[C_FEAT]), bottom_up ? 1 : 0);
            } else if (V >= 4096) {
                float feat[GIR_SCHED_IN];
                sched_bfs_features(g, nf, mf, mu, L, bottom_up, nl, feat);
                if (!bottom_up && mf * alpha > mu) bottom_up = true;
                else if (bottom_up && nf * beta < (double)V) bottom_up = false;
                sched_trace(g, feat, bottom_up ? 1 : 0);
            }
            // levels run on the device until the launch hands back
            if (fresh || (persist_grid > 0 && !handed_back && !bottom_up && vedges <= kPersistMaxEdges)) {
                if (!fresh)
                    GIR_CUDA(g, cudaMemsetAsync(ctl + P_LEVELS, 0, sizeof(unsigned long long) * (kCtlTrace - P_LEVELS),
                                                g->stream));
                PersistArgs pa;
                pa.fw = view(g->fw);
                pa.bw = view(g->bw);
                pa.seen = seen;
                for (int i = 0; i < 3; ++i) {
                    pa.front[i] = front[i];
                    pa.q[i] = q[i];
                    pa.bin_n[i] = g->bin_n[i];
                }
                pa.level = level;
                pa.bins = static_cast<const int32_t*>(g->bins.p);
                pa.V = V;
                pa.all = all;
                pa.E = (double)E;
                pa.mu0 = fresh ? mu : mu + mf;
                pa.alpha = alpha;
                pa.beta = beta;
                pa.lanes = nl;
                pa.L0 = L;
                pa.max_levels = kPersistMaxLevels;
                pa.count_first = fresh ? 1 : 0;
                pa.dir0 = bottom_up ? 1 : 0;
                pa.fixed_dir = V < 4096;
                pa.dir_given = !fresh;
                pa.bu_inside = V <= kPersistBuMaxV;
                pa.net = learned ? static_cast<const float*>(g->sched_w.p) : nullptr;
                pa.ctl = ctl;
                void* kargs[] = {&pa};
                GIR_TRY(timer.run([&]() -> int {
                    GIR_CUDA(g, cudaLaunchCooperativeKernel((const void*)k_bfs_persistent, persist_grid, kPersistThreads,
                                                            kargs, 0, g->stream));
                    return GIR_OK;
                }));
                st.launches++;
                GIR_TRY(read());
                if (hc[P_ERR]) return fail(g, GIR_ERR_TIMEOUT, "bfs: the persistent level loop ran out its barrier bound");
                const int64_t lv = (int64_t)hc[P_LEVELS];
                const bool given = pa.dir_given != 0;
                if (!pa.fixed_dir) {  // the schedule decisions taken inside the launch
                    const int64_t n_tr = std::min<int64_t>(lv + (hc[P_REASON] == R_DONE ? 0 : 1), kPersistTrace);
                    const double* rows = reinterpret_cast<const double*>(hc + kCtlTrace);
                    if (n_tr > kPersistTraceEager) {
                        trace_rows.resize((size_t)n_tr * kTraceW);
                        GIR_CUDA(g, cudaMemcpyAsync(trace_rows.data(), ctl + kCtlTrace, sizeof(double) * trace_rows.size(),
                                                    cudaMemcpyDeviceToHost, g->stream));
                        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
                        rows = trace_rows.data();
                    }
                    for (int64_t r = given ? 1 : 0; r < n_tr; ++r) {
                        const double* t = rows + r * kTraceW;
                        float feat[GIR_SCHED_IN];
                        sched_bfs_features(g, t[0], t[1], t[2], 0, ((int)t[3] & 2) != 0, nl, feat);
                        sched_trace(g, feat, (int32_t)t[3] & 1);
                    }
                }
                L += (int32_t)lv;
                st.iterations += lv;
                st.persistent_levels += lv;
                st.bottom_up += (int64_t)hc[P_BU];
                st.edges += (int64_t)hc[P_EDGES];
                st.reached += (int64_t)hc[P_REACHED];
                nq = (int64_t)(hc[C_Q] >> kQShift);
                vedges = (int64_t)(hc[C_Q] & kQEdges);
                std::memcpy(&mf, &hc[P_MF], sizeof(double));
                std::memcpy(&nf, &hc[P_NF], sizeof(double));
                std::memcpy(&mu, &hc[P_MU], sizeof(double));
                for (uint64_t r = hc[P_ROT]; r > 0; --r) {
                    std::rotate(front, front + 1, front + 3);
                    std::rotate(q, q + 1, q + 3);
                }
                pending = (int)hc[P_DIR];
                handed_back = hc[P_REASON] == R_BIG;  // (a big frontier: one level on the host first)
                fresh = false;
                continue;
            }
            handed_back = false;
            GIR_CUDA(g, cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * C_N, g->stream));
            const LevelMasks km{front[0], seen, front[1], level};
            if (!bottom_up) {
                const int64_t blocks = std::min<int64_t>((vedges / 32 + kBlock / 32) / (kBlock / 32), g->num_sms * 8);
                GIR_TRY(timer.run([&]() -> int {
                    k_td_level<<<(int)blocks, kBlock, 0, g->stream>>>(q[0], nq, vedges, view(g->fw), km, L + 1, q[1], cnt);
                    GIR_LAUNCH(g, "k_td_level");
                    return GIR_OK;
                }));
                st.launches++;
            } else {
                const int32_t* bins = static_cast<const int32_t*>(g->bins.p);
                GIR_TRY(timer.run([&]() -> int {
                    if (g->bin_n[0] > 0) {
                        k_bu_thread<<<grid_for(g, g->bin_n[0], kBlock), kBlock, 0, g->stream>>>(
                            bins, g->bin_n[0], view(g->bw), km, all, g->fw.deg, L + 1, q[1], cnt);
                        GIR_LAUNCH(g, "k_bu_thread");
                        st.launches++;
                    }
                    if (g->bin_n[1] > 0) {
                        k_bu_warp<<<grid_for(g, g->bin_n[1] * 32, kBlock), kBlock, 0, g->stream>>>(
                            bins + g->bin_n[0], g->bin_n[1], view(g->bw), km, all, g->fw.deg, L + 1, q[1], cnt);
                        GIR_LAUNCH(g, "k_bu_warp");
                        st.launches++;
                    }
                    if (g->bin_n[2] > 0) {
                        const int64_t b = g->bin_n[2] < grid ? g->bin_n[2] : grid;
                        k_bu_cta<<<(int)b, kBlock, 0, g->stream>>>(bins + g->bin_n[0] + g->bin_n[1], g->bin_n[2],
                                                                   view(g->bw), km, all, g->fw.deg, L + 1, q[1], cnt);
                        GIR_LAUNCH(g, "k_bu_cta");
                        st.launches++;
                    }
                    return GIR_OK;
                }));
                st.bottom_up++;
            }
            // the frontier's masks become the next level's empty ones
            if (nq * 8 < V) {
                k_clear_front<<<grid_for(g, nq, kBlock), kBlock, 0, g->stream>>>(q[0].v, nq, front[0]);
                GIR_LAUNCH(g, "k_clear_front");
                st.launches++;
            } else {
                GIR_CUDA(g, cudaMemsetAsync(front[0], 0, sizeof(uint64_t) * V, g->stream));
            }
            std::swap(front[0], front[1]);
            std::swap(q[0], q[1]);
            if (learned)
                GIR_TRY(sched_bfs_decide_async(g, cnt, C_PAIRS, C_MEDGES, C_DIR, C_FEAT, nl, mu, bottom_up, alpha, beta));
            GIR_TRY(read());
            take_counters();
            ++L;
            st.iterations++;
        }
        if (level.plane) {
            k_expand_levels<<<grid_for(g, V, kBlock), kBlock, 0, g->stream>>>(level, seen, nl);
            GIR_LAUNCH(g, "k_expand_levels");
            st.launches++;
        }
    }
    GIR_CUDA(g, cudaEventRecord(g->ev1, g->stream));
    GIR_CUDA(g, cudaEventSynchronize(g->ev1));
    float ms = 0;
    GIR_CUDA(g, cudaEventElapsedTime(&ms, g->ev0, g->ev1));
    st.kernel_ms = ms;
    return GIR_OK;
}

}  // namespace gir
