// Level-synchronous frontiers shared by the BFS levels, the two-way reach of the SCC build and the
// spanning forest of the block build: a queue whose entries carry their edge offsets, the
// edge-balanced walk of its rows, and the end of a level inside a cooperative launch.
#pragma once

#include "common.cuh"

namespace gir {

#ifdef __CUDACC__

// A frontier queue is two arrays: the entries and, for each, the number of row entries of the entries
// before it. Appends reserve both at once by one atomicAdd of (entries << 33 | row entries), so the
// offsets ascend with the slots and the next level can cut the frontier's rows into equal runs
// without a scan pass (a level has below 2^31 entries and below 2^33 row entries).
constexpr int kQShift = 33;
constexpr unsigned long long kQEdges = (1ull << kQShift) - 1;

struct Queue {
    int32_t* v;
    uint64_t* off;
};

__device__ __forceinline__ uint64_t warp_incl_u64(uint64_t x) {
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane_id() >= o) x += t;
    }
    return x;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x) {
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Writes a warp's s_n staged entries to the queue from slot `slot` and edge offset `e0` on; deg(e) is
// the row length of entry e.
template <class Deg>
__device__ __forceinline__ void queue_write(const int32_t* s_buf, int s_n, const Queue& q, const Deg& deg,
                                            unsigned long long slot, uint64_t e0) {
    for (int b = 0; b < s_n; b += 32) {
        const int i = b + lane_id();
        const int32_t v = i < s_n ? s_buf[i] : 0;
        const uint64_t d = i < s_n ? (uint64_t)deg(v) : 0ull;
        const uint64_t incl = warp_incl_u64(d);
        if (i < s_n) {
            q.v[slot + i] = v;
            q.off[slot + i] = e0 + incl - d;
        }
        e0 += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// Row entries of a warp's staged queue entries (warp-uniform result).
template <class Deg>
__device__ __forceinline__ uint64_t staged_edges(const int32_t* s_buf, int s_n, const Deg& deg) {
    uint64_t e = 0;
    for (int i = lane_id(); i < s_n; i += 32) e += (uint64_t)deg(s_buf[i]);
    return warp_sum_u64(e);
}

template <class Deg>
__device__ __forceinline__ void queue_flush(int32_t* s_buf, int& s_n, const Queue& q, const Deg& deg,
                                            unsigned long long* cnt) {
    if (s_n == 0) return;
    const uint64_t e = staged_edges(s_buf, s_n, deg);
    unsigned long long at = 0;
    if (lane_id() == 0) at = atomicAdd(cnt, ((unsigned long long)s_n << kQShift) | e);
    at = __shfl_sync(0xffffffffu, at, 0);
    queue_write(s_buf, s_n, q, deg, at >> kQShift, at & kQEdges);
    __syncwarp();
    s_n = 0;
}

// Staged append (warp-uniform call): collects in shared memory, one reservation per kSlots entries.
template <int kSlots = kStage, class Deg>
__device__ __forceinline__ void queue_push(bool pred, int32_t v, int32_t* s_buf, int& s_n, const Queue& q, const Deg& deg,
                                           unsigned long long* cnt) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    const int k = __popc(m);
    if (s_n + k > kSlots) queue_flush(s_buf, s_n, q, deg, cnt);
    if (pred) s_buf[s_n + __popc(m & ((1u << lane_id()) - 1))] = v;
    __syncwarp();
    s_n += k;
}

// End of a level inside a cooperative launch (block-uniform call): the CTA's staged entries go out
// with one reservation, and its warps' two sums with one atomicAdd each (sums may be null).
template <int kWarps>
struct LevelShared {
    unsigned long long sum[kWarps][2];
    uint64_t e[kWarps];
    uint32_t n[kWarps];
    unsigned long long base;
};
template <int kWarps, class Deg>
__device__ __forceinline__ void block_publish(LevelShared<kWarps>& sh, const int32_t* s_buf, int s_n, const Queue& q,
                                              const Deg& deg, unsigned long long* cnt, unsigned long long sum0 = 0,
                                              unsigned long long sum1 = 0, unsigned long long* sums = nullptr) {
    static_assert(kWarps == 32, "one lane of the first warp per warp of the CTA");
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    const uint64_t e_w = staged_edges(s_buf, s_n, deg);
    if (sums) {
        sum0 = warp_sum_u64(sum0);
        sum1 = warp_sum_u64(sum1);
    }
    if (lane == 0) {
        sh.sum[wib][0] = sum0;
        sh.sum[wib][1] = sum1;
        sh.n[wib] = (uint32_t)s_n;
        sh.e[wib] = e_w;
    }
    __syncthreads();
    if (wib == 0) {
        const uint32_t n = sh.n[lane];
        const uint64_t e = sh.e[lane];
        const uint64_t n_in = warp_incl_u64(n), e_in = warp_incl_u64(e);
        sh.n[lane] = (uint32_t)n_in - n;
        sh.e[lane] = e_in - e;
        if (lane == 31) sh.base = n_in ? atomicAdd(cnt, ((unsigned long long)n_in << kQShift) | e_in) : 0ull;
        if (sums) {
            sum0 = warp_sum_u64(sh.sum[lane][0]);
            sum1 = warp_sum_u64(sh.sum[lane][1]);
            if (lane == 0 && sum0) atomicAdd(&sums[0], sum0);
            if (lane == 0 && sum1) atomicAdd(&sums[1], sum1);
        }
    }
    __syncthreads();
    if (s_n) {
        const unsigned long long at = sh.base;
        queue_write(s_buf, s_n, q, deg, (at >> kQShift) + sh.n[wib], (at & kQEdges) + sh.e[wib]);
    }
}

// Largest i in [lo, n) with off[i] <= key (off[lo] <= key): one warp, 32 probes a round.
__device__ __forceinline__ int64_t queue_find(const uint64_t* off, int64_t lo, int64_t n, uint64_t key) {
    int64_t hi = n - 1;
    while (hi > lo) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t i = lo + (int64_t)(lane_id() + 1) * step;
        const bool c = i <= hi && __ldcg((const unsigned long long*)off + i) <= key;
        const int t = __popc(__ballot_sync(0xffffffffu, c));
        if (t > 0) lo += (int64_t)t * step;
        hi = lo + step - 1 < hi ? lo + step - 1 : hi;
    }
    return lo;
}
// The same over the whole queue of n entries and `total` row positions, from a first look at the 32
// entries about where the key would be if all rows were alike: one round instead of three where they
// nearly are (a road network).
__device__ __forceinline__ int64_t queue_guess(const uint64_t* off, int64_t n, int64_t total, int64_t key) {
    int64_t at = (int64_t)((float)key / (float)total * (float)n) - 16;
    at = at + 32 > n ? n - 32 : at;
    at = at < 0 ? 0 : at;
    const int64_t i = at + lane_id();
    const unsigned m =
        __ballot_sync(0xffffffffu, i < n && (int64_t)__ldcg((const unsigned long long*)off + i) <= key);
    if (m == 0) return queue_find(off, 0, at, (uint64_t)key);
    if (m == 0xffffffffu && at + 32 < n) return queue_find(off, at + 31, n, (uint64_t)key);
    return at + __popc(m) - 1;
}

// Visits the row positions [c0, c1) of the frontier (as the queue's offsets count them), by one warp;
// i0 is the largest entry whose offset is at most c0, and c1 - c0 is below 2^31. A warp holds 32 queue
// entries in registers (one load each) and finds a position's entry by shuffles; two positions a
// thread keep two rows of dependent loads in flight. The operation:
//   op.row(entry, beg, pay)    first index of the entry's row, and 64 bits that go with it
//   op.adj(index, pay)         the neighbour at an index of the row (>= 0); may change its copy of pay
//   op.want(w, pay)            the bits the neighbour may take (0: none); a plain read
//   op.apply(w, pay, bits, e)  takes them by an atomic; true when e joins the next queue
//   op.deg(entry)              row length
template <class Op>
__device__ __forceinline__ void walk_rows(const Queue& q, int64_t nq, int64_t total, int64_t c0, int64_t c1, int64_t i0,
                                          Op& op, const Queue& out, unsigned long long* cnt, int32_t* s_buf, int& s_n) {
    constexpr int U = 2;
    const int ln = lane_id();
    int64_t p = c0;
    while (p < c1) {
        const int64_t ij = i0 + ln;
        uint32_t relj = 0xffffffffu;  // the entry's offset from c0 (an entry that starts before c0: 0)
        int64_t begj = 0;             // its row's first index, less that offset
        unsigned long long payj = 0;
        if (ij < nq) {
            const int32_t e = __ldcg(q.v + ij);
            const int64_t off = (int64_t)__ldcg((const unsigned long long*)q.off + ij) - c0;
            relj = off <= 0 ? 0u : (off < 0x7fffffff ? (uint32_t)off : 0x7fffffffu);
            op.row(e, begj, payj);
            begj -= off;
        }
        const int64_t wnext = i0 + 32 < nq ? (int64_t)__ldcg((const unsigned long long*)q.off + i0 + 32) : total;
        const int64_t wend = wnext < c1 ? wnext : c1;
        for (; p < wend; p += 32 * U) {
            int32_t w[U];
            unsigned long long pay[U], bits[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
                const int64_t pos = p + j * 32 + ln;
                const uint32_t rel = (uint32_t)(pos - c0);
                int x = 0;  // largest window entry with offset <= pos (entries without a row share an offset)
#pragma unroll
                for (int b = 16; b; b >>= 1)
                    if (__shfl_sync(0xffffffffu, relj, x + b) <= rel) x += b;
                const int64_t bx = __shfl_sync(0xffffffffu, begj, x);
                pay[j] = __shfl_sync(0xffffffffu, payj, x);
                w[j] = -1;
                if (pos < wend) w[j] = op.adj(bx + rel, pay[j]);
            }
#pragma unroll
            for (int j = 0; j < U; ++j) bits[j] = w[j] >= 0 ? op.want(w[j], pay[j]) : 0ull;
#pragma unroll
            for (int j = 0; j < U; ++j) {
                bool push = false;
                int32_t e = 0;
                if (bits[j]) push = op.apply(w[j], pay[j], bits[j], e);
                queue_push(push, e, s_buf, s_n, out, [&](int32_t x) { return op.deg(x); }, cnt);
            }
        }
        p = wend;
        i0 += 32;
        // (entries without a row keep their slots: jump past a run of them)
        if (p < c1 && i0 + 32 < nq && (int64_t)__ldcg((const unsigned long long*)q.off + i0 + 32) <= p)
            i0 = queue_find(q.off, i0 + 32, nq, (uint64_t)p);
    }
}

// One level's share of a warp: equal runs of the frontier's row positions, at most kRun long, so that
// a short frontier still spreads over every warp.
constexpr int64_t kRun = 32 * 16;
template <class Op>
__device__ __forceinline__ void walk_level(const Queue& q, int64_t nq, int64_t total, int64_t warp, int64_t nwarps,
                                           Op& op, const Queue& out, unsigned long long* cnt, int32_t* s_buf, int& s_n) {
    int64_t run = ((total + nwarps - 1) / nwarps + 31) & ~(int64_t)31;
    run = run < kRun ? run : kRun;
    for (int64_t c0 = warp * run; c0 < total; c0 += nwarps * run) {
        const int64_t c1 = c0 + run < total ? c0 + run : total;
        walk_rows(q, nq, total, c0, c1, queue_guess(q.off, nq, total, c0), op, out, cnt, s_buf, s_n);
    }
}

// ---- Frontier loops of the builds --------------------------------------------------------------
// An operation's whole level loop in one cooperative launch (a CTA of 1,024 threads per SM), one grid
// barrier a level. It ends when the frontier is empty, after max_levels, or when a level's rows hold
// more than max_edges entries (the host launches such a level at full occupancy: k_frontier_level).
// Every level's queue follows the one before it in one pair of arrays, so these have to hold every
// entry ever queued.
constexpr int kLoopThreads = 1024;
enum { W_Q = 0, W_LO = 1, W_LEVELS = 2, W_ERR = 3, W_SLOTS = 4, W_BAR = 16, W_LVL = 32 };
constexpr int kLoopLevels = 64;                        // the most levels of a launch (their sizes go to W_LVL)
constexpr int kLoopWords = W_LVL + kLoopLevels + 1;    // device words

// In: ctl[W_Q] = the frontier (entries << 33 | row entries) at v + ctl[W_LO], the other words zero.
// Out: the same for the level to run next, ctl[W_LEVELS] = levels run, and the packed size of the first
// frontier and of the one after every level from W_LVL on.
template <class Op>
__global__ void __launch_bounds__(kLoopThreads, 1) k_frontier_loop(Op op, Queue all, unsigned long long* ctl,
                                                                   int max_levels, int64_t max_edges) {
    __shared__ int32_t s_stage[32][kStage];
    __shared__ LevelShared<32> sh;
    unsigned int* bar = reinterpret_cast<unsigned int*>(ctl + W_BAR);
    const int wib = threadIdx.x >> 5;
    // (warps numbered across the CTAs first, so that a short frontier spreads over the SMs)
    const int64_t warp = (int64_t)wib * gridDim.x + blockIdx.x, nwarps = (int64_t)gridDim.x * 32;
    unsigned long long packed = __ldcg(ctl + W_Q);
    int64_t lo = (int64_t)__ldcg(ctl + W_LO);
    int lev = 0;
    unsigned met = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl[W_LVL] = packed;
    for (; lev < max_levels; ++lev) {
        const int64_t nq = (int64_t)(packed >> kQShift), total = (int64_t)(packed & kQEdges);
        if (nq == 0 || total > max_edges) break;
        unsigned long long* sl = ctl + W_SLOTS + lev % 3;
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl[W_SLOTS + (lev + 1) % 3] = 0;
        const Queue in{all.v + lo, all.off + lo}, out{all.v + lo + nq, all.off + lo + nq};
        int n_st = 0;
        walk_level(in, nq, total, warp, nwarps, op, out, sl, s_stage[wib], n_st);
        block_publish<32>(sh, s_stage[wib], n_st, out, [&](int32_t x) { return op.deg(x); }, sl);
        if (!grid_barrier(bar, ctl + W_ERR, met)) break;
        lo += nq;
        packed = __ldcg(sl);
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl[W_LVL + 1 + lev] = packed;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // (read by every CTA before its first barrier; unchanged where no level ran)
        ctl[W_Q] = packed;
        ctl[W_LO] = (unsigned long long)lo;
        ctl[W_LEVELS] = (unsigned long long)lev;
    }
}

// One level launched from the host; ctl[W_SLOTS] (zero before) receives the next frontier's size.
constexpr int kLevelThreads = 256;
template <class Op>
__global__ void __launch_bounds__(kLevelThreads) k_frontier_level(Op op, Queue in, int64_t nq, int64_t total, Queue out,
                                                                  unsigned long long* cnt) {
    __shared__ int32_t s_stage[kLevelThreads / 32][kStage];
    int n_st = 0;
    int32_t* s_buf = s_stage[threadIdx.x >> 5];
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    walk_level(in, nq, total, warp, ((int64_t)gridDim.x * blockDim.x) >> 5, op, out, cnt, s_buf, n_st);
    queue_flush(s_buf, n_st, out, [&](int32_t x) { return op.deg(x); }, cnt);
}

// Levels after which a graph of V vertices counts as deep and the builds turn to what needs no levels
// (reciprocal classes for the SCCs, the forest by union-find and Euler tours for the blocks): about
// where the levels so far have cost as much as that will. A level costs 8 us and, in the block build,
// three launches more; the other way costs about 0.35 ms (SCCs) and 0.9 ms (blocks) at 0.65M vertices
// and grows with the vertices. A power-law graph has about ten levels, a road network thousands.
inline int64_t deep_levels(int64_t V) { return 24 + V / 16384; }

// Where a frontier's levels stand: the frontier to run next (entries << 33 | row entries) at `lo` in the
// queue arrays, and the entries of every level so far (the last one: that frontier).
struct FrontierRun {
    unsigned long long packed = 0;
    int64_t lo = 0;
    std::vector<int64_t> levels;
    bool started = false;
    bool done() const { return started && (packed >> kQShift) == 0; }
};

// ---- Bottom-up levels of the builds ------------------------------------------------------------
// Where a frontier's rows hold far more entries than there are vertices left, the vertices left look
// for the frontier instead: a bitmap of the frontier (V / 8 bytes, so the gathers mostly stay in the
// L1) and each row read only as far as its first hit.
__global__ static void k_frontier_bits(const int32_t* q, int64_t n, uint32_t* fwd, uint32_t* bwd) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = q[i], v = e >= 0 ? e : ~e;
        atomicOr((e >= 0 ? fwd : bwd) + (v >> 5), 1u << (v & 31));
    }
}

// First entry w of row [b, b + d) for which hit(w, key), or -1; the row starts on a 16-byte boundary.
// Every lane of the warp calls it (want: this lane has a row, key: a value that goes with it): a lane reads the first 32 entries of its own
// row, four at a time; what is left of longer rows the warp reads together, row after row, as far as
// kLongRow. Rows that go on behind it are left to a second launch by the whole grid (LongRows): one warp took 25 ms
// a level for a hub of 1.5M entries without a hit, of 68.8 ms for the SCCs of that graph (44.1 so).
template <class Hit>
__device__ __forceinline__ int32_t first_hit(const int32_t* adj, int64_t b, int32_t d, bool want, int32_t key, const Hit& hit) {
    int32_t found = -1, at = 0;
    d = d < kLongRow ? d : kLongRow;
    if (want) {
        const int32_t own = d < 32 ? d : 32;
        for (; at + 4 <= own && found < 0; at += 4) {
            const int4 a = *reinterpret_cast<const int4*>(adj + b + at);
            if (hit(a.x, key)) found = a.x;
            else if (hit(a.y, key)) found = a.y;
            else if (hit(a.z, key)) found = a.z;
            else if (hit(a.w, key)) found = a.w;
        }
        for (; at < own && found < 0; ++at) {
            const int32_t w = adj[b + at];
            if (hit(w, key)) found = w;
        }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, want && found < 0 && at < d); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const int64_t rb = __shfl_sync(0xffffffffu, b, src);
        const int32_t rd = __shfl_sync(0xffffffffu, d, src), rkey = __shfl_sync(0xffffffffu, key, src);
        int32_t got = -1;
        for (int32_t k = 32; k < rd && got < 0; k += 32) {
            const int32_t w = k + lane_id() < rd ? adj[rb + k + lane_id()] : -1;
            const unsigned m = __ballot_sync(0xffffffffu, w >= 0 && hit(w, rkey));
            if (m) got = __shfl_sync(0xffffffffu, w, __ffs(m) - 1);
        }
        if (lane_id() == src) found = got;
    }
    return found;
}

// The rows of a level that first_hit left unfinished: queue entries, their number, room for every long row.
struct LongRows {
    int32_t* item;
    unsigned int* n;
    __device__ __forceinline__ void add(int32_t e) const { item[atomicAdd(n, 1u)] = e; }
};

// An operation without bottom-up levels.
struct TopDownOnly {
    bool wants(int64_t, int64_t) const { return false; }
    int launch(gir_dev*, const Queue&, int64_t, const Queue&, unsigned long long*) const { return GIR_OK; }
};

// Runs up to max_levels more levels. Before the first call the caller zeroes ctl (kLoopWords words),
// puts the first frontier at the front of the queue arrays and its packed size in ctl[W_Q].
// kLoopMaxEdges: a larger level runs as its own launch at full occupancy (as the BFS levels do).
constexpr int64_t kLoopMaxEdges = 1ll << 22;
// A large level runs bottom-up where bu.wants(its row entries, entries queued so far).
template <class Op, class BottomUp>
int run_frontier(gir_dev* g, Op op, const BottomUp& bu, Queue q, unsigned long long* ctl, FrontierRun& r,
                 int64_t max_levels) {
    void* hp = nullptr;
    GIR_TRY(pinned(g, kPinnedBytes, &hp));
    unsigned long long* hc = static_cast<unsigned long long*>(hp);
    int loop_ctas = 0;
    GIR_TRY(cooperative_ctas(g, (const void*)k_frontier_loop<Op>, kLoopThreads, &loop_ctas));
    if (loop_ctas == 0 && !r.started) {  // (every level is launched from here: the first frontier's size is read)
        GIR_CUDA(g, cudaMemcpyAsync(hc, ctl + W_Q, sizeof(unsigned long long), cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        r.packed = hc[0];
        r.levels.push_back((int64_t)(r.packed >> kQShift));
        r.started = true;
    }
    while (max_levels > 0 && !r.done()) {
        const int64_t nq = (int64_t)(r.packed >> kQShift), total = (int64_t)(r.packed & kQEdges);
        if (r.started && (total > kLoopMaxEdges || loop_ctas == 0)) {
            GIR_CUDA(g, cudaMemsetAsync(ctl + W_SLOTS, 0, sizeof(unsigned long long), g->stream));
            const Queue in{q.v + r.lo, q.off + r.lo}, out{q.v + r.lo + nq, q.off + r.lo + nq};
            if (total > kLoopMaxEdges && bu.wants(total, r.lo + nq)) {
                GIR_TRY(bu.launch(g, in, nq, out, ctl + W_SLOTS));
            } else {
                k_frontier_level<Op><<<g->num_sms * 8, kLevelThreads, 0, g->stream>>>(op, in, nq, total, out, ctl + W_SLOTS);
                GIR_LAUNCH(g, "k_frontier_level");
            }
            GIR_CUDA(g, cudaMemcpyAsync(hc, ctl + W_SLOTS, sizeof(unsigned long long), cudaMemcpyDeviceToHost, g->stream));
            GIR_CUDA(g, cudaStreamSynchronize(g->stream));
            r.lo += nq;
            r.packed = hc[0];
            r.levels.push_back((int64_t)(r.packed >> kQShift));
            --max_levels;
            continue;
        }
        if (r.started) {
            hc[W_Q] = r.packed;
            hc[W_LO] = (unsigned long long)r.lo;
            for (int k = W_LEVELS; k < W_LVL; ++k) hc[k] = 0;
            GIR_CUDA(g, cudaMemcpyAsync(ctl, hc, sizeof(unsigned long long) * W_LVL, cudaMemcpyHostToDevice, g->stream));
        }
        int levels = (int)(max_levels < kLoopLevels ? max_levels : kLoopLevels);
        int64_t max_edges = kLoopMaxEdges;
        void* args[] = {&op, &q, &ctl, &levels, &max_edges};
        GIR_CUDA(g, cudaLaunchCooperativeKernel((const void*)k_frontier_loop<Op>, g->num_sms, kLoopThreads, args, 0,
                                                g->stream));
        GIR_CUDA(g, cudaMemcpyAsync(hc, ctl, sizeof(unsigned long long) * kLoopWords, cudaMemcpyDeviceToHost, g->stream));
        GIR_CUDA(g, cudaStreamSynchronize(g->stream));
        if (hc[W_ERR]) return fail(g, GIR_ERR_TIMEOUT, "frontier loop: a grid barrier ran out its bound");
        if (!r.started) r.levels.push_back((int64_t)(hc[W_LVL] >> kQShift));
        r.started = true;
        r.packed = hc[W_Q];
        r.lo = (int64_t)hc[W_LO];
        for (int k = 1; k <= (int)hc[W_LEVELS]; ++k) r.levels.push_back((int64_t)(hc[W_LVL + k] >> kQShift));
        max_levels -= (int64_t)hc[W_LEVELS];
    }
    return GIR_OK;
}

#endif

}  // namespace gir
