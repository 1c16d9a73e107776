// traverse.cuh -- persistent push kernels for BFS, SSSP, SSWP and CC over the K-bounded virtual graph.
//
// Reference kernels replaced (rwatling/EEGraph):
//   bfs::{async,sync}_push_{td,dd}   src/bfs.cu:27-273     relax d+1,        atomicMin
//   sssp::{async,sync}_push_{td,dd}  src/sssp.cu:26-299    relax d+w,        atomicMin
//   sswp::{async,sync}_push_{td,dd}  src/sswp.cu:26-271    relax min(d,w),   atomicMax
//   cc::{async,sync}_push_{td,dd}    src/cc.cu:26-271      relax label+w,    atomicMin
//   clearLabel/mixLabels/moveUpLabels/sumLabels  src/gpu_utils.cu:3-34 (frontier upkeep, fused here)
//   the host do { H2D finished; launch; sync; D2H finished } while(!finished) loop, src/eegraph.cu:89-211
//
// One cooperative launch runs the whole traversal. Rounds are separated by a bounded grid barrier
// (common.cuh) instead of a host round trip. A thread expands one part (<= K out-edges of one vertex)
// with aligned 128- or 256-bit streaming loads of targets and weights.
//   TD (topology driven): every round expands every part, as the reference's *_push_td kernels do.
//      SYNC_PUSH_TD keeps the reference's odd/even partner permutation (src/bfs.cu:196-272).
//   DD (data driven): the frontier is a queue of PART ids. A vertex whose value improved is claimed
//      once per round through a round stamp. Claimed vertices collect in per-warp
//      buffers; what is left at a round's end is appended with one reservation per CTA (a hub's parts are
//      written by a whole warp). This
//      replaces label1/label2 + clearLabel; the queue-length counters give --activity (sumLabels).
//      SYNC_PUSH_DD seeds {source}; ASYNC_PUSH_DD seeds every vertex (src/eegraph.cu:41-49).
// Values are updated in place with atomicMin/atomicMax, as in the reference; a vertex whose value is
// still "unreached" (BFS/SSSP: DIST_INFINITY, SSWP: 0) pushes nothing. That keeps SSSP free of the
// INF+w wrap of src/sssp.cu:62 (identical to the reference's SYNC_PUSH_DD results) without changing
// any other fixed point.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdio>

#include "internal.hpp"

namespace eeg {
namespace trav {

// CTA size per operator, two CTAs per SM: 384 threads (80 registers) for BFS, whose group of atomics
// then covers a whole 8-slot part; 512 threads (64 registers) for the others. Measured with K = 8: BFS on
// the 2047^2 grid 1.00 ms, at 512 threads 1.04; SSSP on R-MAT s22 0.634 ms and BFS on the grid within 1 %
// with 768 or 1024 threads and one CTA per SM, more at three CTAs of 384 (56 registers); bucketed rounds
// 5.95 ms on the 4096^2 grid, at 384 threads with 4 or 8 slots in flight 5.85 to 5.90.
template <int OP>
__host__ __device__ constexpr int trav_tpb() {
    return OP == OP_BFS ? 384 : 512;
}

struct TravArgs {
    uint32_t n;
    uint32_t P;
    const uint32_t* __restrict__ vstart;
    const uint32_t* __restrict__ vowner;
    const uint32_t* __restrict__ vcol;
    const uint32_t* __restrict__ vw;
    uint32_t* dist;
    uint32_t* q0;
    uint32_t* q1;
    uint32_t* stamp;
    uint32_t* pushed;      // P: the owner value each part last pushed with (DD; null = every queued part expands)
    const uint32_t* rvstart;  // source-seeded BFS: the transposed graph's parts (null = push rounds only)
    const uint32_t* rvcol;
    uint32_t* plist;          // 2n: the vertices each pull round left unreached (two lists alternate)
    TravCtrl* ctrl;
    uint32_t* activity;
    uint32_t activity_cap;
    uint32_t source;
    uint32_t seed_all;
    uint32_t partner;
    uint32_t max_iters;
    uint32_t it_start;     // first round of this launch (0: also the set-up phase)
    uint64_t timeout_ns;
    uint32_t rounds_limit; // rounds this launch may run (host-loop mode: 1); 0 = until done
    uint32_t delta;        // SSSP/SSWP bucket width (bucketed kernels only)
    uint32_t* fpile;       // 3 x n far piles (bucketed kernels only)
    uint32_t* fflag;       // n far flags (1 = in a pile)
    uint32_t cc_zero;      // CC: relax with weight 0 (connected components)
};

// K weights from slot `at` on (CC in connected-components mode: zeros, nothing loaded).
template <int OP, int K>
__device__ __forceinline__ void load_weights(const TravArgs& a, size_t at, uint32_t (&wt)[K], uint64_t pol) {
    if (OP == OP_CC && a.cc_zero) {
#pragma unroll
        for (int i = 0; i < K; ++i) wt[i] = 0u;
    } else {
        ld_part<K>(a.vw + at, wt, pol);
    }
}

template <int OP>
__device__ __forceinline__ uint32_t init_value(uint32_t v, uint32_t src) {
    if (OP == OP_CC) return v;                       // src/eegraph.cu:546
    if (OP == OP_SSWP) return v == src ? INF : 0u;   // src/eegraph.cu:1551-1559
    return v == src ? 0u : INF;                      // src/eegraph.cu:41-49, 2062-2073
}
template <int OP>
__device__ __forceinline__ bool unreached(uint32_t d) {
    if (OP == OP_BFS || OP == OP_SSSP) return d == INF;
    if (OP == OP_SSWP) return d == 0u;
    return false;
}
// Slots whose atomics are issued together (value atomic + claim, 2 returned values each) under a
// 64-register budget (512-thread CTAs): 4. R-MAT s22, K = 8: SSSP 0.636 ms (2: 0.650), SSWP 0.676 (2:
// 0.717), CC 1.09 (2: 1.11); 8 spills 90 bytes. Bucketed rounds keep their far-buffer state in registers
// too and take 2 (4 spills 96 bytes: 5.95 against 5.84 ms on the 4096^2 grid).
constexpr int ATOMIC_GROUP = 4;

template <int OP>
__device__ __forceinline__ uint32_t relax_value(uint32_t d, uint32_t w) {
    if (OP == OP_BFS) return d + 1u;
    if (OP == OP_SSWP) return d < w ? d : w;
    const uint64_t s = (uint64_t)d + w;              // SSSP / CC: saturate, never wrap
    return s >= INF ? INF : (uint32_t)s;
}
template <int OP>
__device__ __forceinline__ bool better(uint32_t a, uint32_t b) {
    return OP == OP_SSWP ? a > b : a < b;
}
template <int OP>
__device__ __forceinline__ uint32_t atomic_improve(uint32_t* p, uint32_t v) {
    return OP == OP_SSWP ? atomicMax(p, v) : atomicMin(p, v);
}

constexpr int WCAP = 256;  // per-warp append buffer (claimed vertices) before a flush to the queue
constexpr int FCAP = 128;  // per-warp buffer of far vertices (bucketed rounds) before a flush to the pile
constexpr uint32_t PULL_LANE = 4;  // BFS pull rounds: parts a lane walks alone before the warp takes over

// Lane's share of the parts of the buffered vertices: returns the warp's total, *before = the parts of the
// lanes below. Called by all 32 lanes with a warp-uniform `cnt`.
__device__ __forceinline__ uint32_t warp_parts(const uint32_t* __restrict__ vstart, const uint32_t* buf, uint32_t cnt,
                                               uint32_t lane, uint32_t* before) {
    __syncwarp();
    uint32_t sum = 0;
    for (uint32_t e = lane; e < cnt; e += 32u) {
        const uint32_t t = buf[e];
        sum += vstart[t + 1] - vstart[t];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= (uint32_t)off) inc += y;
    }
    *before = inc - sum;
    return __shfl_sync(0xffffffffu, inc, 31);
}

// The part ids of the buffered vertices, from `pos` (this lane's) on; a vertex with more than 32 parts is
// written by the whole warp. Entries at or beyond `cap` are not written (each vertex is claimed once per
// round, so a round never produces more than `cap` = the number of parts; the reader clamps and reports
// an overflow).
__device__ __forceinline__ void warp_write(const uint32_t* __restrict__ vstart, const uint32_t* buf, uint32_t cnt,
                                           uint32_t pos, uint32_t* qnext, uint32_t lane, uint32_t cap) {
    const uint32_t rounds = (cnt + 31u) / 32u;
    for (uint32_t k = 0; k < rounds; ++k) {
        const uint32_t e = k * 32u + lane;
        uint32_t s0 = 0, np = 0;
        if (e < cnt) {
            const uint32_t t = buf[e];
            s0 = vstart[t];
            np = vstart[t + 1] - s0;
            if (np <= 32u)
                for (uint32_t j = 0; j < np; ++j)
                    if (pos + j < cap) qnext[pos + j] = s0 + j;
        }
        uint32_t big = __ballot_sync(0xffffffffu, np > 32u);
        while (big) {  // hub vertices: the whole warp writes their part ids
            const int l = __ffs(big) - 1;
            big &= big - 1u;
            const uint32_t bs0 = __shfl_sync(0xffffffffu, s0, l);
            const uint32_t bnp = __shfl_sync(0xffffffffu, np, l);
            const uint32_t bpos = __shfl_sync(0xffffffffu, pos, l);
            for (uint32_t j = lane; j < bnp; j += 32u)
                if (bpos + j < cap) qnext[bpos + j] = bs0 + j;
        }
        pos += np;
    }
    __syncwarp();
}

// Warp-cooperative append of the warp's claimed vertices to the next queue: one reservation per flush,
// then every claimed vertex's part ids are written. Called by all 32 lanes with a warp-uniform `cnt`.
__device__ __forceinline__ void warp_append(const uint32_t* __restrict__ vstart, uint32_t* parts_ctr, const uint32_t* buf,
                                            uint32_t cnt, uint32_t* qnext, uint32_t lane, uint32_t cap) {
    uint32_t before;
    const uint32_t total = warp_parts(vstart, buf, cnt, lane, &before);
    uint32_t base = 0;
    if (lane == 0 && total) base = atomicAdd(parts_ctr, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    warp_write(vstart, buf, cnt, base + before, qnext, lane, cap);
}

// The same within a round of k_traverse (a full buffer).
__device__ __forceinline__ void warp_flush(const TravArgs& a, const uint32_t* buf, uint32_t cnt, uint32_t* qnext,
                                           uint32_t nxt, bool count_verts, uint32_t lane) {
    uint32_t before;
    const uint32_t total = warp_parts(a.vstart, buf, cnt, lane, &before);
    uint32_t base = 0;
    if (lane == 0) {
        base = (uint32_t)atomicAdd(&a.ctrl->queued[nxt], (unsigned long long)total);
        if (count_verts) atomicAdd(&a.ctrl->qverts[nxt], cnt);
    }
    base = __shfl_sync(0xffffffffu, base, 0);
    warp_write(a.vstart, buf, cnt, base + before, qnext, lane, a.P);
}

// The same vertices' part total, without the parts (a round whose queue is not written).
__device__ __forceinline__ void warp_count(const TravArgs& a, const uint32_t* buf, uint32_t cnt, uint32_t nxt,
                                           uint32_t lane) {
    uint32_t before;
    const uint32_t total = warp_parts(a.vstart, buf, cnt, lane, &before);
    if (lane == 0) {
        atomicAdd(&a.ctrl->queued[nxt], (unsigned long long)total);
        atomicAdd(&a.ctrl->qverts[nxt], cnt);
    }
}

// End of a round: what the CTA's warps still hold, in one reservation per CTA (with one per warp, and the
// vertices counted always, BFS on the 4096^2 grid took 2.24 ms, against 2.07). Called by all threads; qnext
// null: counted only.
template <int NW>
__device__ __forceinline__ void cta_flush(const TravArgs& a, const uint32_t* buf, uint32_t cnt, uint32_t* qnext,
                                          uint32_t nxt, bool count_verts, uint32_t lane, uint2* s_tot) {
    const uint32_t warp = threadIdx.x >> 5;
    uint32_t before = 0, total = 0;
    if (cnt) total = warp_parts(a.vstart, buf, cnt, lane, &before);
    if (lane == 0) s_tot[warp] = make_uint2(total, cnt);
    __syncthreads();
    if (warp == 0) {
        uint2 t = lane < NW ? s_tot[lane] : make_uint2(0u, 0u);
        uint32_t inc = t.x;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= (uint32_t)off) inc += y;
        }
        const uint32_t verts = __reduce_add_sync(0xffffffffu, t.y);
        uint32_t base = 0;
        if (lane == 31u && verts) {
            base = (uint32_t)atomicAdd(&a.ctrl->queued[nxt], (unsigned long long)inc);
            if (count_verts) atomicAdd(&a.ctrl->qverts[nxt], verts);
        }
        base = __shfl_sync(0xffffffffu, base, 31);
        if (lane < NW) s_tot[lane].x = base + inc - t.x;
    }
    __syncthreads();
    if (cnt && qnext) warp_write(a.vstart, buf, cnt, s_tot[warp].x + before, qnext, lane, a.P);
}

// Bucketed rounds, a warp's buffered far vertices: all flag exchanges go out together; a vertex enters the
// pile once (its flag). Returns the number that enter, *bits = this lane's entries among them.
__device__ __forceinline__ uint32_t far_flags(uint32_t* fflag, const uint32_t* buf, uint32_t cnt, uint32_t lane,
                                              uint32_t* bits, uint32_t* before) {
    __syncwarp();
    uint32_t old[FCAP / 32];
#pragma unroll
    for (int k = 0; k < FCAP / 32; ++k) {
        const uint32_t e = k * 32u + lane;
        old[k] = e < cnt ? atomicExch(&fflag[buf[e]], 1u) : 1u;
    }
    uint32_t b = 0;
#pragma unroll
    for (int k = 0; k < FCAP / 32; ++k) b |= (old[k] != 1u ? 1u : 0u) << k;
    *bits = b;
    uint32_t inc = __popc(b);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= (uint32_t)off) inc += y;
    }
    *before = inc - __popc(b);
    return __shfl_sync(0xffffffffu, inc, 31);
}
__device__ __forceinline__ void far_write(const TravArgs& a, const uint32_t* buf, uint32_t bits, uint32_t pos,
                                          uint32_t* pile, uint32_t lane) {
#pragma unroll
    for (int k = 0; k < FCAP / 32; ++k)
        if ((bits >> k) & 1u) {
            if (pos < a.n) pile[pos] = buf[k * 32 + lane];
            else atomicCAS(&a.ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_OVERFLOW);
            ++pos;
        }
    __syncwarp();
}

// The barrier that ends a round, on the word that also counts the next round's parts: the last poll of the
// arrivals brings the queue length along, so a round starts without reading control words (one L2 round
// trip and one CTA barrier less), and the arrival is a release-ordered reduction instead of a fence and an
// atomic. R-MAT s22 SSSP 0.707 -> 0.667 ms, s20 0.250 -> 0.233, s16 97 -> 91 us. Bounded like grid_barrier
// (common.cuh); a CTA that gives up sets the word's top bit for the others that wait there and, for those that have
// gone on to another barrier, the abort word (looked at with the timer, so the common poll costs nothing more).
// Returns false when aborting.
__device__ __forceinline__ bool round_barrier(unsigned long long* w, BarrierWords* bw, uint64_t timeout_ns,
                                              uint32_t* s_len) {
    __shared__ uint32_t s_ok3;
    __syncthreads();
    if (threadIdx.x == 0) {
        red_release_add64(w, 1ull << 32);
        uint32_t ok = 1;
        const uint64_t t0 = global_timer_ns();  // the wait is measured from this CTA's arrival
        uint32_t spins = 0;
        unsigned long long v;
        while (true) {
            v = ld_acquire64(w);
            const uint32_t arrived = (uint32_t)(v >> 32);
            if (arrived & 0x80000000u) { ok = 0; break; }
            if (arrived == gridDim.x) break;
            __nanosleep(32);
            if ((++spins & 7u) == 0) {
                if (ld_relaxed(&bw->abort)) { ok = 0; break; }
                if (global_timer_ns() - t0 > timeout_ns) {
                    atomicCAS(&bw->status, (uint32_t)DEV_OK, (uint32_t)DEV_TIMEOUT);
                    atomicExch(&bw->abort, 1u);
                    atomicOr(w, 1ull << 63);
                    ok = 0;
                    break;
                }
            }
        }
        *s_len = (uint32_t)v;
        s_ok3 = ok;
    }
    __syncthreads();
    return s_ok3 != 0;
}

// Bucketed rounds (SSSP/SSWP, SYNC_PUSH_DD, delta > 0). A claimed vertex whose key (SSSP: distance,
// SSWP: INF - width; smaller is closer in both) is not below the threshold T waits in a far pile (one
// entry per vertex, marked by its flag) instead of entering the next queue. When the queue runs empty,
// a far round sets T = smallest recorded far key + delta and moves every far vertex below T back.
// The fixed point is the same; on high-diameter graphs far fewer edges are rescanned. T and the
// current pile travel in control words keyed by round parity, so every CTA (and every host-loop
// launch) reads the value the previous round settled; three piles rotate so that a pile's length is
// reset two far rounds before it is written again.
// MODE: SSSP and SSWP, bucketed rounds; BFS, pull rounds. Kernels of their own: either takes registers that the
// plain rounds need (with the pull code in it, push-only BFS spilled at K = 16 and pull BFS at K = 8).
template <int OP, int K, bool TD, bool MODE = false>
__global__ void __launch_bounds__(trav_tpb<OP>(), 2) k_traverse(TravArgs a) {
    constexpr int T_TPB = trav_tpb<OP>();
    constexpr bool BKT = MODE && OP != OP_BFS, BFSBU = MODE && OP == OP_BFS;
    __shared__ uint32_t s_buf[TD ? 1 : T_TPB / 32][TD ? 1 : WCAP];
    __shared__ uint2 s_tot[TD ? 1 : T_TPB / 32];
    __shared__ uint32_t s_far[BKT ? T_TPB / 32 : 1][BKT ? FCAP : 1];
    __shared__ uint32_t s_fbase[BKT ? T_TPB / 32 : 1], s_fkey[BKT ? T_TPB / 32 : 1];
    __shared__ uint32_t s_next[2];  // per round (alternating): next of this CTA's 32-entry chunks
    __shared__ uint32_t s_ctl[6];   // this round's control words, read once per CTA

    TravCtrl* ctrl = a.ctrl;
    const uint32_t gtid = blockIdx.x * T_TPB + threadIdx.x;
    const uint32_t gthreads = gridDim.x * T_TPB;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lanemask_lt = (1u << lane) - 1u;
    uint32_t* wbuf = s_buf[TD ? 0 : threadIdx.x >> 5];
    uint32_t* fbuf = s_far[BKT ? threadIdx.x >> 5 : 0];
    const uint64_t pol = l2_evict_first_policy();
    uint32_t epoch = 0;

    // statistics, 32 bits each (a thread's share of 64 rounds is far below 2^32); every 64 rounds a warp's
    // totals go to shared memory. As 64-bit sums they took three more of the 64 registers.
    uint32_t my_parts = 0, my_edges = 0, my_updates = 0;
    __shared__ unsigned long long s_stat[T_TPB / 32][3];
    if (lane < 3u) s_stat[threadIdx.x >> 5][lane] = 0ull;
    __syncwarp();
    auto stat_round = [&]() {
        const uint32_t r0 = __reduce_add_sync(0xffffffffu, my_parts), r1 = __reduce_add_sync(0xffffffffu, my_edges),
                       r2 = __reduce_add_sync(0xffffffffu, my_updates);
        if (lane == 0) {
            s_stat[threadIdx.x >> 5][0] += r0;
            s_stat[threadIdx.x >> 5][1] += r1;
            s_stat[threadIdx.x >> 5][2] += r2;
        }
        my_parts = my_edges = my_updates = 0u;
    };
    // BFS seeded with the source only: every round's queue holds exactly the vertices at level `it`
    // (a round sets values to it+1 only, and a vertex leaves INF once, so atomicMin alone makes each claim
    // unique). Seeding every vertex (ASYNC_PUSH_DD) makes round 0 dense and in place: a vertex reached in
    // it may push again in the same round, so levels in a queue mix and claims need the stamps.
    const bool bfs_levels = OP == OP_BFS && !TD && !a.seed_all;
    // CC: a queued part that already pushed its owner's current value skips its expansion: every target
    // holds at most that value + the weight already (labels only fall), and an improvement of the owner
    // later in the round re-queues it. In the dense all-seeded round 0 most vertices are improved before
    // their own parts are reached and push the improved label, so their round-1 rescan is redundant:
    // edges scanned per reached edge 2.03 -> 1.20 and 1.33 -> 1.22 ms on R-MAT s22 (symmetrised).
    // SSSP and SSWP rescan less for it too (1.59 -> 1.21, 1.65 -> 1.19) but take the same time, and the
    // per-part values cost them 15 % more DRAM traffic, so their kernels leave the check out, as does BFS.
    const bool use_push = OP == OP_CC && !TD && !BKT && a.pushed != nullptr;
    constexpr uint32_t PSENT = OP == OP_SSWP ? 0u : 0xFFFFFFFFu;  // no part ever pushes with it
    // Direction-optimising BFS (source-seeded, one persistent launch): when the frontier's parts are many
    // against the parts of the vertices not yet reached (14x), a round pulls instead of pushing -- every
    // unreached vertex reads the levels of its in-neighbours from the transposed parts, part by part, and
    // takes level it+1 at the first one found at level it (its forward parts are counted and, after the
    // first pull round, appended, so a push round can follow); rounds push again once the frontier holds fewer than n/12 vertices. Every CTA
    // takes the same decision from the same control words. The first pull round walks every vertex and
    // lists the ones with in-edges that it left unreached; a later pull round walks the last list only
    // (a superset of the unreached vertices with in-edges, whatever rounds came between). Same levels;
    // R-MAT s22 from the hub pulls in its two large rounds, the second over 6.5 % of the vertices.
    constexpr int KH = K > 8 && trav_tpb<OP>() == 512 ? 8 : K;  // slots of a part expanded at a time
    constexpr int PVL = K <= 8 ? 4 : 2;  // vertices per lane in a pull round, their loads issued together
    const bool can_bu = BFSBU;  // source-seeded, transposed parts, one persistent launch
    uint32_t seen_parts = 0;  // forward parts of the vertices reached so far
    bool bu = false;          // this round pulls
    uint32_t pj = 0;          // pull rounds so far
    uint32_t it = a.it_start;
    bool all_done = true;  // false when this launch stops only because of rounds_limit
    if (threadIdx.x == 0) s_next[0] = s_next[1] = 0u;
    __syncthreads();
    if (a.it_start == 0) {
        // ---- round 0 set-up: values, stamps, initial frontier
        for (uint32_t v = gtid; v < a.n; v += gthreads) {
            a.dist[v] = init_value<OP>(v, a.source);
            if (!TD && !bfs_levels) a.stamp[v] = 0u;
            if (BKT) a.fflag[v] = 0u;
        }
        if (use_push)
            for (uint32_t q = gtid; q < a.P; q += gthreads) a.pushed[q] = PSENT;
        if (BKT && blockIdx.x == 0 && threadIdx.x == 0) {
            for (int i = 0; i < 3; ++i) {
                ctrl->fcnt[i] = 0u;
                ctrl->fmin[i] = 0xFFFFFFFFu;
            }
            ctrl->fcsel[0] = 0u;  // round 0 (the source's parts) sends every claim to pile 0 (T = 0)
            ctrl->tsel[0] = 0u;
        }
        if (BFSBU && blockIdx.x == 0 && threadIdx.x == 0) ctrl->lcnt[0] = ctrl->lcnt[1] = ctrl->lcnt[2] = ctrl->fcnt[0] = 0u;
        if (!TD && !a.seed_all && blockIdx.x == 0) {
            const uint32_t s0 = a.vstart[a.source], s1 = a.vstart[a.source + 1];
            for (uint32_t j = threadIdx.x; j < s1 - s0; j += T_TPB) a.q0[j] = s0 + j;
            if (threadIdx.x == 0) {
                ctrl->queued[0] = s1 - s0;
                ctrl->qverts[0] = 1u;
            }
        }
        if (!grid_barrier(&ctrl->bw, epoch, a.timeout_ns)) goto finish;
    }

    for (;; ++it) {
        if (a.rounds_limit && it - a.it_start >= a.rounds_limit) {  // host-loop mode: next round, next launch
            all_done = false;
            break;
        }
        const uint32_t cur = it % 3u, nxt = (it + 1u) % 3u, old = (it + 2u) % 3u;
        const bool dense = TD || (a.seed_all && it == 0);
        // The queue length came with the barrier that ended the last round (the launch's first round reads
        // it). What else the round needs is read by one thread per CTA (not by every warp of the grid:
        // those same-address reads queue at one L2 slice) and shared.
        const bool first = it == a.it_start;
        if (threadIdx.x == 0) {
            if (first) s_ctl[0] = (uint32_t)ld_relaxed64(&ctrl->queued[cur]);
            if (can_bu || a.activity) s_ctl[5] = ld_relaxed(&ctrl->qverts[cur]);
            if (can_bu) s_ctl[1] = ld_relaxed(&ctrl->lcnt[(pj + 2u) % 3u]);  // the last pull round's list
            if (BKT) {
                const uint32_t f = ld_relaxed(&ctrl->fcsel[it & 1u]);
                uint32_t c[3], m[3];  // every pile's words, not those of pile f after it is known
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    c[i] = ld_relaxed(&ctrl->fcnt[i]);
                    m[i] = ld_relaxed(&ctrl->fmin[i]);
                }
                s_ctl[1] = f;
                s_ctl[2] = ld_relaxed(&ctrl->tsel[it & 1u]);
                s_ctl[3] = f == 0u ? c[0] : (f == 1u ? c[1] : c[2]);
                s_ctl[4] = f == 0u ? m[0] : (f == 1u ? m[1] : m[2]);
            }
        }
        if (first || can_bu || a.activity || BKT) __syncthreads();
        uint32_t fc = 0, T = 0xFFFFFFFFu, fcount = 0;
        if (BKT) {
            fc = s_ctl[1];
            T = s_ctl[2];
            fcount = s_ctl[3];
        }
        if (it > 0) {
            const uint32_t produced = s_ctl[0];
            if (a.activity && blockIdx.x == 0 && threadIdx.x == 0 && it - 1 < a.activity_cap)
                a.activity[it - 1] = TD ? produced : s_ctl[5];
            if (produced == 0u && fcount == 0u) break;
        }
        const bool was_bu = bu;
        if (can_bu) {
            const uint32_t fparts = s_ctl[0], fverts = s_ctl[5];
            seen_parts += fparts;
            const uint32_t unreached_parts = a.P - (seen_parts < a.P ? seen_parts : a.P);
            bu = bu ? (uint64_t)fverts * 12u >= a.n : (it > 0 && (uint64_t)fparts * 14u > unreached_parts);
        }
        uint32_t len;
        const bool swap = TD && a.partner && (it & 1u);
        if (dense) len = swap ? (a.P + (a.P & 1u)) : a.P;
        else len = s_ctl[0];
        const bool frontier_empty = !dense && len == 0u;
        if (!dense && len > a.P) {  // cannot happen (one claim per vertex per round); never read past the queue
            if (blockIdx.x == 0 && threadIdx.x == 0)
                atomicCAS(&ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_OVERFLOW);
            len = a.P;
        }
        // a pull round walks every vertex, or the last pull round's list
        const uint32_t pcnt = BFSBU ? (pj > 0 && s_ctl[1] < a.n ? s_ctl[1] : a.n) : 0u;
        if (BFSBU && bu) len = (uint32_t)(((uint64_t)pcnt + 32u * PVL - 1u) / (32u * PVL) * 32u);
        bool far_round = false;
        if (frontier_empty) {
            if (!BKT || fcount == 0u) break;
            if (fcount > a.n) {  // one entry per flagged vertex; never read past the pile
                if (blockIdx.x == 0 && threadIdx.x == 0)
                    atomicCAS(&ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_OVERFLOW);
                fcount = a.n;
            }
            far_round = true;
            const uint32_t fm = s_ctl[4];
            T = fm > 0xFFFFFFFFu - a.delta ? 0xFFFFFFFFu : fm + a.delta;
        }
        const uint32_t fdst = far_round ? (fc + 1u) % 3u : fc;  // pile receiving this round's far vertices
        if (it >= a.max_iters) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_ITER_CAP);
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ctrl->queued[old] = 0ull;
            ctrl->qverts[old] = 0u;
            if (BFSBU && bu) ctrl->lcnt[(pj + 1u) % 3u] = 0u;  // the next pull round's list
            if (BKT) {  // what the next round reads; the pile two far rounds back is free again
                ctrl->fcsel[(it + 1u) & 1u] = fdst;
                ctrl->tsel[(it + 1u) & 1u] = T;
                if (far_round) {
                    ctrl->fcnt[(fc + 2u) % 3u] = 0u;
                    ctrl->fmin[(fc + 2u) % 3u] = 0xFFFFFFFFu;
                }
            }
        }
        // The first pull round claims most of the graph, and as a rule the next round pulls too: it counts its
        // claims' parts but does not write them (R-MAT s22 0.199 -> 0.181 ms; s21 to s16, ef 8 to 32: 1 to 13 %
        // less). A push round that follows it all the same collects the vertices at its level here: a scan of the levels and one more barrier, once
        // per run.
        if (BFSBU && was_bu && !bu && pj == 1u) {
            uint32_t* q = (it & 1u) ? a.q1 : a.q0;
            uint32_t cnt = 0;
            auto put = [&]() {
                uint32_t before, base = 0;
                const uint32_t total = warp_parts(a.vstart, wbuf, cnt, lane, &before);
                if (lane == 0) base = atomicAdd(&ctrl->fcnt[0], total);
                base = __shfl_sync(0xffffffffu, base, 0);
                warp_write(a.vstart, wbuf, cnt, base + before, q, lane, a.P);
                cnt = 0;
            };
            for (uint64_t b0 = (uint64_t)(gtid - lane) * 4u; b0 < a.n; b0 += (uint64_t)gthreads * 4u) {
                bool hit[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint64_t v = b0 + 32u * u + lane;
                    hit[u] = v < a.n && a.dist[v] == it;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t mask = __ballot_sync(0xffffffffu, hit[u]);
                    if (!mask) continue;
                    const uint32_t c = __popc(mask);
                    if (cnt + c > (uint32_t)WCAP) put();
                    if (hit[u]) wbuf[cnt + __popc(mask & lanemask_lt)] = (uint32_t)b0 + 32u * u + lane;
                    cnt += c;
                }
            }
            if (cnt) put();
            if (!grid_barrier(&ctrl->bw, epoch, a.timeout_ns)) break;
        }
        const uint32_t* pile_src = BKT ? a.fpile + (size_t)fc * a.n : nullptr;
        uint32_t* pile_dst = BKT ? a.fpile + (size_t)fdst * a.n : nullptr;
        uint32_t fcnt = 0, fkmin = 0xFFFFFFFFu;  // fill of the far buffer (warp-uniform); this lane's smallest key
        // Warp-collective: the lanes with `fl` send vertex t (key `key`) to the far pile, through a per-warp
        // buffer: one flag exchange, one reservation and one minimum per slot and warp (each with its
        // result waited for, the latter two on the same two words for the whole grid) took two thirds of a
        // bucketed round of the 4096^2 grid.
        auto to_far = [&](bool fl, uint32_t t, uint32_t key) {
            const uint32_t fmask = __ballot_sync(0xffffffffu, fl);
            if (!fmask) return;
            const uint32_t c = __popc(fmask);
            if (fcnt + c > (uint32_t)FCAP) {
                uint32_t bits, before, base = 0;
                const uint32_t tot = far_flags(a.fflag, fbuf, fcnt, lane, &bits, &before);
                if (lane == 0 && tot) base = atomicAdd(&ctrl->fcnt[fdst], tot);
                base = __shfl_sync(0xffffffffu, base, 0);
                far_write(a, fbuf, bits, base + before, pile_dst, lane);
                fcnt = 0;
            }
            if (fl) {
                fbuf[fcnt + __popc(fmask & lanemask_lt)] = t;
                fkmin = key < fkmin ? key : fkmin;
            }
            fcnt += c;
        };
        // no __restrict__/const-qualified read-only path here: each queue is rewritten every other round
        const uint32_t* qcur = (it & 1u) ? a.q1 : a.q0;
        uint32_t* qnext = (it & 1u) ? a.q0 : a.q1;
        const uint32_t tag = it + 1u;
        uint32_t changed = 0;
        uint32_t wcnt = 0;  // warp-uniform fill of wbuf
        // This CTA's share of the round is the strided set of 32-entry chunks blockIdx.x + i * gridDim.x;
        // its warps draw from it through a shared counter (this round's; the other one is reset for the
        // next round, whose start is ordered by the grid barrier).
        if (threadIdx.x == 0) s_next[(it + 1u) & 1u] = 0u;
        const uint32_t items = far_round ? fcount : len;
        const uint32_t nch = (items + 31u) / 32u;
        // A round of at most two chunks per warp is a chain of dependent loads: the part ranges of the
        // claimed vertices are fetched while the chunk is still expanded (BFS on the 2047^2 grid 1.28 ->
        // 1.21 ms). In large rounds the fetches only take L1 from the filter reads (R-MAT s22 BFS +2 %).
        const bool small = ((OP == OP_BFS && !BFSBU) || BKT) && items <= 2u * gthreads;
        // In such a round of a low-degree graph (about one part per vertex) BFS leaves the filter reads out of
        // the chain: atomicMin finds out itself, for three or four targets per part, whether one improves
        // (2047^2 grid 1.07 -> 1.00 ms). In the small rounds of a power-law graph nearly all of a part's eight
        // targets are reached already, and the filter spares their atomics (R-MAT s22 0.203 ms, 0.211 without).
        const bool unfiltered = OP == OP_BFS && !TD && bfs_levels && small && a.P - a.P / 8u <= a.n;
        // A pull round's chunks are vertex ranges, and a vertex id's low bits set its degree on R-MAT-like
        // graphs: with chunk b + i * grid (grid = 304 = 16 * 19) a CTA saw the same low bits in every
        // chunk, and CTAs took 115 to 360 thousand cycles over the same chunk counts (R-MAT s22). In a
        // pull round a CTA takes chunk i * grid + (b + i) mod grid of each row i instead: every chunk
        // once, every residue in every CTA.
        const bool rot = BFSBU && bu;
        const uint32_t my_chunks = rot ? (nch + gridDim.x - 1u) / gridDim.x
                                       : (nch > blockIdx.x ? (nch - blockIdx.x + gridDim.x - 1u) / gridDim.x : 0u);

        // Software-pipelined by one chunk: the next chunk is drawn and its queue entries are loaded
        // before the current chunk is expanded, so the queue load is off each part's dependent chain.
        auto draw = [&](uint32_t& pn) -> uint32_t {
            uint32_t ci = 0;
            if (lane == 0) ci = atomicAdd(&s_next[it & 1u], 1u);
            ci = __shfl_sync(0xffffffffu, ci, 0);
            pn = 0xFFFFFFFFu;
            if (ci < my_chunks) {
                uint32_t ch = blockIdx.x + ci;
                if (rot) {
                    while (ch >= gridDim.x) ch -= gridDim.x;
                    ch += ci * gridDim.x;
                } else {
                    ch = blockIdx.x + ci * gridDim.x;
                }
                const uint32_t idx = ch * 32u + lane;
                if (idx < items) {
                    pn = far_round ? pile_src[idx] : ((dense || (BFSBU && bu)) ? idx : qcur[idx]);
                    if (swap) pn ^= 1u;
                }
            }
            return ci;
        };
        uint32_t p_next;
        uint32_t ci_next = draw(p_next);
        for (;;) {
            if (ci_next >= my_chunks) break;
            const uint32_t p = p_next;
            ci_next = draw(p_next);
            if (BKT && far_round) {  // far round: p is a far vertex; move it back when below T
                bool move = false, stay = false;
                uint32_t key = 0;
                if (p < a.n && atomicExch(&a.fflag[p], 0u) == 1u) {
                    const uint32_t dv = a.dist[p];
                    key = OP == OP_SSWP ? INF - dv : dv;
                    if (key < T) move = true;
                    else stay = true;
                }
                to_far(stay, p, key);
                const uint32_t mask = __ballot_sync(0xffffffffu, move);
                if (mask) {
                    const uint32_t c = __popc(mask);
                    if (wcnt + c > (uint32_t)WCAP) {
                        warp_flush(a, wbuf, wcnt, qnext, nxt, can_bu || a.activity, lane);
                        wcnt = 0;
                    }
                    if (move) wbuf[wcnt + __popc(mask & lanemask_lt)] = p;
                    wcnt += c;
                }
                continue;
            }
            if (BFSBU && bu) {  // pull: item p covers PVL vertices, 32 apart; each belongs to this lane alone
                bool want[PVL], claim[PVL];
                uint32_t vv[PVL], s0[PVL], np[PVL];
                const uint64_t vb = (uint64_t)(p >> 5) * (32u * PVL) + (p & 31u);
                const uint32_t* lrd = a.plist + (size_t)((pj + 1u) & 1u) * a.n;  // the last pull round's list
#pragma unroll
                for (int k = 0; k < PVL; ++k) {  // every level and part range first, then every first part
                    const uint64_t li = vb + 32u * k;
                    const bool ok = p < items && li < pcnt;
                    const uint32_t v = ok ? (pj > 0 ? lrd[li] : (uint32_t)li) : 0u;
                    want[k] = claim[k] = false;
                    vv[k] = v;
                    s0[k] = np[k] = 0u;
                    if (ok) {
                        const uint32_t dv = a.dist[v];
                        s0[k] = __ldg(&a.rvstart[v]);
                        np[k] = __ldg(&a.rvstart[v + 1]) - s0[k];
                        want[k] = dv == INF && np[k] > 0u;
                    }
                }
                {
                    uint32_t c[PVL][K];
#pragma unroll
                    for (int k = 0; k < PVL; ++k) {
                        if (want[k]) ld_part<K>(a.rvcol + (size_t)s0[k] * K, c[k], pol);
                        else
#pragma unroll
                            for (int i = 0; i < K; ++i) c[k][i] = NO_EDGE;
                    }
#pragma unroll
                    for (int k = 0; k < PVL; ++k) {
                        bool found = false;
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            if (c[k][i] != NO_EDGE) {
                                found |= a.dist[c[k][i]] == it;
                                ++my_edges;
                            }
                        }
                        if (want[k]) ++my_parts;
                        claim[k] = found;
                    }
                }
#pragma unroll
                for (int k = 0; k < PVL; ++k) {
                    // no parent in the first part: the lane walks the next ones up to PULL_LANE ...
                    const uint32_t lim = want[k] ? (np[k] < PULL_LANE ? np[k] : PULL_LANE) : 0u;
                    for (uint32_t j = 1; j < lim && !claim[k]; ++j) {
                        uint32_t c[K];
                        ld_part<K>(a.rvcol + (size_t)(s0[k] + j) * K, c, pol);
                        bool found = false;
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            if (c[i] != NO_EDGE) {
                                found |= a.dist[c[i]] == it;
                                ++my_edges;
                            }
                        }
                        ++my_parts;
                        claim[k] = found;
                    }
                    // ... and the warp walks the rest of a longer one, 32 parts at a time
                    uint32_t big = __ballot_sync(0xffffffffu, want[k] && !claim[k] && np[k] > PULL_LANE);
                    while (big) {
                        const int l = __ffs(big) - 1;
                        big &= big - 1u;
                        const uint32_t bs0 = __shfl_sync(0xffffffffu, s0[k], l);
                        const uint32_t bnp = __shfl_sync(0xffffffffu, np[k], l);
                        bool any = false;
                        for (uint32_t j0 = PULL_LANE; j0 < bnp && !any; j0 += 32u) {
                            const uint32_t j = j0 + lane;
                            bool found = false;
                            if (j < bnp) {
                                uint32_t c[K];
                                ld_part<K>(a.rvcol + (size_t)(bs0 + j) * K, c, pol);
#pragma unroll
                                for (int i = 0; i < K; ++i) {
                                    if (c[i] != NO_EDGE) {
                                        found |= a.dist[c[i]] == it;
                                        ++my_edges;
                                    }
                                }
                                ++my_parts;
                            }
                            any = __any_sync(0xffffffffu, found);
                        }
                        if ((uint32_t)l == lane) claim[k] = any;
                    }
                    if (claim[k]) {
                        a.dist[vv[k]] = it + 1u;  // no other writer: push and pull rounds never mix
                        ++my_updates;
                    }
                    const uint32_t mask = __ballot_sync(0xffffffffu, claim[k]);
                    if (mask) {
                        const uint32_t cn = __popc(mask);
                        if (wcnt + cn > (uint32_t)WCAP) {
                            if (pj > 0u) warp_flush(a, wbuf, wcnt, qnext, nxt, true, lane);
                            else warp_count(a, wbuf, wcnt, nxt, lane);
                            wcnt = 0;
                        }
                        if (claim[k]) wbuf[wcnt + __popc(mask & lanemask_lt)] = vv[k];
                        wcnt += cn;
                    }
                }
                // the vertices left unreached go on this round's list, one reservation per chunk (buffering
                // them per warp to reserve less often made R-MAT s22's first pull round 12 % slower)
                uint32_t lm[PVL], tot = 0;
#pragma unroll
                for (int k = 0; k < PVL; ++k) {
                    lm[k] = __ballot_sync(0xffffffffu, want[k] && !claim[k]);
                    tot += __popc(lm[k]);
                }
                if (tot) {
                    uint32_t lb = 0;
                    if (lane == 0) lb = atomicAdd(&ctrl->lcnt[pj % 3u], tot);
                    lb = __shfl_sync(0xffffffffu, lb, 0);
                    uint32_t* lwr = a.plist + (size_t)(pj & 1u) * a.n;
#pragma unroll
                    for (int k = 0; k < PVL; ++k) {
                        if (want[k] && !claim[k]) {
                            const uint32_t pos = lb + __popc(lm[k] & lanemask_lt);
                            if (pos < a.n) lwr[pos] = vv[k];  // one entry per vertex: always below n
                        }
                        lb += __popc(lm[k]);
                    }
                }
                continue;
            }
            const bool valid = p < a.P;
            uint32_t col[KH], wt[KH];
            const size_t row = (size_t)p * K;
            uint32_t d = 0;
            bool active = false;
            if (valid) {
                if (bfs_levels) {  // no owner or value load: the level is the round number
                    ld_part<KH>(a.vcol + row, col, pol);
                    d = it;
                    active = true;
                } else {
                    const uint32_t v = __ldg(&a.vowner[p]);
                    uint32_t pv = PSENT;
                    if (!TD) {  // DD: the part is almost surely live -- fetch its row alongside the owner's value
                        ld_part<KH>(a.vcol + row, col, pol);
                        if (OP != OP_BFS) load_weights<OP, KH>(a, row, wt, pol);
                        if (use_push) pv = __ldcg(&a.pushed[p]);  // written in earlier rounds by any CTA
                    }
                    // plain (L1-cached) value reads: the grid barrier's acquire makes the previous round's
                    // values visible; a value improved later in this round re-enqueues its vertex anyway
                    d = a.dist[v];
                    active = !unreached<OP>(d);
                    if (use_push && active) {
                        if (d == pv) active = false;
                        else a.pushed[p] = d;
                    }
                    if (TD && active) {
                        ld_part<KH>(a.vcol + row, col, pol);
                        if (OP != OP_BFS) load_weights<OP, KH>(a, row, wt, pol);
                    }
                }
                if (active) ++my_parts;
            }
            // A 16-slot row is taken in two halves where its targets, values and filter reads together do not
            // fit the registers (they spilled 150 bytes in this loop).
            const bool fetch = (dense || use_push) ? active : valid;
#pragma unroll 1
            for (int h = 0; h < K / KH; ++h) {
                if (h > 0 && fetch) {
                    ld_part<KH>(a.vcol + row + h * KH, col, pol);
                    if (OP != OP_BFS) load_weights<OP, KH>(a, row + h * KH, wt, pol);
                }
                // all filter reads are issued before the first atomic (the compiler may not move a load of
                // dist[] across an atomic on dist[]); a stale value only costs an atomic. Queued parts are
                // almost always live, so their filter reads do not wait for the owner's value.
                uint32_t cd[KH];
#pragma unroll
                for (int i = 0; i < KH; ++i) cd[i] = unfiltered ? INF : ((fetch && col[i] != NO_EDGE) ? a.dist[col[i]] : 0u);
                // What each slot would push, in the place of its weight, and the slots that pass the filter: the
                // filter values and the owner's value are dead before the first atomic (7 % of SSSP's time on
                // R-MAT s22, where they spilled).
                uint32_t hit = 0;
#pragma unroll
                for (int i = 0; i < KH; ++i) {
                    if (active && col[i] != NO_EDGE) {
                        ++my_edges;
                        const uint32_t nd = relax_value<OP>(d, OP == OP_BFS ? 1u : wt[i]);
                        if (OP != OP_BFS && better<OP>(nd, cd[i])) hit |= 1u << i;
                        if (OP != OP_BFS) wt[i] = nd;
                    }
                }
                // The atomics of ATB slots go out before any of their results is used: for each slot whose
                // filter read says the target improves, the value atomic and (DD, except BFS levels) the
                // claim on the target's round stamp are issued together. A won claim means the target
                // improved in this round -- by this lane, or by another after this lane's filter read (that
                // read is no older than the round's start, and values move one way only) -- so the winner
                // appends the target, whoever improved it, and a target improved in a round is appended
                // exactly once.
                // the 384-thread shape has room for a whole part
                constexpr int ATG = BKT ? 2 : (trav_tpb<OP>() == 384 ? 8 : ATOMIC_GROUP);
                constexpr int ATB = KH < ATG ? KH : ATG;
#pragma unroll
                for (int i0 = 0; i0 < KH; i0 += ATB) {
                    uint32_t prev[ATB], ex[ATB];
#pragma unroll
                    for (int j = 0; j < ATB; ++j) {
                        const int i = i0 + j;
                        prev[j] = 0u;
                        ex[j] = tag;
                        // (BFS, with registers to spare, filters here: 0.201 ms on R-MAT s22, 0.213 above)
                        if (OP == OP_BFS && active && col[i] != NO_EDGE && better<OP>(d + 1u, cd[i])) hit |= 1u << i;
                        if ((hit >> i) & 1u) {
                            prev[j] = atomic_improve<OP>(&a.dist[col[i]], OP == OP_BFS ? d + 1u : wt[i]);
                            if (!TD && !bfs_levels) ex[j] = atomicExch(&a.stamp[col[i]], tag);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < ATB; ++j) {
                        const int i = i0 + j;
                        bool claim = false, far = false;
                        uint32_t fkey = 0;
                        const uint32_t t = col[i];
                        if ((hit >> i) & 1u) {
                            const uint32_t nd = OP == OP_BFS ? d + 1u : wt[i];
                            const bool imp = better<OP>(nd, prev[j]);
                            if (imp) ++my_updates;
                            if (TD) {
                                if (imp) changed = 1u;
                            } else if (bfs_levels) {
                                claim = imp;  // atomicMin admits one first improvement
                            } else {
                                claim = ex[j] != tag;
                            }
                            if (BKT && claim) {
                                const uint32_t now = imp ? nd : prev[j];  // the target's value after this atomic
                                const uint32_t key = OP == OP_SSWP ? INF - now : now;
                                if (key >= T) {  // not in this bucket: wait in the far pile
                                    far = true;
                                    fkey = key;
                                    claim = false;
                                }
                            }
                        }
                        if (BKT) to_far(far, t, fkey);
                        if (!TD) {
                            const uint32_t mask = __ballot_sync(0xffffffffu, claim);
                            if (mask) {
                                const uint32_t c = __popc(mask);
                                if (wcnt + c > (uint32_t)WCAP) {
                                    warp_flush(a, wbuf, wcnt, qnext, nxt, can_bu || a.activity, lane);
                                    wcnt = 0;
                                }
                                if (claim) {
                                    wbuf[wcnt + __popc(mask & lanemask_lt)] = t;
                                    if (small) prefetch_l1(a.vstart + t);
                                }
                                wcnt += c;
                            }
                        }
                    }
                }
            }
        }
        if (TD) {
            if (__syncthreads_or(changed) && threadIdx.x == 0) atomicAdd(&ctrl->queued[nxt], 1ull);
        } else if (my_chunks <= 1u) {
            // One warp at most has anything, and makes its reservations itself: no CTA barriers in the rounds of a path
            // (16384 vertices: SSSP
            // 4.20 -> 3.90 us a round, bucketed 5.50 -> 5.07; R-MAT s22 SSSP, whose last rounds are small, 687 -> 672 us).
            if (BKT) {
                const uint32_t km = __reduce_min_sync(0xffffffffu, fkmin);
                uint32_t bits = 0, before = 0, tot = 0, base = 0;
                if (fcnt) tot = far_flags(a.fflag, fbuf, fcnt, lane, &bits, &before);
                if (lane == 0 && tot) base = atomicAdd(&ctrl->fcnt[fdst], tot);
                if (lane == 0 && km != 0xFFFFFFFFu) atomicMin(&ctrl->fmin[fdst], km);
                base = __shfl_sync(0xffffffffu, base, 0);
                if (fcnt) far_write(a, fbuf, bits, base + before, pile_dst, lane);
            }
            if (wcnt) {
                if (BFSBU && bu && pj == 0u) warp_count(a, wbuf, wcnt, nxt, lane);
                else warp_flush(a, wbuf, wcnt, qnext, nxt, can_bu || a.activity, lane);
            }
        } else {
            if (BKT) {  // the far buffers, one reservation per CTA
                constexpr int NW = T_TPB / 32;
                const uint32_t warp = threadIdx.x >> 5;
                uint32_t bits = 0, before = 0, tot = 0;
                if (fcnt) tot = far_flags(a.fflag, fbuf, fcnt, lane, &bits, &before);
                const uint32_t km = __reduce_min_sync(0xffffffffu, fkmin);
                if (lane == 0) {
                    s_fbase[warp] = tot;
                    s_fkey[warp] = km;
                }
                __syncthreads();
                if (warp == 0) {
                    const uint32_t c = lane < NW ? s_fbase[lane] : 0u;
                    const uint32_t k = __reduce_min_sync(0xffffffffu, lane < NW ? s_fkey[lane] : 0xFFFFFFFFu);
                    uint32_t inc = c;
#pragma unroll
                    for (int off = 1; off < 32; off <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
                        if (lane >= (uint32_t)off) inc += y;
                    }
                    uint32_t base = 0;
                    if (lane == 31u && inc) base = atomicAdd(&ctrl->fcnt[fdst], inc);
                    if (lane == 31u && k != 0xFFFFFFFFu) atomicMin(&ctrl->fmin[fdst], k);
                    base = __shfl_sync(0xffffffffu, base, 31);
                    if (lane < NW) s_fbase[lane] = base + inc - c;
                }
                __syncthreads();
                if (fcnt) far_write(a, fbuf, bits, s_fbase[warp] + before, pile_dst, lane);
            }
            cta_flush<T_TPB / 32>(a, wbuf, wcnt, BFSBU && bu && pj == 0u ? nullptr : qnext, nxt, can_bu || a.activity, lane, s_tot);
        }
        if ((it & 63u) == 63u) stat_round();
        if (BFSBU && bu) ++pj;
        if (!round_barrier(&ctrl->queued[nxt], &ctrl->bw, a.timeout_ns, &s_ctl[0])) break;
    }

finish:
    // ---- statistics
    stat_round();
    if (lane == 0) {
        const unsigned long long* st = s_stat[threadIdx.x >> 5];
        if (st[0]) atomicAdd(&ctrl->parts_processed, st[0]);
        if (st[1]) atomicAdd(&ctrl->edges_scanned, st[1]);
        if (st[2]) atomicAdd(&ctrl->updates, st[2]);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctrl->iterations = it;
        ctrl->done = all_done ? 1u : 0u;
        if (BFSBU) ctrl->pull_rounds = pj;
    }
}

// Reached-set statistics: n_r and m_r (out-edges of reached vertices).
// Reached: BFS/SSSP value != DIST_INFINITY, SSWP value != 0 (the source holds DIST_INFINITY), CC all.
template <int OP>
__global__ void k_reached(const uint32_t* __restrict__ dist, const uint32_t* __restrict__ deg, uint32_t n,
                          unsigned long long* out) {
    unsigned long long nr = 0, mr = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t d = dist[v];
        bool r;
        if (OP == OP_CC) r = true;
        else if (OP == OP_SSWP) r = d != 0u;
        else r = d != INF;
        if (r) {
            ++nr;
            mr += deg[v];
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        nr += __shfl_down_sync(0xffffffffu, nr, off);
        mr += __shfl_down_sync(0xffffffffu, mr, off);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&out[0], nr);
        atomicAdd(&out[1], mr);
    }
}

// End of a run: the values into the caller's device array (out may be null) and the reached-set statistics
// in one pass, skipped when the run gave up (its output stays untouched). One pair of atomics per CTA: with
// one per warp, 20 000 of them on two words took as long as the pass.
template <int OP>
__global__ void __launch_bounds__(512) k_finish(const uint32_t* __restrict__ dist, const uint32_t* __restrict__ deg,
                                                uint32_t n, const BarrierWords* bw, uint32_t* __restrict__ out,
                                                int out16, unsigned long long* stats) {
    __shared__ unsigned long long s_n[16], s_m[16];
    const uint32_t status = bw->status;
    if (status != DEV_OK && status != DEV_ITER_CAP) return;
    unsigned long long nr = 0, mr = 0;
    auto one = [&](uint32_t d, uint32_t g) {
        const bool r = OP == OP_CC || (OP == OP_SSWP ? d != 0u : d != INF);
        nr += r ? 1u : 0u;
        mr += r ? g : 0u;
    };
    const uint32_t n4 = n / 4u, t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (uint32_t i = t0; i < n4; i += step) {  // both arrays are 256-byte aligned
        const uint4 d = reinterpret_cast<const uint4*>(dist)[i], g = reinterpret_cast<const uint4*>(deg)[i];
        one(d.x, g.x);
        one(d.y, g.y);
        one(d.z, g.z);
        one(d.w, g.w);
        if (out16) {
            reinterpret_cast<uint4*>(out)[i] = d;
        } else if (out) {
            out[4u * i] = d.x;
            out[4u * i + 1u] = d.y;
            out[4u * i + 2u] = d.z;
            out[4u * i + 3u] = d.w;
        }
    }
    for (uint32_t v = 4u * n4 + t0; v < n; v += step) {
        one(dist[v], deg[v]);
        if (out) out[v] = dist[v];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        nr += __shfl_down_sync(0xffffffffu, nr, off);
        mr += __shfl_down_sync(0xffffffffu, mr, off);
    }
    if ((threadIdx.x & 31u) == 0) {
        s_n[threadIdx.x >> 5] = nr;
        s_m[threadIdx.x >> 5] = mr;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 16; ++w) {
            nr += s_n[w];
            mr += s_m[w];
        }
        atomicAdd(&stats[0], nr);
        atomicAdd(&stats[1], mr);
    }
}

template <int OP, int K, bool TD>
eeg_status launch_one(const TravArgs& args, int device, uint32_t blocks_per_sm_req, cudaStream_t st) {
    constexpr bool CAN_MODE = !TD && (OP == OP_SSSP || OP == OP_SSWP || OP == OP_BFS);
    // bucketed rounds; BFS: pull rounds, from the source in one launch on a graph with transposed parts
    const bool mode = CAN_MODE && !args.seed_all && (OP == OP_BFS ? args.rvstart && args.rounds_limit == 0 : args.delta != 0u);
    auto kern = mode ? k_traverse<OP, K, TD, CAN_MODE> : k_traverse<OP, K, TD, false>;
    constexpr int T_TPB = trav_tpb<OP>();
    // The filter reads of dist[] are L1 hits in part, and L1 is what shared memory leaves: ask for the
    // smallest carveout that still holds the two CTAs per SM the kernel is built for (R-MAT s22: SSSP
    // 0.725 -> 0.706 ms, SSWP 0.726 -> 0.709, CC 1.215 -> 1.193 against the CUDA driver's default). The hint
    // and the occupancy belong to the kernel and the device: asked for once (four runtime calls less per run).
    static std::atomic<int> resident[2][64];
    std::atomic<int>& slot = resident[mode ? 1 : 0][device & 63];
    int per_sm = slot.load(std::memory_order_acquire);
    if (per_sm == 0) {
        EEG_TRY(prefer_l1(kern, 2, device));
        EEG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, T_TPB, 0));
        if (per_sm > 0 && device < 64) slot.store(per_sm, std::memory_order_release);
    }
    if (per_sm <= 0) {
        set_last_error("traversal kernel does not fit on an SM");
        return EEG_ERR_CUDA;
    }
    if (blocks_per_sm_req > 0 && (int)blocks_per_sm_req < per_sm) per_sm = (int)blocks_per_sm_req;
    uint64_t blocks = (uint64_t)per_sm * sm_count(device);
    const uint64_t work = std::max<uint64_t>(args.P, args.n);
    const uint64_t need = (work + T_TPB - 1) / T_TPB;
    if (need < blocks) blocks = std::max<uint64_t>(need, 1);
    TravArgs a = args;
    void* params[] = {(void*)&a};
    EEG_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)blocks), dim3(T_TPB), params, 0, st));
    return EEG_OK;
}

template <int OP, bool TD>
eeg_status launch_k(const TravArgs& args, uint32_t K, int device, uint32_t bps, cudaStream_t st) {
    switch (K) {
        case 4: return launch_one<OP, 4, TD>(args, device, bps, st);
        case 8: return launch_one<OP, 8, TD>(args, device, bps, st);
        case 16: return launch_one<OP, 16, TD>(args, device, bps, st);
        default: set_last_error("K must be 4, 8 or 16"); return EEG_ERR_UNSUPPORTED;
    }
}

// Launch the traversal of one operator; each is defined in its own translation unit traverse_<op>.cu.
eeg_status launch_bfs(const TravArgs& args, bool td, uint32_t K, int device, uint32_t bps, cudaStream_t st);
eeg_status launch_sssp(const TravArgs& args, bool td, uint32_t K, int device, uint32_t bps, cudaStream_t st);
eeg_status launch_sswp(const TravArgs& args, bool td, uint32_t K, int device, uint32_t bps, cudaStream_t st);
eeg_status launch_cc(const TravArgs& args, bool td, uint32_t K, int device, uint32_t bps, cudaStream_t st);

}  // namespace trav
}  // namespace eeg
