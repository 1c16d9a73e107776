// batch.cu -- many BFS/SSSP/SSWP queries, over many graphs of uneven size, in one launch.
//
// No counterpart kernel in the reference: there, every query is a separate eegraph_<algo> call with
// its own host loop (src/main.cu:74-281 runs them one after another).
//
// One launch of k_batch runs a device work queue of queries, largest graphs first (the host sorts them).
// The first `nbig` queries run one after another on the whole grid (rounds separated by the bounded
// grid barrier); the grid is made of thread-block clusters, and then each cluster takes the next query,
// runs the whole traversal with its CTAs -- rounds separated by the hardware cluster barrier, frontier =
// a queue of part ids, the warp-aggregated append of the single-query kernel -- and takes the next one.
// The autotuner picks the cluster size and nbig.
// The launch (with the reset of the work counter) is captured once in a CUDA graph and replayed.
// Queries run the SYNC_PUSH_DD schedule from their source; results equal every variant's.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <numeric>
#include <vector>

#include "traverse.cuh"

namespace cg = cooperative_groups;

namespace eeg {
namespace batch {

constexpr int B_TPB = 512;
struct BGraph {
    uint32_t n, P, K, pad;
    const uint32_t* vstart;
    const uint32_t* vowner;
    const uint32_t* vcol;
    const uint32_t* vw;
};
struct BQuery {
    uint32_t graph, op, source, input_index;
    unsigned long long out_off;
};
struct BCtrl {
    uint32_t qparts[3];
    uint32_t tag;  // running round tag of this cluster (persists across launches)
};
struct BArgs {
    const BGraph* graphs;
    const BQuery* queries;
    uint32_t nq;
    uint32_t max_rounds;
    uint32_t* next;     // work counter
    uint32_t* out;      // output arena
    uint32_t* rounds;   // per query (input order)
    unsigned long long* times;  // per query (input order): start and end (%globaltimer ns) and cluster id
    uint32_t* q0;       // per cluster: 2 * qcap part ids
    uint32_t* stamp;    // per cluster: scap stamps
    BCtrl* ctrl;        // per cluster
    uint64_t qcap, scap;
    uint32_t nbig;      // queries [0, nbig) of the size order run on the whole grid first
    uint32_t pad;
    uint32_t* tq;       // whole-grid queries: 2 * qcap part ids
    uint32_t* tstamp;   //                     scap stamps
    BCtrl* tctrl;
    BarrierWords* bw;   // grid barrier of the whole-grid phase
    uint64_t timeout_ns;
    uint32_t* err;      // set when a queue would exceed its capacity (cannot happen; reported)
};

// The CTAs that run one query together: a thread-block cluster (rounds separated by the hardware
// cluster barrier), or the whole grid (rounds separated by the bounded grid barrier).
struct ClusterTeam {
    cg::cluster_group cl;
    __device__ uint32_t thread_rank() const { return cl.block_rank() * B_TPB + threadIdx.x; }
    __device__ uint32_t nthreads() const { return cl.num_blocks() * B_TPB; }
    __device__ uint32_t cta_rank() const { return cl.block_rank(); }
    __device__ uint32_t ncta() const { return cl.num_blocks(); }
    __device__ bool leader_cta() const { return cl.block_rank() == 0; }
    __device__ bool sync() {
        cl.sync();
        return true;
    }
};
struct GridTeam {
    BarrierWords* bw;
    uint32_t* epoch;
    uint64_t timeout_ns;
    __device__ uint32_t thread_rank() const { return blockIdx.x * B_TPB + threadIdx.x; }
    __device__ uint32_t nthreads() const { return gridDim.x * B_TPB; }
    __device__ uint32_t cta_rank() const { return blockIdx.x; }
    __device__ uint32_t ncta() const { return gridDim.x; }
    __device__ bool leader_cta() const { return blockIdx.x == 0; }
    __device__ bool sync() { return grid_barrier(bw, *epoch, timeout_ns); }
};

constexpr uint32_t ABORTED = 0x80000000u;  // flag beside the rounds run_query returns

// The query a CTA works on, in shared memory: its fields are read where they are used (a broadcast) instead
// of living in registers, or on the stack as references to the kernel's parameters and locals. The bodies still spill
// (16 to 216 bytes of stores, 56 to 328 of loads at 64 registers; with the older expansion 60 to 300).
struct QCtx {
    const uint32_t *vstart, *vowner, *vcol, *vw;
    uint32_t* dist;
    uint32_t *qa, *qb, *stamp;
    BCtrl* ctrl;
    uint32_t* err;
    uint32_t n, P, source, max_rounds, tag0;
};

// One query (SYNC_PUSH_DD from its source) on `team`; returns its rounds, with ABORTED set when a grid barrier
// gave up. Round r uses stamp tag0 + r + 1. Not inlined, so that each (OP, K, team) body gets its own registers.
template <int OP, int K, class Team>
__device__ __noinline__ uint32_t run_query(const QCtx& c, Team team, uint32_t* wbuf) {
    constexpr int KH = K > 8 ? 8 : K;  // slots of a part expanded at a time (trav::k_traverse)
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t crank = team.cta_rank(), ncta = team.ncta();
    __shared__ uint32_t s_next[2];  // per round (alternating): next of this CTA's 32-entry chunks
    if (threadIdx.x == 0) s_next[0] = s_next[1] = 0u;  // ordered before use by the team barrier below
    const uint64_t pol = l2_evict_first_policy();
    {
        const uint32_t tsize = team.nthreads(), n = c.n, source = c.source;
        uint32_t* dist = c.dist;
        for (uint32_t v = team.thread_rank(); v < n; v += tsize) dist[v] = trav::init_value<OP>(v, source);
        if (team.leader_cta()) {
            const uint32_t s0 = c.vstart[source], s1 = c.vstart[source + 1];
            for (uint32_t j = threadIdx.x; j < s1 - s0; j += B_TPB) c.qa[j] = s0 + j;
            if (threadIdx.x == 0) {
                c.ctrl->qparts[0] = s1 - s0;
                c.ctrl->qparts[1] = 0u;
                c.ctrl->qparts[2] = 0u;
            }
        }
    }
    if (!team.sync()) return ABORTED;
    uint32_t it = 0;
    __shared__ uint32_t s_len;  // the round's queue length, read once per CTA
    for (;; ++it) {
        const uint32_t cur = it % 3u, nxt = (it + 1u) % 3u, old = (it + 2u) % 3u;
        if (threadIdx.x == 0) s_len = *(volatile uint32_t*)&c.ctrl->qparts[cur];
        __syncthreads();
        uint32_t len = s_len;
        if (len == 0u || it >= c.max_rounds) break;
        if (len > c.P) {  // one claim per vertex per round bounds a round by P parts; never read past it
            if (threadIdx.x == 0) atomicOr(c.err, 1u);
            len = c.P;
        }
        if (team.leader_cta() && threadIdx.x == 0) c.ctrl->qparts[old] = 0u;
        const uint32_t* qcur = (it & 1u) ? c.qb : c.qa;
        uint32_t* qnext = (it & 1u) ? c.qa : c.qb;
        uint32_t wcnt = 0;
        // this CTA's strided share of the round's 32-entry chunks, drawn by its warps from a shared
        // counter; the other counter is reset for the next round (ordered by the team barrier)
        if (threadIdx.x == 0) s_next[(it + 1u) & 1u] = 0u;
        const uint32_t nch = (len + 31u) / 32u;
        const uint32_t my_chunks = nch > crank ? (nch - crank + ncta - 1u) / ncta : 0u;
        // pipelined by one chunk: the next chunk's queue entries load while this one is expanded
        auto draw = [&](uint32_t& pn) -> uint32_t {
            uint32_t ci = 0;
            if (lane == 0) ci = atomicAdd(&s_next[it & 1u], 1u);
            ci = __shfl_sync(0xffffffffu, ci, 0);
            const uint32_t idx = (crank + ci * ncta) * 32u + lane;
            pn = (ci < my_chunks && idx < len) ? qcur[idx] : 0xFFFFFFFFu;
            return ci;
        };
        uint32_t p_next;
        uint32_t ci_next = draw(p_next);
        for (;;) {
            if (ci_next >= my_chunks) break;
            const uint32_t p = p_next;
            ci_next = draw(p_next);
            const bool valid = p < c.P;
            uint32_t col[KH], wt[KH];
            uint32_t d = 0;
            bool active = false;
            if (valid) {
                ld_part<KH>(c.vcol + (size_t)p * K, col, pol);
                if (OP == OP_BFS) {  // source-seeded BFS: a round's queue holds the vertices at level `it`
                    d = it;
                    active = true;
                } else {
                    const uint32_t v = __ldg(&c.vowner[p]);
                    ld_part<KH>(c.vw + (size_t)p * K, wt, pol);
                    // plain (L1-cached) value reads, as in k_traverse: the team barrier's acquire makes the
                    // previous round's values visible, and a value improved later re-enqueues its vertex
                    d = c.dist[v];
                    active = !trav::unreached<OP>(d);
                }
            }
#pragma unroll 1
            for (int h = 0; h < K / KH; ++h) {
                if (h > 0 && valid) {
                    ld_part<KH>(c.vcol + (size_t)p * K + h * KH, col, pol);
                    if (OP != OP_BFS) ld_part<KH>(c.vw + (size_t)p * K + h * KH, wt, pol);
                }
                // every filter read before the first atomic; then what each slot would push, in the place of
                // its weight, and the slots that pass the filter
                uint32_t cd[KH];
                uint32_t* dist = c.dist;
#pragma unroll
                for (int i = 0; i < KH; ++i) cd[i] = (valid && col[i] != NO_EDGE) ? dist[col[i]] : 0u;
                uint32_t hit = 0;
#pragma unroll
                for (int i = 0; i < KH; ++i) {
                    if (active && col[i] != NO_EDGE) {
                        const uint32_t nd = trav::relax_value<OP>(d, OP == OP_BFS ? 1u : wt[i]);
                        if (trav::better<OP>(nd, cd[i])) hit |= 1u << i;
                        if (OP != OP_BFS) wt[i] = nd;
                    }
                }
                // the atomics of a group of slots go out before any of their results is used; a won claim
                // on the round stamp means the target improved in this round (by this lane or after its
                // filter read), so the winner appends it (the single-query kernel's rule)
                constexpr int ATB = KH < trav::ATOMIC_GROUP ? KH : trav::ATOMIC_GROUP;
#pragma unroll
                for (int i0 = 0; i0 < KH; i0 += ATB) {
                    uint32_t prev[ATB], ex[ATB];
                    const uint32_t tag = c.tag0 + it + 1u;
#pragma unroll
                    for (int j = 0; j < ATB; ++j) {
                        const int i = i0 + j;
                        prev[j] = 0u;
                        ex[j] = tag;
                        if ((hit >> i) & 1u) {
                            prev[j] = trav::atomic_improve<OP>(&dist[col[i]], OP == OP_BFS ? d + 1u : wt[i]);
                            if (OP != OP_BFS) ex[j] = atomicExch(&c.stamp[col[i]], tag);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < ATB; ++j) {
                        const int i = i0 + j;
                        // BFS: atomicMin admits one first improvement
                        const bool claim = ((hit >> i) & 1u) &&
                                           (OP == OP_BFS ? trav::better<OP>(d + 1u, prev[j]) : ex[j] != tag);
                        const uint32_t mask = __ballot_sync(0xffffffffu, claim);
                        if (mask) {
                            const uint32_t cn = __popc(mask);
                            if (wcnt + cn > (uint32_t)trav::WCAP) {
                                trav::warp_append(c.vstart, &c.ctrl->qparts[nxt], wbuf, wcnt, qnext, lane, c.P);
                                wcnt = 0;
                            }
                            if (claim) wbuf[wcnt + __popc(mask & ((1u << lane) - 1u))] = col[i];
                            wcnt += cn;
                        }
                    }
                }
            }
        }
        if (wcnt) trav::warp_append(c.vstart, &c.ctrl->qparts[nxt], wbuf, wcnt, qnext, lane, c.P);
        if (!team.sync()) return it | ABORTED;
    }
    // every CTA has read the final (empty) queue length before the leader initialises the next query
    if (!team.sync()) return it | ABORTED;
    return it;
}

// The query's context into shared memory, then the body for its operator and part size. Called by all threads.
template <class Team>
__device__ __forceinline__ uint32_t dispatch(const BArgs& a, const BQuery& q, Team team, uint32_t* qa, uint32_t* qb,
                                             uint32_t* stamp, BCtrl* ctrl, uint32_t tag, uint32_t* wbuf, QCtx* c) {
    const uint32_t K = a.graphs[q.graph].K;
    __syncthreads();  // the last query's readers are done
    if (threadIdx.x == 0) {
        const BGraph g = a.graphs[q.graph];
        c->vstart = g.vstart;
        c->vowner = g.vowner;
        c->vcol = g.vcol;
        c->vw = g.vw;
        c->dist = a.out + q.out_off;
        c->qa = qa;
        c->qb = qb;
        c->stamp = stamp;
        c->ctrl = ctrl;
        c->err = a.err;
        c->n = g.n;
        c->P = g.P;
        c->source = q.source;
        c->max_rounds = a.max_rounds;
        c->tag0 = tag;
    }
    __syncthreads();
#define EEG_BATCH_K(OPV)                                              \
    switch (K) {                                                      \
        case 4: return run_query<OPV, 4, Team>(*c, team, wbuf);       \
        case 16: return run_query<OPV, 16, Team>(*c, team, wbuf);     \
        default: return run_query<OPV, 8, Team>(*c, team, wbuf);      \
    }
    switch (q.op) {
        case OP_BFS: EEG_BATCH_K(OP_BFS)
        case OP_SSSP: EEG_BATCH_K(OP_SSSP)
        default: EEG_BATCH_K(OP_SSWP)
    }
#undef EEG_BATCH_K
}

__device__ __forceinline__ void record(const BArgs& a, const BQuery& q, uint32_t rounds, unsigned long long t0,
                                       unsigned long long who) {
    a.rounds[q.input_index] = rounds;
    a.times[3 * (size_t)q.input_index] = t0;
    a.times[3 * (size_t)q.input_index + 1] = global_timer_ns();
    a.times[3 * (size_t)q.input_index + 2] = who;
}

__global__ void __launch_bounds__(B_TPB, 2) k_batch(BArgs a) {
    __shared__ uint32_t s_qi;
    __shared__ uint32_t s_buf[B_TPB / 32][trav::WCAP];
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t csize = cl.num_blocks(), crank = cl.block_rank();
    const uint32_t cid = blockIdx.x / csize;
    __shared__ QCtx s_ctx;
    uint32_t* wbuf = s_buf[threadIdx.x >> 5];

    // phase 1: the largest queries, one after another, each on the whole grid
    const uint32_t nbig = min(a.nbig, a.nq);
    if (nbig) {
        uint32_t epoch = 0;
        uint32_t ttag = *(volatile uint32_t*)&a.tctrl->tag;
        GridTeam gt{a.bw, &epoch, a.timeout_ns};
        for (uint32_t qi = 0; qi < nbig; ++qi) {
            const BQuery q = a.queries[qi];
            const unsigned long long t0 = global_timer_ns();
            const uint32_t rounds = dispatch(a, q, gt, a.tq, a.tq + a.qcap, a.tstamp, a.tctrl, ttag, wbuf, &s_ctx);
            ttag += (rounds & ~ABORTED) + 1u;
            if (rounds & ABORTED) break;
            if (blockIdx.x == 0 && threadIdx.x == 0) record(a, q, rounds, t0, ~0ull);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) a.tctrl->tag = ttag;
    }

    // phase 2: the rest from the work counter, one query per cluster
    uint32_t* qa = a.q0 + (size_t)cid * 2 * a.qcap;
    uint32_t* qb = qa + a.qcap;
    uint32_t* stamp = a.stamp + (size_t)cid * a.scap;
    BCtrl* ctrl = a.ctrl + cid;
    uint32_t tag = *(volatile uint32_t*)&ctrl->tag;
    ClusterTeam ct{cl};
    for (;;) {
        if (crank == 0 && threadIdx.x == 0) s_qi = nbig + atomicAdd(a.next, 1u);
        cl.sync();
        const uint32_t qi = *cl.map_shared_rank(&s_qi, 0);
        cl.sync();  // every CTA has read the index before the leader draws the next one
        if (qi >= a.nq) break;
        const BQuery q = a.queries[qi];
        const unsigned long long t0 = global_timer_ns();
        const uint32_t rounds = dispatch(a, q, ct, qa, qb, stamp, ctrl, tag, wbuf, &s_ctx);
        tag += rounds + 1u;
        if (crank == 0 && threadIdx.x == 0) record(a, q, rounds, t0, cid);
    }
    if (crank == 0 && threadIdx.x == 0) ctrl->tag = tag;
}

}  // namespace batch
}  // namespace eeg

using namespace eeg;
using namespace eeg::batch;

struct eeg_batch {
    int device = 0;
    std::vector<eeg_vgraph*> graphs;
    BGraph* d_graphs = nullptr;
    BQuery* d_queries = nullptr;
    uint32_t nq = 0;
    std::vector<unsigned long long> out_off;  // per query, input order
    unsigned long long out_words = 0;
    uint32_t* d_next = nullptr;
    uint32_t* d_rounds = nullptr;
    unsigned long long* d_times = nullptr;
    uint32_t* d_q = nullptr;
    uint32_t* d_stamp = nullptr;
    BCtrl* d_ctrl = nullptr;
    uint64_t qcap = 0, scap = 0;
    uint32_t nclusters = 0, csize = 0, max_rounds = 0;
    uint32_t nbig = 0;                 // queries run on the whole grid first
    uint32_t* d_tq = nullptr;          // their queues and stamps
    uint32_t* d_tstamp = nullptr;
    BCtrl* d_tctrl = nullptr;
    BarrierWords* d_bw = nullptr;
    uint32_t* d_err = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaGraphExec_t exec = nullptr;
    uint32_t* captured_out = nullptr;
};

namespace {

void free_scratch(eeg_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    b->captured_out = nullptr;
    cudaFree(b->d_q);
    cudaFree(b->d_stamp);
    cudaFree(b->d_ctrl);
    b->d_q = b->d_stamp = nullptr;
    b->d_ctrl = nullptr;
    b->nclusters = 0;
}

eeg_status launch(eeg_batch* b, uint32_t* out) {
    BArgs a{};
    a.graphs = b->d_graphs;
    a.queries = b->d_queries;
    a.nq = b->nq;
    a.max_rounds = b->max_rounds;
    a.next = b->d_next;
    a.out = out;
    a.rounds = b->d_rounds;
    a.times = b->d_times;
    a.q0 = b->d_q;
    a.stamp = b->d_stamp;
    a.ctrl = b->d_ctrl;
    a.qcap = b->qcap;
    a.scap = b->scap;
    a.nbig = b->nbig;
    a.tq = b->d_tq;
    a.tstamp = b->d_tstamp;
    a.tctrl = b->d_tctrl;
    a.bw = b->d_bw;
    a.timeout_ns = 1000ull * 1000000ull;  // a round of one query takes microseconds
    a.err = b->d_err;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(b->nclusters * b->csize);
    cfg.blockDim = dim3(B_TPB);
    cfg.stream = b->st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = b->csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    EEG_CUDA(cudaMemsetAsync(b->d_next, 0, sizeof(uint32_t), b->st));
    EEG_CUDA(cudaMemsetAsync(b->d_bw, 0, sizeof(BarrierWords), b->st));
    EEG_CUDA(cudaMemsetAsync(b->d_err, 0, sizeof(uint32_t), b->st));
    EEG_CUDA(cudaLaunchKernelEx(&cfg, k_batch, a));
    return EEG_OK;
}

// (Re)size the per-cluster working memory for cluster size `csize` and capture the launch.
eeg_status configure(eeg_batch* b, uint32_t csize) {
    if (csize != 1 && csize != 2 && csize != 4 && csize != 8) {
        set_last_error("cluster size must be 1, 2, 4 or 8");
        return EEG_ERR_UNSUPPORTED;
    }
    free_scratch(b);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(csize);
    cfg.blockDim = dim3(B_TPB);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int dev = 0;
    EEG_CUDA(cudaGetDevice(&dev));
    EEG_TRY(prefer_l1(k_batch, 2, dev));  // the filter reads' L1 hits, as for the single-graph kernels
    int nclusters = 0;
    EEG_CUDA(cudaOccupancyMaxActiveClusters(&nclusters, k_batch, &cfg));
    if (nclusters <= 0) {
        set_last_error("no cluster of this size fits on the device");
        return EEG_ERR_UNSUPPORTED;
    }
    b->csize = csize;
    b->nclusters = (uint32_t)std::min<int>(nclusters, (int)std::max<uint32_t>(b->nq, 1));
    EEG_CUDA(cudaMalloc((void**)&b->d_q, sizeof(uint32_t) * 2 * b->qcap * b->nclusters));
    EEG_CUDA(cudaMalloc((void**)&b->d_stamp, sizeof(uint32_t) * b->scap * b->nclusters));
    EEG_CUDA(cudaMalloc((void**)&b->d_ctrl, sizeof(BCtrl) * b->nclusters));
    EEG_CUDA(cudaMemsetAsync(b->d_stamp, 0, sizeof(uint32_t) * b->scap * b->nclusters, b->st));
    EEG_CUDA(cudaMemsetAsync(b->d_ctrl, 0, sizeof(BCtrl) * b->nclusters, b->st));
    return EEG_OK;
}

// CTAs per query when the caller leaves the choice open. A query of w edges takes about 39 us of rounds and
// 1.75 ns w (BFS: 0.4 of it) divided by its CTAs; a batch takes at least its longest query, and all queries'
// CTA time over the device's CTAs. The longest query of few or uneven ones is what a small cluster waits
// for, and many small queries pay their rounds once per CTA. Measured against 4 for every batch: 64 graphs of
// up to 2^18 vertices 4.0 -> 2.8 ms (8), 3 graphs of 2^18-2^20 8.6 -> 4.3 (8), 900 queries on graphs of up
// to 2^12 0.75 -> 0.40 (1). 4 stays unless another size promises 15 % (between close ones the model is no
// guide: 148 queries, 8 predicted 4 % faster, 0.28 -> 0.39 ms). The two constants are measured on a GB300 (152 SMs), as
// is everything here: 14 batches of 1 to 900 queries, 2^10 to 2^20 vertices.
//   More clusters need more working memory: one of 4 is not left for a size that needs over a sixteenth of the device's.
uint32_t choose_cluster(const eeg_batch* b, const std::vector<BQuery>& queries) {
    const double ctas = 2.0 * sm_count(b->device);
    auto model = [&](uint32_t c) {
        double longest = 0.0, total = 0.0;
        for (const BQuery& q : queries) {
            const double w = 1.75e-3 * (double)b->graphs[q.graph]->m * (q.op == OP_BFS ? 0.4 : 1.0);
            longest = std::max(longest, 39.0 + w / c);
            total += 39.0 * c + w;
        }
        return std::max(longest, total / ctas);
    };
    auto scratch = [&](uint32_t c) {
        return (double)std::min<size_t>((size_t)(ctas / c), queries.size()) * 4.0 * (2.0 * (double)b->qcap + (double)b->scap);
    };
    size_t free_bytes = 0, total_bytes = 0;
    if (cudaMemGetInfo(&free_bytes, &total_bytes) != cudaSuccess) (void)cudaGetLastError();
    uint32_t best = 4;
    double t = 0.85 * model(4);
    for (uint32_t c : {1u, 2u, 8u}) {
        if (scratch(c) > std::max(scratch(4), (double)total_bytes / 16.0)) continue;
        const double tc = model(c);
        if (tc < t) {
            t = tc;
            best = c;
        }
    }
    return best;
}

eeg_status capture(eeg_batch* b, uint32_t* out) {
    if (b->exec && b->captured_out == out) return EEG_OK;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    cudaGraph_t graph = nullptr;
    EEG_CUDA(cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal));
    eeg_status s = launch(b, out);
    cudaError_t e = cudaStreamEndCapture(b->st, &graph);
    if (s != EEG_OK) {
        if (graph) cudaGraphDestroy(graph);
        return s;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture", __FILE__, __LINE__);
    e = cudaGraphInstantiate(&b->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate", __FILE__, __LINE__);
    b->captured_out = out;
    return EEG_OK;
}

}  // namespace

extern "C" {

EEG_API eeg_status eeg_batch_create(eeg_vgraph* const* graphs, uint32_t num_graphs, eeg_batch** out) {
    if (!out || !graphs || num_graphs == 0) {
        set_last_error("eeg_batch_create: no graphs");
        return EEG_ERR_INVALID;
    }
    *out = nullptr;
    eeg_batch* b = new eeg_batch();
    EEG_CUDA(cudaGetDevice(&b->device));
    std::vector<BGraph> hg(num_graphs);
    for (uint32_t i = 0; i < num_graphs; ++i) {
        eeg_vgraph* vg = graphs[i];
        if (!vg || vg->device != b->device || !vg->fwd_parts || (!vg->fwd.vw && vg->fwd.P)) {
            delete b;
            set_last_error("eeg_batch_create: graph missing, on another device, without weights or without "
                           "forward parts (EEG_VG_REVERSE_ONLY)");
            return EEG_ERR_INVALID;
        }
        b->graphs.push_back(vg);
        hg[i] = BGraph{vg->n, (uint32_t)vg->fwd.P, vg->K, 0, vg->fwd.vstart, vg->fwd.vowner, vg->fwd.vcol, vg->fwd.vw};
        b->qcap = std::max<uint64_t>(b->qcap, std::max<uint64_t>(vg->fwd.P, 1));
        b->scap = std::max<uint64_t>(b->scap, std::max<uint32_t>(vg->n, 1));
    }
    auto fail = [&](eeg_status s) {
        eeg_batch_destroy(b);
        return s;
    };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreate(&b->ev[0])) != cudaSuccess || (e = cudaEventCreate(&b->ev[1])) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_graphs, sizeof(BGraph) * num_graphs)) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_next, sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_tq, sizeof(uint32_t) * 2 * b->qcap)) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_tstamp, sizeof(uint32_t) * b->scap)) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_tctrl, sizeof(BCtrl))) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_bw, sizeof(BarrierWords))) != cudaSuccess ||
        (e = cudaMalloc((void**)&b->d_err, sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMemset(b->d_tstamp, 0, sizeof(uint32_t) * b->scap)) != cudaSuccess ||
        (e = cudaMemset(b->d_tctrl, 0, sizeof(BCtrl))) != cudaSuccess ||
        (e = cudaMemcpy(b->d_graphs, hg.data(), sizeof(BGraph) * num_graphs, cudaMemcpyHostToDevice)) != cudaSuccess)
        return fail(cuda_fail(e, "eeg_batch_create", __FILE__, __LINE__));
    *out = b;
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_set_queries(eeg_batch* b, const eeg_query* queries, uint32_t nq, uint32_t cluster_size,
                                         unsigned long long* out_words) {
    if (!b || (nq && !queries)) {
        set_last_error("eeg_batch_set_queries: null argument");
        return EEG_ERR_INVALID;
    }
    EEG_CUDA(cudaSetDevice(b->device));
    std::vector<BQuery> hq(nq);
    b->out_off.assign(nq, 0);
    unsigned long long off = 0;
    uint32_t max_n = 1;
    for (uint32_t i = 0; i < nq; ++i) {
        const eeg_query& q = queries[i];
        if (q.graph >= b->graphs.size() || (q.algo != EEG_BFS && q.algo != EEG_SSSP && q.algo != EEG_SSWP) ||
            q.source >= b->graphs[q.graph]->n) {
            set_last_error("eeg_batch_set_queries: query " + std::to_string(i) +
                           " has a bad graph index, algorithm (BFS/SSSP/SSWP) or source");
            return EEG_ERR_INVALID;
        }
        const int op = q.algo == EEG_BFS ? OP_BFS : (q.algo == EEG_SSSP ? OP_SSSP : OP_SSWP);
        hq[i] = BQuery{q.graph, (uint32_t)op, q.source, i, off};
        b->out_off[i] = off;
        off += b->graphs[q.graph]->n;
        max_n = std::max(max_n, b->graphs[q.graph]->n);
    }
    // largest graphs first, so the long queries start early and the short ones fill the tail
    std::stable_sort(hq.begin(), hq.end(), [&](const BQuery& x, const BQuery& y) {
        return b->graphs[x.graph]->fwd.P > b->graphs[y.graph]->fwd.P;
    });
    cudaFree(b->d_queries);
    cudaFree(b->d_rounds);
    cudaFree(b->d_times);
    b->d_queries = nullptr;
    b->d_rounds = nullptr;
    b->d_times = nullptr;
    EEG_CUDA(cudaMalloc((void**)&b->d_queries, sizeof(BQuery) * std::max<uint32_t>(nq, 1)));
    EEG_CUDA(cudaMalloc((void**)&b->d_rounds, sizeof(uint32_t) * std::max<uint32_t>(nq, 1)));
    EEG_CUDA(cudaMalloc((void**)&b->d_times, 3 * sizeof(unsigned long long) * std::max<uint32_t>(nq, 1)));
    if (nq) EEG_CUDA(cudaMemcpy(b->d_queries, hq.data(), sizeof(BQuery) * nq, cudaMemcpyHostToDevice));
    b->nq = nq;
    b->out_words = off;
    b->max_rounds = max_n + 2u;
    if (out_words) *out_words = off;
    const uint32_t size = cluster_size ? cluster_size : choose_cluster(b, hq);
    eeg_status s = configure(b, size);
    if (s != EEG_OK && cluster_size == 0 && size != 4) {  // the choice was ours: 4 if that fits
        (void)cudaGetLastError();
        s = configure(b, 4);
    }
    return s;
}

EEG_API eeg_status eeg_batch_query_offset(const eeg_batch* b, uint32_t query, unsigned long long* offset) {
    if (!b || !offset || query >= b->nq) {
        set_last_error("eeg_batch_query_offset: bad argument");
        return EEG_ERR_INVALID;
    }
    *offset = b->out_off[query];
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_run(eeg_batch* b, uint32_t* out, void* stream, float* ms) {
    if (!b || (b->nq && !out)) {
        set_last_error("eeg_batch_run: null argument");
        return EEG_ERR_INVALID;
    }
    EEG_CUDA(cudaSetDevice(b->device));
    if (b->nq == 0) return EEG_OK;
    EEG_TRY(capture(b, out));
    cudaStream_t user = (cudaStream_t)stream;
    // order after the caller's stream, run on the batch's own (capturable) stream, then back
    EEG_CUDA(cudaEventRecord(b->ev[0], user));
    EEG_CUDA(cudaStreamWaitEvent(b->st, b->ev[0], 0));
    EEG_CUDA(cudaEventRecord(b->ev[0], b->st));
    EEG_CUDA(cudaGraphLaunch(b->exec, b->st));
    EEG_CUDA(cudaEventRecord(b->ev[1], b->st));
    EEG_CUDA(cudaStreamWaitEvent(user, b->ev[1], 0));
    EEG_CUDA(cudaEventSynchronize(b->ev[1]));
    if (ms) EEG_CUDA(cudaEventElapsedTime(ms, b->ev[0], b->ev[1]));
    uint32_t err = 0;
    EEG_CUDA(cudaMemcpy(&err, b->d_err, sizeof(err), cudaMemcpyDeviceToHost));
    if (err) {
        set_last_error("eeg_batch_run: internal error: a frontier queue exceeded its capacity");
        return EEG_ERR_CUDA;
    }
    if (b->nbig) {
        BarrierWords bw{};
        EEG_CUDA(cudaMemcpy(&bw, b->d_bw, sizeof(bw), cudaMemcpyDeviceToHost));
        if (bw.status == DEV_TIMEOUT) {
            // Some CTAs of the launch were not resident (another stream's kernels held SMs), so the
            // whole-grid phase gave up and its queries' results are incomplete. Run the batch again with
            // every query on the clusters, whose barriers need no more than the cluster co-resident.
            const uint32_t keep = b->nbig;
            EEG_TRY(eeg_batch_set_grid_queries(b, 0));
            const eeg_status s = eeg_batch_run(b, out, stream, ms);
            const eeg_status s2 = eeg_batch_set_grid_queries(b, keep);
            return s != EEG_OK ? s : s2;
        }
    }
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_set_grid_queries(eeg_batch* b, uint32_t count) {
    if (!b) {
        set_last_error("eeg_batch_set_grid_queries: null argument");
        return EEG_ERR_INVALID;
    }
    if (b->nbig != count && b->exec) {  // the captured launch holds the old count
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
        b->captured_out = nullptr;
    }
    b->nbig = count;
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_get_config(const eeg_batch* b, uint32_t* cluster_size, uint32_t* grid_queries) {
    if (!b) {
        set_last_error("eeg_batch_get_config: null argument");
        return EEG_ERR_INVALID;
    }
    if (cluster_size) *cluster_size = b->csize;
    if (grid_queries) *grid_queries = std::min(b->nbig, b->nq);
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_rounds(const eeg_batch* b, uint32_t* rounds) {
    if (!b || !rounds) {
        set_last_error("eeg_batch_rounds: null argument");
        return EEG_ERR_INVALID;
    }
    if (b->nq) EEG_CUDA(cudaMemcpy(rounds, b->d_rounds, sizeof(uint32_t) * b->nq, cudaMemcpyDeviceToHost));
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_query_times(const eeg_batch* b, unsigned long long* times) {
    if (!b || !times) {
        set_last_error("eeg_batch_query_times: null argument");
        return EEG_ERR_INVALID;
    }
    if (b->nq) EEG_CUDA(cudaMemcpy(times, b->d_times, 3 * sizeof(unsigned long long) * b->nq, cudaMemcpyDeviceToHost));
    return EEG_OK;
}

EEG_API eeg_status eeg_batch_autotune(eeg_batch* b, uint32_t* out, uint32_t* chosen_cluster_size, float* best_ms) {
    if (!b || (b->nq && !out)) {
        set_last_error("eeg_batch_autotune: null argument");
        return EEG_ERR_INVALID;
    }
    float best = 3.0e38f;
    uint32_t best_c = 4, best_big = 0;
    for (uint32_t c : {1u, 2u, 4u, 8u}) {
        if (configure(b, c) != EEG_OK) continue;
        for (uint32_t nb : {0u, 1u, 2u, 4u, 8u, 16u, 32u, 64u}) {
            if (nb > b->nq) break;
            eeg_batch_set_grid_queries(b, nb);
            float t = 0.f, sum = 0.f;
            bool ok = true;
            for (int rep = 0; rep < 3 && ok; ++rep) {  // first replay warms up; keep the faster of the others
                ok = eeg_batch_run(b, out, nullptr, &t) == EEG_OK;
                if (rep > 0) sum = rep == 1 ? t : std::min(sum, t);
            }
            if (ok && sum < best) {
                best = sum;
                best_c = c;
                best_big = nb;
            }
        }
    }
    EEG_TRY(configure(b, best_c));
    eeg_batch_set_grid_queries(b, best_big);
    if (chosen_cluster_size) *chosen_cluster_size = best_c;
    if (best_ms) *best_ms = best;
    return EEG_OK;
}

EEG_API void eeg_batch_destroy(eeg_batch* b) {
    if (!b) return;
    cudaSetDevice(b->device);
    free_scratch(b);
    cudaFree(b->d_graphs);
    cudaFree(b->d_queries);
    cudaFree(b->d_next);
    cudaFree(b->d_rounds);
    cudaFree(b->d_times);
    cudaFree(b->d_tq);
    cudaFree(b->d_tstamp);
    cudaFree(b->d_tctrl);
    cudaFree(b->d_bw);
    cudaFree(b->d_err);
    if (b->ev[0]) cudaEventDestroy(b->ev[0]);
    if (b->ev[1]) cudaEventDestroy(b->ev[1]);
    if (b->st) cudaStreamDestroy(b->st);
    delete b;
}

}  // extern "C"
