// pagerank_dd.cu -- data-driven PageRank: a residual frontier over the forward virtual graph.
//
// Reference: pr::sync_push_dd and pr::async_push_dd (src/pr.cu:110-169, 227-288) with their driver
// (src/eegraph.cu:1046-1232). Every vertex holds a residual `delta` (initially 1-d = 0.15) and a value
// (initially 0); a vertex whose residual exceeds the activation threshold `acc` (--accuracy,
// src/argument_parsing.cpp:119-121) adds it to its value and pushes d * delta / outdeg to each
// out-neighbour, and only vertices that received a push in the previous round are looked at again.
// Its fixed point is the one of the topology-driven kernels, x = (1-d) + d A^T D^-1 x (the mass of
// vertices without out-edges dropped): at every moment x* = x + (I - d P^T)^-1 r, so stopping when no
// residual exceeds acc leaves ||x* - x||_1 <= ||r||_1 / (1-d).
//
// GB300 form: one cooperative persistent launch; each round has two phases separated by the bounded
// grid barrier.
//   A (vertices): a dense scan of the residuals -- every vertex whose residual t exceeds acc (no push
//     lands in this phase, so a plain read and reset is exact) adds t to its FP64 value, records its push
//     amount d * t / outdeg, and its parts join the round's part queue (one reservation per warp; the
//     whole warp writes a hub's part ids). The scan reads 8 bytes per vertex per round; the vertices it
//     activates are the ones the reference's labels would hold.
//   B (parts): each queued part pushes its owner's amount to its <= K targets with FP64 reductions
//     (atomic adds whose old value nobody waits for). A round that queues no part ends the run: every
//     residual is then <= acc.
// Residuals and values are FP64 (a hub's residual collects ~10^5 pushes per round; FP32 accumulation
// would not hold the 1e-6 L1 bound); the output is FP32. Tracking which pushes lift a residual past acc
// instead of scanning needs the atomics' old values: 25 % slower on R-MAT s22 (154.6 against 123.4 ms),
// every returning FP64 atomic a long-scoreboard wait.
// Long steps (ACC; runs without --accuracy and without a round cap, on graphs of at least a part per four vertices): with the threshold derived from the
// tolerance nearly every vertex stays active for ~135 rounds of 0.84 each, and a round is a Jacobi sweep in
// residual form. So these runs take the step lengths of the control in common.cuh (its evidence is one round
// old when the step is taken): a round with step length alpha adds alpha t to the value, keeps (1 - alpha) t
// as residual and pushes alpha times the amount. Every residual takes part until none exceeds acc (|r|: they
// may be negative): with only those above acc, the last decade lost its single mode and some graphs took 60
// rounds instead of 22-26. So the rounds need no queue: phase A walks the vertices, phase B all parts. A phase
// A that finds nothing above acc is undone from the recorded residuals. R-MAT s17, K = 8:
// 10.5 -> 0.66 ms (with the hot targets below; a graph's first run also sets those up, 0.88 ms).
// Hot targets: reductions to one 128-byte line are done one after another (4 ns each on one address, 1 to 1.5 ns
// within a line by the times below; on lines of their own 175 G/s), so the pushes to an R-MAT graph's first vertices, which share
// lines, set the round's time. Vertices with more than m / 32768 in-edges (and more than 64) therefore
// collect in 32 places, one per lane and each in a line of its own, summed when phase A reads the vertex;
// their ids in a private copy of the targets say so (built once per graph, like the pull sweeps' ranks;
// none where no vertex is hot). R-MAT s17, K = 8: 2.34 -> 1.84 ms with a vertex's 32 places side by side and
// m / 4096; a line each 0.90 -> 0.74 ms, m / 32768 0.66 ms (s20: 4.9 -> 4.3 -> 3.4 ms; m / 8192 and m / 16384
// lie between; graphs of even degree have no hot vertex and do not change).
// Phase A of the long steps was bound by FP64 instructions (the unit takes a warp's in about 16 cycles): a
// division per vertex and round, and ten adds per warp for the two sums. d / outdeg is kept (computed once
// per run), the CTA's sums are added by two warps, and loads that do not depend on each other go out
// together: with one-load barrier polls 1.19 -> 0.98 ms (s17), 0.65 -> 0.43 ms (100003 x 12, even degrees).
// The reference's two DD kernels differ only in when a vertex's label is cleared (in the kernel that
// processes it, or by clearLabel after it); with the residual taken once per round in a phase of its
// own that makes no difference, so SYNC_PUSH_DD and ASYNC_PUSH_DD run these same rounds.
#include <algorithm>

#include "internal.hpp"

namespace eeg {
namespace {

constexpr int DD_TPB = 512;
constexpr uint32_t HOT = 0x80000000u;  // private target ids: index of a hot vertex (graphs below 2^31 vertices)
constexpr uint32_t HOT_CAP = 32768;

struct DDArgs {
    uint32_t n;
    uint32_t P;
    const uint32_t* __restrict__ vstart;
    const uint32_t* __restrict__ vowner;
    const uint32_t* __restrict__ vcol;
    const uint32_t* __restrict__ deg;
    const uint32_t* __restrict__ hot;    // nhot hot vertices
    const uint32_t* __restrict__ hbits;  // bit per vertex: hot
    uint32_t nhot;
    uint32_t hstride;                    // nhot rounded up to whole 128-byte lines
    double* rep;                         // 32 x hstride partial residuals
    double* r;
    double* xv;
    double* amt;
    double* taken;  // long steps: each vertex's residual in the last round
    double* share;  // long steps: d / outdeg (0 without out-edges)
    float* x;
    uint32_t* pq;
    PRDDCtrl* ctrl;
    double acc;
    double damping;
    double base;
    uint32_t max_iters;
    uint64_t timeout_ns;
};

// Warp-collective: append the parts [s0, s0 + np) of each lane's vertex to the part queue.
__device__ __forceinline__ void append_parts(uint32_t s0, uint32_t np, uint32_t* ctr, uint32_t* pq, uint32_t cap,
                                             uint32_t lane) {
    uint32_t inc = np;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= (uint32_t)off) inc += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    if (total == 0u) return;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(ctr, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t pos = base + inc - np;
    if (np <= 32u)
        for (uint32_t j = 0; j < np; ++j)
            if (pos + j < cap) pq[pos + j] = s0 + j;
    uint32_t big = __ballot_sync(0xffffffffu, np > 32u);
    while (big) {  // hub vertices: the whole warp writes their part ids
        const int l = __ffs(big) - 1;
        big &= big - 1u;
        const uint32_t bs0 = __shfl_sync(0xffffffffu, s0, l);
        const uint32_t bnp = __shfl_sync(0xffffffffu, np, l);
        const uint32_t bpos = __shfl_sync(0xffffffffu, pos, l);
        for (uint32_t j = lane; j < bnp; j += 32u)
            if (bpos + j < cap) pq[bpos + j] = bs0 + j;
    }
}

template <int K, bool ACC>
__global__ void __launch_bounds__(DD_TPB, 2) k_pagerank_dd(DDArgs a) {
    __shared__ uint32_t s_len;
    __shared__ double s_red[2][DD_TPB / 32];
    __shared__ double s_sum[2][ACC ? DD_TPB : 1];
    PRDDCtrl* ctrl = a.ctrl;
    const uint32_t gtid = blockIdx.x * DD_TPB + threadIdx.x;
    const uint32_t gthreads = gridDim.x * DD_TPB;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t gwarp = gtid >> 5, nwarps = gthreads >> 5;
    const uint64_t pol = l2_evict_first_policy();
    uint32_t epoch = 0;
    uint32_t it = 0;
    unsigned long long my_pushes = 0, my_parts = 0, my_taken = 0;
    __shared__ Extrapolation s_ex;
    bool stepped = false;  // the last round took a long step
    double undo = 0.0;     // ACC: step length of a phase A whose residuals are to be put back
    if (threadIdx.x == 0) extrapolation_init(s_ex);

    for (uint32_t v = gtid; v < a.n; v += gthreads) {
        a.r[v] = a.base;
        a.xv[v] = 0.0;
        if (ACC) {
            const uint32_t d = __ldg(&a.deg[v]);
            a.share[v] = d ? a.damping / (double)d : 0.0;
        }
    }
    for (uint32_t i = gtid; i < a.hstride * 32u; i += gthreads) a.rep[i] = 0.0;
    if (!grid_barrier_sync(&ctrl->bw, epoch, a.timeout_ns)) goto finish;

    for (;; ++it) {
        const uint32_t cur = it % 3u, nxt = (it + 1u) % 3u;
        if (it >= a.max_iters) {
            if (blockIdx.x == 0 && threadIdx.x == 0)
                atomicCAS(&ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_ITER_CAP);
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {  // last read in round it-2
            ctrl->plen[nxt] = 0u;
            ctrl->rsum[nxt] = 0.0;
            ctrl->probe[nxt] = 0.0;
        }
        const double alpha = (double)s_ex.alpha;
        const double rho = s_ex.cand != 0.f ? 1.0 - 1.0 / (double)s_ex.cand : 0.0;  // measured for when not 0
        double rs = 0.0, qs = 0.0;
        // ---- phase A: every vertex whose residual exceeds acc takes it (a dense scan of the residuals)
        uint32_t above = 0;  // ACC: this thread saw a residual above acc
        // vertex v with residual t: taken when it exceeds acc; its parts [s0, s0 + np) then push
        auto take = [&](uint32_t v, double t, uint32_t& s0, uint32_t& np) {
            const bool act = t > a.acc;
            if (act) {
                a.r[v] = 0.0;
                a.xv[v] = __ldcg(&a.xv[v]) + t;
                ++my_taken;
                const uint32_t d = __ldg(&a.deg[v]);
                if (d) {
                    a.amt[v] = a.damping * t / (double)d;
                    s0 = __ldg(&a.vstart[v]);
                    np = __ldg(&a.vstart[v + 1]) - s0;
                }
            }
            return act;
        };
        // ACC: every vertex is taken. Value, share and last residual are loaded beside t.
        auto step = [&](uint32_t v, double t, double xo, double share, double last) {
            const double at = alpha != 1.0 ? alpha * t : t;
            if (rho != 0.0) qs += fabs(t - rho * last);
            rs += fabs(t);
            above |= fabs(t) > a.acc ? 1u : 0u;
            a.taken[v] = t;
            a.amt[v] = at * share;
            a.r[v] = alpha != 1.0 ? (1.0 - alpha) * t : 0.0;
            a.xv[v] = xo + at;
            my_taken += t != 0.0 ? 1u : 0u;
        };
        // hot vertices: a lane sums one vertex's partial residuals (32 vertices per warp, spread over the CTAs)
        for (uint32_t h0 = (threadIdx.x / 32u * gridDim.x + blockIdx.x) * 32u; h0 < a.nhot; h0 += nwarps * 32u) {
            const uint32_t h = h0 + lane;
            uint32_t s0 = 0, np = 0;
            if (h < a.nhot) {
                const uint32_t v = __ldg(&a.hot[h]);
                const double r0 = __ldcg(&a.r[v]), xo = __ldcg(&a.xv[v]);
                const double share = ACC ? __ldcg(&a.share[v]) : 0.0;
                const double last = ACC && rho != 0.0 ? __ldcg(&a.taken[v]) : 0.0;
                double sum = 0.0;
#pragma unroll 8
                for (uint32_t l = 0; l < 32u; ++l) sum += __ldcg(&a.rep[(size_t)l * a.hstride + h]);
#pragma unroll 8
                for (uint32_t l = 0; l < 32u; ++l) a.rep[(size_t)l * a.hstride + h] = 0.0;
                const double t = r0 + sum;
                if (ACC)
                    step(v, t, xo, share, last);
                else if (!take(v, t, s0, np))
                    a.r[v] = t;
            }
            if (!ACC) append_parts(s0, np, &ctrl->plen[cur], a.pq, a.P, lane);
        }
        for (uint32_t b0 = gwarp * 32u; b0 < a.n; b0 += nwarps * 32u) {
            const uint32_t v = b0 + lane;
            uint32_t s0 = 0, np = 0;
            const uint32_t hb = a.nhot ? __ldg(&a.hbits[b0 >> 5]) : 0u;
            if (ACC) {
                double t = 0.0, xo = 0.0, share = 0.0, last = 0.0;
                if (v < a.n) {
                    t = __ldcg(&a.r[v]);
                    xo = __ldcg(&a.xv[v]);
                    share = __ldcg(&a.share[v]);
                    if (rho != 0.0) last = __ldcg(&a.taken[v]);
                }
                if (v < a.n && !((hb >> lane) & 1u)) step(v, t, xo, share, last);
            } else {
                if (v < a.n && !((hb >> lane) & 1u)) take(v, __ldcg(&a.r[v]), s0, np);
                append_parts(s0, np, &ctrl->plen[cur], a.pq, a.P, lane);
            }
        }
        if (ACC) {  // two warps add the CTA's sums
            s_sum[0][threadIdx.x] = rs;
            s_sum[1][threadIdx.x] = qs;
            above = __syncthreads_or(above);
            if (threadIdx.x < 64u) {
                const uint32_t which = threadIdx.x >> 5;
                double sum = 0.0;
                if (which == 0u || rho != 0.0) {
#pragma unroll 4
                    for (int w = 0; w < DD_TPB / 32; ++w) sum += s_sum[which][w * 32 + lane];
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
                    if (lane == 0u) atomicAdd(which ? &ctrl->probe[cur] : &ctrl->rsum[cur], sum);
                }
                if (threadIdx.x == 0 && above) atomicAdd(&ctrl->plen[cur], 1u);
            }
        }
        if (!grid_barrier_sync(&ctrl->bw, epoch, a.timeout_ns)) break;
        if (threadIdx.x == 0) {
            s_len = ld_relaxed(&ctrl->plen[cur]);
            if (ACC) {
                const double rt = __ldcg(&ctrl->rsum[cur]);
                if (alpha != 1.0) {  // this round takes the step: rt is the residual before it
                    s_ex.alpha = 1.f;
                    s_ex.r_before = rt;
                    s_ex.r_prev = 0.0;
                } else {
                    if (stepped && !(rt <= s_ex.r_before)) s_ex.off = 1u;
                    extrapolation_next(s_ex, rt, __ldcg(&ctrl->probe[cur]), a.damping);
                }
            }
        }
        stepped = alpha != 1.0;
        __syncthreads();
        uint32_t npq = s_len;
        __syncthreads();
        if (npq == 0u) {  // nothing pushes: every residual stays <= acc
            undo = alpha;
            break;
        }
        if (!ACC && npq > a.P) {
            if (blockIdx.x == 0 && threadIdx.x == 0)
                atomicCAS(&ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_OVERFLOW);
            npq = a.P;
        }
        // ---- phase B: push the amounts along the queued parts (reductions: no value comes back)
        if (ACC) npq = a.P;
        constexpr int U = K >= 16 ? 1 : 2;  // chunks in flight per warp
        for (uint64_t b0 = (uint64_t)gwarp * 32u; b0 < npq; b0 += (uint64_t)nwarps * 32u * U) {
            uint32_t col[U][K];
            double am[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t i = b0 + (uint64_t)u * nwarps * 32u + lane;
                am[u] = 0.0;
                if (i < npq) {
                    const uint32_t p = ACC ? (uint32_t)i : __ldcg(&a.pq[i]);
                    const uint32_t owner = __ldg(&a.vowner[p]);
                    ld_part<K>(a.vcol + (size_t)p * K, col[u], pol);
                    am[u] = __ldcg(&a.amt[owner]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (am[u] == 0.0) continue;  // past the end, or nothing to push
                ++my_parts;
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (col[u][k] != NO_EDGE) {
                        double* at = a.r + col[u][k];
                        if (a.nhot && (col[u][k] & HOT)) at = a.rep + (size_t)lane * a.hstride + (col[u][k] & ~HOT);
                        atomicAdd(at, am[u]);
                        ++my_pushes;
                    }
            }
        }
        if (!grid_barrier_sync(&ctrl->bw, epoch, a.timeout_ns)) break;
    }
finish:
    {
        // the output, and what is left: residual mass (error bound resid / (1-d)) and the value norm
        double rs = 0.0, xs = 0.0;
        for (uint32_t v = gtid; v < a.n; v += gthreads) {
            double xv = __ldcg(&a.xv[v]);
            double rv = __ldcg(&a.r[v]);
            if (ACC && undo != 0.0) {
                rv = __ldcg(&a.taken[v]);
                xv -= undo * rv;
            }
            a.x[v] = (float)xv;
            if (a.nhot && ((__ldg(&a.hbits[v >> 5]) >> (v & 31u)) & 1u)) rv = 0.0;  // counted below
            rs += fabs(rv);
            xs += xv;
        }
        for (uint32_t h = gtid; h < a.nhot; h += gthreads) {  // pushes not taken (the round cap) count too
            const uint32_t v = __ldg(&a.hot[h]);
            double rv = ACC && undo != 0.0 ? __ldcg(&a.taken[v]) : __ldcg(&a.r[v]);
            for (uint32_t l = 0; l < 32u; ++l) rv += __ldcg(&a.rep[(size_t)l * a.hstride + h]);
            rs += fabs(rv);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            rs += __shfl_down_sync(0xffffffffu, rs, off);
            xs += __shfl_down_sync(0xffffffffu, xs, off);
            my_pushes += __shfl_down_sync(0xffffffffu, my_pushes, off);
            my_parts += __shfl_down_sync(0xffffffffu, my_parts, off);
            my_taken += __shfl_down_sync(0xffffffffu, my_taken, off);
        }
        if (lane == 0) {
            s_red[0][threadIdx.x >> 5] = rs;
            s_red[1][threadIdx.x >> 5] = xs;
            if (my_pushes) atomicAdd(&ctrl->pushes, my_pushes);
            if (my_parts) atomicAdd(&ctrl->parts, my_parts);
            if (my_taken) atomicAdd(&ctrl->consumed, my_taken);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double r2 = 0.0, x2 = 0.0;
            for (int w = 0; w < DD_TPB / 32; ++w) {
                r2 += s_red[0][w];
                x2 += s_red[1][w];
            }
            atomicAdd(&ctrl->resid, r2);
            atomicAdd(&ctrl->norm, x2);
            if (blockIdx.x == 0) ctrl->iterations = it;
        }
    }
}

// ---- hot targets (once per graph)
__global__ void k_dd_indeg(uint64_t slots, const uint32_t* __restrict__ col, uint32_t* cnt) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = col[i];
        if (c != NO_EDGE) atomicAdd(&cnt[c], 1u);
    }
}
// cnt[v] (in-degree) -> v's private id; hot vertices listed in hot[1..], their number in hot[0], bits in hbits
__global__ void k_dd_hot(uint32_t n, uint32_t limit, uint32_t* cnt, uint32_t* hot, uint32_t* hbits) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        uint32_t id = v;
        if (cnt[v] > limit) {
            const uint32_t h = atomicAdd(&hot[0], 1u);
            hot[1u + h] = v;
            atomicOr(&hbits[v >> 5], 1u << (v & 31u));
            id = HOT | h;
        }
        cnt[v] = id;
    }
}
__global__ void k_dd_cols(uint64_t slots, const uint32_t* __restrict__ col, const uint32_t* __restrict__ id,
                          uint32_t* __restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = col[i];
        out[i] = c == NO_EDGE ? NO_EDGE : id[c];
    }
}

template <int K>
eeg_status launch_dd(const DDArgs& a, bool acc, int device, uint32_t bps, cudaStream_t st) {
    auto kern = acc ? k_pagerank_dd<K, true> : k_pagerank_dd<K, false>;
    int per_sm = 0;
    EEG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, DD_TPB, 0));
    if (per_sm <= 0) {
        set_last_error("data-driven PageRank kernel does not fit on an SM");
        return EEG_ERR_CUDA;
    }
    if (bps > 0 && (int)bps < per_sm) per_sm = (int)bps;
    uint64_t blocks = (uint64_t)per_sm * sm_count(device);
    const uint64_t work = std::max<uint64_t>(a.P, a.n);
    const uint64_t need = (work + DD_TPB - 1) / DD_TPB;
    if (need < blocks) blocks = std::max<uint64_t>(need, 1);
    DDArgs args = a;
    void* params[] = {(void*)&args};
    EEG_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)blocks), dim3(DD_TPB), params, 0, st));
    return EEG_OK;
}

}  // namespace

static uint32_t hot_stride(uint32_t nhot) { return (nhot + 15u) / 16u * 16u; }

// A graph whose private targets (as many words as its own) do not fit runs without hot targets.
static eeg_status ensure_dd_hot(eeg_vgraph* vg, cudaStream_t st) {
    Workspace& ws = vg->ws;
    if (ws.dd_hot_ready) return EEG_OK;
    const uint64_t slots = vg->fwd.P * vg->K;
    const uint64_t limit = std::max<uint64_t>(64, vg->m >> 15);  // sum of in-degrees = m: below HOT_CAP hot vertices
    ws.dd_nhot = 0;
    if (slots && vg->n < HOT && vg->m > limit) {
        const size_t words = ((size_t)vg->n + 31) / 32;
        uint32_t* cnt = nullptr;
        auto set_up = [&]() -> eeg_status {
            if (!ws.dd_hot) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_hot, sizeof(uint32_t) * (HOT_CAP + 1 + words)));
            const cudaError_t e = cudaMallocAsync((void**)&cnt, sizeof(uint32_t) * vg->n, st);
            if (e != cudaSuccess) {
                cnt = nullptr;
                return cuda_fail(e, "cudaMallocAsync(in-degrees)", __FILE__, __LINE__);
            }
            EEG_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * vg->n, st));
            EEG_CUDA(cudaMemsetAsync(ws.dd_hot, 0, sizeof(uint32_t) * (HOT_CAP + 1 + words), st));
            const uint64_t cap = (uint64_t)sm_count(vg->device) * 8;
            const unsigned gs = (unsigned)std::min<uint64_t>((slots + 255) / 256, cap * 2);
            const unsigned gv = (unsigned)std::min<uint64_t>(((uint64_t)vg->n + 255) / 256, cap);
            k_dd_indeg<<<gs, 256, 0, st>>>(slots, vg->fwd.vcol, cnt);
            k_dd_hot<<<gv, 256, 0, st>>>(vg->n, (uint32_t)limit, cnt, ws.dd_hot, ws.dd_hot + HOT_CAP + 1);
            uint32_t nhot = 0;
            EEG_CUDA(cudaMemcpyAsync(&nhot, ws.dd_hot, sizeof(nhot), cudaMemcpyDeviceToHost, st));
            EEG_CUDA(cudaStreamSynchronize(st));
            if (nhot) {
                if (!ws.dd_col) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_col, sizeof(uint32_t) * slots));
                if (!ws.dd_rep) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_rep, sizeof(double) * 32 * (size_t)hot_stride(nhot)));
                k_dd_cols<<<gs, 256, 0, st>>>(slots, vg->fwd.vcol, cnt, ws.dd_col);
            }
            EEG_CUDA(cudaGetLastError());
            ws.dd_nhot = nhot;
            return EEG_OK;
        };
        const eeg_status s = set_up();
        if (cnt) cudaFreeAsync(cnt, st);
        if (s == EEG_ERR_NOMEM) {
            (void)cudaGetLastError();
            vg_free(vg, ws.dd_col);
            ws.dd_col = nullptr;
        } else {
            EEG_TRY(s);
        }
    }
    ws.dd_hot_ready = true;
    return EEG_OK;
}

eeg_status run_pagerank_dd(eeg_vgraph* vg, eeg_variant variant, const eeg_options& o, cudaStream_t st,
                           eeg_result* res) {
    (void)variant;
    if (vg->n == 0) {
        set_last_error("empty graph");
        return EEG_ERR_INVALID;
    }
    if (!vg->fwd_parts) {
        set_last_error("data-driven PageRank pushes along out-edges: this graph was built without its forward "
                       "parts (EEG_VG_REVERSE_ONLY); use a topology-driven variant or build the forward graph");
        return EEG_ERR_INVALID;
    }
    Workspace& ws = vg->ws;
    const size_t n = std::max<uint32_t>(vg->n, 1);
    const size_t P = std::max<uint64_t>(vg->fwd.P, 1);
    if (!ws.x) EEG_TRY(vg_alloc(vg, (void**)&ws.x, sizeof(float) * n));
    if (!ws.dd_r) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_r, sizeof(double) * n));
    if (!ws.dd_x) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_x, sizeof(double) * n));
    if (!ws.dd_amt) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_amt, sizeof(double) * n));
    // long steps: the threshold and the schedule are the library's own (no --accuracy, no round cap)
    // and phase A is not most of the work: where few vertices have out-edges (fewer parts than n/4), nearly all of them are
    // idle after the first round, and a queue's scan of the residuals takes a seventh of a long step's phase A (2^26
    // vertices, 1 M edges: 3.1 ms, 11.5 with long steps; a cycle with 4 M leaves 0.33, 0.65. A tree, two vertices per
    // part, still loses, 0.62 and 0.95 in 20 and 23 rounds; R-MAT graphs, whose mass circulates, gain from there on)
    bool accel = !(o.pr_accuracy > 0.f) && o.max_iterations == 0 && vg->fwd.P * 4u >= vg->n;
    if (accel) {  // two arrays more; where they do not fit, the rounds keep a queue
        eeg_status s = EEG_OK;
        if (!ws.dd_taken) s = vg_alloc(vg, (void**)&ws.dd_taken, sizeof(double) * n);
        if (s == EEG_OK && !ws.dd_share) s = vg_alloc(vg, (void**)&ws.dd_share, sizeof(double) * n);
        if (s == EEG_ERR_NOMEM) {
            (void)cudaGetLastError();
            accel = false;
        } else {
            EEG_TRY(s);
        }
    }
    if (!accel && !ws.dd_pq) EEG_TRY(vg_alloc(vg, (void**)&ws.dd_pq, sizeof(uint32_t) * P));
    if (!ws.ddctrl) EEG_CUDA(cudaMalloc((void**)&ws.ddctrl, sizeof(PRDDCtrl)));
    if (!ws.ev[0]) {
        EEG_CUDA(cudaEventCreate(&ws.ev[0]));
        EEG_CUDA(cudaEventCreate(&ws.ev[1]));
    }
    EEG_TRY(ensure_dd_hot(vg, st));
    EEG_CUDA(cudaMemsetAsync(ws.ddctrl, 0, sizeof(PRDDCtrl), st));
    const double damping = o.pr_damping > 0.f ? (double)o.pr_damping : 0.85;
    const double tol = o.pr_tolerance > 0.f ? (double)o.pr_tolerance : 1e-7;
    DDArgs a{};
    a.n = vg->n;
    a.P = (uint32_t)vg->fwd.P;
    a.vstart = vg->fwd.vstart;
    a.vowner = vg->fwd.vowner;
    a.vcol = ws.dd_nhot ? ws.dd_col : vg->fwd.vcol;
    a.deg = vg->fwd.deg;
    a.nhot = ws.dd_nhot;
    a.hstride = hot_stride(ws.dd_nhot);
    a.hot = ws.dd_hot ? ws.dd_hot + 1 : nullptr;
    a.hbits = ws.dd_hot ? ws.dd_hot + HOT_CAP + 1 : nullptr;
    a.rep = ws.dd_rep;
    a.r = ws.dd_r;
    a.xv = ws.dd_x;
    a.amt = ws.dd_amt;
    a.taken = ws.dd_taken;
    a.share = ws.dd_share;
    a.x = ws.x;
    a.pq = ws.dd_pq;
    a.ctrl = ws.ddctrl;
    a.damping = damping;
    a.base = 1.0 - damping;
    // The reference's activation threshold when given; otherwise one that meets the tolerance: every
    // value ends >= 1-d, so residuals <= tol*(1-d)^2 bound ||x*-x||_1 <= n*acc/(1-d) <= tol*||x||_1.
    a.acc = o.pr_accuracy > 0.f ? (double)o.pr_accuracy : tol * (1.0 - damping) * (1.0 - damping);
    a.max_iters = o.max_iterations ? o.max_iterations : 10000u;
    a.timeout_ns = wait_limit_ns(o);

    EEG_CUDA(cudaEventRecord(ws.ev[0], st));
    eeg_status s;
    switch (vg->K) {
        case 4: s = launch_dd<4>(a, accel, vg->device, o.blocks_per_sm, st); break;
        case 8: s = launch_dd<8>(a, accel, vg->device, o.blocks_per_sm, st); break;
        case 16: s = launch_dd<16>(a, accel, vg->device, o.blocks_per_sm, st); break;
        default: set_last_error("K must be 4, 8 or 16"); return EEG_ERR_UNSUPPORTED;
    }
    if (s != EEG_OK) return s;
    EEG_CUDA(cudaEventRecord(ws.ev[1], st));
    PRDDCtrl hc;
    EEG_CUDA(cudaMemcpyAsync(&hc, ws.ddctrl, sizeof(PRDDCtrl), cudaMemcpyDeviceToHost, st));
    EEG_CUDA(cudaStreamSynchronize(st));
    float ms = 0.f;
    EEG_CUDA(cudaEventElapsedTime(&ms, ws.ev[0], ws.ev[1]));
    if (res) {
        res->kernel_ms = ms;
        res->iterations = hc.iterations;
        res->edges_scanned = hc.pushes;
        res->parts_processed = hc.parts;
        res->updates = hc.consumed;
        res->pr_residual = hc.resid;
        res->pr_l1_norm = hc.norm;
        res->launches = 1;
    }
    if (hc.bw.status == DEV_TIMEOUT) {
        set_last_error("grid barrier wait exceeded the timeout");
        return EEG_ERR_TIMEOUT;
    }
    if (hc.bw.status == DEV_ITER_CAP) {
        set_last_error("data-driven PageRank did not empty its frontier within the round cap");
        return EEG_ERR_ITER_CAP;
    }
    if (hc.bw.status == DEV_OVERFLOW) {
        set_last_error("internal error: a PageRank frontier exceeded its capacity");
        return EEG_ERR_CUDA;
    }
    return EEG_OK;
}

}  // namespace eeg
