// ppr.cu -- differentiable personalised PageRank: forward solve, implicit adjoint solve and the
// edge / teleport gradients over the K-bounded virtual graph. A project-added form: the reference's
// PageRank (src/pr.cu:3-288) is unweighted, unpersonalised and has no adjoint.
//
// Model, per column, with row-normalised weights W_uv = w_uv / s_u (s_u = sum of u's out-weights):
//   forward  X = (1-d) T + d W^T X    -- pull over the transposed graph: x_v gathers rows X_u
//   adjoint  L = G + d W L            -- pull over the forward graph:   l_u gathers rows L_v
//   dLoss/dW_uv = d <X_u, L_v>,  dLoss/dw_uv = (dLoss/dW_uv - sum_v' dLoss/dW_uv' W_uv') / s_u,
//   dLoss/dT = (1-d) L.
// Neither solve needs atomics on values, a transpose at run time or stored iterates.
//
// Work decomposition (both directions, both forms): the part list is cut into chunks of <= 128 slots.
// A chunk holds whole vertices, except that a vertex with more than 128 slots (a hub) gets chunks of
// its own. Each hub chunk writes a partial; the last chunk of a group of 32 to arrive sums the group
// (compensated FP32, in chunk order) and the last group sums the groups. Deterministic, and a sweep
// needs one grid barrier (Jacobi, double-buffered iterates).
//   Batched rows (2..64 columns; rows padded to W = 32 or 64 FP32, 128 or 256 B): a warp owns a chunk and
//   splits into G = 128/W lane groups of W/4 lanes; group g takes slots g, g+G, ... of each part and
//   lane q of a group the float4 of columns 4q..4q+3, so one gather instruction moves G rows.
//   Single column (the plain form): a lane owns a slot; part sums by K-lane butterflies, vertex sums by
//   a segmented warp scan.
// Two forms of a sweep (template parameter RES):
//   Residual form (runs without an explicit sweep cap): a sweep gathers the rows of the residual f, the
//   iterate moves by alpha g with g = d * (gathered sum), and the step length alpha comes from the
//   extrapolation control (common.cuh): 94 + 78 sweeps of forward and adjoint become 21 + 21 on R-MAT
//   graphs, which the gathers through L2 bound (R-MAT s18 x 64 columns, step with gradients 27.0 -> 8.6 ms). The first
//   sweep gathers the source rows themselves; rows without parts in the direction keep a zero residual.
//   The iterate is accumulated in FP32, so two last value-form sweeps (x = s b + d sum) replace the
//   rounding of the additions by that of one sweep: relative L2 error of the adjoint at R-MAT s18 in a
//   CPU model 9.1e-8 without them, 5.2e-8 with one, 2.8e-8 with two (plain sweeps: 1.0e-7).
//   After long steps a forward solve also ends only when no element is further from its end than the bound of
//   common.cuh allows (see look()).
//   Value form (runs with an explicit cap, whose result after k sweeps is the k-th Jacobi iterate).
// Stop test: d/(1-d) * ||Y_{k+1}-Y_k||_1 <= tol * ||Y_{k+1}||_1 over all columns, reduced in FP64
// (FP32 per-chunk partials, FP64 per lane and across the grid); everything else is FP32.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.hpp"

namespace eeg {
namespace {

constexpr uint32_t PPR_SLOTS = 128;  // slots per work chunk
constexpr uint32_t PPR_GROUP = 32;   // hub chunks per first-level group
constexpr uint32_t PPR_W = 64;       // widest row of the batched form (FP32 columns)
constexpr int PPR_TPB = 256;
constexpr uint32_t NONE = 0xFFFFFFFFu;
constexpr unsigned FULL = 0xFFFFFFFFu;

struct Chunk {
    uint32_t p0, p1;  // parts [p0, p1)
    uint32_t hub;     // hub table index, or NONE
    uint32_t idx;     // index of this chunk within its hub
};
struct Hub {
    uint32_t v;       // vertex
    uint32_t first;   // first partial slot
    uint32_t count;   // chunks
    uint32_t gfirst;  // first group
};

// Device tables of one direction.
struct DirTab {
    const uint32_t* __restrict__ vowner;
    const uint32_t* __restrict__ vcol;
    const float* __restrict__ w;  // normalised weight of each slot
    const Chunk* __restrict__ chunk;
    uint32_t nchunks;
    const Hub* __restrict__ hub;
    uint32_t* garrive;  // arrivals per group (monotone over the sweeps of one launch)
    uint32_t* harrive;  // group completions per hub
    float* partial;     // hub chunk partials (slots x width)
    float* gpartial;    // group partials (groups x width)
    const uint32_t* __restrict__ vstart;
};

// What a sweep of the solve does at a vertex's end (uniform over the grid). VALUE: x = s b + d sum.
// Residual form, g = d sum: FIRST (gathers the source rows), PLAIN (y += g, f = g), PROBE (PLAIN, and q
// for the control), STEP (y += alpha g, f = (1 - alpha) f + alpha g).
enum Sweep : int { SW_VALUE = 0, SW_FIRST = 1, SW_PLAIN = 2, SW_PROBE = 3, SW_STEP = 4 };

struct SolveArgs {
    DirTab g;
    uint32_t n;
    const float* __restrict__ b;  // n x width source rows
    float scale_b;                // 1-d (forward) or 1 (adjoint)
    float d;
    float scale_lo, d_lo;         // their low parts (runs without a cap; 0 in value-form runs)
    float* y0;      // iterates (residual form: residuals)
    float* y1;
    float* y;       // residual form: the iterate
    float* res;     //                and the buffer of the result (y1 may share it: not read in the last sweep)
    PRCtrl* ctrl;
    uint32_t max_iters;
    double tol;
    VertexBound bound;  // residual form, forward
    uint64_t timeout_ns;
};

struct GradArgs {
    DirTab g;               // forward direction
    const float* __restrict__ X;
    const float* __restrict__ L;
    float d;
    float* gslot;           // dLoss/dW per forward slot
    float* r;               // sum_v dLoss/dW_uv W_uv per vertex
    uint32_t accumulate;
};

// ------------------------------------------------------------------ small helpers
__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ void fma4(float4& acc, float w, const float4& x) {
    acc.x = fmaf(w, x.x, acc.x);
    acc.y = fmaf(w, x.y, acc.y);
    acc.z = fmaf(w, x.z, acc.z);
    acc.w = fmaf(w, x.w, acc.w);
}
__device__ __forceinline__ float4 shfl_xor4(const float4& v, int o) {
    return make_float4(__shfl_xor_sync(FULL, v.x, o), __shfl_xor_sync(FULL, v.y, o), __shfl_xor_sync(FULL, v.z, o),
                       __shfl_xor_sync(FULL, v.w, o));
}
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
// d acc + s b, both factors as (high, low) pairs
__device__ __forceinline__ float affine(float d, float dl, float acc, float s, float sl, float b) {
    return fmaf(d, acc, fmaf(dl, acc, fmaf(sl, b, s * b)));
}
__device__ __forceinline__ float4 affine4(float d, float dl, const float4& acc, float s, float sl, const float4& b) {
    return make_float4(affine(d, dl, acc.x, s, sl, b.x), affine(d, dl, acc.y, s, sl, b.y),
                       affine(d, dl, acc.z, s, sl, b.z), affine(d, dl, acc.w, s, sl, b.w));
}
__device__ __forceinline__ float l1diff4(const float4& a, const float4& b) {
    return fabsf(a.x - b.x) + fabsf(a.y - b.y) + fabsf(a.z - b.z) + fabsf(a.w - b.w);
}
__device__ __forceinline__ float l14(const float4& a) { return fabsf(a.x) + fabsf(a.y) + fabsf(a.z) + fabsf(a.w); }
__device__ __forceinline__ float dot4(const float4& a, const float4& b) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));
}
__device__ __forceinline__ uint32_t ld_nc(const uint32_t* p) { return __ldg(p); }

// Element j (run-time index) of a register array without local-memory indexing.
template <int N, typename T>
__device__ __forceinline__ T pick(const T (&a)[N], uint32_t j) {
    T r = a[0];
#pragma unroll
    for (int i = 1; i < N; ++i)
        if ((uint32_t)i == j) r = a[i];
    return r;
}

// Lane-group transpose reduction: each lane holds N values (one per slot of its group of NQ lanes);
// afterwards lane q holds the sum over the group's lanes of value index(q) (see red_index). log2(N)
// halving steps, then plain butterflies.
template <int N, int NQ>
__device__ __forceinline__ float tred(float (&v)[N], uint32_t q) {
    int n = N;
#pragma unroll
    for (int o = NQ / 2; o >= 1; o >>= 1) {
        if (n >= 2) {
            const bool up = (q & (uint32_t)o) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i < n / 2) {
                    const float send = up ? v[i] : v[i + n / 2];
                    const float keep = up ? v[i + n / 2] : v[i];
                    v[i] = keep + __shfl_xor_sync(FULL, send, o);
                }
            }
            n >>= 1;
        } else {
            v[0] += __shfl_xor_sync(FULL, v[0], o);
        }
    }
    return v[0];
}
template <int N, int NQ>
__device__ __forceinline__ uint32_t red_index(uint32_t q) {
    uint32_t i = 0;
    int n = N;
#pragma unroll
    for (int o = NQ / 2; o >= 1; o >>= 1) {
        if (n >= 2) {
            if (q & (uint32_t)o) i += (uint32_t)(n / 2);
            n >>= 1;
        }
    }
    return i;
}

// Sum of a float4 over the warp's lane groups (lanes q, q+NQ, ...); every lane gets its q's total.
template <int NQ>
__device__ __forceinline__ float4 across_groups(float4 v) {
#pragma unroll
    for (int o = NQ; o < 32; o <<= 1) v = add4(v, shfl_xor4(v, o));
    return v;
}

// Compensated sum of partial rows [first, first+cnt) (NQ float4 each); lane groups take rows in turn;
// every lane of the warp returns the same float4 for its q.
template <int NQ>
__device__ float4 sum_rows(const float4* base, uint32_t first, uint32_t cnt, uint32_t grp, uint32_t q) {
    constexpr uint32_t G = 32 / NQ;
    float4 hi = f4(0.f), lo = f4(0.f);
    for (uint32_t i = grp; i < cnt; i += G) {
        const float4 p = __ldcg(base + (size_t)(first + i) * NQ + q);
        pair_add(hi.x, lo.x, p.x, 0.f);
        pair_add(hi.y, lo.y, p.y, 0.f);
        pair_add(hi.z, lo.z, p.z, 0.f);
        pair_add(hi.w, lo.w, p.w, 0.f);
    }
#pragma unroll
    for (int o = NQ; o < 32; o <<= 1) {
        const float4 ho = shfl_xor4(hi, o), lo2 = shfl_xor4(lo, o);
        pair_add(hi.x, lo.x, ho.x, lo2.x);
        pair_add(hi.y, lo.y, ho.y, lo2.y);
        pair_add(hi.z, lo.z, ho.z, lo2.z);
        pair_add(hi.w, lo.w, ho.w, lo2.w);
    }
    return hi;
}

// Slot j*G + grp of a part row (grp run-time, the array index compile-time: no local memory).
template <int G, int K>
__device__ __forceinline__ uint32_t group_slot(const uint32_t (&row)[K], int j, uint32_t grp) {
    uint32_t r = row[j * G];
#pragma unroll
    for (int g = 1; g < G; ++g)
        if (grp == (uint32_t)g) r = row[j * G + g];
    return r;
}

// Rows gathered per lane per step: 8, so U = 8/H parts per step (16/K at W = 64, 32/K at W = 32).
template <int K, int G>
struct RowStep {
    static constexpr int H = K / G;  // slots of a part per lane group
    static constexpr int U = 8 / H;  // parts per step
};

// Neighbour ids and weights of this lane group's slots (j*G + grp) of parts pp .. pp+U-1 of a chunk
// (NONE and 0 past its np parts). Two groups (W = 64): whole rows by 256-bit loads, then a selection;
// more groups: the group's slots one by one (the whole rows would take 2*U*K registers).
template <int K, int G>
__device__ __forceinline__ void load_group_slots(const DirTab& g, uint32_t p0, uint32_t pp, uint32_t np, uint32_t grp,
                                                 uint64_t pol, uint32_t (&colg)[RowStep<K, G>::U][K / G],
                                                 uint32_t (&wbg)[RowStep<K, G>::U][K / G]) {
    constexpr int U = RowStep<K, G>::U, H = K / G;
    if constexpr (G <= 2) {
        uint32_t col[U][K], wb[U][K];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (pp + u < np) {
                const size_t row = (size_t)(p0 + pp + u) * K;
                ld_part<K>(g.vcol + row, col[u], pol);
                ld_part<K>(reinterpret_cast<const uint32_t*>(g.w) + row, wb[u], pol);
            } else {
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    col[u][j] = NONE;
                    wb[u][j] = 0u;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < H; ++j) {
                colg[u][j] = group_slot<G>(col[u], j, grp);
                wbg[u][j] = group_slot<G>(wb[u], j, grp);
            }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < H; ++j) {
                colg[u][j] = NONE;
                wbg[u][j] = 0u;
                if (pp + u < np) {
                    const size_t at = (size_t)(p0 + pp + u) * K + (size_t)(j * G) + grp;
                    colg[u][j] = ld_nc(g.vcol + at);
                    wbg[u][j] = __float_as_uint(__ldg(g.w + at));
                }
            }
    }
}
// Compensated sum of scalar partials [first, first+cnt); all lanes return the same value.
__device__ float sum_scalars(const float* base, uint32_t first, uint32_t cnt, uint32_t lane) {
    float hi = 0.f, lo = 0.f;
    for (uint32_t i = lane; i < cnt; i += 32) pair_add(hi, lo, __ldcg(base + first + i), 0.f);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const float h2 = __shfl_xor_sync(FULL, hi, o), l2 = __shfl_xor_sync(FULL, lo, o);
        pair_add(hi, lo, h2, l2);
    }
    return hi;
}

// Arrival at a counter; true in the warp that completes `target` arrivals. Warp-collective.
__device__ __forceinline__ bool arrive_last(uint32_t* ctr, uint32_t target, uint32_t lane) {
    uint32_t last = 0;
    if (lane == 0) {
        __threadfence();
        last = (atomicAdd(ctr, 1u) + 1u == target) ? 1u : 0u;
    }
    last = __shfl_sync(FULL, last, 0);
    if (last) __threadfence();
    return last != 0;
}

// Next chunk of this CTA's strided share of the chunk list (blockIdx.x + i * gridDim.x: CTAs get
// similar mixes of hub and leaf chunks), drawn by its warps through a shared counter so that no warp
// idles while another of the CTA still has chunks queued. NONE when the share is used up. Warp-collective.
__device__ __forceinline__ uint32_t next_chunk(uint32_t* ctr, uint32_t nchunks, uint32_t lane) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(ctr, 1u);
    i = __shfl_sync(FULL, i, 0);
    const uint64_t c = blockIdx.x + (uint64_t)i * gridDim.x;
    return c < nchunks ? (uint32_t)c : NONE;
}

// Hub chunk delivery, batched rows. `tot` is the chunk's row (same in every lane group). Returns true
// in the warp that completes the hub for this sweep (`mult` = sweeps completed including this one), with
// the hub's full row in `out` and its vertex in `v`. Warp-collective.
template <int NQ>
__device__ bool hub_rows(const DirTab& g, const Chunk& ch, const float4& tot, uint32_t mult, uint32_t lane,
                         float4& out, uint32_t& v) {
    const uint32_t grp = lane / NQ, q = lane % NQ;
    const Hub H = g.hub[ch.hub];
    float4* part = reinterpret_cast<float4*>(g.partial);
    float4* gpart = reinterpret_cast<float4*>(g.gpartial);
    if (grp == 0) {
        part[(size_t)(H.first + ch.idx) * NQ + q] = tot;
        __threadfence();
    }
    __syncwarp();
    const uint32_t gi = ch.idx / PPR_GROUP, g0 = gi * PPR_GROUP;
    const uint32_t gs = min(PPR_GROUP, H.count - g0);
    if (!arrive_last(&g.garrive[H.gfirst + gi], mult * gs, lane)) return false;
    const float4 s1 = sum_rows<NQ>(part, H.first + g0, gs, grp, q);
    const uint32_t ng = (H.count + PPR_GROUP - 1) / PPR_GROUP;
    v = H.v;
    if (ng == 1) {
        out = s1;
        return true;
    }
    if (grp == 0) {
        gpart[(size_t)(H.gfirst + gi) * NQ + q] = s1;
        __threadfence();
    }
    __syncwarp();
    if (!arrive_last(&g.harrive[ch.hub], mult * ng, lane)) return false;
    out = sum_rows<NQ>(gpart, H.gfirst, ng, grp, q);
    return true;
}
// Same for one scalar per chunk.
__device__ bool hub_scalar(const DirTab& g, const Chunk& ch, float tot, uint32_t mult, uint32_t lane, float& out,
                           uint32_t& v) {
    const Hub H = g.hub[ch.hub];
    if (lane == 0) {
        g.partial[H.first + ch.idx] = tot;
        __threadfence();
    }
    __syncwarp();
    const uint32_t gi = ch.idx / PPR_GROUP, g0 = gi * PPR_GROUP;
    const uint32_t gs = min(PPR_GROUP, H.count - g0);
    if (!arrive_last(&g.garrive[H.gfirst + gi], mult * gs, lane)) return false;
    const float s1 = sum_scalars(g.partial, H.first + g0, gs, lane);
    const uint32_t ng = (H.count + PPR_GROUP - 1) / PPR_GROUP;
    v = H.v;
    if (ng == 1) {
        out = s1;
        return true;
    }
    if (lane == 0) {
        g.gpartial[H.gfirst + gi] = s1;
        __threadfence();
    }
    __syncwarp();
    if (!arrive_last(&g.harrive[ch.hub], mult * ng, lane)) return false;
    out = sum_scalars(g.gpartial, H.gfirst, ng, lane);
    return true;
}

// End of a sweep: reduce the residual / norm (and the probe), barrier, stop test. Returns 0 = continue,
// 1 = converged, 2 = grid aborting. With RES the control's next step is in *ex (shared).
template <bool RES>
__device__ __forceinline__ int end_sweep(const SolveArgs& a, uint32_t s, double dr, double dn, double dq, int mode,
                                         Extrapolation* ex, uint32_t& epoch) {
    PRCtrl* ctrl = a.ctrl;
    const bool probe = RES && mode == SW_PROBE;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        dr += __shfl_down_sync(FULL, dr, off);
        dn += __shfl_down_sync(FULL, dn, off);
        if (probe) dq += __shfl_down_sync(FULL, dq, off);
    }
    // one set of atomics per CTA: with one per warp, thousands of them queued at the same words every sweep (single
    // column, 490 K vertices of a grid 30.1 -> 24.4 us a sweep, R-MAT s18 54.3 -> 48.1)
    __shared__ double s_part[3][PPR_TPB / 32];
    if ((threadIdx.x & 31u) == 0) {
        s_part[0][threadIdx.x >> 5] = dr;
        s_part[1][threadIdx.x >> 5] = dn;
        s_part[2][threadIdx.x >> 5] = dq;
    }
    __syncthreads();
    if (threadIdx.x < 3u && (threadIdx.x < 2u || probe)) {
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < PPR_TPB / 32; ++w) sum += s_part[threadIdx.x][w];
        if (sum != 0.0) atomicAdd(threadIdx.x == 0u ? &ctrl->resid[s % 3] : (threadIdx.x == 1u ? &ctrl->norm[s % 3] : &ctrl->probe[s % 3]), sum);
    }
    if (!grid_barrier(&ctrl->bw, epoch, a.timeout_ns)) return 2;
    __shared__ double s_rn[2];  // one read per CTA instead of one per warp
    if (threadIdx.x == 0) {
        s_rn[0] = __ldcg(&ctrl->resid[s % 3]);
        s_rn[1] = __ldcg(&ctrl->norm[s % 3]);
        if (RES) extrapolation_next(*ex, s_rn[0], __ldcg(&ctrl->probe[s % 3]), (double)a.d);
    }
    __syncthreads();
    const double resid = s_rn[0], norm = s_rn[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // slot (s+2)%3 was last read before barrier s and is next accumulated after barrier s+1
        ctrl->resid[(s + 2) % 3] = 0.0;
        ctrl->norm[(s + 2) % 3] = 0.0;
        if (RES) {
            ctrl->probe[(s + 2) % 3] = 0.0;
            ctrl->far[(s + 2) % 3] = 0u;
        }
        ctrl->last_resid = resid;
        ctrl->last_norm = norm;
    }
    if (RES && mode == SW_STEP) return 0;  // its residual is that of the step's start
    const double tol = RES && ex->steps ? 0.25 * a.tol : a.tol;
    return ((double)a.d / (1.0 - (double)a.d) * resid <= tol * norm) ? 1 : 0;
}

// A solve with long steps whose L1 test is met after sweep s looks at every element of its iterate (see
// VertexBound): 0 = one is off, and the control's next step is set for it; 1 = none is; 2 = the grid is aborting.
// Forward solves only: their values are sums of one sign, so each has a size of its own to be measured by (a source with
// a negative entry leaves the look out: what cancels has none, and would keep the solve sweeping).
// (Adjoints, whose values cancel, came out as close as from plain sweeps, element by element, in the same 64-bit
// model.) Symmetrised R-MAT s14-s17, 32 seeds a column: elements 1e-4 to 1e-3 off without it, 8e-7 with it, 3e-7 to
// 2e-6 with plain sweeps; 15 to 25 more sweeps. The estimate (before two more plain sweeps) is there 1e-3 and more, on
// directed graphs mostly below 6e-6 with elements 1e-9 to 6e-8 off: 64 tol at the first look, then 8 tol (at 8 tol
// from the start directed graphs took one sweep more). The look takes 35 us of 3.4 ms (R-MAT s18, 64 columns). Not
// inlined: the gather loop needs the registers.
constexpr double PPR_FIRST = 64.0, PPR_LATER = 8.0;
static __device__ __noinline__ int look(const SolveArgs& a, uint32_t width, uint32_t s, uint32_t epoch, Extrapolation* ex) {
    const float most = ex->looks ? a.bound.later : a.bound.first;
    const float *f = (s & 1u) ? a.y0 : a.y1, *fo = (s & 1u) ? a.y1 : a.y0, *y = a.y;
    const uint64_t count = (uint64_t)a.n * width;
    uint32_t far = 0;
    const bool signs = ex->looks == 0u;  // the first look also looks for a negative source
    const float4* b4 = reinterpret_cast<const float4*>(a.b);
    auto one = [&](float fv, float yv, uint64_t i) {
        far |= vertex_off<true>(most, a.bound.d, fv, yv, [&]() { return fo[i]; }) ? 1u : 0u;
    };
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
#pragma unroll 2
    for (uint64_t i = t0; i < count / 4u; i += step) {
        const float4 fv = reinterpret_cast<const float4*>(f)[i], yv = reinterpret_cast<const float4*>(y)[i];
        one(fv.x, yv.x, 4u * i);
        one(fv.y, yv.y, 4u * i + 1u);
        one(fv.z, yv.z, 4u * i + 2u);
        one(fv.w, yv.w, 4u * i + 3u);
        if (signs && width > 1u) {
            const float4 b = b4[i];
            far |= fminf(fminf(b.x, b.y), fminf(b.z, b.w)) < 0.f ? 2u : 0u;
        }
    }
    for (uint64_t i = count / 4u * 4u + t0; i < count; i += step) one(f[i], y[i], i);
    if (signs && width == 1u)  // a single column's source need not be aligned
        for (uint64_t i = t0; i < count; i += step) far |= a.b[i] < 0.f ? 2u : 0u;
    far = (__syncthreads_or(far & 1u) ? 1u : 0u) | (__syncthreads_or(far & 2u) ? 2u : 0u);
    if (threadIdx.x == 0 && far) atomicOr(&a.ctrl->far[s % 3u], far);
    if (!grid_barrier(&a.ctrl->bw, epoch, a.timeout_ns)) return 2;
    __shared__ uint32_t s_far;
    if (threadIdx.x == 0) {
        const uint32_t found = __ldcg(&a.ctrl->far[s % 3u]);
        s_far = found == 1u ? 1u : 0u;
        if (s_far) vertices_off(*ex, (double)a.d);
    }
    __syncthreads();
    return s_far ? 0 : 1;
}

// One element of a vertex's end in residual form: yv the iterate's (FIRST: the source row's) old value, fo
// the old residual (PROBE and STEP), acc the gathered sum. Returns the new residual; yv becomes the new
// iterate. A long step cancels: its products go in as exact pairs.
__device__ __forceinline__ float res_elem(const SolveArgs& a, int mode, float alpha, float acc, float fo, float& yv,
                                          float& q) {
    float g = fmaf(a.d_lo, acc, a.d * acc);
    if (mode == SW_FIRST) {
        g = fmaf(a.scale_lo, g, a.scale_b * g);
        yv = fmaf(a.scale_lo, yv, a.scale_b * yv);
    } else if (mode == SW_PROBE) {
        q += fabsf(fmaf(-(1.f - 1.f / alpha), fo, g));
    } else if (mode == SW_STEP) {
        const float add = alpha * g, add_lo = fmaf(alpha, g, -add), b = 1.f - alpha;
        const float p = b * fo, p_lo = fmaf(b, fo, -p);
        float f, e, s, es;
        two_sum(p, add, f, e);
        two_sum(yv, add, s, es);
        yv = __fadd_rn(s, __fadd_rn(es, add_lo));
        return __fadd_rn(f, __fadd_rn(e, __fadd_rn(p_lo, add_lo)));
    }
    yv += g;
    return g;
}

// ------------------------------------------------------------------ batched rows: solve
// The vertex's end: its sum over the lane groups, then the new rows. bv: the source row (VALUE) or the
// iterate's old row (FIRST: the source row); ov: the old iterate (VALUE) or residual (PROBE, STEP).
struct SweepEnd {
    int mode;
    float alpha;  // STEP: the step length; PROBE: the one measured for
    float4* out;  // VALUE: iterates; residual form: residuals
    float4* y;    // residual form: iterates
};
template <int NQ, bool RES>
__device__ __forceinline__ void finish_row(const SolveArgs& a, const SweepEnd& e, uint32_t v, const float4& sum, float4 bv,
                                           const float4& ov, uint32_t grp, uint32_t q, float& rr, float& nn, float& qq) {
    if (!RES || e.mode == SW_VALUE) {
        const float4 y = affine4(a.d, a.d_lo, sum, a.scale_b, a.scale_lo, bv);
        if (grp == 0) {
            e.out[(size_t)v * NQ + q] = y;
            rr += l1diff4(y, ov);
            nn += l14(y);
        }
        return;
    }
    if (grp == 0) {
        float4 f;
        f.x = res_elem(a, e.mode, e.alpha, sum.x, ov.x, bv.x, qq);
        f.y = res_elem(a, e.mode, e.alpha, sum.y, ov.y, bv.y, qq);
        f.z = res_elem(a, e.mode, e.alpha, sum.z, ov.z, bv.z, qq);
        f.w = res_elem(a, e.mode, e.alpha, sum.w, ov.w, bv.w, qq);
        e.out[(size_t)v * NQ + q] = f;
        e.y[(size_t)v * NQ + q] = bv;
        rr += l14(f);
        nn += l14(bv);
    }
}

// A chunk's neighbour ids and weights (at most 128 each), staged in shared memory while the chunk before is
// worked on: 16-byte asynchronous copies, four slots per lane and array (rows are 16-byte aligned).
struct Stage {
    uint32_t col[PPR_SLOTS];
    float w[PPR_SLOTS];
};
__device__ __forceinline__ void stage_chunk(const DirTab& g, Stage* s, uint32_t p0, uint32_t slots, uint32_t K, uint32_t lane) {
    if (4u * lane < slots) {
        const size_t at = (size_t)p0 * K + 4u * lane;
        const uint32_t dc = (uint32_t)__cvta_generic_to_shared(s->col + 4u * lane);
        const uint32_t dw = (uint32_t)__cvta_generic_to_shared(s->w + 4u * lane);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dc), "l"(g.vcol + at) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dw), "l"(g.w + at) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The solve is latency-bound: nothing but the row gathers is left on a step's chain of loads -- the chunk's ids
// and weights come from shared memory, and the next chunk's description, owners, ids and weights are fetched
// while the current one is gathered; for 64 columns what is the same in the whole grid, and the FP64 sums,
// are kept in shared memory (8 row gathers take 32 of a lane's registers; 32 columns, whose vertices end twice
// as often per gather, keep them in registers: 125 against 147 us a sweep). R-MAT s18 x 64 columns, one sweep: 183 us with
// the ids loaded step by step and 150 bytes spilled, 158 us so with 3 CTAs per SM (24 warps; 56 bytes spilled).
//   The kinds of vertex end, inlined together, still spill: 168 bytes of stores and 192 to 268 of loads at 64 registers, 164
// to 232 and 144 to 204 for 32 columns. A function per kind of sweep, called once per sweep, spills 24 to 112 in the loops
// that count and is slower on R-MAT (s18 156 -> 164 us, 32 columns 125 -> 141).
//   CTAS = 4 (64 registers): more rows in flight where they come from beyond L2 or its far half:
// s18 158 -> 155 us, s20 625 -> 575; but s16 51 -> 53, 100 K vertices with K = 16 50 -> 55. So 4 is taken
// for rows above 48 MB. NQ = W/4 lanes per row.
constexpr size_t PPR_MANY_ROWS = (size_t)48 << 20;
template <int K, int NQ, bool RES, int CTAS>
__global__ void __launch_bounds__(PPR_TPB, CTAS) k_ppr_rows(const __grid_constant__ SolveArgs a) {
    constexpr int G = 32 / NQ;               // lane groups (rows per gather instruction)
    constexpr int H = K / G;                 // slots per group per part
    constexpr int U = RowStep<K, G>::U;      // parts per step: 8 row gathers in flight per lane
    constexpr bool KEEP = NQ == 8;           // sweep state and sums in registers
    static_assert(H >= 1 && H <= 8, "K must be at least the number of lane groups");
    const uint32_t lane = threadIdx.x & 31u, grp = lane / NQ, q = lane % NQ;
    __shared__ uint32_t s_next[2];  // per sweep (alternating): next of this CTA's chunks
    __shared__ __align__(16) Stage s_stage[PPR_TPB / 32][2];
    if (threadIdx.x == 0) s_next[0] = s_next[1] = 0u;
    __syncthreads();
    Stage* stage = s_stage[threadIdx.x >> 5];
    __shared__ SweepEnd s_end;            // this sweep's end of a vertex
    __shared__ double s_sum[KEEP ? 1 : 3][KEEP ? 1 : PPR_TPB];  // each thread's residual, norm and probe of the sweep
    const float4* b = reinterpret_cast<const float4*>(a.b);
    __shared__ Extrapolation s_ex;
    uint32_t epoch = 0, s = 0;
    bool conv = false;
    uint32_t tail = 0;  // residual form: value-form sweeps left before the end
    if (threadIdx.x == 0) extrapolation_init(s_ex);
    {
        float4* y0 = reinterpret_cast<float4*>(a.y0);
        float4* y1 = reinterpret_cast<float4*>(a.y1);
        float4* yy = reinterpret_cast<float4*>(a.y);
        float4* re = reinterpret_cast<float4*>(a.res);
        const uint64_t tot = (uint64_t)a.n * NQ;
        for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot;
             i += (uint64_t)gridDim.x * blockDim.x) {
            if (RES) {  // only the rows no sweep writes: iterate s b, residual 0
                const uint32_t v = (uint32_t)(i / NQ);
                if (a.g.vstart[v + 1] != a.g.vstart[v]) continue;
            }
            const float4 v = b[i];
            const float4 y = affine4(0.f, 0.f, f4(0.f), a.scale_b, a.scale_lo, v);
            if (RES) {
                y0[i] = y1[i] = f4(0.f);
                yy[i] = y;
            } else {
                y0[i] = y;
                y1[i] = y;
            }
        }
        if (!grid_barrier(&a.ctrl->bw, epoch, a.timeout_ns)) goto finish;
        for (; s < a.max_iters || tail; ++s) {
            SweepEnd e;  // the same in every thread; kept in shared memory for the vertices' ends
            e.mode = SW_VALUE;
            e.alpha = 1.f;
            e.out = (s & 1u) ? y0 : y1;
            e.y = yy;
            const float4* in = (s & 1u) ? y1 : y0;
            const float4* own = b;  // the row a vertex's end adds to
            if (RES && tail) {
                in = tail == 2u ? yy : y0;
                e.out = tail == 2u ? y0 : re;
            } else if (RES) {
                e.mode = s == 0u ? SW_FIRST : (s_ex.alpha != 1.f ? SW_STEP : (s_ex.cand != 0.f ? SW_PROBE : SW_PLAIN));
                e.alpha = e.mode == SW_STEP ? s_ex.alpha : s_ex.cand;
                if (s == 0u) in = b;
                else own = yy;
            }
            // the rows whose old values a vertex's end reads; the other sweeps skip the load
            const bool want_old = !RES || e.mode == SW_PROBE || e.mode == SW_STEP;
            const int mode = e.mode;
            double dr = 0.0, dn = 0.0, dq = 0.0;
            if (!KEEP) {
                s_sum[0][threadIdx.x] = s_sum[1][threadIdx.x] = s_sum[2][threadIdx.x] = 0.0;
                if (threadIdx.x == 0) s_end = e;
                __syncthreads();
            }
            const SweepEnd& end = KEEP ? e : s_end;
            if (threadIdx.x == 0) s_next[(s + 1u) & 1u] = 0u;  // next sweep's; ordered by the sweep's grid barrier
            // the next chunk: its parts and hub index (z); no parts when the share is used up
            auto draw = [&](uint32_t& c, uint3& parts) {
                c = next_chunk(&s_next[s & 1u], a.g.nchunks, lane);
                const Chunk h = c != NONE ? a.g.chunk[c] : Chunk{0u, 0u, NONE, 0u};
                parts = make_uint3(h.p0, h.p1, h.hub);
            };
            auto fetch = [&](uint3 parts, uint32_t st) -> uint32_t {  // its rows into stage st; its owners
                stage_chunk(a.g, stage + st, parts.x, (parts.y - parts.x) * K, K, lane);
                return lane < parts.y - parts.x ? ld_nc(a.g.vowner + parts.x + lane) : NONE;
            };
            uint32_t c, c_next;
            uint3 parts, parts_next;
            draw(c, parts);
            uint32_t sid = 0;
            uint32_t own_l = fetch(parts, sid);
            draw(c_next, parts_next);
            for (; c != NONE; c = c_next, parts = parts_next, draw(c_next, parts_next)) {
                const uint32_t own_next = fetch(parts_next, sid ^ 1u);
                asm volatile("cp.async.wait_group 1;" ::: "memory");  // this chunk's stage has landed
                __syncwarp();
                const Stage& sg = stage[sid];
                const uint32_t np = parts.y - parts.x;
                uint32_t cur = __shfl_sync(FULL, own_l, 0);
                float4 bv = own[(size_t)cur * NQ + q];
                float4 ov = want_old ? in[(size_t)cur * NQ + q] : f4(0.f);
                float4 acc = f4(0.f);
                float rr = 0.f, nn = 0.f, qq = 0.f;
                for (uint32_t pp = 0; pp < np; pp += U) {
                    float4 xv[U][H];
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int j = 0; j < H; ++j) {
                            const uint32_t id = pp + u < np ? sg.col[(pp + u) * K + j * G + grp] : NONE;
                            xv[u][j] = id != NONE ? in[(size_t)id * NQ + q] : f4(0.f);
                        }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (pp + u < np) {
                            const uint32_t o = __shfl_sync(FULL, own_l, pp + u);
                            if (o != cur) {
                                finish_row<NQ, RES>(a, end, cur, across_groups<NQ>(acc), bv, ov, grp, q, rr, nn, qq);
                                acc = f4(0.f);
                                cur = o;
                                bv = own[(size_t)cur * NQ + q];
                                if (want_old) ov = in[(size_t)cur * NQ + q];
                            }
#pragma unroll
                            for (int j = 0; j < H; ++j) fma4(acc, sg.w[(pp + u) * K + j * G + grp], xv[u][j]);
                        }
                    }
                }
                const float4 tot = across_groups<NQ>(acc);
                if (parts.z == NONE) {
                    finish_row<NQ, RES>(a, end, cur, tot, bv, ov, grp, q, rr, nn, qq);
                } else {
                    float4 full;
                    uint32_t v;
                    if (hub_rows<NQ>(a.g, a.g.chunk[c], tot, s + 1, lane, full, v))
                        finish_row<NQ, RES>(a, end, v, full, own[(size_t)v * NQ + q],
                                            want_old ? in[(size_t)v * NQ + q] : f4(0.f), grp, q, rr, nn, qq);
                }
                if (KEEP) {
                    dr += (double)rr;
                    dn += (double)nn;
                    if (RES) dq += (double)qq;
                } else {
                    s_sum[0][threadIdx.x] += (double)rr;
                    s_sum[1][threadIdx.x] += (double)nn;
                    if (RES) s_sum[2][threadIdx.x] += (double)qq;
                }
                own_l = own_next;
                sid ^= 1u;
                __syncwarp();  // every lane has read the stage before it is filled again
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (RES && tail) {  // rows without parts: the value is s b
                for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < tot;
                     i += (uint64_t)gridDim.x * blockDim.x) {
                    const uint32_t v = (uint32_t)(i / NQ);
                    if (a.g.vstart[v + 1] == a.g.vstart[v]) end.out[i] = yy[i];
                }
                if (--tail) {
                    if (!grid_barrier(&a.ctrl->bw, epoch, a.timeout_ns)) goto finish;
                    continue;
                }
                conv = true;
                ++s;
                break;
            }
            if (!KEEP) {
                dr = s_sum[0][threadIdx.x];
                dn = s_sum[1][threadIdx.x];
                dq = s_sum[2][threadIdx.x];
            }
            const int st = end_sweep<RES>(a, s, dr, dn, dq, mode, &s_ex, epoch);
            if (st == 2) goto finish;
            if (st == 1) {
                if (RES) {
                    const int seen = s_ex.steps && s + 1u < a.bound.sweeps ? look(a, 4u * NQ, s, epoch++, &s_ex) : 1;
                    if (seen == 2) goto finish;
                    if (seen == 1) tail = 2u;
                } else {
                    ++s;
                    conv = true;
                    break;
                }
            }
        }
    }
    if (!conv && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&a.ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_ITER_CAP);
finish:
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctrl->iterations = s;
}

// ------------------------------------------------------------------ single column: solve
template <int K, bool RES>
__global__ void __launch_bounds__(PPR_TPB, 4) k_ppr_scalar(const __grid_constant__ SolveArgs a) {
    constexpr int PPS = 32 / K;                   // parts per 32-slot step
    constexpr int STEPS = (int)PPR_SLOTS / 32;    // steps per chunk
    const uint32_t lane = threadIdx.x & 31u;
    __shared__ uint32_t s_next[2];  // per sweep (alternating): next of this CTA's chunks
    if (threadIdx.x == 0) s_next[0] = s_next[1] = 0u;
    __syncthreads();
    const float* b = a.b;
    __shared__ Extrapolation s_ex;
    uint32_t epoch = 0, s = 0;
    bool conv = false;
    uint32_t tail = 0;  // residual form: value-form sweeps left before the end
    if (threadIdx.x == 0) extrapolation_init(s_ex);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (RES && a.g.vstart[i + 1] != a.g.vstart[i]) continue;  // only the rows no sweep writes
        const float y = fmaf(a.scale_lo, b[i], a.scale_b * b[i]);
        if (RES) {
            a.y0[i] = a.y1[i] = 0.f;
            a.y[i] = y;
        } else {
            a.y0[i] = y;
            a.y1[i] = y;
        }
    }
    if (!grid_barrier(&a.ctrl->bw, epoch, a.timeout_ns)) goto finish;
    for (; s < a.max_iters || tail; ++s) {
        const float* in = (s & 1u) ? a.y1 : a.y0;
        float* out = (s & 1u) ? a.y0 : a.y1;
        const float* own = b;  // the value a vertex's end adds to
        int mode = SW_VALUE;
        float alpha = 1.f;
        if (RES && tail) {
            in = tail == 2u ? a.y : a.y0;
            out = tail == 2u ? a.y0 : a.res;
        } else if (RES) {
            mode = s == 0u ? SW_FIRST : (s_ex.alpha != 1.f ? SW_STEP : (s_ex.cand != 0.f ? SW_PROBE : SW_PLAIN));
            alpha = mode == SW_STEP ? s_ex.alpha : s_ex.cand;
            if (s == 0u) in = b;
            else own = a.y;
        }
        const bool want_old = !RES || mode == SW_PROBE || mode == SW_STEP;
        double dr = 0.0, dn = 0.0, dq = 0.0;
        // one vertex's end, by one lane
        auto finish_one = [&](uint32_t v, float sum, float& rr, float& nn, float& qq) {
            float ov = want_old ? in[v] : 0.f, bv = own[v];
            if (!RES || mode == SW_VALUE) {
                const float y = affine(a.d, a.d_lo, sum, a.scale_b, a.scale_lo, bv);
                rr += fabsf(y - ov);
                nn += fabsf(y);
                out[v] = y;
            } else {
                const float f = res_elem(a, mode, alpha, sum, ov, bv, qq);
                out[v] = f;
                a.y[v] = bv;
                rr += fabsf(f);
                nn += fabsf(bv);
            }
        };
        if (threadIdx.x == 0) s_next[(s + 1u) & 1u] = 0u;  // next sweep's; ordered by the sweep's grid barrier
        for (uint32_t c; (c = next_chunk(&s_next[s & 1u], a.g.nchunks, lane)) != NONE;) {
            const Chunk ch = a.g.chunk[c];
            const uint32_t np = ch.p1 - ch.p0;
            const uint32_t nsl = np * K;
            const size_t base = (size_t)ch.p0 * K;
            const uint32_t own_l = lane < np ? ld_nc(a.g.vowner + ch.p0 + lane) : NONE;
            uint32_t col[STEPS];
            float wv[STEPS], xv[STEPS];
#pragma unroll
            for (int st = 0; st < STEPS; ++st) {
                const uint32_t idx = (uint32_t)st * 32u + lane;
                col[st] = idx < nsl ? ld_nc(a.g.vcol + base + idx) : NONE;
                wv[st] = idx < nsl ? __ldg(a.g.w + base + idx) : 0.f;
            }
#pragma unroll
            for (int st = 0; st < STEPS; ++st) xv[st] = col[st] != NONE ? in[col[st]] : 0.f;
            float psum = 0.f;
#pragma unroll
            for (int st = 0; st < STEPS; ++st) {
                if ((uint32_t)st * 32u < nsl) {
                    float v = wv[st] * xv[st];
#pragma unroll
                    for (int o = K / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
#pragma unroll
                    for (int i = 0; i < PPS; ++i) {
                        const float t = __shfl_sync(FULL, v, i * K);
                        if (lane == (uint32_t)(st * PPS + i)) psum = t;
                    }
                }
            }
            // vertex sums: segmented inclusive scan over the part lanes
            const uint32_t prev = __shfl_up_sync(FULL, own_l, 1);
            const bool head = lane == 0 || own_l != prev;
            const uint32_t hm = __ballot_sync(FULL, head);
            const uint32_t start = 31u - __clz(hm & (((lane == 31u) ? 0u : (2u << lane)) - 1u));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float t = __shfl_up_sync(FULL, psum, o);
                if (lane >= (uint32_t)o && lane - (uint32_t)o >= start) psum += t;
            }
            float rr = 0.f, nn = 0.f, qq = 0.f;
            if (ch.hub == NONE) {
                const uint32_t next = __shfl_down_sync(FULL, own_l, 1);
                const bool lastl = lane < np && (lane == np - 1 || next != own_l);
                if (lastl) finish_one(own_l, psum, rr, nn, qq);
            } else {
                const float tot = __shfl_sync(FULL, psum, np - 1);
                float full;
                uint32_t v;
                if (hub_scalar(a.g, ch, tot, s + 1, lane, full, v) && lane == 0) finish_one(v, full, rr, nn, qq);
            }
            dr += (double)rr;
            dn += (double)nn;
            if (RES) dq += (double)qq;
        }
        if (RES && tail) {  // rows without parts: the value is s b
            for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n;
                 i += (uint64_t)gridDim.x * blockDim.x)
                if (a.g.vstart[i + 1] == a.g.vstart[i]) out[i] = a.y[i];
            if (--tail) {
                if (!grid_barrier(&a.ctrl->bw, epoch, a.timeout_ns)) goto finish;
                continue;
            }
            conv = true;
            ++s;
            break;
        }
        const int st = end_sweep<RES>(a, s, dr, dn, dq, mode, &s_ex, epoch);
        if (st == 2) goto finish;
        if (st == 1) {
            if (RES) {
                const int seen = s_ex.steps && s + 1u < a.bound.sweeps ? look(a, 1u, s, epoch++, &s_ex) : 1;
                if (seen == 2) goto finish;
                if (seen == 1) tail = 2u;
            } else {
                ++s;
                conv = true;
                break;
            }
        }
    }
    if (!conv && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&a.ctrl->bw.status, (uint32_t)DEV_OK, (uint32_t)DEV_ITER_CAP);
finish:
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ctrl->iterations = s;
}

// ------------------------------------------------------------------ gradients
// Batched rows: g_uv = d <X_u, L_v> per forward slot; r_u = sum_v g_uv W_uv per vertex.
template <int K, int NQ>
__global__ void __launch_bounds__(PPR_TPB, 2) k_ppr_grad_rows(GradArgs a) {
    constexpr int G = 32 / NQ;
    constexpr int H = K / G;
    constexpr int U = RowStep<K, G>::U;
    static_assert(H >= 1 && H <= NQ, "K must be at least the number of lane groups");
    const uint32_t lane = threadIdx.x & 31u, grp = lane / NQ, q = lane % NQ;
    __shared__ uint32_t s_next[2];  // per sweep (alternating): next of this CTA's chunks
    if (threadIdx.x == 0) s_next[0] = s_next[1] = 0u;
    __syncthreads();
    const uint64_t pol = l2_evict_first_policy();
    const float4* X = reinterpret_cast<const float4*>(a.X);
    const float4* L = reinterpret_cast<const float4*>(a.L);
    const uint32_t ri = red_index<H, NQ>(q);
    const uint32_t jme = (uint32_t)G * ri + grp;               // slot this lane reports after the reduction
    const bool writer = (q & (uint32_t)(NQ / H - 1)) == 0u;    // one lane per reduced value
    for (uint32_t c; (c = next_chunk(&s_next[0], a.g.nchunks, lane)) != NONE;) {
        const Chunk ch = a.g.chunk[c];
        const uint32_t np = ch.p1 - ch.p0;
        const uint32_t own_l = lane < np ? ld_nc(a.g.vowner + ch.p0 + lane) : NONE;
        uint32_t cur = __shfl_sync(FULL, own_l, 0);
        float4 xu = X[(size_t)cur * NQ + q];
        float racc = 0.f;
        for (uint32_t pp = 0; pp < np; pp += U) {
            uint32_t colg[U][H], wbg[U][H];
            load_group_slots<K, G>(a.g, ch.p0, pp, np, grp, pol, colg, wbg);
            float4 lv[U][H];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    const uint32_t id = colg[u][j];
                    lv[u][j] = id != NONE ? L[(size_t)id * NQ + q] : f4(0.f);
                }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (pp + u < np) {
                    const uint32_t o = __shfl_sync(FULL, own_l, pp + u);
                    if (o != cur) {
                        float t = racc;
#pragma unroll
                        for (int off = 16; off >= 1; off >>= 1) t += __shfl_xor_sync(FULL, t, off);
                        if (lane == 0) a.r[cur] = a.accumulate ? a.r[cur] + t : t;
                        racc = 0.f;
                        cur = o;
                        xu = X[(size_t)cur * NQ + q];
                    }
                    float dv[H];
#pragma unroll
                    for (int j = 0; j < H; ++j) dv[j] = dot4(xu, lv[u][j]);
                    const float dsum = tred<H, NQ>(dv, q);
                    const uint32_t id = pick<H>(colg[u], ri);  // slot jme of the part
                    if (writer && id != NONE) {
                        const float g = a.d * dsum;
                        const size_t slot = (size_t)(ch.p0 + pp + u) * K + jme;
                        a.gslot[slot] = a.accumulate ? a.gslot[slot] + g : g;
                        racc = fmaf(g, __uint_as_float(pick<H>(wbg[u], ri)), racc);
                    }
                }
            }
        }
        float t = racc;
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) t += __shfl_xor_sync(FULL, t, off);
        if (ch.hub == NONE) {
            if (lane == 0) a.r[cur] = a.accumulate ? a.r[cur] + t : t;
        } else {
            float full;
            uint32_t v;
            if (hub_scalar(a.g, ch, t, 1u, lane, full, v) && lane == 0) a.r[v] = a.accumulate ? a.r[v] + full : full;
        }
    }
}

// Single column: the same per slot, X and L scalars.
template <int K>
__global__ void __launch_bounds__(PPR_TPB, 4) k_ppr_grad_scalar(GradArgs a) {
    constexpr int PPS = 32 / K;
    constexpr int STEPS = (int)PPR_SLOTS / 32;
    const uint32_t lane = threadIdx.x & 31u;
    __shared__ uint32_t s_next[2];  // per sweep (alternating): next of this CTA's chunks
    if (threadIdx.x == 0) s_next[0] = s_next[1] = 0u;
    __syncthreads();
    for (uint32_t c; (c = next_chunk(&s_next[0], a.g.nchunks, lane)) != NONE;) {
        const Chunk ch = a.g.chunk[c];
        const uint32_t np = ch.p1 - ch.p0;
        const uint32_t nsl = np * K;
        const size_t base = (size_t)ch.p0 * K;
        const uint32_t own_l = lane < np ? ld_nc(a.g.vowner + ch.p0 + lane) : NONE;
        uint32_t col[STEPS];
        float wv[STEPS], gv[STEPS];
#pragma unroll
        for (int st = 0; st < STEPS; ++st) {
            const uint32_t idx = (uint32_t)st * 32u + lane;
            col[st] = idx < nsl ? ld_nc(a.g.vcol + base + idx) : NONE;
            wv[st] = idx < nsl ? __ldg(a.g.w + base + idx) : 0.f;
        }
#pragma unroll
        for (int st = 0; st < STEPS; ++st) {
            const uint32_t o = __shfl_sync(FULL, own_l, st * PPS + (int)(lane / K));
            gv[st] = 0.f;
            if (col[st] != NONE) {
                gv[st] = a.d * (a.X[o] * a.L[col[st]]);
                const size_t slot = base + (uint32_t)st * 32u + lane;
                a.gslot[slot] = a.accumulate ? a.gslot[slot] + gv[st] : gv[st];
            }
        }
        float psum = 0.f;
#pragma unroll
        for (int st = 0; st < STEPS; ++st) {
            if ((uint32_t)st * 32u < nsl) {
                float v = gv[st] * wv[st];
#pragma unroll
                for (int o = K / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
#pragma unroll
                for (int i = 0; i < PPS; ++i) {
                    const float t = __shfl_sync(FULL, v, i * K);
                    if (lane == (uint32_t)(st * PPS + i)) psum = t;
                }
            }
        }
        const uint32_t prev = __shfl_up_sync(FULL, own_l, 1);
        const bool head = lane == 0 || own_l != prev;
        const uint32_t hm = __ballot_sync(FULL, head);
        const uint32_t start = 31u - __clz(hm & (((lane == 31u) ? 0u : (2u << lane)) - 1u));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(FULL, psum, o);
            if (lane >= (uint32_t)o && lane - (uint32_t)o >= start) psum += t;
        }
        if (ch.hub == NONE) {
            const uint32_t next = __shfl_down_sync(FULL, own_l, 1);
            if (lane < np && (lane == np - 1 || next != own_l))
                a.r[own_l] = a.accumulate ? a.r[own_l] + psum : psum;
        } else {
            const float tot = __shfl_sync(FULL, psum, np - 1);
            float full;
            uint32_t v;
            if (hub_scalar(a.g, ch, tot, 1u, lane, full, v) && lane == 0) a.r[v] = a.accumulate ? a.r[v] + full : full;
        }
    }
}

// Per-edge outputs in input edge order.
__global__ void k_ppr_scatter(uint64_t nslots, uint32_t K, const uint32_t* __restrict__ veid,
                              const uint32_t* __restrict__ vowner, const float* __restrict__ gslot,
                              const float* __restrict__ r, const float* __restrict__ s, float* dwn, float* dw) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nslots; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t e = veid[i];
        if (e == NONE) continue;
        const float g = gslot[i];
        if (dwn) dwn[e] = g;
        if (dw) {
            const uint32_t u = vowner[i / K];
            const float su = s[u];
            dw[e] = su > 0.f ? (g - r[u]) / su : 0.f;
        }
    }
}

// out = (1-d) L  (dLoss/dT)
__global__ void k_ppr_scale(uint64_t count, float f, const float* __restrict__ in, float* __restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = f * in[i];
}

// ------------------------------------------------------------------ weights
// s_u = sum of u's raw out-weights over the forward chunks (a lane owns a slot, as in k_ppr_grad_scalar; a
// hub's chunks deliver partials: with a warp per vertex, R-MAT s18's first vertex alone took 0.27 ms), in a
// fixed order; vertices without out-edges keep the zero they were set to. Flags negative / non-finite weights.
template <int K>
__global__ void __launch_bounds__(PPR_TPB, 4) k_ppr_out_sums(DirTab g, const uint32_t* __restrict__ veid,
                                                             const float* __restrict__ w, float* __restrict__ s, uint32_t* bad) {
    constexpr int PPS = 32 / K;
    constexpr int STEPS = (int)PPR_SLOTS / 32;
    const uint32_t lane = threadIdx.x & 31u;
    __shared__ uint32_t s_next;
    if (threadIdx.x == 0) s_next = 0u;
    __syncthreads();
    uint32_t wrong = 0;
    for (uint32_t c; (c = next_chunk(&s_next, g.nchunks, lane)) != NONE;) {
        const Chunk ch = g.chunk[c];
        const uint32_t np = ch.p1 - ch.p0, nsl = np * K;
        const size_t base = (size_t)ch.p0 * K;
        const uint32_t own_l = lane < np ? ld_nc(g.vowner + ch.p0 + lane) : NONE;
        uint32_t e[STEPS];
        float x[STEPS];
#pragma unroll
        for (int st = 0; st < STEPS; ++st) {
            const uint32_t idx = (uint32_t)st * 32u + lane;
            e[st] = idx < nsl ? ld_nc(veid + base + idx) : NONE;
        }
#pragma unroll
        for (int st = 0; st < STEPS; ++st) x[st] = e[st] != NONE ? __ldg(w + e[st]) : 0.f;
        float psum = 0.f;
#pragma unroll
        for (int st = 0; st < STEPS; ++st) {
            if (!(x[st] >= 0.f) || !isfinite(x[st])) wrong = 1u;
            if ((uint32_t)st * 32u < nsl) {
                float v = x[st];
#pragma unroll
                for (int o = K / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
#pragma unroll
                for (int i = 0; i < PPS; ++i) {
                    const float t = __shfl_sync(FULL, v, i * K);
                    if (lane == (uint32_t)(st * PPS + i)) psum = t;
                }
            }
        }
        const uint32_t prev = __shfl_up_sync(FULL, own_l, 1);
        const uint32_t hm = __ballot_sync(FULL, lane == 0 || own_l != prev);
        const uint32_t start = 31u - __clz(hm & (((lane == 31u) ? 0u : (2u << lane)) - 1u));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(FULL, psum, o);
            if (lane >= (uint32_t)o && lane - (uint32_t)o >= start) psum += t;
        }
        if (ch.hub == NONE) {
            const uint32_t next = __shfl_down_sync(FULL, own_l, 1);
            if (lane < np && (lane == np - 1 || next != own_l)) s[own_l] = psum;
        } else {
            const float tot = __shfl_sync(FULL, psum, np - 1);
            float full;
            uint32_t v;
            if (hub_scalar(g, ch, tot, 1u, lane, full, v) && lane == 0) s[v] = full;
        }
    }
    if (__any_sync(FULL, wrong) && lane == 0) atomicOr(bad, 1u);
}
// Normalised weight per slot. Forward: the slot's source is the part owner; transposed: the slot's
// neighbour.
__global__ void k_ppr_norm(uint64_t nslots, uint32_t K, int transposed, const uint32_t* __restrict__ veid,
                           const uint32_t* __restrict__ vowner, const uint32_t* __restrict__ vcol,
                           const float* __restrict__ w, const float* __restrict__ s, float* __restrict__ wn) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nslots; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t e = veid[i];
        float r = 0.f;
        if (e != NONE) {
            const uint32_t u = transposed ? vcol[i] : vowner[i / K];
            const float su = s[u];
            r = su > 0.f ? w[e] / su : 0.f;
        }
        wn[i] = r;
    }
}

unsigned grid_1d(uint64_t work, int device) {
    const uint64_t cap = (uint64_t)sm_count(device) * 8;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((work + PPR_TPB - 1) / PPR_TPB, cap));
}

}  // namespace

// Host-held device tables of one direction.
struct PPRDir {
    Chunk* chunk = nullptr;
    uint32_t nchunks = 0;
    Hub* hub = nullptr;
    uint32_t nhubs = 0, nslots = 0, ngroups = 0;
    uint32_t* garrive = nullptr;
    uint32_t* harrive = nullptr;
    float* partial = nullptr;
    float* gpartial = nullptr;
    float* w = nullptr;  // normalised weight per slot
};

}  // namespace eeg

struct eeg_ppr {
    eeg_vgraph* vg = nullptr;
    uint32_t C = 1, W = 1;
    eeg::PPRDir fwd, rev;
    float* w_raw = nullptr;  // m
    float* s = nullptr;      // n
    uint32_t* bad = nullptr;
    float* Y[2] = {nullptr, nullptr};  // forward iterates (X in one of them until the next forward)
    float* Lb[2] = {nullptr, nullptr}; // adjoint iterates; residuals of the solves in residual form
    float* b = nullptr;                // staged input rows (n x W)
    float* gslot = nullptr;            // forward slots
    float* r = nullptr;                // n
    float* stage_m = nullptr;          // 2m: host-bound edge outputs
    float* stage_nw = nullptr;         // n x W: host-bound / repacked row outputs
    eeg::PRCtrl* ctrl = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    int xi = -1;  // Y buffer holding X after the last forward
    bool have_w = false, have_g = false;
    uint64_t bytes = 0;
};

namespace eeg {
namespace {

eeg_status ppr_alloc(eeg_ppr* p, void** ptr, size_t bytes) {
    EEG_TRY(vg_alloc(p->vg, ptr, bytes));
    p->bytes += bytes;
    return EEG_OK;
}

void free_pdir(eeg_ppr* p, PPRDir& d) {
    vg_free(p->vg, d.chunk);
    vg_free(p->vg, d.hub);
    vg_free(p->vg, d.garrive);
    vg_free(p->vg, d.harrive);
    vg_free(p->vg, d.partial);
    vg_free(p->vg, d.gpartial);
    vg_free(p->vg, d.w);
    d = PPRDir{};
}

// Cut one direction's parts into chunks (host; from vstart).
eeg_status build_chunks(eeg_ppr* p, const VDir& vd, PPRDir& d) {
    eeg_vgraph* vg = p->vg;
    const uint32_t n = vg->n, K = vg->K;
    const uint32_t CH = PPR_SLOTS / K;
    // Small graphs: chunks only as large as it takes to give every resident warp one. A chunk's vertices end one after
    // another (some 230 instructions each), so with full chunks a sweep of a 150^2 grid, 16 columns, was one warp's 16
    // vertices: 26.8 us, 18.6 so (64 columns 20.6 -> 15.9; a path of 5000 vertices 16.6 -> 11.6). A single column's chunk is
    // worked on by all lanes at once.
    const uint64_t warps = (uint64_t)sm_count(vg->device) * 24u;
    const uint32_t pack = p->W == 1 ? CH : (uint32_t)std::min<uint64_t>(CH, std::max<uint64_t>(1, (vd.P + warps - 1) / warps));
    std::vector<uint32_t> vs((size_t)n + 1);
    EEG_CUDA(cudaMemcpy(vs.data(), vd.vstart, sizeof(uint32_t) * ((size_t)n + 1), cudaMemcpyDeviceToHost));
    std::vector<Chunk> ch;
    std::vector<Hub> hubs;
    ch.reserve((size_t)(vd.P / CH) + 16);
    uint32_t slots = 0, groups = 0;
    uint32_t v = 0;
    while (v < n) {
        const uint32_t np = vs[v + 1] - vs[v];
        if (np == 0) {
            ++v;
            continue;
        }
        if (np > CH) {
            const uint32_t count = (np + CH - 1) / CH;
            const uint32_t h = (uint32_t)hubs.size();
            hubs.push_back(Hub{v, slots, count, groups});
            for (uint32_t i = 0; i < count; ++i)
                ch.push_back(Chunk{vs[v] + i * CH, std::min(vs[v] + (i + 1) * CH, vs[v + 1]), h, i});
            slots += count;
            groups += (count + PPR_GROUP - 1) / PPR_GROUP;
            ++v;
            continue;
        }
        const uint32_t p0 = vs[v];
        uint32_t p1 = vs[v + 1];
        ++v;
        while (v < n && vs[v + 1] - vs[v] <= CH && vs[v + 1] - p0 <= pack) {
            p1 = vs[v + 1];
            ++v;
        }
        ch.push_back(Chunk{p0, p1, NONE, 0});
    }
    d.nchunks = (uint32_t)ch.size();
    d.nhubs = (uint32_t)hubs.size();
    d.nslots = slots;
    d.ngroups = groups;
    EEG_TRY(ppr_alloc(p, (void**)&d.chunk, sizeof(Chunk) * std::max<size_t>(ch.size(), 1)));
    EEG_TRY(ppr_alloc(p, (void**)&d.hub, sizeof(Hub) * std::max<size_t>(hubs.size(), 1)));
    EEG_TRY(ppr_alloc(p, (void**)&d.garrive, sizeof(uint32_t) * std::max<uint32_t>(groups, 1)));
    EEG_TRY(ppr_alloc(p, (void**)&d.harrive, sizeof(uint32_t) * std::max<uint32_t>(d.nhubs, 1)));
    EEG_TRY(ppr_alloc(p, (void**)&d.partial, sizeof(float) * p->W * std::max<uint32_t>(slots, 1)));
    EEG_TRY(ppr_alloc(p, (void**)&d.gpartial, sizeof(float) * p->W * std::max<uint32_t>(groups, 1)));
    EEG_TRY(ppr_alloc(p, (void**)&d.w, sizeof(float) * std::max<size_t>((size_t)vd.P * K, 4)));
    if (!ch.empty())
        EEG_CUDA(cudaMemcpy(d.chunk, ch.data(), sizeof(Chunk) * ch.size(), cudaMemcpyHostToDevice));
    if (!hubs.empty())
        EEG_CUDA(cudaMemcpy(d.hub, hubs.data(), sizeof(Hub) * hubs.size(), cudaMemcpyHostToDevice));
    return EEG_OK;
}

DirTab tab(const VDir& vd, const PPRDir& d) {
    DirTab t{};
    t.vowner = vd.vowner;
    t.vcol = vd.vcol;
    t.w = d.w;
    t.chunk = d.chunk;
    t.nchunks = d.nchunks;
    t.hub = d.hub;
    t.garrive = d.garrive;
    t.harrive = d.harrive;
    t.partial = d.partial;
    t.gpartial = d.gpartial;
    t.vstart = vd.vstart;
    return t;
}

eeg_status reset_counters(const PPRDir& d, cudaStream_t st) {
    EEG_CUDA(cudaMemsetAsync(d.garrive, 0, sizeof(uint32_t) * std::max<uint32_t>(d.ngroups, 1), st));
    EEG_CUDA(cudaMemsetAsync(d.harrive, 0, sizeof(uint32_t) * std::max<uint32_t>(d.nhubs, 1), st));
    return EEG_OK;
}

template <typename Kern>
eeg_status launch_coop(Kern kern, void* arg, int device, uint32_t bps, uint64_t work_warps, cudaStream_t st) {
    int per_sm = 0;
    EEG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, PPR_TPB, 0));
    if (per_sm <= 0) {
        set_last_error("personalised PageRank kernel does not fit on an SM");
        return EEG_ERR_CUDA;
    }
    if (bps > 0 && (int)bps < per_sm) per_sm = (int)bps;
    uint64_t blocks = (uint64_t)per_sm * sm_count(device);
    const uint64_t need = (work_warps * 32 + PPR_TPB - 1) / PPR_TPB;
    if (need < blocks) blocks = std::max<uint64_t>(need, 1);
    void* params[] = {arg};
    EEG_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)blocks), dim3(PPR_TPB), params, 0, st));
    return EEG_OK;
}

template <int K, bool RES>
eeg_status launch_solve(eeg_ppr* p, SolveArgs& a, uint32_t bps, cudaStream_t st) {
    const uint64_t work = std::max<uint64_t>(a.g.nchunks, ((uint64_t)a.n * 16 + 31) / 32);
    if (p->W == 1) return launch_coop(k_ppr_scalar<K, RES>, &a, p->vg->device, bps, work, st);
    if (p->W == 32) return launch_coop(k_ppr_rows<K, 8, RES, 3>, &a, p->vg->device, bps, work, st);
    if (RES && (size_t)a.n * PPR_W * sizeof(float) > PPR_MANY_ROWS)
        return launch_coop(k_ppr_rows<K, 16, RES, RES ? 4 : 3>, &a, p->vg->device, bps, work, st);
    return launch_coop(k_ppr_rows<K, 16, RES, 3>, &a, p->vg->device, bps, work, st);
}

template <int K>
eeg_status launch_grad(eeg_ppr* p, GradArgs& a, cudaStream_t st) {
    const int dev = p->vg->device;
    const uint64_t cap = (uint64_t)sm_count(dev) * (p->W == 1 ? 4 : 2) * (PPR_TPB / 32);
    const uint64_t warps = std::max<uint64_t>(1, std::min<uint64_t>(a.g.nchunks, cap));
    const unsigned blocks = (unsigned)((warps * 32 + PPR_TPB - 1) / PPR_TPB);
    if (p->W == 1)
        k_ppr_grad_scalar<K><<<blocks, PPR_TPB, 0, st>>>(a);
    else if (p->W == 32)
        k_ppr_grad_rows<K, 8><<<blocks, PPR_TPB, 0, st>>>(a);
    else
        k_ppr_grad_rows<K, 16><<<blocks, PPR_TPB, 0, st>>>(a);
    EEG_CUDA(cudaGetLastError());
    return EEG_OK;
}

// Source rows for a solve: the caller's array when it already has the internal layout, else staged.
eeg_status stage_rows(eeg_ppr* p, const float* in, int on_device, cudaStream_t st, const float** out) {
    const uint32_t n = p->vg->n;
    const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    if (on_device && p->C == p->W && ((uintptr_t)in & 15u) == 0) {
        *out = in;
        return EEG_OK;
    }
    if (p->C == p->W)
        EEG_CUDA(cudaMemcpyAsync(p->b, in, sizeof(float) * (size_t)n * p->W, kind, st));
    else
        EEG_CUDA(cudaMemcpy2DAsync(p->b, sizeof(float) * p->W, in, sizeof(float) * p->C, sizeof(float) * p->C, n, kind, st));
    *out = p->b;
    return EEG_OK;
}

eeg_status unstage_rows(eeg_ppr* p, const float* src, float* dst, int on_device, cudaStream_t st) {
    const uint32_t n = p->vg->n;
    const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    if (p->C == p->W)
        EEG_CUDA(cudaMemcpyAsync(dst, src, sizeof(float) * (size_t)n * p->W, kind, st));
    else
        EEG_CUDA(cudaMemcpy2DAsync(dst, sizeof(float) * p->C, src, sizeof(float) * p->W, sizeof(float) * p->C, n, kind, st));
    return EEG_OK;
}

// X = p->Y[p->xi] is kept by an adjoint solve. *result: the buffer holding the solution.
eeg_status solve(eeg_ppr* p, bool adjoint, const float* bsrc, const eeg_options& o, cudaStream_t st,
                 eeg_result* res, float** result) {
    eeg_vgraph* vg = p->vg;
    const VDir& vd = adjoint ? vg->fwd : vg->rev;
    PPRDir& d = adjoint ? p->fwd : p->rev;
    const float damping = o.pr_damping > 0.f ? o.pr_damping : 0.85f;
    SolveArgs a{};
    a.g = tab(vd, d);
    a.n = vg->n;
    a.b = bsrc;
    a.scale_b = adjoint ? 1.0f : 1.0f - damping;
    a.d = damping;
    const bool res_form = o.max_iterations == 0;
    if (res_form) {
        const double d64 = o.pr_damping > 0.f ? (double)o.pr_damping : 0.85, s64 = adjoint ? 1.0 : 1.0 - d64;
        a.d_lo = (float)(d64 - (double)a.d);
        a.scale_b = (float)s64;
        a.scale_lo = (float)(s64 - (double)a.scale_b);
    }
    if (!res_form) {
        a.y0 = adjoint ? p->Lb[0] : p->Y[0];
        a.y1 = adjoint ? p->Lb[1] : p->Y[1];
    } else if (!adjoint) {  // residuals in the adjoint's buffers
        a.y0 = p->Lb[0];
        a.y1 = p->Lb[1];
        a.y = p->Y[0];
        a.res = p->Y[1];
    } else {  // the forward's other buffer is free
        a.y0 = p->Y[p->xi ^ 1];
        a.y1 = p->Lb[0];
        a.y = p->Lb[1];
        a.res = p->Lb[0];
    }
    a.ctrl = p->ctrl;
    a.max_iters = o.max_iterations ? o.max_iterations : 10000u;
    a.tol = o.pr_tolerance > 0.f ? (double)o.pr_tolerance : 1e-7;
    if (!adjoint) a.bound = vertex_bound(a.tol, (double)a.d, PPR_FIRST, PPR_LATER);
    a.timeout_ns = wait_limit_ns(o);
    EEG_CUDA(cudaMemsetAsync(p->ctrl, 0, sizeof(PRCtrl), st));
    EEG_TRY(reset_counters(d, st));
#define EEG_PPR_SOLVE(KV) \
    EEG_TRY(res_form ? (launch_solve<KV, true>(p, a, o.blocks_per_sm, st)) : (launch_solve<KV, false>(p, a, o.blocks_per_sm, st)))
    switch (vg->K) {
        case 4: EEG_PPR_SOLVE(4); break;
        case 8: EEG_PPR_SOLVE(8); break;
        case 16: EEG_PPR_SOLVE(16); break;
        default: set_last_error("K must be 4, 8 or 16"); return EEG_ERR_UNSUPPORTED;
    }
#undef EEG_PPR_SOLVE
    PRCtrl hc;
    EEG_CUDA(cudaMemcpyAsync(&hc, p->ctrl, sizeof(PRCtrl), cudaMemcpyDeviceToHost, st));
    EEG_CUDA(cudaStreamSynchronize(st));
    // residual form, cap of 10000 sweeps reached: the iterate as it stands
    if (!res_form) *result = (hc.iterations & 1u) ? a.y1 : a.y0;
    else *result = hc.bw.status == DEV_ITER_CAP ? a.y : a.res;
    const double m = (double)vg->m, n = (double)vg->n;
    res->iterations += hc.iterations;
    res->pr_residual = hc.last_resid;
    res->pr_l1_norm = hc.last_norm;
    res->edges_scanned += (uint64_t)hc.iterations * vg->m;
    res->algorithmic_bytes += (double)hc.iterations * (8.0 * m + (double)p->W * (4.0 * m + 8.0 * n));
    res->launches += 1;
    if (hc.bw.status == DEV_TIMEOUT) {
        set_last_error("grid barrier wait exceeded the timeout");
        return EEG_ERR_TIMEOUT;
    }
    if (hc.bw.status == DEV_ITER_CAP) {
        set_last_error("personalised PageRank did not reach the tolerance within the sweep cap");
        return EEG_ERR_ITER_CAP;
    }
    return EEG_OK;
}

}  // namespace
}  // namespace eeg

using namespace eeg;

extern "C" {

EEG_API eeg_status eeg_ppr_create(eeg_vgraph* vg, uint32_t columns, eeg_ppr** out) {
    if (!vg || !out) {
        set_last_error("null argument");
        return EEG_ERR_INVALID;
    }
    *out = nullptr;
    if (columns == 0 || columns > PPR_W) {
        set_last_error("columns must be in [1, 64]");
        return EEG_ERR_INVALID;
    }
    if (!vg->fwd_parts) {
        set_last_error("personalised PageRank needs the forward parts (not EEG_VG_REVERSE_ONLY)");
        return EEG_ERR_INVALID;
    }
    if (!vg->has_rev || vg->rev_alias || !(vg->flags & EEG_VG_EDGE_IDS) || !vg->fwd.veid || !vg->rev.veid) {
        set_last_error("personalised PageRank needs a graph built with EEG_VG_REVERSE | EEG_VG_EDGE_IDS");
        return EEG_ERR_INVALID;
    }
    if (vg->n == 0) {
        set_last_error("empty graph");
        return EEG_ERR_INVALID;
    }
    EEG_CUDA(cudaSetDevice(vg->device));
    eeg_ppr* p = new eeg_ppr();
    p->vg = vg;
    p->C = columns;
    p->W = columns == 1 ? 1u : (columns <= 32 ? 32u : PPR_W);  // row width: 128-B rows up to 32 columns
    const size_t n = vg->n, rows = n * p->W;
    eeg_status s = EEG_OK;
    auto run = [&]() -> eeg_status {
        EEG_TRY(build_chunks(p, vg->fwd, p->fwd));
        EEG_TRY(build_chunks(p, vg->rev, p->rev));
        EEG_TRY(ppr_alloc(p, (void**)&p->w_raw, sizeof(float) * std::max<uint64_t>(vg->m, 1)));
        EEG_TRY(ppr_alloc(p, (void**)&p->s, sizeof(float) * n));
        EEG_TRY(ppr_alloc(p, (void**)&p->bad, sizeof(uint32_t)));
        for (int i = 0; i < 2; ++i) {
            EEG_TRY(ppr_alloc(p, (void**)&p->Y[i], sizeof(float) * rows));
            EEG_TRY(ppr_alloc(p, (void**)&p->Lb[i], sizeof(float) * rows));
        }
        EEG_TRY(ppr_alloc(p, (void**)&p->b, sizeof(float) * rows));
        EEG_CUDA(cudaMemset(p->b, 0, sizeof(float) * rows));  // padding columns stay zero
        EEG_TRY(ppr_alloc(p, (void**)&p->gslot, sizeof(float) * std::max<size_t>((size_t)vg->fwd.P * vg->K, 4)));
        EEG_TRY(ppr_alloc(p, (void**)&p->r, sizeof(float) * n));
        EEG_CUDA(cudaMalloc((void**)&p->ctrl, sizeof(PRCtrl)));
        EEG_CUDA(cudaEventCreate(&p->ev[0]));
        EEG_CUDA(cudaEventCreate(&p->ev[1]));
        return EEG_OK;
    };
    s = run();
    if (s != EEG_OK) {
        eeg_ppr_destroy(p);
        return s;
    }
    *out = p;
    return EEG_OK;
}

EEG_API eeg_status eeg_ppr_set_weights(eeg_ppr* p, const float* w, int on_device) {
    if (!p || (!w && p->vg->m > 0)) {
        set_last_error("null argument");
        return EEG_ERR_INVALID;
    }
    eeg_vgraph* vg = p->vg;
    EEG_CUDA(cudaSetDevice(vg->device));
    const uint32_t K = vg->K;
    if (vg->m > 0)
        EEG_CUDA(cudaMemcpy(p->w_raw, w, sizeof(float) * vg->m, on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
    EEG_CUDA(cudaMemset(p->bad, 0, sizeof(uint32_t)));
    EEG_CUDA(cudaMemset(p->s, 0, sizeof(float) * vg->n));
    EEG_TRY(reset_counters(p->fwd, 0));
    if (p->fwd.nchunks) {
        const DirTab g = tab(vg->fwd, p->fwd);
        const unsigned blocks = grid_1d((uint64_t)p->fwd.nchunks * 32, vg->device);
        if (K == 4) k_ppr_out_sums<4><<<blocks, PPR_TPB>>>(g, vg->fwd.veid, p->w_raw, p->s, p->bad);
        else if (K == 8) k_ppr_out_sums<8><<<blocks, PPR_TPB>>>(g, vg->fwd.veid, p->w_raw, p->s, p->bad);
        else k_ppr_out_sums<16><<<blocks, PPR_TPB>>>(g, vg->fwd.veid, p->w_raw, p->s, p->bad);
    }
    const uint64_t fs = (uint64_t)vg->fwd.P * K, rs = (uint64_t)vg->rev.P * K;
    if (fs)
        k_ppr_norm<<<grid_1d(fs, vg->device), PPR_TPB>>>(fs, K, 0, vg->fwd.veid, vg->fwd.vowner, vg->fwd.vcol, p->w_raw,
                                                         p->s, p->fwd.w);
    if (rs)
        k_ppr_norm<<<grid_1d(rs, vg->device), PPR_TPB>>>(rs, K, 1, vg->rev.veid, vg->rev.vowner, vg->rev.vcol, p->w_raw,
                                                         p->s, p->rev.w);
    EEG_CUDA(cudaGetLastError());
    uint32_t bad = 0;
    EEG_CUDA(cudaMemcpy(&bad, p->bad, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (bad) {
        p->have_w = false;
        set_last_error("edge weights must be finite and >= 0");
        return EEG_ERR_INVALID;
    }
    p->have_w = true;
    p->xi = -1;
    return EEG_OK;
}

EEG_API eeg_status eeg_ppr_forward(eeg_ppr* p, const float* teleport, int in_on_device, float* x_out,
                                   int out_on_device, const eeg_options* opts, void* stream, eeg_result* res) {
    if (!p || !teleport) {
        set_last_error("null argument");
        return EEG_ERR_INVALID;
    }
    if (!p->have_w) {
        set_last_error("set the edge weights first (eeg_ppr_set_weights)");
        return EEG_ERR_INVALID;
    }
    eeg_options o;
    eeg_options_init(&o);
    if (opts) o = *opts;
    cudaStream_t st = (cudaStream_t)stream;
    EEG_CUDA(cudaSetDevice(p->vg->device));
    eeg_result r;
    memset(&r, 0, sizeof(r));
    p->xi = -1;
    const float* bsrc = nullptr;
    EEG_CUDA(cudaEventRecord(p->ev[0], st));
    EEG_TRY(stage_rows(p, teleport, in_on_device, st, &bsrc));
    float* X = nullptr;
    eeg_status s = solve(p, false, bsrc, o, st, &r, &X);
    if (s != EEG_OK && s != EEG_ERR_ITER_CAP) return s;
    p->xi = X == p->Y[1] ? 1 : 0;
    if (x_out) EEG_TRY(unstage_rows(p, X, x_out, out_on_device, st));
    EEG_CUDA(cudaEventRecord(p->ev[1], st));
    EEG_CUDA(cudaEventSynchronize(p->ev[1]));
    float ms = 0.f;
    EEG_CUDA(cudaEventElapsedTime(&ms, p->ev[0], p->ev[1]));
    r.kernel_ms = ms;
    r.reached_vertices = p->vg->n;
    r.reached_edges = p->vg->m;
    r.gteps = ms > 0 ? (double)r.iterations * (double)p->vg->m / (ms * 1e-3) / 1e9 : 0.0;
    if (res) *res = r;
    return s;
}

EEG_API eeg_status eeg_ppr_adjoint(eeg_ppr* p, const float* dl_dx, int in_on_device, float* dl_dteleport,
                                   float* dl_dw, float* dl_dwn, int out_on_device, int accumulate,
                                   const eeg_options* opts, void* stream, eeg_result* res) {
    if (!p || !dl_dx) {
        set_last_error("null argument");
        return EEG_ERR_INVALID;
    }
    if (p->xi < 0) {
        set_last_error("run eeg_ppr_forward first");
        return EEG_ERR_INVALID;
    }
    eeg_options o;
    eeg_options_init(&o);
    if (opts) o = *opts;
    eeg_vgraph* vg = p->vg;
    cudaStream_t st = (cudaStream_t)stream;
    EEG_CUDA(cudaSetDevice(vg->device));
    const float damping = o.pr_damping > 0.f ? o.pr_damping : 0.85f;
    eeg_result r;
    memset(&r, 0, sizeof(r));
    const float* bsrc = nullptr;
    EEG_CUDA(cudaEventRecord(p->ev[0], st));
    EEG_TRY(stage_rows(p, dl_dx, in_on_device, st, &bsrc));
    float* L = nullptr;
    eeg_status s = solve(p, true, bsrc, o, st, &r, &L);
    if (s != EEG_OK && s != EEG_ERR_ITER_CAP) return s;
    // edge gradients
    GradArgs g{};
    g.g = tab(vg->fwd, p->fwd);
    g.X = p->Y[p->xi];
    g.L = L;
    g.d = damping;
    g.gslot = p->gslot;
    g.r = p->r;
    g.accumulate = (accumulate && p->have_g) ? 1u : 0u;
    EEG_TRY(reset_counters(p->fwd, st));
    switch (vg->K) {
        case 4: EEG_TRY(launch_grad<4>(p, g, st)); break;
        case 8: EEG_TRY(launch_grad<8>(p, g, st)); break;
        case 16: EEG_TRY(launch_grad<16>(p, g, st)); break;
        default: set_last_error("K must be 4, 8 or 16"); return EEG_ERR_UNSUPPORTED;
    }
    p->have_g = true;
    r.launches += 1;
    const uint64_t fs = (uint64_t)vg->fwd.P * vg->K;
    if ((dl_dw || dl_dwn) && fs) {
        float* dwn = dl_dwn;
        float* dw = dl_dw;
        if (!out_on_device) {
            if (!p->stage_m) EEG_TRY(ppr_alloc(p, (void**)&p->stage_m, sizeof(float) * 2 * std::max<uint64_t>(vg->m, 1)));
            dwn = dl_dwn ? p->stage_m : nullptr;
            dw = dl_dw ? p->stage_m + vg->m : nullptr;
        }
        k_ppr_scatter<<<grid_1d(fs, vg->device), PPR_TPB, 0, st>>>(fs, vg->K, vg->fwd.veid, vg->fwd.vowner, p->gslot,
                                                                   p->r, p->s, dwn, dw);
        EEG_CUDA(cudaGetLastError());
        r.launches += 1;
        if (!out_on_device) {
            if (dl_dwn) EEG_CUDA(cudaMemcpyAsync(dl_dwn, dwn, sizeof(float) * vg->m, cudaMemcpyDeviceToHost, st));
            if (dl_dw) EEG_CUDA(cudaMemcpyAsync(dl_dw, dw, sizeof(float) * vg->m, cudaMemcpyDeviceToHost, st));
        }
    }
    if (dl_dteleport) {
        const uint64_t cnt = (uint64_t)vg->n * p->W;
        const bool direct = out_on_device && p->C == p->W;
        if (!direct && !p->stage_nw) EEG_TRY(ppr_alloc(p, (void**)&p->stage_nw, sizeof(float) * cnt));
        float* dst = direct ? dl_dteleport : p->stage_nw;
        const float s32 = o.pr_damping > 0.f ? (float)(1.0 - (double)o.pr_damping) : (float)0.15;
        k_ppr_scale<<<grid_1d(cnt, vg->device), PPR_TPB, 0, st>>>(cnt, s32, L, dst);
        EEG_CUDA(cudaGetLastError());
        r.launches += 1;
        if (!direct) EEG_TRY(unstage_rows(p, dst, dl_dteleport, out_on_device, st));
    }
    EEG_CUDA(cudaEventRecord(p->ev[1], st));
    EEG_CUDA(cudaEventSynchronize(p->ev[1]));
    float ms = 0.f;
    EEG_CUDA(cudaEventElapsedTime(&ms, p->ev[0], p->ev[1]));
    r.kernel_ms = ms;
    r.reached_vertices = vg->n;
    r.reached_edges = vg->m;
    // gradient pass: per edge 8 B (target + weight) + 4 B gradient + one gathered row of the adjoint
    r.algorithmic_bytes += (double)vg->m * (12.0 + 4.0 * p->W) + (double)vg->n * 4.0 * p->W;
    r.gteps = ms > 0 ? (double)r.iterations * (double)vg->m / (ms * 1e-3) / 1e9 : 0.0;
    if (res) *res = r;
    return s;
}

EEG_API void eeg_ppr_destroy(eeg_ppr* p) {
    if (!p) return;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(p->vg->device);
    cudaDeviceSynchronize();  // no kernel may still use the arrays
    free_pdir(p, p->fwd);
    free_pdir(p, p->rev);
    eeg_vgraph* vg = p->vg;
    vg_free(vg, p->w_raw);
    vg_free(vg, p->s);
    vg_free(vg, p->bad);
    for (int i = 0; i < 2; ++i) {
        vg_free(vg, p->Y[i]);
        vg_free(vg, p->Lb[i]);
    }
    vg_free(vg, p->b);
    vg_free(vg, p->gslot);
    vg_free(vg, p->r);
    vg_free(vg, p->stage_m);
    vg_free(vg, p->stage_nw);
    if (p->ctrl) cudaFree(p->ctrl);
    if (p->ev[0]) cudaEventDestroy(p->ev[0]);
    if (p->ev[1]) cudaEventDestroy(p->ev[1]);
    cudaSetDevice(prev);
    delete p;
}

}  // extern "C"
