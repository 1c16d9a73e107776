// builder.cu -- GPU construction of the K-bounded virtual graph.
//
// Replaces VirtualGraph::VirtualGraph + VirtualGraph::MakeGraph (reference src/virtual_graph.cpp:3-112,
// UM twin src/um_virtual_graph.cu:36-111), which build an interleaved host array on one core and
// drop every edge whose slot index reaches num_edges (src/virtual_graph.cpp:86-88). Here:
//
// The low 11 bits of the owner id are a vertex's place in its bucket, the bits above them name the bucket:
//   1. partition    stable, by bucket, in tiles of 8192 edges: (low bits, neighbour[, weight]). One pass up
//                   to 2^22 vertices; above, the bucket bits are sorted in passes of at most 11 bits. The
//                   first pass reads the caller's arrays (shift, both directions, range check).
//   2. counts       per tile of one bucket and vertex; prefix sums over a bucket's tiles give the degrees
//   3. part counts  np[v] = ceil(deg[v] / K); vstart = exclusive scan; vstart[n] = P
//   4. owners       vowner of every part, unused slots of a vertex's last part
//   5. placement    stable, each tile: edge of rank r of vertex v -> slot vstart[v]*K + r (part r/K)
// A sparse graph (see sorted_by_vertex) is partitioned by all bits of the owner id instead: 2. is then the runs of
// equal owners, and 5. an edge's place in its run.
// What bounds it is memory traffic: 8-bit radix passes over all 22 bits, a preparing copy, run detection,
// cleared slots and a separate placement moved 9.7 GB for 67 M weighted edges; this moves 4 GB (2.95 ->
// 1.98 ms from device arrays; now the tile kernels' shared-memory and store throughput, 0.65 ms each).
//
// The result is lossless and deterministic. Part p of vertex v holds out-edges [ (p - vstart[v]) * K,
// +K ) of v in one K-slot row, in input order (the order MakeGraph gives them), so a thread reads a
// whole part with one or two aligned 256-bit loads.
#include <algorithm>
#include <cstdio>

#include "internal.hpp"

namespace eeg {

// ------------------------------------------------------------------ device-wide scan
namespace {

constexpr int SCAN_TPB = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr uint64_t SCAN_TILE = (uint64_t)SCAN_TPB * SCAN_ITEMS;

__device__ __forceinline__ uint32_t scan_op(uint32_t a, uint32_t b, int op) {
    return op == SCAN_ADD ? a + b : (a > b ? a : b);
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, int op) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= (uint32_t)off) x = scan_op(x, y, op);
    }
    return x;
}

// CTA scan of one value per thread (blockDim == SCAN_TPB). Returns the EXCLUSIVE prefix
// (identity 0 for thread 0) and sets *total to the CTA aggregate.
__device__ __forceinline__ uint32_t cta_exclusive(uint32_t x, int op, uint32_t* s_warp, uint32_t* s_inc,
                                                  uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = warp_inclusive(x, op);
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) s_warp[lane] = warp_inclusive(s_warp[lane], op);  // 32 warps
    __syncthreads();
    inc = warp > 0 ? scan_op(s_warp[warp - 1], inc, op) : inc;
    s_inc[threadIdx.x] = inc;
    __syncthreads();
    uint32_t ex = threadIdx.x > 0 ? s_inc[threadIdx.x - 1] : 0u;
    *total = s_warp[31];
    __syncthreads();
    return ex;
}

__global__ void __launch_bounds__(SCAN_TPB) k_scan_reduce(const uint32_t* __restrict__ in, uint64_t n,
                                                          uint32_t* __restrict__ partials, int op) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_inc[SCAN_TPB];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        uint64_t idx = base + (uint64_t)i * SCAN_TPB + threadIdx.x;
        if (idx < n) acc = scan_op(acc, in[idx], op);
    }
    uint32_t total;
    cta_exclusive(acc, op, s_warp, s_inc, &total);
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

// Single CTA: exclusive scan of the tile partials, in place.
__global__ void __launch_bounds__(SCAN_TPB) k_scan_partials(uint32_t* partials, uint64_t nt, int op) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_inc[SCAN_TPB];
    uint32_t carry = 0;
    for (uint64_t base = 0; base < nt; base += SCAN_TPB) {
        uint64_t idx = base + threadIdx.x;
        uint32_t x = idx < nt ? partials[idx] : 0u;
        uint32_t total;
        uint32_t ex = cta_exclusive(x, op, s_warp, s_inc, &total);
        if (idx < nt) partials[idx] = threadIdx.x == 0 ? carry : scan_op(carry, ex, op);
        carry = scan_op(carry, total, op);
    }
}

__global__ void __launch_bounds__(SCAN_TPB) k_scan_apply(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                         uint64_t n, const uint32_t* __restrict__ partials,
                                                         int inclusive, int op) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_inc[SCAN_TPB];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    // each thread owns SCAN_ITEMS consecutive items (blocked arrangement keeps scan order)
    uint32_t v[SCAN_ITEMS];
    const uint64_t t0 = base + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        uint64_t idx = t0 + i;
        v[i] = idx < n ? in[idx] : 0u;
        acc = scan_op(acc, v[i], op);
    }
    uint32_t total;
    uint32_t ex = cta_exclusive(acc, op, s_warp, s_inc, &total);
    const uint32_t tile_prefix = partials[blockIdx.x];
    uint32_t run = threadIdx.x == 0 ? tile_prefix : scan_op(tile_prefix, ex, op);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        uint64_t idx = t0 + i;
        uint32_t before = run;
        run = scan_op(run, v[i], op);
        if (idx < n) out[idx] = inclusive ? run : before;
    }
}

}  // namespace

uint64_t device_scan_tmp_words(uint64_t n) { return (n + SCAN_TILE - 1) / SCAN_TILE + 1; }

eeg_status device_scan_u32(const uint32_t* in, uint32_t* out, uint64_t n, bool inclusive, ScanOp op,
                           uint32_t* tmp, cudaStream_t st) {
    if (n == 0) return EEG_OK;
    const uint64_t nt = (n + SCAN_TILE - 1) / SCAN_TILE;
    k_scan_reduce<<<(unsigned)nt, SCAN_TPB, 0, st>>>(in, n, tmp, (int)op);
    k_scan_partials<<<1, SCAN_TPB, 0, st>>>(tmp, nt, (int)op);
    k_scan_apply<<<(unsigned)nt, SCAN_TPB, 0, st>>>(in, out, n, tmp, inclusive ? 1 : 0, (int)op);
    EEG_CUDA(cudaGetLastError());
    return EEG_OK;
}

// ------------------------------------------------------------------ builder kernels
namespace {

constexpr int B_TPB = 256;
// Tiles of the partition and the placement: warp w of a tile owns keys [w*512, w*512+512) of it and takes
// them 32 at a time, in order, so ranks keep the input order. 2048 bins leave runs of at least 4 keys per
// bin on average (16-byte writes; 4096-key tiles would halve them and double the count tables). Two CTAs
// per SM, so that one ranks while the other loads or writes: the tile's words share the shared memory of
// the per-warp counters (102-110 KB), and the neighbours and payloads are loaded only when their places
// are known (64 registers).
constexpr int S_TPB = 512;
constexpr int S_WARPS = S_TPB / 32;
constexpr int S_ITEMS = 16;
constexpr int S_TILE = S_TPB * S_ITEMS;
constexpr int S_BITS = 11;
constexpr int S_BINS = 1 << S_BITS;
constexpr int S_CHUNK = 64;  // tiles per prefix chunk
static_assert(S_TILE <= 65535, "per-tile ranks and starts are 16-bit");
static_assert(S_BINS == 4 * S_TPB, "a thread owns four bins");

// The caller's edges as arcs: arc e < m_in is input edge e, with sym arc m_in + e its reverse. Owner and
// neighbour 0-based; an endpoint outside [0, n) raises err (the build is then refused).
struct Arcs {
    const uint32_t* __restrict__ a;  // owners
    const uint32_t* __restrict__ b;  // neighbours
    const uint32_t* __restrict__ w;  // weights (null: 1), unused with eid
    uint64_t m_in, m;
    uint32_t n, shift;
    int sym, eid;
    uint32_t* err;
};
// Tiles of the first pass: the input edges in order, then (sym) once more for the reverses, so that a tile has
// one direction. Loads in the tile kernels are unconditional (clamped to the tile's last arc) and checks come
// after all of them: a check behind each load, or an atomic between two, makes a thread wait for one load
// after the other (40 of 48 thousand cycles per tile).
struct ArcTile {
    const uint32_t* __restrict__ owner;
    const uint32_t* __restrict__ nb;
    const uint32_t* __restrict__ w;
    uint32_t first;  // arc index of the tile's first arc (payload with eid)
    uint32_t count;
};
__device__ __forceinline__ ArcTile arc_tile(const Arcs& s, uint32_t tile) {
    const uint32_t nt = (uint32_t)((s.m_in + S_TILE - 1) / S_TILE);
    const bool rev = tile >= nt;
    const uint64_t e0 = (uint64_t)(rev ? tile - nt : tile) * S_TILE;
    ArcTile r;
    r.owner = (rev ? s.b : s.a) + e0;
    r.nb = (rev ? s.a : s.b) + e0;
    r.w = s.w ? s.w + e0 : nullptr;
    r.first = (uint32_t)(e0 + (rev ? s.m_in : 0ull));
    r.count = (uint32_t)min((uint64_t)S_TILE, s.m_in - e0);
    return r;
}
__device__ __forceinline__ uint32_t checked(const Arcs& s, uint32_t id, bool& bad) {
    id -= s.shift;
    bad |= id >= s.n;
    return id >= s.n ? 0u : id;
}

// A count in shared memory; when the whole warp counts the same bin (sorted edge lists), by one lane.
__device__ __forceinline__ void count_bin(uint32_t* h, bool valid, uint32_t bin, uint32_t lane) {
    const uint32_t v = valid ? bin : 0xFFFFFFFFu;
    if (__all_sync(0xffffffffu, v == __shfl_sync(0xffffffffu, v, 0))) {
        if (valid && lane == 0) atomicAdd(&h[bin], 32u);
    } else if (valid) {
        atomicAdd(&h[bin], 1u);
    }
}

// Partition, counts of one tile per bin (key >> lo) & (bins - 1): hist[tile][bin]. The first pass (RAW) takes
// the owners from the arcs and leaves a copy where the placement of the pass would read them from host
// memory again (copy non-null).
template <bool RAW>
__global__ void __launch_bounds__(S_TPB) k_bin_counts(Arcs s, const uint32_t* __restrict__ key, uint32_t* __restrict__ copy,
                                                      uint64_t m, uint32_t lo, uint32_t bins, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[S_BINS];
    for (uint32_t i = threadIdx.x; i < bins; i += S_TPB) h[i] = 0u;
    __syncthreads();
    const uint32_t* at = key + (RAW ? 0ull : (uint64_t)blockIdx.x * S_TILE);
    uint32_t count = 0;
    if (RAW) {
        const ArcTile a = arc_tile(s, blockIdx.x);
        at = a.owner;
        count = a.count;
    } else {
        count = (uint32_t)min((uint64_t)S_TILE, m - (uint64_t)blockIdx.x * S_TILE);
    }
    uint32_t k[S_ITEMS];
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) k[j] = __ldg(at + min(j * (uint32_t)S_TPB + threadIdx.x, count - 1u));
    if (RAW) {
        bool bad = false;
#pragma unroll
        for (int j = 0; j < S_ITEMS; ++j) k[j] = checked(s, k[j], bad);
        if (bad) atomicOr(s.err, 1u);
    }
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) {
        const uint32_t i = j * (uint32_t)S_TPB + threadIdx.x;
        if (RAW && copy && i < count) copy[(uint64_t)blockIdx.x * S_TILE + i] = k[j];
        count_bin(h, i < count, (k[j] >> lo) & (bins - 1u), threadIdx.x & 31u);
    }
    __syncthreads();
    uint32_t* out = hist + (size_t)blockIdx.x * bins;
    for (uint32_t i = threadIdx.x; i < bins; i += S_TPB) out[i] = h[i];
}

// hist[tile][bin] -> prefix within its chunk of S_CHUNK tiles; csum[chunk][bin] = the chunk's total
__global__ void __launch_bounds__(256) k_tile_prefix(uint32_t* hist, uint32_t ntiles, uint32_t bins, uint32_t* csum) {
    const uint32_t d = blockIdx.y * 256u + threadIdx.x;
    if (d >= bins) return;
    const uint32_t t0 = blockIdx.x * S_CHUNK, t1 = min(t0 + (uint32_t)S_CHUNK, ntiles);
    uint32_t run = 0;
    for (uint32_t t = t0; t < t1; t += 8u) {
        uint32_t x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = t + j < t1 ? hist[(size_t)(t + j) * bins + d] : 0u;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (t + j < t1) hist[(size_t)(t + j) * bins + d] = run;
            run += x[j];
        }
    }
    csum[(size_t)blockIdx.x * bins + d] = run;
}
// csum[chunk][bin] -> prefix over the chunks; tot[bin]
__global__ void __launch_bounds__(256) k_chunk_prefix(uint32_t* csum, uint32_t nchunks, uint32_t bins, uint32_t* tot) {
    const uint32_t d = blockIdx.x * 256u + threadIdx.x;
    if (d >= bins) return;
    uint32_t run = 0;
    for (uint32_t c = 0; c < nchunks; c += 8u) {
        uint32_t x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = c + j < nchunks ? csum[(size_t)(c + j) * bins + d] : 0u;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (c + j < nchunks) csum[(size_t)(c + j) * bins + d] = run;
            run += x[j];
        }
    }
    tot[d] = run;
}

// One CTA: exclusive scan of f(i), i < count, written to out[i]; out[count] = the total.
template <class F>
__device__ void scan_to(F f, uint32_t count, uint32_t* out) {
    __shared__ uint32_t s_warp[32], s_inc[SCAN_TPB];
    uint32_t carry = 0;
    for (uint32_t base = 0; base < count; base += SCAN_TPB) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t x = i < count ? f(i) : 0u;
        uint32_t total;
        const uint32_t ex = cta_exclusive(x, SCAN_ADD, s_warp, s_inc, &total);
        if (i < count) out[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) out[count] = carry;
}
__global__ void __launch_bounds__(SCAN_TPB) k_bin_starts(const uint32_t* tot, uint32_t bins, uint32_t* start) {
    scan_to([&](uint32_t i) { return tot[i]; }, bins, start);
}
// Tiles of the buckets: tstart = first tile of each (a bucket without edges has none), tbucket = each tile's bucket
__global__ void __launch_bounds__(SCAN_TPB) k_bucket_tiles(const uint32_t* __restrict__ bstart, uint32_t nb,
                                                           uint32_t* tstart, uint32_t* tbucket) {
    scan_to([&](uint32_t i) { return (bstart[i + 1] - bstart[i] + (uint32_t)S_TILE - 1u) / (uint32_t)S_TILE; }, nb, tstart);
    __syncthreads();
    // a bucket of many tiles (2048 of them: 70 us by one thread) is written by the whole CTA
    __shared__ uint32_t s_many[SCAN_TPB], s_count;
    for (uint32_t base = 0; base < nb; base += SCAN_TPB) {
        if (threadIdx.x == 0) s_count = 0u;
        __syncthreads();
        const uint32_t i = base + threadIdx.x;
        const uint32_t t0 = i < nb ? tstart[i] : 0u, t1 = i < nb ? tstart[i + 1] : 0u;
        if (t1 - t0 > 16u) s_many[atomicAdd(&s_count, 1u)] = i;
        else
            for (uint32_t t = t0; t < t1; ++t) tbucket[t] = i;
        __syncthreads();
        for (uint32_t k = 0; k < s_count; ++k)
            for (uint32_t t = tstart[s_many[k]] + threadIdx.x; t < tstart[s_many[k] + 1]; t += SCAN_TPB) tbucket[t] = s_many[k];
        __syncthreads();
    }
}
// Bucket starts from keys sorted by bucket (more than one partition pass): entry i closes every bucket up to its own
__global__ void k_bucket_starts(const uint32_t* __restrict__ key, uint64_t m, uint32_t nb, uint32_t* __restrict__ bstart) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t from = i == 0 ? 0u : (key[i - 1] >> S_BITS) + 1u, to = i == m ? nb : key[i] >> S_BITS;
        for (uint32_t b = from; b <= to; ++b) bstart[b] = (uint32_t)i;
    }
}

// Stable places of a tile's keys in bin order. bin_of(j) is the bin of this lane's key of its warp's round j
// (>= bins: none); cnt [S_WARPS][bins] is scratch, free again on return. place_of(place, j) = the key's index
// among the tile's keys ordered by bin (two to a register), dstart[bin] = the bin's first index. Called by all threads.
__device__ __forceinline__ uint32_t place_of(const uint32_t (&place)[S_ITEMS / 2], int j) {
    return (place[j >> 1] >> ((j & 1) * 16)) & 0xFFFFu;
}
template <class Bin>
__device__ __forceinline__ void tile_places(Bin bin_of, uint32_t bins, uint16_t* cnt, uint16_t* dstart,
                                            uint32_t* s_warp, uint32_t (&place)[S_ITEMS / 2]) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint4* z = reinterpret_cast<uint4*>(cnt);
    for (uint32_t i = threadIdx.x; i < S_WARPS * bins / 8u; i += S_TPB) z[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    uint16_t* mine = cnt + (size_t)warp * bins;
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) {
        const uint32_t d = bin_of(j);
        // lanes of the same bin, bit by bit (__match_any_sync, which takes time with every distinct value
        // among the lanes, is no faster here)
        uint32_t peers = __ballot_sync(0xffffffffu, d < bins);
#pragma unroll 1
        for (int bit = 0; bit < S_BITS; ++bit) {
            const uint32_t set = __ballot_sync(0xffffffffu, (d >> bit) & 1u);
            peers &= (d >> bit) & 1u ? set : ~set;
        }
        const uint32_t rk = __popc(peers & ((1u << lane) - 1u));
        const uint32_t before = d < bins ? mine[d] : 0u;
        __syncwarp();
        if (d < bins && rk == 0) mine[d] = (uint16_t)(before + __popc(peers));
        __syncwarp();
        if (j & 1) place[j >> 1] |= (before + rk) << 16;
        else place[j >> 1] = before + rk;
    }
    __syncthreads();
    // four bins per thread: offsets of each warp's keys inside the bin, and the bin's length
    uint32_t len[4] = {0u, 0u, 0u, 0u};
    const uint32_t d0 = 4u * threadIdx.x;
    if (d0 < bins) {
#pragma unroll
        for (int w = 0; w < S_WARPS; ++w) {
            uint2* at = reinterpret_cast<uint2*>(cnt + (size_t)w * bins + d0);
            const uint2 c = *at;
            *at = make_uint2(len[0] | len[1] << 16, len[2] | len[3] << 16);
            len[0] += c.x & 0xFFFFu;
            len[1] += c.x >> 16;
            len[2] += c.y & 0xFFFFu;
            len[3] += c.y >> 16;
        }
    }
    uint32_t total;
    uint32_t run = block_exclusive_sum(len[0] + len[1] + len[2] + len[3], s_warp, &total);
    if (d0 < bins) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            dstart[d0 + q] = (uint16_t)run;
            run += len[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) {
        const uint32_t d = bin_of(j);
        if (d < bins) place[j >> 1] += ((uint32_t)dstart[d] + mine[d]) << ((j & 1) * 16);
    }
    __syncthreads();
}

// Shared memory of the two tile kernels (bytes): the tile's words in the place of the counters (16-byte
// aligned for any number of bins: both sizes are multiples of 16 from four bins on), then per bin the output
// offset and the first index.
__host__ __device__ constexpr size_t max_size(size_t a, size_t b) { return a > b ? a : b; }
__host__ __device__ constexpr size_t partition_tile(uint32_t bins, bool payload) {
    return max_size((size_t)S_WARPS * bins * 2, (size_t)S_TILE * (payload ? 12 : 8));
}
__host__ __device__ constexpr size_t place_tile(bool payload) {
    return max_size((size_t)S_WARPS * S_BINS * 2, (size_t)S_TILE * (payload ? 10 : 6));
}
constexpr size_t partition_smem(uint32_t bins, bool payload) { return partition_tile(bins, payload) + (size_t)bins * (4 + 2); }
constexpr size_t place_smem(bool payload) { return place_tile(payload) + (size_t)S_BINS * (8 + 2); }
static_assert(S_WARPS * 4 * 2 % 16 == 0 && S_TILE * 6 % 16 == 0, "16-byte aligned counters");
// What the kernels are allowed to be launched with belongs to the process: the largest that any build asks for,
// always, so that builds in several threads do not take it from each other.
constexpr size_t PARTITION_SMEM = partition_smem(S_BINS, true), PLACE_SMEM = place_smem(true);

// Partition, scatter of one tile: a key's place = its bin's start + the bin's keys in earlier tiles + its rank
// in the tile. The tile goes through shared memory in bin order, so a bin's run is written by consecutive
// threads. KOut = uint16_t: only the low S_BITS of the key are kept (the bucket is known from the place).
template <bool RAW, typename KOut>
__global__ void __launch_bounds__(S_TPB, 2) k_partition(Arcs s, const uint32_t* __restrict__ key,
                                                        const uint32_t* __restrict__ nb, const uint32_t* __restrict__ pay,
                                                        uint64_t m, uint32_t lo, uint32_t bins,
                                                        const uint32_t* __restrict__ hist, const uint32_t* __restrict__ csum,
                                                        const uint32_t* __restrict__ start, KOut* __restrict__ key_out,
                                                        uint32_t* __restrict__ nb_out, uint32_t* __restrict__ pay_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_warp[33];
    uint16_t* s_cnt = reinterpret_cast<uint16_t*>(smem);
    uint32_t* s_key = reinterpret_cast<uint32_t*>(smem);  // over the counters, once the places are known
    uint32_t* s_nb = s_key + S_TILE;
    uint32_t* s_pay = s_nb + S_TILE;
    uint32_t* s_goff = reinterpret_cast<uint32_t*>(smem + partition_tile(bins, pay_out != nullptr));
    uint16_t* s_dstart = reinterpret_cast<uint16_t*>(s_goff + bins);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t first = warp * (32u * S_ITEMS) + lane;  // this lane's keys: first, first + 32, ...
    ArcTile a{};
    const uint64_t e0 = (uint64_t)blockIdx.x * S_TILE;
    if (RAW) a = arc_tile(s, blockIdx.x);
    else a.count = (uint32_t)min((uint64_t)S_TILE, m - e0);
    const uint32_t total = a.count;
    const uint32_t* kp = key ? key + e0 : a.owner;
    const uint32_t* np = RAW ? a.nb : nb + e0;
    uint32_t k[S_ITEMS], x[S_ITEMS];
    uint32_t place[S_ITEMS / 2];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) k[j] = __ldg(kp + min(first + j * 32u, total - 1u));  // coalesced
    for (uint32_t d = threadIdx.x; d < bins; d += S_TPB)
        s_goff[d] = start[d] + csum[(size_t)(blockIdx.x / S_CHUNK) * bins + d] + hist[(size_t)blockIdx.x * bins + d];
    if (RAW && !key) {
#pragma unroll
        for (int j = 0; j < S_ITEMS; ++j) k[j] = checked(s, k[j], bad);
    }
    tile_places([&](int j) { return first + j * 32u < total ? (k[j] >> lo) & (bins - 1u) : 0xFFFFFFFFu; }, bins, s_cnt,
                s_dstart, s_warp, place);
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j)
        if (first + j * 32u < total) s_key[place_of(place, j)] = k[j];
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) x[j] = __ldg(np + min(first + j * 32u, total - 1u));
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) {
        if (RAW) x[j] = checked(s, x[j], bad);
        if (first + j * 32u < total) s_nb[place_of(place, j)] = x[j];
    }
    if (RAW && bad) atomicOr(s.err, 1u);
    if (pay_out) {
        const uint32_t* pp = RAW ? (s.eid ? nullptr : a.w) : pay + e0;
        if (pp) {
#pragma unroll
            for (int j = 0; j < S_ITEMS; ++j) x[j] = __ldg(pp + min(first + j * 32u, total - 1u));
        } else {  // arc indices, or weights all 1
#pragma unroll
            for (int j = 0; j < S_ITEMS; ++j) x[j] = s.eid ? a.first + first + j * 32u : 1u;
        }
#pragma unroll
        for (int j = 0; j < S_ITEMS; ++j)
            if (first + j * 32u < total) s_pay[place_of(place, j)] = x[j];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < total; i += S_TPB) {
        const uint32_t kk = s_key[i];
        const uint32_t d = (kk >> lo) & (bins - 1u);
        const uint32_t gp = s_goff[d] + (i - s_dstart[d]);
        key_out[gp] = (KOut)(sizeof(KOut) == 2 ? kk & (uint32_t)(S_BINS - 1) : kk);
        nb_out[gp] = s_nb[i];
        if (pay_out) pay_out[gp] = s_pay[i];
    }
}

// Placement, counts of one tile of a bucket per vertex of the bucket: cnt[tile][vertex]
template <typename KeyT>
__global__ void __launch_bounds__(S_TPB) k_vertex_counts(const KeyT* __restrict__ key, const uint32_t* __restrict__ bstart,
                                                         const uint32_t* __restrict__ tstart,
                                                         const uint32_t* __restrict__ tbucket, uint32_t nb,
                                                         uint32_t* __restrict__ cnt) {
    __shared__ uint32_t h[S_BINS];
    if (blockIdx.x >= tstart[nb]) return;
    const uint32_t b = tbucket[blockIdx.x];
    const uint32_t e0 = bstart[b] + (blockIdx.x - tstart[b]) * (uint32_t)S_TILE;
    const uint32_t e1 = e0 + min(bstart[b + 1] - e0, (uint32_t)S_TILE);
    for (uint32_t i = threadIdx.x; i < (uint32_t)S_BINS; i += S_TPB) h[i] = 0u;
    __syncthreads();
    uint32_t k[S_ITEMS];
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) {
        const uint64_t e = min((uint64_t)e0 + j * S_TPB + threadIdx.x, (uint64_t)e1 - 1u);
        k[j] = (uint32_t)key[e] & (uint32_t)(S_BINS - 1);
    }
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j)
        count_bin(h, (uint64_t)e0 + j * S_TPB + threadIdx.x < e1, k[j], threadIdx.x & 31u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < (uint32_t)S_BINS; i += S_TPB) cnt[(size_t)blockIdx.x * S_BINS + i] = h[i];
}

// cnt[tile][vertex] -> prefix over the bucket's tiles; deg[v], np[v] = ceil(deg/K) (np[n] = 0) and the
// max-degree vertex (lowest id among ties). A CTA takes 256 vertices of one bucket: a thread per vertex where
// the bucket has few tiles (the CTAs of grid row 0); where it has many (a hub's bucket has hundreds), each
// grid row takes 32 of the vertices, with eight spans of the tiles. R-MAT s22: one chain of loads per vertex
// everywhere 0.17 ms, spans everywhere 0.16.
constexpr uint32_t FEW_TILES = 32;
__global__ void __launch_bounds__(256) k_degrees(uint32_t* cnt, const uint32_t* __restrict__ tstart, uint32_t n, uint32_t K,
                                                 uint32_t* __restrict__ deg, uint32_t* __restrict__ np,
                                                 unsigned long long* __restrict__ best) {
    __shared__ uint32_t s_sum[8][32];
    const uint32_t lane = threadIdx.x & 31u, span = threadIdx.x >> 5;
    unsigned long long mine = 0;
    auto settle = [&](uint32_t v, uint32_t total) {
        if (v >= n) return;
        deg[v] = total;
        np[v] = (total + K - 1) / K;
        const unsigned long long key = ((unsigned long long)total << 32) | (unsigned long long)(0xFFFFFFFFu - v);
        mine = key > mine ? key : mine;
    };
    // prefix of the tiles [a, b) of one vertex from `run` on, eight loads at a time
    auto prefix = [&](uint32_t* at, uint32_t a, uint32_t b, uint32_t run) {
        for (uint32_t t = a; t < b; t += 8u) {
            uint32_t x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = t + j < b ? at[(size_t)(t + j) * S_BINS] : 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (t + j < b) at[(size_t)(t + j) * S_BINS] = run;
                run += x[j];
            }
        }
        return run;
    };
    for (uint64_t v0 = (uint64_t)blockIdx.x * 256u; v0 < n; v0 += (uint64_t)gridDim.x * 256u) {  // 256 divides a bucket
        const uint32_t t0 = tstart[v0 >> S_BITS], tiles = tstart[(v0 >> S_BITS) + 1] - t0;
        if (tiles <= FEW_TILES) {
            if (blockIdx.y) continue;
            const uint32_t v = (uint32_t)v0 + threadIdx.x;
            settle(v, prefix(cnt + (v & (S_BINS - 1)), t0, t0 + tiles, 0u));
            continue;
        }
        const uint32_t a = t0 + (uint32_t)((uint64_t)tiles * span / 8u), b = t0 + (uint32_t)((uint64_t)tiles * (span + 1u) / 8u);
        const uint32_t v = (uint32_t)v0 + blockIdx.y * 32u + lane;
        uint32_t* at = cnt + (v & (S_BINS - 1));
        uint32_t sum = 0;
#pragma unroll 8
        for (uint32_t t = a; t < b; ++t) sum += at[(size_t)t * S_BINS];
        s_sum[span][lane] = sum;
        __syncthreads();
        uint32_t run = 0, total = 0;
#pragma unroll
        for (uint32_t q = 0; q < 8u; ++q) {
            run += q < span ? s_sum[q][lane] : 0u;
            total += s_sum[q][lane];
        }
        prefix(at, a, b, run);
        if (span == 0u) settle(v, total);
        __syncthreads();
    }
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) np[n] = 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, mine, off);
        mine = o > mine ? o : mine;
    }
    if (lane == 0u && mine) atomicMax(best, mine);
}

// Edges sorted by vertex: first[v] = v's first edge, end[v] = one past its last; vertices without edges keep the zero
// that end was cleared to.
__global__ void k_runs(const uint32_t* __restrict__ key, uint64_t m, uint32_t* __restrict__ first, uint32_t* __restrict__ end) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = key[i];
        if (i == 0 || key[i - 1] != v) first[v] = (uint32_t)i;
        if (i + 1 == m || key[i + 1] != v) end[v] = (uint32_t)i + 1u;
    }
}
// end[v] -> deg[v] (in place), np[v] = ceil(deg/K) (np[n] = 0) and the max-degree vertex (lowest id among ties). Four
// vertices per thread; where they have no edges, nothing but np is written.
__global__ void __launch_bounds__(256) k_run_degrees(const uint32_t* __restrict__ first, uint32_t n, uint32_t K,
                                                     uint32_t* __restrict__ deg, uint32_t* __restrict__ np,
                                                     unsigned long long* __restrict__ best) {
    unsigned long long mine = 0;
    auto one = [&](uint32_t v, uint32_t e) {
        if (!e) return 0u;
        const uint32_t d = e - first[v];
        deg[v] = d;
        const unsigned long long key = ((unsigned long long)d << 32) | (unsigned long long)(0xFFFFFFFFu - v);
        mine = key > mine ? key : mine;
        return (d + K - 1) / K;
    };
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = t0; i < n / 4u; i += step) {  // both arrays are 256-byte aligned
        const uint4 e = reinterpret_cast<const uint4*>(deg)[i];
        const uint32_t v = (uint32_t)i * 4u;
        uint4 p = make_uint4(0u, 0u, 0u, 0u);
        if (e.x | e.y | e.z | e.w) p = make_uint4(one(v, e.x), one(v + 1u, e.y), one(v + 2u, e.z), one(v + 3u, e.w));
        reinterpret_cast<uint4*>(np)[i] = p;
    }
    for (uint64_t v = n / 4u * 4u + t0; v < n; v += step) np[v] = one((uint32_t)v, deg[v]);
    if (t0 == 0) np[n] = 0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, mine, off);
        mine = o > mine ? o : mine;
    }
    if ((threadIdx.x & 31u) == 0u && mine) atomicMax(best, mine);
}
// Placement from edges sorted by vertex (payloads as in k_place).
__global__ void k_place_runs(const uint32_t* __restrict__ key, const uint32_t* __restrict__ nb, const uint32_t* __restrict__ pay,
                             uint64_t m, uint32_t K, const uint32_t* __restrict__ first, const uint32_t* __restrict__ vstart,
                             uint32_t* __restrict__ vcol, uint32_t* __restrict__ vw, const uint32_t* __restrict__ w_in,
                             uint32_t* __restrict__ veid, uint64_t m_in) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = key[i];
        const size_t slot = (size_t)vstart[v] * K + (uint32_t)((uint32_t)i - first[v]);
        vcol[slot] = nb[i];
        if (veid) {
            const uint32_t e = pay[i];
            veid[slot] = e;
            if (vw) vw[slot] = w_in ? w_in[(m_in && e >= m_in) ? e - m_in : e] : 1u;
        } else if (vw) {
            vw[slot] = pay[i];
        }
    }
}

// Owner of every part, and the unused slots of each vertex's last part (targets and edge indices NO_EDGE,
// weights 0). The owners of a vertex of more than 32 parts are written by its whole warp, those of one of more than
// HUB_PARTS (on hubs: their number, then their ids) by k_hub_owners' whole grid: a vertex of 2 M parts took its warp
// 340 us. The unused slots end a row aligned
// to its size, so they are written in at most one store each of 4, 8 and 16 bytes (and one more 16 for K =
// 16): a store of 32 lanes here touches 32 sectors whatever its width, 0.16 ms on R-MAT s22 word by word.
__device__ __forceinline__ void pad_row(uint32_t* p, size_t i, size_t end, uint32_t x) {
    if ((i & 1u) && i < end) p[i++] = x;
    if ((i & 2u) && i < end) {
        *reinterpret_cast<uint2*>(p + i) = make_uint2(x, x);
        i += 2;
    }
    for (; i < end; i += 4) *reinterpret_cast<uint4*>(p + i) = make_uint4(x, x, x, x);
}
constexpr uint32_t HUB_PARTS = 4096;
__global__ void k_owners(uint32_t n, uint32_t K, const uint32_t* __restrict__ vstart, const uint32_t* __restrict__ deg,
                         uint32_t* __restrict__ vowner, uint32_t* __restrict__ vcol, uint32_t* __restrict__ vw,
                         uint32_t* __restrict__ veid, uint32_t* __restrict__ hubs) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t v0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; v0 < n;
         v0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = v0 + lane;
        uint32_t s0 = 0, np = 0;
        if (v < n) {
            s0 = vstart[v];
            np = vstart[v + 1] - s0;
            if (np) {
                const size_t end = (size_t)(s0 + np) * K;
                const size_t used = (size_t)s0 * K + deg[v];
                pad_row(vcol, used, end, NO_EDGE);
                if (vw) pad_row(vw, used, end, 0u);
                if (veid) pad_row(veid, used, end, NO_EDGE);
                if (np <= 32u)
                    for (uint32_t j = 0; j < np; ++j) vowner[s0 + j] = (uint32_t)v;
                else if (np > HUB_PARTS) hubs[1u + atomicAdd(&hubs[0], 1u)] = (uint32_t)v;
            }
        }
        uint32_t big = __ballot_sync(0xffffffffu, np > 32u && np <= HUB_PARTS);
        while (big) {
            const int l = __ffs(big) - 1;
            big &= big - 1u;
            const uint32_t bs = __shfl_sync(0xffffffffu, s0, l), bn = __shfl_sync(0xffffffffu, np, l);
            for (uint32_t j = lane; j < bn; j += 32u) vowner[bs + j] = (uint32_t)v0 + (uint32_t)l;
        }
    }
}

__global__ void k_hub_owners(const uint32_t* __restrict__ hubs, const uint32_t* __restrict__ vstart, uint32_t* __restrict__ vowner) {
    for (uint32_t h = 0; h < hubs[0]; ++h) {
        const uint32_t v = hubs[1u + h], end = vstart[v + 1];
        for (uint64_t p = (uint64_t)vstart[v] + blockIdx.x * blockDim.x + threadIdx.x; p < end; p += gridDim.x * blockDim.x)
            vowner[p] = v;
    }
}

// Placement of one tile of a bucket: edge of rank r of vertex v -> slot vstart[v]*K + r, through shared memory
// in vertex order (the partition's scheme). With veid the payload is the arc index: the weight is gathered
// from the input array by it (arc e >= m_in of a symmetrised build is the reverse of input edge e - m_in;
// m_in is 0 otherwise) and the index is kept per slot.
template <typename KeyT>
__global__ void __launch_bounds__(S_TPB, 2) k_place(const KeyT* __restrict__ key, const uint32_t* __restrict__ nb,
                                                    const uint32_t* __restrict__ pay, const uint32_t* __restrict__ bstart,
                                                    const uint32_t* __restrict__ tstart,
                                                    const uint32_t* __restrict__ tbucket, uint32_t nbuckets, uint32_t n,
                                                    uint32_t K, const uint32_t* __restrict__ cnt,
                                                    const uint32_t* __restrict__ vstart, uint32_t* __restrict__ vcol,
                                                    uint32_t* __restrict__ vw, const uint32_t* __restrict__ w_in,
                                                    uint32_t* __restrict__ veid, uint64_t m_in) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_warp[33];
    uint16_t* s_cnt = reinterpret_cast<uint16_t*>(smem);
    uint32_t* s_nb = reinterpret_cast<uint32_t*>(smem);  // over the counters, once the places are known
    uint16_t* s_key = reinterpret_cast<uint16_t*>(s_nb + S_TILE);
    uint32_t* s_pay = reinterpret_cast<uint32_t*>(s_key + S_TILE);
    unsigned long long* s_goff = reinterpret_cast<unsigned long long*>(smem + place_tile(pay != nullptr));
    uint16_t* s_dstart = reinterpret_cast<uint16_t*>(s_goff + S_BINS);
    if (blockIdx.x >= tstart[nbuckets]) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t b = tbucket[blockIdx.x];
    const uint32_t e0 = bstart[b] + (blockIdx.x - tstart[b]) * (uint32_t)S_TILE;
    const uint32_t total = min(bstart[b + 1] - e0, (uint32_t)S_TILE);  // at least 1
    const uint32_t wbase = warp * (32u * S_ITEMS) + lane;
    const KeyT* kp = key + e0;
    const uint32_t* np = nb + e0;
    KeyT bin[S_ITEMS];
    uint32_t x[S_ITEMS];
    uint32_t place[S_ITEMS / 2];
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) bin[j] = kp[min(wbase + j * 32u, total - 1u)];
    for (uint32_t d = threadIdx.x; d < (uint32_t)S_BINS; d += S_TPB) {
        const uint32_t vx = (b << S_BITS) + d;
        s_goff[d] = vx < n ? (unsigned long long)vstart[vx] * K + cnt[(size_t)blockIdx.x * S_BINS + d] : 0ull;
    }
    tile_places([&](int j) { return wbase + j * 32u < total ? (uint32_t)bin[j] & (uint32_t)(S_BINS - 1) : 0xFFFFFFFFu; },
                S_BINS, s_cnt, s_dstart, s_warp, place);
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j) x[j] = __ldg(np + min(wbase + j * 32u, total - 1u));
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j)
        if (wbase + j * 32u < total) s_key[place_of(place, j)] = (uint16_t)((uint32_t)bin[j] & (uint32_t)(S_BINS - 1));
#pragma unroll
    for (int j = 0; j < S_ITEMS; ++j)
        if (wbase + j * 32u < total) s_nb[place_of(place, j)] = x[j];
    if (pay) {
        const uint32_t* pp = pay + e0;
#pragma unroll
        for (int j = 0; j < S_ITEMS; ++j) x[j] = __ldg(pp + min(wbase + j * 32u, total - 1u));
#pragma unroll
        for (int j = 0; j < S_ITEMS; ++j)
            if (wbase + j * 32u < total) s_pay[place_of(place, j)] = x[j];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < total; i += S_TPB) {
        const uint32_t d = s_key[i];
        const size_t slot = (size_t)(s_goff[d] + (i - s_dstart[d]));
        vcol[slot] = s_nb[i];
        if (veid) {
            const uint32_t e = s_pay[i];
            veid[slot] = e;
            if (vw) vw[slot] = w_in ? w_in[(m_in && e >= m_in) ? e - m_in : e] : 1u;
        } else if (vw) {
            vw[slot] = s_pay[i];  // a weighted direction always carries a payload
        }
    }
}

// Out-degree histogram of the input edges (with sym, of both directions); endpoints outside [0, n)
// are counted nowhere (the transposed build reports them). The lowest OUTDEG_HOT ids count in shared
// memory first, each CTA adding its non-zero counters at the end: generators that do not permute ids
// (R-MAT) put their hubs there, and per-edge global atomics on a hub's counter queue at one L2 slice.
constexpr uint32_t OUTDEG_HOT = 8192;
__global__ void __launch_bounds__(256) k_outdeg(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                                                uint64_t m, uint32_t n, uint32_t shift, int sym,
                                                uint32_t* __restrict__ deg) {
    __shared__ uint32_t s_cnt[OUTDEG_HOT];
    for (uint32_t i = threadIdx.x; i < OUTDEG_HOT; i += blockDim.x) s_cnt[i] = 0u;
    __syncthreads();
    auto count = [&](uint32_t v) {
        if (v < OUTDEG_HOT) atomicAdd(&s_cnt[v], 1u);
        else atomicAdd(&deg[v], 1u);
    };
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = a[e] - shift, t = b[e] - shift;
        if (s < n && t < n) {
            count(s);
            if (sym) count(t);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < OUTDEG_HOT && i < n; i += blockDim.x)
        if (s_cnt[i]) atomicAdd(&deg[i], s_cnt[i]);
}
// Largest degree and its smallest vertex, packed (degree << 32 | ~vertex) into one 64-bit max.
__global__ void k_deg_best(const uint32_t* __restrict__ deg, uint32_t n, unsigned long long* best) {
    unsigned long long b = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if (deg[v]) b = max(b, ((unsigned long long)deg[v] << 32) | (0xFFFFFFFFu - v));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_down_sync(0xffffffffu, b, o));
    if ((threadIdx.x & 31u) == 0 && b) atomicMax(best, b);
}

}  // namespace

int sm_count(int device) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || v <= 0) v = 132;
    return v;
}

static unsigned grid_for(uint64_t work, int device) {
    uint64_t blocks = (work + B_TPB - 1) / B_TPB;
    uint64_t cap = (uint64_t)sm_count(device) * 16;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    return (unsigned)blocks;
}

namespace {
// stream-ordered temporaries released on every exit path
struct TempSet {
    cudaStream_t st;
    void* p[32] = {nullptr};
    int k = 0;
    explicit TempSet(cudaStream_t s) : st(s) {}
    eeg_status get(void** out, size_t bytes) {
        if (k == 32) {
            set_last_error("builder: too many temporaries");
            return EEG_ERR_INVALID;
        }
        cudaError_t e = cudaMallocAsync(out, bytes ? bytes : 4, st);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync(builder temporaries)", __FILE__, __LINE__);
        p[k++] = *out;
        return EEG_OK;
    }
    ~TempSet() {
        for (int i = 0; i < k; ++i) cudaFreeAsync(p[i], st);
    }
};
}  // namespace

eeg_status build_out_degrees(eeg_vgraph* vg, VDir* d, const uint32_t* d_src, const uint32_t* d_dst, cudaStream_t st) {
    const uint32_t n = vg->n;
    const bool sym = (vg->flags & EEG_VG_SYMMETRIZE) != 0;
    const uint64_t m_in = sym ? vg->m / 2 : vg->m;
    const uint32_t shift = (vg->flags & EEG_VG_SHIFT_ONE) ? 1u : 0u;
    EEG_TRY(vg_alloc(vg, (void**)&d->deg, sizeof(uint32_t) * (size_t)(n + 1)));
    TempSet T(st);
    unsigned long long* best = nullptr;
    EEG_TRY(T.get((void**)&best, sizeof(unsigned long long)));
    EEG_CUDA(cudaMemsetAsync(d->deg, 0, sizeof(uint32_t) * (size_t)(n + 1), st));
    EEG_CUDA(cudaMemsetAsync(best, 0, sizeof(unsigned long long), st));
    // two CTAs per SM: each flushes its shared counters once
    if (m_in)
        k_outdeg<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>((m_in + 255) / 256, (uint64_t)sm_count(vg->device) * 2)),
                   256, 0, st>>>(d_src, d_dst, m_in, n, shift, sym ? 1 : 0, d->deg);
    k_deg_best<<<grid_for(n, vg->device), B_TPB, 0, st>>>(d->deg, n, best);
    EEG_CUDA(cudaGetLastError());
    unsigned long long hb = 0;
    EEG_CUDA(cudaMemcpyAsync(&hb, best, sizeof(hb), cudaMemcpyDeviceToHost, st));
    EEG_CUDA(cudaStreamSynchronize(st));
    vg->max_deg = (uint32_t)(hb >> 32);
    vg->max_deg_vertex = hb ? 0xFFFFFFFFu - (uint32_t)(hb & 0xFFFFFFFFu) : 0u;
    d->P = 0;
    vg->bytes += sizeof(uint32_t) * (size_t)(n + 1);
    return EEG_OK;
}

// Sparse graphs are sorted down to the vertex instead of into buckets: a bucket costs its tile (64 KB of counters
// cleared twice, 8 KB of counts written and read), however few edges it has. Device arrays, forward and weighted, ms:
// 2^26 vertices with 1 M edges 4.19 -> 1.02, with 8 M 5.1 -> 1.8, with 64 M 7.8 -> 5.7 (128 M: 9.8, 9.2 this way); 2^24
// with 8 M 1.62 -> 1.00, with 32 M 2.50 (2.39 this way, symmetrised 3.15 and 3.21); 2^22 with 2 M 0.43 -> 0.35, with
// 4 M 0.51 (0.51); 2^20 with 0.5 M 0.21 (0.21). Up to 2^22 vertices the buckets take one pass, this two.
static bool sorted_by_vertex(uint32_t n, uint64_t m) {
    return m > 0 && n > (1u << 20) && (n > (1u << 22) ? 2 * m < 3ull * n : 4 * m < 3ull * n);
}

// Build one direction. reverse: edges (s,t) are inserted as (t,s) -- the transposed graph. Each vertex's
// edges keep the input order (the order the reference's MakeGraph gives them) and the layout is
// deterministic. With EEG_VG_SYMMETRIZE the vg->m arcs are the vg->m / 2 input edges followed by their
// reverses. host_in: the input arrays are page-locked host memory, each read once over the link.
eeg_status build_direction(eeg_vgraph* vg, VDir* d, const uint32_t* d_src, const uint32_t* d_dst,
                           const uint32_t* d_w, bool reverse, bool host_in, cudaStream_t st) {
    const uint32_t n = vg->n, K = vg->K;
    const uint64_t m = vg->m;
    const bool sym = (vg->flags & EEG_VG_SYMMETRIZE) != 0;
    const uint64_t m_in = sym ? m / 2 : m;  // input edges
    const bool with_w = (d_w != nullptr) || (!reverse && vg->weighted);
    const bool eid = (vg->flags & EEG_VG_EDGE_IDS) != 0;
    const bool payload = with_w || eid;  // a third word per edge: weight, or edge index
    const uint32_t bits = n > 1 ? 32u - (uint32_t)__builtin_clz(n - 1) : 1u;
    const bool by_vertex = sorted_by_vertex(n, m);
    const uint32_t low = by_vertex ? 0u : (uint32_t)S_BITS;
    const uint32_t high = bits > low ? bits - low : 0u;  // bits to partition by
    const uint32_t passes = std::max<uint32_t>(1u, (high + S_BITS - 1) / S_BITS);
    const uint32_t nb_buckets = n ? ((n - 1) >> S_BITS) + 1u : 1u;
    // the first pass's tiles have one direction each (later passes have no more of them)
    const uint64_t ntiles = ((m_in + S_TILE - 1) / S_TILE) * (sym ? 2u : 1u);
    const uint64_t ntiles2 = (m + S_TILE - 1) / S_TILE;
    const uint64_t nchunks = (ntiles + S_CHUNK - 1) / S_CHUNK;
    const uint64_t vtiles = m / S_TILE + std::min<uint64_t>(nb_buckets, m);  // most tiles the buckets can have
    const bool low_keys = passes == 1 && !by_vertex;  // the partition keeps the low bits only

    EEG_TRY(vg_alloc(vg, (void**)&d->deg, sizeof(uint32_t) * (size_t)(n + 1)));
    EEG_TRY(vg_alloc(vg, (void**)&d->vstart, sizeof(uint32_t) * (size_t)(n + 1)));
    TempSet T(st);
    uint32_t *np = nullptr, *tmp = nullptr, *err = nullptr;
    EEG_TRY(T.get((void**)&np, sizeof(uint32_t) * (size_t)(n + 1)));
    EEG_TRY(T.get((void**)&err, 16));
    EEG_TRY(T.get((void**)&tmp, sizeof(uint32_t) * device_scan_tmp_words((uint64_t)n + 1)));
    unsigned long long* best = (unsigned long long*)(err + 2);
    EEG_CUDA(cudaMemsetAsync(err, 0, 16, st));

    // ---- partition by bucket
    void* key = nullptr;                       // uint16_t low bits (one pass) or the uint32_t owners
    uint32_t *nb = nullptr, *pay = nullptr;    // partitioned
    uint32_t *bstart = nullptr, *tstart = nullptr, *tbucket = nullptr, *vcnt = nullptr, *first = nullptr;
    if (m > 0) {
        Arcs s{};
        s.a = reverse ? d_dst : d_src;
        s.b = reverse ? d_src : d_dst;
        s.w = with_w ? d_w : nullptr;
        s.m_in = m_in;
        s.m = m;
        s.n = n;
        s.shift = (vg->flags & EEG_VG_SHIFT_ONE) ? 1u : 0u;
        s.sym = sym ? 1 : 0;
        s.eid = eid ? 1 : 0;
        s.err = err;
        const uint32_t max_bins = 1u << std::max(2u, (high + passes - 1) / passes);
        uint32_t *hist = nullptr, *csum = nullptr, *tot = nullptr, *start = nullptr, *copy = nullptr;
        EEG_TRY(T.get((void**)&hist, sizeof(uint32_t) * ntiles * max_bins));
        EEG_TRY(T.get((void**)&csum, sizeof(uint32_t) * nchunks * max_bins));
        EEG_TRY(T.get((void**)&tot, sizeof(uint32_t) * max_bins));
        EEG_TRY(T.get((void**)&start, sizeof(uint32_t) * (max_bins + 1)));
        if (host_in) EEG_TRY(T.get((void**)&copy, sizeof(uint32_t) * m));
        uint32_t* in_key = nullptr;  // null: the arcs
        uint32_t *in_nb = nullptr, *in_pay = nullptr;
        void* out_keys[2] = {nullptr, nullptr};
        uint32_t *out_nbs[2] = {nullptr, nullptr}, *out_pays[2] = {nullptr, nullptr};
        uint32_t lo = low;
        for (uint32_t p = 0; p < passes; ++p) {
            const bool last = p + 1 == passes;
            // bits of this pass (at least 2: the tile kernels take four bins per thread)
            const uint32_t pbits = std::max(2u, last ? std::max(bits, lo) - lo : (high + passes - 1) / passes);
            const uint32_t bins = 1u << pbits;
            // two sets of outputs in turn: the third pass's are the first's
            if (p < 2) {
                EEG_TRY(T.get(&out_keys[p], (low_keys ? sizeof(uint16_t) : sizeof(uint32_t)) * m));
                EEG_TRY(T.get((void**)&out_nbs[p], sizeof(uint32_t) * m));
                if (payload) EEG_TRY(T.get((void**)&out_pays[p], sizeof(uint32_t) * m));
            }
            void* out_key = out_keys[p & 1u];
            uint32_t *out_nb = out_nbs[p & 1u], *out_pay = out_pays[p & 1u];
            const uint64_t nt = p == 0 ? ntiles : ntiles2, nc = (nt + S_CHUNK - 1) / S_CHUNK;
            if (p == 0)
                k_bin_counts<true><<<(unsigned)nt, S_TPB, 0, st>>>(s, nullptr, copy, m, lo, bins, hist);
            else
                k_bin_counts<false><<<(unsigned)nt, S_TPB, 0, st>>>(s, in_key, nullptr, m, lo, bins, hist);
            k_tile_prefix<<<dim3((unsigned)nc, (bins + 255u) / 256u), 256, 0, st>>>(hist, (uint32_t)nt, bins, csum);
            k_chunk_prefix<<<(bins + 255u) / 256u, 256, 0, st>>>(csum, (uint32_t)nc, bins, tot);
            k_bin_starts<<<1, SCAN_TPB, 0, st>>>(tot, bins, start);
            const size_t smem = partition_smem(bins, payload);
            const uint32_t* kin = p == 0 ? copy : in_key;
            auto go = [&](auto kern, auto* kout) -> eeg_status {
                EEG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PARTITION_SMEM));
                kern<<<(unsigned)nt, S_TPB, smem, st>>>(s, kin, in_nb, in_pay, m, lo, bins, hist, csum, start, kout,
                                                            out_nb, out_pay);
                return EEG_OK;
            };
            if (low_keys) EEG_TRY(go(k_partition<true, uint16_t>, (uint16_t*)out_key));
            else if (p == 0) EEG_TRY(go(k_partition<true, uint32_t>, (uint32_t*)out_key));
            else EEG_TRY(go(k_partition<false, uint32_t>, (uint32_t*)out_key));
            EEG_CUDA(cudaGetLastError());
            in_key = low_keys ? nullptr : (uint32_t*)out_key;
            in_nb = out_nb;
            in_pay = out_pay;
            key = out_key;
            lo += pbits;
        }
        nb = in_nb;
        pay = in_pay;
        if (by_vertex) {
            EEG_TRY(T.get((void**)&first, sizeof(uint32_t) * (size_t)n));
            EEG_CUDA(cudaMemsetAsync(d->deg, 0, sizeof(uint32_t) * (size_t)n, st));
            k_runs<<<grid_for(m, vg->device), B_TPB, 0, st>>>((const uint32_t*)key, m, first, d->deg);
        } else {
            // ---- tiles of the buckets, counts per vertex
            EEG_TRY(T.get((void**)&tstart, sizeof(uint32_t) * ((size_t)nb_buckets + 1)));
            EEG_TRY(T.get((void**)&tbucket, sizeof(uint32_t) * vtiles));
            EEG_TRY(T.get((void**)&vcnt, sizeof(uint32_t) * vtiles * S_BINS));
            if (low_keys) {
                bstart = start;  // bins at least the buckets; their starts run on to m
            } else {
                EEG_TRY(T.get((void**)&bstart, sizeof(uint32_t) * ((size_t)nb_buckets + 1)));
                k_bucket_starts<<<grid_for(m + 1, vg->device), B_TPB, 0, st>>>((const uint32_t*)key, m, nb_buckets, bstart);
            }
            k_bucket_tiles<<<1, SCAN_TPB, 0, st>>>(bstart, nb_buckets, tstart, tbucket);
            if (low_keys)
                k_vertex_counts<uint16_t><<<(unsigned)vtiles, S_TPB, 0, st>>>((const uint16_t*)key, bstart, tstart, tbucket,
                                                                              nb_buckets, vcnt);
            else
                k_vertex_counts<uint32_t><<<(unsigned)vtiles, S_TPB, 0, st>>>((const uint32_t*)key, bstart, tstart, tbucket,
                                                                              nb_buckets, vcnt);
        }
    } else if (!by_vertex) {  // no edges: no tile in any bucket
        EEG_TRY(T.get((void**)&tstart, sizeof(uint32_t) * ((size_t)nb_buckets + 1)));
        EEG_CUDA(cudaMemsetAsync(tstart, 0, sizeof(uint32_t) * ((size_t)nb_buckets + 1), st));
    }
    if (by_vertex)
        k_run_degrees<<<grid_for((uint64_t)n, vg->device), 256, 0, st>>>(first, n, K, d->deg, np, best);
    else
        k_degrees<<<dim3(grid_for((uint64_t)n, vg->device), 8), 256, 0, st>>>(vcnt, tstart, n, K, d->deg, np, best);
    EEG_TRY(device_scan_u32(np, d->vstart, (uint64_t)n + 1, false, SCAN_ADD, tmp, st));

    uint32_t hbuf[4] = {0, 0, 0, 0};
    uint32_t P32 = 0;
    EEG_CUDA(cudaMemcpyAsync(hbuf, err, 16, cudaMemcpyDeviceToHost, st));
    EEG_CUDA(cudaMemcpyAsync(&P32, d->vstart + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    EEG_CUDA(cudaStreamSynchronize(st));
    if (hbuf[0]) {
        set_last_error("edge endpoint outside [0, num_nodes)");
        return EEG_ERR_INVALID;
    }
    const unsigned long long kbest = ((unsigned long long)hbuf[3] << 32) | hbuf[2];
    if (!reverse) {
        vg->max_deg = (uint32_t)(kbest >> 32);
        vg->max_deg_vertex = kbest ? 0xFFFFFFFFu - (uint32_t)(kbest & 0xFFFFFFFFu) : 0u;
    }
    const uint64_t P = P32;
    d->P = P;
    const size_t slots = (size_t)P * K;
    EEG_TRY(vg_alloc(vg, (void**)&d->vowner, sizeof(uint32_t) * (size_t)std::max<uint64_t>(P, 1)));
    EEG_TRY(vg_alloc(vg, (void**)&d->vcol, sizeof(uint32_t) * std::max<size_t>(slots, 4)));
    if (with_w) EEG_TRY(vg_alloc(vg, (void**)&d->vw, sizeof(uint32_t) * std::max<size_t>(slots, 4)));
    if (eid) EEG_TRY(vg_alloc(vg, (void**)&d->veid, sizeof(uint32_t) * std::max<size_t>(slots, 4)));

    if (P > 0) {
        uint32_t* hubs = nullptr;
        if ((kbest >> 32) > (uint64_t)HUB_PARTS * K) {  // each of them has more edges than that
            EEG_TRY(T.get((void**)&hubs, sizeof(uint32_t) * (m / ((uint64_t)HUB_PARTS * K) + 2)));
            EEG_CUDA(cudaMemsetAsync(hubs, 0, sizeof(uint32_t), st));
        }
        k_owners<<<grid_for(n, vg->device), B_TPB, 0, st>>>(n, K, d->vstart, d->deg, d->vowner, d->vcol, d->vw, d->veid, hubs);
        if (hubs) k_hub_owners<<<(unsigned)sm_count(vg->device) * 2, B_TPB, 0, st>>>(hubs, d->vstart, d->vowner);
        if (by_vertex) {
            k_place_runs<<<grid_for(m, vg->device), B_TPB, 0, st>>>((const uint32_t*)key, nb, pay, m, K, first, d->vstart, d->vcol,
                                                                    d->vw, with_w ? d_w : nullptr, d->veid, sym ? m_in : 0);
        } else {
            const size_t psm = place_smem(payload);
            auto go = [&](auto kern, auto* k) -> eeg_status {
                EEG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PLACE_SMEM));
                kern<<<(unsigned)vtiles, S_TPB, psm, st>>>(k, nb, pay, bstart, tstart, tbucket, nb_buckets, n, K, vcnt,
                                                                 d->vstart, d->vcol, d->vw, with_w ? d_w : nullptr, d->veid,
                                                                 sym ? m_in : 0);
                return EEG_OK;
            };
            if (low_keys) EEG_TRY(go(k_place<uint16_t>, (const uint16_t*)key));
            else EEG_TRY(go(k_place<uint32_t>, (const uint32_t*)key));
        }
    }
    EEG_CUDA(cudaGetLastError());
    vg->bytes += sizeof(uint32_t) * ((size_t)(n + 1) * 2 + (size_t)P + slots * (1 + (with_w ? 1 : 0) + (eid ? 1 : 0)));
    return EEG_OK;
}

}  // namespace eeg
