// Subgraph rewrites applied after a sampling pass
// (crates/aethergraph-core/src/loader/sampler.rs:964-1040 apply_subgraph_type):
//   mirror  (bidirectional): the sampled edges stay, then the reverse of edge i is
//           appended, in the order of i, unless its (src_local, dst_local) pair is
//           already among the sampled edges or an earlier appended reverse;
//   induce  (induced): the edges become every stored edge between two sampled
//           nodes, ordered by the expanded node's local index, then row position.
// Both are exact restatements for parallel hardware: "first in order wins" is an
// atomicMin over edge positions in a hash table of pairs, "in order" is a prefix
// sum over keep flags.  Hash probes are bounded by the table size.
#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "internal.h"

using namespace ag;

namespace {

constexpr uint64_t kEmptyKey = ~0ull;

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
    return x;
}

// Finds `key` or claims an empty slot for it; returns the slot, or ~0 when the
// table is full (cannot happen at load <= 1/2; the caller records it).
__device__ __forceinline__ uint64_t find_or_insert(unsigned long long *keys, uint64_t mask, uint64_t key) {
    uint64_t slot = mix64(key) & mask;
    for (uint64_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long cur = keys[slot];
        if (cur == key) return slot;
        if (cur == kEmptyKey) {
            const unsigned long long prev = atomicCAS(&keys[slot], (unsigned long long)kEmptyKey, (unsigned long long)key);
            if (prev == kEmptyKey || prev == key) return slot;
        }
        slot = (slot + 1) & mask;
    }
    return ~0ull;
}

__device__ __forceinline__ uint64_t find(const unsigned long long *keys, uint64_t mask, uint64_t key) {
    uint64_t slot = mix64(key) & mask;
    for (uint64_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long cur = keys[slot];
        if (cur == key) return slot;
        if (cur == kEmptyKey) return ~0ull;
        slot = (slot + 1) & mask;
    }
    return ~0ull;
}

__device__ __forceinline__ uint64_t pair_key(uint32_t a, uint32_t b) { return ((uint64_t)a << 32) | b; }

// Phase 1: every sampled pair enters the table with value 0 ("forward").
__global__ void k_mirror_forward(const uint32_t *__restrict__ sl, const uint32_t *__restrict__ dl, uint64_t n,
                                 unsigned long long *keys, uint32_t *vals, uint64_t mask, uint32_t *err) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t slot = find_or_insert(keys, mask, pair_key(sl[i], dl[i]));
        if (slot == ~0ull) { atomicOr(err, 1u); continue; }
        atomicMin(&vals[slot], 0u);
    }
}

// Phase 2: the reverse pair of edge i competes with value i + 1; a pair that is a
// forward pair keeps 0, otherwise the smallest i wins.
__global__ void k_mirror_reverse(const uint32_t *__restrict__ sl, const uint32_t *__restrict__ dl, uint64_t n,
                                 unsigned long long *keys, uint32_t *vals, uint64_t mask, uint32_t *err) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t slot = find_or_insert(keys, mask, pair_key(dl[i], sl[i]));
        if (slot == ~0ull) { atomicOr(err, 1u); continue; }
        atomicMin(&vals[slot], (uint32_t)(i + 1));
    }
}

__global__ void k_mirror_flags(const uint32_t *__restrict__ sl, const uint32_t *__restrict__ dl, uint64_t n,
                               const unsigned long long *keys, const uint32_t *vals, uint64_t mask, uint32_t *flags) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t slot = find(keys, mask, pair_key(dl[i], sl[i]));
        flags[i] = (slot != ~0ull && vals[slot] == (uint32_t)(i + 1)) ? 1u : 0u;
    }
}

// Appends the winners behind the n sampled edges.  rank = exclusive prefix of flags.
__global__ void k_mirror_append(uint32_t *edge_src, uint32_t *edge_dst, uint32_t *sl, uint32_t *dl, uint64_t *edge_ids,
                                uint64_t n, const uint32_t *__restrict__ flags, const uint32_t *__restrict__ rank) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!flags[i]) continue;
        const uint64_t o = n + rank[i];
        edge_src[o] = edge_dst[i]; edge_dst[o] = edge_src[i];
        sl[o] = dl[i]; dl[o] = sl[i];
        if (edge_ids) edge_ids[o] = edge_ids[i];
    }
}

// int64 [2, e]: row 0 the neighbor's local index, row 1 the expanded node's.
__global__ void k_edge_index_local(const uint32_t *__restrict__ sl, const uint32_t *__restrict__ dl, uint64_t e, int64_t *out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < e; i += (uint64_t)gridDim.x * blockDim.x) {
        out[i] = (int64_t)dl[i];
        out[e + i] = (int64_t)sl[i];
    }
}

uint64_t pow2_at_least(uint64_t v) {
    uint64_t p = 1024;
    while (p < v) p <<= 1;
    return p;
}

uint32_t grid_for(uint64_t n) { return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)kSMs * 8)); }

struct Scratch {
    cudaStream_t st;
    void *p[6] = {};
    bool idle = false;  // nothing queued on `st` uses the blocks any more
    ~Scratch() {
        if (!idle) cudaStreamSynchronize(st);
        for (void *q : p) workspace_free(q);
    }
};

}  // namespace

// In place on the device arrays of one sampled subgraph.  The four u32 edge arrays
// (and edge_ids when given) hold n_edges entries and room for 2 * n_edges;
// edge_index_local (optional) has room for [2, 2 * n_edges] and is rewritten for the
// new edge count.  *n_edges_out (host) receives the new count.  Synchronous.
extern "C" int32_t ag_subgraph_mirror(int32_t device, uint64_t n_edges, uint64_t cap_edges, uint32_t *edge_src,
                                      uint32_t *edge_dst, uint32_t *src_local, uint32_t *dst_local, uint64_t *edge_ids,
                                      int64_t *edge_index_local, uint64_t *n_edges_out, void *stream) {
    if (!n_edges_out) return fail(AG_ERR_VALUE, "ag_subgraph_mirror: null argument");
    *n_edges_out = n_edges;
    if (n_edges == 0) return AG_OK;
    if (!edge_src || !edge_dst || !src_local || !dst_local) return fail(AG_ERR_VALUE, "ag_subgraph_mirror: null edge array");
    if (cap_edges < 2 * n_edges) return fail(AG_ERR_VALUE, "ag_subgraph_mirror: capacity %llu < 2 x %llu edges",
                                             (unsigned long long)cap_edges, (unsigned long long)n_edges);
    if (n_edges >= 0x7FFFFFFFull) return fail(AG_ERR_VALUE, "ag_subgraph_mirror: too many edges");
    DeviceGuard guard(device);
    if (!guard.ok) return AG_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t cap = pow2_at_least(4 * n_edges), mask = cap - 1;  // <= 2n keys: load <= 1/2
    Scratch sc{st};
    unsigned long long *keys = nullptr; uint32_t *vals = nullptr, *flags = nullptr, *rank = nullptr, *err = nullptr;
    AG_CUDA(workspace_alloc(&sc.p[0], cap * 8)); keys = (unsigned long long *)sc.p[0];
    AG_CUDA(workspace_alloc(&sc.p[1], cap * 4)); vals = (uint32_t *)sc.p[1];
    AG_CUDA(workspace_alloc(&sc.p[2], (n_edges + 1) * 4)); flags = (uint32_t *)sc.p[2];
    AG_CUDA(workspace_alloc(&sc.p[3], (n_edges + 1) * 4)); rank = (uint32_t *)sc.p[3];
    AG_CUDA(workspace_alloc(&sc.p[4], 4)); err = (uint32_t *)sc.p[4];
    AG_CUDA(cudaMemsetAsync(keys, 0xFF, cap * 8, st));
    AG_CUDA(cudaMemsetAsync(vals, 0xFF, cap * 4, st));
    AG_CUDA(cudaMemsetAsync(err, 0, 4, st));
    AG_CUDA(cudaMemsetAsync(flags + n_edges, 0, 4, st));
    const uint32_t grid = grid_for(n_edges);
    k_mirror_forward<<<grid, 256, 0, st>>>(src_local, dst_local, n_edges, keys, vals, mask, err);
    k_mirror_reverse<<<grid, 256, 0, st>>>(src_local, dst_local, n_edges, keys, vals, mask, err);
    k_mirror_flags<<<grid, 256, 0, st>>>(src_local, dst_local, n_edges, keys, vals, mask, flags);
    size_t temp_bytes = 0;
    AG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, flags, rank, (int)(n_edges + 1), st));
    AG_CUDA(workspace_alloc(&sc.p[5], std::max<size_t>(temp_bytes, 16)));
    AG_CUDA(cub::DeviceScan::ExclusiveSum(sc.p[5], temp_bytes, flags, rank, (int)(n_edges + 1), st));
    k_mirror_append<<<grid, 256, 0, st>>>(edge_src, edge_dst, src_local, dst_local, edge_ids, n_edges, flags, rank);
    uint32_t added = 0, herr = 0;
    AG_CUDA(cudaMemcpyAsync(&added, rank + n_edges, 4, cudaMemcpyDeviceToHost, st));
    AG_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st));
    AG_CUDA(cudaStreamSynchronize(st));
    sc.idle = true;
    if (herr) return fail(AG_ERR_WORKER, "ag_subgraph_mirror: pair table overflow");
    const uint64_t total = n_edges + added;
    if (edge_index_local) {
        k_edge_index_local<<<grid_for(total), 256, 0, st>>>(src_local, dst_local, total, edge_index_local);
        AG_CUDA(cudaStreamSynchronize(st));
    }
    AG_CUDA(cudaGetLastError());
    *n_edges_out = total;
    return AG_OK;
}

// ------------------------------------------------------------------ induce --
namespace {

// The rows of the sampled nodes, one after the other in local order, form one list of
// positions: the result is the hits of that list, in list order.  Every warp takes an
// equal stretch of it, whatever rows it crosses, counts its hits (first walk) and, once
// the counts are scanned, writes them behind the stretches before it (second walk).
//
// Rows differ by five orders of magnitude (a hub of an R-MAT graph of 64 M edges has
// over 100 K neighbours, most vertices a few), so a warp per row leaves the two walks to
// the warp with the longest one: 200 seeds, fanouts 10, 5 on that graph reach 3200 nodes
// and 5.7 M positions, 2660 + 3080 us at 4 % of the warps busy; in equal stretches 39 + 44 us.
// Bound by latency: half of the warps resident, 36 and 47 % of the issue slots used, 6 % of the
// DRAM rate; a warp waits nine cycles an issue for loads, four at the barriers of the filter
// (counting walk) or seven for loads (filling walk).
// One block per SM, so that the filter below is built once for 32 warps and the counts that
// are scanned are one per block (256-thread blocks: 55 + 48 us, of it 25 us for the scan of
// 4736 warp counts and up to 10 us for building the filter in waves of blocks).
constexpr int kWalkThreads = 1024;
constexpr uint32_t kWalkWarps = kWalkThreads / 32;
constexpr uint32_t kWalkMin = 128;   // positions a warp takes at least
constexpr uint32_t kWalkUnroll = 4;  // 32-position chunks in flight in a long row
// Most neighbours are not in the sample, and a probe of the node table is 32 scattered
// reads for a warp.  A bitmap of the nodes' hashes in shared memory answers for most of
// them: kFilterMin - kFilterMax words a block, 16 bits or more per node where that fits
// (up to 1 / 16 of the misses pass), built by every block from the node list; none above
// kFilterNodes nodes, where it would be over a quarter full and slow to build.
constexpr uint32_t kFilterMin = 1024, kFilterMax = 16384;
constexpr uint64_t kFilterNodes = 1 << 17;

__device__ __forceinline__ uint32_t node_slot(uint32_t v, uint32_t mask) { return (uint32_t)(mix64(v) & mask); }

// The sampled nodes are distinct: table of node << 32 | local index, and every node's row.
__global__ void k_induce_insert(const uint64_t *__restrict__ offsets, uint64_t num_graph_nodes, uint64_t num_edges,
                                const uint32_t *__restrict__ nodes, uint64_t n, unsigned long long *table, uint32_t mask,
                                uint64_t *row_off, uint64_t *row_len, uint32_t *err) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = nodes[i];
        uint64_t lo = 0, hi = 0;
        if ((uint64_t)v < num_graph_nodes) { lo = offsets[v]; hi = offsets[(uint64_t)v + 1]; }
        row_off[i] = lo;
        row_len[i] = (hi > lo && hi <= num_edges) ? hi - lo : 0;
        const unsigned long long entry = ((unsigned long long)v << 32) | (uint32_t)i;
        uint32_t slot = node_slot(v, mask);
        bool done = false;
        for (uint32_t probe = 0; probe <= mask && !done; ++probe) {
            done = atomicCAS(&table[slot], (unsigned long long)kEmptyKey, entry) == kEmptyKey;
            slot = (slot + 1) & mask;
        }
        if (!done) atomicOr(err, 1u);
    }
}

// Local index of node v, or 0xFFFFFFFF (never one: a plan holds fewer than 2^30 nodes).
__device__ __forceinline__ uint32_t node_lookup(const unsigned long long *__restrict__ table, uint32_t mask, uint32_t v) {
    uint32_t slot = node_slot(v, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long e = __ldg(table + slot);
        if (e == kEmptyKey) return 0xFFFFFFFFu;
        if ((uint32_t)(e >> 32) == v) return (uint32_t)e;
        slot = (slot + 1) & mask;
    }
    return 0xFFFFFFFFu;
}

struct InduceWalk {
    const uint32_t *dst, *nodes;
    uint64_t n;
    const uint64_t *row_off;    // [n] first CSR position of every node's row
    const uint64_t *row_start;  // [n + 1] its first position in the list
    const unsigned long long *table;
    uint32_t mask, warps;
    uint32_t filter_words;      // a power of two, or 0: no filter
    uint64_t *warp_start;       // [warps] hits of the block's earlier warps
    uint64_t *block_start;      // [warps / kWalkWarps] hits of the block, then (scanned) of the blocks before it
    uint64_t *total;            // [0] all hits, [1] blocks that have counted
};

struct InduceOut {
    uint32_t *edge_src, *edge_dst, *sl, *dl;
    uint64_t *edge_ids;
    int64_t *edge_index_local;
    uint64_t n_edges;
};

// Row that holds position g of the list, searched from row `lo` on.
__device__ __forceinline__ uint64_t row_of(const uint64_t *__restrict__ row_start, uint64_t n, uint64_t lo, uint64_t g) {
    uint64_t hi = n;  // row_start[lo] <= g < row_start[hi]
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (__ldg(row_start + mid) <= g) lo = mid; else hi = mid;
    }
    return lo;
}

// A node's bit in the filter: another hash than the table's.
__device__ __forceinline__ uint32_t filter_bit(uint32_t v, uint32_t words) { return (v * 0x9E3779B1u) >> (32 - 5 - (31 - __clz(words))); }

// Both walks.  In a long row the warp reads kWalkUnroll chunks of it at once.  Elsewhere the
// positions lie in several rows: the lanes hold the ends of the next 32 rows and every lane
// finds its rows among them by shuffles (a search through memory per lane took 4 us for 32
// positions), kWalkUnroll chunks at once (one at a time: 1 us each); only positions beyond
// those 32 rows fall back to the search.
template <bool FILL>
__global__ void __launch_bounds__(kWalkThreads)
k_induce_walk(InduceWalk a, InduceOut o) {
    extern __shared__ uint32_t s_filter[];
    if (a.filter_words) {
        for (uint32_t i = threadIdx.x; i < a.filter_words; i += kWalkThreads) s_filter[i] = 0;
        __syncthreads();
        for (uint64_t i = threadIdx.x; i < a.n; i += kWalkThreads) {
            const uint32_t bit = filter_bit(__ldg(a.nodes + i), a.filter_words);
            atomicOr(&s_filter[bit >> 5], 1u << (bit & 31));
        }
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31, w = (blockIdx.x * kWalkThreads + threadIdx.x) >> 5;
    const uint64_t all = a.row_start[a.n];
    const uint64_t share = ((all + a.warps - 1) / a.warps + 31) & ~31ull;
    const uint64_t per = share > kWalkMin ? share : kWalkMin;
    uint64_t g = min(all, (uint64_t)w * per);
    const uint64_t stop = min(all, g + per);
    uint64_t out = FILL ? a.block_start[blockIdx.x] + a.warp_start[w] : 0;
    uint64_t count = 0;
    // hits of 32 positions: lane's neighbour v at CSR position pos in the row of local index r
    auto take = [&](uint32_t hit, uint32_t v, uint64_t pos, uint32_t r, uint32_t node) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit != 0xFFFFFFFFu);
        if (FILL) {
            if (hit != 0xFFFFFFFFu) {
                const uint64_t at = out + __popc(m & ((1u << lane) - 1));
                o.edge_src[at] = node; o.edge_dst[at] = v; o.sl[at] = r; o.dl[at] = hit;
                if (o.edge_ids) o.edge_ids[at] = pos;
                if (o.edge_index_local) { o.edge_index_local[at] = (int64_t)hit; o.edge_index_local[o.n_edges + at] = (int64_t)r; }
            }
            out += __popc(m);
        } else {
            count += __popc(m);
        }
    };
    auto find = [&](uint32_t v) {
        if (!a.filter_words) return node_lookup(a.table, a.mask, v);
        const uint32_t bit = filter_bit(v, a.filter_words);
        return ((s_filter[bit >> 5] >> (bit & 31)) & 1u) ? node_lookup(a.table, a.mask, v) : 0xFFFFFFFFu;
    };
    uint64_t row = g < stop ? row_of(a.row_start, a.n, 0, g) : 0;  // row_start[row] <= g
    while (g < stop) {
        const uint64_t row_end = __ldg(a.row_start + min(row + 1 + lane, a.n));  // of row + lane
        const uint32_t skip = __popc(__ballot_sync(0xFFFFFFFFu, row_end <= g));   // rows that end at or before g
        if (skip == 32) { row = row_of(a.row_start, a.n, row, g); continue; }
        const uint64_t end = min(stop, __shfl_sync(0xFFFFFFFFu, row_end, skip));
        if (end - g >= 32 * kWalkUnroll) {  // a long row: whole chunks of it
            row += skip;
            const uint64_t base = __ldg(a.row_off + row) - __ldg(a.row_start + row);  // list position -> CSR position
            const uint32_t node = FILL ? __ldg(a.nodes + row) : 0;
            for (; end - g >= 32 * kWalkUnroll; g += 32 * kWalkUnroll) {
                uint32_t v[kWalkUnroll], hit[kWalkUnroll];
#pragma unroll
                for (uint32_t u = 0; u < kWalkUnroll; ++u) v[u] = ld_stream_u32(a.dst + base + g + u * 32 + lane);
#pragma unroll
                for (uint32_t u = 0; u < kWalkUnroll; ++u) hit[u] = find(v[u]);
#pragma unroll
                for (uint32_t u = 0; u < kWalkUnroll; ++u) take(hit[u], v[u], base + g + u * 32 + lane, (uint32_t)row, node);
            }
            continue;
        }
        uint32_t at[kWalkUnroll], v[kWalkUnroll], hit[kWalkUnroll];
        uint64_t pos[kWalkUnroll];
#pragma unroll
        for (uint32_t u = 0; u < kWalkUnroll; ++u) {
            const uint64_t mine = g + u * 32 + lane;
            uint32_t r = 0;  // rows of the window that end at or before this lane's position
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1)
                if (__shfl_sync(0xFFFFFFFFu, row_end, r + step - 1) <= mine) r += step;
            const bool past = __shfl_sync(0xFFFFFFFFu, row_end, 31) <= mine;  // the window ends before it
            at[u] = (uint32_t)row + r; pos[u] = 0; v[u] = 0;
            if (mine < stop) {
                if (past) at[u] = (uint32_t)row_of(a.row_start, a.n, row, mine);
                pos[u] = __ldg(a.row_off + at[u]) + (mine - __ldg(a.row_start + at[u]));
                v[u] = ld_stream_u32(a.dst + pos[u]);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < kWalkUnroll; ++u) hit[u] = g + u * 32 + lane < stop ? find(v[u]) : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t u = 0; u < kWalkUnroll; ++u) {
            const uint32_t node = (FILL && hit[u] != 0xFFFFFFFFu) ? __ldg(a.nodes + at[u]) : 0;
            take(hit[u], v[u], pos[u], at[u], node);
        }
        g += 32 * kWalkUnroll;
        row = __shfl_sync(0xFFFFFFFFu, at[kWalkUnroll - 1], 31);  // at most the row of the next position
    }
    if (FILL) return;
    // Hits before every warp within its block; the block that counts last scans the blocks.
    __shared__ uint64_t s_sum[kWalkWarps];
    __shared__ bool s_last;
    auto scan_warp = [&](uint64_t v) {  // inclusive, over the lanes
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t up = __shfl_up_sync(0xFFFFFFFFu, v, d);
            if ((int)lane >= d) v += up;
        }
        return v;
    };
    if (lane == 0) s_sum[threadIdx.x >> 5] = count;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint64_t mine = s_sum[lane], upto = scan_warp(mine);
        a.warp_start[blockIdx.x * kWalkWarps + lane] = upto - mine;
        if (lane == 31) a.block_start[blockIdx.x] = upto;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd((unsigned long long *)(a.total + 1), 1ull) == gridDim.x - 1;
        __threadfence();  // before the other threads' reads, by the barrier
    }
    __syncthreads();
    if (!s_last) return;
    uint64_t before = 0;
    for (uint32_t base = 0; base < gridDim.x; base += kWalkThreads) {
        const uint32_t i = base + threadIdx.x;
        const uint64_t mine = i < gridDim.x ? __ldcg(a.block_start + i) : 0, upto = scan_warp(mine);
        __syncthreads();
        if (lane == 31) s_sum[threadIdx.x >> 5] = upto;
        __syncthreads();
        if (threadIdx.x < 32) s_sum[lane] = scan_warp(s_sum[lane]);
        __syncthreads();
        const uint64_t earlier = before + (threadIdx.x >= 32 ? s_sum[(threadIdx.x >> 5) - 1] : 0);
        if (i < gridDim.x) a.block_start[i] = earlier + upto - mine;
        before += s_sum[kWalkWarps - 1];
    }
    if (threadIdx.x == 0) a.total[0] = before;
}

}  // namespace

struct ag_induce_plan {
    int device = 0;
    uint64_t n_edges = 0;
    cudaStream_t stream = nullptr;  // the last call's
    void *scratch = nullptr;
    InduceWalk walk{};
};

extern "C" void ag_subgraph_induce_free(ag_induce_plan *p) {
    if (!p) return;
    DeviceGuard guard(p->device);
    if (p->scratch) cudaStreamSynchronize(p->stream);  // already idle unless a call failed
    workspace_free(p->scratch);
    delete p;
}

// Step 1 of the induced rewrite: indexes the n_nodes sampled nodes (device u32 ids,
// distinct) and counts the stored edges between them; *n_edges_out (host) sizes the
// arrays for step 2.  `nodes_dev` must stay valid until the plan is freed.  Synchronous.
extern "C" int32_t ag_subgraph_induce_plan(const ag_graph *g, const uint32_t *nodes_dev, uint64_t n_nodes, void *stream,
                                           ag_induce_plan **out, uint64_t *n_edges_out) {
    if (!g || !out || !n_edges_out || (!nodes_dev && n_nodes)) return fail(AG_ERR_VALUE, "ag_subgraph_induce_plan: null argument");
    if (n_nodes >= 0x40000000ull) return fail(AG_ERR_VALUE, "ag_subgraph_induce_plan: too many nodes");
    DeviceGuard guard(g->device);
    if (!guard.ok) return AG_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    ag_induce_plan *p = new ag_induce_plan();
    p->device = g->device; p->stream = st;
    *out = nullptr; *n_edges_out = 0;
    if (n_nodes == 0) { *out = p; return AG_OK; }
    auto bail = [&](int32_t rc) { ag_subgraph_induce_free(p); return rc; };
#define AG_PLAN_CUDA(expr) do { const cudaError_t e_ = (expr); if (e_ != cudaSuccess) \
        return bail(fail(AG_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_))); } while (0)
    const uint64_t cap = pow2_at_least(2 * n_nodes);
    const uint32_t blocks = (uint32_t)kSMs, warps = blocks * kWalkWarps;
    size_t temp_bytes = 0;
    AG_PLAN_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, (uint64_t *)nullptr, (uint64_t *)nullptr, (int)(n_nodes + 1), st));
    // one allocation: table, row offsets, row lengths and their scan, the warps' counts, totals, scan scratch
    const uint64_t words = cap + n_nodes + 2 * (n_nodes + 1) + warps + blocks + 3;
    const uint64_t temp_at = (words * 8 + 255) & ~255ull;
    AG_PLAN_CUDA(workspace_alloc(&p->scratch, temp_at + temp_bytes));
    unsigned long long *table = (unsigned long long *)p->scratch;
    uint64_t *row_off = (uint64_t *)(table + cap), *row_len = row_off + n_nodes, *row_start = row_len + n_nodes + 1;
    uint64_t *warp_start = row_start + n_nodes + 1, *block_start = warp_start + warps, *total = block_start + blocks;  // total[2]: error bits
    AG_PLAN_CUDA(cudaMemsetAsync(table, 0xFF, cap * 8, st));
    AG_PLAN_CUDA(cudaMemsetAsync(total, 0, 24, st));
    AG_PLAN_CUDA(cudaMemsetAsync(row_len + n_nodes, 0, 8, st));
    k_induce_insert<<<grid_for(n_nodes), 256, 0, st>>>(g->offsets, g->num_nodes, g->num_edges, nodes_dev, n_nodes, table,
                                                       (uint32_t)(cap - 1), row_off, row_len, (uint32_t *)(total + 2));
    AG_PLAN_CUDA(cub::DeviceScan::ExclusiveSum((uint8_t *)p->scratch + temp_at, temp_bytes, row_len, row_start, (int)(n_nodes + 1), st));
    // cap >= 2 n: 16 bits or more per node
    const uint32_t filter = n_nodes > kFilterNodes ? 0 : (uint32_t)std::min<uint64_t>(std::max<uint64_t>(cap / 4, kFilterMin), kFilterMax);
    AG_PLAN_CUDA(cudaFuncSetAttribute(k_induce_walk<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFilterMax * 4));
    AG_PLAN_CUDA(cudaFuncSetAttribute(k_induce_walk<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFilterMax * 4));
    p->walk = InduceWalk{g->dst, nodes_dev, n_nodes, row_off, row_start, table, (uint32_t)(cap - 1), warps, filter, warp_start, block_start, total};
    k_induce_walk<false><<<blocks, kWalkThreads, filter * 4, st>>>(p->walk, InduceOut{});
    AG_PLAN_CUDA(cudaGetLastError());
    uint64_t got[3] = {0, 0, 0};
    AG_PLAN_CUDA(cudaMemcpyAsync(got, total, 24, cudaMemcpyDeviceToHost, st));
    AG_PLAN_CUDA(cudaStreamSynchronize(st));
#undef AG_PLAN_CUDA
    if ((uint32_t)got[2]) return bail(fail(AG_ERR_WORKER, "ag_subgraph_induce_plan: node table overflow"));
    p->n_edges = got[0];
    *n_edges_out = got[0];
    *out = p;
    return AG_OK;
}

// Step 2: writes the plan's edges (cap_edges >= the planned count).  edge_ids and
// edge_index_local ([2, n_edges] int64) are optional.  Synchronous.
extern "C" int32_t ag_subgraph_induce_fill(ag_induce_plan *p, uint64_t cap_edges, uint32_t *edge_src, uint32_t *edge_dst,
                                           uint32_t *src_local, uint32_t *dst_local, uint64_t *edge_ids,
                                           int64_t *edge_index_local, void *stream) {
    if (!p) return fail(AG_ERR_VALUE, "ag_subgraph_induce_fill: null plan");
    if (p->n_edges == 0) return AG_OK;
    if (!edge_src || !edge_dst || !src_local || !dst_local) return fail(AG_ERR_VALUE, "ag_subgraph_induce_fill: null edge array");
    if (cap_edges < p->n_edges) return fail(AG_ERR_VALUE, "ag_subgraph_induce_fill: capacity %llu < %llu edges",
                                            (unsigned long long)cap_edges, (unsigned long long)p->n_edges);
    DeviceGuard guard(p->device);
    if (!guard.ok) return AG_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    p->stream = st;
    const InduceOut o{edge_src, edge_dst, src_local, dst_local, edge_ids, edge_index_local, p->n_edges};
    k_induce_walk<true><<<p->walk.warps / kWalkWarps, kWalkThreads, p->walk.filter_words * 4, st>>>(p->walk, o);
    AG_CUDA(cudaGetLastError());
    AG_CUDA(cudaStreamSynchronize(st));
    return AG_OK;
}
