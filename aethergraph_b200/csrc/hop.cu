// One-hop Philox reservoir sampling: the fast-mode sampler of the reference
// (CPU: crates/aethergraph-core/src/internal/philox.rs:59-82 `reservoir_sample`;
// GPU: crates/aether-stream/src/gpu/kernels/sampler/sampler.cu `warp_sample_neighbors`,
// launched by sampler/mod.rs:180-230).  Same inputs, same outputs, same bits:
// for every requested node a row of `fanout` slots —
//   degree == 0 or node outside the graph: count 0;
//   fanout > 32: `fanout` draws with replacement, slot d = row[philox(d) % degree];
//   fanout >= degree: the row itself, count = degree;
//   else Algorithm R keyed by the scan position t (draw t decides j = r % (t + 1)),
// unused slots hold AG_SAMPLE_PAD, counts[row] says how many are real.
//
// Algorithm R looks sequential in t, but every decision j(t) is a pure function
// of (seed, layer, node, t), and the reservoir's final slot j simply holds the
// element with the LARGEST t that chose j (or element j itself if none did).  So
// the t's are evaluated in parallel with a per-slot maximum; nothing waits for
// another and the result is bit-identical.
#include "common.cuh"
#include "internal.h"

namespace ag {
namespace {

constexpr int kHopThreads = 256;
constexpr uint32_t kHopRows = 32;      // most rows a block takes at a time, four per warp
constexpr uint64_t kHopLong = 2048;    // rows from here on are the whole block's work

__device__ __forceinline__ void hop_row(const uint64_t *offsets, uint64_t num_nodes, uint64_t num_edges, uint64_t node,
                                        uint64_t &begin, uint64_t &degree) {
    begin = degree = 0;
    if (node >= num_nodes) return;
    begin = __ldg(offsets + node);
    const uint64_t end = __ldg(offsets + node + 1);
    degree = (end >= begin && end <= num_edges) ? end - begin : 0;
}

// fanout > 32: `fanout` draws with replacement, a warp per row.
__global__ void __launch_bounds__(kHopThreads)
k_hop_replace(const uint64_t *__restrict__ offsets, const uint32_t *__restrict__ neighbors, uint64_t num_nodes,
              uint64_t num_edges, const uint64_t *__restrict__ nodes, uint32_t *__restrict__ output,
              uint32_t *__restrict__ counts, uint64_t node_count, uint32_t fanout, uint64_t seed, uint32_t layer) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t stride = ((uint64_t)gridDim.x * kHopThreads) >> 5;
    for (uint64_t row = ((uint64_t)blockIdx.x * kHopThreads + threadIdx.x) >> 5; row < node_count; row += stride) {
        uint32_t *out = output + row * fanout;
        const uint64_t node = nodes[row];
        uint64_t begin, degree;
        hop_row(offsets, num_nodes, num_edges, node, begin, degree);
        for (uint32_t d = lane; d < fanout; d += 32) {
            uint32_t v = AG_SAMPLE_PAD;
            if (degree) {
                const uint32_t r = philox_u32(seed, layer, node, d);
                const uint64_t at = degree <= 0xFFFFFFFFull ? r % (uint32_t)degree : r % degree;  // the 64-bit remainder is slow
                v = ld_stream_u32(neighbors + begin + at);
            }
            out[d] = v;
        }
        if (lane == 0) counts[row] = degree ? fanout : 0;
    }
}

// Decisions t in [fanout, degree) of one row, four per generator call (draw t is word t % 4
// of block t / 4): `who` of `of` threads, each taking every of-th block of four.
template <typename T>
__device__ __forceinline__ void reservoir_scan(uint64_t seed, uint32_t layer, uint64_t node, T degree, uint32_t fanout,
                                               uint32_t who, uint32_t of, uint32_t *last) {
    for (T g = (fanout >> 2) + who; g * 4 < degree; g += of) {
        const uint4 r = philox4x32_10(seed, layer, node, (uint32_t)g);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const T t = g * 4 + e;
            const uint32_t word = e == 0 ? r.x : e == 1 ? r.y : e == 2 ? r.z : r.w;
            if (t < fanout || t >= degree) continue;
            const uint32_t j = word % (uint32_t)(t + 1);
            if (j < fanout) atomicMax(&last[j], (uint32_t)t);
        }
    }
}

// Rows of hundreds of neighbours: bound by the generator and the remainder, about 45 instructions
// a decision with a generator call each and a third of that with four per call; and by the
// longest row: a row of 150 K neighbours takes one warp longer than 100 K ordinary rows take
// the GPU.  Rows with at most 32 decisions: latency, so a decision per lane (100 K rows of 40
// neighbours, fanout 25: 33 us, 41 with four per call), one barrier a round, and 45 registers
// instead of 48 for the row in 32 bits.  300 K rows of a 4 M vertex / 100 M edge R-MAT graph,
// fanout 25: 92 us, 290 and more with a warp per row and a call per decision; 300 K rows of 300
// neighbours 231 and 372, of 10 neighbours 62 and 61 (fanout 8: 86 and 79).
__global__ void __launch_bounds__(kHopThreads)
k_hop_reservoir(const uint64_t *__restrict__ offsets, const uint32_t *__restrict__ neighbors, uint64_t num_nodes,
                uint64_t num_edges, const uint64_t *__restrict__ nodes, uint32_t *__restrict__ output,
                uint32_t *__restrict__ counts, uint64_t node_count, uint32_t fanout, uint64_t seed, uint32_t layer, uint32_t round) {
    constexpr uint32_t kWarps = kHopThreads / 32;
    __shared__ uint32_t s_last[kWarps + 1][32];  // per warp, and for the block: largest t that chose slot j
    __shared__ uint32_t s_long[kHopRows];        // rows of this round left to the block
    __shared__ uint32_t s_longs;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto row_of = [&](uint64_t row, uint64_t &node, uint64_t &begin, uint64_t &degree) {
        node = nodes[row];
        hop_row(offsets, num_nodes, num_edges, node, begin, degree);
    };
    if (threadIdx.x == 0) s_longs = 0;
    __syncthreads();
    for (uint64_t base = (uint64_t)blockIdx.x * round; base < node_count; base += (uint64_t)gridDim.x * round) {
        bool left = false;  // a row of this warp is left to the block
        for (uint32_t i = warp; i < round && base + i < node_count; i += kWarps) {
            uint32_t *out = output + (base + i) * fanout;
            uint64_t node, begin, length;
            row_of(base + i, node, begin, length);
            if (length >= kHopLong) {  // more than any fanout of this kernel
                if (lane == 0) s_long[atomicAdd(&s_longs, 1u)] = i;
                left = true;
                continue;
            }
            const uint32_t degree = (uint32_t)length, taken = min(degree, fanout);
            uint32_t from = lane;  // this lane's neighbour
            if (degree > fanout) {
                s_last[warp][lane] = lane;  // slot j starts with element j
                __syncwarp();
                if (degree <= fanout + 32) {  // a decision per lane
                    const uint32_t t = fanout + lane;
                    const uint32_t j = philox_u32(seed, layer, node, t) % (t + 1);
                    if (t < degree && j < fanout) atomicMax(&s_last[warp][j], t);
                } else {
                    reservoir_scan(seed, layer, node, degree, fanout, lane, 32, s_last[warp]);
                }
                __syncwarp();
                from = s_last[warp][lane];
                __syncwarp();
            }
            if (lane < fanout) out[lane] = lane < taken ? ld_stream_u32(neighbors + begin + from) : AG_SAMPLE_PAD;
            if (lane == 0) counts[base + i] = taken;
        }
        if (!__syncthreads_or(left)) continue;
        for (uint32_t l = 0; l < s_longs; ++l) {
            const uint64_t row = base + s_long[l];
            uint64_t node, begin, degree;
            row_of(row, node, begin, degree);
            if (threadIdx.x < 32) s_last[kWarps][lane] = lane;
            __syncthreads();
            reservoir_scan(seed, layer, node, degree, fanout, threadIdx.x, kHopThreads, s_last[kWarps]);
            __syncthreads();
            if (threadIdx.x < fanout) output[row * fanout + threadIdx.x] = ld_stream_u32(neighbors + begin + s_last[kWarps][threadIdx.x]);
            if (threadIdx.x == 0) counts[row] = fanout;
            __syncthreads();
        }
        if (threadIdx.x == 0) s_longs = 0;
        __syncthreads();
    }
}

}  // namespace
}  // namespace ag

using namespace ag;

extern "C" int32_t ag_sample_hop_reservoir(const ag_graph *g, const uint64_t *nodes_dev, uint64_t node_count,
                                           uint32_t fanout, uint64_t seed, uint32_t layer,
                                           uint32_t *neighbors_out_dev, uint32_t *counts_out_dev, void *stream) {
    if (!g || !neighbors_out_dev || !counts_out_dev || (!nodes_dev && node_count))
        return fail(AG_ERR_VALUE, "ag_sample_hop_reservoir: null argument");
    if (fanout == 0) return fail(AG_ERR_VALUE, "fanout must be >= 1");
    if (node_count == 0) return AG_OK;
    DeviceGuard guard(g->device);
    if (!guard.ok) return AG_ERR_CUDA;
    // A row per warp up to twice what fills the GPU (8 blocks of 8 warps per SM), four beyond: 15 K
    // rows of 1500 neighbours 42 us, 57 with four; 100 K rows of 10 neighbours 36 us, 31 with four.
    const uint32_t round = fanout > 32 || node_count <= (uint64_t)kSMs * 128 ? kHopThreads / 32 : kHopRows;
    const uint64_t blocks = std::min<uint64_t>((node_count + round - 1) / round, (uint64_t)kSMs * 32);
    if (fanout > 32)
        k_hop_replace<<<(uint32_t)blocks, kHopThreads, 0, (cudaStream_t)stream>>>(
            g->offsets, g->dst, g->num_nodes, g->num_edges, nodes_dev, neighbors_out_dev, counts_out_dev, node_count, fanout, seed, layer);
    else
        k_hop_reservoir<<<(uint32_t)blocks, kHopThreads, 0, (cudaStream_t)stream>>>(
            g->offsets, g->dst, g->num_nodes, g->num_edges, nodes_dev, neighbors_out_dev, counts_out_dev, node_count, fanout, seed,
            layer, round);
    AG_CUDA(cudaGetLastError());
    return AG_OK;
}
