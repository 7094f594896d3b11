// Homogeneous k-hop neighbor sampler with frontier dedup and relabel.
//
// Computes exactly what the reference's NeighborSampler::sample computes
// (crates/aethergraph-core/src/loader/sampler.rs:845-961 with the hop loop at
// :754-842 and the per-node dispatch at :1178-1235), but as a short chain of
// data-parallel kernels instead of one sequential loop.  A batch with H hops
// is 2H + 1 launches (2H + 2 with more than kFusedSeeds seeds):
//
//   insert_seeds   every seed is inserted into a hash table keyed by vertex id
//                  with atomicMin(position): the smallest position that names a
//                  vertex is its first sighting.  A batch of few seeds does this
//                  at the head of assign(0).
//   assign(s)      s = 0 .. H.  The items of stage s are the seeds (s = 0) or
//                  the edges hop s - 1 emitted, in position order.  One
//                  single-pass scan over them turns the first-sighting flags
//                  into local ids (= discovery order, exactly the order the
//                  sequential reference assigns them in) and appends the new
//                  vertices to `nodes`; the same scan carries how many edges and
//                  how many RNG draws each new vertex needs at hop s, so the new
//                  vertices leave the kernel as a frontier with their row
//                  bounds, edge slots and draw offsets attached.
//   pick(s)        s = 0 .. H - 1.  A group of lanes per frontier vertex
//                  reproduces the reference's choice of row positions — take-all
//                  (:1312-1328), Floyd (:1332-1380), with replacement
//                  (:1289-1308) or the weighted Efraimidis-Spirakis keys
//                  (:1418-1469) — writes the edges of hop s at their scanned
//                  slots and inserts the destinations into the table as the
//                  items of stage s + 1.
//                  Every item also learns its vertex's final local id here (its own
//                  if it is the first sighting, else the one the first sighting got,
//                  for which it may have to wait a moment), so dst_local / seed_locals
//                  and the int64 views the Python API exposes are written by the same
//                  kernel; the block that finishes last in the last stage writes the
//                  batch's counts.
//
// The reference draws from one sequential WyRand stream per batch.  WyRand's
// state is an additive counter, so draw d is a pure function of (seed, d); the
// scan of per-vertex draw counts gives every vertex the index of its first
// draw, and the parallel picks are bit-identical to the sequential ones.
//
// Batches are independent, so one launch chain serves a whole GROUP of them:
// every kernel's grid has the batch as its y dimension and each batch brings
// its own parameter block, dedup table, scan descriptors and output buffers.
// A group of 16 batches of 1024 seeds costs the same few launches as one.
#include <string.h>

#include <algorithm>
#include <string>
#include <type_traits>
#include <vector>

#include <sched.h>

#include "common.cuh"
#include "internal.h"
#include "sampler.cuh"

namespace ag {

namespace {

constexpr int kTile = 512;      // threads per block of the assign kernel
// Most items per thread of the assign kernel.  The last stage holds no row bounds per item,
// so it can afford twice as many table probes in flight per thread.
constexpr int kMaxIPT = 4, kMaxIPTLast = 8;
constexpr int kPickThreads = 256;
constexpr int kLargeK = 1024;   // largest fanout the k > 32 path keeps in shared memory

enum : int { kModeUniform = 0, kModeReplace = 1, kModeWeighted = 2, kModeWeightedReplace = 3 };
enum : int { kPickSmall = 0, kPickLarge = 1, kPickWeighted = 2 };

// A long row of a weighted hop, split into n_slices slices (0: it did not fit the queue).
struct __align__(16) HubRow {
    uint32_t batch, vertex;  // position in the batch's frontier
    uint32_t slice_base, n_slices;
};

// Parameter block of one batch; a group's blocks sit in one device array that
// the kernels index with blockIdx.y.
struct SampleParams {
    const uint64_t *offsets;
    const uint32_t *dst;
    const float *weights;
    uint64_t num_nodes, num_edges;
    DedupTable table;
    BatchState *state;
    TileDesc *tiles;
    uint32_t epoch_base;  // stage s scans under epoch_base + s
    uint32_t n_seeds;
    const uint32_t *seeds;
    uint64_t seed;
    int rng_mode;
    int mode;
    uint64_t start_draw;  // absolute index of the batch's first RNG draw (0 for a freshly seeded batch)
    uint32_t num_hops;
    // outputs
    uint32_t *nodes;
    uint32_t *edge_src, *edge_dst, *src_local, *dst_local, *seed_locals;
    uint64_t *edge_ids;
    uint64_t cap_nodes, cap_edges;
    int64_t *n_id, *edge_index_local, *e_id, *seed_index;
    ag_sample_counts *counts;
    // scratch
    uint32_t *slot_of_seed;
    uint32_t *slot_of_edge;
    FrontierEntry *frontier;
    uint64_t frontier_cap;
    // weighted only, shared by the batches of a chain: the rows left to k_pick_hub_slices
    // rows, thresholds and done counts twice: [0] the hop's rows, [1] those whose guess was too low
    HubRow *hub_rows;                // [2][hub_cap]
    unsigned long long *hub_count;   // [2] rows queued << 32 | slices handed out
    uint32_t *hub_thr, *hub_done;    // [2][hub_cap] per row: lowest k-th best key so far (float bits), slices finished
    float *hub_guess;                // [hub_cap] the threshold the row started with
    double *hub_key;                 // [hub_cap][k] the slices' best (key, position) pairs
    uint32_t *hub_pos;
    uint32_t hub_cap, hub_slice;     // slices the arrays hold, positions per slice
    uint32_t alone, pad;             // no other chain runs beside this one (chain_release)
};

// Row bounds with the reference's guard (graph/csr.rs:318-335): an inverted
// pair or one past num_edges is an empty row.
__device__ __forceinline__ void row_bounds(const uint64_t *offsets, uint64_t num_nodes,
                                           uint64_t num_edges, uint32_t id, uint64_t &off,
                                           uint64_t &deg) {
    off = 0; deg = 0;
    if ((uint64_t)id >= num_nodes) return;
    const uint64_t a = __ldg(offsets + id), b = __ldg(offsets + id + 1);
    if (a > b || b > num_edges) return;
    off = a; deg = b - a;
}

// How many edges and draws a row of `deg` asks for at fanout k
// (sampler.rs:1226-1233 uniform, :1289-1308 replace, :1427-1457 weighted).
__device__ __forceinline__ void row_demand(int mode, uint64_t deg, uint32_t k, uint32_t &take,
                                           uint64_t &draws) {
    take = 0; draws = 0;
    if (deg == 0 || k == 0) return;
    if (mode == kModeReplace || mode == kModeWeightedReplace) { take = k; draws = k; return; }
    if ((uint64_t)k >= deg) { take = (uint32_t)deg; return; }
    take = k;
    draws = (mode == kModeWeighted) ? deg : (uint64_t)k;
}

// ------------------------------------------------------------ seed insert --
// Where the parts of a chain's staged block are.  Order: parameter blocks, gather
// arguments (if any), seeds (if the caller's are in host memory).
struct StageLayout {
    SampleParams *params_dev;          // the device copies
    GatherArgs *gather_dev;            // null: nothing to gather
    uint32_t seeds_at, seed_stride;    // first word of the seeds (0: in device memory already), seeds reserved per batch
};
static_assert(sizeof(SampleParams) % 8 == 0 && sizeof(GatherArgs) % 8 == 0, "staged blocks are made of 8-byte words");

__device__ __forceinline__ uint32_t insert_seed(const SampleParams &p, uint32_t i, uint32_t id) {
    if ((uint64_t)id >= p.num_nodes) {
        atomicOr(&p.state->error, kErrBadSeed);
        return 0xFFFFFFFFu;
    }
    return table_insert_min(p.table, id, enc_pending(p.table.gen, 0, i), &p.state->error);
}

__global__ void k_insert_seeds(const SampleParams *__restrict__ pa) {
    const SampleParams &p = pa[blockIdx.y];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.n_seeds) p.slot_of_seed[i] = insert_seed(p, i, p.seeds[i]);
}

// ----------------------------------------------------------------- expand --
__device__ __forceinline__ uint32_t draw_u32(const SampleParams &p, uint32_t hop, uint32_t vertex,
                                             uint64_t dbase, uint32_t slot) {
    if (p.rng_mode == AG_RNG_PHILOX) return philox_u32(p.seed, hop, vertex, slot);
    return (uint32_t)wyrand_at(p.seed, dbase + slot);  // next_u32: genstamp.rs:199-201
}

// Edge t of vertex fe at hop `hop` (= item fe.ebase + t of stage hop + 1), its
// destination d already loaded from CSR position pos.
__device__ __forceinline__ void emit_edge_loaded(const SampleParams &p, uint32_t hop, uint32_t edges_before,
                                                 const FrontierEntry &fe, uint32_t t, uint64_t pos, uint32_t d) {
    const uint32_t e_rel = fe.ebase + t;
    const uint64_t e = (uint64_t)edges_before + e_rel;
    if (e >= p.cap_edges || e_rel >= kMaxPos) { atomicOr(&p.state->error, kErrCapacity); return; }
    if (p.edge_src) p.edge_src[e] = fe.id;
    p.edge_dst[e] = d;
    if (p.edge_ids) p.edge_ids[e] = pos;
    if (p.e_id && p.edge_ids) p.e_id[e] = (int64_t)pos;
    p.src_local[e] = fe.local;
    if ((uint64_t)d >= p.num_nodes) {
        // Only reachable on a graph that skipped validation; the reference drops
        // such an edge (sampler.rs:736-739), which a slot-scanned layout cannot.
        atomicOr(&p.state->error, kErrBadDst);
        p.slot_of_edge[e] = 0xFFFFFFFFu;
        return;
    }
    p.slot_of_edge[e] = table_insert_min(p.table, d, enc_pending(p.table.gen, hop + 1, e_rel), &p.state->error);
}

__device__ __forceinline__ void emit_edge(const SampleParams &p, uint32_t hop, uint32_t edges_before,
                                          const FrontierEntry &fe, uint32_t t, uint64_t pos) {
    const uint32_t e_rel = fe.ebase + t;
    if ((uint64_t)edges_before + e_rel >= p.cap_edges || e_rel >= kMaxPos) { atomicOr(&p.state->error, kErrCapacity); return; }
    emit_edge_loaded(p, hop, edges_before, fe, t, pos, ld_stream_u32(p.dst + pos));
}

__device__ __forceinline__ bool key_less(double ka, uint32_t pa, double kb, uint32_t pb) {
    return ka < kb || (ka == kb && pa < pb);
}

// Fanout <= G <= 32: G lanes per vertex, lane t owns edge slot t.  A lane group works
// on two vertices per round, so the two destination loads (random sectors of the CSR)
// and the table probes behind them are in flight together.
template <int G>
__device__ __forceinline__ void pick_small(const SampleParams &p, uint32_t hop, uint32_t k, uint32_t edges_before,
                                           const FrontierEntry *fes, uint32_t n) {
    constexpr int U = 2;
    const uint32_t t = threadIdx.x % G;
    const uint32_t gshift = (threadIdx.x & 31) & ~(G - 1);
    const uint32_t gmask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u);
    constexpr uint32_t kPerBlock = kPickThreads / G;
    // Grid-stride over the frontier; the loop bound is block-uniform.
    for (uint32_t base = blockIdx.x * kPerBlock * U; base < n; base += gridDim.x * kPerBlock * U) {
        FrontierEntry fe[U];
        uint32_t pick[U];
        bool emit[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t j = base + u * kPerBlock + threadIdx.x / G;
            const bool active = j < n;
            fe[u] = FrontierEntry{};
            if (active) fe[u] = fes[j];
            const uint32_t deg = fe[u].deg;
            const bool sampled = active && p.mode != kModeReplace && deg > k;  // Floyd row
            pick[u] = t;                                                         // take-all: row order
            uint32_t ip = 0;
            if (active && p.mode == kModeReplace && deg > 0 && t < k) {
                // sampler.rs:1298-1300: k independent draws over the whole row
                pick[u] = (uint32_t)(((uint64_t)draw_u32(p, hop, fe[u].id, fe[u].dbase, t) * deg) >> 32);
            } else if (sampled && t < k) {
                // sampler.rs:1345-1346: i runs over deg-k .. deg-1, j = rand_below(i + 1)
                ip = deg - k + t;
                pick[u] = (uint32_t)(((uint64_t)draw_u32(p, hop, fe[u].id, fe[u].dbase, t) * ((uint64_t)ip + 1)) >> 32);
            }
            // Floyd's "already taken?" is sequential in t (sampler.rs:1347-1352):
            // resolve slot s against the finished slots below it, one ballot per s.
            if (__any_sync(0xffffffffu, sampled)) {
                for (uint32_t s = 1; s < k; ++s) {
                    const uint32_t js = __shfl_sync(0xffffffffu, pick[u], s, G);
                    const bool hit = sampled && t < s && pick[u] == js;
                    const uint32_t m = (__ballot_sync(0xffffffffu, hit) >> gshift) & gmask;
                    if (sampled && t == s && m) pick[u] = ip;
                }
            }
            uint32_t take = 0;
            uint64_t draws;
            if (active) row_demand(p.mode, deg, k, take, draws);
            emit[u] = t < take;
        }
        uint32_t d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) d[u] = emit[u] ? ld_stream_u32(p.dst + fe[u].off + pick[u]) : 0u;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (emit[u]) emit_edge_loaded(p, hop, edges_before, fe[u], t, fe[u].off + pick[u], d[u]);
    }
}

// Fanout > 32: one warp per vertex (four warps per block); finished picks live
// in shared memory so later slots can be checked against all earlier ones.
__device__ __forceinline__ void pick_large(const SampleParams &p, uint32_t hop, uint32_t k, uint32_t edges_before,
                                           const FrontierEntry *fes, uint32_t n, uint32_t *s_picks) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *picks = s_picks + warp * kLargeK;
    for (uint32_t j = blockIdx.x * 4 + warp; j < n; j += gridDim.x * 4) {
        const FrontierEntry fe = fes[j];
        const uint32_t deg = fe.deg;
        uint32_t take;
        uint64_t draws;
        row_demand(p.mode, deg, k, take, draws);
        const bool sampled = p.mode != kModeReplace && deg > k;
        __syncwarp();
        for (uint32_t c = 0; c < take; c += 32) {
            const uint32_t t = c + lane;
            const bool in = t < take;
            uint32_t pick = t, ip = 0;
            bool hit_prev = false;
            if (in && p.mode == kModeReplace) {
                pick = (uint32_t)(((uint64_t)draw_u32(p, hop, fe.id, fe.dbase, t) * deg) >> 32);
            } else if (in && sampled) {
                ip = deg - k + t;
                pick = (uint32_t)(((uint64_t)draw_u32(p, hop, fe.id, fe.dbase, t) * ((uint64_t)ip + 1)) >> 32);
                for (uint32_t q = 0; q < c; ++q) hit_prev |= (picks[q] == pick);
            }
            if (sampled) {
                for (uint32_t s = 0; s < 32; ++s) {
                    const uint32_t js = __shfl_sync(0xffffffffu, pick, s);
                    const bool hit = in && (uint32_t)lane < s && pick == js;
                    const uint32_t m = __ballot_sync(0xffffffffu, hit);
                    if (in && (uint32_t)lane == s && (m || hit_prev)) pick = ip;
                }
                if (in) picks[t] = pick;
                __syncwarp();
            }
            if (in) emit_edge(p, hop, edges_before, fe, t, fe.off + pick);
        }
    }
}

// Weighted sampling without replacement, fanout <= 32, one warp per vertex or slice of its row.
// Selection follows sampler.rs:1418-1469: one 64-bit draw per row position in
// row order, key = -ln(u) / w in f64 with u = ((bits >> 11) + 1) * 2^-53
// (sampler.rs:52-55), +inf for a weight that is not finite and positive; the k
// smallest keys win.  The winners are emitted in ascending (key, position)
// order; the reference's own order comes from Rust's select_nth_unstable_by and
// is not defined by its source tree.  The warp streams the row 32 positions at a
// time and keeps the k best so far sorted across its lanes.

// Compare-exchange with the lane `stride` away; this lane keeps the smaller pair if `small`.
__device__ __forceinline__ void warp_exchange(double &key, uint32_t &pos, int stride, bool small) {
    const double ok = __shfl_xor_sync(0xffffffffu, key, stride);
    const uint32_t op = __shfl_xor_sync(0xffffffffu, pos, stride);
    if (key_less(ok, op, key, pos) == small) { key = ok; pos = op; }
}

// Sorts the warp's 32 (key, position) pairs ascending across the lanes (bitonic).
__device__ __forceinline__ void warp_sort_pairs(double &key, uint32_t &pos, int lane) {
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1)
            warp_exchange(key, pos, stride, ((lane & size) == 0) == ((lane & stride) == 0));
    }
}

constexpr int kInsertFew = 6;  // winners inserted one by one (about 35 instructions each)

// Inserts the chunk's candidates (one per lane, cpos == ~0 for none) that beat the
// current k-th best into the sorted lanes.
__device__ __forceinline__ void topk_insert_chunk(double key, uint32_t cpos, double &best_key, uint32_t &best_pos,
                                                  uint32_t k, int lane) {
    for (bool again = false;; again = true) {
        const double tk = __shfl_sync(0xffffffffu, best_key, k - 1);
        const uint32_t tp = __shfl_sync(0xffffffffu, best_pos, k - 1);
        const uint32_t m = __ballot_sync(0xffffffffu, cpos != 0xFFFFFFFFu && key_less(key, cpos, tk, tp));
        if (!m) break;
        if (!again && __popc(m) > kInsertFew) {
            // Many: sort them, keep the smaller of best[i] and candidate[31 - i] (the 32 smallest
            // of the 64, a bitonic sequence) and sort that: 21 exchange steps.
            warp_sort_pairs(key, cpos, lane);
            const double rk = __shfl_sync(0xffffffffu, key, 31 - lane);
            const uint32_t rp = __shfl_sync(0xffffffffu, cpos, 31 - lane);
            if (key_less(rk, rp, best_key, best_pos)) { best_key = rk; best_pos = rp; }
#pragma unroll
            for (int stride = 16; stride > 0; stride >>= 1) warp_exchange(best_key, best_pos, stride, (lane & stride) == 0);
            break;
        }
        const int src = __ffs(m) - 1;
        const double ck = __shfl_sync(0xffffffffu, key, src);
        const uint32_t cp = __shfl_sync(0xffffffffu, cpos, src);
        // (ck, cp) lands after every entry that is smaller, the rest shift up by one.
        const uint32_t smaller = __ballot_sync(0xffffffffu, key_less(best_key, best_pos, ck, cp));
        const int at = __popc(smaller);
        const double up_k = __shfl_up_sync(0xffffffffu, best_key, 1);
        const uint32_t up_p = __shfl_up_sync(0xffffffffu, best_pos, 1);
        if (lane == at) { best_key = ck; best_pos = cp; }
        else if (lane > at) { best_key = up_k; best_pos = up_p; }
        if (lane == src) cpos = 0xFFFFFFFFu;
    }
}

// Exact key of position `pos` of the row (sampler.rs:1440-1452): u from the position's
// own draw, key = -ln(u) / w, +inf for a weight that is not a positive finite number.
__device__ __forceinline__ double weighted_key(const SampleParams &p, uint32_t hop, const FrontierEntry &fe, uint32_t pos) {
    const uint64_t bits = (p.rng_mode == AG_RNG_PHILOX)
        ? (((uint64_t)philox_u32(p.seed, hop, fe.id, 2 * pos) << 32) | philox_u32(p.seed, hop, fe.id, 2 * pos + 1))
        : wyrand_at(p.seed, fe.dbase + pos);
    const double w = (double)__ldg(p.weights + fe.off + pos);
    if (!(isfinite(w) && w > 0.0)) return __longlong_as_double(0x7FF0000000000000ll);
    const double u = ((double)(bits >> 11) + 1.0) * (1.0 / 9007199254740992.0);
    return -log(u) / w;
}

// Streams positions [begin, end) of the row of `fe` into the warp's sorted best k
// (all sentinels on entry).
//
// Almost every position loses against the k-th best key, and the exact key costs an
// f64 log and divide, so the stream works in two stages.  Stage 1, all lanes, single
// precision, no log: with uf >= u (u's top 23 bits, rounded up),
//     -ln(u) >= -ln(uf) >= 2 (1 - uf) / (1 + uf)
// (the first term of the series of ln, all terms positive), tight where it matters: a
// winner of a long row has u near 1.  If 2 (1 - uf) exceeds (1 + uf) * thr * w by more
// than the rounding of the three f32 products (3 * 2^-24 relative, 1e-5 is granted;
// 1 + uf and 1 - uf are exact), the exact key cannot be below the threshold and the
// position is dropped.  A weight that is not positive and finite has key +inf, which a
// finite threshold beats: 0, negative weights and NaN are dropped by the same comparison,
// +inf (and a product that overflows) survives to stage 2.  Survivors are only queued
// (`buf`, kQueue slots of the warp's shared memory).  Stage 2, whenever 32 are queued: every
// lane evaluates one queued position exactly and the winners are inserted.
//
// Without a threshold the first 32 positions are evaluated at once, which holds k of them.
// If the k-th best key is still +inf then, a later position whose key is +inf as well comes
// after the k held (equal keys go by position), so weights that are not positive can be
// dropped from there on: the factor +inf keeps exactly the positive ones.
//
// The threshold is the lowest of `guess`, the k-th best key at the last flush and, when
// several warps stream slices of one row, `shared_thr`, the lowest k-th best any of them
// holds (the bit pattern of a non-negative float orders like the float).  Without the
// guess (+inf) it is always an upper bound of the row's final k-th best key, so stage 1
// only ever discards certain losers and the output is exactly that of evaluating every
// position.  With a guess the same holds if the k-th best found is at most the guess;
// the caller checks that and streams again without one if not.
//
// Bound: instructions, about 30 for 32 positions in stage 1 and 500 for a flush, so what
// counts is the multiply of the random stream (wyrand_top32) and the number of flushes
// (guess_threshold, and the first chunk on its own where there is no threshold).  One place
// in the code flushes: with three inlined copies the kernels spill.  kChunks * 32 positions are loaded and filtered together and only
// then asked for survivors, with one vote, while the next ones are loaded.
constexpr uint32_t kChunks = 4;
constexpr uint32_t kQueue = 32 + 32 * kChunks;  // what a flush leaves (fewer than 32) and one round's survivors

template <bool PHILOX>
__device__ __forceinline__ void topk_stream_rng(const SampleParams &p, uint32_t hop, const FrontierEntry &fe, uint32_t begin,
                                                uint32_t end, uint32_t k, int lane, double &best_key, uint32_t &best_pos,
                                                uint32_t *buf, float guess, uint32_t *shared_thr) {
    uint32_t queued = 0;  // warp-uniform
    bool fresh = true;    // nothing inserted yet
    float thr = guess;
    auto threshold = [&] { return shared_thr ? fminf(thr, __uint_as_float(__ldcg(shared_thr))) : thr; };
    const float *w = p.weights + fe.off + begin + lane;
    constexpr uint64_t kStep = 0xa0761d6478bd642full;  // from one draw's state to the next (wyrand_at)
    const uint64_t seed = p.seed;
    uint32_t first = begin + lane;  // this lane's position in the next chunk
    uint64_t state = seed + (fe.dbase + first + 1ull) * kStep;
    float wf[kChunks];  // the weights of the next kChunks * 32 positions; past the end: negative, dropped
#pragma unroll
    for (uint32_t u = 0; u < kChunks; ++u) wf[u] = u * 32 + lane < end - begin ? __ldg(w + u * 32) : -1.0f;
    uint32_t left = end - begin;
    __syncwarp();  // the queue may have been another stream's
    if (!(__shfl_sync(0xffffffffu, threshold(), 0) <= 3.0e38f)) {  // no threshold: the first chunk as it is
        buf[lane] = first;
        queued = min(32u, left);
        wf[0] = -1.0f;
    }
    for (bool drain = queued > 0;;) {
        // evaluate 32 queued positions exactly, one per lane, and insert the winners
        while (queued >= 32 || (drain && queued > 0)) {
            const uint32_t count = min(queued, 32u);
            queued -= count;
            __syncwarp();
            double key = __longlong_as_double(0x7FF0000000000000ll);
            uint32_t cpos = 0xFFFFFFFFu;
            if ((uint32_t)lane < count) {
                cpos = buf[queued + lane];
                key = weighted_key(p, hop, fe, cpos);
            }
            if (fresh) {
                warp_sort_pairs(key, cpos, lane);
                best_key = key; best_pos = cpos;
                fresh = false;
            } else {
                topk_insert_chunk(key, cpos, best_key, best_pos, k, lane);
            }
            const double kth = __shfl_sync(0xffffffffu, best_key, k - 1);
            thr = fminf(thr, (float)kth);
            if (shared_thr) {
                const float up = __double2float_ru(kth);  // rounded up: still an upper bound
                if (lane == 0 && up < 3.0e38f) atomicMin(shared_thr, __float_as_uint(up));
            }
        }
        if (left == 0) break;
        // those after them are on their way while these are filtered
        float ahead[kChunks];
#pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u)
            ahead[u] = left > 32 * kChunks && u * 32 + lane < left - 32 * kChunks ? __ldg(w + 32 * kChunks + u * 32) : -1.0f;
        const float t = threshold();
        const float ts = (t >= 1.0e-30f && t <= 3.0e38f) ? t * 1.00001f : __uint_as_float(0x7F800000u);
        bool kept[kChunks], any = false;
#pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u) {
            const uint32_t top = PHILOX ? philox_u32(seed, hop, fe.id, 2 * (first + u * 32))
                                        : wyrand_top32(state + u * 32 * kStep);
            const float above = __uint_as_float(0x3F800000u | (top >> 9)) + 1.1920928955078125e-07f;  // 1 + uf
            const float below = 2.0f - above;                                                           // 1 - uf
            kept[u] = 2.0f * below <= above * (ts * wf[u]);
            any = any || kept[u];
        }
        if (__any_sync(0xffffffffu, any)) {
            __syncwarp();  // the queue's last reads are done
#pragma unroll
            for (uint32_t u = 0; u < kChunks; ++u) {
                const uint32_t m = __ballot_sync(0xffffffffu, kept[u]);
                if (kept[u]) buf[queued + __popc(m & ((1u << lane) - 1u))] = first + u * 32;
                queued += __popc(m);
            }
        }
        w += 32 * kChunks;
        first += 32 * kChunks;
        state += 32 * kChunks * kStep;
#pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u) wf[u] = ahead[u];
        left -= min(left, 32 * kChunks);
        drain = left == 0;
    }
}

__device__ __forceinline__ void topk_stream(const SampleParams &p, uint32_t hop, const FrontierEntry &fe, uint32_t begin,
                                            uint32_t end, uint32_t k, int lane, double &best_key, uint32_t &best_pos,
                                            uint32_t *buf, float guess, uint32_t *shared_thr = nullptr) {
    best_key = __longlong_as_double(0x7FF0000000000000ll);
    best_pos = 0xFFFFFFFFu;  // sentinel: sorts after every real (key, position)
    if (p.rng_mode == AG_RNG_PHILOX) topk_stream_rng<true>(p, hop, fe, begin, end, k, lane, best_key, best_pos, buf, guess, shared_thr);
    else topk_stream_rng<false>(p, hop, fe, begin, end, k, lane, best_key, best_pos, buf, guess, shared_thr);
}

// A threshold that about `want` of a row's `n` keys should fall below, given its positive
// weights' mean: keys are exponential with rate w, so n (1 - exp(-t mean)) = want for equal
// weights.  A hint only (see topk_stream): without one the threshold starts at +inf and
// comes down flush by flush, four or five of them in a row of 500.
__device__ __forceinline__ float guess_threshold(float mean, float n, float want) {
    const float t = -__logf(1.0f - want / n) / mean;
    return (want < 0.75f * n && t > 1.0e-30f && t < 3.0e38f) ? t : __uint_as_float(0x7F800000u);
}

// A lane's share of a row's weight above which the row counts as skewed, in means.  Weights of
// one size stay below, log-normal ones of sigma 1 nearly always.  Eight batches of 1024 seeds,
// fanouts 15, 10, rows of 128 to 2048 positions: Pareto weights (exponent 1/2) 765 us, 1810
// from the mean alone (most rows streamed twice); log-normal 655.
constexpr float kSkew = 6.0f;

// Sum of `count` weights of a row, `step` apart, that are positive and finite (warp-wide).
// *skewed: a lane's share is far from the others', so the mean says little about the keys.
__device__ __forceinline__ float weight_sum(const float *w, uint32_t count, uint64_t step, int lane, bool *skewed) {
    float sum = 0.0f;
    for (uint32_t c = 0; c < count; c += 32 * kChunks) {
        float v[kChunks];
#pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u) {
            const uint32_t i = c + u * 32 + lane;
            v[u] = i < count ? __ldg(w + i * step) : 0.0f;
        }
#pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u) sum += (v[u] > 0.0f && v[u] < 3.0e38f) ? v[u] : 0.0f;
    }
    const float share = sum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    *skewed = __any_sync(0xffffffffu, !(share > 0.0f && share * 32.0f < sum * kSkew));
    return sum;
}

// The threshold for a skewed row: of the sampled weights about `target` keys should fall below
// t.  A key does with probability 1 - exp(-t w), bounded by min(t w, 1); the sum of the bounds
// is concave in t and linear between the places where a weight reaches 1, so from the left
// Newton's steps approach the place where it is `target`, and a third more makes up for the
// bound.  +inf if fewer weights than that are positive.
__device__ __forceinline__ float skewed_threshold(const float *w, uint32_t count, uint64_t step, float t, float target, int lane) {
    const float inff = __uint_as_float(0x7F800000u);
    if (!(t < 3.0e38f)) return inff;
    for (int round = 0; round < 12; ++round) {
        float rest = 0.0f, full = 0.0f;  // weights with t w < 1, number of the others
        for (uint32_t i = lane; i < count; i += 32) {
            const float v = __ldg(w + i * step);
            if (!(v > 0.0f && v < 3.0e38f)) continue;
            if (t * v < 1.0f) rest += v; else full += 1.0f;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            rest += __shfl_xor_sync(0xffffffffu, rest, o);
            full += __shfl_xor_sync(0xffffffffu, full, o);
        }
        if (full >= target) break;
        if (!(rest > 0.0f)) return inff;
        const float next = (target - full) / rest;
        if (!(next > 1.05f * t)) break;
        t = next;
    }
    t *= 1.33f;
    return t > 1.0e-30f && t < 3.0e38f ? t : inff;
}

// Warps per block of the weighted picks: few, so that a block's slots are free again as
// soon as its own rows are done (rows of a hop differ by a factor of 2000).
constexpr int kWeightedThreads = 64;

// Rows longer than kHubDegree are split into slices, a warp each, by k_pick_hub_slices;
// a warp alone takes about 1 us per 1000 positions, so the rows left to one warp end
// together with the rest of the hop.
constexpr uint32_t kHubDegree = 2048;
constexpr uint32_t kMaxHubSlices = 65536;   // slices a chain's queue holds; a row that does not fit stays with its warp
constexpr uint32_t kMaxSlicesPerRow = 256;  // the merge of a row is one warp's work
constexpr uint32_t kGuessDegree = 128;      // rows from here on get a threshold to start with
constexpr uint32_t kSampledWeights = 512;   // weights, evenly spaced, that a row's mean is taken from

__device__ __forceinline__ uint32_t hub_slice_len(uint32_t deg, uint32_t slice) {
    return max(slice, (deg / kMaxSlicesPerRow + 32u) & ~31u);
}

// Queues a long row for k_pick_hub_slices<again> with a threshold to start from; false if its
// slices do not fit the queue.  Warp-wide.
__device__ __forceinline__ bool queue_long_row(const SampleParams &p, uint32_t again, uint32_t batch, uint32_t vertex, uint32_t deg,
                                               float thr, int lane) {
    bool queued = false;
    if (lane == 0) {
        const uint32_t len = hub_slice_len(deg, again ? kHubDegree : p.hub_slice), slices = (deg - 1) / len + 1;
        // one atomic for both counters: the rows' slice ranges ascend in queue order
        const unsigned long long at = atomicAdd(p.hub_count + again, (1ull << 32) | slices);
        const uint32_t h = (uint32_t)(at >> 32), base = (uint32_t)at;
        queued = (uint64_t)base + slices <= p.hub_cap;
        if (h < p.hub_cap) {
            const uint32_t to = again * p.hub_cap + h;
            p.hub_rows[to] = HubRow{batch, vertex, base, queued ? slices : 0u};
            p.hub_thr[to] = __float_as_uint(thr);
            p.hub_done[to] = 0;
            if (!again) p.hub_guess[h] = thr;
        }
    }
    return __shfl_sync(0xffffffffu, queued, 0);
}

__device__ __forceinline__ void pick_weighted(const SampleParams &p, uint32_t hop, uint32_t k, uint32_t edges_before,
                                              const FrontierEntry *fes, uint32_t n, uint32_t *queue) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k == 0) return;
    for (uint32_t j = blockIdx.x * (kWeightedThreads / 32) + warp; j < n; j += gridDim.x * (kWeightedThreads / 32)) {
        const FrontierEntry fe = fes[j];
        const uint32_t deg = fe.deg;
        if (deg == 0) continue;
        if (k >= deg) {
            for (uint32_t t = lane; t < deg; t += 32) emit_edge(p, hop, edges_before, fe, t, fe.off + t);
            continue;
        }
        if (deg > kHubDegree) {  // queue the row for the slice kernel
            // Many more than k: a wrong guess costs the whole row again.
            bool skewed;
            const float guess = guess_threshold(weight_sum(p.weights + fe.off, kSampledWeights, deg / kSampledWeights, lane, &skewed) / kSampledWeights,
                                                (float)deg, 4.0f * (float)k + 64.0f);
            if (queue_long_row(p, 0, blockIdx.y, j, deg, guess, lane)) continue;
        }
        const float inff = __uint_as_float(0x7F800000u);
        float guess = inff;
        if (deg >= kGuessDegree) {
            // enough to be right nineteen times in twenty or better, few enough for one flush
            const float want = (float)k + 2.0f * sqrtf((float)k) + 2.0f;
            const uint32_t count = min(deg, kSampledWeights), step = deg > kSampledWeights ? deg / kSampledWeights : 1;
            const float *w = p.weights + fe.off;
            bool skewed;
            guess = guess_threshold(weight_sum(w, count, step, lane, &skewed) / (float)count, (float)deg, want);
            if (skewed) guess = skewed_threshold(w, count, step, guess, want * ((float)count / (float)deg), lane);
        }
        double best_key;
        uint32_t best_pos;
        for (;; guess = inff) {  // again without the guess if it was too low
            topk_stream(p, hop, fe, 0, deg, k, lane, best_key, best_pos, queue + warp * kQueue, guess);
            if (__shfl_sync(0xffffffffu, best_key, k - 1) <= (double)guess) break;
        }
        if ((uint32_t)lane < k) emit_edge(p, hop, edges_before, fe, lane, fe.off + best_pos);
    }
}

// One stage: assign local ids to the first sightings among the stage's items
// and (has_next) queue the new vertices, with their row bounds, edge slots and
// draw offsets, as the frontier the pick kernel of hop `stage` expands.  Every
// item also writes the final local id of its vertex (dst_local / seed_locals and
// the int64 views): its own if it is the first sighting, the one already in the
// table if the vertex was registered by an earlier stage, and otherwise the one
// an earlier item of this stage is about to store — a short, bounded wait that is
// taken only after the block has passed its next barrier, so a block never waits
// for a store of its own.
__device__ __forceinline__ StageInfo load_stage_cg(const StageInfo *s) {
    // other blocks of this launch wrote it: read it from L2, not from a stale L1 line
    const uint4 a = __ldcg((const uint4 *)s), b = __ldcg((const uint4 *)s + 1);
    StageInfo r;
    r.n_nodes = a.x; r.n_edges = a.y; r.frontier_n = a.z; r.hop_edges = a.w;
    r.draws = ((uint64_t)b.y << 32) | b.x; r.hop_draws = ((uint64_t)b.w << 32) | b.z;
    return r;
}

__device__ __forceinline__ void write_item_local(const SampleParams &p, uint32_t stage, uint32_t n_edges_before,
                                                 uint32_t item, uint32_t local) {
    if (stage == 0) {
        p.seed_locals[item] = local;
        if (p.seed_index) p.seed_index[item] = (int64_t)local;
    } else {
        const uint64_t e = (uint64_t)n_edges_before + item;
        if (e >= p.cap_edges) return;
        p.dst_local[e] = local;
        if (p.edge_index_local) p.edge_index_local[e] = (int64_t)local;  // row 0: sampled neighbor
    }
}

// Weighted picks with replacement (sampler.rs:1383-1412): the reference sums the row's
// weights in f64 in row order, draws u = next_u64 * (total / u64::MAX) k times and takes,
// for each draw, the first position whose running sum exceeds u.  The running sums must
// be the reference's own, rounding included, so every lane of the warp that owns the row
// adds the weights in the same row order (redundantly: the loads are warp-wide
// broadcasts) — once for the total, once more to place its own draw.  Lane t owns draw t
// of the current round of 32.
__global__ void __launch_bounds__(kPickThreads)
k_pick_weighted_replace(const SampleParams *pa, uint32_t hop, uint32_t k) {
    __shared__ __align__(16) SampleParams s_params;
    chain_sync();
    const SampleParams &p = chain_block(pa + blockIdx.y, s_params);
    chain_release(p.alone);
    const StageInfo nx = p.state->stage[hop + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t j = blockIdx.x * (kPickThreads / 32) + warp; j < nx.frontier_n; j += gridDim.x * (kPickThreads / 32)) {
        const FrontierEntry fe = p.frontier[j];
        const uint32_t deg = fe.deg;
        if (deg == 0 || k == 0) continue;
        const float *w = p.weights + fe.off;
        double total = 0.0;
        for (uint32_t i = 0; i < deg; ++i) total += (double)__ldg(w + i);
        const double scale = total / 18446744073709551615.0;  // u64::MAX as f64
        for (uint32_t t0 = 0; t0 < k; t0 += 32) {
            const uint32_t t = t0 + lane;
            const bool mine = t < k;
            const uint64_t bits = (p.rng_mode == AG_RNG_PHILOX)
                ? (((uint64_t)philox_u32(p.seed, hop, fe.id, 2 * t) << 32) | philox_u32(p.seed, hop, fe.id, 2 * t + 1))
                : wyrand_at(p.seed, fe.dbase + t);
            const double u = __ull2double_rn(bits) * scale;
            uint32_t idx = deg - 1;  // partition_point(c <= u) clamped to the last position
            bool placed = !mine;
            double c = 0.0;
            for (uint32_t i = 0; i < deg; ++i) {
                c += (double)__ldg(w + i);
                if (!placed && !(c <= u)) { idx = i; placed = true; }
                if (__all_sync(0xffffffffu, placed)) break;
            }
            if (mine) emit_edge(p, hop, nx.n_edges, fe, t, fe.off + idx);
        }
    }
}

// Weighted picks with a fanout above 32 (up to kLargeK): one block per frontier vertex.
// The block streams the row, every thread evaluating the exact key of one position per
// round (sampler.rs:1440-1452), and collects the positions that beat the current k-th
// best in a shared buffer; when the buffer fills up it is sorted (bitonic, ascending
// (key, position)) and cut back to the best k, which tightens the threshold.  The k
// smallest (key, position) pairs are a property of the row alone, so neither the order
// in which threads append nor the moments of the cuts change the result; the winners
// are emitted in ascending order like the fanout <= 32 path.
constexpr int kWLThreads = 256;
constexpr int kWLBuf = 2048;  // >= kLargeK + kWLThreads

__device__ __forceinline__ void wl_sort(double *key, uint32_t *pos) {  // whole block, kWLBuf entries
    for (uint32_t size = 2; size <= (uint32_t)kWLBuf; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (uint32_t t = threadIdx.x; t < (uint32_t)kWLBuf / 2; t += kWLThreads) {
                const uint32_t lo = 2 * t - (t & (stride - 1));  // index with bit `stride` clear
                const uint32_t hi = lo + stride;
                const bool up = (lo & size) == 0;
                const double ka = key[lo], kb = key[hi];
                const uint32_t pa = pos[lo], pb = pos[hi];
                if (key_less(kb, pb, ka, pa) == up) { key[lo] = kb; pos[lo] = pb; key[hi] = ka; pos[hi] = pa; }
            }
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kWLThreads)
k_pick_weighted_large(const SampleParams *pa, uint32_t hop, uint32_t k) {
    __shared__ double s_key[kWLBuf];
    __shared__ uint32_t s_pos[kWLBuf];
    __shared__ uint32_t s_fill;
    __shared__ __align__(16) SampleParams s_params;
    chain_sync();
    const SampleParams &p = chain_block(pa + blockIdx.y, s_params);
    chain_release(p.alone);
    const StageInfo nx = p.state->stage[hop + 1];
    const double inf = __longlong_as_double(0x7FF0000000000000ll);
    for (uint32_t j = blockIdx.x; j < nx.frontier_n; j += gridDim.x) {
        const FrontierEntry fe = p.frontier[j];
        const uint32_t deg = fe.deg;
        if (deg == 0 || k == 0) continue;
        if (k >= deg) {  // take-all, row order, no draws
            for (uint32_t t = threadIdx.x; t < deg; t += kWLThreads) emit_edge(p, hop, nx.n_edges, fe, t, fe.off + t);
            continue;
        }
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < (uint32_t)kWLBuf; t += kWLThreads) { s_key[t] = inf; s_pos[t] = 0xFFFFFFFFu; }
        if (threadIdx.x == 0) s_fill = 0;
        __syncthreads();
        double thr_key = inf;            // the k-th best so far (block-uniform)
        uint32_t thr_pos = 0xFFFFFFFFu;
        for (uint32_t c = 0; c < deg; c += kWLThreads) {
            const uint32_t pos = c + threadIdx.x;
            if (pos < deg) {
                const double key = weighted_key(p, hop, fe, pos);
                if (key_less(key, pos, thr_key, thr_pos)) {
                    const uint32_t at = atomicAdd(&s_fill, 1u);  // < kWLBuf: at most k + one round are ever held
                    s_key[at] = key; s_pos[at] = pos;
                }
            }
            __syncthreads();
            if (s_fill + kWLThreads > (uint32_t)kWLBuf || c + kWLThreads >= deg) {
                wl_sort(s_key, s_pos);
                const uint32_t keep = min(s_fill, k);
                for (uint32_t t = keep + threadIdx.x; t < (uint32_t)kWLBuf; t += kWLThreads) { s_key[t] = inf; s_pos[t] = 0xFFFFFFFFu; }
                if (keep == k) { thr_key = s_key[k - 1]; thr_pos = s_pos[k - 1]; }
                __syncthreads();
                if (threadIdx.x == 0) s_fill = keep;
                __syncthreads();
            }
        }
        for (uint32_t t = threadIdx.x; t < k; t += kWLThreads) emit_edge(p, hop, nx.n_edges, fe, t, fe.off + s_pos[t]);
    }
}

// Called by one thread once every block of the batch's last kernel has finished.
__device__ __forceinline__ void publish_counts(const SampleParams &p, BatchState *bs) {
    __threadfence();
    const StageInfo fin = load_stage_cg(&bs->stage[p.num_hops + 1]);
    ag_sample_counts c{};
    c.num_nodes = (uint32_t)min((uint64_t)fin.n_nodes, p.cap_nodes);
    c.num_edges = (uint32_t)min((uint64_t)fin.n_edges, p.cap_edges);
    c.num_seeds = p.n_seeds;
    c.num_hops = p.num_hops;
    for (uint32_t st = 0; st <= p.num_hops; ++st) c.nodes_per_hop[st] = __ldcg(&bs->nodes_per_stage[st]);
    for (uint32_t h = 0; h < p.num_hops; ++h) c.edges_per_hop[h] = load_stage_cg(&bs->stage[h + 1]).hop_edges;
    c.draws = fin.draws - load_stage_cg(&bs->stage[0]).draws;
    c.error = atomicOr(&bs->error, 0u);
    if ((uint64_t)fin.n_nodes > p.cap_nodes || (uint64_t)fin.n_edges > p.cap_edges) c.error |= kErrCapacity;
    *p.counts = c;
    bs->stream_pos = fin.draws;  // a bare sampler keeps consuming the same stream
    bs->error = 0;               // ready for the handle's next batch
    bs->ticket = 0;
    bs->done_blocks = 0;
}

// The body of an assign kernel.  FUSED: stage 0 of a batch whose seeds fit one tile; the
// one block inserts the seeds itself and needs neither ticket nor look-back.
template <bool HAS_NEXT, int IPT, bool FUSED>
__device__ __forceinline__ void assign_stage(const SampleParams &p, uint32_t stage, uint32_t k) {
    constexpr bool has_next = HAS_NEXT;  // the last stage queues no frontier
    constexpr int kIPT = IPT, kTileItems = kTile * IPT;
    __shared__ uint32_t s_tile;
    __shared__ ScanVal s_warp[kTile / 32];
    __shared__ ScanVal s_prefix;
    __shared__ uint32_t s_seeds[FUSED ? kTileItems : 1];

    BatchState *bs = p.state;
    StageInfo si = bs->stage[stage];
    if (stage == 0) {
        // A reseeded batch starts its stream at draw 0; otherwise the handle's stream
        // continues where its previous batch stopped (the host keeps that position).
        si = StageInfo{};
        si.draws = p.start_draw;
    }
    const uint32_t count = (stage == 0) ? p.n_seeds : si.hop_edges;
    const uint32_t n_tiles = max(1u, (count + kTileItems - 1) / kTileItems);
    const uint32_t edges_before_next = si.n_edges + ((stage == 0) ? 0u : count);  // where hop `stage` starts
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gen = p.table.gen;
    const uint32_t *slots_in = (stage == 0) ? p.slot_of_seed : p.slot_of_edge + si.n_edges;

    // The grid is sized for a typical batch, not for the worst case: a block
    // keeps drawing tile tickets until they run out.  Tickets are handed out in
    // order, so the tiles a look-back (or a pending vertex) waits for are always
    // already running.  A thread owns kIPT consecutive items of its tile (launch_assign
    // picks kIPT), so that many table probes (and row-bound loads) are in flight per
    // thread, and the barriers, the ticket and the look-back are paid once per
    // kTile * kIPT items.
    for (;;) {
        if (!FUSED) {
            if (threadIdx.x == 0) s_tile = atomicAdd(&bs->ticket, 1u);
            __syncthreads();
        }
        const uint32_t tile = FUSED ? 0u : s_tile;
        if (tile >= n_tiles) {
            // n_tiles + gridDim.x tickets are drawn in all; the last one resets the counter.
            if (threadIdx.x == 0 && tile == n_tiles + gridDim.x - 1) bs->ticket = 0;
            break;
        }
        const uint32_t item0 = tile * kTileItems + threadIdx.x * kIPT;

        // First sighting?  The table holds the pending mark of the smallest
        // position that named the vertex.
        uint32_t slot[kIPT], id[kIPT], cur32[kIPT];
        bool first[kIPT];
        if (FUSED) {
            // a coalesced read of the seeds, then each thread takes its own
#pragma unroll
            for (int j = 0; j < kIPT; ++j) {
                const uint32_t i = threadIdx.x + j * kTile;
                if (i < count) s_seeds[i] = p.seeds[i];
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kIPT; ++j) slot[j] = (item0 + j < count) ? insert_seed(p, item0 + j, s_seeds[item0 + j]) : 0xFFFFFFFFu;
            __threadfence();  // every seed is in the table before any of them is looked at
            __syncthreads();
        } else {
#pragma unroll
            for (int j = 0; j < kIPT; ++j) slot[j] = (item0 + j < count) ? slots_in[item0 + j] : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int j = 0; j < kIPT; ++j) {
            id[j] = 0; cur32[j] = 0; first[j] = false;
            if (slot[j] != 0xFFFFFFFFu) {
                const uint64_t cur = __ldcg((const unsigned long long *)&p.table.slots[slot[j]]);
                cur32[j] = (uint32_t)cur;
                first[j] = (cur32[j] == enc_pending(gen, stage, item0 + j));
                id[j] = (uint32_t)(cur >> 32);
            }
        }
        ScanVal tv{0u, 0u, 0ull};  // this thread's items together
        uint64_t off[kIPT];
        uint32_t deg[kIPT];
#pragma unroll
        for (int j = 0; j < kIPT; ++j) {
            off[j] = 0; deg[j] = 0;
            if (first[j]) {
                tv.flags += 1u;
                if (has_next) {
                    uint64_t d64;
                    row_bounds(p.offsets, p.num_nodes, p.num_edges, id[j], off[j], d64);
                    if (d64 > 0xFFFFFFFFull) { atomicOr(&bs->error, kErrCapacity); d64 = 0; }
                    deg[j] = (uint32_t)d64;
                    uint32_t take; uint64_t draws;
                    row_demand(p.mode, d64, k, take, draws);
                    tv.take += take; tv.draws += draws;
                }
            }
        }

        // Block scan of the threads' totals: warp scans, then the warp totals.
        const ScanVal incl = warp_inclusive_scan(tv, lane);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            ScanVal w = (lane < kTile / 32) ? s_warp[lane] : ScanVal{0, 0, 0};
            const ScanVal wi = warp_inclusive_scan(w, lane);
            const ScanVal block_total = ScanVal{__shfl_sync(0xffffffffu, wi.flags, 31),
                                                __shfl_sync(0xffffffffu, wi.take, 31),
                                                __shfl_sync(0xffffffffu, wi.draws, 31)};
            if (lane < kTile / 32) s_warp[lane] = ScanVal{wi.flags - w.flags, wi.take - w.take, wi.draws - w.draws};
            const ScanVal prefix = FUSED ? ScanVal{0, 0, 0}
                                         : lookback_exclusive(p.tiles, tile, p.epoch_base + stage, block_total, lane, &bs->error);
            if (lane == 0) {
                s_prefix = prefix;
                if (tile == n_tiles - 1) {
                    // Totals of the stage: hand over to the next one.
                    const ScanVal tot = prefix + block_total;
                    StageInfo nx;
                    nx.n_nodes = si.n_nodes + tot.flags;
                    nx.n_edges = edges_before_next;
                    nx.frontier_n = tot.flags;
                    nx.hop_edges = tot.take;
                    nx.draws = si.draws + tot.draws;
                    nx.hop_draws = 0;
                    bs->stage[stage + 1] = nx;
                    bs->nodes_per_stage[stage] = tot.flags;
                    if (p.hub_count) p.hub_count[0] = p.hub_count[1] = 0;  // the hop's queues start empty (every batch says so)
                    if (stage == 0) bs->stage[0] = si;  // what the counts measure the draws against
                }
            }
        }
        __syncthreads();
        // exclusive prefix of this thread's first item
        ScanVal run = s_prefix + s_warp[warp];
        run.flags += incl.flags - tv.flags; run.take += incl.take - tv.take; run.draws += incl.draws - tv.draws;
        uint32_t pending = 0;  // bit j: item j's vertex is registered by an earlier item of this stage
#pragma unroll
        for (int j = 0; j < kIPT; ++j) {
            const uint32_t item = item0 + j;
            if (first[j]) {
                const uint32_t local = si.n_nodes + run.flags;
                if ((uint64_t)local >= p.cap_nodes || (uint64_t)local >= kMaxPos ||
                    (has_next && (uint64_t)run.flags >= p.frontier_cap)) {
                    atomicOr(&bs->error, kErrCapacity);
                    if (has_next && (uint64_t)run.flags < p.frontier_cap) p.frontier[run.flags] = FrontierEntry{};
                    // the batch has failed; its other items must still not wait for this vertex
                    p.table.slots[slot[j]] = ((uint64_t)id[j] << 32) | enc_final(gen, local & kPosMask);
                    write_item_local(p, stage, si.n_edges, item, 0xFFFFFFFFu);
                } else {
                    p.nodes[local] = id[j];
                    if (p.n_id) p.n_id[local] = (int64_t)id[j];
                    p.table.slots[slot[j]] = ((uint64_t)id[j] << 32) | enc_final(gen, local);  // readers accept either form
                    write_item_local(p, stage, si.n_edges, item, local);
                    if (has_next) {
                        FrontierEntry fe;
                        fe.off = off[j];
                        fe.dbase = si.draws + run.draws;
                        fe.id = id[j];
                        fe.local = local;
                        fe.deg = deg[j];
                        fe.ebase = run.take;
                        p.frontier[run.flags] = fe;
                    }
                }
                run.flags += 1u;
                if (has_next) {
                    uint32_t take; uint64_t draws;
                    row_demand(p.mode, deg[j], k, take, draws);
                    run.take += take; run.draws += draws;
                }
            } else if (item < count) {
                if (slot[j] == 0xFFFFFFFFu) write_item_local(p, stage, si.n_edges, item, 0xFFFFFFFFu);
                else if (!(cur32[j] & kPendingBit)) write_item_local(p, stage, si.n_edges, item, cur32[j] & kPosMask);  // an earlier stage's vertex
                else pending |= 1u << j;
            }
        }
        // The first sighting of a pending vertex is an earlier item of this stage: in this
        // tile (stored before the barrier below) or in a tile with a smaller ticket, whose
        // block is running and waits for nothing later than itself.
        __syncthreads();
        if (pending) {
#pragma unroll
            for (int j = 0; j < kIPT; ++j) {
                if (!(pending & (1u << j))) continue;
                uint32_t v = (uint32_t)__ldcg((const unsigned long long *)&p.table.slots[slot[j]]), spins = 0;
                while (v & kPendingBit) {
                    if (++spins > kSpinLimit) { atomicOr(&bs->error, kErrSpinTimeout); break; }
                    __nanosleep(40);
                    v = (uint32_t)__ldcg((const unsigned long long *)&p.table.slots[slot[j]]);
                }
                write_item_local(p, stage, si.n_edges, item0 + j, (v & kPendingBit) ? 0xFFFFFFFFu : (v & kPosMask));
            }
        }
        if (FUSED) break;
    }

    if (has_next) return;
    if (p.edge_index_local) {
        // Last stage: every edge of the batch exists, so the row offset of the int64
        // [2, E] local edge index is known.  Row 1 = the expanded vertex's local id.
        const uint64_t total = min((uint64_t)edges_before_next, p.cap_edges);
        for (uint64_t e = (uint64_t)blockIdx.x * kTile + threadIdx.x; e < total; e += (uint64_t)gridDim.x * kTile)
            p.edge_index_local[total + e] = (int64_t)p.src_local[e];
    }
    // The block that finishes last publishes the batch's counts (every
    // error bit any block raised is in by then) and leaves the state ready for the
    // handle's next batch.
    __shared__ bool s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&bs->done_blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    publish_counts(p, bs);
}

template <bool HAS_NEXT, int IPT>
__global__ void __launch_bounds__(kTile, 2)
k_assign(const SampleParams *pa, uint32_t stage, uint32_t k) {
    __shared__ __align__(16) SampleParams s_params;
    chain_sync();
    const SampleParams &p = chain_block(pa + blockIdx.y, s_params);
    chain_release(p.alone);
    assign_stage<HAS_NEXT, IPT, false>(p, stage, k);
}

// Seed insertion and stage 0 in one launch, a block per batch.
constexpr uint32_t kFusedSeeds = kTile * kMaxIPT;

template <int IPT>
__global__ void __launch_bounds__(kTile, 2)
k_assign_seeds(const SampleParams *__restrict__ pa, uint32_t k) {
    chain_release(pa[blockIdx.y].alone);
    assign_stage<true, IPT, true>(pa[blockIdx.y], 0, k);
}

// The same with the staged block in the kernel's parameters.
template <int IPT, int BYTES>
__global__ void __launch_bounds__(kTile, 2)
k_assign_seeds_packed(const __grid_constant__ PackedWords<BYTES> c, const StageLayout at, uint32_t k) {
    __shared__ __align__(16) SampleParams p;
    constexpr uint32_t kWords = sizeof(SampleParams) / 8, kGatherWords = sizeof(GatherArgs) / 8;
    const uint32_t words = kWords + (at.gather_dev ? kGatherWords : 0u);
    for (uint32_t i = threadIdx.x; i < words; i += kTile) {
        if (i < kWords) {
            const uint64_t v = c.w[blockIdx.y * kWords + i];
            ((uint64_t *)&p)[i] = v;
            ((uint64_t *)(at.params_dev + blockIdx.y))[i] = v;
        } else {
            ((uint64_t *)(at.gather_dev + blockIdx.y))[i - kWords] = c.w[gridDim.y * kWords + blockIdx.y * kGatherWords + i - kWords];
        }
    }
    __syncthreads();
    chain_release(p.alone);
    if (threadIdx.x == 0 && at.seeds_at) p.seeds = (const uint32_t *)(c.w + at.seeds_at) + blockIdx.y * at.seed_stride;
    __syncthreads();
    assign_stage<true, IPT, true>(p, 0, k);
}

// Hop `hop`: expand the frontier stage `hop` queued (stage[hop + 1] holds its
// size and where the hop's edges start).  The lanes of the whole grid share the
// frontier, so even a hop with few vertices spreads over the GPU.
//
// Latency-bound, so resident warps count: six blocks of 256 threads per SM, which leaves 40
// registers a thread.  Asked for one block the compiler takes 48 to 53, and the long chains of
// two workers lose 1.3 % (64 batches of 1024 seeds, fanouts 25, 10, on 100 M vertices / 2 B
// edges: 6.54 ms for 512 batches against 6.45).
template <int G, int PICK>
__global__ void __launch_bounds__(PICK == kPickLarge ? 128 : PICK == kPickWeighted ? kWeightedThreads : kPickThreads, PICK == kPickWeighted ? 14 : PICK == kPickLarge ? 12 : 6)
k_pick(const SampleParams *pa, uint32_t hop, uint32_t k) {
    __shared__ uint32_t s_picks[PICK == kPickLarge ? 4 : 1][PICK == kPickLarge ? kLargeK : 1];
    __shared__ uint32_t s_queue[PICK == kPickWeighted ? (kWeightedThreads / 32) * kQueue : 1];  // weighted: queued positions per warp
    __shared__ __align__(16) SampleParams s_params;
    chain_sync();
    const SampleParams &p = chain_block(pa + blockIdx.y, s_params);
    chain_release(p.alone);
    const StageInfo nx = p.state->stage[hop + 1];
    if constexpr (PICK == kPickWeighted) pick_weighted(p, hop, k, nx.n_edges, p.frontier, nx.frontier_n, s_queue);
    else if constexpr (PICK == kPickLarge) pick_large(p, hop, k, nx.n_edges, p.frontier, nx.frontier_n, &s_picks[0][0]);
    else pick_small<G>(p, hop, k, nx.n_edges, p.frontier, nx.frontier_n);
}

// The queued rows of a weighted hop, a warp per slice, whatever batch of the chain they
// belong to.  Every slice leaves its best k; the warp that finishes a row's last slice
// merges them and emits.  (key, position) is a total order, so the k smallest — and their
// emission order — do not depend on how the row was split or which warp merges.
//
// Why slices: a row of 500 K positions takes one block of 512 threads 450 us, whatever the rest
// of the chain does.  Twelve batches of 512 seeds, fanouts 15, 10, 5, on a graph of 10 M vertices
// and 200 M edges (28 M positions a batch): 5330 us with a block per row, 2070 us in slices.
//
// A guessed threshold below the row's k-th best key shows at the merge.  The row is then queued
// once more and a second launch (AGAIN) streams it in slices without a guess.  512 seeds,
// fanouts 15, 10, rows of up to 220 K positions: log-normal weights 175 us; one weight of a
// row 1e6 times the others 240 (870 if the merging warp streams the row alone); eight positive
// weights a row, the rest zero, 210 (3870 alone).
template <bool AGAIN>
__global__ void __launch_bounds__(kWeightedThreads, 14)
k_pick_hub_slices(const SampleParams *pa, uint32_t hop, uint32_t k) {
    __shared__ uint32_t s_queue[(kWeightedThreads / 32) * kQueue];
    __shared__ __align__(16) SampleParams s_params[kWeightedThreads / 32];
    chain_sync();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the parameter block of the batch this warp is at; what concerns the queue is in every one
    const SampleParams &p = s_params[warp];
    uint32_t batch = 0;
    auto load_params = [&] {
        __syncwarp();
        for (uint32_t i = lane; i < sizeof(SampleParams) / 8; i += 32) ((uint64_t *)&s_params[warp])[i] = ((const uint64_t *)(pa + batch))[i];
        __syncwarp();
    };
    load_params();
    chain_release(p.alone);
    const double inf = __longlong_as_double(0x7FF0000000000000ll);
    const unsigned long long count = p.hub_count[AGAIN];
    const uint32_t rows = min((uint32_t)(count >> 32), p.hub_cap), slices = min((uint32_t)count, p.hub_cap);
    const uint32_t half = AGAIN ? p.hub_cap : 0u;
    for (uint32_t slice = blockIdx.x * (kWeightedThreads / 32) + warp; slice < slices; slice += gridDim.x * (kWeightedThreads / 32)) {
        // the last row whose slices start at or before this one; 32 probes a step
        uint32_t lo = 0, n = rows;
        while (n > 1) {
            const uint32_t step = (n + 31) / 32, at = lane * step;
            const uint32_t m = __ballot_sync(0xffffffffu, at < n && p.hub_rows[half + lo + at].slice_base <= slice);
            const uint32_t hit = 31 - __clz(m);  // lane 0 always holds
            lo += hit * step;
            n = min(step, n - hit * step);
        }
        const HubRow row = p.hub_rows[half + lo];
        if (row.n_slices == 0) continue;  // did not fit: its own warp has done it
        if (row.batch != batch) { batch = row.batch; load_params(); }
        const FrontierEntry fe = p.frontier[row.vertex];
        const uint32_t deg = fe.deg, len = hub_slice_len(deg, AGAIN ? kHubDegree : p.hub_slice);
        const uint64_t first = (uint64_t)(slice - row.slice_base) * len;
        uint32_t begin = (uint32_t)min((uint64_t)deg, first), end = (uint32_t)min((uint64_t)deg, first + len);
        float guess = AGAIN ? __uint_as_float(0x7F800000u) : p.hub_guess[lo];
        uint32_t *shared_thr = p.hub_thr + half + lo;
        double best_key;
        uint32_t best_pos;
        bool mine = true;  // this warp finishes the row
        for (bool whole = row.n_slices == 1;; whole = true) {
            topk_stream(p, hop, fe, begin, end, k, lane, best_key, best_pos, s_queue + warp * kQueue, guess, shared_thr);
            if (!whole) {
                const uint64_t at = (uint64_t)slice * k;
                if ((uint32_t)lane < k) { p.hub_key[at + lane] = best_key; p.hub_pos[at + lane] = best_pos; }
                __threadfence();
                __syncwarp();
                uint32_t before = 0;
                if (lane == 0) { before = atomicAdd(p.hub_done + half + lo, 1u); __threadfence(); }
                mine = __shfl_sync(0xffffffffu, before, 0) == row.n_slices - 1;
                if (!mine) break;
                __syncwarp();  // lane 0's fence comes before the other lanes' reads
                const uint64_t from = (uint64_t)row.slice_base * k;
                const uint32_t cands = row.n_slices * k;
                for (uint32_t c = 0; c < cands; c += 32) {
                    const uint32_t i = c + lane;
                    // this slice's own best are in the lanes already
                    const bool have = i < cands && i / k != slice - row.slice_base;
                    const double ck = have ? __ldcg(p.hub_key + from + i) : inf;
                    const uint32_t cp = have ? __ldcg(p.hub_pos + from + i) : 0xFFFFFFFFu;
                    topk_insert_chunk(ck, cp, best_key, best_pos, k, lane);
                }
            }
            if (AGAIN || __shfl_sync(0xffffffffu, best_key, k - 1) <= (double)guess) break;
            // The guess was too low: the row once more without one, by this warp if the queue is full.
            // (What was found bounds the k-th best key from above, if k were found.)
            const float bound = __double2float_ru(__shfl_sync(0xffffffffu, best_key, k - 1));
            if (queue_long_row(p, 1, row.batch, row.vertex, deg, bound, lane)) { mine = false; break; }
            begin = 0; end = deg; guess = __uint_as_float(0x7F800000u); shared_thr = nullptr;
        }
        if (!mine) continue;
        if ((uint32_t)lane < k) emit_edge(p, hop, p.state->stage[hop + 1].n_edges, fe, lane, fe.off + best_pos);
    }
}

uint64_t next_pow2(uint64_t v) {
    uint64_t p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Items per thread of an assign launch: the fewest with which the tiles of all batches
// are resident at once (two blocks per SM).  A small stage is bound by the latency of its
// dependent loads (slot, table entry, row bounds), so it wants its items on as many SMs
// as there are; only a stage that fills the GPU gains from more items per thread.
// (Always four, last stage eight: the last stage of 128 seeds with fanouts 15, 10 ran 22 us
// on two blocks, now 13; a call of 1024 seeds with fanouts 25, 10 went from 167 to 140 us.)
template <bool HAS_NEXT>
void launch_assign(uint64_t items, uint32_t n_batches, cudaStream_t st, const SampleParams *pa, uint32_t stage, uint32_t k) {
    const uint64_t resident = (uint64_t)kSMs * 2 * kTile;
    const int most = HAS_NEXT ? kMaxIPT : kMaxIPTLast;
    int ipt = 1;
    while (ipt < most && items * n_batches > resident * ipt) ipt *= 2;
    const uint64_t per = (uint64_t)kTile * ipt, blocks = (items + per - 1) / per;
    // The grid covers the worst case only up to a few waves of resident blocks over the
    // whole group; the kernel draws tile tickets beyond that, so a batch far below its
    // bound does not pay for thousands of empty blocks.
    const dim3 grid((uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(blocks, std::max<uint64_t>(1, (uint64_t)kSMs * 8 / n_batches))), n_batches);
    switch (ipt) {
        case 1: launch_chained(k_assign<HAS_NEXT, 1>, grid, dim3(kTile), st, pa, stage, k); break;
        case 2: launch_chained(k_assign<HAS_NEXT, 2>, grid, dim3(kTile), st, pa, stage, k); break;
        case 4: launch_chained(k_assign<HAS_NEXT, 4>, grid, dim3(kTile), st, pa, stage, k); break;
        default: launch_chained(k_assign<HAS_NEXT, HAS_NEXT ? kMaxIPT : kMaxIPTLast>, grid, dim3(kTile), st, pa, stage, k); break;
    }
}

void launch_pick(int mode, uint32_t k, uint64_t frontier_est, uint32_t n_batches, cudaStream_t st,
                 const SampleParams *pa, uint32_t hop) {
    // About two waves of resident blocks over the whole group; the lanes stride beyond.
    auto blocks_for = [&](uint64_t vertices, uint64_t per_block) {
        const uint64_t b = (vertices + per_block - 1) / per_block;
        return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(b, std::max<uint64_t>(1, (uint64_t)kSMs * 16 / n_batches)));
    };
    if (mode == kModeWeightedReplace) {
        launch_chained(k_pick_weighted_replace, dim3(blocks_for(frontier_est, kPickThreads / 32), n_batches), dim3(kPickThreads), st, pa, hop, k);
    } else if (mode == kModeWeighted && k > 32) {
        launch_chained(k_pick_weighted_large, dim3(blocks_for(frontier_est, 1), n_batches), dim3(kWLThreads), st, pa, hop, k);
    } else if (mode == kModeWeighted) {
        const uint64_t blocks = std::min<uint64_t>((frontier_est + kWeightedThreads / 32 - 1) / (kWeightedThreads / 32),
                                                   std::max<uint64_t>(1, (uint64_t)kSMs * 128 / n_batches));
        launch_chained(k_pick<32, kPickWeighted>, dim3((uint32_t)std::max<uint64_t>(1, blocks), n_batches), dim3(kWeightedThreads), st, pa, hop, k);
        // rows longer than kHubDegree were only queued: a warp per slice of them, and once more for
        // those whose guess was too low (as a rule none)
        launch_chained(k_pick_hub_slices<false>, dim3((uint32_t)kSMs * 16), dim3(kWeightedThreads), st, pa, hop, k);
        launch_chained(k_pick_hub_slices<true>, dim3((uint32_t)kSMs * 4), dim3(kWeightedThreads), st, pa, hop, k);
    } else if (k > 32) {
        launch_chained(k_pick<32, kPickLarge>, dim3(blocks_for(frontier_est, 4), n_batches), dim3(128), st, pa, hop, k);
    } else {
        const uint32_t G = k <= 4 ? 4 : k <= 8 ? 8 : k <= 16 ? 16 : 32;
        const dim3 grid(blocks_for(frontier_est, 2 * kPickThreads / G), n_batches);  // two vertices per lane group and round
        switch (G) {
            case 4: launch_chained(k_pick<4, kPickSmall>, grid, dim3(kPickThreads), st, pa, hop, k); break;
            case 8: launch_chained(k_pick<8, kPickSmall>, grid, dim3(kPickThreads), st, pa, hop, k); break;
            case 16: launch_chained(k_pick<16, kPickSmall>, grid, dim3(kPickThreads), st, pa, hop, k); break;
            default: launch_chained(k_pick<32, kPickSmall>, grid, dim3(kPickThreads), st, pa, hop, k); break;
        }
    }
}

}  // namespace
}  // namespace ag

using namespace ag;

struct ag_sampler {
    const ag_graph *g = nullptr;
    ag_sampling_config cfg{};
    int device = 0;
    int mode = kModeUniform;
    uint64_t seed = 0;
    // RNG stream position of the handle (draws consumed by earlier batches).  Kept on the
    // host from the counts of every finished continuing batch, so it survives scratch
    // growth and state resets; `pending_pos` marks a launched batch not yet accounted.
    uint64_t stream_pos = 0;
    bool pending_pos = false;
    uint32_t epoch = 0;
    uint32_t gen = 0;    // table generation of the next launch
    uint32_t group = 1;  // batches one launch chain can carry
    // sizing (per batch)
    uint64_t cap_seeds = 0, max_nodes = 0, max_edges = 0, max_hop_edges = 0;
    uint64_t table_cap = 0, n_tiles = 0;
    // scratch (device), each `group` times the per-batch size, carved out of one block
    uint8_t *scratch = nullptr;
    uint64_t *table = nullptr;
    FrontierEntry *frontier = nullptr;
    uint64_t max_frontier = 0;
    uint32_t *slot_of_seed = nullptr, *slot_of_edge = nullptr;
    // weighted only: the queue of long rows, one for the chain (hub_rows is the allocation)
    HubRow *hub_rows = nullptr;
    unsigned long long *hub_count = nullptr;
    uint32_t *hub_thr = nullptr, *hub_done = nullptr, *hub_pos = nullptr;
    float *hub_guess = nullptr;
    double *hub_key = nullptr;
    uint32_t hub_cap = 0;
    TileDesc *tiles = nullptr;
    BatchState *state = nullptr;
    uint8_t *stage_dev = nullptr;   // parameter blocks, gather arguments and seeds of the chain (see StageLayout)
    // pinned host
    ag_sample_counts *counts_host = nullptr;
    bool yield_wait = false;  // ag_sample_group_wait polls and yields instead of spinning in the runtime
    uint8_t *stage_host = nullptr;
    cudaEvent_t done = nullptr;
    bool in_flight = false, dirty = true;
    uint32_t in_flight_n = 0;
    // A loader's handle gathers on its own low-priority stream, behind an event:
    // sampling kernels of other handles (latency-bound, few resources) then slip
    // in between the short-lived blocks of a running gather (bandwidth-bound).
    // A handle that runs alone has no such neighbours and gathers on the caller's
    // stream: the hop to another stream and back cost a call 5 us or so.  Made when
    // the first such chain is launched.
    cudaStream_t gstream = nullptr;
    bool pipelined = false;  // a loader's, or one of a group: sampler_set_pipelined
    cudaEvent_t sampled = nullptr;
    // Sharded stores: the remote part of a chain's rows is fetched by a launch of its own on
    // this stream (between the two priorities), beside the local part on gstream.  Made when
    // the first such chain is launched.
    cudaStream_t rstream = nullptr;
    int gpriority = 0, rpriority = 0;
    cudaEvent_t remote_done = nullptr;
    uint64_t est_rows_tight = 0;  // rows per batch the last chain produced, with little headroom (sort padding)
    SortScratch sort;  // sharded feature stores: the chain's row ids in address order (gather.cu)
    // The arguments of the chain in flight, kept so that it can be launched once more:
    // the dedup tables are sized from the node counts of earlier chains (small tables stay
    // in L2), and a batch that outgrows its table is sampled again with the full-size one.
    struct Launch {
        uint32_t n_batches = 0;
        std::vector<const uint32_t *> seeds;
        std::vector<uint64_t> n_seeds, batch_seeds;
        bool has_batch_seeds = false;
        int32_t seeds_mem = AG_MEM_HOST;
        const ag_features *feats = nullptr;
        std::vector<ag_subgraph_buffers> bufs;
        cudaStream_t stream = nullptr;
        bool reduced_table = false;
    } last;
    // Grid-size estimates from the last group's real counts (the bounds before
    // the first one); kernels stride past an estimate that turns out too small.
    uint64_t est_nodes = 0;
    uint64_t est_items[AG_MAX_HOPS + 2] = {0};
    // optional per-group device timing
    bool profile = false, gathered = false;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    // buffers handed out by ag_sample (library-allocated variant)
    std::vector<void *> owned;
};

namespace {

void compute_bounds(const ag_sampler *s, uint64_t n_seeds, uint64_t *max_nodes, uint64_t *max_edges,
                    uint64_t *max_hop_edges) {
    const uint64_t N = s->g->num_nodes;
    uint64_t f = std::min<uint64_t>(n_seeds, N), nodes = f, edges = 0, mhe = 0;
    for (uint32_t h = 0; h < s->cfg.num_hops; ++h) {
        const uint64_t e = f * s->cfg.fanout[h];
        edges += e;
        mhe = std::max(mhe, e);
        f = std::min<uint64_t>(e, N);
        nodes += f;
    }
    if (max_nodes) *max_nodes = std::min<uint64_t>(nodes, N);
    if (max_edges) *max_edges = edges;
    if (max_hop_edges) *max_hop_edges = mhe;
}

void free_scratch(ag_sampler *s) {
    workspace_free(s->scratch); workspace_free(s->stage_host);
    s->scratch = nullptr; s->stage_host = s->stage_dev = nullptr;
    s->table = nullptr; s->frontier = nullptr; s->tiles = nullptr; s->hub_rows = nullptr;
    s->slot_of_seed = s->slot_of_edge = nullptr;
}

// A finished continuing batch (no per-batch seed) moves the handle's stream on by
// the draws it consumed; called wherever the host has just waited for the batch.
void account_stream(ag_sampler *s) {
    if (s->pending_pos) s->stream_pos += s->counts_host[0].draws;
    s->pending_pos = false;
}

// Sizes of a batch of n_seeds seeds; refuses one past the per-batch limits.
int32_t size_batch(ag_sampler *s, uint64_t n_seeds) {
    const uint64_t cap = std::max<uint64_t>(n_seeds, 1);
    compute_bounds(s, cap, &s->max_nodes, &s->max_edges, &s->max_hop_edges);
    if (s->max_nodes >= kMaxPos || s->max_hop_edges >= kMaxPos || cap >= kMaxPos || s->max_edges >= 0xFFFFFFFFull)
        return fail(AG_ERR_VALUE, "batch too large: %llu seeds with this fanout can reach %llu nodes and %llu edges "
                    "in a hop (limit %llu each)", (unsigned long long)n_seeds, (unsigned long long)s->max_nodes,
                    (unsigned long long)s->max_hop_edges, (unsigned long long)kMaxPos - 1);
    return AG_OK;
}

// Scratch for `group` batches of up to n_seeds seeds each: one device block (an allocation
// takes 0.1 to 1.5 ms when the driver has to map memory) and one pinned one.
int32_t ensure_scratch(ag_sampler *s, uint64_t n_seeds) {
    if (n_seeds <= s->cap_seeds && s->table) return AG_OK;
    if (s->in_flight) { AG_CUDA(cudaEventSynchronize(s->done)); s->in_flight = false; account_stream(s); }
    free_scratch(s);
    s->cap_seeds = 0;
    const uint64_t cap = std::max<uint64_t>(n_seeds, 1), G = s->group;
    AG_TRY(size_batch(s, n_seeds));
    s->table_cap = std::max<uint64_t>(1024, next_pow2(2 * s->max_nodes));
    // the frontier of a hop holds at most the vertices the previous stage found
    s->max_frontier = std::max<uint64_t>(std::min<uint64_t>(std::max(cap, s->max_hop_edges), s->g->num_nodes), 1);
    s->n_tiles = std::max<uint64_t>(std::max(cap, s->max_hop_edges) / kTile + 2, 2);
    s->hub_cap = 0;
    uint64_t hop_k = 1;
    if (s->mode == kModeWeighted) {
        // A batch expands a vertex once, and a row of d > kHubDegree positions is at most
        // 2 d / kHubDegree slices.
        const uint64_t most = 2 * (s->g->num_edges / kHubDegree) * G;
        for (uint32_t h = 0; h < s->cfg.num_hops; ++h) hop_k = std::max<uint64_t>(hop_k, std::min<uint32_t>(s->cfg.fanout[h], 32u));
        s->hub_cap = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(most, 1), kMaxHubSlices);
    }
    const uint64_t stage = G * (sizeof(SampleParams) + sizeof(GatherArgs) + (cap + 1) / 2 * 8), hubs = s->hub_cap;
    AG_CUDA(workspace_alloc_host(&s->stage_host, stage));
    uint8_t *base = nullptr;
    for (int pass = 0; pass < 2; ++pass) {  // the sizes, then the places
        uint64_t off = 0;
        auto carve = [&](auto **p, uint64_t bytes) {
            if (pass) *(uint8_t **)p = base + off;
            off += (bytes + 255) & ~255ull;
        };
        carve(&s->table, G * s->table_cap * 8);
        carve(&s->frontier, G * s->max_frontier * sizeof(FrontierEntry));
        carve(&s->slot_of_seed, G * cap * 4);
        carve(&s->slot_of_edge, G * std::max<uint64_t>(s->max_edges, 1) * 4);
        carve(&s->tiles, G * s->n_tiles * sizeof(TileDesc));
        carve(&s->stage_dev, stage);
        if (hubs) {
            carve(&s->hub_rows, 2 * hubs * sizeof(HubRow)); carve(&s->hub_count, 16);
            carve(&s->hub_key, hubs * hop_k * 8); carve(&s->hub_pos, hubs * hop_k * 4);
            carve(&s->hub_thr, 2 * hubs * 4); carve(&s->hub_done, 2 * hubs * 4); carve(&s->hub_guess, hubs * 4);
        }
        if (!pass) {
            AG_CUDA(workspace_alloc(&base, off));
            s->scratch = base;
        }
    }
    s->cap_seeds = cap;
    s->epoch = 0;
    s->dirty = true;
    return AG_OK;
}

}  // namespace

extern "C" int32_t ag_sampler_create_group(const ag_graph *g, const ag_sampling_config *cfg, uint32_t group,
                                           ag_sampler **out) {
    if (!g || !cfg || !out) return fail(AG_ERR_VALUE, "ag_sampler_create: null argument");
    if (group == 0 || group > 256) return fail(AG_ERR_VALUE, "group size must be between 1 and 256 (got %u)", group);
    if (cfg->num_hops == 0 || cfg->num_hops > AG_MAX_HOPS)
        return fail(AG_ERR_VALUE, "num_neighbors must list between 1 and %d hops (got %u)", AG_MAX_HOPS, cfg->num_hops);
    // SamplerConfigError::WeightsMissing (sampler.rs:331-337)
    if (cfg->weighted && !g->weights)
        return fail(AG_ERR_VALUE, "weighted sampling requested, but the graph has no edge weights");
    if (cfg->rng_mode != AG_RNG_WYRAND_EXACT && cfg->rng_mode != AG_RNG_PHILOX)
        return fail(AG_ERR_VALUE, "unknown rng_mode %d", cfg->rng_mode);
    for (uint32_t h = 0; h < cfg->num_hops; ++h) {
        if (cfg->fanout[h] > (uint32_t)kLargeK)
            return fail(AG_ERR_VALUE, "fanout of at most %d per hop is supported (hop %u asks %u)", kLargeK, h, cfg->fanout[h]);
    }
    DeviceGuard guard(g->device);
    if (!guard.ok) return AG_ERR_CUDA;
    ag_sampler *s = new ag_sampler();
    s->g = g;
    s->cfg = *cfg;
    s->device = g->device;
    s->group = group;
    s->pipelined = group > 1;
    s->mode = cfg->weighted ? (cfg->replace ? kModeWeightedReplace : kModeWeighted) : (cfg->replace ? kModeReplace : kModeUniform);
    s->seed = cfg->seed;
    int32_t st = AG_OK;
    do {
        if (workspace_alloc(&s->state, group * sizeof(BatchState)) != cudaSuccess ||  // cleared by the first launch (`dirty`)
            workspace_alloc_host(&s->counts_host, group * sizeof(ag_sample_counts)) != cudaSuccess ||
            cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&s->sampled, cudaEventDisableTiming) != cudaSuccess) {
            st = fail(AG_ERR_CUDA, "sampler allocation failed: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        int lo = 0, hi = 0;
        cudaDeviceGetStreamPriorityRange(&lo, &hi);  // lo = least urgent
        // AG_GATHER_PRIORITY=high: the gather streams as urgent as the sampling streams (A/B measurements)
        static const bool gather_high = [] { const char *v = getenv("AG_GATHER_PRIORITY"); return v && v[0] == 'h'; }();
        s->gpriority = gather_high ? hi : lo;
        s->rpriority = (lo + hi) / 2;
        // Without a size to expect, the first batch brings it.
        st = cfg->max_seeds ? ensure_scratch(s, cfg->max_seeds) : size_batch(s, 1);
    } while (0);
    if (st != AG_OK) { ag_sampler_free(s); return st; }
    *out = s;
    return AG_OK;
}

extern "C" int32_t ag_sampler_create(const ag_graph *g, const ag_sampling_config *cfg, ag_sampler **out) {
    return ag_sampler_create_group(g, cfg, 1, out);
}

extern "C" void ag_sampler_free(ag_sampler *s) {
    if (!s) return;
    DeviceGuard guard(s->device);
    if (s->in_flight && s->done) cudaEventSynchronize(s->done);
    free_scratch(s);
    s->sort.release();
    for (void *p : s->owned) cudaFree(p);
    workspace_free(s->state); workspace_free(s->counts_host);
    if (s->done) cudaEventDestroy(s->done);
    if (s->sampled) cudaEventDestroy(s->sampled);
    workspace_stream_free(s->gstream, s->gpriority);
    workspace_stream_free(s->rstream, s->rpriority);
    if (s->remote_done) cudaEventDestroy(s->remote_done);
    for (auto &e : s->ev) if (e) cudaEventDestroy(e);
    delete s;
}

extern "C" int32_t ag_sampler_reseed(ag_sampler *s, uint64_t seed) {
    if (!s) return fail(AG_ERR_VALUE, "ag_sampler_reseed: null sampler");
    if (s->in_flight) {  // the batch in flight still belongs to the old stream
        DeviceGuard guard(s->device);
        cudaEventSynchronize(s->done);
    }
    s->seed = seed;
    s->stream_pos = 0;
    s->pending_pos = false;
    return AG_OK;
}

void ag::sampler_set_pipelined(ag_sampler *s) { s->pipelined = true; }

// A loader's worker threads wait for their chains by polling the event and yielding
// the core between polls instead of spinning inside the runtime: with three workers
// per GPU and eight GPUs per host the spinning waits alone would occupy most of the
// host's cores, which the consumer's own thread needs; on an idle core a yield returns
// at once, so nothing is lost when there are cores to spare.  (Sleeping on the event
// — cudaEventBlockingSync — was measured too: -9 % on one GPU, the wake-up is too slow.)
int32_t ag::sampler_set_yielding_wait(ag_sampler *s, bool on) {
    s->yield_wait = on;
    return AG_OK;
}

extern "C" int32_t ag_sampler_set_profiling(ag_sampler *s, int32_t on) {
    if (!s) return fail(AG_ERR_VALUE, "ag_sampler_set_profiling: null sampler");
    DeviceGuard guard(s->device);
    if (!guard.ok) return AG_ERR_CUDA;
    if (on && !s->ev[0])
        for (auto &e : s->ev) AG_CUDA(cudaEventCreate(&e));
    s->profile = on != 0;
    return AG_OK;
}

extern "C" int32_t ag_sampler_bounds(const ag_sampler *s, uint64_t n_seeds, uint64_t *max_nodes, uint64_t *max_edges) {
    if (!s) return fail(AG_ERR_VALUE, "ag_sampler_bounds: null sampler");
    compute_bounds(s, n_seeds, max_nodes, max_edges, nullptr);
    return AG_OK;
}

// One launch chain for `n_batches` independent batches.  batch b uses
// seeds[b] / n_seeds[b] / bufs[b] and, when batch_seeds != NULL, restarts its
// RNG stream at draw 0 of batch_seeds[b]; with batch_seeds == NULL the handle's
// own stream continues (only meaningful for a single batch).
namespace {
int32_t launch_saved(ag_sampler *s, bool relaunch);
}  // namespace

extern "C" int32_t ag_sample_group_into(ag_sampler *s, uint32_t n_batches, const uint32_t *const *seeds,
                                        const uint64_t *n_seeds, int32_t seeds_mem, const uint64_t *batch_seeds,
                                        const ag_features *feats, ag_subgraph_buffers *bufs, void *stream) {
    if (!s || !bufs || !seeds || !n_seeds) return fail(AG_ERR_VALUE, "ag_sample_group_into: null argument");
    if (n_batches == 0 || n_batches > s->group)
        return fail(AG_ERR_VALUE, "group of %u batches does not fit a sampler created for %u", n_batches, s->group);
    const ag_graph *g = s->g;
    uint64_t max_n = 0;
    bool want_x = false;
    for (uint32_t b = 0; b < n_batches; ++b) {
        const ag_subgraph_buffers &B = bufs[b];
        if (!seeds[b] && n_seeds[b]) return fail(AG_ERR_VALUE, "ag_sample_group_into: null seeds");
        if (!B.nodes || !B.edge_dst || !B.src_local || !B.dst_local || !B.seed_locals)
            return fail(AG_ERR_VALUE, "nodes, edge_dst, src_local, dst_local and seed_locals buffers are required");
        if (B.cap_seeds < n_seeds[b]) return fail(AG_ERR_VALUE, "seed_locals capacity %llu < %llu seeds",
                                                  (unsigned long long)B.cap_seeds, (unsigned long long)n_seeds[b]);
        if (n_seeds[b] >= kMaxPos) return fail(AG_ERR_VALUE, "too many seeds");
        max_n = std::max(max_n, n_seeds[b]);
        want_x = want_x || (feats && B.x);
        // Seeds::new (sampler.rs:230-239): name the first id at or past num_nodes.
        if (seeds_mem == AG_MEM_HOST)
            for (uint64_t i = 0; i < n_seeds[b]; ++i)
                if ((uint64_t)seeds[b][i] >= g->num_nodes)
                    return fail(AG_ERR_SAMPLING, "seed node %u (position %llu) is out of range for %llu nodes",
                                seeds[b][i], (unsigned long long)i, (unsigned long long)g->num_nodes);
    }
    if (feats && want_x && feats->row_stride != 1 && !feats->shards)
        return fail(AG_ERR_VALUE, "a cyclic feature shard is read through a sharded view");
    if (feats && want_x && feats->device != s->device)
        return fail(AG_ERR_VALUE, "feature store lives on device %d, sampler on %d", feats->device, s->device);
    DeviceGuard guard(s->device);
    if (!guard.ok) return AG_ERR_CUDA;
    if (s->in_flight) { AG_CUDA(cudaEventSynchronize(s->done)); s->in_flight = false; account_stream(s); }
    ag_sampler::Launch &L = s->last;
    L.n_batches = n_batches;
    L.seeds.assign(seeds, seeds + n_batches);
    L.n_seeds.assign(n_seeds, n_seeds + n_batches);
    L.has_batch_seeds = batch_seeds != nullptr;
    if (batch_seeds) L.batch_seeds.assign(batch_seeds, batch_seeds + n_batches);
    L.seeds_mem = seeds_mem;
    L.feats = feats;
    L.bufs.assign(bufs, bufs + n_batches);
    L.stream = (cudaStream_t)stream;
    return launch_saved(s, false);
}

namespace {
// Time zero of the profiled intervals on a GPU: an event recorded once, on the stream of
// the first profiled launch there.  Called with a null stream it only returns the event.
cudaEvent_t profile_origin(int device, cudaStream_t st) {
    static std::mutex m;
    static cudaEvent_t origin[64] = {nullptr};
    std::lock_guard<std::mutex> lk(m);
    if (device < 0 || device >= 64) return nullptr;
    if (!origin[device] && st) {
        cudaEvent_t e = nullptr;
        if (cudaEventCreate(&e) == cudaSuccess && cudaEventRecord(e, st) == cudaSuccess) origin[device] = e;
        else if (e) cudaEventDestroy(e);
    }
    return origin[device];
}

int32_t launch_saved_impl(ag_sampler *s, bool relaunch);

// Queues the chain described by s->last.  relaunch: the same chain once more with
// full-size dedup tables (host seeds are already in the handle's staged block).
// A failure part way through leaves kernels of the chain queued: wait for them and
// mark the handle's device state unknown, so that the next call clears it instead of
// reusing staging buffers, table generation and batch state under running kernels.
int32_t launch_saved(ag_sampler *s, bool relaunch) {
    const int32_t st = launch_saved_impl(s, relaunch);
    if (st != AG_OK) {
        const std::string msg = ag_last_error();
        cudaStreamSynchronize(s->last.stream);
        if (s->gstream) cudaStreamSynchronize(s->gstream);
        if (s->rstream) cudaStreamSynchronize(s->rstream);
        cudaGetLastError();
        s->dirty = true;
        s->pending_pos = false;
        s->in_flight = false;
        set_error("%s", msg.c_str());
    }
    return st;
}

int32_t launch_saved_impl(ag_sampler *s, bool relaunch) {
    const ag_sampler::Launch &L = s->last;
    const uint32_t n_batches = L.n_batches;
    const uint32_t *const *seeds = L.seeds.data();
    const uint64_t *n_seeds = L.n_seeds.data();
    const uint64_t *batch_seeds = L.has_batch_seeds ? L.batch_seeds.data() : nullptr;
    const int32_t seeds_mem = L.seeds_mem;
    const ag_features *feats = L.feats;
    const ag_subgraph_buffers *bufs = L.bufs.data();
    const ag_graph *g = s->g;
    uint64_t max_n = 0;
    bool want_x = false;
    for (uint32_t b = 0; b < n_batches; ++b) {
        max_n = std::max(max_n, n_seeds[b]);
        want_x = want_x || (feats && bufs[b].x);
    }
    cudaStream_t st = L.stream;
    AG_TRY(ensure_scratch(s, max_n));
    if (s->profile) {
        profile_origin(s->device, st);
        AG_CUDA(cudaEventRecord(s->ev[0], st));
    }
    if (s->dirty || s->gen >= kGens) {
        // Every slot free again.  A launch marks its entries with its generation,
        // so this real clear is only needed once the generations have cycled (or
        // after a failed launch left the table in an unknown state).
        AG_CUDA(cudaMemsetAsync(s->table, 0xFF, (uint64_t)s->group * s->table_cap * 8, st));
        s->gen = 0;
    }
    if (s->dirty) {
        AG_CUDA(cudaMemsetAsync(s->state, 0, s->group * sizeof(BatchState), st));
        AG_CUDA(cudaMemsetAsync(s->tiles, 0, (uint64_t)s->group * s->n_tiles * sizeof(TileDesc), st));
        s->epoch = 0;
        s->dirty = false;
    }
    const uint32_t H = s->cfg.num_hops;
    if (s->epoch + (H + 2) > 0x3FFFFF00u) {  // the epoch lives in 30 bits of the tile status
        AG_CUDA(cudaMemsetAsync(s->tiles, 0, (uint64_t)s->group * s->n_tiles * sizeof(TileDesc), st));
        s->epoch = 0;
    }
    // Tables sized for twice the nodes the last chains really produced (with headroom)
    // instead of the worst-case bound: a chain's tables then fit in L2.
    uint64_t used_cap = s->table_cap;
    if (!relaunch && s->est_nodes) used_cap = std::min(s->table_cap, std::max<uint64_t>(1024, next_pow2(2 * s->est_nodes)));
    s->last.reduced_table = used_cap < s->table_cap;
    uint32_t log2cap = 0;
    while ((1ull << log2cap) < used_cap) ++log2cap;
    const uint64_t ecap = std::max<uint64_t>(s->max_edges, 1);

    // The staged block (see PackedWords): as kernel parameters where the seeds are inserted by
    // stage 0 and the block is small, else copied to the device.
    const bool host_seeds = seeds_mem == AG_MEM_HOST;
    const uint32_t nmax = (uint32_t)max_n, seed_stride = (nmax + 1) & ~1u;
    const uint64_t gather_at = n_batches * sizeof(SampleParams), seeds_at = gather_at + (want_x ? n_batches * sizeof(GatherArgs) : 0);
    const uint64_t stage_bytes = seeds_at + (host_seeds ? (uint64_t)n_batches * seed_stride * 4 : 0);
    const bool fused = nmax <= kFusedSeeds;
    const uint64_t packed_most = nmax <= kTile ? kPackedSmall : nmax <= kTile * 2 ? kPackedMedium : kPackedLarge;
    const bool packed = fused && stage_bytes <= packed_most;
    SampleParams *params_host = (SampleParams *)s->stage_host;
    GatherArgs *gather_host = (GatherArgs *)(s->stage_host + gather_at), *gather_dev = (GatherArgs *)(s->stage_dev + gather_at);
    uint32_t *seeds_host = (uint32_t *)(s->stage_host + seeds_at);
    const uint32_t *seeds_dev = (const uint32_t *)(s->stage_dev + seeds_at);
    uint64_t b_nodes = 0;
    for (uint32_t b = 0; b < n_batches; ++b) {
        const ag_subgraph_buffers &B = bufs[b];
        const uint32_t n = (uint32_t)n_seeds[b];
        SampleParams p{};
        p.offsets = g->offsets; p.dst = g->dst; p.weights = g->weights;
        p.num_nodes = g->num_nodes; p.num_edges = g->num_edges;
        p.table = DedupTable{s->table + (uint64_t)b * used_cap, (uint32_t)(used_cap - 1), 32u - log2cap, s->gen};
        p.state = s->state + b;
        p.tiles = s->tiles + (uint64_t)b * s->n_tiles;
        p.epoch_base = s->epoch + 1;
        p.n_seeds = n;
        if (host_seeds) {  // (packed: the kernel fills in where they are)
            if (n && !relaunch) memcpy(seeds_host + (uint64_t)b * seed_stride, seeds[b], (size_t)n * 4);
            p.seeds = seeds_dev + (uint64_t)b * seed_stride;
        } else {
            p.seeds = seeds[b];
        }
        p.seed = batch_seeds ? batch_seeds[b] : s->seed;
        p.rng_mode = s->cfg.rng_mode; p.mode = s->mode;
        p.alone = s->pipelined ? 0u : 1u;
        p.start_draw = batch_seeds ? 0ull : s->stream_pos;
        p.num_hops = H;
        p.nodes = B.nodes; p.edge_src = B.edge_src; p.edge_dst = B.edge_dst;
        p.src_local = B.src_local; p.dst_local = B.dst_local; p.seed_locals = B.seed_locals;
        p.edge_ids = s->cfg.track_edge_ids ? B.edge_ids : nullptr;
        p.cap_nodes = B.cap_nodes; p.cap_edges = B.cap_edges;
        p.n_id = B.n_id; p.edge_index_local = B.edge_index_local; p.e_id = B.e_id; p.seed_index = B.seed_index;
        p.counts = s->counts_host + b;  // pinned: one posted write, visible once the chain's event is
        p.slot_of_seed = s->slot_of_seed + (uint64_t)b * s->cap_seeds;
        p.slot_of_edge = s->slot_of_edge + (uint64_t)b * ecap;
        p.frontier = s->frontier + (uint64_t)b * s->max_frontier;
        p.frontier_cap = s->max_frontier;
        if (s->hub_rows) {
            p.hub_rows = s->hub_rows; p.hub_count = s->hub_count; p.hub_thr = s->hub_thr; p.hub_done = s->hub_done; p.hub_guess = s->hub_guess;
            p.hub_key = s->hub_key; p.hub_pos = s->hub_pos; p.hub_cap = s->hub_cap;
            // about as many slices whatever the chain's length, a few times what runs at once
            p.hub_slice = (uint32_t)std::min<uint64_t>(kHubDegree * std::max<uint64_t>(next_pow2(n_batches) / 2, 1), 16 * kHubDegree);
        }
        params_host[b] = p;
        uint64_t bn, be;
        compute_bounds(s, n, &bn, &be, nullptr);
        b_nodes = std::max(b_nodes, bn);
        if (want_x) {
            GatherArgs ga{};
            if (feats && B.x) {
                set_gather_source(ga, feats);
                ga.ids = B.nodes; ga.ids64 = 0;
                ga.n = std::min<uint64_t>(bn, B.cap_x ? std::min(B.cap_x, B.cap_nodes) : B.cap_nodes);
                // rows to gather = nodes registered by the last stage (read on the device)
                ga.n_dev = &s->state[b].stage[H + 1].n_nodes;
                ga.out = B.x;
            }
            gather_host[b] = ga;
        }
    }
    s->pending_pos = (batch_seeds == nullptr);  // a continuing batch advances the handle's stream
    s->epoch += H + 2;
    s->gen += 1;
    const SampleParams *pa = (const SampleParams *)s->stage_dev;
    const uint32_t k0 = s->cfg.fanout[0];
    if (packed) {
        const StageLayout at{(SampleParams *)s->stage_dev, want_x ? gather_dev : nullptr, host_seeds ? (uint32_t)(seeds_at / 8) : 0u, seed_stride};
        auto launch = [&](auto ipt, auto words) {
            constexpr int kIPT = decltype(ipt)::value, kBytes = decltype(words)::value;
            PackedWords<kBytes> c;
            memcpy(&c, s->stage_host, stage_bytes);
            k_assign_seeds_packed<kIPT, kBytes><<<dim3(1, n_batches), kTile, 0, st>>>(c, at, k0);
        };
        if (nmax <= kTile) launch(std::integral_constant<int, 1>{}, std::integral_constant<int, kPackedSmall>{});
        else if (nmax <= kTile * 2) launch(std::integral_constant<int, 2>{}, std::integral_constant<int, kPackedMedium>{});
        else launch(std::integral_constant<int, kMaxIPT>{}, std::integral_constant<int, kPackedLarge>{});
    } else {
        AG_CUDA(cudaMemcpyAsync(s->stage_dev, s->stage_host, stage_bytes, cudaMemcpyHostToDevice, st));
        if (!fused) k_insert_seeds<<<dim3((nmax + 255) / 256, n_batches), 256, 0, st>>>(pa);
        else if (nmax <= kTile) k_assign_seeds<1><<<dim3(1, n_batches), kTile, 0, st>>>(pa, k0);
        else if (nmax <= kTile * 2) k_assign_seeds<2><<<dim3(1, n_batches), kTile, 0, st>>>(pa, k0);
        else k_assign_seeds<kMaxIPT><<<dim3(1, n_batches), kTile, 0, st>>>(pa, k0);
    }
    uint64_t items = nmax;  // bound on the items of the stage being launched
    for (uint32_t stage = 0; stage <= H; ++stage) {
        const bool has_next = stage < H;
        const uint32_t k = has_next ? s->cfg.fanout[stage] : 0;
        const uint64_t expect = (stage && s->est_items[stage]) ? std::min(items, s->est_items[stage]) : items;
        if (stage == 0 && fused) {}  // done above
        else if (has_next) launch_assign<true>(expect, n_batches, st, pa, stage, k);
        else launch_assign<false>(expect, n_batches, st, pa, stage, k);
        if (has_next && k) {
            // the new vertices of this stage are at most its items
            launch_pick(s->mode, k, std::min<uint64_t>(expect, g->num_nodes), n_batches, st, pa, stage);
        }
        items = std::min<uint64_t>(items, g->num_nodes) * k;
    }
    AG_CUDA(cudaGetLastError());
    if (s->profile) AG_CUDA(cudaEventRecord(s->ev[1], st));
    s->gathered = false;
    if (want_x) {
        bool aligned = ((uintptr_t)feats->payload % 16) == 0;
        for (uint32_t b = 0; b < n_batches; ++b) aligned = aligned && ((uintptr_t)bufs[b].x % 16) == 0;
        const uint64_t rows = s->est_nodes ? std::min(b_nodes, s->est_nodes) : b_nodes;
        const uint32_t row_bytes = (uint32_t)(feats->dim * elem_size(feats->dtype));
        const bool sorted = sorted_gather_applies(feats, row_bytes, aligned);
        // Rows of a sharded store are fetched in address order, each distinct row of the chain
        // once.  Making and sorting the keys is small, latency-bound work like the sampling
        // kernels: it stays on the (high-priority) sampling stream.  (The handle's previous
        // chain has finished — its event was waited for — so the sort scratch is free.)
        const uint64_t sort_rows = s->est_rows_tight ? std::min(rows, s->est_rows_tight) : rows;  // less padding to sort
        if (sorted) AG_CUDA(launch_sort_keys(GatherArgs{}, gather_dev, n_batches, sort_rows, feats, s->sort, st));
        cudaStream_t gs = st;
        if (s->pipelined || sorted) {
            // sampling chain -> event -> gather on the low-priority stream -> event -> caller's stream
            if (!s->gstream) AG_CUDA(workspace_stream(&s->gstream, s->gpriority));
            gs = s->gstream;
            AG_CUDA(cudaEventRecord(s->sampled, st));
            AG_CUDA(cudaStreamWaitEvent(gs, s->sampled, 0));
        }
        if (s->profile) AG_CUDA(cudaEventRecord(s->ev[2], gs));
        if (sorted) {
            if (!s->rstream) AG_CUDA(workspace_stream(&s->rstream, s->rpriority));
            if (!s->remote_done) AG_CUDA(cudaEventCreateWithFlags(&s->remote_done, cudaEventDisableTiming));
            AG_CUDA(cudaStreamWaitEvent(s->rstream, s->sampled, 0));
            AG_CUDA(launch_sorted_fetch(GatherArgs{}, gather_dev, n_batches, sort_rows, row_bytes, (uint32_t)feats->dim,
                                        feats->dtype, feats, s->sort, gs, s->rstream));
            AG_CUDA(cudaEventRecord(s->remote_done, s->rstream));
            AG_CUDA(cudaStreamWaitEvent(gs, s->remote_done, 0));
        } else {
            AG_CUDA(launch_gather_group(gather_dev, n_batches, row_bytes, (uint32_t)feats->dim, rows, aligned,
                                        feats->dtype, feats->shards != nullptr, gs, gs == st));
        }
        if (s->profile) AG_CUDA(cudaEventRecord(s->ev[3], gs));
        AG_CUDA(cudaEventRecord(s->done, gs));
        if (gs != st) AG_CUDA(cudaStreamWaitEvent(st, s->done, 0));  // the caller's stream stays ordered behind the gather
        s->gathered = true;
    } else {
        AG_CUDA(cudaEventRecord(s->done, st));
    }
    s->in_flight = true;
    s->in_flight_n = n_batches;
    return AG_OK;
}
}  // namespace

// Waits for the group queued last; counts[b] receives batch b's counts.  Returns
// the first batch error (the other batches' counts are still valid).
extern "C" int32_t ag_sample_group_wait(ag_sampler *s, ag_sample_counts *counts, int32_t *statuses) {
    if (!s) return fail(AG_ERR_VALUE, "ag_sample_wait: null sampler");
    if (!s->in_flight) return fail(AG_ERR_VALUE, "ag_sample_wait: no batch in flight");
    DeviceGuard guard(s->device);
    if (!guard.ok) return AG_ERR_CUDA;
    auto wait_done = [&]() -> cudaError_t {
        if (!s->yield_wait) return cudaEventSynchronize(s->done);
        cudaError_t q;
        while ((q = cudaEventQuery(s->done)) == cudaErrorNotReady) sched_yield();
        return q;
    };
    cudaError_t e = wait_done();
    s->in_flight = false;
    if (e == cudaSuccess && s->last.reduced_table) {
        bool full = false;
        for (uint32_t b = 0; b < s->in_flight_n; ++b) full = full || (s->counts_host[b].error & kErrTableFull);
        if (full) {
            // A batch outgrew the table its chain was given: once more, with the full-size tables.
            s->dirty = true;
            s->est_nodes = 0;
            AG_TRY(launch_saved(s, true));
            e = wait_done();
            s->in_flight = false;
        }
    }
    if (e != cudaSuccess) {
        s->dirty = true;
        s->pending_pos = false;
        return fail(AG_ERR_CUDA, "sampling kernels failed: %s", cudaGetErrorString(e));
    }
    account_stream(s);
    float sample_ms = 0.f, gather_ms = 0.f, gather_begin = 0.f;
    if (s->profile) {
        cudaEventElapsedTime(&sample_ms, s->ev[0], s->ev[1]);
        if (s->gathered) {
            cudaEventElapsedTime(&gather_ms, s->ev[2], s->ev[3]);
            if (cudaEvent_t origin = profile_origin(s->device, nullptr)) cudaEventElapsedTime(&gather_begin, origin, s->ev[2]);
        }
    }
    // Next group's grids follow what this one really produced (with headroom).
    uint64_t mx_nodes = 0, mx_items[AG_MAX_HOPS + 2] = {0};
    for (uint32_t b = 0; b < s->in_flight_n; ++b) {
        const ag_sample_counts &c = s->counts_host[b];
        mx_nodes = std::max<uint64_t>(mx_nodes, c.num_nodes);
        for (uint32_t h = 0; h < c.num_hops && h < AG_MAX_HOPS; ++h)
            mx_items[h + 1] = std::max<uint64_t>(mx_items[h + 1], c.edges_per_hop[h]);
    }
    s->est_nodes = mx_nodes + mx_nodes / 4 + 256;
    s->est_rows_tight = mx_nodes + mx_nodes / 16 + 64;
    for (uint32_t h = 1; h <= s->cfg.num_hops; ++h) s->est_items[h] = mx_items[h] + mx_items[h] / 4 + 512;
    int32_t first = AG_OK;
    for (uint32_t b = 0; b < s->in_flight_n; ++b) {
        ag_sample_counts c = s->counts_host[b];
        c.sample_ms = sample_ms / s->in_flight_n;
        c.gather_ms = gather_ms / s->in_flight_n;
        c.gather_begin_ms = gather_begin;
        c.gather_end_ms = (double)gather_begin + gather_ms;
        if (counts) counts[b] = c;
        int32_t st = AG_OK;
        if (c.error & kErrBadSeed) st = fail(AG_ERR_SAMPLING, "a seed node is out of range for %llu nodes", (unsigned long long)s->g->num_nodes);
        else if (c.error & kErrCapacity) st = fail(AG_ERR_VALUE, "output buffers too small for the sampled subgraph");
        else if (c.error & kErrBadDst) st = fail(AG_ERR_LOAD, "graph holds a destination outside [0, num_nodes); load it with full validation");
        else if (c.error) st = fail(AG_ERR_WORKER, "sampler kernels reported error bits 0x%x", c.error);
        if (st != AG_OK && (c.error & (kErrSpinTimeout | kErrTableFull))) s->dirty = true;
        if (statuses) statuses[b] = st;
        if (st != AG_OK && first == AG_OK) first = st;
    }
    return first;
}

extern "C" int32_t ag_sample_into(ag_sampler *s, const uint32_t *seeds, uint64_t n_seeds, int32_t seeds_mem,
                                  const ag_features *feats, ag_subgraph_buffers *buf, void *stream) {
    if (!s || !buf || (!seeds && n_seeds)) return fail(AG_ERR_VALUE, "ag_sample_into: null argument");
    const uint32_t *sp[1] = {seeds};
    const uint64_t ns[1] = {n_seeds};
    return ag_sample_group_into(s, 1, sp, ns, seeds_mem, nullptr, feats, buf, stream);
}

extern "C" int32_t ag_sample_wait(ag_sampler *s, ag_sample_counts *counts) {
    if (s && s->in_flight && s->in_flight_n != 1) return fail(AG_ERR_VALUE, "ag_sample_wait: a group is in flight; use ag_sample_group_wait");
    return ag_sample_group_wait(s, counts, nullptr);
}

extern "C" int32_t ag_sample(ag_sampler *s, const uint32_t *seeds, uint64_t n_seeds, const ag_features *feats,
                             int32_t want_int64, ag_subgraph_buffers *buf, void *stream) {
    if (!s || !buf) return fail(AG_ERR_VALUE, "ag_sample: null argument");
    DeviceGuard guard(s->device);
    if (!guard.ok) return AG_ERR_CUDA;
    uint64_t mn, me;
    compute_bounds(s, n_seeds, &mn, &me, nullptr);
    ag_subgraph_buffers b{};
    b.cap_nodes = std::max<uint64_t>(mn, 1); b.cap_edges = std::max<uint64_t>(me, 1);
    b.cap_seeds = std::max<uint64_t>(n_seeds, 1);
    std::vector<void *> mine;
    auto alloc = [&](void **ptr, uint64_t bytes) -> bool {
        if (device_malloc(ptr, bytes) != cudaSuccess) return false;
        mine.push_back(*ptr);
        return true;
    };
    bool ok = alloc((void **)&b.nodes, b.cap_nodes * 4) && alloc((void **)&b.edge_src, b.cap_edges * 4) &&
              alloc((void **)&b.edge_dst, b.cap_edges * 4) && alloc((void **)&b.src_local, b.cap_edges * 4) &&
              alloc((void **)&b.dst_local, b.cap_edges * 4) && alloc((void **)&b.seed_locals, b.cap_seeds * 4);
    if (ok && s->cfg.track_edge_ids) ok = alloc((void **)&b.edge_ids, b.cap_edges * 8);
    if (ok && want_int64) {
        ok = alloc((void **)&b.n_id, b.cap_nodes * 8) && alloc((void **)&b.edge_index_local, b.cap_edges * 16) &&
             alloc((void **)&b.seed_index, b.cap_seeds * 8);
        if (ok && s->cfg.track_edge_ids) ok = alloc((void **)&b.e_id, b.cap_edges * 8);
    }
    if (ok && feats) ok = alloc((void **)&b.x, b.cap_nodes * feats->dim * 4);
    if (!ok) {
        for (void *q : mine) cudaFree(q);
        return fail(AG_ERR_CUDA, "ag_sample: out of device memory: %s", cudaGetErrorString(cudaGetLastError()));
    }
    const int32_t st = ag_sample_into(s, seeds, n_seeds, AG_MEM_HOST, feats, &b, stream);
    if (st != AG_OK) { for (void *q : mine) cudaFree(q); return st; }
    s->owned.insert(s->owned.end(), mine.begin(), mine.end());
    *buf = b;
    return AG_OK;
}

extern "C" int32_t ag_subgraph_release(ag_sampler *s, ag_subgraph_buffers *buf) {
    if (!s || !buf) return fail(AG_ERR_VALUE, "ag_subgraph_release: null argument");
    DeviceGuard guard(s->device);
    if (s->in_flight) { cudaEventSynchronize(s->done); }
    void *ptrs[] = {buf->nodes, buf->edge_src, buf->edge_dst, buf->edge_ids, buf->src_local, buf->dst_local,
                    buf->seed_locals, buf->n_id, buf->edge_index_local, buf->e_id, buf->seed_index, buf->x};
    for (void *q : ptrs) {
        if (!q) continue;
        auto it = std::find(s->owned.begin(), s->owned.end(), q);
        if (it != s->owned.end()) { cudaFree(q); s->owned.erase(it); }
    }
    *buf = ag_subgraph_buffers{};
    return AG_OK;
}
