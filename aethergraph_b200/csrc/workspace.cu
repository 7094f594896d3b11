// Device memory, pinned memory and streams that short-lived handles use and give back.
//
// An epoch driver makes a loader per epoch and drops it: twenty scratch arrays per
// worker, two arrays per batch in flight, streams and staging buffers.  cudaMalloc and
// cudaFree of megabytes take 0.3 - 1.7 ms each while kernels run (cudaFree waits for the
// whole device), so ten batches of 128 seeds spent 12 - 24 ms on 0.3 ms of kernels.
// Blocks that a handle gives back are kept for the next handle that asks for about the size.
//
//   * Bounded: kMaxHeld bytes per device and kMaxHeldHost pinned; the blocks kept longest go first.
//   * Given back: when the last graph and feature store are freed, and whenever a device
//     allocation of the library fails, which is then tried again (device_malloc).  Another
//     allocator of the process asks for it with ag_release_kept_memory.
//   * Ordered: a block is given back only once all work on it has finished, so the next
//     owner needs no event; contents are whatever they were.
//   * One lock, held for list operations only; any thread may take and give.
#include <list>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace ag {
namespace {

constexpr size_t kMaxHeld = 512ull << 20;
constexpr size_t kMaxHeldHost = 64ull << 20;
constexpr size_t kMaxStreams = 16;  // idle streams kept per device and priority
constexpr int kHost = -1;           // the "device" of pinned blocks

struct Block {
    int device;
    size_t bytes;
    void *ptr;
};
struct IdleStream {
    int device, priority;
    cudaStream_t stream;
};

struct Cache {
    std::mutex m;
    std::list<Block> idle;                     // oldest first
    std::unordered_map<int, size_t> held;      // bytes in `idle` per device
    std::unordered_map<void *, Block> live;
    std::vector<IdleStream> streams;
    uint64_t users = 0;
};
Cache &cache() {  // never destroyed: handles may be freed during process exit
    static Cache *c = new Cache();
    return *c;
}

// What is asked of the driver for a block.  Large blocks: whole 2 MiB pages, which the driver
// maps in any case, so that a loader of several GB holds no more than it asked for.  Below that
// eight sizes per power of two, so that requests which differ from call to call meet again.
constexpr size_t kPage = 2ull << 20;
size_t block_size(size_t bytes) {
    if (bytes >= kPage) return (bytes + kPage - 1) / kPage * kPage;
    size_t step = 512;
    while (step * 16 <= bytes) step *= 2;
    return (std::max<size_t>(bytes, 1) + step - 1) / step * step;
}

void really_free(const std::vector<Block> &blocks) {
    for (const Block &b : blocks) {
        if (b.device == kHost) { cudaFreeHost(b.ptr); continue; }
        DeviceGuard guard(b.device);
        cudaFree(b.ptr);
    }
}

// Caller holds the lock.
void take_idle(Cache &c, bool everything, int device, size_t keep, std::vector<Block> *out) {
    for (auto it = c.idle.begin(); it != c.idle.end();) {
        if (everything || (it->device == device && c.held[device] > keep)) {
            c.held[it->device] -= it->bytes;
            out->push_back(*it);
            it = c.idle.erase(it);
        } else {
            ++it;
        }
    }
}

void drop_all() {
    Cache &c = cache();
    std::vector<Block> blocks;
    std::vector<IdleStream> streams;
    {
        std::lock_guard<std::mutex> lk(c.m);
        take_idle(c, true, 0, 0, &blocks);
        streams.swap(c.streams);
    }
    really_free(blocks);
    for (const IdleStream &s : streams) { DeviceGuard guard(s.device); cudaStreamDestroy(s.stream); }
}

cudaError_t take(int device, void **out, size_t bytes) {
    Cache &c = cache();
    const size_t want = block_size(bytes);
    *out = nullptr;
    {
        // the smallest kept block that holds the request and is at most an eighth larger
        std::lock_guard<std::mutex> lk(c.m);
        auto best = c.idle.end();
        for (auto it = c.idle.begin(); it != c.idle.end(); ++it) {
            if (it->device != device || it->bytes < want || it->bytes > want + want / 8) continue;
            if (best == c.idle.end() || it->bytes <= best->bytes) best = it;  // of equal ones the newest
        }
        if (best != c.idle.end()) {
            const Block b = *best;
            c.idle.erase(best);
            c.held[device] -= b.bytes;
            c.live.emplace(b.ptr, b);
            *out = b.ptr;
            return cudaSuccess;
        }
    }
    void *p = nullptr;
    cudaError_t e;
    if (device == kHost) {
        e = cudaHostAlloc(&p, want, cudaHostAllocDefault);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            drop_all();
            e = cudaHostAlloc(&p, want, cudaHostAllocDefault);
        }
    } else {
        e = device_malloc(&p, want);
    }
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(c.m);
    c.live.emplace(p, Block{device, want, p});
    *out = p;
    return cudaSuccess;
}

void give(void *p) {
    if (!p) return;
    Cache &c = cache();
    std::vector<Block> out;
    {
        std::lock_guard<std::mutex> lk(c.m);
        auto it = c.live.find(p);
        if (it == c.live.end()) return;
        const Block b = it->second;
        c.live.erase(it);
        const size_t limit = b.device == kHost ? kMaxHeldHost : kMaxHeld;
        if (c.users == 0 || b.bytes > limit) {
            out.push_back(b);
        } else {
            take_idle(c, false, b.device, limit - b.bytes, &out);
            c.idle.push_back(b);
            c.held[b.device] += b.bytes;
        }
    }
    really_free(out);
}

}  // namespace

cudaError_t device_malloc(void **out, size_t bytes) {
    const cudaError_t e = cudaMalloc(out, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    drop_all();
    return cudaMalloc(out, bytes);
}

void workspace_drop() { drop_all(); }

cudaError_t workspace_alloc(void **out, size_t bytes) {
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) { *out = nullptr; return e; }
    return take(device, out, bytes);
}
cudaError_t workspace_alloc_host(void **out, size_t bytes) { return take(kHost, out, bytes); }
void workspace_free(void *p) { give(p); }

cudaError_t workspace_stream(cudaStream_t *out, int priority) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    {
        Cache &c = cache();
        std::lock_guard<std::mutex> lk(c.m);
        for (size_t i = 0; i < c.streams.size(); ++i) {
            if (c.streams[i].device != device || c.streams[i].priority != priority) continue;
            *out = c.streams[i].stream;
            c.streams[i] = c.streams.back();
            c.streams.pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreateWithPriority(out, cudaStreamNonBlocking, priority);
}

void workspace_stream_free(cudaStream_t stream, int priority) {
    if (!stream) return;
    int device = 0;
    Cache &c = cache();
    if (cudaGetDevice(&device) == cudaSuccess) {
        std::lock_guard<std::mutex> lk(c.m);
        size_t same = 0;
        for (const IdleStream &s : c.streams) same += s.device == device && s.priority == priority;
        if (c.users && same < kMaxStreams) {
            c.streams.push_back(IdleStream{device, priority, stream});
            return;
        }
    }
    cudaStreamDestroy(stream);
}

WorkspaceUser::WorkspaceUser() {
    Cache &c = cache();
    std::lock_guard<std::mutex> lk(c.m);
    ++c.users;
}
WorkspaceUser::WorkspaceUser(const WorkspaceUser &) : WorkspaceUser() {}
WorkspaceUser::~WorkspaceUser() {
    bool last;
    {
        Cache &c = cache();
        std::lock_guard<std::mutex> lk(c.m);
        last = --c.users == 0;
    }
    if (last) drop_all();
}

}  // namespace ag

extern "C" void ag_release_kept_memory(void) { ag::workspace_drop(); }
