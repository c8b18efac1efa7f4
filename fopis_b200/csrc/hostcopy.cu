// hostcopy.cu — copies between the device and a caller's pageable memory.
//
// cudaMemcpy stages pageable memory through one thread: 4.2 GB/s into freshly
// allocated pages (that thread takes every page fault), 9 GB/s out of them,
// where the link carries 54. Here chunks go through a ring of pinned slots, the
// calling thread issuing the device copies and a few threads copying between
// the slots and the caller's memory, so faults and memory copies run in
// parallel and beside the link. A potential of 139 MB into a new array: 33 ->
// 9.6 ms; out of one: 12 -> 6 ms. Smaller copies, and memory that is already
// pinned, go straight to cudaMemcpyAsync.
//
// The pinned ring (8 MB) is shared by the contexts of the process, one copy at a
// time, allocated by the first copy that needs it and freed with the last
// context.
#include "internal.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>

namespace fopis {

namespace {

constexpr size_t kSlot = 512 * 1024;
constexpr int kSlots = 16;
// Below this an allocator that has freed such a block before hands out pages that
// are mapped already, where cudaMemcpy moves 18-20 GB/s and the threads, started for
// each copy, are no faster (18 MB: 1.0 against 1.6 ms); above it every allocation is
// new pages. (A first read of a smaller field pays its page faults here too.)
constexpr size_t kStaged = 32 << 20;

std::mutex g_ring_mutex;
char* g_ring = nullptr;
int g_contexts = 0;

bool pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged || a.type == cudaMemoryTypeDevice;
}

struct Chunk { char *dev, *host; size_t bytes; };

// The counters of one staged copy. Chunk i uses slot i % kSlots and belongs to
// worker i % workers.
struct Ring {
    std::vector<Chunk> chunks;
    std::atomic<int> open{0};                            // chunks below this may be taken up by their worker
    std::unique_ptr<std::atomic<bool>[]> done;           // worker finished with chunk i
    std::atomic<bool> stop{false};
    std::vector<std::thread> threads;

    bool wait(const std::atomic<int>& n, int i) const {
        while (n.load(std::memory_order_acquire) <= i) {
            if (stop.load(std::memory_order_relaxed)) return false;
            std::this_thread::yield();
        }
        return true;
    }
    void wait_done(int i) const {
        while (!done[i].load(std::memory_order_acquire)) std::this_thread::yield();
    }
    // False when the system gives no threads: the caller copies plainly.
    bool start(bool to_host) {
        done.reset(new std::atomic<bool>[chunks.size()]);
        for (size_t i = 0; i < chunks.size(); ++i) done[i].store(false);
        const int cores = (int)std::thread::hardware_concurrency();
        const int workers = std::max(1, std::min({8, cores / 2, (int)chunks.size() / 2}));
        auto work = [this, workers, to_host](int w) {
            for (int i = w; i < (int)chunks.size(); i += workers) {
                if (!wait(open, i)) return;
                char* slot = g_ring + (size_t)(i % kSlots) * kSlot;
                if (to_host) std::memcpy(chunks[i].host, slot, chunks[i].bytes);
                else std::memcpy(slot, chunks[i].host, chunks[i].bytes);
                done[i].store(true, std::memory_order_release);
            }
        };
        try {
            for (int w = 0; w < workers; ++w) threads.emplace_back(work, w);
        } catch (const std::system_error&) {
            end();
            return false;
        }
        return true;
    }
    void end() {
        stop.store(true);
        for (auto& t : threads) t.join();
        threads.clear();
    }
    ~Ring() { end(); }
};

// Waits for the copies between the device and the slots when a copy ends early, by
// an error: the next one, another context's perhaps, fills the slots anew.
struct Drain {
    cudaStream_t st;
    bool staged = false;
    ~Drain() { if (staged) cudaStreamSynchronize(st); }
};

// Takes the ring and cuts the segments into chunks; false when the copy should
// not be staged.
bool begin(Ctx& c, const CopySegment* s, int n, Ring& r, std::unique_lock<std::mutex>& lock) {
    size_t total = 0;
    for (int q = 0; q < n; ++q) total += s[q].bytes;
    if (total < kStaged) return false;
    for (int q = 0; q < n; ++q) if (pinned(s[q].host)) return false;
    lock = std::unique_lock<std::mutex>(g_ring_mutex);
    if (!g_ring && cudaHostAlloc((void**)&g_ring, kSlots * kSlot, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_ring = nullptr;
        lock.unlock();
        return false;
    }
    if (!c.copy_ev[0])
        for (auto& e : c.copy_ev) FOPIS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (int q = 0; q < n; ++q)
        for (size_t off = 0; off < s[q].bytes; off += kSlot)
            r.chunks.push_back(Chunk{(char*)s[q].dev + off, (char*)s[q].host + off, std::min(kSlot, s[q].bytes - off)});
    return true;
}

}  // namespace

static_assert(sizeof(Ctx::copy_ev) / sizeof(cudaEvent_t) == kSlots, "an event per slot");

void hostcopy_open() {
    std::lock_guard<std::mutex> lock(g_ring_mutex);
    ++g_contexts;
}

void hostcopy_close(Ctx& c) {
    for (auto& e : c.copy_ev) if (e) { cudaEventDestroy(e); e = nullptr; }
    std::lock_guard<std::mutex> lock(g_ring_mutex);
    if (--g_contexts == 0 && g_ring) {
        cudaFreeHost(g_ring);
        g_ring = nullptr;
    }
}

// Device to host in stream order; the memory is filled when it returns.
void copy_to_host(Ctx& c, const CopySegment* s, int n) {
    std::unique_lock<std::mutex> lock;   // released after the threads are joined and the slots at rest
    Drain drain{c.st};
    Ring r;
    if (!begin(c, s, n, r, lock) || !r.start(true)) {
        for (int q = 0; q < n; ++q)
            FOPIS_CUDA(cudaMemcpyAsync(s[q].host, s[q].dev, s[q].bytes, cudaMemcpyDeviceToHost, c.st));
        FOPIS_CUDA(cudaStreamSynchronize(c.st));
        return;
    }
    drain.staged = true;
    const int total = (int)r.chunks.size();
    for (int issued = 0, landed = 0; landed < total;) {
        if (issued < total && issued - landed < kSlots &&
            (issued < kSlots || r.done[issued - kSlots].load(std::memory_order_acquire))) {
            const Chunk& k = r.chunks[issued];
            FOPIS_CUDA(cudaMemcpyAsync(g_ring + (size_t)(issued % kSlots) * kSlot, k.dev, k.bytes, cudaMemcpyDeviceToHost, c.st));
            FOPIS_CUDA(cudaEventRecord(c.copy_ev[issued % kSlots], c.st));
            ++issued;
        } else if (landed < issued) {
            FOPIS_CUDA(cudaEventSynchronize(c.copy_ev[landed % kSlots]));
            r.open.store(++landed, std::memory_order_release);
        } else {
            std::this_thread::yield();   // every slot waits for its worker
        }
    }
    for (int i = 0; i < total; ++i) r.wait_done(i);
    drain.staged = false;
}

// Host to device in stream order; the memory has been read when it returns,
// without wait only once the stream has passed.
void copy_to_device(Ctx& c, const CopySegment* s, int n, bool wait) {
    std::unique_lock<std::mutex> lock;
    Drain drain{c.st};
    Ring r;
    const bool staged = begin(c, s, n, r, lock);
    const int total = (int)r.chunks.size();
    r.open.store(std::min(total, kSlots));
    if (!staged || !r.start(false)) {
        for (int q = 0; q < n; ++q)
            FOPIS_CUDA(cudaMemcpyAsync(s[q].dev, s[q].host, s[q].bytes, cudaMemcpyHostToDevice, c.st));
        if (wait) FOPIS_CUDA(cudaStreamSynchronize(c.st));
        return;
    }
    drain.staged = true;
    for (int i = 0; i < total; ++i) {
        r.wait_done(i);
        const Chunk& k = r.chunks[i];
        FOPIS_CUDA(cudaMemcpyAsync(k.dev, g_ring + (size_t)(i % kSlots) * kSlot, k.bytes, cudaMemcpyHostToDevice, c.st));
        FOPIS_CUDA(cudaEventRecord(c.copy_ev[i % kSlots], c.st));
        const int back = i - kSlots / 2;   // keep half the ring on the link, hand the rest to the workers
        if (back >= 0 && back + kSlots < total) {
            FOPIS_CUDA(cudaEventSynchronize(c.copy_ev[back % kSlots]));
            r.open.store(back + kSlots + 1, std::memory_order_release);
        }
    }
    drain.staged = false;
    FOPIS_CUDA(cudaStreamSynchronize(c.st));   // the slots are free for the next copy
}

}  // namespace fopis
