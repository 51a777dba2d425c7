// Large copies between ordinary (pageable) host memory and the device.
//
// The runtime stages a pageable copy through page-locked memory with one
// thread: 8-10 GB/s to the device, 21 GB/s back into memory already touched and
// 4-5 GB/s into fresh pages, which that thread also has to fault in; the link
// carries 50. Here several threads move the chunks of a copy through a block of
// page-locked slots (two per thread, so that a thread fills or empties one
// while the other travels). Whole calls with ordinary NumPy arrays, before and
// after: construct_umap_graph at 1M points, k = 15 (120 MB up, 250 MB down; a
// copy of its results left out at the same time) 127 -> 28.5 ms, densMAP layout
// of 200k points, k = 30 (72 MB up) 19.5 -> 16.0, exact kNN of 200k points (24 MB
// up, 48 down) 20.8 -> 15.8 ms.
//
// The block is one per process, page-locked for every device, allocated at the
// first large copy and given back by umapcu_release_cached. A copy that finds
// it taken by another thread's goes through the runtime as before, and so does
// one whose context is not its device's primary one: the helping threads, and
// the block, belong to primary contexts.
#include <cuda.h>

#include <atomic>
#include <mutex>
#include <thread>

#include "internal.cuh"

namespace umapcu {
namespace {

constexpr size_t kChunk = (size_t)1 << 20;
constexpr unsigned kMaxThreads = 8;
// Copies below these gain nothing over the runtime's: starting the threads takes
// 0.1-0.2 ms. Up, from touched pages: 4 MB 0.24 (the runtime) and 0.26 ms, 8 MB
// 0.45 and 0.42, 16 MB 0.83 and 0.62. Down into touched pages, as the allocator
// hands them out again: 6 MB 0.46 and 0.54, 16 MB 1.18 and 1.08, 32 MB 2.3 and
// 1.5; into fresh ones 8 MB 1.7 and 0.83, 32 MB 6.6 and 1.8.
constexpr size_t kLeastUp = (size_t)8 << 20, kLeastDown = (size_t)16 << 20;

std::mutex g_mu;
uint8_t *g_block = nullptr;  // the idle block; null while taken or not allocated
bool g_taken = false;

unsigned copy_threads()
{
    static const unsigned n = std::min(kMaxThreads, std::thread::hardware_concurrency() / 2);
    return n;
}

// Whether the calling thread's context is the primary one of device dev.
bool primary_context(int dev)
{
    struct Calls {
        decltype(&cuCtxGetCurrent) current = nullptr;
        decltype(&cuDevicePrimaryCtxRetain) retain = nullptr;
        decltype(&cuDevicePrimaryCtxRelease) release = nullptr;
        Calls()
        {
            auto get = [](const char *name, auto &f) {
                cudaDriverEntryPointQueryResult found;
                void *p = nullptr;
                if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &found) == cudaSuccess &&
                    found == cudaDriverEntryPointSuccess)
                    f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(p);
                else cudaGetLastError();
            };
            get("cuCtxGetCurrent", current);
            get("cuDevicePrimaryCtxRetain", retain);
            get("cuDevicePrimaryCtxRelease", release);
        }
    };
    static const Calls f;
    if (!f.current || !f.retain || !f.release) return false;
    CUcontext mine = nullptr, primary = nullptr;
    // (a runtime device is the driver's of the same number)
    if (f.current(&mine) != CUDA_SUCCESS || !mine || f.retain(&primary, dev) != CUDA_SUCCESS) return false;
    f.release(dev);
    return mine == primary;
}

struct Block {
    uint8_t *p = nullptr;
    bool mine = false;
    Block()
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_taken) return;
        if (!g_block &&
            cudaHostAlloc((void **)&g_block, 2 * kChunk * copy_threads(), cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            g_block = nullptr;
            return;
        }
        p = g_block;
        g_block = nullptr;
        g_taken = mine = true;
    }
    ~Block()
    {
        if (!mine) return;
        std::lock_guard<std::mutex> lk(g_mu);
        g_block = p;
        g_taken = false;
    }
    Block(const Block &) = delete;
    Block &operator=(const Block &) = delete;
};

struct Slot {
    uint8_t *p = nullptr;
    cudaEvent_t done = nullptr;
    size_t at = 0, bytes = 0;  // the chunk on its way
    cudaError_t init(uint8_t *mem)
    {
        p = mem;
        return cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
    }
    ~Slot()
    {
        if (!done) return;
        cudaEventSynchronize(done);  // the slot's memory outlives its copy
        cudaEventDestroy(done);
    }
};

// One thread's share: chunks taken from `next` until none is left.
cudaError_t move_chunks(uint8_t *dst, const uint8_t *src, size_t bytes, bool to_device, uint8_t *mem,
                        std::atomic<size_t> &next, cudaStream_t s)
{
    Slot slot[2];
    cudaError_t e;
    for (int i = 0; i < 2; i++)
        if ((e = slot[i].init(mem + i * kChunk)) != cudaSuccess) return e;
    auto finish = [&](Slot &k) {  // the slot's chunk has arrived
        if (!k.bytes) return cudaSuccess;
        const cudaError_t r = cudaEventSynchronize(k.done);
        if (r == cudaSuccess && !to_device) memcpy(dst + k.at, k.p, k.bytes);
        k.bytes = 0;
        return r;
    };
    for (int i = 0;; i ^= 1) {
        const size_t at = next.fetch_add(kChunk);
        if (at >= bytes) {
            e = finish(slot[i]);
            const cudaError_t f = finish(slot[i ^ 1]);
            return e != cudaSuccess ? e : f;
        }
        Slot &k = slot[i];
        if ((e = finish(k)) != cudaSuccess) return e;
        k.at = at;
        k.bytes = std::min(kChunk, bytes - at);
        if (to_device) {
            memcpy(k.p, src + at, k.bytes);
            e = cudaMemcpyAsync(dst + at, k.p, k.bytes, cudaMemcpyHostToDevice, s);
        } else {
            e = cudaMemcpyAsync(k.p, src + at, k.bytes, cudaMemcpyDeviceToHost, s);
        }
        if (e == cudaSuccess) e = cudaEventRecord(k.done, s);
        if (e != cudaSuccess) {
            k.bytes = 0;
            return e;
        }
    }
}

}  // namespace

bool staged_copy(void *dst, const void *src, size_t bytes, bool to_device, cudaStream_t s)
{
    if (bytes < (to_device ? kLeastUp : kLeastDown) || copy_threads() < 2) return false;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, to_device ? src : dst) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type != cudaMemoryTypeUnregistered) return false;  // page-locked already
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (!primary_context(dev)) return false;
    Block block;
    if (!block.p) return false;
    if (!to_device) sync(s);  // not by the copying threads, which would spin
    const unsigned n = (unsigned)std::min<size_t>(copy_threads(), (bytes + kChunk - 1) / kChunk);
    std::atomic<size_t> next{0};
    cudaError_t err[kMaxThreads] = {};
    auto work = [&](unsigned t) {
        if (t) err[t] = cudaSetDevice(dev);  // the calling thread's context is as it should be
        if (err[t] == cudaSuccess)
            err[t] = move_chunks(static_cast<uint8_t *>(dst), static_cast<const uint8_t *>(src), bytes, to_device,
                                 block.p + 2 * kChunk * t, next, s);
    };
    std::vector<std::thread> threads;
    threads.reserve(n);
    try {
        for (unsigned t = 1; t < n; t++) threads.emplace_back(work, t);
    } catch (const std::exception &) {  // fewer threads then: the chunks are shared out as they go
    }
    work(0);
    for (std::thread &t : threads) t.join();
    for (unsigned t = 0; t < n; t++) check_cuda(err[t], "staged copy");
    return true;
}

void release_copy_block()
{
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_block) cudaFreeHost(g_block);
    g_block = nullptr;
}

}  // namespace umapcu
