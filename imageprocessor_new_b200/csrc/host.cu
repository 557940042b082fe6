// Large results into ordinary host memory.
//
// A device copy into pageable memory runs at some 10 GB/s (the driver stages it and one thread copies
// and takes the destination's page faults); a page-locked result would be fast but stay page-locked for
// as long as the caller keeps it. Here the data comes in chunks into a few pinned slots and a few host
// threads copy the chunks out as they land, so the transfer, the copies and the faults overlap: 30 MB
// in 1.0 instead of 1.8 ms, 120 MB (its pages fresh from the system each time) in 7.6 instead of 57 ms with
// 2 MB chunks and eight threads; up to 8 MB the direct copy is as fast.

#include <string.h>

#include <algorithm>
#include <atomic>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"

using namespace spx;

namespace {

constexpr int kMaxSlots = 16;
constexpr int kMaxThreads = 8;

struct Transfer {
    char* dst;
    const char* pinned;
    size_t bytes, chunk;
    int chunks, slots, device;
    cudaEvent_t event[kMaxSlots];
    std::atomic<int> issued{0};             // chunks whose device copy and event are queued
    std::atomic<int> next{0};               // next chunk a thread takes
    std::atomic<int> landed[kMaxSlots];     // chunks copied out of each slot
    std::atomic<bool> failed{false};

    void copy_out(int k) {
        const int slot = k % slots;
        if (cudaEventSynchronize(event[slot]) != cudaSuccess) failed = true;
        const size_t lo = (size_t)k * chunk, n = std::min(chunk, bytes - lo);
        if (!failed) memcpy(dst + lo, pinned + (size_t)slot * chunk, n);
        landed[slot].fetch_add(1, std::memory_order_release);
    }
    void work() {
        cudaSetDevice(device);
        for (int k = next.fetch_add(1); k < chunks; k = next.fetch_add(1)) {
            while (issued.load(std::memory_order_acquire) <= k && !failed) std::this_thread::yield();
            if (issued.load(std::memory_order_acquire) <= k) return;
            copy_out(k);
        }
    }
};

}  // namespace

extern "C" {

int spx_download(void* dst, const void* src, size_t bytes, void* pinned, size_t pinned_bytes, size_t chunk, int threads,
                 void* stream) {
    SPX_REQUIRE(chunk > 0 && pinned_bytes >= chunk && threads >= 1, "bad arguments");
    if (bytes == 0) return SPX_OK;
    SPX_REQUIRE(dst && src && pinned, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Transfer t;
    t.dst = static_cast<char*>(dst);
    t.pinned = static_cast<const char*>(pinned);
    t.bytes = bytes;
    t.chunk = chunk;
    t.chunks = (int)((bytes + chunk - 1) / chunk);
    t.slots = (int)std::min<size_t>({(size_t)kMaxSlots, pinned_bytes / chunk, (size_t)t.chunks});
    SPX_CUDA(cudaGetDevice(&t.device));
    int made = 0;
    cudaError_t err = cudaSuccess;
    for (; made < t.slots && err == cudaSuccess; ++made) {
        t.landed[made] = 0;
        err = cudaEventCreateWithFlags(&t.event[made], cudaEventDisableTiming);
    }
    if (err != cudaSuccess) --made;
    std::vector<std::thread> pool;
    if (err == cudaSuccess) {
        try {
            pool.reserve(kMaxThreads);
            for (int i = 0; i < std::min({threads, kMaxThreads, t.chunks}); ++i) pool.emplace_back([&t] { t.work(); });
        } catch (const std::exception&) {
            // Fewer threads than asked for; with none this thread copies the chunks out itself, below.
        }
        for (int k = 0; k < t.chunks && err == cudaSuccess && !t.failed; ++k) {
            const int slot = k % t.slots, round = k / t.slots;
            // The slot's previous chunk has been copied out (by a thread, or here when there is none).
            while (t.landed[slot].load(std::memory_order_acquire) < round && !t.failed) {
                if (pool.empty()) t.copy_out(t.next.fetch_add(1));
                else std::this_thread::yield();
            }
            const size_t lo = (size_t)k * chunk;
            err = cudaMemcpyAsync(static_cast<char*>(pinned) + (size_t)slot * chunk, static_cast<const char*>(src) + lo,
                                  std::min(chunk, bytes - lo), cudaMemcpyDeviceToHost, s);
            if (err == cudaSuccess) err = cudaEventRecord(t.event[slot], s);
            if (err == cudaSuccess) t.issued.store(k + 1, std::memory_order_release);
        }
        if (err != cudaSuccess) t.failed = true;
        if (pool.empty() && !t.failed)
            for (int k = t.next.load(); k < t.chunks; ++k) t.copy_out(k);
        for (std::thread& th : pool) th.join();
    }
    const bool failed = t.failed;
    if (failed || err != cudaSuccess) cudaStreamSynchronize(s);  // no copy into the slots outlives the call
    for (int i = 0; i < made; ++i) cudaEventDestroy(t.event[i]);
    if (err == cudaSuccess && failed) err = cudaGetLastError();
    if (err != cudaSuccess || failed) {
        set_error("download failed: %s", cudaGetErrorString(err));
        return SPX_ERR_CUDA;
    }
    return SPX_OK;
}

}  // extern "C"
