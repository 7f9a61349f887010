// Copies into pageable host memory through a pinned buffer (see host_copy.h).
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace emg {
namespace {

constexpr size_t CHUNK = 2u << 20;   // bytes per slot
constexpr int SLOTS = 16;            // 32 MB pinned, two slots per thread
constexpr size_t MIN_BYTES = 8u << 20;  // below this the plain copy costs less than starting threads

std::mutex buffer_mu;  // held for the length of a staged copy: one at a time uses the buffer
unsigned char* buffer = nullptr;

// The buffer, page-locked for every device; null when there is none to be had. It
// is host memory of the library's own that is registered with the driver, so a
// device reset takes the page lock and not the memory: it is then locked again.
unsigned char* locked_buffer() {
    if (!buffer) buffer = static_cast<unsigned char*>(std::aligned_alloc(CHUNK, CHUNK * SLOTS));
    if (!buffer) return nullptr;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, buffer) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (at.type != cudaMemoryTypeHost && cudaHostRegister(buffer, CHUNK * SLOTS, cudaHostRegisterPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return buffer;
}

// host threads emptying the slots: at most one per two slots
int worker_count() {
    const unsigned n = std::thread::hardware_concurrency();
    return (int)std::min<unsigned>(SLOTS / 2, std::max(1u, n / 2));
}

}  // namespace

void release_host_buffer() {
    std::lock_guard<std::mutex> lock(buffer_mu);  // waits for a copy that uses it
    if (!buffer) return;
    if (cudaHostUnregister(buffer) != cudaSuccess) cudaGetLastError();
    std::free(buffer);
    buffer = nullptr;
}

cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    auto plain = [&] {
        const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
        return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
    };
    if (bytes < MIN_BYTES) return plain();
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
        cudaGetLastError();
        return plain();
    }
    if (at.type != cudaMemoryTypeUnregistered) return plain();  // pinned: full link speed already
    std::unique_lock<std::mutex> lock(buffer_mu, std::try_to_lock);
    const int nw = worker_count();
    if (!lock.owns_lock() || nw < 2) return plain();
    if (!locked_buffer()) return plain();
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    std::atomic<int> failed{(int)cudaSuccess};
    // worker w moves chunks w, w + nw, ...: the next one crosses the bus into its
    // second slot while it copies the one before out of the first
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(dev);
        cudaEvent_t ev[2] = {nullptr, nullptr};
        for (auto& x : ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
        unsigned char* slot[2] = {buffer + (size_t)(2 * w) * CHUNK, buffer + (size_t)(2 * w + 1) * CHUNK};
        auto fetch = [&](size_t c, int b) {
            const size_t off = c * CHUNK, n = std::min(CHUNK, bytes - off);
            e = cudaMemcpyAsync(slot[b], static_cast<const unsigned char*>(src) + off, n, cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaEventRecord(ev[b], stream);
        };
        int b = 0;
        if (e == cudaSuccess && (size_t)w < chunks) fetch((size_t)w, 0);
        for (size_t c = (size_t)w; e == cudaSuccess && c < chunks; c += (size_t)nw, b ^= 1) {
            if (c + nw < chunks) fetch(c + nw, b ^ 1);
            if (e != cudaSuccess) break;
            e = cudaEventSynchronize(ev[b]);
            if (e == cudaSuccess)
                std::memcpy(static_cast<unsigned char*>(dst) + c * CHUNK, slot[b], std::min(CHUNK, bytes - c * CHUNK));
        }
        for (auto& x : ev)
            if (x) cudaEventDestroy(x);
        if (e != cudaSuccess) failed.store((int)e);
    };
    std::vector<std::thread> threads;
    int started = 1;
    try {
        threads.reserve((size_t)nw);
        for (; started < nw; started++) threads.emplace_back(work, started);
    } catch (...) {  // no thread to be had: this one takes the shares that are left
    }
    work(0);
    for (int w = started; w < nw; w++) work(w);
    for (auto& t : threads) t.join();
    if (failed.load() != (int)cudaSuccess) {
        cudaStreamSynchronize(stream);  // nothing may still write to the buffer
        return (cudaError_t)failed.load();
    }
    return cudaSuccess;
}

}  // namespace emg
