// Host arrays of a call on their way to the device and back (HostIo), with the
// pinned memory they are staged through (PinPool).  Host code only, so that it
// can be tested against a stand-in for the CUDA runtime.
#pragma once

#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>

namespace bbrt {

// A grow-only device buffer, freed when it goes out of scope.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    cudaError_t ensure(size_t n) {
        if (n <= bytes) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaSuccess) bytes = n;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
};

// Pinned host memory for calls on host arrays (HostIo), shared by the scenes:
// pinning 1 MB takes about a millisecond, more than a small call.  A call
// borrows a block and gives it back; there are at most kMax of each kind, and
// all are freed with the last scene.  A call that gets none (all are out, or
// the system pins no more) copies without.
class PinPool {
public:
    static constexpr int kSlots = 16;
    static constexpr size_t kSlot = 512 << 10;
    static constexpr size_t kBytes[2] = { 1 << 20, kSlots * kSlot };   // a small call's block; slots of a large one
    static constexpr int kMax[2] = { 16, 4 };
    static PinPool& get() {
        static PinPool* p = new PinPool;   // outlives the last scene
        return *p;
    }
    // A block, or null.
    char* take(int kind) {
        {
            std::lock_guard<std::mutex> g(mu_);
            if (n_[kind] > 0) return free_[kind][--n_[kind]];
            if (made_[kind] == kMax[kind]) return nullptr;
            ++made_[kind];
        }
        void* p = nullptr;
        if (cudaHostAlloc(&p, kBytes[kind], cudaHostAllocPortable) == cudaSuccess) return static_cast<char*>(p);
        cudaGetLastError();
        std::lock_guard<std::mutex> g(mu_);
        --made_[kind];
        return nullptr;
    }
    void give(int kind, char* p) {
        std::lock_guard<std::mutex> g(mu_);
        free_[kind][n_[kind]++] = p;
    }
    // A scene's share in the pool's life; its calls have ended when it goes.
    struct User {
        User() {
            PinPool& p = get();
            std::lock_guard<std::mutex> g(p.mu_);
            ++p.users_;
        }
        ~User() {
            PinPool& p = get();
            std::lock_guard<std::mutex> g(p.mu_);
            if (--p.users_ > 0) return;
            for (int k = 0; k < 2; ++k)
                for (; p.n_[k] > 0; --p.made_[k]) cudaFreeHost(p.free_[k][--p.n_[k]]);
        }
        User(const User&) = delete;
        User& operator=(const User&) = delete;
    };

private:
    std::mutex mu_;
    char* free_[2][16] = {};
    int n_[2] = { 0, 0 }, made_[2] = { 0, 0 };
    int users_ = 0;
};

// The host arrays of one call on their way to the device and back.  A copy
// from or to pageable memory goes through the driver's staging on one thread
// (about 4 GB/s into pages that are not yet there) and costs several
// microseconds however small, so, by the call's bytes:
//   at most kZeroCopy    the kernels read and write a pinned block, no copies
//                        (96 queries: 58 us, 67 with one copy each way, 75
//                        with the driver's staging; 61 recorded paths 142,
//                        148, 258 us);
//   at most kOneCopy     one copy each way between that block and the device
//                        (inputs of at most that, whatever the outputs: 4,099
//                        rays with 1.8 MB of results 0.38 ms, in chunks 0.48);
//   more                 array by array: chunks through pinned slots by several
//                        threads, which also spread the page faults of the
//                        caller's arrays (262,147 recorded paths, 97 MB of
//                        results: 24 ms with the driver's staging, 8.4 ms this
//                        way on 16 cores); pinned arrays are copied directly.
// Array by array too, at any size, where an array is device memory (its copy is
// CUDA's to make or to refuse: the host cannot read it), and with the driver's
// staging where the pool has no block.
struct HostIo {
    static constexpr size_t kZeroCopy = 64 << 10, kOneCopy = PinPool::kBytes[0], kChunk = PinPool::kSlot;
    static constexpr int kMaxArrays = 12, kMaxThreads = PinPool::kSlots;
    struct Array {
        char* host;
        size_t bytes, off;
        bool in, direct;   // direct: one CUDA copy from or to the caller's memory
    };
    DevBuf& block;       // the scene's device block ...
    cudaEvent_t* slot_ev;   // ... and its event per copying thread (created here)
    int device;
    cudaStream_t st;
    Array a[kMaxArrays];
    int n = 0;
    size_t in_bytes = 0, total = 0;
    char* base = nullptr;   // the block the kernels use
    char* held[2] = { nullptr, nullptr };   // pinned memory borrowed from the pool

    HostIo(DevBuf& block_, cudaEvent_t* slot_ev_, int device_, cudaStream_t st_)
        : block(block_), slot_ev(slot_ev_), device(device_), st(st_) {}
    HostIo(const HostIo&) = delete;
    HostIo& operator=(const HostIo&) = delete;
    ~HostIo() {
        if (opened && !done) cudaStreamSynchronize(st);   // a failed call: nothing may still use the memory
        for (int k = 0; k < 2; ++k)
            if (held[k]) PinPool::get().give(k, held[k]);
    }

    // Inputs first, then outputs (a null array is skipped); at(i) after open().
    int add(const void* host, size_t bytes, bool in) {
        if (!host || bytes == 0) return -1;
        a[n] = { static_cast<char*>(const_cast<void*>(host)), bytes, total, in, false };
        total += (bytes + 255) & ~static_cast<size_t>(255);
        if (in) in_bytes = total;
        return n++;
    }
    template <class T>
    T* at(int i) const { return i < 0 ? nullptr : reinterpret_cast<T*>(base + a[i].off); }

    cudaError_t open() {
        opened = true;
        by_array[0] = total > kOneCopy;      // outputs
        by_array[1] = in_bytes > kOneCopy;   // inputs
        for (int k = 0; k < n; ++k) {
            cudaPointerAttributes pa;
            if (cudaPointerGetAttributes(&pa, a[k].host) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            a[k].direct = pa.type == cudaMemoryTypeDevice || (pa.type == cudaMemoryTypeHost && total > kOneCopy);
            by_array[a[k].in] |= a[k].direct;
        }
        if (!by_array[0] || !by_array[1]) {
            held[0] = PinPool::get().take(0);
            if (!held[0]) by_array[0] = by_array[1] = true;
        }
        if (!by_array[0] && !by_array[1] && total <= kZeroCopy) {
            base = held[0];
        } else {
            const cudaError_t e = block.ensure(total);
            if (e != cudaSuccess) return e;
            base = static_cast<char*>(block.p);
        }
        if (by_array[1]) return arrays(true);
        for (int k = 0; k < n; ++k)
            if (a[k].in) std::memcpy(held[0] + a[k].off, a[k].host, a[k].bytes);
        if (base == held[0] || !in_bytes) return cudaSuccess;
        return cudaMemcpyAsync(base, held[0], in_bytes, cudaMemcpyHostToDevice, st);
    }

    // The results are in the caller's arrays when this returns.
    cudaError_t close() {
        cudaError_t e = cudaSuccess;
        if (by_array[0]) e = arrays(false);
        else if (base != held[0] && total > in_bytes)
            e = cudaMemcpyAsync(held[0] + in_bytes, base + in_bytes, total - in_bytes, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        done = true;
        if (!by_array[0])
            for (int k = 0; k < n; ++k)
                if (!a[k].in) std::memcpy(a[k].host, held[0] + a[k].off, a[k].bytes);
        return cudaSuccess;
    }

private:
    bool opened = false, done = false, by_array[2] = { false, false };

    cudaError_t arrays(bool up) {
        const cudaMemcpyKind kind = up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
        size_t first[kMaxArrays + 1] = {};   // first chunk of each array that is staged
        for (int k = 0; k < n; ++k)
            first[k + 1] = first[k] + (a[k].in == up && !a[k].direct ? (a[k].bytes + kChunk - 1) / kChunk : 0);
        const size_t chunks = first[n];
        if (chunks && !held[1]) held[1] = PinPool::get().take(1);
        for (int k = 0; k < n; ++k) {
            if (a[k].in != up || (!a[k].direct && held[1])) continue;
            char* dev = base + a[k].off;
            const cudaError_t e = cudaMemcpyAsync(up ? dev : a[k].host, up ? a[k].host : dev, a[k].bytes, kind, st);
            if (e != cudaSuccess) return e;
        }
        if (chunks == 0 || !held[1]) return cudaSuccess;
        for (int k = 0; k < kMaxThreads; ++k) {
            if (slot_ev[k]) continue;
            const cudaError_t e = cudaEventCreateWithFlags(&slot_ev[k], cudaEventDisableTiming);
            if (e != cudaSuccess) return e;
        }
        const int threads = static_cast<int>(std::min<size_t>(chunks, std::min(kMaxThreads, omp_get_max_threads())));
        std::atomic<size_t> next{ 0 };
        std::atomic<int> err{ cudaSuccess };
        #pragma omp parallel num_threads(threads)
        {
            const int me = omp_get_thread_num();
            char* slot = held[1] + kChunk * me;
            cudaError_t e = cudaSetDevice(device);
            for (size_t c = next++; e == cudaSuccess && c < chunks; c = next++) {
                int k = 0;
                while (c >= first[k + 1]) ++k;
                const size_t at = (c - first[k]) * kChunk, bytes = std::min(kChunk, a[k].bytes - at);
                char *host = a[k].host + at, *dev = base + a[k].off + at;
                if (up) std::memcpy(slot, host, bytes);
                e = cudaMemcpyAsync(up ? dev : slot, up ? slot : dev, bytes, kind, st);
                if (e == cudaSuccess) e = cudaEventRecord(slot_ev[me], st);
                if (e == cudaSuccess) e = cudaEventSynchronize(slot_ev[me]);
                if (e == cudaSuccess && !up) std::memcpy(host, slot, bytes);
            }
            if (e != cudaSuccess) err = e;
        }
        return static_cast<cudaError_t>(err.load());
    }
};

}  // namespace bbrt
