// HostIo and PinPool against a stand-in for the CUDA runtime, in which device
// memory cannot be touched by the host and a copy whose direction does not
// match its pointers is refused.
//   host_io copy BYTES KINDS   one call with two inputs and two outputs of BYTES
//                              bytes each; KINDS: h(ost), p(inned) or d(evice)
//                              for each of the four.  Prints "ok" when every
//                              output holds what the "kernel" wrote and it read
//                              the inputs, or the CUDA error that refused the call
//   host_io pool               blocks of the pool at its limits, and calls without
#include "../../billardballraytracing3d_b200/csrc/host_io.hpp"

#include <sys/mman.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <map>
#include <string>
#include <vector>

namespace {

struct Mapping { size_t bytes; char* view; };   // device range, and a view of it the stand-in uses
std::map<char*, Mapping> device_memory;
std::map<char*, size_t> pinned;
std::mutex mu;
int pin_calls = 0, pin_limit = 1 << 30;

template <class M>
auto find(M& m, const void* p, size_t (*size)(const typename M::mapped_type&)) {
    auto it = m.upper_bound(const_cast<char*>(static_cast<const char*>(p)));
    if (it == m.begin()) return m.end();
    --it;
    return static_cast<const char*>(p) < it->first + size(it->second) ? it : m.end();
}
char* device_view(const void* p) {   // null: not device memory
    auto it = find(device_memory, p, +[](const Mapping& x) { return x.bytes; });
    return it == device_memory.end() ? nullptr : it->second.view + (static_cast<const char*>(p) - it->first);
}
// Host view of any address: what a kernel sees.
char* view(void* p) {
    char* v = device_view(p);
    return v ? v : static_cast<char*>(p);
}

}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) {
    std::lock_guard<std::mutex> g(mu);
    const int fd = memfd_create("dev", 0);
    if (fd < 0 || ftruncate(fd, bytes)) return cudaErrorMemoryAllocation;
    char* hidden = static_cast<char*>(mmap(nullptr, bytes, PROT_NONE, MAP_SHARED, fd, 0));
    char* seen = static_cast<char*>(mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_SHARED, fd, 0));
    close(fd);
    device_memory[hidden] = { bytes, seen };
    *p = hidden;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> g(mu);
    auto it = device_memory.find(static_cast<char*>(p));
    munmap(it->first, it->second.bytes);
    munmap(it->second.view, it->second.bytes);
    device_memory.erase(it);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    std::lock_guard<std::mutex> g(mu);
    if (++pin_calls > pin_limit) return cudaErrorMemoryAllocation;
    *p = std::malloc(bytes);
    pinned[static_cast<char*>(*p)] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::lock_guard<std::mutex> g(mu);
    pinned.erase(static_cast<char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> g(mu);
    *a = {};
    a->type = device_view(p) ? cudaMemoryTypeDevice
              : find(pinned, p, +[](const size_t& x) { return x; }) != pinned.end() ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    std::lock_guard<std::mutex> g(mu);
    char *d = device_view(dst), *s = device_view(src);
    if (kind == cudaMemcpyHostToDevice ? (!d || s) : (d || !s)) return cudaErrorInvalidValue;
    std::memcpy(d ? d : dst, s ? s : src, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(8); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

namespace {

// One call: the "kernel" writes outputs from the inputs.  "ok", "wrong" or the error.
std::string call(size_t bytes, const char* kinds) {
    bbrt::DevBuf block;
    cudaEvent_t slot_ev[bbrt::PinPool::kSlots] = {};
    void* a[4];
    for (int k = 0; k < 4; ++k) {
        if (kinds[k] == 'd') cudaMalloc(&a[k], bytes);
        else if (kinds[k] == 'p') cudaHostAlloc(&a[k], bytes, 0);
        else a[k] = std::malloc(bytes);
        std::memset(view(static_cast<char*>(a[k])), k < 2 ? 3 + k : 0xEE, bytes);
    }
    std::string res;
    {
        bbrt::HostIo io(block, slot_ev, 0, nullptr);
        int at[4];
        for (int k = 0; k < 4; ++k) at[k] = io.add(a[k], bytes, k < 2);
        cudaError_t e = io.open();
        if (e == cudaSuccess) {
            char* v[4];
            for (int k = 0; k < 4; ++k) v[k] = view(io.at<char>(at[k]));
            for (size_t j = 0; j < bytes; ++j) {
                v[2][j] = static_cast<char>(v[0][j] + 16 * v[1][j] + j % 7);
                v[3][j] = static_cast<char>(v[0][j] * v[1][j] + j % 5);
            }
            e = io.close();
        }
        if (e != cudaSuccess) res = "error " + std::to_string(static_cast<int>(e));
    }
    if (res.empty()) {
        res = "ok";
        for (size_t j = 0; j < bytes; ++j)
            if (view(static_cast<char*>(a[2]))[j] != static_cast<char>(3 + 64 + j % 7) ||
                view(static_cast<char*>(a[3]))[j] != static_cast<char>(12 + j % 5)) {
                res = "wrong";
                break;
            }
    }
    return res;
}

}  // namespace

int main(int argc, char** argv) {
    if (argc == 4 && std::string(argv[1]) == "copy") {
        bbrt::PinPool::User user;
        std::printf("%s\n", call(std::strtoull(argv[2], nullptr, 10), argv[3]).c_str());
        return 0;
    }
    // the pool at its limits
    bbrt::PinPool& pool = bbrt::PinPool::get();
    {
        bbrt::PinPool::User user;
        std::vector<char*> held[2];
        for (int kind = 0; kind < 2; ++kind)
            while (char* p = pool.take(kind)) held[kind].push_back(p);
        std::printf("blocks %zu %zu pinned %zu\n", held[0].size(), held[1].size(), pinned.size());
        // calls of every size class while all blocks are out: no more is pinned
        const int before = pin_calls;
        for (size_t bytes : { 1000, 100000, 3000000 }) std::printf("out %s\n", call(bytes, "hhhh").c_str());
        std::printf("pinned by them %d\n", pin_calls - before);
        for (int kind = 0; kind < 2; ++kind)
            for (char* p : held[kind]) pool.give(kind, p);
    }
    std::printf("after the last scene %zu\n", pinned.size());
    pin_limit = pin_calls;   // the system pins no more
    {
        bbrt::PinPool::User user;
        for (size_t bytes : { 1000, 100000, 3000000 }) std::printf("none %s\n", call(bytes, "hhhh").c_str());
    }
    return 0;
}
