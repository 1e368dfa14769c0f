// pt_mapped.h - small buffers of mapped host memory that kernels write and the host reads
// (a stepped day's rows, the error word of a network's waits).
//
// Allocating one takes 105 us and freeing it 160 (GB300), as long as two stepped days of a
// small engine, and whoever makes an engine or a network makes one.  So buffers that are
// given back are kept for the next, up to kMappedKept of them and kMappedBytes in all;
// pt_trim_device_memory frees them.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <mutex>
#include <vector>

namespace ptm {

constexpr size_t kMappedKept = 64, kMappedBytes = 4 << 20, kMappedLeast = 256;

struct Mapped {
    void *ptr = nullptr;
    size_t bytes = 0;
};

struct MappedPool {
    std::mutex mu;
    std::vector<Mapped> kept;
    size_t bytes = 0;   // of those kept
};

inline MappedPool &mapped_pool()
{
    static MappedPool *p = new MappedPool();   // (not destroyed: engines may outlive static objects)
    return *p;
}

// At least `bytes` bytes, portable, contents unspecified.
inline cudaError_t mapped_take(size_t bytes, Mapped *out)
{
    size_t n = kMappedLeast;
    while (n < bytes) n *= 2;
    {
        MappedPool &p = mapped_pool();
        std::lock_guard<std::mutex> lock(p.mu);
        for (size_t i = 0; i < p.kept.size(); i++)
            if (p.kept[i].bytes == n) {
                *out = p.kept[i];
                p.bytes -= n;
                p.kept.erase(p.kept.begin() + (long)i);
                return cudaSuccess;
            }
    }
    void *ptr = nullptr;
    const cudaError_t e = cudaHostAlloc(&ptr, n, cudaHostAllocMapped | cudaHostAllocPortable);
    if (e == cudaSuccess) *out = {ptr, n};
    return e;
}

// `idle`: nothing that writes the buffer is in flight.  Where that could not be waited for
// (beside a capture) it is freed and not kept.
inline void mapped_give(Mapped &m, bool idle)
{
    if (!m.ptr) return;
    if (idle) {
        MappedPool &p = mapped_pool();
        std::lock_guard<std::mutex> lock(p.mu);
        if (p.kept.size() < kMappedKept && p.bytes + m.bytes <= kMappedBytes) {
            p.kept.push_back(m);
            p.bytes += m.bytes;
            m = Mapped{};
            return;
        }
    }
    cudaFreeHost(m.ptr);
    m = Mapped{};
}

inline void mapped_trim()
{
    std::vector<Mapped> all;
    {
        MappedPool &p = mapped_pool();
        std::lock_guard<std::mutex> lock(p.mu);
        all.swap(p.kept);
        p.bytes = 0;
    }
    for (Mapped &m : all) cudaFreeHost(m.ptr);
}

}  // namespace ptm
