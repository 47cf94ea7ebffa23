// Device allocations made by the engine since the library was loaded.  Asking
// the driver how much memory is in use takes half a millisecond; an answer stays
// good, as far as this library goes, until this number changes.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace cgb {

inline std::atomic<uint64_t>& device_allocs() {
    static std::atomic<uint64_t> n{0};
    return n;
}

template <class T>
inline cudaError_t device_malloc(T** p, size_t bytes) {
    device_allocs().fetch_add(1, std::memory_order_relaxed);
    return cudaMalloc((void**)p, bytes);
}

}  // namespace cgb
