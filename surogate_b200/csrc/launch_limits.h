// Dynamic shared memory above 48 KB has to be allowed per kernel AND per device before the first launch there.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>

namespace sg {

// Allows `kernel` `bytes` of dynamic shared memory on the current device, once per device: bit d of `done` (one word per kernel) says that
// device d has it.  False when the runtime refuses; the next launch then asks again.  Safe from several threads: the attribute is the same
// for all of them.
inline bool raise_smem_limit(const void* kernel, int bytes, std::atomic<uint64_t>& done) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return false;
    const uint64_t bit = dev < 64 ? uint64_t{1} << dev : 0;      // beyond 64 devices: asked at every launch
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        cudaGetLastError();      // reported here, not by the next launch check
        return false;
    }
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

}  // namespace sg
