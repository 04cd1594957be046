// Block flags of the carry scans' decoupled look-back.
#pragma once
#include <cuda/atomic>

#include <cstdint>

namespace bgpu {

constexpr uint32_t kSpinLimit = 1u << 22;  // bounded look-back wait, then error exit

// Flag word: [63:4] epoch, [3:2] status (1 aggregate, 2 inclusive), [1] G/carry, [0] P.
__device__ __forceinline__ uint64_t make_flag(uint64_t epoch, uint32_t status, uint32_t g,
                                              uint32_t pbit) {
    return (epoch << 4) | ((uint64_t)status << 2) | ((uint64_t)g << 1) | pbit;
}

// Bounded wait for a look-back flag word of the current epoch: returns it, or
// 0 after `limit` polls with bit 0 of the error word set.  The only wait of
// the carry scans; the diagnostic k_wait_selftest runs it on its own.
__device__ __forceinline__ uint64_t wait_flag(const uint64_t* flag, uint64_t epoch, uint32_t limit,
                                              uint32_t* err) {
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_device> w(
        *reinterpret_cast<unsigned long long*>(const_cast<uint64_t*>(flag)));
    for (uint32_t spins = 0;; ++spins) {
        const uint64_t f = w.load(cuda::memory_order_acquire);
        if ((f >> 4) == epoch) return f;
        if (spins >= limit) {
            atomicOr(err, 1u);
            return 0;
        }
        __nanosleep(32);
    }
}

}  // namespace bgpu
