// digit_counts.cuh -- how often each digit of the keys occurs, for every pass of the radix
// sort (sort.cu) at once.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace fgb {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kMaxPasses = 4;

// A CTA's counts, in shared memory.
struct DigitCounts {
    uint32_t of[kMaxPasses][kRadix];

    __device__ __forceinline__ void clear() {
        for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += blockDim.x) (&of[0][0])[i] = 0;
    }
    // (To add once where a warp's lanes agree costs more than it saves, 30 against 28 us for
    // the kernel that makes the keys of 1 M particles, although their high digits mostly do.)
    __device__ __forceinline__ void add(uint32_t key, int passes) {
        for (int p = 0; p < passes; ++p) atomicAdd(&of[p][(key >> (p * kRadixBits)) & (kRadix - 1)], 1u);
    }
    __device__ __forceinline__ void give(uint32_t *__restrict__ hist, int passes) const {
        for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) {
            const uint32_t v = (&of[0][0])[i];
            if (v) atomicAdd(&hist[i], v);
        }
    }
};

}  // namespace fgb
