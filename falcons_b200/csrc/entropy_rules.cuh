// Rules of the entropy stage that guard its memory accesses, callable on host and device.
#pragma once
#include <cuda_runtime.h>

namespace fb2 {

// Whether the items [first, first + count) are among the first n, for any `first` (the sum itself could wrap).
__host__ __device__ __forceinline__ bool range_within(unsigned long long first, unsigned long long count,
                                                      unsigned long long n) {
    return count <= n && first <= n - count;
}

}  // namespace fb2
