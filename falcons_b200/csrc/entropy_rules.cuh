// Rules of the entropy stage that guard its memory accesses, callable on host and device.
#pragma once
#include <cuda_runtime.h>

namespace fb2 {

// Parts of a chain of n codes that decode side by side: one every `part` codes, or (part 0: no checkpoints) one in
// all, which takes at most kWholeChain codes, the decoder's 32-bit count.  ~0: more than that.
constexpr unsigned long long kWholeChain = 0xFFFFFFFFull;
__host__ __device__ __forceinline__ unsigned long long chain_part_count(unsigned long long n, unsigned long long part) {
    if (n == 0) return 0;
    if (part) return 1 + (n - 1) / part;
    return n <= kWholeChain ? 1 : ~0ull;
}

}  // namespace fb2
