// Shared between the two LM-head kernels (lm_head.cu, lm_head_umma.cu): the argmax candidate record
// and its ordering.
#pragma once

namespace tz {

struct LmBest { float val; int idx; };

__device__ __forceinline__ bool better(float v, int i, float bv, int bi) {
    // greedy argmax keeps the first maximum (TenzoEngine.cpp:1749 of the reference, strict '>'):
    // larger value, or same value at a lower index
    return v > bv || (v == bv && i < bi);
}

// The layer before the LM head asks for this much of the table; the one-sequence kernel asks for the next piece while its
// own activations are being prepared (together they stay below the 126 MB of L2).
constexpr size_t kLmPrefetchBefore = (size_t)64 << 20, kLmPrefetchMore = (size_t)24 << 20;

constexpr int kLmuMaxTiles = 2048;   // 128-row vocabulary tiles the tensor-core path's scratch is sized for (vocab <= 262144)

}  // namespace tz
