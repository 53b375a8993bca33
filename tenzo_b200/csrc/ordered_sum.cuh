// Sequential fp32 sums of non-negative values, evaluated in parallel with the bits of the sequential loop.
#pragma once
#include "common.cuh"

namespace tz {

// s = ((s + e[0]) + e[1]) + ... by one warp, every addition rounded to nearest even as in the loop, for e[i] >= 0.
//
// While the running sum s stays inside one binade [B, 2B) it is a multiple of u = ulp(B), and RN(s + e) - s is e rounded to
// a multiple of u; only a tie looks at s, and only at whether s / u is even. So over a run of elements the sum advances by
// one of two amounts, chosen by the parity of the mantissa it starts from, and both are found by running the loop from B and
// from B + u - without knowing s. Each lane does that for one segment. Which binade a segment lies in follows from a
// prefix sum in any order: both it and the loop are within n 2^-24 of the true sum, relatively, so a segment whose ends lie
// inside a binade by more than that is certain to stay in it. The few others (the sum can double only so often) are added
// element by element, and so are the first 64, where it doubles all the time.
//
// Cycles for n values, this against the plain loop with its loads: 2048: 6 800 and 10 800; 864: 5 000 and 4 700 (about 300 a
// segment that is added one by one, 315 a group of eight that is not).
//
// `e` is in shared memory, 16-byte aligned, and readable up to ordered_sum_padded(n) floats, zeros beyond n. All 32 lanes
// call it with the same arguments and get the same result.
constexpr int kOrderedHead = 64;
__host__ __device__ constexpr int ordered_sum_segment(int n) {          // elements a lane takes behind the head: whole 16-byte pieces, an odd number of them (no bank conflicts)
    const int pieces = n > kOrderedHead ? (n - kOrderedHead + 127) >> 7 : 1;
    return 4 * (pieces | 1);
}
__host__ __device__ constexpr int ordered_sum_padded(int n) { return kOrderedHead + 32 * ordered_sum_segment(n); }

// The plain loop over n values (n a multiple of 4): eight 16-byte loads, then their 32 additions. Loading the next batch during
// the additions is slower: a wait for one batch then also waits for the loads of the next.
__device__ __forceinline__ float chain_sum(const float* e, int n, float s) {
    const float4* p = reinterpret_cast<const float4*>(e);
    int j = 0;
#pragma unroll 1
    for (; j + 8 <= n >> 2; j += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = p[j + u];
#pragma unroll
        for (int u = 0; u < 8; ++u) { s += v[u].x; s += v[u].y; s += v[u].z; s += v[u].w; }
    }
#pragma unroll 1
    for (; j < n >> 2; ++j) { const float4 v = p[j]; s += v.x; s += v.y; s += v.z; s += v.w; }
    return s;
}

__device__ __forceinline__ float ordered_sum_warp(const float* e, int n, float s) {
    constexpr uint32_t kExp = 0x7f800000u;
    const int lane = threadIdx.x & 31;
    if (n <= kOrderedHead) return chain_sum(e, (n + 3) & ~3, s);
    const int L4 = ordered_sum_segment(n) >> 2;
    const float4* segs = reinterpret_cast<const float4*>(e + kOrderedHead);
    const float4* mine = segs + lane * L4;
    float p0 = 0.0f, p1 = 0.0f;
#pragma unroll 4
    for (int j = 0; j < L4; ++j) {
        const float4 v = mine[j];
        p0 += v.x + v.y;
        p1 += v.z + v.w;
    }
    const float part = p0 + p1;
    float incl = part;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {                   // (independent of the head's chain below, and hidden by it)
        const float up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    s = chain_sum(e, kOrderedHead, s);
    const float margin = (float)n * 0x1p-23f;            // twice the bound
    const float from = s + (incl - part), to = s + incl;
    const uint32_t B = __float_as_uint(from) & kExp;
    const bool inside = B != 0u && B != kExp && (__float_as_uint(from - from * margin) & kExp) == B && (__float_as_uint(to + to * margin) & kExp) == B;
    const float start0 = __uint_as_float(B), start1 = __uint_as_float(B | 1u);
    float c0 = start0, c1 = start1;
#pragma unroll 4
    for (int j = 0; j < L4; ++j) {
        const float4 v = mine[j];
        c0 += v.x; c1 += v.x;
        c0 += v.y; c1 += v.y;
        c0 += v.z; c1 += v.z;
        c0 += v.w; c1 += v.w;
    }
    // starting at B, not at s, the loop may leave the binade where the sum does not: then the segment is not used either
    const uint32_t use = __ballot_sync(0xffffffffu, inside && (__float_as_uint(c0) & kExp) == B && (__float_as_uint(c1) & kExp) == B);
    // Inside a binade the sum's bits count units of u, so the amounts are integers: i0 from an even mantissa and, the two runs
    // keeping a distance of 0, 1 or 2 units, i0 + (-1, 0 or 1) from an odd one. Nine cycles a segment: S + i0 + (S & 1) di.
    const int i0 = (int)(__float_as_uint(c0) - B), di = (int)(__float_as_uint(c1) - (B | 1u)) - i0;
    const int word = (i0 << 2) | (di + 1);
    const int n_seg = (n - kOrderedHead + 4 * L4 - 1) / (4 * L4);
    int S = __float_as_int(s);
#pragma unroll 1
    for (int i = 0; i < n_seg; i += 8) {
        int w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __shfl_sync(0xffffffffu, word, i + k);
        const uint32_t sure = use >> i & 0xffu;
        if (sure == 0xffu) {                             // (segments behind the last are empty: i0 = 0)
#pragma unroll
            for (int k = 0; k < 8; ++k) S += (w[k] >> 2) + (S & 1) * ((w[k] & 3) - 1);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (sure >> k & 1u) {
                    S += (w[k] >> 2) + (S & 1) * ((w[k] & 3) - 1);
                } else if (i + k < n_seg) {
                    S = __float_as_int(chain_sum(reinterpret_cast<const float*>(segs + (i + k) * L4), 4 * L4, __int_as_float(S)));
                }
            }
        }
    }
    s = __int_as_float(S);
    return s;
}

}  // namespace tz
