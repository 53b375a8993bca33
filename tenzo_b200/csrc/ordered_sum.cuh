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
// HEAD = false: for a sum that goes on, where the first elements are like all others.
//
// `e` is in shared memory, 16-byte aligned, and readable up to ordered_sum_padded(n, HEAD) floats, zeros beyond n. All 32 lanes
// call it with the same arguments and get the same result.
constexpr int kOrderedHead = 64;
__host__ __device__ constexpr int ordered_sum_segment(int n) {          // elements a lane takes of n: whole 16-byte pieces, an odd number of them (no bank conflicts)
    return 4 * ((n > 0 ? (n + 127) >> 7 : 1) | 1);
}
__host__ __device__ constexpr int ordered_sum_padded(int n, bool head = true) {
    return head ? kOrderedHead + 32 * ordered_sum_segment(n - kOrderedHead) : 32 * ordered_sum_segment(n);
}
// Two amounts in a row, each from an even and from an odd mantissa: again such a pair.
__device__ __forceinline__ void join_steps(int& even, int& odd, int next_even, int next_odd) {
    even += even & 1 ? next_odd : next_even;
    odd += odd & 1 ? next_even : next_odd;
}

// The plain loop over n values (n a multiple of 4): eight 16-byte loads, then their 32 additions (of zeros behind the last value, which
// change nothing). Loading the next batch during the additions is slower: a wait for one batch then also waits for the loads of
// the next.
__device__ __forceinline__ float chain_sum(const float* e, int n, float s) {
    const float4* p = reinterpret_cast<const float4*>(e);
#pragma unroll 1
    for (int j = 0; j < n >> 2; j += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = j + u < n >> 2 ? p[j + u] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int u = 0; u < 8; ++u) { s += v[u].x; s += v[u].y; s += v[u].z; s += v[u].w; }
    }
    return s;
}

template <bool HEAD>
__device__ __forceinline__ float ordered_sum_warp(const float* e, int n, float s) {
    constexpr uint32_t kExp = 0x7f800000u;
    constexpr int head = HEAD ? kOrderedHead : 0;
    const int lane = threadIdx.x & 31;
    if (n <= kOrderedHead) return chain_sum(e, (n + 3) & ~3, s);
    const int L4 = ordered_sum_segment(n - head) >> 2;
    const float4* segs = reinterpret_cast<const float4*>(e + head);
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
    if (HEAD) s = chain_sum(e, kOrderedHead, s);
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
    // Inside a binade the sum's bits count units of u, so the amounts are integers, and two segments in a row are one: five rounds of
    // shuffles leave in the last lane of every run of sure lanes what the run comes to. (Walked one by one, the 32 segments took
    // more instructions than their additions.) Segments behind the last are empty, their amounts zero.
    int even = (int)(__float_as_uint(c0) - B), odd = (int)(__float_as_uint(c1) - (B | 1u));
    if (use == 0xffffffffu) {                                // (most of a long sum's chunks)
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ne = __shfl_down_sync(0xffffffffu, even, o), no = __shfl_down_sync(0xffffffffu, odd, o);
            join_steps(even, odd, ne, no);
        }
        const int S = __float_as_int(s);
        return __int_as_float(S + __shfl_sync(0xffffffffu, S & 1 ? odd : even, 0));
    }
    const uint32_t first = ~use | (~use << 1) | 1u;          // lanes that no sure lane's amounts are added to from below
    int f = (int)(first >> lane & 1u);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int pe = __shfl_up_sync(0xffffffffu, even, o), po = __shfl_up_sync(0xffffffffu, odd, o);
        const int pf = __shfl_up_sync(0xffffffffu, f, o);
        if (!f && lane >= o) {
            join_steps(pe, po, even, odd);
            even = pe;
            odd = po;
            f = pf;
        }
    }
    int S = __float_as_int(s);
#pragma unroll 1
    for (int k = 0; k < 32;) {
        const uint32_t unsure = ~use & (0xffffffffu << k);
        const int end = unsure ? __ffs(unsure) - 1 : 32;     // the first lane from k on that is not sure
        if (end > k) {
            const int je = __shfl_sync(0xffffffffu, even, end - 1), jo = __shfl_sync(0xffffffffu, odd, end - 1);
            S += S & 1 ? jo : je;
        }
        if (end < 32) S = __float_as_int(chain_sum(reinterpret_cast<const float*>(segs + end * L4), 4 * L4, __int_as_float(S)));
        k = end + 1;
    }
    return __int_as_float(S);
}

}  // namespace tz
