// Sequential fp32 sums of non-negative values, evaluated in parallel with the bits of the sequential loop.
#pragma once
#include "common.cuh"

namespace tz {

// s = ((s + e[0]) + e[1]) + ... by one warp, every addition rounded to nearest even as in the loop, for e[i] >= 0.
//
// While the running sum s stays inside one binade [B, 2B) it is a multiple of u = ulp(B), and RN(s + e) - s is e rounded to
// a multiple of u; only a tie looks at s, and only at whether s / u is even. So over a run of elements the sum advances by
// one of two amounts, chosen by the parity of the mantissa it starts from, and both are found by running the loop from B and
// from B + u - without knowing s. Each lane does that for one segment, with B guessed from an approximate prefix sum; the
// segments are then applied in order. A segment whose guess was wrong, or in which the sum leaves the binade (it can
// double only so often), is added element by element: the guess decides the speed, never the result.
//
// A dependent addition takes 4.5 cycles, so the plain loop over 4096 values is 18 000 cycles; this is about 3 000.
//
// `e` is in shared memory, 16-byte aligned, and readable up to ordered_sum_padded(n) floats, zeros beyond n. All 32 lanes
// call it with the same arguments and get the same result.
__host__ __device__ __forceinline__ int ordered_sum_segment(int n) { return 4 * (((n + 127) >> 7) | 1); }   // odd number of 16-byte pieces: no bank conflicts
__host__ __device__ __forceinline__ int ordered_sum_padded(int n) { return 32 * ordered_sum_segment(n); }

__device__ __forceinline__ float ordered_sum_warp(const float* e, int n, float s) {
    constexpr uint32_t kExp = 0x7f800000u;
    const int lane = threadIdx.x & 31, L4 = ordered_sum_segment(n) >> 2;
    const float4* seg = reinterpret_cast<const float4*>(e) + lane * L4;
    float p0 = 0.0f, p1 = 0.0f;
    for (int j = 0; j < L4; ++j) {
        const float4 v = seg[j];
        p0 += v.x + v.y;
        p1 += v.z + v.w;
    }
    const float part = p0 + p1;
    float incl = part;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    uint32_t B = __float_as_uint(s + (incl - part)) & kExp;
    const float start0 = __uint_as_float(B), start1 = __uint_as_float(B | 1u);
    float c0 = start0, c1 = start1;
    for (int j = 0; j < L4; ++j) {
        const float4 v = seg[j];
        c0 += v.x; c1 += v.x;
        c0 += v.y; c1 += v.y;
        c0 += v.z; c1 += v.z;
        c0 += v.w; c1 += v.w;
    }
    if (B == kExp || (__float_as_uint(c0) & kExp) != B || (__float_as_uint(c1) & kExp) != B) B = 0u;   // 0: element by element
    const float d0 = c0 - start0, d1 = c1 - start1;      // exact: multiples of u below B
    auto serial = [&](int i) {
        const float4* p = reinterpret_cast<const float4*>(e) + i * L4;
        for (int j = 0; j < L4; ++j) {
            const float4 v = p[j];
            s += v.x; s += v.y; s += v.z; s += v.w;
        }
    };
    const int n_seg = (n + 4 * L4 - 1) / (4 * L4);
    for (int i = 0; i < n_seg; i += 4) {                 // four segments at a time; the lanes behind the last hold zeros
        float r[5];
        r[0] = s;
        const uint32_t Bs = __float_as_uint(s) & kExp;
        bool fits = Bs != 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t Bi = __shfl_sync(0xffffffffu, B, i + k);
            const float a0 = __shfl_sync(0xffffffffu, d0, i + k), a1 = __shfl_sync(0xffffffffu, d1, i + k);
            r[k + 1] = r[k] + ((__float_as_uint(r[k]) & 1u) ? a1 : a0);   // exact while it stays in the binade
            fits = fits && Bi == Bs;
        }
        if (fits && (__float_as_uint(r[4]) & kExp) == Bs) {
            s = r[4];
            continue;
        }
#pragma unroll 1
        for (int k = i; k < i + 4 && k < n_seg; ++k) {
            const uint32_t Bi = __shfl_sync(0xffffffffu, B, k);
            const float a0 = __shfl_sync(0xffffffffu, d0, k), a1 = __shfl_sync(0xffffffffu, d1, k);
            const uint32_t sb = __float_as_uint(s);
            const float t = s + ((sb & 1u) ? a1 : a0);
            if (Bi != 0u && (sb & kExp) == Bi && (__float_as_uint(t) & kExp) == Bi) s = t;
            else serial(k);
        }
    }
    return s;
}

}  // namespace tz
