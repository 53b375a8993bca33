// Decode attention in the reference's operation order for contexts of up to 256 keys: one CTA per sequence and head group, every
// phase by all of its 256 threads, K and V in shared memory as they come. Same function and same bits as attention.cu and
// attention_split.cu (FusedKVCache::forward_attention_raw and PagedKVCache::forward_attention_raw,
// src/runtime/TenzoEngine.cpp:242-445, :447-533, :657-694, :823-851 of the reference).
//
// What bounds it: latency. A short context is some hundred dependent steps - position, rows and query, rotation, scores, maximum,
// exponentials, their sum in key order, weights, value sums in key order - so the phases are laid out for few barriers (seven)
// and for all threads: up to 64 keys four threads share a key (a head each), up to 128 two, above that a thread has a key.
// The scores stay in the thread's registers until they are exponentials.
// Microseconds of a call in a graph, 20/5 heads, against what the automatic choice took before (one kernel for one sequence, three
// for many): one sequence of 64 keys 4.8 -> 3.6, of 211 6.7 -> 5.6; 63 prompt rows 16.6 -> 7.2, 255 44.6 -> 39.1; 12 sequences up to 200 keys
// 12.6 -> 6.8, 64 up to 256 23.5 -> 19.2, 256 up to 256 54.5 -> 52.5; block pools, 64 up to 200 25.9 -> 18.3. At 256 keys and many items it is
// bound by its instructions as the three kernels are, and the line lies there.
// Part of attention.cu, whose error flag it sets: a flag of its own would be one more synchronising copy, 13 us, wherever the flags are
// read (each greedy call, each step of several sequences).
#pragma once
#include <cuda.h>

#include "attn_common.cuh"
#include "ordered_sum.cuh"
#include "../../include/tenzo_kernels.h"

namespace tz {

constexpr int kShortThreads = 256, kShortKeys = 256;

struct ShortLaunch {
    tenzo_attention_args a;
    bool early;                      // position, cache rows and scales are read before the wait for the previous kernel
};

// [K rows][V rows] | exponentials [GH][stride] | weights [keys][GH] | queries [GH][128] | new rows [2][128]
struct ShortSmem {
    int rows, keys, stride;          // cache rows, key slots (64, 128 or 256), floats between heads' exponentials
    __host__ __device__ ShortSmem(int max_len) : rows((max_len + 15) & ~15), keys(max_len <= 64 ? 64 : max_len <= 128 ? 128 : 256), stride(keys + 4) {}
    __host__ __device__ size_t bytes(int gh) const { return (size_t)2 * rows * kHd + 4 * ((size_t)gh * stride + (size_t)keys * gh + (size_t)gh * kHd + 2 * kHd); }
};

__device__ __forceinline__ void short_cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// The dot products of one key row (16-byte pieces permuted by row & 7) with H heads.
template <int H, bool PAGED>
__device__ __forceinline__ void short_dots(const unsigned char* row, uint32_t swz, const float* q, float ks, float sm_scale, float (&out)[4]) {
    constexpr int NA = PAGED ? 16 : 8;      // contiguous cache: eight FMA lanes, element e in lane e mod 8 (:682-691); block pools: sixteen (:371-386)
    float acc[H][NA];
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int j = 0; j < NA; ++j) acc[h][j] = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint4 kb = *reinterpret_cast<const uint4*>(row + (((uint32_t)c ^ swz) << 4));
        const uint32_t w[4] = {kb.x ^ 0x80808080u, kb.y ^ 0x80808080u, kb.z ^ 0x80808080u, kb.w ^ 0x80808080u};
        float kf[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) kf[e] = s8_to_f(w[e >> 2], e & 3);
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int e4 = 0; e4 < 4; ++e4) {
                const float4 q4 = *reinterpret_cast<const float4*>(q + h * kHd + c * 16 + e4 * 4);
                const float qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float& d = acc[h][(e4 * 4 + e) % NA];
                    d = __fmaf_rn(qv[e], kf[e4 * 4 + e], d);
                }
            }
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const float* ac = acc[h];
        if constexpr (PAGED) {
            float dot = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) dot = __fadd_rn(dot, __fadd_rn(ac[j], ac[j + 8]));
            out[h] = __fmul_rn(__fmul_rn(dot, ks), sm_scale);                          // :388
        } else {
            out[h] = (ac[0] + ac[1] + ac[2] + ac[3] + ac[4] + ac[5] + ac[6] + ac[7]) * (ks * sm_scale);   // :691
        }
    }
}

template <int GH, bool PAGED>
__global__ void __launch_bounds__(kShortThreads) attn_short_kernel(const ShortLaunch L) {
    const tenzo_attention_args& a = L.a;
    extern __shared__ __align__(16) unsigned char s_k[];
    __shared__ float s_red[kShortThreads / 32][4], s_inv[GH], s_new_scale[2];
    const ShortSmem lay(a.max_len);
    unsigned char* s_v = s_k + lay.rows * kHd;
    float* s_e = reinterpret_cast<float*>(s_v + lay.rows * kHd);
    float* s_w = s_e + GH * lay.stride;
    float* s_q = s_w + lay.keys * GH;
    float* s_new = s_q + GH * kHd;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = a.n_q / a.n_kv;
    const int head0 = blockIdx.x * GH, kvh = head0 / G, seq = blockIdx.y;
    if (a.use_pdl && !L.early) pdl_wait();
    const int pos = __ldcg(a.pos + seq), T = pos + 1;
    if (pos < 0 || pos >= a.max_len) {
        if (tid == 0) atomicExch(&g_attn_timeouts, 2);
        return;
    }
    const size_t base = ((size_t)a.layer * a.n_kv + kvh) * a.max_seq;
    const int* table = PAGED ? a.block_table + (size_t)seq * a.table_stride : nullptr;
    auto row = [&](int t) -> size_t {
        if constexpr (PAGED) return (((size_t)__ldg(table + (t >> 4)) * a.n_layers + a.layer) * a.n_kv + kvh) * 16 + (size_t)(t & 15);
        else return base + t;
    };
    const size_t seq_kv = PAGED ? 0 : (size_t)seq * a.seq_stride_kv, seq_sc = PAGED ? 0 : (size_t)seq * a.seq_stride_sc;
    int8_t* ck = a.cache_k + seq_kv;
    int8_t* cv = a.cache_v + seq_kv;
    float* sk = a.scale_k + seq_sc;
    float* sv = a.scale_v + seq_sc;
    const int cached = a.append ? pos : T;             // keys whose rows are in the cache
    for (int i = tid; i < cached * 8; i += kShortThreads) {
        const int t = i >> 3, c = i & 7, at = t * kHd + ((c ^ (t & 7)) << 4);
        const size_t r = row(t) * kHd + c * 16;
        short_cp_async16(s_k + at, ck + r);
        short_cp_async16(s_v + at, cv + r);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // Keys and heads of this thread.
    const int nk = T <= 64 ? 64 : T <= 128 ? 128 : 256, key = tid & (nk - 1), hpt = GH * nk >= kShortThreads ? GH * nk / kShortThreads : 1;
    const int h0 = tid / nk * hpt;
    const bool mine = key < T && h0 < GH;
    float ks = 0.0f, vs = 0.0f;
    if (key < cached) {
        const size_t r = row(key);
        ks = __ldcg(sk + r);
        vs = __ldcg(sv + r);
    }
    const int i = tid & (kHd / 2 - 1);                 // this thread's pair of a rotated vector
    float c = 1.0f, sn = 0.0f;
    if (a.rope_cos) {
        c = __ldg(a.rope_cos + (size_t)pos * (kHd / 2) + i);
        sn = __ldg(a.rope_sin + (size_t)pos * (kHd / 2) + i);
    }
    if (a.use_pdl && L.early) pdl_wait();

    // ---- rotation of the queries and the new key (:459-480), the new row (:483-533) -----------------------------------------------
    {
        const float* qh = a.q + (size_t)seq * a.q_stride + (size_t)head0 * kHd;
        const float* kh = a.k + (size_t)seq * a.kv_stride + (size_t)kvh * kHd;
        const float* vh = a.v + (size_t)seq * a.kv_stride + (size_t)kvh * kHd;
        const int g = tid >> 6;
        float q0 = 0.0f, q1 = 0.0f, n0 = 0.0f, n1 = 0.0f;
        if (g < GH) {
            q0 = __ldcg(qh + g * kHd + i);
            q1 = __ldcg(qh + g * kHd + i + kHd / 2);
        }
        const bool new_k = a.append && g == 3, new_v = a.append && g == 2;
        if (new_k || new_v) {
            n0 = __ldcg((new_k ? kh : vh) + i);
            n1 = __ldcg((new_k ? kh : vh) + i + kHd / 2);
        }
        if (g < GH) rope_rotate(q0, q1, a.rope_cos != nullptr, c, sn, s_q[g * kHd + i], s_q[g * kHd + i + kHd / 2]);
        if (new_k || new_v) {
            float* o = s_new + (new_k ? 0 : kHd);
            rope_rotate(n0, n1, new_k && a.rope_cos != nullptr, c, sn, o[i], o[i + kHd / 2]);
        }
    }
    if (a.append) {
        __syncthreads();
        if (warp < 2) {                                // warp 0: key row, warp 1: value row
            const float4 x4 = *reinterpret_cast<const float4*>(s_new + warp * kHd + lane * 4);
            const float x[4] = {x4.x, x4.y, x4.z, x4.w};
            float amax = 1e-8f;
#pragma unroll
            for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fabsf(x[j]));
            amax = warp_max(amax);
            const float s = amax / 127.0f, inv = 1.0f / s;                           // :522, :527
            uint32_t packed = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                packed |= ((uint32_t)(uint8_t)(int8_t)(int)fminf(fmaxf(roundf(x[j] * inv), -128.0f), 127.0f)) << (8 * j);   // :530
            *reinterpret_cast<uint32_t*>((warp == 0 ? s_k : s_v) + pos * kHd + (((lane >> 2) ^ (pos & 7)) << 4) + (lane & 3) * 4) = packed;
            if (lane == 0) s_new_scale[warp] = s;
            if (head0 % G == 0) {
                const size_t r = row(pos);
                reinterpret_cast<uint32_t*>((warp == 0 ? ck : cv) + r * kHd)[lane] = packed;
                if (lane == 0) (warp == 0 ? sk : sv)[r] = s;
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (a.use_pdl) pdl_launch_dependents();
    if (a.append && key == pos) { ks = s_new_scale[0]; vs = s_new_scale[1]; }

    // ---- scores (:678-694), their maximum, exponentials (:826) --------------------------------------------------------------------
    const float sm_scale = 1.0f / sqrtf((float)kHd);   // :660
    float x[4] = {-1e30f, -1e30f, -1e30f, -1e30f};     // :670
    if (mine) {
        const unsigned char* kr = s_k + key * kHd;
        const uint32_t swz = (uint32_t)key & 7u;
        const float* q = s_q + h0 * kHd;
        if (GH >= 4 && hpt == 4) short_dots<4 < GH ? 4 : GH, PAGED>(kr, swz, q, ks, sm_scale, x);
        else if (GH >= 2 && hpt == 2) short_dots<2 < GH ? 2 : GH, PAGED>(kr, swz, q, ks, sm_scale, x);
        else short_dots<1, PAGED>(kr, swz, q, ks, sm_scale, x);
    }
#pragma unroll
    for (int h = 0; h < GH; ++h)
        if (h < hpt) {
            const float m = warp_max(fmaxf(-1e30f, x[h]));
            if (lane == 0) s_red[warp][h] = m;
        }
    __syncthreads();
    const unsigned long long tab = kExp2fTab[lane];
    const uint32_t tab_lo = (uint32_t)tab, tab_hi = (uint32_t)(tab >> 32);
    const int group_warps = nk >> 5, warp0 = tid / nk * group_warps;
#pragma unroll
    for (int h = 0; h < GH; ++h)
        if (h < hpt) {
            float m = -1e30f;
            for (int w = 0; w < group_warps; ++w) m = fmaxf(m, s_red[warp0 + w][h]);
            const float e = expf_reference_bits_lanes(mine ? x[h] - m : 0.0f, tab_lo, tab_hi);
            x[h] = mine ? e : 0.0f;
            if (h0 < GH) s_e[(h0 + h) * lay.stride + key] = x[h];
        }
    __syncthreads();
    if (warp < GH) {                                   // :824-829
        const float sum = chain_sum(s_e + warp * lay.stride, (T + 3) & ~3, 0.0f);
        if (lane == 0) s_inv[warp] = PAGED ? 1.0f / __fadd_rn(sum, 1e-8f) : 1.0f / sum;          // :400 for block pools
    }
    __syncthreads();
    // ---- weights p_t * s_v[t] (:830, :844): zero behind the last key ---------------------------------------------------------------
    if (h0 < GH) {
#pragma unroll
        for (int h = 0; h < GH; ++h)
            if (h < hpt) {
                const float p = x[h] * s_inv[h0 + h];
                s_w[key * GH + h0 + h] = !mine || (PAGED && p < 1e-7f) ? 0.0f : p * vs;        // block pools drop keys under 1e-7 (:416)
            }
    }
    __syncthreads();
    // ---- value sums in key order (:842-851): a thread has one dim of half the heads ------------------------------------------------
    constexpr int HV = GH >= 2 ? GH / 2 : 1;
    const int d = tid & (kHd - 1), hv = (tid >> 7) * HV;
    if (hv >= GH) return;
    float acc[HV];
#pragma unroll
    for (int h = 0; h < HV; ++h) acc[h] = 0.0f;
    const unsigned char* vp = s_v + (d & 15);
    const int piece = d >> 4;
    constexpr int U = 8;
    float w[2][U][HV];
    int vb[2][U];
    auto load = [&](int b, int t0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int8_t* p = reinterpret_cast<const int8_t*>(vp + (t0 + u) * kHd + ((piece ^ u) << 4));         // t0 is a multiple of eight
            vb[b][u] = *p;
            asm("" : "+r"(vb[b][u]));
#pragma unroll
            for (int h = 0; h < HV; ++h) w[b][u][h] = s_w[(t0 + u) * GH + hv + h];
        }
    };
    auto add = [&](int b) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float f = (float)vb[b][u];
#pragma unroll
            for (int h = 0; h < HV; ++h) acc[h] = __fmaf_rn(f, w[b][u][h], acc[h]);
        }
    };
    const int steps = (T + U - 1) / U;                 // (rows behind the last key: whatever bytes there are, with weight zero)
    load(0, 0);
    for (int s = 0; s < steps; s += 2) {
        if (s + 1 < steps) load(1, (s + 1) * U);
        add(0);
        if (s + 1 >= steps) break;
        if (s + 2 < steps) load(0, (s + 2) * U);
        add(1);
    }
    float* out = a.out + ((size_t)seq * a.n_q + head0 + hv) * kHd + d;
#pragma unroll
    for (int h = 0; h < HV; ++h) out[h * kHd] = acc[h];
}

// Up to 256 keys. `tiles` and `heads_per_cta` ask for one of the other forms; the rows go to shared memory in 16-byte pieces.
static bool attn_short_chosen(const tenzo_attention_args& a) {
    if (a.mode != 0 || a.tiles != 0 || a.heads_per_cta != 0 || a.max_len > kShortKeys) return false;
    if ((reinterpret_cast<uintptr_t>(a.cache_k) & 15) || (reinterpret_cast<uintptr_t>(a.cache_v) & 15)) return false;
    return a.block_table || a.seq_stride_kv % 16 == 0;
}

template <int GH, bool PAGED>
static int short_launch(const ShortLaunch& L, cudaStream_t st) {
    cudaError_t e = allow_smem(attn_short_kernel<GH, PAGED>, ShortSmem(kShortKeys).bytes(GH));
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(L.a.n_q / GH), (unsigned)L.a.batch, 1);
    cfg.blockDim = dim3(kShortThreads, 1, 1);
    cfg.dynamicSmemBytes = ShortSmem(L.a.max_len).bytes(GH);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = L.a.use_pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, attn_short_kernel<GH, PAGED>, L);
}

static int attn_short_run(const tenzo_attention_args& a, cudaStream_t st) {
    ShortLaunch L;
    L.a = a;
    if (L.a.q_stride <= 0) L.a.q_stride = a.n_q * kHd;
    if (L.a.kv_stride <= 0) L.a.kv_stride = a.n_kv * kHd;
    // (as the form for few items in attention.cu: with an append the rows before the new one are inputs that no kernel of the
    // step writes)
    L.early = a.append && !a.block_table && (long long)a.batch * a.n_kv < 64;
    int gh = a.n_q / a.n_kv > 4 ? 4 : a.n_q / a.n_kv;
    while (gh > 1 && (long long)a.batch * (a.n_q / gh) < 148) gh >>= 1;
    if (a.block_table) return gh == 4 ? short_launch<4, true>(L, st) : gh == 2 ? short_launch<2, true>(L, st) : short_launch<1, true>(L, st);
    return gh == 4 ? short_launch<4, false>(L, st) : gh == 2 ? short_launch<2, false>(L, st) : short_launch<1, false>(L, st);
}

}  // namespace tz
