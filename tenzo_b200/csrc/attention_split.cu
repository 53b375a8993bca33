// Decode attention in the reference's operation order over the whole machine: scores, softmax and value sums as three
// kernels with the score vectors in a scratch buffer between them. Same function and same bits as attention.cu
// (FusedKVCache::forward_attention_raw and PagedKVCache::forward_attention_raw, src/runtime/TenzoEngine.cpp:242-445,
// :447-533, :657-694, :823-851 of the reference), for callers that bring the scratch.
//
// Why three kernels. The order fixes only chains: the eight (paged: sixteen) FMA lanes of one score, the sum of a head's
// exponentials, and the sum over the keys for one head and one output dim. attention.cu keeps an item (sequence, kv head)
// in one CTA whose phases each use the warps that their own chains allow, with the score vectors filling shared memory so
// that an SM holds one CTA: 46 cycles per key and SM. Split at the phase boundaries, every phase spreads over all SMs:
//   scores   one warp per 64-key tile, any tile of any item: 4 heads x 128 FMA + 256 conversions per key, 8 LDS.128 of the
//            key row and 64 broadcast LDS.128 of the query per key pair;
//   softmax  one CTA per item or head; the ordered sum of the exponentials in parallel segments (ordered_sum.cuh);
//   values   consumer warps that own the chains of an (item, dims, heads) unit, fed by producer warps.
// What bounds it. A (key, item) takes some 70 warp instructions (35.6 in the scores, 6.3 in the softmax, 28 in the value sums; 16 +
// 16 of them are the multiply-adds whose order is fixed), so 592 schedulers need 60 us a million. 64 x 8192 keys, 20/5 heads:
// 672 us in one kernel, here 272, 104 us a million (277 before the sums of the softmax were joined and the value sums took two dims
// a load). The distance to 60: the three kernels follow one another without overlap (111, 35 and 126 us at 64 x 8192), the
// softmax lasts as long as its summing warps' chains, and the last round of the value sums is as long as its longest item (they
// are dealt out by index). The scores' loop cannot go below 30 cycles of a scheduler a (key, item): a byte permute or a logical
// operation holds its pipe for two cycles and adds to the multiply-adds instead of hiding under them, and a packed f32x2 multiply-add holds its
// pipe for as long as two plain ones. Four keys a lane, packed multiply-adds, conversion by an integer MMA and persistent CTAs
// were all written and took 108 to 167 us against 111 here.
// One sequence of 6003 keys: 98 us in one kernel, here 41 (6, 10.5 and 24 us).
// Launched back to back with programmatic serialisation but without an early trigger: kernels that let their dependents in
// before their own wait pile up on the SMs, and a small grid is then placed on the few that have room (one sequence of
// 6003 keys took 211 us that way).
#include <cuda.h>

#include <cstring>
#include <utility>

#include "attn_common.cuh"
#include "ordered_sum.cuh"
#include "umma.cuh"
#include "../../include/tenzo_kernels.h"

namespace tz {

constexpr int kScoreWarps = 8;
constexpr int kSpTile = 64;                       // keys of a score tile: two per lane
constexpr int kSpTileBytes = kSpTile * kHd;

struct SplitLaunch {
    tenzo_attention_args a;
    int gh;                          // query heads that share one pass over the keys (an item: sequence, kv head, head group)
    int groups;                      // items per sequence: n_q / gh
    int tp;                          // keys per item in the scratch (max_len rounded up to 4)
    int span, n_spans;               // keys per score CTA
    int seq0;                        // first sequence of this pass
    bool shared_cache;               // every query row reads sequence 0's cache (seq_stride 0 / table_stride 0)
    float* scores;                   // [item][tp][gh]: scores, then exponentials
    float* span_max;                 // [item][n_spans][gh]
    float* inv_sum;                  // [item][gh]
};

__device__ int g_split_timeouts = 0;   // 1: a bounded wait on a tile copy gave up; 2: a position outside [0, max_len)

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int row, int seq, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_addr(dst)), "l"(map), "r"(x), "r"(row), "r"(seq), "r"(smem_addr(bar)) : "memory");
}

template <int N>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {       // N = 4, 8 or 16 bytes
    if constexpr (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(N) : "memory");
}

// Where the keys of one (sequence, kv head) lie: row of key t in cache_k / cache_v and scale_k / scale_v.
template <bool PAGED>
struct KeyRows {
    const int* table;
    size_t base;                     // contiguous: rows before key 0 of this sequence, layer and head
    int n_layers, layer, n_kv, kvh;
    __device__ __forceinline__ KeyRows(const tenzo_attention_args& a, int seq, int kvh_) : table(nullptr), base(0), n_layers(a.n_layers), layer(a.layer), n_kv(a.n_kv), kvh(kvh_) {
        if constexpr (PAGED) table = a.block_table + (size_t)seq * a.table_stride;
        else base = ((size_t)a.layer * a.n_kv + kvh_) * a.max_seq;
    }
    __device__ __forceinline__ size_t row(int t) const {
        if constexpr (PAGED) return (((size_t)__ldg(table + (t >> 4)) * n_layers + layer) * n_kv + kvh) * 16 + (size_t)(t & 15);
        else return base + t;
    }
    // The 64 rows of a K tile, 128-byte swizzle; every lane calls it, after lane 0's expect_tx of tile_bytes.
    __device__ __forceinline__ void load_tile(unsigned char* dst, const CUtensorMap* map, int t0, int T, int map_seq, uint64_t* bar, int lane) const {
        if constexpr (PAGED) {
            if (lane < kSpTile / 16 && t0 + 16 * lane < T) tma_load_2d(dst + lane * 16 * kHd, map, 0, (int)row(t0 + 16 * lane), bar);
        } else {
            if (lane == 0) tma_load_3d(dst, map, 0, (int)base + t0, map_seq, bar);
        }
    }
    __device__ __forceinline__ unsigned tile_bytes(int t0, int T) const {
        if constexpr (PAGED) return (unsigned)min(kSpTile / 16, (T - t0 + 15) >> 4) * 16u * kHd;
        else return (unsigned)kSpTileBytes;
    }
};

// A warp takes tiles warp, warp + 8, ... of its CTA's key span through a tile buffer of its own (one: three or four warps
// share a scheduler, and the others compute while one waits).
template <int GH, bool PAGED>
__global__ void __launch_bounds__(kScoreWarps * 32, 2) split_scores_kernel(const SplitLaunch L, const __grid_constant__ CUtensorMap kmap) {
    const tenzo_attention_args& a = L.a;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* s_tiles = smem_raw + (((smem_addr(smem_raw) + 1023u) & ~1023u) - smem_addr(smem_raw));
    __shared__ __align__(16) float s_q[GH * kHd];
    __shared__ __align__(16) float s_new[2 * kHd];
    __shared__ __align__(16) int8_t s_new8[kHd];
    __shared__ float s_new_scale;
    __shared__ float s_red[kScoreWarps][GH];
    __shared__ uint64_t s_bar[kScoreWarps];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = blockIdx.y, seq = L.seq0 + blockIdx.z, head0 = grp * GH, G = a.n_q / a.n_kv, kvh = head0 / G;
    const size_t item = (size_t)blockIdx.z * L.groups + grp;
    if (lane == 0) {
        mbar_init(&s_bar[warp], 1);
        mbar_init_fence();
    }
    if (a.use_pdl) pdl_wait();
    const int pos = __ldcg(a.pos + seq), T = pos + 1, k0 = blockIdx.x * L.span, k1 = min(T, k0 + L.span);
    if (pos < 0 || pos >= a.max_len) {
        if (tid == 0) atomicExch(&g_split_timeouts, 2);
        return;
    }
    if (k0 >= T) return;
    const KeyRows<PAGED> rows(a, seq, kvh);
    const int map_seq = L.shared_cache ? 0 : seq;
    const size_t sc_base = (PAGED || L.shared_cache) ? 0 : (size_t)seq * a.seq_stride_sc;
    const float* sk = a.scale_k + sc_base;
    unsigned char* tile = s_tiles + (size_t)warp * kSpTileBytes;
    auto request = [&](int t0) {
        if (lane == 0) mbar_expect_tx(&s_bar[warp], rows.tile_bytes(t0, T));
        __syncwarp();
        rows.load_tile(tile, &kmap, t0, T, map_seq, &s_bar[warp], lane);
    };
    int t0 = k0 + warp * kSpTile;
    if (t0 < k1) request(t0);

    const float* cs = a.rope_cos ? a.rope_cos + (size_t)pos * (kHd / 2) : nullptr;
    const float* sn = a.rope_sin ? a.rope_sin + (size_t)pos * (kHd / 2) : nullptr;
    for (int idx = tid; idx < GH * (kHd / 2); idx += kScoreWarps * 32) {            // :459-480
        const int g = idx / (kHd / 2), i = idx % (kHd / 2);
        const float* qh = a.q + (size_t)seq * a.q_stride + (size_t)(head0 + g) * kHd;
        rope_pair(__ldcg(qh + i), __ldcg(qh + i + kHd / 2), cs, sn, i, s_q[g * kHd + i], s_q[g * kHd + i + kHd / 2]);
    }
    const bool has_new = a.append && pos < k1;       // this CTA's span ends with the new token
    if (has_new) {                                   // :483-533; the first head group of a kv head stores the rows
        if (tid < kHd / 2) {
            const float* kh = a.k + (size_t)seq * a.kv_stride + (size_t)kvh * kHd;
            rope_pair(__ldcg(kh + tid), __ldcg(kh + tid + kHd / 2), cs, sn, tid, s_new[tid], s_new[tid + kHd / 2]);
        } else if (tid >= kHd) {
            s_new[tid] = __ldcg(a.v + (size_t)seq * a.kv_stride + (size_t)kvh * kHd + tid - kHd);
        }
        __syncthreads();
        if (warp < 2) {
            const float4 v = *reinterpret_cast<const float4*>(s_new + warp * kHd + lane * 4);
            const float x[4] = {v.x, v.y, v.z, v.w};
            float amax = 1e-8f;
#pragma unroll
            for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fabsf(x[j]));
            amax = warp_max(amax);
            const float s = amax / 127.0f, inv = 1.0f / s;                           // :522, :527
            uint32_t packed = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                packed |= ((uint32_t)(uint8_t)(int8_t)(int)fminf(fmaxf(roundf(x[j] * inv), -128.0f), 127.0f)) << (8 * j);   // :530
            if (warp == 0) {
                reinterpret_cast<uint32_t*>(s_new8)[lane] = packed;
                if (lane == 0) s_new_scale = s;
            }
            if (head0 % G == 0) {
                const size_t r = rows.row(pos);
                int8_t* dst = (warp == 0 ? a.cache_k : a.cache_v) + ((PAGED || L.shared_cache) ? 0 : (size_t)seq * a.seq_stride_kv) + r * kHd;
                reinterpret_cast<uint32_t*>(dst)[lane] = packed;
                if (lane == 0) (warp == 0 ? a.scale_k : a.scale_v)[sc_base + r] = s;
            }
        }
    }
    __syncthreads();

    const float sm_scale = 1.0f / sqrtf((float)kHd);   // :660
    float tmax[GH];
#pragma unroll
    for (int g = 0; g < GH; ++g) tmax[g] = -1e30f;     // :670
    bool timed_out = false;
    float* out = L.scores + item * (size_t)L.tp * GH;
    for (int use = 0; t0 < k1; t0 += kScoreWarps * kSpTile, ++use) {
        float ksc[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int t = t0 + 32 * s + lane;
            ksc[s] = t < T && !(has_new && t == pos) ? __ldcg(sk + rows.row(t)) : s_new_scale;
        }
        if (lane == 0 && !mbar_wait_bounded(&s_bar[warp], (unsigned)use & 1u)) timed_out = true;
        __syncwarp();
        const unsigned char* row[2];
        uint32_t swz[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const bool is_new = has_new && t0 + 32 * s + lane == pos;
            row[s] = is_new ? reinterpret_cast<const unsigned char*>(s_new8) : tile + (32 * s + lane) * kHd;
            swz[s] = is_new ? 0u : (uint32_t)(lane & 7);
        }
        // contiguous cache: eight FMA lanes, element e in lane e mod 8 (:682-691); block pools: sixteen (:371-386)
        constexpr int NA = PAGED ? 16 : 8;
        constexpr int HP = PAGED && GH > 2 ? 2 : GH;    // heads per pass over the row: 2 x HP x NA accumulators live
#pragma unroll
        for (int h0 = 0; h0 < GH; h0 += HP) {
            if (h0 > 0) asm volatile("" ::: "memory");   // convert the row again rather than keep 128 floats of it
            float acc[2][HP][NA];
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int g = 0; g < HP; ++g)
#pragma unroll
                    for (int j = 0; j < NA; ++j) acc[s][g][j] = 0.0f;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float kf[2][16];
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const uint4 kb = *reinterpret_cast<const uint4*>(row[s] + (((uint32_t)c ^ swz[s]) << 4));
                    const uint32_t w[4] = {kb.x ^ 0x80808080u, kb.y ^ 0x80808080u, kb.z ^ 0x80808080u, kb.w ^ 0x80808080u};
#pragma unroll
                    for (int e = 0; e < 16; ++e) kf[s][e] = s8_to_f(w[e >> 2], e & 3);
                }
#pragma unroll
                for (int g = 0; g < HP; ++g)
#pragma unroll
                    for (int e4 = 0; e4 < 4; ++e4) {
                        const float4 q4 = *reinterpret_cast<const float4*>(s_q + (h0 + g) * kHd + c * 16 + e4 * 4);
                        const float qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                float& d = acc[s][g][(e4 * 4 + e) % NA];
                                d = __fmaf_rn(qv[e], kf[s][e4 * 4 + e], d);
                            }
                    }
            }
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int t = t0 + 32 * s + lane;
                float v[HP];
#pragma unroll
                for (int g = 0; g < HP; ++g) {
                    const float* ac = acc[s][g];
                    if constexpr (PAGED) {
                        float dot = 0.0f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) dot = __fadd_rn(dot, __fadd_rn(ac[j], ac[j + 8]));
                        v[g] = __fmul_rn(__fmul_rn(dot, ksc[s]), sm_scale);                          // :388
                    } else {
                        v[g] = (ac[0] + ac[1] + ac[2] + ac[3] + ac[4] + ac[5] + ac[6] + ac[7]) * (ksc[s] * sm_scale);   // :691
                    }
                }
                if (t < k1) {
#pragma unroll
                    for (int g = 0; g < HP; ++g) tmax[h0 + g] = fmaxf(tmax[h0 + g], v[g]);
                    float* o = out + (size_t)t * GH + h0;
                    if constexpr (HP == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                    else if constexpr (HP == 2) *reinterpret_cast<float2*>(o) = make_float2(v[0], v[1]);
                    else o[0] = v[0];
                }
            }
        }
        __syncwarp();                                  // every lane has read the tile
        if (t0 + kScoreWarps * kSpTile < k1) request(t0 + kScoreWarps * kSpTile);
    }
    if (timed_out) atomicExch(&g_split_timeouts, 1);
#pragma unroll
    for (int g = 0; g < GH; ++g) {
        const float m = warp_max(tmax[g]);
        if (lane == 0) s_red[warp][g] = m;
    }
    __syncthreads();
    if (tid < GH) {
        float m = s_red[0][tid];
#pragma unroll
        for (int w = 1; w < kScoreWarps; ++w) m = fmaxf(m, s_red[w][tid]);
        L.span_max[(item * L.n_spans + blockIdx.x) * GH + tid] = m;
    }
}

// Scores -> exponentials (in place) and 1 / sum, for HS heads of an item per CTA. Chunks of keys go through two
// shared-memory buffers: while HS warps add up one chunk, each a head in key order, the others evaluate the next. Many
// items: four heads a CTA and small chunks, so that all CTAs are resident at once; few: one head, long chunks (fewer sums).
// (64 x 8192 keys, 20/5 heads: 46 -> 36 us, 1536 prompt rows 114 -> 102, one sequence of 6003 keys 11.3 -> 10.1, against chunks of 1024
// with a head each, zeros evaluated up to 1216, and segments walked one by one.)
// MANY: more items than three CTAs an SM hold. The summing warps are what an item takes its time for, so half the evaluating
// threads and five CTAs an SM then (a prompt of 1536 rows: 27.75 -> 27.05 ms in all, 640 items of 4096 keys 40 -> 37 us; but
// 320 items of 8192 keys 49 -> 55).
template <int HS, bool MANY> struct SoftShape {
    // keys of the first chunk, and of the others, whose sums need no head: the summing warp's segments hold them without a rest
    static constexpr int eval = HS == 1 ? 512 : MANY ? 128 : 256, threads = eval + 32 * HS, chunk = HS == 1 ? 4032 : HS == 2 ? 1984 : 960, next = chunk - kOrderedHead;
    static constexpr int resident = HS == 1 ? 2 : MANY ? 5 : 3;
};
template <int GH, int HS, bool PAGED, bool MANY>
__global__ void __launch_bounds__(SoftShape<HS, MANY>::threads, SoftShape<HS, MANY>::resident) split_softmax_kernel(const SplitLaunch L) {
    const tenzo_attention_args& a = L.a;
    constexpr int kEval = SoftShape<HS, MANY>::eval, kSoftChunk = SoftShape<HS, MANY>::chunk, kSoftNext = SoftShape<HS, MANY>::next;
    static_assert(ordered_sum_padded(kSoftChunk) == kSoftChunk && ordered_sum_padded(kSoftNext, false) == kSoftNext, "");
    extern __shared__ __align__(16) float s_e[];       // [2][HS][padded chunk]
    __shared__ float s_max[HS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sw = warp - kEval / 32;   // sw >= 0: summing warp of head sw
    const size_t item = blockIdx.x / (GH / HS);
    const int h0 = (int)(blockIdx.x % (GH / HS)) * HS;
    const int chunk = min(kSoftChunk, L.tp), padded = ordered_sum_padded(chunk);
    const unsigned long long tab = kExp2fTab[lane];
    const uint32_t tab_lo = (uint32_t)tab, tab_hi = (uint32_t)(tab >> 32);
    if (a.use_pdl) pdl_wait();
    const int seq = L.seq0 + (int)(item / L.groups), T = __ldcg(a.pos + seq) + 1;
    if (T <= 0 || T > a.max_len) return;
    constexpr int U = 4;                               // keys a thread has in flight
    float x[U][HS];
    float* e = L.scores + item * (size_t)L.tp * GH + h0;
    auto load = [&](int i, int n, int t0) {            // scores of keys t0 + i + u * threads
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = i + u * kEval;
            const float* p = e + (size_t)(t0 + k) * GH;
#pragma unroll
            for (int h = 0; h < HS; ++h) x[u][h] = 0.0f;
            if (k < n) {
                if constexpr (HS == 4) {
                    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
                    x[u][0] = v.x; x[u][1] = v.y; x[u][2] = v.z; x[u][3] = v.w;
                } else if constexpr (HS == 2) {
                    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
                    x[u][0] = v.x; x[u][1] = v.y;
                } else {
                    x[u][0] = __ldcg(p);
                }
            }
        }
    };
    if (sw < 0) load(tid, min(kSoftChunk, T), 0);
    if (sw >= 0) {
        const int spans = (T + L.span - 1) / L.span;
        float m = -1e30f;
        for (int i = lane; i < spans; i += 32) m = fmaxf(m, __ldcg(L.span_max + (item * L.n_spans + i) * GH + h0 + sw));
        m = warp_max(m);
        if (lane == 0) s_max[sw] = m;
    }
    __syncthreads();
    float mx[HS];
#pragma unroll
    for (int h = 0; h < HS; ++h) mx[h] = s_max[h];
    auto evaluate = [&](int c, bool loaded) {          // chunk c: e_t = expf(score_t - max) (:826), zeros behind the last key
        const int t0 = c == 0 ? 0 : kSoftChunk + (c - 1) * kSoftNext, n = min(c == 0 ? kSoftChunk : kSoftNext, T - t0);
        const int n_pad = c > 0 ? ordered_sum_padded(n, false) : n <= kOrderedHead ? kOrderedHead : ordered_sum_padded(n);
        float* dst = s_e + (size_t)(c & 1) * HS * padded;
        for (int i0 = 0; i0 < n_pad; i0 += U * kEval) {
            if (!loaded || i0 > 0) load(i0 + tid, n, t0);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = i0 + u * kEval + tid;
                if (k - lane >= n_pad) break;          // whole warps: the table look-up is a shuffle
#pragma unroll
                for (int h = 0; h < HS; ++h) {
                    x[u][h] = expf_reference_bits_lanes(k < n ? x[u][h] - mx[h] : 0.0f, tab_lo, tab_hi);
                    if (k >= n) x[u][h] = 0.0f;
                    dst[h * padded + k] = x[u][h];
                }
                if (k < n) {
                    float* p = e + (size_t)(t0 + k) * GH;
                    if constexpr (HS == 4) *reinterpret_cast<float4*>(p) = make_float4(x[u][0], x[u][1], x[u][2], x[u][3]);
                    else if constexpr (HS == 2) *reinterpret_cast<float2*>(p) = make_float2(x[u][0], x[u][1]);
                    else p[0] = x[u][0];
                }
            }
        }
    };
    const int n_chunks = T <= kSoftChunk ? 1 : 1 + (T - kSoftChunk + kSoftNext - 1) / kSoftNext;
    float sum = 0.0f;
    if (sw < 0) evaluate(0, true);
    __syncthreads();
    for (int c = 0; c < n_chunks; ++c) {
        const float* mine = s_e + (size_t)(c & 1) * HS * padded + sw * padded;
        if (sw < 0) { if (c + 1 < n_chunks) evaluate(c + 1, false); }
        else if (c == 0) sum = ordered_sum_warp<true>(mine, min(kSoftChunk, T), 0.0f);                                             // :824-829
        else sum = ordered_sum_warp<false>(mine, min(kSoftNext, T - kSoftChunk - (c - 1) * kSoftNext), sum);
        __syncthreads();
    }
    if (sw >= 0 && lane == 0) L.inv_sum[item * GH + h0 + sw] = PAGED ? 1.0f / __fadd_rn(sum, 1e-8f) : 1.0f / sum;   // :400 for block pools
}

// Value sums: a consumer lane owns one or two output dims of GV heads, one chain per head and dim, and walks the keys in
// order (:842-851). Producer warps keep a three-stage ring of key chunks filled and form the weights p_t * s_v[t]
// (:830, :844), so that the consumers only load, convert and multiply-add. Hand-over by named barriers (a poll of an
// mbarrier costs its warp more than a chunk's barrier does). Two shapes (heavy_items), and a third for up to 160 heads in all:
//   heavy  two neighbouring dims a lane and all heads: the fewest instructions and shared-memory cycles an item. Two items a CTA,
//          two consumer warps each; V bytes by bulk copy, two to a load and converted by the consumers (one load a dim: 131 us
//          against 126 at 64 x 8192 keys, 222 and 212 for 1536 prompt rows; what the kernel waits for most is shared memory);
//   light  32 dims and all heads a CTA, one consumer warp: for when there are fewer items than schedulers. Four producer
//          warps convert V to floats, which leaves the consumer a load, the weights and the FMAs. One
//          consumer a CTA because the floats pass the shared-memory pipe twice: four of them, at 13 cycles a key, waited for it;
//   few    one head and 64 dims a CTA, a dim a lane (split_values_few_kernel).
constexpr int kValueThreads = 192;                    // heavy: four consumer warps, one a scheduler, and two producers; light: 1 + 4
constexpr int kValueKeys = 64, kValueStages = 3;
template <int GV>
struct HeavyRing {
    static constexpr int v_bytes = kValueKeys * kHd, w_floats = kValueKeys * GV;
    static constexpr int group_bytes = kValueStages * (v_bytes + 8 * w_floats + 4 * kValueKeys);
    static constexpr int bytes = 2 * group_bytes;
};
template <int GV>
struct LightRing {
    static constexpr int v_floats = kValueKeys * 32, w_floats = kValueKeys * GV;
    static constexpr int bytes = kValueStages * 4 * (v_floats + w_floats);
};

// The two signed bytes of a sign-extended 16-bit load, one converted by the special-function pipe (from 8 bits) and one like an
// FMA (from 32): both from 32 bits, with a permute for the lower byte, is slower (128 us against 126).
__device__ __forceinline__ void bytes_of(int pair, int& lo, int& hi) {
    lo = (int)(int8_t)pair;
    hi = (int)(int8_t)(pair >> 8);
}

// What an item's value sums read.
template <int GH, bool PAGED>
struct ValueItem {
    int seq, head0, T;
    KeyRows<PAGED> rows;
    const int8_t* cv;
    const float *sv, *e, *inv;
    __device__ __forceinline__ ValueItem(const SplitLaunch& L, int item, int sub_head)
        : seq(L.seq0 + item / L.groups), head0((item % L.groups) * GH + sub_head), T(__ldcg(L.a.pos + seq) + 1), rows(L.a, seq, head0 / (L.a.n_q / L.a.n_kv)) {
        const bool one = PAGED || L.shared_cache;
        cv = L.a.cache_v + (one ? 0 : (size_t)seq * L.a.seq_stride_kv);
        sv = L.a.scale_v + (one ? 0 : (size_t)seq * L.a.seq_stride_sc);
        e = L.scores + (size_t)item * L.tp * GH + sub_head;
        inv = L.inv_sum + (size_t)item * GH + sub_head;
        if (T > L.a.max_len) T = 0;                    // refused by the score kernel
    }
};

template <int GV, bool PAGED>
__device__ __forceinline__ void store_weights(float* o, const float (&e)[GV], const float (&inv)[GV], float vs) {
    float wt[GV];
#pragma unroll
    for (int g = 0; g < GV; ++g) {
        const float p = e[g] * inv[g];
        wt[g] = (PAGED && p < 1e-7f) ? 0.0f : p * vs;  // block pools drop keys under 1e-7 (:416); a zero weight changes no sum
    }
    if constexpr (GV == 4) *reinterpret_cast<float4*>(o) = make_float4(wt[0], wt[1], wt[2], wt[3]);
    else if constexpr (GV == 2) *reinterpret_cast<float2*>(o) = make_float2(wt[0], wt[1]);
    else o[0] = wt[0];
}

template <int GV>
__device__ __forceinline__ void load_vec(const float* p, float (&v)[GV]) {
    if constexpr (GV == 4) {
        const float4 q = __ldcg(reinterpret_cast<const float4*>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else if constexpr (GV == 2) {
        const float2 q = __ldcg(reinterpret_cast<const float2*>(p));
        v[0] = q.x; v[1] = q.y;
    } else {
        v[0] = __ldcg(p);
    }
}

// The producer warp of a group of consumers: V rows as they come, weights of GV heads, a ring of kValueStages chunks of KEYS keys.
template <int GH, int GV, int KEYS, bool PAGED>
__device__ __forceinline__ void produce_values(const ValueItem<GH, PAGED>& it, int n_chunks, unsigned char* s_v, float* s_e, float* s_w, float* s_s,
                                               uint64_t* s_bar, int bar_full, int bar_free, int count) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        for (int i = 0; i < kValueStages; ++i) mbar_init(&s_bar[i], 1);
        mbar_init_fence();
    }
    __syncwarp();
    float inv[GV];
    load_vec<GV>(it.inv, inv);
    // Block pools: lane l holds block l of the next chunk, fetched a chunk ahead (an address that waits for the table puts its round
    // trip on every chunk).
    auto block_of = [&](int c) { return PAGED && lane < KEYS / 16 && c * KEYS + 16 * lane < it.T ? __ldg(it.rows.table + c * (KEYS / 16) + lane) : 0; };
    auto row_of = [&](int block) { return (((size_t)block * it.rows.n_layers + it.rows.layer) * it.rows.n_kv + it.rows.kvh) * 16; };
    int next_block = block_of(0);
    auto request = [&](int c) {
        if (c < n_chunks) {
            const int block = next_block;
            next_block = block_of(c + 1);
            const int st = c % kValueStages, t0 = c * KEYS, n = min(KEYS, it.T - t0);
            if (lane == 0) mbar_expect_tx(&s_bar[st], (unsigned)n * kHd);
            __syncwarp();
            unsigned char* dst = s_v + st * (KEYS * kHd);
            if constexpr (PAGED) {
                if (16 * lane < n) bulk_g2s(dst + lane * 16 * kHd, it.cv + row_of(block) * kHd, (unsigned)min(16, n - 16 * lane) * kHd, &s_bar[st]);
            } else {
                if (lane == 0) bulk_g2s(dst, it.cv + it.rows.row(t0) * kHd, (unsigned)n * kHd, &s_bar[st]);
            }
#pragma unroll
            for (int i = 0; i < KEYS / 32; ++i) {
                const int k = 32 * i + lane;
                const size_t r = PAGED ? row_of(__shfl_sync(0xffffffffu, block, k >> 4)) + (k & 15) : it.rows.row(t0 + k);
                if (k < n) {
                    cp_async<4 * GV>(s_e + st * (KEYS * GV) + k * GV, it.e + (size_t)(t0 + k) * GH);
                    cp_async<4>(s_s + st * KEYS + k, it.sv + r);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");       // one group a chunk, empty behind the last
    };
    bool timed_out = false;
    for (int c = 0; c < kValueStages - 1; ++c) request(c);
    for (int c = 0; c < n_chunks; ++c) {
        const int st = c % kValueStages;
        asm volatile("cp.async.wait_group %0;" ::"n"(kValueStages - 2) : "memory");
#pragma unroll
        for (int i = 0; i < KEYS / 32; ++i) {                              // a lane's own copies
            const int k = 32 * i + lane;
            float ev[GV];
#pragma unroll
            for (int g = 0; g < GV; ++g) ev[g] = s_e[st * (KEYS * GV) + k * GV + g];
            store_weights<GV, PAGED>(s_w + st * (KEYS * GV) + k * GV, ev, inv, s_s[st * KEYS + k]);
        }
        if (!mbar_wait_bounded(&s_bar[st], (unsigned)(c / kValueStages) & 1u)) timed_out = true;
        named_barrier_arrive(bar_full + st, count);
        if (c > 0 && c + kValueStages - 1 < n_chunks) named_barrier_sync(bar_free + (c - 1) % kValueStages, count);   // chunk c - 1 has been read
        request(c + kValueStages - 1);
    }
    if (timed_out) atomicExch(&g_split_timeouts, 1);
}

template <int GH, bool PAGED>
__device__ __forceinline__ void split_values_heavy(const SplitLaunch& L, unsigned char* smem, uint64_t (*s_bars)[kValueStages], int block, int n_items) {
    using Ring = HeavyRing<GH>;
    constexpr int U = 8, kCount = 96;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = warp < 4 ? warp >> 1 : warp - 4, item = 2 * block + grp;
    if (grp >= 2 || item >= n_items) return;
    const ValueItem<GH, PAGED> it(L, item, 0);
    if (it.T <= 0) return;
    unsigned char* s_v = smem + (size_t)grp * Ring::group_bytes;                                 // [stages][keys][128]
    float* s_e = reinterpret_cast<float*>(s_v + kValueStages * Ring::v_bytes);                   // [stages][keys][GH]
    float* s_w = s_e + kValueStages * Ring::w_floats;                                            // [stages][keys][GH]
    float* s_s = s_w + kValueStages * Ring::w_floats;                                            // [stages][keys]
    const int bar_full = 1 + grp * 2 * kValueStages, bar_free = bar_full + kValueStages;
    const int n_chunks = (it.T + kValueKeys - 1) / kValueKeys;
    if (warp >= 4) {
        produce_values<GH, GH, kValueKeys, PAGED>(it, n_chunks, s_v, s_e, s_w, s_s, s_bars[grp], bar_full, bar_free, kCount);
        return;
    }
    const int part = warp & 1;
    float acc[GH][2];
#pragma unroll
    for (int g = 0; g < GH; ++g) acc[g][0] = acc[g][1] = 0.0f;
    for (int c = 0; c < n_chunks; ++c) {
        const int st = c % kValueStages;
        named_barrier_sync(bar_full + st, kCount);
        const int8_t* vp = reinterpret_cast<const int8_t*>(s_v + st * Ring::v_bytes) + 64 * part + 2 * lane;
        const float* wp = s_w + st * Ring::w_floats;
        const int n = min(kValueKeys, it.T - c * kValueKeys);
        auto load_v = [&](int k) { return (int)*reinterpret_cast<const int16_t*>(vp + k * kHd); };
        if (n == kValueKeys) {
            // three batches of eight keys under way, interleaved key by key: raw bytes on their way from shared memory,
            // bytes being converted, and values being summed
            int raw[U];
            float f[2][U][2], w[2][U][GH];
            auto load_w = [&](int k, int b, int i) {           // the i-th 16 bytes of eight keys' weights
                const float4 q = reinterpret_cast<const float4*>(wp + k * GH)[i];
                w[b][(4 * i) / GH][(4 * i) % GH] = q.x;
                w[b][(4 * i + 1) / GH][(4 * i + 1) % GH] = q.y;
                w[b][(4 * i + 2) / GH][(4 * i + 2) % GH] = q.z;
                w[b][(4 * i + 3) / GH][(4 * i + 3) % GH] = q.w;
            };
            auto convert = [&](int b, int u) {
                int lo, hi;
                bytes_of(raw[u], lo, hi);
                f[b][u][0] = (float)lo;
                f[b][u][1] = (float)hi;
            };
#pragma unroll
            for (int u = 0; u < U; ++u) raw[u] = load_v(u);
#pragma unroll
            for (int i = 0; i < U * GH / 4; ++i) load_w(0, 0, i);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                convert(0, u);
                raw[u] = load_v(U + u);
            }
#pragma unroll
            for (int k = 0; k < kValueKeys; k += U) {
                const int b = (k / U) & 1;
#pragma unroll
                for (int u = 0; u < U; ++u) {
#pragma unroll
                    for (int d = 0; d < 2; ++d)
#pragma unroll
                        for (int g = 0; g < GH; ++g) acc[g][d] = __fmaf_rn(f[b][u][d], w[b][u][g], acc[g][d]);
                    if (k + U < kValueKeys) convert(b ^ 1, u);
                    if (k + 2 * U < kValueKeys) raw[u] = load_v(k + 2 * U + u);
                    if (k + U < kValueKeys)
#pragma unroll
                        for (int i = u * GH / 4; i < (u + 1) * GH / 4; ++i) load_w(k + U, b ^ 1, i);
                }
            }
        } else {                                       // the last chunk
#pragma unroll 4
            for (int k = 0; k < n; ++k) {
                int lo, hi;
                bytes_of(load_v(k), lo, hi);
#pragma unroll
                for (int g = 0; g < GH; ++g) {
                    acc[g][0] = __fmaf_rn((float)lo, wp[k * GH + g], acc[g][0]);
                    acc[g][1] = __fmaf_rn((float)hi, wp[k * GH + g], acc[g][1]);
                }
            }
        }
        if (c + kValueStages < n_chunks) named_barrier_arrive(bar_free + st, kCount);
    }
    float* out = L.a.out + ((size_t)it.seq * L.a.n_q + it.head0) * kHd + 64 * part + 2 * lane;
#pragma unroll
    for (int g = 0; g < GH; ++g)
#pragma unroll
        for (int d = 0; d < 2; ++d) out[g * kHd + d] = acc[g][d];
}

// All heads and 32 dims of an item a CTA. Producer warp p converts keys 16 p .. 16 p + 15 of a chunk (in block pools: one block),
// one 16-byte piece a lane, fetched four chunks ahead. Word j of piece q of key r goes to the 16 bytes (2 j + q) ^ 2 (r & 3)
// of the key's row, which keeps the stores of a warp free of bank conflicts; consumer lane l reads the floats of dim
// 16 ((l >> 2) & 1) + 4 (l >> 3) + (l & 3).
template <int GH, bool PAGED>
__device__ __forceinline__ void split_values_light(const SplitLaunch& L, unsigned char* smem, int block, int item0) {
    using Ring = LightRing<GH>;
    constexpr int GV = GH, kCount = 160, kAhead = 4;
    const int lane = threadIdx.x & 31, warp = ((threadIdx.x >> 5) + block) % 6;      // consumers of successive CTAs on different schedulers
    const int part = block & 3, group = block >> 2;
    if (warp == 5) return;
    const ValueItem<GH, PAGED> it(L, item0 + group, 0);
    if (it.T <= 0) return;
    float* s_v = reinterpret_cast<float*>(smem);                                                 // [stages][keys][32]
    float* s_w = s_v + kValueStages * Ring::v_floats;                                            // [stages][keys][GV]
    const int n_chunks = (it.T + kValueKeys - 1) / kValueKeys;
    if (warp > 0) {
        const int p = warp - 1, r = lane >> 1, q = lane & 1;
        uint4 v[kAhead];
        float ev[kAhead][GV], vs[kAhead], inv[GV];
        load_vec<GV>(it.inv, inv);
        auto fetch = [&](int c, int b) {
            const int t0 = c * kValueKeys + 16 * p, n = it.T - t0;
            v[b] = make_uint4(0u, 0u, 0u, 0u);
            vs[b] = 0.0f;
#pragma unroll
            for (int g = 0; g < GV; ++g) ev[b][g] = 0.0f;
            if (n > 0) {
                const size_t row0 = it.rows.row(t0);
                if (r < n) v[b] = ld_cg_u4(it.cv + (row0 + r) * kHd + 32 * part + 16 * q);
                if (lane < 16 && lane < n) {
                    load_vec<GV>(it.e + (size_t)(t0 + lane) * GH, ev[b]);
                    vs[b] = __ldcg(it.sv + row0 + lane);
                }
            }
        };
        auto put = [&](int c, int b) {
            const int st = c % kValueStages;
            float* dst = s_v + st * Ring::v_floats + (16 * p + r) * 32;
            const uint32_t w4[4] = {v[b].x ^ 0x80808080u, v[b].y ^ 0x80808080u, v[b].z ^ 0x80808080u, v[b].w ^ 0x80808080u};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(dst + 4 * ((2 * j + q) ^ (2 * (r & 3)))) = make_float4(s8_to_f(w4[j], 0), s8_to_f(w4[j], 1), s8_to_f(w4[j], 2), s8_to_f(w4[j], 3));
            if (lane < 16) store_weights<GV, PAGED>(s_w + st * Ring::w_floats + (16 * p + lane) * GV, ev[b], inv, vs[b]);
        };
#pragma unroll
        for (int b = 0; b < kAhead; ++b) fetch(b, b);
        for (int c0 = 0; c0 < n_chunks; c0 += kAhead) {
#pragma unroll
            for (int b = 0; b < kAhead; ++b) {
                const int c = c0 + b;
                if (c >= n_chunks) break;
                if (c >= kValueStages) named_barrier_sync(1 + kValueStages + c % kValueStages, kCount);
                put(c, b);
                named_barrier_arrive(1 + c % kValueStages, kCount);
                fetch(c + kAhead, b);
            }
        }
        return;
    }
    float acc[GV];
#pragma unroll
    for (int g = 0; g < GV; ++g) acc[g] = 0.0f;
    int col[4];                                        // this lane's column in the rows of keys 0..3 mod 4
#pragma unroll
    for (int i = 0; i < 4; ++i) col[i] = 4 * ((lane >> 2) ^ (2 * i)) + (lane & 3);
    // Sixteen (eight) keys a step; a chunk's last step is summed while the next chunk's first one is on its way from shared memory,
    // so that the chain does not stop at the hand-over.
    constexpr int U = GV == 1 ? 16 : 8;
    float f[U], w[U * GV];
    auto load = [&](int st, int k) {
        const float* vp = s_v + st * Ring::v_floats + k * 32;
        const float4* wp = reinterpret_cast<const float4*>(s_w + st * Ring::w_floats + k * GV);
#pragma unroll
        for (int u = 0; u < U; ++u) f[u] = vp[u * 32 + col[u & 3]];
#pragma unroll
        for (int i = 0; i < U * GV / 4; ++i) {
            const float4 x = wp[i];
            w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
        }
    };
    auto sum = [&](const float (&fs)[U], const float (&ws)[U * GV]) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int g = 0; g < GV; ++g) acc[g] = __fmaf_rn(fs[u], ws[u * GV + g], acc[g]);
    };
    const int full = it.T / kValueKeys;                // whole chunks
    if (full > 0) {
        named_barrier_sync(1, kCount);
        load(0, 0);
    }
    for (int c = 0; c < full; ++c) {
        const int st = c % kValueStages;
#pragma unroll
        for (int k = U; k <= kValueKeys; k += U) {
            float f0[U], w0[U * GV];
#pragma unroll
            for (int u = 0; u < U; ++u) f0[u] = f[u];
#pragma unroll
            for (int u = 0; u < U * GV; ++u) w0[u] = w[u];
            if (k < kValueKeys) {
                load(st, k);
            } else {
                if (c + kValueStages < n_chunks) named_barrier_arrive(1 + kValueStages + st, kCount);    // every key of the chunk is in registers
                if (c + 1 < full) {
                    named_barrier_sync(1 + (c + 1) % kValueStages, kCount);
                    load((c + 1) % kValueStages, 0);
                }
            }
            sum(f0, w0);
        }
    }
    if (full < n_chunks) {                             // the keys behind the last whole chunk
        const int st = full % kValueStages, n = it.T - full * kValueKeys;
        named_barrier_sync(1 + st, kCount);
        const float* vp = s_v + st * Ring::v_floats;
        const float* wp = s_w + st * Ring::w_floats;
#pragma unroll 1
        for (int k = 0; k < n; k += 4)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < n) {
                    const float v = vp[(k + u) * 32 + col[u]];
#pragma unroll
                    for (int g = 0; g < GV; ++g) acc[g] = __fmaf_rn(v, wp[(k + u) * GV + g], acc[g]);
                }
    }
    float* out = L.a.out + ((size_t)it.seq * L.a.n_q + it.head0) * kHd + 32 * part + 16 * ((lane >> 2) & 1) + 4 * (lane >> 3) + (lane & 3);
#pragma unroll
    for (int g = 0; g < GV; ++g) out[g * kHd] = acc[g];
}

// Few heads (up to eight sequences of 20): a CTA has one head and 64 dims, a dim a lane and a consumer warp a scheduler, and beside a chain's
// multiply-add there is only a byte load, a conversion and a quarter of a weight load a key. A batch of eight keys is
// summed while the next is converted and the one after that is on its way from shared memory, over the chunks' ends too.
// 24.2 us for one sequence of 6003 keys and 44.9 for 12000 are 3.5 us and 6.8 cycles a key, where the chain alone would take the
// multiply-add's 4.6: 3.9 warp instructions a key (producers included), 37 % of the issue slots used, stalls mostly fixed latencies.
// Chunks of 256 keys: a chunk costs the producer warp some 700 cycles whatever it holds. One sequence of 6003 keys: 30.4 us with V
// converted to floats by four producer warps (8.8 cycles a key, as long as the producers took), here 33.2 with chunks of 64 keys,
// 25.7 of 128 and 24.0 of 256; two sequences up to 5000 32.0 -> 20.7.
constexpr int kFewThreads = 96, kFewKeys = 256;
constexpr int kFewBytes = kValueStages * (kFewKeys * kHd + 12 * kFewKeys);
template <int GH, bool PAGED>
__global__ void __launch_bounds__(kFewThreads) split_values_few_kernel(const SplitLaunch L) {
    extern __shared__ __align__(128) unsigned char s_v[];                                        // [stages][keys][128]
    __shared__ uint64_t s_bar[kValueStages];
    float* s_e = reinterpret_cast<float*>(s_v + kValueStages * kFewKeys * kHd);                // [stages][keys]
    float* s_w = s_e + kValueStages * kFewKeys;
    float* s_s = s_w + kValueStages * kFewKeys;
    constexpr int U = 8, kBatches = kFewKeys / U, bar_full = 1, bar_free = 1 + kValueStages;
    if (L.a.use_pdl) pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = blockIdx.x & 1, unit = blockIdx.x >> 1;
    const ValueItem<GH, PAGED> it(L, unit / GH, unit % GH);
    if (it.T <= 0) return;
    const int n_chunks = (it.T + kFewKeys - 1) / kFewKeys, full = it.T / kFewKeys;
    if (warp == 2) {
        produce_values<GH, 1, kFewKeys, PAGED>(it, n_chunks, s_v, s_e, s_w, s_s, s_bar, bar_full, bar_free, kFewThreads);
        return;
    }
    const int dim = 64 * half + 32 * warp + lane;
    float acc = 0.0f, f[2][U], w[2][U];
    int raw[U];
    auto load_v = [&](int st, int k) {                 // (a load that extends the sign, converted from 32 bits: that conversion issues like an FMA)
        int x = reinterpret_cast<const int8_t*>(s_v)[(st * kFewKeys + k) * kHd + dim];
        asm("" : "+r"(x));
        return x;
    };
    auto load_w = [&](int st, int k, int b, int i) {   // the i-th four of eight weights
        const float4 q = *reinterpret_cast<const float4*>(s_w + st * kFewKeys + k + 4 * i);
        w[b][4 * i] = q.x; w[b][4 * i + 1] = q.y; w[b][4 * i + 2] = q.z; w[b][4 * i + 3] = q.w;
    };
    if (full > 0) {
        named_barrier_sync(bar_full, kFewThreads);
#pragma unroll
        for (int u = 0; u < U; ++u) raw[u] = load_v(0, u);
        load_w(0, 0, 0, 0);
        load_w(0, 0, 0, 1);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f[0][u] = (float)raw[u];
            raw[u] = load_v(0, U + u);
        }
    }
    int st = 0;
    for (int c = 0; c < full; ++c) {
        const int next = st + 1 == kValueStages ? 0 : st + 1;
        const bool more = c + 1 < full;
#pragma unroll
        for (int j = 0; j < kBatches; ++j) {           // batch j is summed, j + 1 converted, j + 2 loaded
            const int b = j & 1;
            if (j == kBatches - 2 && more) named_barrier_sync(bar_full + next, kFewThreads);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                acc = __fmaf_rn(f[b][u], w[b][u], acc);
                if (j < kBatches - 1 || more) f[b ^ 1][u] = (float)raw[u];
                if (j < kBatches - 2) raw[u] = load_v(st, (j + 2) * U + u);
                else if (more) raw[u] = load_v(next, (j + 2 - kBatches) * U + u);
                if ((u & 3) == 3) {
                    if (j < kBatches - 1) load_w(st, (j + 1) * U, b ^ 1, u >> 2);
                    else if (more) load_w(next, 0, b ^ 1, u >> 2);
                }
            }
            if (j == kBatches - 2 && c + kValueStages < n_chunks) named_barrier_arrive(bar_free + st, kFewThreads);      // the chunk is in registers
        }
        st = next;
    }
    if (full < n_chunks) {                             // the keys behind the last whole chunk
        const int n = it.T - full * kFewKeys;
        named_barrier_sync(bar_full + st, kFewThreads);
#pragma unroll 4
        for (int k = 0; k < n; ++k) acc = __fmaf_rn((float)load_v(st, k), s_w[st * kFewKeys + k], acc);
    }
    L.a.out[((size_t)it.seq * L.a.n_q + it.head0) * kHd + dim] = acc;
}

// The first `heavy` items in the heavy shape, the rest in the light one.
template <int GH, bool PAGED>
__global__ void __launch_bounds__(kValueThreads, 3) split_values_kernel(const SplitLaunch L, int heavy) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t s_bars[2][kValueStages];
    if (L.a.use_pdl) pdl_wait();
    const int heavy_blocks = (heavy + 1) / 2;
    if ((int)blockIdx.x < heavy_blocks) split_values_heavy<GH, PAGED>(L, smem_raw, s_bars, blockIdx.x, heavy);
    else split_values_light<GH, PAGED>(L, smem_raw, blockIdx.x - heavy_blocks, heavy);
}

// ---- host side ---------------------------------------------------------------------------------------------------------
static int split_group(int n_q, int n_kv) { const int g = n_q / n_kv; return g > 4 ? 4 : g; }

static size_t split_bytes_per_seq(int n_q, int max_len) {
    const size_t tp = ((size_t)max_len + 3) & ~(size_t)3, spans = ((size_t)max_len + kScoreWarps * kSpTile - 1) / (kScoreWarps * kSpTile);
    return (size_t)n_q * (tp + spans + 1) * sizeof(float);
}
// Scores of one pass: a batch whose scores need more goes through in several passes, so that they stay in L2 (126 MB)
// between the kernels and the scratch stays bounded.
constexpr size_t kSplitPassBytes = (size_t)64 << 20;

size_t attn_split_workspace_bytes(int batch, int n_q, int max_len) {
    const size_t per_seq = split_bytes_per_seq(n_q, max_len), all = per_seq * (size_t)batch;
    const size_t cap = kSplitPassBytes > per_seq ? kSplitPassBytes : per_seq;
    return (all < cap ? all : cap) + 256;
}

bool attn_split_possible(const tenzo_attention_args& a) {
    if (!a.workspace || (reinterpret_cast<uintptr_t>(a.workspace) & 15) || a.workspace_bytes < split_bytes_per_seq(a.n_q, a.max_len) + 64) return false;
    if ((reinterpret_cast<uintptr_t>(a.cache_k) & 15) || (reinterpret_cast<uintptr_t>(a.cache_v) & 15) ) return false;
    if (a.block_table) return a.n_pool_blocks > 0 && (long long)a.n_pool_blocks * a.n_layers * a.n_kv * 16 < (1LL << 31);
    return a.seq_stride_kv % 16 == 0 && (long long)(a.layer + 1) * a.n_kv * a.max_seq < (1LL << 31);
}

// The K cache as a byte tensor {128, rows, sequences} read in boxes of 64 rows; block pools: {128, rows of the pool} in boxes
// of one block's 16 rows. Rows past the layers up to this one are zero-filled and never used.
static int k_tensor_map(const SplitLaunch& L, CUtensorMap* out) {
    const tenzo_attention_args& a = L.a;
    if (a.block_table)
        return encode_2d(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.cache_k, kHd, (uint64_t)a.n_pool_blocks * a.n_layers * a.n_kv * 16, kHd, kHd, 16u, CU_TENSOR_MAP_SWIZZLE_128B);
    const uint64_t rows = (uint64_t)(a.layer + 1) * a.n_kv * a.max_seq;
    const bool one = L.shared_cache || a.batch == 1;
    return encode_3d_bytes(out, a.cache_k, kHd, rows, one ? 1u : (uint64_t)a.batch, one ? rows * kHd : (uint64_t)a.seq_stride_kv, kHd, (uint32_t)kSpTile, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <typename... KArgs, typename... Args>
static cudaError_t split_launch(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool pdl, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// How the value sums of `items` items are cut. Heavy items run best when each of the 592 schedulers (148 SMs) has the same
// number of their warps, so whole rounds of 296 items are heavy; a rest that would leave most SMs idle for a round, and a
// batch as small as that, is light (64 x 8192 keys, 20/5 heads: 276 us all heavy, 253 with 24 of the 320 items light; 60 items of
// 1500 36.8 all heavy and 35.7 all light, 70 items 37.5 and 36.3, 80 items 42.1 and 48.1; 100 items of 2048 54.8 and 62.3). Behind a whole round
// an SM takes one light CTA, 37 items in all; two of them are slower than another heavy one (value sums of 3000 keys a sequence in us, the rest
// light and all heavy: 320 items 49.2 and 58.9, 335 75.6 and 59.0, 370 75.4 and 59.4). Behind
// two rounds and more it is a few per cent either way, and which depends on the lengths, which the host does not know: two light CTAs an SM cost equal lengths
// what a heavy round saves, and ragged ones end sooner with them. The line is a compromise between those (whole calls in us, the rest light and all heavy; equal 1800 keys,
// spread over a factor of two, spread from 100 to 3000 keys: 630 items 127.4 and 127.7, 112.0 and 108.0, 144.2 and 156.0; 640 130.8 and 128.0, 108.1 and 109.5,
// 132.8 and 130.2; 650 133.6 and 128.5, 113.8 and 114.7, 149.0 and 156.4; 675 140.3 and 131.7, 114.7 and 113.2, 150.4 and 160.3; 690 141.8 and 133.2, 119.5 and 115.7, 139.3 and
// 148.2; 945 175.7 and 174.1, 149.1 and 148.2, 178.6 and 186.6; 1240 214.9 and 213.5, 178.7 and 177.7, 226.0 and 224.6). Up to kFewHeads heads, a consumer warp a scheduler, take the form of one head a CTA
// (light and this form, value sums in us: 60 heads up to 3000 keys 20.1 and 14.4, 80 heads of 6000 44.2 and 35.0, 120 heads up to 1500 13.8 and 11.2, 128
// of 16/16 up to 2000 18.1 and 14.0, 160 up to 1500 15.8 and 12.7 and of 6000 66.1 and 66.4; 240 heads up to 1500 16.9 and 17.9).
constexpr int kFewHeads = 160;
static int heavy_items(long long items) {
    const long long rest = items % 296;
    return (int)(rest <= (items < 296 ? 70 : items < 592 ? 37 : 60) ? items - rest : items);
}

}  // namespace tz
#include "attention_rows.cuh"        // many query rows over one cache
namespace tz {

template <int GH, bool PAGED>
static cudaError_t launch_values(const SplitLaunch& L, int items, cudaStream_t st) {
    if (items * GH <= kFewHeads) {
        cudaError_t e = allow_smem(split_values_few_kernel<GH, PAGED>, kFewBytes);
        if (e != cudaSuccess) return e;
        return split_launch(split_values_few_kernel<GH, PAGED>, dim3((unsigned)(items * GH * 2)), kFewThreads, kFewBytes, st, L.a.use_pdl != 0, L);
    }
    const int heavy = heavy_items(items), smem = heavy ? HeavyRing<GH>::bytes : LightRing<GH>::bytes;
    static_assert(HeavyRing<GH>::bytes >= LightRing<GH>::bytes, "");
    cudaError_t e = allow_smem(split_values_kernel<GH, PAGED>, HeavyRing<GH>::bytes);
    if (e != cudaSuccess) return e;
    const int blocks = (heavy + 1) / 2 + (items - heavy) * 4;
    return split_launch(split_values_kernel<GH, PAGED>, dim3((unsigned)blocks), kValueThreads, smem, st, L.a.use_pdl != 0, L, heavy);
}

template <int GH, int HS, bool PAGED, bool MANY = false>
static cudaError_t launch_softmax(const SplitLaunch& L, long long items, cudaStream_t st) {
    using Shape = SoftShape<HS, MANY>;
    const int chunk = L.tp < Shape::chunk ? L.tp : Shape::chunk;
    const size_t smem = (size_t)2 * HS * ordered_sum_padded(chunk) * sizeof(float);
    static_assert(2 * HS * ordered_sum_padded(Shape::chunk) * sizeof(float) <= 47 * 1024, "more than a kernel may have without asking");
    return split_launch(split_softmax_kernel<GH, HS, PAGED, MANY>, dim3((unsigned)(items * (GH / HS))), Shape::threads, smem, st, L.a.use_pdl != 0, L);
}

template <int GH, bool PAGED>
static cudaError_t split_pass(const SplitLaunch& L, int n_seq, cudaStream_t st) {
    CUtensorMap km;
    if (k_tensor_map(L, &km)) return cudaErrorInvalidValue;
    const size_t smem = 1024 + (size_t)kScoreWarps * kSpTileBytes;
    cudaError_t e = allow_smem(split_scores_kernel<GH, PAGED>, smem);
    if (e != cudaSuccess) return e;
    e = split_launch(split_scores_kernel<GH, PAGED>, dim3((unsigned)L.n_spans, (unsigned)L.groups, (unsigned)n_seq), kScoreWarps * 32, smem, st, L.a.use_pdl != 0, L, km);
    if (e != cudaSuccess) return e;
    const long long items = (long long)n_seq * L.groups;
    if (GH > 1 && items > 3 * 148) e = launch_softmax<GH, GH, PAGED, GH != 1>(L, items, st);
    else e = GH == 1 || items >= 148 ? launch_softmax<GH, GH, PAGED>(L, items, st) : launch_softmax<GH, 1, PAGED>(L, items, st);
    if (e != cudaSuccess) return e;
    return launch_values<GH, PAGED>(L, (int)items, st);
}

static int split_rows_per_pass(const tenzo_attention_args& a) {
    const size_t per_seq = split_bytes_per_seq(a.n_q, a.max_len), cap = kSplitPassBytes > per_seq ? kSplitPassBytes : per_seq;
    const size_t room = a.workspace_bytes - 64 < cap ? a.workspace_bytes - 64 : cap;
    const int fit = room / per_seq < (size_t)a.batch ? (int)(room / per_seq) : a.batch, passes = (a.batch + fit - 1) / fit;
    return (a.batch + passes - 1) / passes;
}

int attn_split_kernels(const tenzo_attention_args& a) {
    if (const int rows = attn_rows_per_pass(a)) return 4 * ((a.batch + rows - 1) / rows);
    const int per_pass = split_rows_per_pass(a);
    return 3 * ((a.batch + per_pass - 1) / per_pass);
}

// Against the one kernel of attention.cu, above the 256 keys that attention_short.cuh takes (us in a graph, one kernel and three). With heads
// for every SM the three win (12 x 1500: 50 and 34). With fewer the one kernel is a chain as long as the context, the three have
// their fixed cost: one sequence of 512 keys 10.1 and 11.9, of 640 13.0 and 12.8, of 768 15.1 and 12.6, of 1024 19.2 and 15.3; from block
// pools, where the one kernel reads through the table key by key, 400 13.4 and 14.5, 512 15.4 and 14.3, 1024 26.0 and 17.0. Above two sequences'
// heads it is less: 80 heads 768 keys 15.3 and 15.5, 900 18.3 and 17.6, pools 512 15.3 and 15.0, 640 18.5 and 17.5. max_len is an upper bound that
// callers round up, so each line lies a step further.
constexpr int kLineHeads = 40;
bool attn_split_preferred(const tenzo_attention_args& a) {
    const long long heads = (long long)a.batch * a.n_q;
    if (heads >= 256) return true;
    if (heads >= 148) return a.max_len > 256;
    if (a.block_table) return a.max_len > (heads <= kLineHeads ? 512 : 640);
    return a.max_len > (heads <= kLineHeads ? 768 : 1024);
}

int attn_split_run(const tenzo_attention_args& a, cudaStream_t st) {
    if (const int rows = attn_rows_per_pass(a)) return attn_rows_run(a, rows, st);
    SplitLaunch L;
    L.a = a;
    if (L.a.q_stride <= 0) L.a.q_stride = a.n_q * kHd;
    if (L.a.kv_stride <= 0) L.a.kv_stride = a.n_kv * kHd;
    L.shared_cache = a.batch > 1 && !a.block_table && a.seq_stride_kv == 0;
    L.tp = (a.max_len + 3) & ~3;
    const int per_pass = split_rows_per_pass(a);
    // Heads per pass over the keys: as many as share the kv head, fewer when the score CTAs would not cover the SMs.
    const int base_span = kScoreWarps * kSpTile;
    L.gh = split_group(a.n_q, a.n_kv);
    while (L.gh > 1 && (long long)per_pass * (a.n_q / L.gh) * ((a.max_len + base_span - 1) / base_span) < 148) L.gh >>= 1;
    L.groups = a.n_q / L.gh;
    // Keys per score CTA: longer spans spread the rotation and the first tile's latency over more keys, as long as every SM
    // still gets several CTAs.
    L.span = base_span;
    while (L.span < 4 * base_span && (long long)per_pass * L.groups * ((a.max_len + 2 * L.span - 1) / (2 * L.span)) >= 8 * 148) L.span *= 2;
    L.n_spans = (a.max_len + L.span - 1) / L.span;
    L.scores = static_cast<float*>(a.workspace);
    L.span_max = L.scores + (size_t)per_pass * a.n_q * L.tp;
    L.inv_sum = L.span_max + (size_t)per_pass * a.n_q * L.n_spans;
    for (L.seq0 = 0; L.seq0 < a.batch; L.seq0 += per_pass) {
        const int n = a.batch - L.seq0 < per_pass ? a.batch - L.seq0 : per_pass;
        cudaError_t e;
        if (a.block_table)
            e = L.gh == 4 ? split_pass<4, true>(L, n, st) : L.gh == 2 ? split_pass<2, true>(L, n, st) : split_pass<1, true>(L, n, st);
        else
            e = L.gh == 4 ? split_pass<4, false>(L, n, st) : L.gh == 2 ? split_pass<2, false>(L, n, st) : split_pass<1, false>(L, n, st);
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

const int* attn_split_timeouts_flag() {
    void* p = nullptr;
    return cudaGetSymbolAddress(&p, g_split_timeouts) == cudaSuccess ? static_cast<const int*>(p) : nullptr;
}
int attn_split_take_timeouts() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_split_timeouts, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_split_timeouts, &zero, sizeof zero);
    return v;
}

}  // namespace tz

extern "C" size_t tenzo_cuda_attention_rows_workspace_bytes(int batch, int n_q, int n_kv, int max_len) {
    if (batch <= 0 || n_q <= 0 || n_kv <= 0 || n_q % n_kv || n_q / n_kv > 8 || max_len <= 0) return 0;
    const size_t split = tz::attn_split_workspace_bytes(batch, n_q, max_len), rows = tz::rows_workspace_bytes(batch, n_q, n_kv, max_len);
    return split > rows ? split : rows;
}

extern "C" size_t tenzo_cuda_attention_exact_workspace_bytes(int batch, int n_q, int n_kv, int max_len) {
    if (batch <= 0 || n_q <= 0 || n_kv <= 0 || n_q % n_kv || max_len <= 0) return 0;
    return tz::attn_split_workspace_bytes(batch, n_q, max_len);
}
