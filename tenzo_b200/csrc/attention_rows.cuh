// Attention in the reference's operation order for many query rows over ONE cache (the rows of a prompt), in scratch of the caller's.
// Same function and same bits as attention.cu (FusedKVCache::forward_attention_raw, src/runtime/TenzoEngine.cpp:447-533,
// :657-694, :823-851 of the reference).
//
// What the rows share. attention_split.cu takes an item (row, kv head) by itself: every key's bytes are loaded and made floats
// once for its four heads, 12 of the 30 cycles a scheduler spends on them. Here the 64 query vectors of a kv head that
// 64 / G neighbouring rows have (G heads a kv head) go through the keys together, and both contractions are matrix products
// whose order of summation is the reference's:
//   scores   chain j of eight (elements j, j + 8, ...) is a product over 16 elements; a lane holds 8 vectors x 8 keys of one
//            chain, runs its 16 multiply-adds, adds it to the sum of the chains before, and goes on with the next chain;
//   softmax  sixteen warps evaluate the exponentials of 32 (row, head) pairs, a lane of another adds up a pair's in order;
//   values   a lane holds 8 vectors x 8 dims, one chain each, and walks the keys; the weights e / sum * scale_v are zero behind a row's
//            last key, which changes no sum.
// The cache's bytes become floats once a call (rows_prepare_kernel), in the order in which a tile holds them, so that a tile's half is one bulk
// copy. (Converted by every CTA on its way into shared memory, 1536 rows took 383 us, with 37 % of the value sums' time in it.)
//
// What bounds it: the pipe of the multiply-adds. A key of a kv head's four vectors is 8 packed multiply-adds of 2.3 cycles a warp in either
// product, 92 us each for 1536 rows (20/5 heads); the loops in place take 158 and 133 (the kernels by themselves under a profiler; pipe 66 and 73 % busy; a loop of
// this shape alone takes 105: what it copies into register pairs and loads shares the issue slots), the softmax 55, the preparation 15. A whole call, back to back in
// a graph, in us, as items (attention_split.cu) and here: 1536 rows 565 and 336, 600 rows 123 and 82, 300 rows 50 and 40, 256 rows behind 2744 keys 323 and 288, 4000 rows
// 3751 and 2289; 16/16 heads, 300 rows 119 and 39, 1500 rows 1122 and 279; 32/8, 1000 rows 418 and 251.
#pragma once
#include "attn_common.cuh"
#include "../../include/tenzo_kernels.h"

namespace tz {

constexpr int kRowVecs = 64;                       // query vectors of a tile
constexpr int kRowThreads = 256;
constexpr int kRowKeys = 128;                      // keys of a score tile
constexpr int kRowChunk = 32;                      // keys of a value chunk
constexpr int kRowQFloats = kHd * kRowVecs;        // a tile's rotated query vectors

struct RowsLaunch {
    tenzo_attention_args a;
    int G;                           // heads that share a kv head: 1, 2, 4 or 8
    int rows;                        // query rows of a tile: 64 / G
    int n;                           // query rows of this pass
    int row0;                        // the first of them
    int tp;                          // floats of a (row, head) in the scratch: max_len rounded up to 4
    float* scores;                   // [n][n_q][tp]: scores, then exponentials
    float* inv_sum;                  // [n][n_q]
    int* max;                        // [n][n_q]: the largest score, see ordered_bits
    int n_tiles;                     // tiles of the pass
    int key_tiles;                   // 128-key tiles of the cache up to max_len
    int span;                        // key tiles a score CTA goes through
    float* k;                        // [key tiles][n_kv][128 elements][128 keys], see rows_prepare_kernel
    float* v;                        // [n_kv][key tiles * 128][128]
    float* q;                        // [tiles][n_kv][128 elements][64 vectors]
};

// Keys of row r of the pass; 0 for a row that is not there, or whose position is refused.
__device__ __forceinline__ int row_keys(const RowsLaunch& L, int r) {
    if (r >= L.n) return 0;
    const int pos = __ldcg(L.a.pos + L.row0 + r);
    return pos < 0 || pos >= L.a.max_len ? 0 : pos + 1;
}
// The most keys a row of the tile has; every lane calls it.
__device__ __forceinline__ int tile_keys(const RowsLaunch& L, int tile, int rows) {
    const int lane = threadIdx.x & 31;
    int T = 0;
    for (int i = lane; i < rows; i += 32) T = max(T, row_keys(L, tile * rows + i));
    return __reduce_max_sync(0xffffffffu, T);
}
// The last tiles have the most keys, as a rule, and go first.
__device__ __forceinline__ int tile_of(const RowsLaunch& L, int rows, int index) { return (L.n + rows - 1) / rows - 1 - index; }

// Floats as integers of the same order, for a maximum by atomics (there are no NaN among them: a running fmaxf drops those).
__device__ __forceinline__ int ordered_bits(float x) { const int b = __float_as_int(x); return b ^ ((b >> 31) & 0x7fffffff); }
__device__ __forceinline__ float from_ordered_bits(int b) { return __int_as_float(b ^ ((b >> 31) & 0x7fffffff)); }

// acc[p][k] += a_p * b_k (FIRST: 0 + a_p * b_k): pairs of vectors p (two quads), four columns
template <bool FIRST = false>
__device__ __forceinline__ void outer4(f32x2 (&acc)[4][4], const float* qa, const float* qb, const float* kp) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(qa), y = *reinterpret_cast<const ulonglong2*>(qb);
    const float4 u = *reinterpret_cast<const float4*>(kp);
    const f32x2 q[4] = {x.x, x.y, y.x, y.y};
    const float k[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const f32x2 kk = pack2(k[j], k[j]);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            if constexpr (FIRST) asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(acc[p][j]) : "l"(q[p]), "l"(kk), "l"(0ull));
            else fma2(acc[p][j], q[p], kk);
        }
    }
}

// What the tiles are made of, in the order in which they lie in shared memory. Blocks of query vectors: rotated (:459-480), element e of vector
// v at 64 e + 4 (v / 4 ^ e mod 8) + v mod 4; lanes are eight elements x the four vectors of a quad. Behind them, in the first pass, blocks of 32 keys
// of a kv head: K as floats, element 8 i + j of key t in row 16 j + i of its key tile (the sixteen elements of a chain together), and V as floats.
constexpr int kRowPrepKeys = 32;
__global__ void __launch_bounds__(256) rows_prepare_kernel(const RowsLaunch L) {
    const tenzo_attention_args& a = L.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (a.use_pdl) pdl_wait();
    const int q_blocks = L.n_tiles * a.n_kv * 2;
    if ((int)blockIdx.x >= q_blocks) {
        const int kvh = (blockIdx.x - q_blocks) % a.n_kv, t0 = (blockIdx.x - q_blocks) / a.n_kv * kRowPrepKeys;
        const size_t base = ((size_t)a.layer * a.n_kv + kvh) * a.max_seq;
        const ByteFloats bytes;
        f32x2 lo, hi;
        float f[4];
        {   // a lane a key, a warp sixteen elements of it
            const uint4 w = __ldcg(reinterpret_cast<const uint4*>(a.cache_k + (base + min(t0 + lane, a.max_len - 1)) * kHd) + warp);
            const uint32_t w4[4] = {w.x, w.y, w.z, w.w};
            float* tile = L.k + ((size_t)(t0 / kRowKeys) * a.n_kv + kvh) * (kHd * kRowKeys) + t0 % kRowKeys + lane;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                bytes.pairs(w4[e], lo, hi);
                unpack2(lo, f[0], f[1]);
                unpack2(hi, f[2], f[3]);
#pragma unroll
                for (int c = 0; c < 4; ++c) tile[(16 * (4 * (e & 1) + c) + 2 * warp + (e >> 1)) * kRowKeys] = f[c];     // element 16 warp + 4 e + c
            }
        }
#pragma unroll
        for (int i = 0; i < kRowPrepKeys / 8; ++i) {
            const int t = t0 + 8 * i + warp;
            bytes.pairs(__ldcg(reinterpret_cast<const uint32_t*>(a.cache_v + (base + min(t, a.max_len - 1)) * kHd) + lane), lo, hi);
            *reinterpret_cast<ulonglong2*>(L.v + ((size_t)kvh * L.key_tiles * kRowKeys + t) * kHd + 4 * lane) = make_ulonglong2(lo, hi);
        }
        return;
    }
    const int unit = blockIdx.x >> 1, part = blockIdx.x & 1, tile = unit / a.n_kv, kvh = unit % a.n_kv;
    float* out = L.q + (size_t)unit * kRowQFloats;
    if (threadIdx.x < 32) {
        const int v = 32 * part + threadIdx.x, r = tile * L.rows + v / L.G;
        if (r < L.n) L.max[(size_t)r * a.n_q + kvh * L.G + v % L.G] = ordered_bits(-1e30f);       // :670
    }
    const int i = 8 * warp + (lane & 7);                         // of 64
#pragma unroll
    for (int qi = 0; qi < 8; ++qi) {
        const int quad = 8 * part + qi;
        const int v = 4 * quad + (lane >> 3), r = min(tile * L.rows + v / L.G, L.n - 1);
        const int pos = max(0, min(__ldcg(a.pos + L.row0 + r), a.max_len - 1));
        const float* qh = a.q + (size_t)(L.row0 + r) * a.q_stride + (size_t)(kvh * L.G + v % L.G) * kHd;
        const float* cs = a.rope_cos ? a.rope_cos + (size_t)pos * (kHd / 2) : nullptr;
        const float* sn = a.rope_sin ? a.rope_sin + (size_t)pos * (kHd / 2) : nullptr;
        float r0, r1;
        rope_pair(__ldcg(qh + i), __ldcg(qh + i + kHd / 2), cs, sn, i, r0, r1);
        float* o = out + i * kRowVecs + 4 * (quad ^ (i & 7)) + (lane >> 3);
        o[0] = r0;
        o[kHd / 2 * kRowVecs] = r1;                              // (element i + 64 has the same low bits)
    }
}

// Scores of 64 vectors x a span of key tiles. Shared memory: q, and two buffers of half a key tile (four chains of 128 keys, 32 KB), each
// brought in by a bulk copy while the other is computed on.
constexpr int kRowHalf = kHd / 2 * kRowKeys;
constexpr int kRowScoreBytes = (kRowQFloats + 2 * kRowHalf) * 4;
__global__ void __launch_bounds__(kRowThreads, 2) rows_scores_kernel(const RowsLaunch L) {
    const tenzo_attention_args& a = L.a;
    extern __shared__ __align__(128) float smem[];
    __shared__ uint64_t s_bar[3];
    __shared__ int s_keys[kRowVecs];                             // keys of the tile's rows
    float* s_q = smem;
    float* s_k = smem + kRowQFloats;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = blockIdx.y % a.n_kv, tile = tile_of(L, L.rows, blockIdx.y / a.n_kv), first = blockIdx.x * L.span;
    if (tid == 0) {
        for (int i = 0; i < 3; ++i) mbar_init(&s_bar[i], 1);
        mbar_init_fence();
    }
    if (a.use_pdl) pdl_wait();
    const int T = tile_keys(L, tile, L.rows);
    if (tid < L.rows) {
        s_keys[tid] = row_keys(L, tile * L.rows + tid);
        if (blockIdx.x == 0 && s_keys[tid] == 0 && tile * L.rows + tid < L.n) atomicExch(&g_split_timeouts, 2);
    }
    const int n_halves = 2 * (min((first + L.span) * kRowKeys, (T + kRowKeys - 1) / kRowKeys * kRowKeys) / kRowKeys - first);
    if (n_halves <= 0) return;
    auto request = [&](int h) {                                  // (by thread 0)
        mbar_expect_tx(&s_bar[h & 1], kRowHalf * 4);
        bulk_g2s(s_k + (h & 1) * kRowHalf, L.k + ((size_t)(first + (h >> 1)) * a.n_kv + kvh) * (2 * kRowHalf) + (h & 1) * kRowHalf, kRowHalf * 4, &s_bar[h & 1]);
    };
    if (tid == 0) {
        mbar_expect_tx(&s_bar[2], kRowQFloats * 4);
        bulk_g2s(s_q, L.q + ((size_t)tile * a.n_kv + kvh) * kRowQFloats, kRowQFloats * 4, &s_bar[2]);
        request(0);
        request(1);
    }
    // warps 2 x 4 over (32 vectors, 32 keys); lanes 4 x 8: vectors 4 vg .. and 16 + 4 vg .., keys 4 kg .. The second four go through the keys'
    // quarters the other way round, so that the warps whose quarter of the last key tile is behind every row's last key, and which leave it out,
    // are of different schedulers (calls apart, each waited for: 300 rows 49.8 -> 47.7 us, 600 rows 94.9 -> 91.8, 1000 of 32/8 heads 261.8 -> 259.0, 1537 355.2 -> 352.2, 256 behind 2744 keys 297.4
    // and 298.3; a branch around the products instead of a shorter loop: 1537 rows 357.3).
    const int kg = lane & 7, vq = 8 * (warp >> 2) + (lane >> 3), kw = 32 * (warp < 4 ? warp : 7 - warp), k0 = kw + 4 * kg;
    const int n_mine = (first + (n_halves >> 1) - 1) * kRowKeys + kw < T ? n_halves : n_halves - 2;
    const float* sk = a.scale_k + ((size_t)a.layer * a.n_kv + kvh) * a.max_seq;
    const float sm_scale = 1.0f / sqrtf((float)kHd);             // :660
    f32x2 sum[4][4];
    bool timed_out = false;
    __syncthreads();
    if (lane == 0 && !mbar_wait_bounded(&s_bar[2], 0u)) timed_out = true;
#pragma unroll 1
    for (int h = 0; h < n_mine; ++h) {
        if (lane == 0 && !mbar_wait_bounded(&s_bar[h & 1], (unsigned)(h >> 1) & 1u)) timed_out = true;
        __syncwarp();
        const float* sh = s_k + (h & 1) * kRowHalf + k0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            f32x2 acc[4][4];
            const int chain = 4 * (h & 1) + j;                   // (the low bits of the chain's elements)
            const float* qa = s_q + chain * kRowVecs + 4 * (vq ^ chain);
            const float* qb = s_q + chain * kRowVecs + 4 * ((vq + 4) ^ chain);
            outer4<true>(acc, qa, qb, sh + 16 * j * kRowKeys);
#pragma unroll
            for (int i = 1; i < 16; ++i) outer4(acc, qa + 8 * kRowVecs * i, qb + 8 * kRowVecs * i, sh + (16 * j + i) * kRowKeys);
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int c = 0; c < 4; ++c) sum[p][c] = j == 0 && !(h & 1) ? acc[p][c] : add2(sum[p][c], acc[p][c]);     // chains left to right (:691)
        }
        __syncthreads();
        if (tid == 0 && h + 2 < n_halves) request(h + 2);
        if (!(h & 1)) continue;
        const int t0 = (first + (h >> 1)) * kRowKeys;
        float ks[4], m[8];                                       // m: maxima of vectors 4 vq .. and 4 (vq + 4) .. over this lane's keys
#pragma unroll
        for (int c = 0; c < 4; ++c) ks[c] = __ldg(sk + min(t0 + k0 + c, T - 1)) * sm_scale;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float v[2][4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                unpack2(sum[p][c], v[0][c], v[1][c]);
                v[0][c] *= ks[c];                                // :691
                v[1][c] *= ks[c];
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int vec = 4 * (p < 2 ? vq : vq + 4) + 2 * (p & 1) + e, r = vec / L.G;
                const int left = s_keys[r] - t0 - k0;            // keys of the row from this lane's first on
                m[2 * p + e] = -1e30f;                           // :670
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (c < left) m[2 * p + e] = fmaxf(m[2 * p + e], v[e][c]);
                if (left > 0)
                    *reinterpret_cast<float4*>(L.scores + ((size_t)(tile * L.rows + r) * a.n_q + kvh * L.G + vec % L.G) * L.tp + t0 + k0) = make_float4(v[e][0], v[e][1], v[e][2], v[e][3]);
            }
        }
        // eight maxima over the eight lanes of a key group: each step halves the vectors a lane has, and lane kg ends with vector kg's
#pragma unroll
        for (int n = 4; n > 0; n >>= 1)
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const bool up = kg & n;
                const float mine = up ? m[i + n] : m[i], other = __shfl_xor_sync(0xffffffffu, up ? m[i] : m[i + n], n);
                m[i] = fmaxf(mine, other);
            }
        const int vec = 4 * (kg < 4 ? vq : vq + 4) + (kg & 3), r = vec / L.G;
        if (s_keys[r] > t0 + kw) atomicMax(L.max + (size_t)(tile * L.rows + r) * a.n_q + kvh * L.G + vec % L.G, ordered_bits(m[0]));
    }
    for (int h = n_mine; h < n_halves; ++h) __syncthreads();     // (thread 0 never comes here: its quarter is the first)
    if (timed_out) atomicExch(&g_split_timeouts, 1);
}

// Scores -> exponentials (in place) and 1 / sum. There are more (row, head) pairs than the machine has lanes for, so a lane of the summing warp
// adds up a pair's exponentials one after another as the reference does, while the other warps evaluate the next chunk: 32 pairs a
// CTA, chunks of 128 keys through two buffers. (A warp a pair with ordered_sum.cuh's segments: 139 us for 1536 rows, some thousand
// instructions a pair beside the exponentials; here 55.) Bound by the instructions of the exponential.
constexpr int kRowSoftWarps = 16, kRowSoftChunk = 128, kRowSoftStride = kRowSoftChunk + 4;
__global__ void __launch_bounds__(32 * (kRowSoftWarps + 1), 2) rows_softmax_kernel(const RowsLaunch L) {
    const tenzo_attention_args& a = L.a;
    __shared__ __align__(16) float s_e[2][32 * kRowSoftStride];
    constexpr int kOwn = 32 / kRowSoftWarps;                     // pairs an evaluating warp has
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long tab = kExp2fTab[lane];
    const uint32_t tab_lo = (uint32_t)tab, tab_hi = (uint32_t)(tab >> 32);
    if (a.use_pdl) pdl_wait();
    const int pairs = L.n * a.n_q, first = pairs - 32 * ((int)blockIdx.x + 1);         // from the last rows on; the last CTA may start below 0
    auto keys_of = [&](int pair) { return pair < 0 ? 0 : row_keys(L, pair / a.n_q); };
    const int T_lane = keys_of(first + lane), T_max = __reduce_max_sync(0xffffffffu, T_lane), n_chunks = (T_max + kRowSoftChunk - 1) / kRowSoftChunk;
    if (warp == kRowSoftWarps) {
        float sum = 0.0f;
        for (int c = 0; c < n_chunks; ++c) {
            __syncthreads();                                     // chunk c is in place (and c - 1 was read)
            const float4* p = reinterpret_cast<const float4*>(s_e[c & 1] + lane * kRowSoftStride);
            const int n = min(kRowSoftChunk, T_max - c * kRowSoftChunk);      // (zeros behind a pair's last key change no sum)
#pragma unroll 1
            for (int j = 0; j < (n + 3) >> 2; j += 8) {
                float4 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = p[j + u];
#pragma unroll
                for (int u = 0; u < 8; ++u) { sum += v[u].x; sum += v[u].y; sum += v[u].z; sum += v[u].w; }        // :824-829
            }
        }
        if (T_lane > 0) L.inv_sum[first + lane] = 1.0f / sum;
        return;
    }
    float* row[kOwn];
    int T[kOwn];
    float mx[kOwn];
#pragma unroll
    for (int h = 0; h < kOwn; ++h) {
        T[h] = __shfl_sync(0xffffffffu, T_lane, kOwn * warp + h);
        row[h] = L.scores + (size_t)max(0, first + kOwn * warp + h) * L.tp + lane;
        mx[h] = from_ordered_bits(__ldcg(L.max + max(0, first + kOwn * warp + h)));
    }
    float x[kOwn][4];
    auto load = [&](int t) {
#pragma unroll
        for (int h = 0; h < kOwn; ++h)
#pragma unroll
            for (int u = 0; u < 4; ++u) x[h][u] = t + 32 * u + lane < T[h] ? __ldcg(row[h] + t + 32 * u) : -INFINITY;
    };
    load(0);
    for (int c = 0; c < n_chunks; ++c) {
        const int t = c * kRowSoftChunk;
        float* d = s_e[c & 1] + kOwn * warp * kRowSoftStride + lane;
        float e[kOwn][4];
#pragma unroll
        for (int h = 0; h < kOwn; ++h)
#pragma unroll
            for (int u = 0; u < 4; ++u) e[h][u] = x[h][u] - mx[h];               // (behind the last key -inf for every maximum, which is -1e30 at least: zero)
        if (c + 1 < n_chunks) load(t + kRowSoftChunk);
#pragma unroll
        for (int h = 0; h < kOwn; ++h)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                e[h][u] = expf_reference_bits_lanes(e[h][u], tab_lo, tab_hi);                                          // :826
                d[h * kRowSoftStride + 32 * u] = e[h][u];
                if (t + 32 * u + lane < T[h]) row[h][t + 32 * u] = e[h][u];
            }
        __syncthreads();
    }
}

// Value sums of 32 vectors x 128 dims: chunks of 32 keys; V's floats by bulk copies into three buffers, the weights [32 keys][vectors] (quads of
// vectors exchanged by the key's quad) through registers into two. Three CTAs an SM: the buffers are 56 KB, and a fourth lacks 512 bytes for its barriers.
// With two buffers there are four, and they wait more for their copies: 1024 rows 171 -> 180 us in all, 4000 2289 -> 2335, 1536 336 -> 338.
constexpr int kRowValueVecs = 32, kRowValueThreads = 4 * kRowValueVecs, kRowValueStages = 3;
constexpr int kRowVFloats = kRowChunk * kHd, kRowWFloats = kRowChunk * kRowValueVecs;
constexpr int kRowValueBytes = (kRowValueStages * kRowVFloats + 2 * kRowWFloats) * 4;
__global__ void __launch_bounds__(kRowValueThreads, 3) rows_values_kernel(const RowsLaunch L) {
    const tenzo_attention_args& a = L.a;
    extern __shared__ __align__(128) float smem[];
    __shared__ uint64_t s_bar[kRowValueStages];
    float* s_weights = smem + kRowValueStages * kRowVFloats;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rows = kRowValueVecs / L.G;
    const int kvh = blockIdx.x % a.n_kv, tile = tile_of(L, rows, blockIdx.x / a.n_kv);
    if (tid == 0) {
        for (int i = 0; i < kRowValueStages; ++i) mbar_init(&s_bar[i], 1);
        mbar_init_fence();
    }
    if (a.use_pdl) pdl_wait();
    const int T = tile_keys(L, tile, rows), n_chunks = (T + kRowChunk - 1) / kRowChunk;
    if (T == 0) return;
    const float* sv = a.scale_v + ((size_t)a.layer * a.n_kv + kvh) * a.max_seq;
    auto request = [&](int c, int st) {                          // (by thread 0)
        mbar_expect_tx(&s_bar[st], kRowVFloats * 4);
        bulk_g2s(smem + st * kRowVFloats, L.v + ((size_t)kvh * L.key_tiles * kRowKeys + c * kRowChunk) * kHd, kRowVFloats * 4, &s_bar[st]);
    };
    if (tid == 0)
        for (int c = 0; c < min(n_chunks, kRowValueStages - 1); ++c) request(c, c);
    // weights: vectors kRowValueVecs / 2 * it + 4 warp + (lane >> 3), keys 4 (lane & 7) ..
    const int kq = lane & 7, v4 = lane >> 3;
    const float* erow[2];
    float inv[2];
    int Tr[2];
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const int vec = kRowValueVecs / 2 * it + 4 * warp + v4, r = tile * rows + vec / L.G;
        Tr[it] = row_keys(L, r);
        const size_t pair = (size_t)min(r, L.n - 1) * a.n_q + kvh * L.G + vec % L.G;
        erow[it] = L.scores + pair * L.tp + 4 * kq;
        inv[it] = Tr[it] > 0 ? __ldcg(L.inv_sum + pair) : 0.0f;
    }
    float4 e[2];
    float s[4];
    auto fetch = [&](int c) {
        const int t = c * kRowChunk;
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            e[it] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (t + 4 * kq < Tr[it]) e[it] = __ldcg(reinterpret_cast<const float4*>(erow[it] + t));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = __ldg(sv + min(t + 4 * kq + j, T - 1));
    };
    auto put = [&](int c) {
        const int t = c * kRowChunk + 4 * kq;
#pragma unroll
        for (int it = 0; it < 2; ++it) {                         // e / sum * scale (:830, :844); the row's scratch holds no exponentials behind its last key
            float* d = s_weights + (c & 1) * kRowWFloats + 4 * kq * kRowValueVecs + 4 * ((kRowValueVecs / 8 * it + warp) ^ kq) + v4;
            d[0] = t < Tr[it] ? e[it].x * inv[it] * s[0] : 0.0f;
            d[kRowValueVecs] = t + 1 < Tr[it] ? e[it].y * inv[it] * s[1] : 0.0f;
            d[2 * kRowValueVecs] = t + 2 < Tr[it] ? e[it].z * inv[it] * s[2] : 0.0f;
            d[3 * kRowValueVecs] = t + 3 < Tr[it] ? e[it].w * inv[it] * s[3] : 0.0f;
        }
    };
    const int vq = 8 * (warp >> 2) + (lane >> 3), d0 = 32 * (warp & 3) + 4 * (lane & 7);
    f32x2 acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int d = 0; d < 4; ++d) acc[p][d] = 0;
    bool timed_out = false;
    fetch(0);
    put(0);
    __syncthreads();
    int st = 0, round = 0;
#pragma unroll 1
    for (int c = 0; c < n_chunks; ++c) {
        if (c + 1 < n_chunks) fetch(c + 1);
        if (tid == 0 && c + kRowValueStages - 1 < n_chunks) request(c + kRowValueStages - 1, st == 0 ? kRowValueStages - 1 : st - 1);     // where chunk c - 1 was
        if (lane == 0 && !mbar_wait_bounded(&s_bar[st], (unsigned)round & 1u)) timed_out = true;
        __syncwarp();
        const float* s_w = s_weights + (c & 1) * kRowWFloats;
        const float* s_v = smem + st * kRowVFloats + d0;
#pragma unroll
        for (int k = 0; k < kRowChunk; ++k)
            outer4(acc, s_w + k * kRowValueVecs + 4 * (vq ^ (k >> 2)), s_w + k * kRowValueVecs + 4 * ((vq + 4) ^ (k >> 2)), s_v + k * kHd);         // :842-851
        if (c + 1 < n_chunks) put(c + 1);
        __syncthreads();
        if (++st == kRowValueStages) { st = 0; ++round; }
    }
    if (timed_out) atomicExch(&g_split_timeouts, 1);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        float o[2][4];
#pragma unroll
        for (int d = 0; d < 4; ++d) unpack2(acc[p][d], o[0][d], o[1][d]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int vec = 4 * (p < 2 ? vq : vq + 4) + 2 * (p & 1) + e, r = tile * rows + vec / L.G;
            if (row_keys(L, r) == 0) continue;
            float* out = a.out + ((size_t)(L.row0 + r) * a.n_q + kvh * L.G + vec % L.G) * kHd + d0;
#pragma unroll
            for (int d = 0; d < 4; ++d) out[d] = o[e][d];
        }
    }
}

// ---- host side ---------------------------------------------------------------------------------------------------------
static int rows_key_tiles(int max_len) { return (max_len + kRowKeys - 1) / kRowKeys; }
static size_t rows_key_bytes(int n_kv, int max_len) { return (size_t)2 * rows_key_tiles(max_len) * n_kv * kHd * kRowKeys * sizeof(float); }
static size_t rows_tile_bytes(int n_q, int n_kv, int max_len) {                    // of one tile's queries, scores, maxima and sums
    const size_t tp = ((size_t)max_len + 3) & ~(size_t)3;
    return ((size_t)kRowVecs / (n_q / n_kv) * n_q * (tp + 2) + (size_t)n_kv * kRowQFloats) * sizeof(float);
}
// Scratch of one pass at most, beside the keys'. It is as large as a prompt of 1700 rows needs whole (20/5 heads), of which about half is touched: 1536 rows
// take 338 us in one pass, 384 in two, 444 in three (whose last tiles leave SMs idle three times), 575 in six; the three kernels 565.
constexpr size_t kRowsPassBytes = (size_t)256 << 20;

// Rows of a pass in the caller's scratch; 0: another form. A CTA of the value sums has the whole chains of 32 vectors, so there has to be one for
// every SM in a pass, or a few SMs take as long for the last key (64 rows at 3000 keys, 40 CTAs: 107 us as items, 190 here). In us here and as items, 20/5
// heads, one pass: 225 rows 31 and 36, 240 behind 3000 keys 302 and 320; several, by the CTAs of each: 512 rows behind 6000 keys 160 CTAs 1178 and 1517,
// 1024 behind 8000 220 CTAs 2645 and 3939, behind 3000 320 CTAs 1131 and 1544, 8000 from the start 250 CTAs 9304 and 14444, 4500 410 CTAs 3029 and 4791.
// A whole prompt's few last tiles at each pass' end cost most where the scratch holds little of it: 1536 rows in 160 CTAs a pass 575 and 565, in 240 448;
// 32/8 heads, 1000 rows, 176 CTAs 409 and 418.
constexpr int kRowsValueCtas = 148;
static int rows_in_pass(int batch, int n_q, int n_kv, int max_len, size_t scratch) {
    const int per_tile = kRowVecs / (n_q / n_kv), tiles = (batch + per_tile - 1) / per_tile;
    const size_t keys = rows_key_bytes(n_kv, max_len), tile = rows_tile_bytes(n_q, n_kv, max_len);
    if (scratch < keys + tile + 64) return 0;
    size_t fit = (scratch - 64 - keys) / tile;
    if (fit > kRowsPassBytes / tile) fit = kRowsPassBytes > tile ? kRowsPassBytes / tile : 1;
    const int passes = fit < (size_t)tiles ? (int)((tiles + fit - 1) / fit) : 1, tiles_pass = (tiles + passes - 1) / passes;
    return tiles_pass * (kRowVecs / kRowValueVecs) * n_kv < kRowsValueCtas ? 0 : tiles_pass * per_tile;
}
static int attn_rows_per_pass(const tenzo_attention_args& a) {
    if (a.tiles != 0 || a.batch < 2 || a.block_table || a.seq_stride_kv != 0 || a.append || a.heads_per_cta != 0) return 0;
    return rows_in_pass(a.batch, a.n_q, a.n_kv, a.max_len, a.workspace_bytes);
}

// Scratch for `batch` rows and up to max_len keys: what the longest cache wants that this form takes with it; 0 if it takes none (fewer
// rows than it has CTAs for).
static size_t rows_workspace_bytes(int batch, int n_q, int n_kv, int max_len) {
    const int per_tile = kRowVecs / (n_q / n_kv), tiles = (batch + per_tile - 1) / per_tile;
    if ((long long)tiles * (kRowVecs / kRowValueVecs) * n_kv < kRowsValueCtas) return 0;
    for (int len = max_len; len > 0; len = (len - 1) / kRowKeys * kRowKeys) {
        const size_t tile = rows_tile_bytes(n_q, n_kv, len), all = tile * (size_t)tiles, cap = kRowsPassBytes > tile ? kRowsPassBytes : tile;
        const size_t bytes = rows_key_bytes(n_kv, len) + (all < cap ? all : cap) + 64;
        if (rows_in_pass(batch, n_q, n_kv, len, bytes)) return bytes;
    }
    return 0;
}

static int attn_rows_run(const tenzo_attention_args& a, int rows_per_pass, cudaStream_t st) {
    RowsLaunch L;
    L.a = a;
    if (L.a.q_stride <= 0) L.a.q_stride = a.n_q * kHd;
    L.G = a.n_q / a.n_kv;
    L.rows = kRowVecs / L.G;
    L.tp = (a.max_len + 3) & ~3;
    L.key_tiles = rows_key_tiles(a.max_len);
    cudaError_t e = allow_smem(rows_scores_kernel, kRowScoreBytes);
    if (e == cudaSuccess) e = allow_smem(rows_values_kernel, kRowValueBytes);
    for (L.row0 = 0; e == cudaSuccess && L.row0 < a.batch; L.row0 += rows_per_pass) {
        L.n = a.batch - L.row0 < rows_per_pass ? a.batch - L.row0 : rows_per_pass;
        L.n_tiles = (L.n + L.rows - 1) / L.rows;
        const unsigned units = (unsigned)(L.n_tiles * a.n_kv);
        // Two key tiles a score CTA where that leaves enough of them (1536 rows: 164 -> 159 us; 300 rows 16.8 -> 22.4).
        L.span = (long long)units * L.key_tiles >= 16 * 148 ? 2 : 1;
        L.k = static_cast<float*>(a.workspace);
        L.v = L.k + (size_t)L.key_tiles * a.n_kv * kHd * kRowKeys;
        L.q = L.v + (size_t)L.key_tiles * a.n_kv * kHd * kRowKeys;
        L.scores = L.q + (size_t)units * kRowQFloats;
        L.inv_sum = L.scores + (size_t)L.n * a.n_q * L.tp;
        L.max = reinterpret_cast<int*>(L.inv_sum + (size_t)L.n * a.n_q);
        const int value_rows = kRowValueVecs / L.G;
        const bool pdl = a.use_pdl != 0;
        const unsigned key_blocks = L.row0 == 0 ? (unsigned)((a.max_len + kRowPrepKeys - 1) / kRowPrepKeys * a.n_kv) : 0u;
        e = split_launch(rows_prepare_kernel, dim3(2 * units + key_blocks), 256, 0, st, pdl, L);
        if (e == cudaSuccess) e = split_launch(rows_scores_kernel, dim3((unsigned)((L.key_tiles + L.span - 1) / L.span), units), kRowThreads, kRowScoreBytes, st, pdl, L);
        if (e == cudaSuccess) e = split_launch(rows_softmax_kernel, dim3((unsigned)((L.n * a.n_q + 31) / 32)), 32 * (kRowSoftWarps + 1), 0, st, pdl, L);
        if (e == cudaSuccess) e = split_launch(rows_values_kernel, dim3((unsigned)((L.n + value_rows - 1) / value_rows * a.n_kv)), kRowValueThreads, kRowValueBytes, st, pdl, L);
    }
    return e == cudaSuccess ? 0 : (int)e;
}

}  // namespace tz
