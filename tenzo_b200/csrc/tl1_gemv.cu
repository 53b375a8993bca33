// TL1 ternary GEMV / skinny GEMM for sm_100a on the int8 tensor-core path (mma.sync m16n8k32,
// u8 x s8 -> s32), with the RMSNorm + absmax(31) activation quantiser fused into its prologue at
// batch 1 and the reference's three epilogues (store / residual add / squared-ReLU GLU).
//
// What it replaces in the reference CPU engine (src/runtime/TenzoEngine.cpp): rms_norm_raw
// (:148-166), build_lut (:22-62), compute_single_block (:64-127) and their call sites (:1542-1628).
//
// How the arithmetic is organised on the GPU
//   * The reference looks every 4-bit index up in a 16-entry table of clamp(w0*a0+w1*a1). With
//     |a| <= 31 the clamp can never fire, so the accumulator is the plain integer dot product
//     sum_k w[r][k]*a[k]; any exact integer evaluation gives the same int32.
//   * Weights stay in the reference's layout [N/64][K/2][32 B]. Lane (g = lane>>2, t = lane&3) of a
//     warp reads, for a "set" of 16 column pairs, the four 32-bit words at byte 4g of column pairs
//     16s+4i+t (i = 0..3) from the staged copy (bank-conflict free). A 4x4 byte transpose
//     (8 PRMT) turns them into T[j] = row pair 4g+j at those four column pairs.
//   * A byte of the layout is c0 | c1<<2 | c2<<4 | c3<<6 with codes c = w+1 in {0,1,2}: (c0,c1) =
//     row c at columns (2p,2p+1), (c2,c3) = row c+32. Masking without shifting gives bytes
//     c0, 4c1, 16c2, 64c3 — four ready-made u8 A fragments of mma.m16n8k32:
//        a0 = T&0x03.. (row 4g+j, even cols)    a2 = T&0x0C.. (row 4g+j, odd cols, x4)
//        a1 = T&0x30.. (row 32+4g+j, even, x16) a3 = T&0xC0.. (row 32+4g+j, odd, x64)
//     The B fragment holds the int8 activations of up to 8 sequences, even columns pre-multiplied
//     by 4 (|4a| <= 124), so the low rows accumulate 4*sum(c*a) and the high rows 64*sum(c*a).
//     One LOP3 per fragment register, four MMAs per 512 weight bytes per 8 sequences, and the
//     tensor core does the reduction over k that a dot-product kernel would do with shuffles.
//   * sum(w*a) = sum(c*a) - sum(a); sum(a) per sequence is accumulated while the activations are
//     staged.
//   * K can be split across the CTAs of a thread-block cluster (2, 4 or 8): partials meet in the
//     leader CTA's shared memory through distributed-shared-memory atomicAdd (integer, hence
//     order-free and exact) between hardware cluster barriers; the leader runs the epilogue.
//   * Each CTA brings its weight bytes into shared memory with 1-D bulk asynchronous copies (TMA)
//     completing on mbarriers, issued by one thread as the very first thing the kernel does: tens
//     of kilobytes per SM are in flight from a handful of instructions, which ordinary loads cannot
//     do (the load/store unit's request queue saturates at a fraction of the HBM latency-bandwidth
//     product). Every wait on an mbarrier is bounded; a give-up raises a flag the host can read.
//   * Nothing that does not depend on the previous kernel waits for it: the bulk copies, the norm
//     weights and an L2 prefetch of the NEXT kernel's weights are issued before griddepcontrol.wait.
//   * batch == 1: every CTA normalises and quantises the activation itself (bit-identical to the
//     reference, see common.cuh) and only packs the columns of its own K range.
//     batch > 1: act_quant_kernel (norm_quant.cu) has written packed int8 activations to a
//     workspace; CTAs stage their K range for 8 or 32 sequences and reuse every weight word for all.
#include <cooperative_groups.h>
#include <type_traits>

#include "common.cuh"
#include "attn_common.cuh"
#include "../../include/tenzo_kernels.h"

namespace tz {

namespace cg = cooperative_groups;

#ifndef TZ_FUSED_WARPS
#define TZ_FUSED_WARPS 16
#endif
constexpr int kFusedWarps = TZ_FUSED_WARPS;    // batch 1: one CTA per row block; two fit on an SM so consecutive kernels overlap
constexpr int kBatchedWarps = 16;

struct GemvLaunch {
    tenzo_tl1_gemv_args a;
    int ksplit;      // cluster size along K
    int units;       // CTAs along the row dimension (n_blocks, or n_blocks/2 in GLU mode)
    int nsets;       // ceil(K/2 / 16)
    const uint32_t* act_words;   // batch > 1: [batch][nsets][4][2] packed activations
    const float* act_inv;        // batch > 1: [batch] m/31
};

__device__ __forceinline__ float seg_scale_for(const tenzo_tl1_gemv_args& a, int block) {
    return block < a.seg_end[0] ? a.seg_scale[0] : (block < a.seg_end[1] ? a.seg_scale[1] : a.seg_scale[2]);
}

__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ld_stream_u32(const void* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Optional in-kernel timeline (compile with -DTZ_TRACE): first and last CTA record their SM's cycle counter at
// stage boundaries into g_trace (16 words per record; stamps 0-6 are the stages, 8-12 lie inside the prologue; word 15:
// block index, grid size in the upper half), read and reset by tenzo_trace_gemv(); compiled out of the library build.
#ifdef TZ_TRACE
__device__ unsigned long long g_trace[4096 * 16];
__device__ unsigned int g_trace_n;
#define TZ_TRACE_DECL unsigned long long tr[16] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}
#define TZ_STAMP(k) do { if (threadIdx.x == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1)) tr[k] = (unsigned long long)clock64(); } while (0)
#define TZ_TRACE_FLUSH do { if (threadIdx.x == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1)) { \
    const unsigned slot = atomicAdd(&g_trace_n, 1u); \
    if (slot < 4096) { for (int k = 0; k < 15; ++k) g_trace[slot * 16 + k] = tr[k]; \
                       g_trace[slot * 16 + 15] = blockIdx.x | ((unsigned long long)gridDim.x << 32); } } } while (0)
#else
#define TZ_TRACE_DECL do {} while (0)
#define TZ_STAMP(k) do {} while (0)
#define TZ_TRACE_FLUSH do {} while (0)
#endif

#ifndef TZ_GEMV_CHUNKS
#define TZ_GEMV_CHUNKS 1
#endif
// Bulk copies (and mbarriers) per row block. One: a bulk copy costs about the same whatever its size (measured: an SM
// completes roughly one copy per 0.45 us up to 16 KB), so splitting a 40 KB slice into eight pieces to start computing on
// the first cost more than it gained (decode went 820 -> 865 tok/s with one copy).
constexpr int kChunks = TZ_GEMV_CHUNKS;

__device__ int g_tl1_repeats = 0;  // one-sequence products whose presumed integers did not stand (tl1_one_kernel)
__device__ int g_tl1_timeouts = 0; // set when a bounded mbarrier wait gave up (the result of that launch is invalid)

template <int NT, bool FUSED>
struct GemvSmem {
    static constexpr int SL = FUSED ? 1 : 8 * NT;                       // sequences per CTA
    // 32-bit words: s_d[128*SL] | s_sa4[SL] | s_inv[SL] | scratch[32] | mbarriers[2*kChunks x 2 words]
    //               | s_b[sets*SL*8] | weights[nb_cta*sets*128] | (fused) x[K]
    static __host__ __device__ int head_words() { return (128 * SL + 2 * SL + 32 + 2 + 4 * kChunks + 3) & ~3; }
    static __host__ __device__ size_t bytes(int sets_per_cta, int K, int nb_cta) {
        return (size_t)(head_words() + sets_per_cta * SL * 8 + nb_cta * sets_per_cta * 128 + (FUSED ? K : 0)) * 4;
    }
};

template <int NT, bool FUSED>
__global__ void __launch_bounds__((FUSED ? kFusedWarps : kBatchedWarps) * 32, FUSED ? 2 : 1) tl1_mma_kernel(const GemvLaunch L) {
    constexpr int kGemvWarps = FUSED ? kFusedWarps : kBatchedWarps;
    constexpr int kGemvThreads = kGemvWarps * 32;
    using Lay = GemvSmem<NT, FUSED>;
    constexpr int SL = Lay::SL;
    const tenzo_tl1_gemv_args& a = L.a;
    extern __shared__ __align__(16) uint32_t smem[];
    int* s_d = reinterpret_cast<int*>(smem);                 // [rows_cta][SL] scaled accumulators
    int* s_sa4 = s_d + 128 * SL;                             // [SL] 4 * sum(a) over this CTA's columns
    float* s_inv = reinterpret_cast<float*>(s_sa4 + SL);     // [SL] m/31 per sequence
    float* s_f = s_inv + SL;                                 // [32] reduction scratch
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + ((128 * SL + 2 * SL + 32 + 1) & ~1));   // [2][kChunks]
    uint32_t* s_b = smem + Lay::head_words();                // [sets][SL][4 t][2] packed activations

    TZ_TRACE_DECL;
    TZ_STAMP(0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const int unit = blockIdx.x / L.ksplit, split = blockIdx.x % L.ksplit, seq0 = blockIdx.y * SL;
    const bool glu = a.epilogue == TENZO_EPI_RELU2_GLU;
    const int nb_cta = glu ? 2 : 1;                 // row blocks handled by this CTA
    const int wb = kGemvWarps / nb_cta;             // warps per row block
    const int my_blk = glu ? (warp & 1) : 0;        // which of the CTA's row blocks this warp feeds
    const int wi = glu ? (warp >> 1) : warp;        // index among the warps of that row block
    const int kh = a.K >> 1;                        // column pairs
    cg::cluster_group cluster = cg::this_cluster();

    // K range of this CTA in sets of 16 column pairs (512 weight bytes per row block per set)
    const int s_begin = (int)(((long long)L.nsets * split) / L.ksplit);
    const int s_end = (int)(((long long)L.nsets * (split + 1)) / L.ksplit);
    const int n_cta_sets = s_end - s_begin;
    const int my_sets = (n_cta_sets - wi + wb - 1) / wb;   // this warp takes sets wi, wi+wb, ... of the range
    uint32_t* s_wt = s_b + n_cta_sets * SL * 8;              // [nb_cta][n_cta_sets][128 words] weights as in memory
    float* s_x = reinterpret_cast<float*>(s_wt + nb_cta * n_cta_sets * 128);   // fused only: x[K]
    const int sets_per_chunk = (n_cta_sets + kChunks - 1) / kChunks;

    // ---- weights: bulk-copy this CTA's slice of each row block into shared memory ----------------
    // They do not depend on the previous kernel, so they are requested before anything else.
    const unsigned range_bytes = (unsigned)(min(s_end * 512, kh * 32) - s_begin * 512);
    if (tid == 0) {
        for (int i = 0; i < nb_cta * kChunks; ++i) mbar_init(&s_bar[i], 1);
        mbar_init_fence();
        for (int bk = 0; bk < nb_cta; ++bk) {
            const int block = bk ? unit + L.units : unit;
            const uint8_t* src = a.w + (size_t)block * kh * 32 + (size_t)s_begin * 512;
            for (int c = 0; c < kChunks; ++c) {
                const unsigned off = (unsigned)c * sets_per_chunk * 512;
                const unsigned bytes = off < range_bytes ? min((unsigned)sets_per_chunk * 512, range_bytes - off) : 0u;
                mbar_expect_tx(&s_bar[bk * kChunks + c], bytes);   // zero bytes completes the phase at once
                if (bytes)
                    bulk_g2s(reinterpret_cast<uint8_t*>(s_wt + bk * n_cta_sets * 128) + off, src + off, bytes, &s_bar[bk * kChunks + c]);
            }
        }
    }
    l2_prefetch_slice(a.prefetch, a.prefetch_bytes);

    const int rows_cta = nb_cta * 64;
    for (int i = tid; i < rows_cta * SL; i += kGemvThreads) s_d[i] = 0;
    for (int i = tid; i < SL; i += kGemvThreads) s_sa4[i] = 0;
    constexpr int kWRegs = 16;                      // norm weights held in registers while waiting (K <= 16*threads)
    float wreg[kWRegs];
    const bool has_w = FUSED && a.do_norm && a.norm_w;
    const bool w_in_regs = has_w && a.K <= kWRegs * kGemvThreads;
    if (w_in_regs) {
#pragma unroll
        for (int r = 0; r < kWRegs; ++r) {
            const int i = tid + r * kGemvThreads;
            wreg[r] = i < a.K ? __ldg(a.norm_w + i) : 0.0f;   // model constant: no need to wait for the previous kernel
        }
    }
    if (L.ksplit > 1 || !FUSED) __syncthreads();    // batched: the staging loop below adds into s_sa4 from every warp, so the
                                                    // zeroes above must be in place first (one sequence: barriers follow anyway)
    if (L.ksplit > 1) cluster.barrier_arrive();     // "my s_d is zeroed": peers may add into it after their wait

    TZ_STAMP(1);
    if (a.use_pdl) pdl_wait();
    TZ_STAMP(2);
    if (FUSED && a.use_pdl) pdl_launch_dependents();   // one sequence: the next kernel's CTAs may come in and fetch their weights from here on

    float resid_v = 0.0f;                           // batch 1: fetched now so the epilogue does not wait on it
    if (FUSED && a.epilogue == TENZO_EPI_RESIDUAL && split == 0 && tid < 64)
        resid_v = __ldcg(a.resid + (size_t)seq0 * a.out_stride + unit * 64 + tid);

    if (FUSED) {
        // ---- RMSNorm + absmax(31) quantiser, recomputed identically by every CTA: x staged in shared memory, two passes over it ----------------
        const float* x = a.x + (size_t)seq0 * a.x_stride;
        const bool vec = ((a.K & 3) == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
        if (vec) {
            for (int i = tid; i < (a.K >> 2); i += kGemvThreads)
                reinterpret_cast<float4*>(s_x)[i] = __ldcg(reinterpret_cast<const float4*>(x) + i);
        } else {
            for (int i = tid; i < a.K; i += kGemvThreads) s_x[i] = __ldcg(x + i);
        }
        __syncthreads();
        float m = 0.0f;
        if (a.do_norm) {
            const float ss = sumsq_reference_order(s_x, a.K, s_f);
            const float inv_rms = rms_inv(ss, a.K, a.eps);
            if (w_in_regs) {
#pragma unroll
                for (int r = 0; r < kWRegs; ++r) {
                    const int i = tid + r * kGemvThreads;
                    if (i < a.K) {
                        const float y = s_x[i] * inv_rms * wreg[r];   // x * inv_rms * w, left to right (:158)
                        s_x[i] = y;
                        m = fmaxf(m, fabsf(y));
                    }
                }
            } else {
                for (int i = tid; i < a.K; i += kGemvThreads) {
                    const float y = rms_apply(s_x[i], inv_rms, has_w ? a.norm_w : nullptr, i);
                    s_x[i] = y;
                    m = fmaxf(m, fabsf(y));
                }
            }
        } else {
            for (int i = tid; i < a.K; i += kGemvThreads) m = fmaxf(m, fabsf(s_x[i]));
        }
        m = fmaxf(block_max_nonneg(m, s_f), 1e-6f); // TenzoEngine.cpp:28-32 (m: running maximum of |y| from 0)
        const float to_q = 31.0f / m;               // :34
        if (tid == 0) s_inv[0] = m / 31.0f;         // :35
        // pack only this CTA's columns: one 32-bit fragment word per (set, t, even/odd)
        int sa = 0;
        for (int wd = tid; wd < n_cta_sets * 8; wd += kGemvThreads) {
            const int s = s_begin + (wd >> 3), tt = (wd >> 1) & 3, odd = wd & 1;
            uint32_t word = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int col = 2 * (16 * s + 4 * i + tt) + odd;
                const int q = col < a.K ? (int)roundf(s_x[col] * to_q) : 0;   // :41-42, half away from zero
                sa += q;
                word |= (uint32_t)(uint8_t)(int8_t)(odd ? q : 4 * q) << (8 * i);
            }
            s_b[wd] = word;
        }
        sa = warp_sum_i(sa);
        if (lane == 0 && sa) atomicAdd(&s_sa4[0], 4 * sa);
        if ((a.a_out || a.inv_out) && blockIdx.x == 0) {                      // parity-check outputs
            for (int i = tid; i < a.K; i += kGemvThreads)
                if (a.a_out) a.a_out[(size_t)seq0 * a.K + i] = (int8_t)(int)roundf(s_x[i] * to_q);
            if (a.inv_out && tid == 0) a.inv_out[seq0] = m / 31.0f;
        }
    } else {
        // ---- stage this CTA's K range of the pre-quantised activations of SL sequences -----------
        for (int idx = tid; idx < n_cta_sets * SL * 2; idx += kGemvThreads) {
            const int half = idx & 1, n = (idx >> 1) % SL, sl = (idx >> 1) / SL;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (seq0 + n < a.batch)
                v = __ldcg(reinterpret_cast<const uint4*>(L.act_words + ((size_t)(seq0 + n) * L.nsets + s_begin + sl) * 8) + half);
            reinterpret_cast<uint4*>(s_b + ((size_t)sl * SL + n) * 8)[half] = v;
            int sa4 = dp4a_ss(0x01010101u, v.x, 0);     // even-column words already carry the factor 4
            sa4 = dp4a_ss(0x04040404u, v.y, sa4);
            sa4 = dp4a_ss(0x01010101u, v.z, sa4);
            sa4 = dp4a_ss(0x04040404u, v.w, sa4);
            if (sa4) atomicAdd(&s_sa4[n], sa4);
        }
        for (int n = tid; n < SL; n += kGemvThreads) s_inv[n] = seq0 + n < a.batch ? __ldcg(L.act_inv + seq0 + n) : 0.0f;
    }
    __syncthreads();
    TZ_STAMP(3);
    if (!FUSED && a.use_pdl) pdl_launch_dependents();

    // ---- main loop: weights from shared memory, four MMAs per set per 8 sequences -----------------
    int acc[NT][4][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][j][e] = 0;
    // Per-lane cursors advance by one stride per set: no index arithmetic in the loop. Words past the
    // copied range (ragged K) are stale shared memory, but the activation bytes they meet are zero.
    const uint32_t* wt = s_wt + my_blk * n_cta_sets * 128 + (16 * wi + t4) * 8 + g;      // column pair 16*sl + 4*i + t4, byte 4g
    const uint32_t* bp = s_b + ((size_t)wi * SL + g) * 8 + t4 * 2;                        // B fragment words of sequence g
    const int wt_step = 16 * wb * 8, bp_step = wb * SL * 8;
    int next_wait = 0, chunk = 0;                                                         // first set of the next chunk to wait for
    bool timed_out = false;
    for (int u = 0, sl = wi; u < my_sets; ++u, sl += wb, wt += wt_step, bp += bp_step) {
        while (sl >= next_wait) {
            // one lane polls (operations on one mbarrier serialise); the warp barrier passes the
            // acquired visibility on to the other lanes
            if (lane == 0 && !mbar_wait_bounded(&s_bar[my_blk * kChunks + chunk], 0)) timed_out = true;
            __syncwarp();
            ++chunk;
            next_wait += sets_per_chunk;
        }
        const uint32_t W0 = wt[0], W1 = wt[32], W2 = wt[64], W3 = wt[96];
        // 4x4 byte transpose: T[j] = (W0.j, W1.j, W2.j, W3.j) = row pair 4g+j at this lane's four column pairs
        const uint32_t p0 = prmt(W0, W1, 0x5140u), p1 = prmt(W2, W3, 0x5140u);
        const uint32_t p2 = prmt(W0, W1, 0x7362u), p3 = prmt(W2, W3, 0x7362u);
        const uint32_t T[4] = {prmt(p0, p1, 0x5410u), prmt(p0, p1, 0x7632u), prmt(p2, p3, 0x5410u), prmt(p2, p3, 0x7632u)};
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            uint2 b = make_uint2(0, 0);
            if (nt * 8 + g < SL) b = *reinterpret_cast<const uint2*>(bp + nt * 64);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mma_u8s8(acc[nt][j], T[j] & 0x03030303u, T[j] & 0x30303030u, T[j] & 0x0C0C0C0Cu, T[j] & 0xC0C0C0C0u, b.x, b.y);
        }
    }
    if (timed_out) atomicExch(&g_tl1_timeouts, 1);
    TZ_STAMP(4);

    // ---- warps of a row block meet in shared memory ---------------------------------------------
    if (my_sets > 0) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int n = nt * 8 + 2 * t4 + e;          // sequence (column of D) held in c[e] and c[2+e]
                if (n < SL) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        atomicAdd(&s_d[(my_blk * 64 + 4 * g + j) * SL + n], acc[nt][j][e]);            // x4
                        atomicAdd(&s_d[(my_blk * 64 + 32 + 4 * g + j) * SL + n], acc[nt][j][2 + e]);   // x64
                    }
                }
            }
    }
    __syncthreads();

    // ---- split-K meeting point: the cluster leader's shared memory -----------------------------
    if (L.ksplit > 1) {
        cluster.barrier_wait();                     // every peer has zeroed its s_d (arrive above)
        if (split != 0) {
            int* remote = cluster.map_shared_rank(s_d, 0);
            for (int i = tid; i < rows_cta * SL; i += kGemvThreads) {
                const int v = s_d[i];
                if (v) atomicAdd(remote + i, v);
            }
            for (int n = tid; n < SL; n += kGemvThreads) atomicAdd(remote + 128 * SL + n, s_sa4[n]);
        }
        cluster.sync();                             // all remote adds have landed in the leader
        if (split != 0) return;
    }

    TZ_STAMP(5);
    // ---- epilogue -----------------------------------------------------------------------------
    for (int idx = tid; idx < 64 * SL; idx += kGemvThreads) {
        const int r = idx / SL, n = idx % SL, seq = seq0 + n;
        if (seq >= a.batch) continue;
        const int sum_a = s_sa4[n] >> 2;
        const float inv_act = s_inv[n];
        float v[2];
#pragma unroll
        for (int bk = 0; bk < 2; ++bk) {
            if (bk >= nb_cta) break;
            const int blk = bk ? unit + L.units : unit;
            const int raw = s_d[(bk * 64 + r) * SL + n];
            const int accv = (r < 32 ? (raw >> 2) : (raw >> 6)) - sum_a;
            if (a.acc_out) a.acc_out[(size_t)seq * a.n_blocks * 64 + blk * 64 + r] = accv;
            v[bk] = (float)accv * (inv_act * seg_scale_for(a, blk));   // :1554, :118
        }
        const size_t o = (size_t)seq * a.out_stride + unit * 64 + r;
        if (a.epilogue == TENZO_EPI_STORE) {
            a.out[o] = v[0];
        } else if (a.epilogue == TENZO_EPI_RESIDUAL) {
            a.out[o] = (FUSED ? resid_v : __ldcg(a.resid + o)) + v[0];   // :1590
        } else {
            const float rl = fmaxf(0.0f, v[0]);
            a.out[o] = (rl * rl) * v[1];                                 // :1618-1619
        }
    }
    TZ_STAMP(6);
    TZ_TRACE_FLUSH;
}

// ---- one sequence, K a multiple of 32 up to 8192, 16-byte aligned vectors -----------------------------------------------------
// The product of tl1_mma_kernel<1, true> with everything that can be taken off the path between the input vector and it.
//   * The sum of squares. In the reference's order that is eight chains of K/8 dependent additions (2 600 cycles at K = 2560,
//     6 300 at 6912 in place), and the quantiser needs 1 / rms from it. But (x / rms * w) * (31 / max|x / rms * w|) depends
//     on 1 / rms in its last bits only: so x * w is quantised as it is, the product runs on that, and a warp of its own adds
//     up the chains meanwhile. Then every thread checks its elements with the exact 1 / rms: if each quantised value lies
//     less than half a unit from the exact quotient and no |y| exceeds that of the presumed maximum, the integers are the
//     reference's, and only the scale is taken from the exact values; else (some quotient within 1e-6 of a half) the
//     activations are quantised again, as the reference does it, and the product repeated. Same results either way, bit for
//     bit. Of 20 000 products of normal vectors 35 were repeated at K = 2560, 68 at 4096 and 94 at 6912, of squared-ReLU ones 4
//     to 12 (counted: tenzo_cuda_tl1_gemv_take_repeats); nearly all whose largest |y| is under the floor of 1e-6, but not zero. What the check covers need not be exact before it: 31 / max is an approximate
//     quotient, the rounding is an addition of 1.5 * 2^23. Nor need it be a number: a NaN or an overflow in x * w fails the
//     check (the exact value is a NaN too, or the presumed integer is none of +-31 where that of the maximum has to be).
//   * Cluster meetings. A CTA takes half a 64-row block (16 of the 32 bytes of each column pair: rows c and c + 32) over the
//     whole of K instead of a block over half of K; whole blocks where halves would be more than one CTA an SM.
//   * Byte shuffling. A weight word goes into the tensor core as it lies in memory, four rows of one column pair, masked but not
//     transposed: its bytes are the k index there, and column n of B has the activation in byte n and zeroes elsewhere, so
//     that column n of D is row n of the word.
// A worker owns 16-byte pieces of x (piece f = t, t + 512, ...: elements 4f .. 4f + 3) from the load to the packed bytes.
// The chain warp is warp 0: the scheduler prefers it.
// What bounds it: latency. Of the 2.9 us of a K = 2560 product 0.5 us are the load of x, 0.2 the maximum, 0.6 the quantiser, 0.7
// the product, 0.8 the rest of the chain and the check. In a decode step (launches overlapped) 3840 x 2560 4.8 -> 4.3 us,
// 2560 x 2560 4.9 -> 3.9, gate|up 13824 x 2560 6.1 -> 5.2, 2560 x 6912 8.8 -> 7.2, against the kernel above. Then three
// waits less, 24.51 -> 24.02 ms for 32 tokens of a 2B-shaped model: the presumed maximum's element is handed over in shared memory (it
// was read again from L2, and 300 to 1000 cycles of every product waited for that: 24.31), the chain's loads run a batch ahead of its
// additions (24.10), and one block's MMAs go to two sums in turn. In cycles after the wait, 2560 x 2560: 960 for x and its squares, 700
// quantiser, 240 barrier and weights, 1600 product, 700 check, 600 scale and store.
constexpr int kOneWorkers = kFusedWarps * 32, kOneThreads = kOneWorkers + 32;
constexpr int kOneMaxK = 8192;

struct OneSmem {
    // 32-bit words: s_d[128] | s_f[64] | s_b[sets * 8] | squares by chains [8][stride] | weights [nb_cta][K/2 column pairs][4 HB words]
    static constexpr int head_words = 128 + 64;
    static __host__ __device__ constexpr int stride(int K) { return (K >> 3) | 4; }        // an odd number of 16-byte pieces: eight rows' pieces in different banks
    static constexpr size_t bytes(int K, int nb_cta, int hb) { return (size_t)(head_words + (K >> 2) + 8 * stride(K) + nb_cta * (K >> 1) * 4 * hb) * 4; }
    static constexpr size_t most() { return bytes(kOneMaxK, 2, 1); }             // = bytes(kOneMaxK, 1, 2); two whole blocks a CTA only where they fit it
};

// Barrier of the 512 workers that also ors a flag.
__device__ __forceinline__ bool workers_any(bool v) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"(v ? 1u : 0u), "n"(kOneWorkers) : "memory");
    return r != 0;
}

template <int P, int HB>      // pieces a worker owns at most; halves of a row block a CTA takes
__global__ void __launch_bounds__(kOneThreads, 2) tl1_one_kernel(const GemvLaunch L) {
    const tenzo_tl1_gemv_args& a = L.a;
    extern __shared__ __align__(16) uint32_t smem[];
    constexpr int kRows = 32 * HB;                                   // rows of a block in this CTA
    int* s_d = reinterpret_cast<int*>(smem);                         // [nb_cta][kRows] accumulators: low-nibble rows x4, high-nibble rows x64
    float* s_f = reinterpret_cast<float*>(smem + 128);               // [0,16) maxima, 32: 1/rms
    int* s_sa = reinterpret_cast<int*>(s_f + 36);                    // sum of the activations
    unsigned long long* s_top = reinterpret_cast<unsigned long long*>(s_f + 38);   // x and its weight where x * w is largest (one 64-bit word: stores of equal ones do not mix)
    uint32_t* s_b = smem + OneSmem::head_words;                      // [sets][8]: word c of set b holds activations 32 b + c + 8 j as bytes j, even c times 4
    float* s_sq = reinterpret_cast<float*>(s_b + (a.K >> 2));        // [8][stride]
    const int stride = OneSmem::stride(a.K), n_pieces = a.K >> 2, kh = a.K >> 1, n_sets = a.K >> 5;
    unsigned char* s_wt = reinterpret_cast<unsigned char*>(s_sq + 8 * stride);     // [nb_cta][kh][16 HB]
    const bool glu = a.epilogue == TENZO_EPI_RELU2_GLU;
    const int nb_cta = glu ? 2 : 1;
    const int unit = HB == 2 ? blockIdx.x : blockIdx.x >> 1, half = HB == 2 ? 0 : blockIdx.x & 1;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x < 32) {
        // ---- the chain warp ----------------------------------------------------------------------------------------------------
        if (a.use_pdl) pdl_wait();
        if (!a.do_norm) return;
        named_barrier_sync(3, kOneThreads);                          // the squares are in place
        // The fixed cost of every faster form is more than it saves here: 320 additions are 1666 cycles (864: 3900); sixteen segments of
        // the chains by eight warps, walked from presumed sums and joined, 2270 (2840), five parts by three warps 1930 (3250).
        const float sum = lane < 8 ? sequential_sum(s_sq + lane * stride, a.K >> 3) : 0.0f;
        float ss = __shfl_sync(0xffffffffu, sum, 0);
#pragma unroll
        for (int j = 1; j < 8; ++j) ss = __fadd_rn(ss, __shfl_sync(0xffffffffu, sum, j));      // the eight lanes left to right (common.cuh)
        if (lane == 0) s_f[32] = rms_inv(ss, a.K, a.eps);
        named_barrier_arrive(4, kOneThreads);
        return;
    }

    // ---- before the producer has finished: this CTA's weights, the next kernel's, the norm weights --------------------------------
    const int tid = threadIdx.x - 32, warp = tid >> 5;
    for (int bk = 0; bk < nb_cta; ++bk) {
        const uint8_t* src = a.w + (size_t)(bk ? unit + L.units : unit) * kh * 32 + 16 * half;
        for (int i = tid; i < kh * HB; i += kOneWorkers) {           // 16-byte pieces: HB a column pair
            const uint8_t* p = HB == 2 ? src + (size_t)i * 16 : src + (size_t)i * 32;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(s_wt + ((size_t)bk * kh * HB + i) * 16)), "l"(p) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    l2_prefetch_workers(a.prefetch, a.prefetch_bytes, tid, kOneWorkers);
    if (tid < 128) s_d[tid] = 0;
    if (tid == 0) {
        *s_sa = 0;
        *s_top = 0x7fffffffull;                                      // no number, if no element is one
    }
    const bool has_w = a.do_norm && a.norm_w;
    constexpr bool kKeep = P <= 2;                                   // w and the result stay in registers for the check, else they are read again
    // Pieces beyond the vector read its first one: a load under a condition would be waited for before the next.
    auto load_w = [&](int j, float (&w)[4]) {
        const int f = tid + j * kOneWorkers;
        const float4 v = has_w ? __ldg(reinterpret_cast<const float4*>(a.norm_w) + (f < n_pieces ? f : 0)) : make_float4(1.f, 1.f, 1.f, 1.f);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    };
    auto load_x = [&](int j, float (&x)[4]) {
        const int f = tid + j * kOneWorkers;
        const float4 v = __ldcg(reinterpret_cast<const float4*>(a.x) + (f < n_pieces ? f : 0));
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    };
    float xr[P][4], wr[P][4];
#pragma unroll
    for (int j = 0; j < P; ++j)
        load_w(j, wr[j]);                                            // model constants
    if (a.use_pdl) pdl_wait();
    const int my_row = tid & (kRows - 1), out_row = unit * 64 + (my_row < kRows / 2 ? 16 * half + my_row : 32 + 16 * half + my_row - kRows / 2);
    float resid_v = 0.0f;
    if (a.epilogue == TENZO_EPI_RESIDUAL && tid < kRows) resid_v = __ldcg(a.resid + out_row);

    auto normed = [&](float x, float inv_rms, float w) {             // x * inv_rms * w, left to right (:158)
        const float y = x * inv_rms;
        return has_w ? y * w : y;
    };
    auto workers_max = [&](float m) {                                // maximum over the workers of values >= 0
        m = warp_max_nonneg(m);
        if (lane == 0) s_f[warp] = m;
        named_barrier_sync(1, kOneWorkers);
        return warp_max_nonneg(s_f[lane & 15]);
    };
    constexpr float kRound = 12582912.0f;                            // 1.5 * 2^23: v + kRound holds round(v) in its low bits
    float r[kKeep ? P : 1][4];                                       // kRound + the quantised values
    // Element 4f + k goes to byte (f >> 1) & 3 of word (set f >> 3, c = 4 (f & 1) + k); even columns carry the factor 4.
    uint8_t* s_b8 = reinterpret_cast<uint8_t*>(s_b) + ((tid >> 3) * 8 + 4 * (tid & 1)) * 4 + ((tid >> 1) & 3);
    auto put = [&](int j, const float (&v)[4]) {                     // takes kRound + the values, returns their sum
        const uint32_t q0 = __float_as_uint(v[0]), q1 = __float_as_uint(v[1]), q2 = __float_as_uint(v[2]), q3 = __float_as_uint(v[3]);
        uint8_t* d = s_b8 + j * (4 * kOneWorkers);
        d[0] = (uint8_t)(q0 << 2);
        d[4] = (uint8_t)q1;
        d[8] = (uint8_t)(q2 << 2);
        d[12] = (uint8_t)q3;
        if constexpr (kKeep)
#pragma unroll
            for (int k = 0; k < 4; ++k) r[j][k] = v[k];
        return (int)(q0 + q1 + q2 + q3 - 4u * __float_as_uint(kRound));
    };
    auto quantised = [&](int j, float (&q)[4]) {
        if constexpr (kKeep) {
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = r[j][k] - kRound;
        } else {
            const uint4 u = *reinterpret_cast<const uint4*>(s_b + (tid >> 3) * 8 + 4 * (tid & 1) + j * kOneWorkers);
            const uint32_t sel = 0x7540u + ((tid >> 1) & 3);         // the thread's byte of a word, as a float: 2^23 + 128 + the signed byte
            auto byte_of = [&](uint32_t v) { return __uint_as_float(prmt(v ^ 0x80808080u, 0x4B000000u, sel)); };
            q[0] = __fmaf_rn(byte_of(u.x), 0.25f, -2097184.0f);
            q[1] = byte_of(u.y) - 8388736.0f;
            q[2] = __fmaf_rn(byte_of(u.z), 0.25f, -2097184.0f);
            q[3] = byte_of(u.w) - 8388736.0f;
        }
    };
    auto add_sa = [&](int sa) {
        sa = warp_sum_i(sa);
        if (lane == 0 && sa) atomicAdd(s_sa, sa);
    };
    // As the reference does it (:28-42): this thread's values, their maximum over the vector m. What is no number (a NaN element,
    // or an infinite one, whose quotient is one) becomes the integer 0, as in the conversion of the other kernels; the rest lies
    // within +-31.
    auto exact_quantise = [&](float m, auto value) {
        const float to_q = 31.0f / fmaxf(m, 1e-6f);
        int sa = 0;
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (tid + j * kOneWorkers < n_pieces) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float y = value(j, k) * to_q;
                    v[k] = y == y ? roundf(y) + kRound : kRound;     // half away from zero
                }
                sa += put(j, v);
            }
        add_sa(sa);
    };

#pragma unroll
    for (int j = 0; j < P; ++j)
        load_x(j, xr[j]);
    float m = 0.0f;
    if (a.do_norm) {
        auto z = [&](int j, int k) { return xr[j][k] * wr[j][k]; };
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (tid + j * kOneWorkers < n_pieces) {
                const int f = tid + j * kOneWorkers;
                float* d = s_sq + (4 * (f & 1)) * stride + (f >> 1);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    d[k * stride] = __fmul_rn(xr[j][k], xr[j][k]);
                    m = fmaxf(m, fabsf(z(j, k)));
                }
            }
        const float m_own = m;
        m = warp_max_nonneg(m);
        if (lane == 0) s_f[warp] = m;
        if (a.use_pdl) pdl_launch_dependents();                      // x is here: the next kernel's CTAs may come in and ask for their weights
        named_barrier_sync(3, kOneThreads);
        m = warp_max_nonneg(s_f[lane & 15]);
        // The products x * w again rather than kept: they would take the registers that hold w.
        auto forget = [&] {
#pragma unroll
            for (int j = 0; j < P; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) asm volatile("" : "+f"(wr[j][k]));
        };
        forget();
        if (m_own == m) {                                            // whose element it is (any of equal ones)
#pragma unroll
            for (int j = 0; j < P; ++j)
                if (tid + j * kOneWorkers < n_pieces)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (fabsf(z(j, k)) == m) *s_top = (unsigned long long)__float_as_uint(wr[j][k]) << 32 | __float_as_uint(xr[j][k]);
        }
        forget();
        const float to_q = __fdividef(31.0f, fmaxf(m, 1e-30f));
        int sa = 0;
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (tid + j * kOneWorkers < n_pieces) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = __fmaf_rn(z(j, k), to_q, kRound);
                sa += put(j, v);
            }
        add_sa(sa);
    } else {
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (tid + j * kOneWorkers < n_pieces)
#pragma unroll
                for (int k = 0; k < 4; ++k) m = fmaxf(m, fabsf(xr[j][k]));
        if (a.use_pdl) pdl_launch_dependents();
        m = workers_max(m);
        exact_quantise(m, [&](int j, int k) { return xr[j][k]; });
    }

    const int g = lane >> 2, t4 = lane & 3;
    // Weight word i of this lane: column pair 4 i + t4 of the set, or (halves) 4 (2 i + (g >> 2)) + t4; B has the activation of
    // that pair in byte g & 3: byte i (2 i + (g >> 2)) of the packed words.
    constexpr int kWords = 2 * HB;
    const uint32_t sel0 = (0x4444u & ~(0xfu << (4 * (g & 3)))) | ((HB == 2 ? 0u : (uint32_t)(g >> 2)) << (4 * (g & 3)));
    const uint32_t sel_step = (HB == 2 ? 1u : 2u) << (4 * (g & 3));
    const uint32_t w_off = HB == 2 ? t4 * 32 + 4 * g : (4 * (g >> 2) + t4) * 16 + 4 * (g & 3);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    bool checked = !a.do_norm;
#pragma unroll 1
    for (;;) {
        named_barrier_sync(1, kOneWorkers);                          // packed words and weights are in place
        int acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        auto product = [&](auto blocks) {
            constexpr int NB = decltype(blocks)::value;
            // One block: the warps of the chain's scheduler stay out of the way, the chain is what the CTA waits for then (two
            // blocks: the product is). Down at K = 6912 7.6 -> 7.2 us.
            const int pw = NB == 2 ? kFusedWarps : kFusedWarps * 3 / 4, pi = NB == 2 ? warp : warp - (warp >> 2);
            if (NB == 1 && (warp & 3) == 3) return;
            const unsigned char* wt = s_wt + (size_t)pi * (256 * HB) + w_off;
            const size_t blk = (size_t)kh * (16 * HB);
            const uint2* bp = reinterpret_cast<const uint2*>(s_b + pi * 8) + t4;
#pragma unroll 2
            for (int s = pi; s < n_sets; s += pw, wt += 256 * HB * pw, bp += 4 * pw) {
                uint32_t W[NB][kWords];
                const uint2 b = *bp;
#pragma unroll
                for (int bk = 0; bk < NB; ++bk)
#pragma unroll
                    for (int i = 0; i < kWords; ++i) W[bk][i] = *reinterpret_cast<const uint32_t*>(wt + bk * blk + 128 * i);
#pragma unroll
                for (int i = 0; i < kWords; ++i) {
                    const uint32_t be = prmt(b.x, 0u, sel0 + i * sel_step), bo = prmt(b.y, 0u, sel0 + i * sel_step);
#pragma unroll
                    for (int bk = 0; bk < NB; ++bk) {
                        const uint32_t w = W[bk][i];
                        mma_u8s8(acc[NB == 1 ? i & 1 : bk], w & 0x03030303u, w & 0x30303030u, w & 0x0C0C0C0Cu, w & 0xC0C0C0C0u, be, bo);
                    }
                }
            }
        };
        if (glu) product(std::integral_constant<int, 2>{});
        else product(std::integral_constant<int, 1>{});
        if (!glu)                                                    // (of one block: two sums, for MMAs that do not wait for the one before)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[0][e] += acc[1][e];
        // D: rows g (low nibbles) and g + 8 (high ones), columns 2 t4, 2 t4 + 1: byte rows 4 g + column; of halves, columns 4-7
        // belong to the words of lanes g >= 4 and the other columns to those below. The warps meet.
        if (HB == 2 ? t4 < 2 : (t4 >> 1) == (g >> 2)) {
            int* d = s_d + 4 * (HB == 2 ? g : g & 3) + 2 * (t4 & 1);
#pragma unroll
            for (int bk = 0; bk < 2; ++bk, d += kRows) {
                if (bk >= nb_cta) break;
                atomicAdd(d, acc[bk][0]);                            // x4
                atomicAdd(d + 1, acc[bk][1]);
                atomicAdd(d + kRows / 2, acc[bk][2]);                // x64
                atomicAdd(d + kRows / 2 + 1, acc[bk][3]);
            }
        }
        if (checked) {
            named_barrier_sync(1, kOneWorkers);
            break;
        }
        // ---- the exact 1 / rms is known by now (or soon): do the integers stand? --------------------------------------------------
        if constexpr (!kKeep)
#pragma unroll
            for (int j = 0; j < P; ++j) load_w(j, wr[j]);
        named_barrier_sync(4, kOneThreads);
        float inv_rms = s_f[32];
        const unsigned long long top = *s_top;
        const float m_top = fabsf(normed(__uint_as_float((uint32_t)top), inv_rms, __uint_as_float((uint32_t)(top >> 32)))), to_q = 31.0f / fmaxf(m_top, 1e-6f);
        bool good = true;
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (tid + j * kOneWorkers < n_pieces) {
                float q[4];
                quantised(j, q);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float v = normed(xr[j][k], inv_rms, wr[j][k]);
                    good = good && fabsf(v) <= m_top && fabsf(v * to_q - q[k]) < 0.5f;
                }
            }
        m = m_top;
        if (!workers_any(!good)) break;                              // (also: every warp's sums are in s_d)
        asm volatile("" : "+f"(inv_rms));                            // (the check's values again, not kept: registers)
        float mm = 0.0f;
#pragma unroll
        for (int j = 0; j < P; ++j)
            if (tid + j * kOneWorkers < n_pieces)
#pragma unroll
                for (int k = 0; k < 4; ++k) mm = fmaxf(mm, fabsf(normed(xr[j][k], inv_rms, wr[j][k])));
        if (tid < 128) s_d[tid] = 0;
        if (tid == 0) *s_sa = 0;
        m = workers_max(mm);                                         // (its barrier also: the zeroes are in place)
        asm volatile("" : "+f"(inv_rms));
        exact_quantise(m, [&](int j, int k) { return normed(xr[j][k], inv_rms, wr[j][k]); });
        checked = true;
    }
    const float inv_act = fmaxf(m, 1e-6f) / 31.0f;                   // :35
    if (blockIdx.x == 0) {                                           // parity-check outputs
        if (checked && a.do_norm && tid == 0) atomicAdd(&g_tl1_repeats, 1);
        if (a.inv_out && tid == 0) a.inv_out[0] = inv_act;
        if (a.a_out)
#pragma unroll
            for (int j = 0; j < P; ++j)
                if (tid + j * kOneWorkers < n_pieces) {
                    float q[4];
                    quantised(j, q);
#pragma unroll
                    for (int k = 0; k < 4; ++k) a.a_out[4 * (tid + j * kOneWorkers) + k] = (int8_t)(int)q[k];
                }
    }
    if (tid < kRows) {
        const int sum_a = *s_sa;
        float v[2];
#pragma unroll
        for (int bk = 0; bk < 2; ++bk) {
            if (bk >= nb_cta) break;
            const int raw = s_d[bk * kRows + tid];
            const int accv = (tid < kRows / 2 ? (raw >> 2) : (raw >> 6)) - sum_a;
            if (a.acc_out) a.acc_out[out_row + (bk ? L.units * 64 : 0)] = accv;
            v[bk] = (float)accv * (inv_act * seg_scale_for(a, bk ? unit + L.units : unit));   // :1554, :118
        }
        float* o = a.out + out_row;
        if (a.epilogue == TENZO_EPI_STORE) {
            *o = v[0];
        } else if (a.epilogue == TENZO_EPI_RESIDUAL) {
            *o = resid_v + v[0];                                       // :1590
        } else {
            const float rl = fmaxf(0.0f, v[0]);
            *o = (rl * rl) * v[1];                                     // :1618-1619
        }
    }
}

// Cluster size along K: 1, 2, 4 or 8. Enough CTAs to put one on every SM, few enough sets per warp
// that a warp's loads are all in flight at once, a K range whose packed activations fit in shared
// memory, never more CTAs than sets.
static int pick_ksplit(int n_blocks, int K, int epilogue, int batch) {
    const int nsets = ((K >> 1) + 15) / 16;
    const int nb_cta = epilogue == TENZO_EPI_RELU2_GLU ? 2 : 1;
    const int units = n_blocks / nb_cta;
    int ks = 1;
    if (batch == 1) {
        // one CTA per row block, two resident per SM: weights (512 B per set per row block) + x must fit ~100 KB
        auto bytes = [&](int k) { return (size_t)((nsets + k - 1) / k + 1) * (512 * nb_cta + 32) + (size_t)K * 4 + 2048; };
        while (ks < 8 && ks * 2 <= nsets && (units * ks < 32 || bytes(ks) > 100 * 1024)) ks *= 2;
    } else {
        const int sl = batch <= 8 ? 8 : 32, seq_tiles = (batch + sl - 1) / sl;
        auto bytes = [&](int k) { return (size_t)((nsets + k - 1) / k + 1) * (512 * nb_cta + 32 * sl) + (size_t)sl * 520 + 1024; };
        while (ks < 8 && ks * 2 <= nsets && (units * ks * seq_tiles < 148 || bytes(ks) > 200 * 1024)) ks *= 2;
    }
    return ks;
}

// act_quant_kernel lives in norm_quant.cu
cudaError_t launch_act_quant(const float* x, const float* norm_w, int do_norm, float eps, int K, int batch, int x_stride,
                             uint32_t* words, float* inv, int8_t* a_out, int8_t* a_mma, int* sum_out, int use_pdl, cudaStream_t st);
// tcgen05 GEMM for nine or more sequences (tl1_umma.cu)
bool tl1_umma_applicable(const tenzo_tl1_gemv_args& a);
int launch_tl1_umma(const tenzo_tl1_gemv_args& a, const int8_t* a8, const float* inv, const int* sum_a, cudaStream_t st);
int tl1_umma_take_timeouts();
const int* tl1_timeouts_flag() {
    void* p = nullptr;
    return cudaGetSymbolAddress(&p, g_tl1_timeouts) == cudaSuccess ? static_cast<const int*>(p) : nullptr;
}

template <int NT, bool FUSED>
static cudaError_t launch_gemv(const GemvLaunch& L, cudaStream_t st) {
    using Lay = GemvSmem<NT, FUSED>;
    const tenzo_tl1_gemv_args& a = L.a;
    const int sets_per_cta = (L.nsets + L.ksplit - 1) / L.ksplit + 1;
    const size_t smem = Lay::bytes(sets_per_cta, a.K, a.epilogue == TENZO_EPI_RELU2_GLU ? 2 : 1);
    constexpr size_t kMostSmem = 220 * 1024;
    if (smem > kMostSmem) return cudaErrorInvalidValue;
    if (smem > 48 * 1024) {
        cudaError_t ea = allow_smem(tl1_mma_kernel<NT, FUSED>, kMostSmem);
        if (ea != cudaSuccess) return ea;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(L.units * L.ksplit), (unsigned)((a.batch + Lay::SL - 1) / Lay::SL), 1);
    cfg.blockDim = dim3((FUSED ? kFusedWarps : kBatchedWarps) * 32, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (L.ksplit > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = (unsigned)L.ksplit;
        attr[n_attr].val.clusterDim.y = 1;
        attr[n_attr].val.clusterDim.z = 1;
        ++n_attr;
    }
    if (a.use_pdl) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    return cudaLaunchKernelEx(&cfg, tl1_mma_kernel<NT, FUSED>, L);
}

static bool tl1_one_applicable(const tenzo_tl1_gemv_args& a) {
    const bool w = a.do_norm && a.norm_w;
    return a.batch == 1 && a.K % 32 == 0 && a.K <= kOneMaxK && ((reinterpret_cast<uintptr_t>(a.x) | (w ? reinterpret_cast<uintptr_t>(a.norm_w) : 0)) & 15) == 0;
}

static cudaError_t launch_tl1_one(const GemvLaunch& L, cudaStream_t st) {
    const tenzo_tl1_gemv_args& a = L.a;
    const int nb_cta = a.epilogue == TENZO_EPI_RELU2_GLU ? 2 : 1;
    // Half blocks double the CTAs and halve their loops, but every CTA quantises the whole vector: they pay while each has an SM of
    // its own. Products back to back in a graph, overlapped, half and whole blocks in us: 2560 wide 60 units 3.93 and 4.02,
    // 74 4.02 and 4.19, 80 4.90 and 4.35, 108 5.25 and 4.53, 148 5.79 and 4.87, 224 9.57 and 6.40; with GLU 80 6.19 and 4.87,
    // 108 6.66 and 5.13, 224 12.9 and 7.4; 4096 wide 60 4.70 and 4.68, 96 6.2 and 5.2, 224 with GLU 18.5 and 12.4; 1280 wide
    // 60 3.50 and 3.51, 90 4.39 and 3.76. Only at 6912 whole blocks win from 40 units on already (6.73 and 6.32).
    const int hb = 2 * L.units > 148 && OneSmem::bytes(a.K, nb_cta, 2) <= OneSmem::most() ? 2 : 1;
    const size_t smem = OneSmem::bytes(a.K, nb_cta, hb);
    auto kernel = a.K <= 8 * kOneWorkers ? (hb == 2 ? tl1_one_kernel<2, 2> : tl1_one_kernel<2, 1>) : (hb == 2 ? tl1_one_kernel<4, 2> : tl1_one_kernel<4, 1>);
    if (smem > 48 * 1024) {
        cudaError_t e = allow_smem(kernel, OneSmem::most());
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(L.units * (3 - hb)), 1, 1);
    cfg.blockDim = dim3(kOneThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, L);
}

}  // namespace tz

extern "C" int tenzo_cuda_tl1_gemv_ksplit(int n_blocks, int K, int epilogue) {
    if (n_blocks <= 0 || K <= 0) return 1;
    return tz::pick_ksplit(n_blocks, K, epilogue, 1);
}

namespace tz {
// Self-test of the give-up path of the bounded waits: barrier A is told to expect 32 bytes that nobody sends, so the wait
// on it (a short one: 2^8 polls) runs out, the kernel raises the same flag a real give-up raises and carries on; barrier
// B tracks the one 16-byte copy the kernel does issue and is waited for before the CTA's shared memory goes away. Nothing
// here can fault or hang: both waits are bounded, and the only memory touched is the kernel's own.
__global__ void __launch_bounds__(32) wait_expiry_selftest_kernel(const unsigned char* src16) {
    __shared__ __align__(16) unsigned char s_dst[16];
    __shared__ uint64_t s_bar[2];
    if (threadIdx.x == 0) {
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        mbar_init_fence();
        mbar_expect_tx(&s_bar[0], 32);
        mbar_expect_tx(&s_bar[1], 16);
        bulk_g2s(s_dst, src16, 16, &s_bar[1]);
        bool done = false;
        for (int it = 0; it < (1 << 8) && !done; ++it) done = mbar_test(&s_bar[0], 0);
        if (!done) atomicExch(&g_tl1_timeouts, 1);
        mbar_wait_bounded(&s_bar[1], 0);
    }
}
}  // namespace tz

extern "C" int tenzo_cuda_selftest_wait_expiry(void* stream) {
    static unsigned char* src = nullptr;
    if (!src) {
        if (cudaMalloc((void**)&src, 256) != cudaSuccess) return (int)cudaErrorMemoryAllocation;
        cudaMemset(src, 0, 256);
    }
    tz::wait_expiry_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(src);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}

extern "C" int tenzo_cuda_tl1_gemv_take_timeouts(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, tz::g_tl1_timeouts, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(tz::g_tl1_timeouts, &zero, sizeof zero);
    const int u = tz::tl1_umma_take_timeouts();
    if (u < 0) return -1;
    return v | u;
}

extern "C" int tenzo_cuda_tl1_gemv_take_repeats(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, tz::g_tl1_repeats, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(tz::g_tl1_repeats, &zero, sizeof zero);
    return v;
}

extern "C" size_t tenzo_cuda_tl1_gemv_workspace_bytes(int batch, int K) {
    if (batch <= 1 || K <= 0) return 0;
    const size_t nsets = ((size_t)(K >> 1) + 15) / 16;
    // packed activations (words path) or the int8 matrix in act_quant_kernel's a_mma order (tensor-core path), then inv[batch], then sum_a[batch]
    const size_t act = (size_t)batch * nsets * 32 > (size_t)batch * K ? (size_t)batch * nsets * 32 : (size_t)batch * K;
    return ((act + 15) & ~(size_t)15) + 2 * (size_t)batch * sizeof(float) + 64;
}

extern "C" int tenzo_cuda_tl1_gemv(const tenzo_tl1_gemv_args* args, void* stream) {
    using namespace tz;
    if (!args || !args->x || !args->w || !args->out) return -1;
    const tenzo_tl1_gemv_args& a = *args;
    if (a.n_blocks <= 0 || a.K <= 0 || (a.K & 1) || a.batch <= 0) return -1;
    if ((reinterpret_cast<uintptr_t>(a.w) & 15) != 0) return -1;   /* bulk copies start on 16-byte boundaries */
    if (a.epilogue < 0 || a.epilogue > 2) return -1;
    if (a.epilogue == TENZO_EPI_RESIDUAL && !a.resid) return -1;
    if (a.epilogue == TENZO_EPI_RELU2_GLU && (a.n_blocks & 1)) return -1;
    if (a.K > 16384) return -5;   /* same bound as the reference engine's scratch vectors (:1227) */
    if (a.batch > 1 && (!a.workspace || (reinterpret_cast<uintptr_t>(a.workspace) & 15) != 0)) return -1;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    GemvLaunch L;
    L.a = a;
    L.nsets = ((a.K >> 1) + 15) / 16;
    L.units = a.epilogue == TENZO_EPI_RELU2_GLU ? a.n_blocks / 2 : a.n_blocks;
    L.ksplit = pick_ksplit(a.n_blocks, a.K, a.epilogue, a.batch);
    L.act_words = nullptr;
    L.act_inv = nullptr;
    cudaError_t e;
    if (a.batch == 1) {
        e = tl1_one_applicable(a) ? launch_tl1_one(L, st) : launch_gemv<1, true>(L, st);
    } else {
        uint32_t* words = static_cast<uint32_t*>(a.workspace);
        const size_t act_bytes = (((size_t)a.batch * L.nsets * 32 > (size_t)a.batch * a.K ? (size_t)a.batch * L.nsets * 32 : (size_t)a.batch * a.K) + 15) & ~(size_t)15;
        float* inv = reinterpret_cast<float*>(static_cast<unsigned char*>(a.workspace) + act_bytes);
        if (tl1_umma_applicable(a)) {
            int8_t* a8 = static_cast<int8_t*>(a.workspace);
            int* sums = reinterpret_cast<int*>(inv + a.batch);
            e = launch_act_quant(a.x, a.norm_w, a.do_norm, a.eps, a.K, a.batch, a.x_stride, nullptr, inv, a.a_out, a8, sums, a.use_pdl, st);
            if (e != cudaSuccess) return (int)e;
            if (a.inv_out && (e = cudaMemcpyAsync(a.inv_out, inv, (size_t)a.batch * sizeof(float), cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return (int)e;
            return launch_tl1_umma(a, a8, inv, sums, st);
        }
        e = launch_act_quant(a.x, a.norm_w, a.do_norm, a.eps, a.K, a.batch, a.x_stride, words, inv, a.a_out, nullptr, nullptr, a.use_pdl, st);
        if (e != cudaSuccess) return (int)e;
        if (a.inv_out) {
            e = cudaMemcpyAsync(a.inv_out, inv, (size_t)a.batch * sizeof(float), cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return (int)e;
        }
        L.act_words = words;
        L.act_inv = inv;
        L.a.a_out = nullptr;
        L.a.inv_out = nullptr;
        e = a.batch <= 8 ? launch_gemv<1, false>(L, st) : launch_gemv<4, false>(L, st);
    }
    return e == cudaSuccess ? 0 : (int)e;
}

#ifdef TZ_TRACE
// Measurement builds only: copies up to max_records timeline records (16 words each) to `out`, resets the buffer and
// returns how many were copied.
extern "C" __attribute__((visibility("default"))) int tenzo_trace_gemv(unsigned long long* out, int max_records) {
    unsigned int n = 0;
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (cudaMemcpyFromSymbol(&n, tz::g_trace_n, sizeof n) != cudaSuccess) return -1;
    if (n > 4096u) n = 4096u;
    if ((int)n > max_records) n = (unsigned)max_records;
    if (n && cudaMemcpyFromSymbol(out, tz::g_trace, (size_t)n * 16 * sizeof(unsigned long long)) != cudaSuccess) return -1;
    const unsigned int zero = 0;
    if (cudaMemcpyToSymbol(tz::g_trace_n, &zero, sizeof zero) != cudaSuccess) return -1;
    return (int)n;
}
#endif
