// Batched TL1 bitlinear on the 5th-generation tensor cores (tcgen05.mma kind::i8, accumulators AND the weight
// operand in tensor memory) for sm_100a. Used by tenzo_cuda_tl1_gemv when there are at least nine sequences.
//
// Replaces, for many sequences at once, the same reference code as tl1_gemv.cu
// (src/runtime/TenzoEngine.cpp:22-166 and the call shapes :1547-1628 of the reference): integer
// accumulators are exact, so the result is bit-identical to the one-sequence path.
//
//   D[128 weight rows][N sequences] (int32, TMEM) += A[128][K] (u8 codes 0,1,2 times 1,4 or 16,64, TMEM) * B[K][N] (s8
//   activations times 4,1, smem); sum_k w*a = sum_k code*a - sum_k a   (w = code - 1; the per-sequence sum comes from the
//   quantiser)
//
// One CTA per 128-row tile (two 64-row TL1 blocks; for the GLU epilogue the gate block and its up block, so the
// activation is applied inside the CTA). K is walked in 128-byte chunks through two rings, 8 or 12 slots of codes in tensor
// memory and 4 or 12 activation tiles in shared memory (multiples of four: see UmmaSmem::a_slots_for); 21 warps per CTA:
//   warp 0 (lane 0)     bulk-copies the packed 2-bit weights eight chunks at a time (2 x 16 KB) into a ring of two or
//                       three groups; the first groups are requested by one lane each first thing in the kernel
//                       (weights depend on no earlier kernel); lanes 1-31 fetch the per-sequence scale and sum for
//                       the epilogue;
//   warps 2-17          (four groups of four; group g takes chunks g, g + 4, ..., two per iteration when there are
//                       twelve activation tiles) expand the 2-bit codes to bytes in registers and write them straight into
//                       the slot's 32 columns of tensor memory (tcgen05.st 16x256b: no shared-memory A tile, no
//                       proxy fence). Lane quarter q of a group takes one nibble half of one row block; a thread's
//                       four TMEM lanes are the four rows of ONE packed word, so a thread loads sixteen words per
//                       chunk and every byte of them is used. The row order inside a quarter is therefore permuted
//                       (TMEM lane l holds row 4*(l&7) + (l>>3)); the epilogue undoes it. Up to 96 sequences there are as
//                       many activation slots as code slots, and the warps of a group take turns TMA-loading the chunk's
//                       activation tile [N][128 B] (128-byte swizzle) right after they have seen the slot free;
//   warps 1, 18-20      (lane 0 each) take every fourth chunk: one poll of the slot's barrier (expand arrivals + the
//                       TMA's bytes), four tcgen05.mma (K = 32 each, A from tensor memory), one commit that frees the
//                       slot. A poll costs the issuing thread about 180 cycles, a commit about 80 and the loop
//                       another 270 (measured), more than the MMAs of a chunk take below 256 sequences, so one
//                       issuing thread bounds the loop; four hide it. Integer accumulation is order-free, and the
//                       expanding warps zero the accumulators while they wait for weights, so the threads need no
//                       order among them (when chunk 0 had to overwrite them first, the others lost 850 cycles). From 97
//                       sequences on there are four activation tiles only. With one ring for both, codes and MMAs then took
//                       turns (900 cycles a chunk for 516 of math); now the codes run eight chunks ahead, and each issuing
//                       thread requests the next tile of its own slot as soon as its MMAs have completed (one thread that
//                       requested all of them was the slowest role, 970 cycles a chunk): 640 cycles a chunk.
// After the last chunk every issuing thread commits to one barrier, which starts the epilogue on all sixteen expand
// warps (the groups on alternate 32-sequence column units; TMEM lane = weight row, tcgen05.ld 16 sequences at a
// time, scale / residual / ReLU^2*GLU, the unit assembled in shared memory and sent off by its own TMA store while
// the next one is computed).
// Few row tiles (the out, down and q|k|v projections have 20 to 30) would leave most SMs idle, so many sequences are then spread over
// several CTAs a row tile, or K is split (pick_umma_shape)
// across the 2, 4 or 8 CTAs of a thread-block cluster: each accumulates its share of the chunks in its own tensor
// memory and parks its int32 partial tile in shared memory; after a hardware cluster barrier every CTA takes the
// units of four sequences u = rank, rank + ksplit, ..., adds its peers' partials for them through distributed
// shared memory (integer sums: order-free, exact), runs the epilogue on them and stores them (a reduce-scatter:
// the epilogue work is spread over the cluster instead of queueing on one leader).
// Every mbarrier wait is bounded; a wait that gives up sets g_umma_timeouts, the roles fall through
// to the end and the TMEM allocation is released on every path.
#include <cooperative_groups.h>

#include <cstdlib>

#include "umma.cuh"
#include "../../include/tenzo_kernels.h"

namespace cg = cooperative_groups;

namespace tz {

constexpr int kExpandGroups = 4;               // groups of four warps that expand alternate chunks (and run the epilogue)
constexpr int kUmmaThreads = 32 * (2 + 4 * kExpandGroups + 3);   // warp 0 producer, warp 1 and the last three MMA issue, the rest expand
// From nine sequences on: up to eight, one mma.sync column group holds them all (8.8 us for quantiser and 3840 x 2560 product,
// 11.9 for 2560 x 6912; here 8.9 and 13.2), with more it takes four (21 and 25 us; here 9.0 and 13.5).
constexpr int kUmmaMinBatch = 9;
constexpr int kMmaThreads = 4;
constexpr int kMaxSlots = 16;                  // ring of chunk slots: as many as tensor memory and shared memory allow
constexpr int kPGroup = 8;                     // chunks of packed weights per bulk copy (16 KB per row block)
constexpr int kMaxPGroups = 3;                 // such groups in the ring (3 up to 64 sequences, else 2): 64 KB of packed weights in flight behind the group in use
constexpr int kKc = 128;                       // bytes of K per chunk (one swizzle atom row)
constexpr int kTileRows = 128;
constexpr int kPBytes = 2 * (kKc / 2) * 32;    // packed weights of one chunk, two row blocks: 4 KB
constexpr int kMaxN = 256;
constexpr int kTmemCols = 512;                 // columns 0..N-1 accumulators, then 32 columns per slot for the A operand
constexpr int kSmemBudget = 216 * 1024;        // activation ring + packed-weight ring

struct UmmaLaunch {
    tenzo_tl1_gemv_args a;
    const float* inv;        // [batch] m/31
    const int* sum_a;        // [batch] sum_k a_k
    int units;               // tiles along the rows
    int n_box;               // sequences per CTA, a multiple of 16 (<= 256)
    int n_slots;             // ring slots (A in tensor memory)
    int b_slots;             // activation tiles in shared memory: as many, or four (then the issuing threads request them)
    int n_pgroups;           // groups of kPGroup chunks in the packed-weight ring
    int ksplit;              // CTAs of a cluster that share one tile's K range (1 = no cluster)
    int store_cols;          // sequences per TMA store of the epilogue (32; 16 up to 64 sequences, 4 with a cluster or up to 32)
};

__device__ int g_umma_timeouts = 0;

// Optional in-kernel timeline (compile with -DTZ_UMMA_TRACE): CTA-local clock64 stamps per phase, read back through
// tenzo_trace_umma; compiled out of the library build.
#ifdef TZ_UMMA_TRACE
__device__ long long g_umma_trace[160 * 16];
#define UT(i) (g_umma_trace[(blockIdx.x % 160) * 16 + (i)] = clock64())
__device__ long long g_umma_chunks[64 * 8];      // CTA 0: per chunk, when each role reached it
#define UC(j, k) do { if (blockIdx.x == 0 && blockIdx.z == 0 && (j) < 64) g_umma_chunks[(j) * 8 + (k)] = clock64(); } while (0)
#define UTG(i) do { long long t_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_)); g_umma_trace[(blockIdx.x % 160) * 16 + (i)] = t_; } while (0)
#else
#define UT(i) ((void)0)
#define UC(j, k) ((void)0)
#define UTG(i) ((void)0)
#endif

// Optional self-check (compile with -DTZ_UMMA_CHECK): every shared-memory range handed to a copy engine and every
// tensor-memory column range is checked against the allocation first; a violation is recorded (code, value, limit) and
// the access skipped. Read back through tenzo_check_umma; compiled out of the library build.
#ifdef TZ_UMMA_CHECK
__device__ unsigned long long g_umma_check[4];
__device__ __forceinline__ bool umma_check(bool good, int code, unsigned long long v, unsigned long long lim) {
    if (!good && atomicCAS(&g_umma_check[0], 0ull, (unsigned long long)code) == 0ull) { g_umma_check[1] = v; g_umma_check[2] = lim; g_umma_check[3] = blockIdx.x; }
    return good;
}
#define UCHK(good, code, v, lim) umma_check((good), (code), (unsigned long long)(v), (unsigned long long)(lim))
#else
#define UCHK(good, code, v, lim) true
#endif

__device__ __forceinline__ float umma_seg_scale(const tenzo_tl1_gemv_args& a, int block) {
    return block < a.seg_end[0] ? a.seg_scale[0] : (block < a.seg_end[1] ? a.seg_scale[1] : a.seg_scale[2]);
}

struct UmmaSmem {
    // [1024-aligned] ring b_slots x { B n_box*128 } | packed ring n_pgroups x 2 blocks x 16 KB | barriers | tmem slot | inv[256] | sum_a[256]
    static __host__ __device__ int pgroups_for(int n_box) { return n_box <= 64 ? kMaxPGroups : 2; }
    static __host__ __device__ int tmem_a(int n_box) { return (n_box + 31) & ~31; }          // first column of the A slots
    // Both numbers are multiples of four (the expand groups and the issuing threads): slot s then always belongs to group s % 4 and
    // thread s % 4, so every phase of a slot's barriers is seen, in order, by the same waiter. (A parity wait
    // cannot tell phase k from phase k - 2: with five slots a thread that ran ahead of its neighbour took a slot's
    // previous phase for the one it waited for and multiplied a tile that had not arrived.)
    static __host__ __device__ int a_slots_for(int n_box) {                                  // by tensor memory: 12 up to 128 sequences, 8 at 256
        const int r = (kTmemCols - tmem_a(n_box)) / 32;
        return (r < kMaxSlots ? r : kMaxSlots) & ~3;
    }
    // By shared memory: 12 or more up to 96 sequences, else 4. Eight, which would fit up to 144, are one iteration of all expanding warps: with four
    // the codes run ahead of the tiles instead (28672 x 4096 with GLU at 128 sequences 30.7 -> 28.4 us, 2560 x 6912 24.0 -> 22.4; at 96, from twelve
    // to four, 25.6 -> 26.8).
    static __host__ __device__ int b_slots_for(int n_box) {
        const int r = (kSmemBudget - pgroups_for(n_box) * kPGroup * kPBytes) / (n_box * kKc), a = a_slots_for(n_box), b = (r < a ? r : a) & ~3;
        return b < 12 ? 4 : b;
    }
    static constexpr int n_bars = 2 * kMaxSlots + 2 * kMaxPGroups + 3;
    static __host__ __device__ size_t bytes(int n_box) {
        return 1024 + (size_t)b_slots_for(n_box) * n_box * kKc + (size_t)pgroups_for(n_box) * kPGroup * kPBytes + ((8 * n_bars + 15) & ~15) + 16 + 2 * kMaxN * 4;
    }
};

// Slot and round of a chunk in a ring of n slots, stepped without a division (by at most n): n is a run-time number, and the
// divisions were on the way of every hand-over (13824 x 2560 with GLU at 12 sequences 13.9 -> 12.7 us, 28672 x 4096 29.2 -> 25.7).
struct RingPos {
    int slot, round;
    __device__ __forceinline__ void step(int by, int n) {
        slot += by;
        if (slot >= n) { slot -= n; ++round; }
    }
};

// NC sequences of the epilogue: r = accumulators of TMEM lane m (weight row `row`, `rr` inside its block).
template <int EPI, int NC>
__device__ __forceinline__ void umma_epilogue_block(const tenzo_tl1_gemv_args& a, uint32_t (&r)[NC], const float* s_inv, const int* s_sum, float wscale,
                                                    int shift, int c0, int seq0, int block, int rr, int row, bool up_half, float* s_out_cols, float* s_glu_cols, bool ok) {
    float v[NC];
#pragma unroll
    for (int i = 0; i < NC; i += 4) {
        const int4 sv = *reinterpret_cast<const int4*>(s_sum + c0 + i);
        const float4 iv = *reinterpret_cast<const float4*>(s_inv + c0 + i);
        const int s4[4] = {sv.x, sv.y, sv.z, sv.w};
        const float i4[4] = {iv.x, iv.y, iv.z, iv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int accv = ((int)r[i + e] >> shift) - s4[e];
            r[i + e] = (uint32_t)accv;
            v[i + e] = (float)accv * (i4[e] * wscale);      // :1554, :118
        }
    }
    if (a.acc_out && ok && block >= 0) {
#pragma unroll
        for (int i = 0; i < NC; ++i)
            if (seq0 + c0 + i < a.batch) a.acc_out[(size_t)(seq0 + c0 + i) * a.n_blocks * 64 + block * 64 + rr] = (int)r[i];
    }
    if (EPI == TENZO_EPI_RELU2_GLU) {
        if (up_half) {                                   // the up value, and ReLU(gate)^2: multiplied once both are in place
#pragma unroll
            for (int i = 0; i < NC; ++i) s_glu_cols[i * 64 + rr] = v[i];
        } else {
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                const float rl = fmaxf(0.0f, v[i]);
                s_out_cols[i * 64 + rr] = rl * rl;                               // :1618
            }
        }
    } else if (EPI == TENZO_EPI_RESIDUAL) {
        float res[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int seq = seq0 + c0 + i;
            res[i] = (seq < a.batch && block >= 0) ? __ldcg(a.resid + (size_t)seq * a.out_stride + block * 64 + rr) : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) s_out_cols[i * 128 + row] = res[i] + v[i];                          // :1590
    } else {
#pragma unroll
        for (int i = 0; i < NC; ++i) s_out_cols[i * 128 + row] = v[i];
    }
}

template <int EPI, bool CLUSTER>
__global__ void __launch_bounds__(kUmmaThreads, 1) tl1_umma_kernel(const UmmaLaunch L, const __grid_constant__ CUtensorMap amap,
                                                                   const __grid_constant__ CUtensorMap omap) {
    const tenzo_tl1_gemv_args& a = L.a;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base_off = ((smem_addr(smem_raw) + 1023u) & ~1023u) - smem_addr(smem_raw);
    unsigned char* ring = smem_raw + base_off;
    const int N = L.n_box, R = L.n_slots, RB = L.b_slots, slot_bytes = N * kKc;
    const bool b_ahead = RB < R;                       // the codes run further ahead than the activation tiles do
    const int PG = L.n_pgroups;
    unsigned char* pring = ring + (size_t)RB * slot_bytes;                       // [PG][2 row blocks][kPGroup chunks][64][32] packed weights
    uint64_t* bars = reinterpret_cast<uint64_t*>(pring + (size_t)PG * kPGroup * kPBytes);
    const uint32_t tmem_a0 = (uint32_t)UmmaSmem::tmem_a(N);
    uint64_t* bar_full = bars;                         // [R] A expanded (one arrival per expanding warp) and the activation tile landed
    uint64_t* bar_empty = bars + kMaxSlots;            // [R] the slot's MMAs have completed
    uint64_t* bar_p = bars + 2 * kMaxSlots;            // [PG] packed weights have landed
    uint64_t* bar_pfree = bar_p + kMaxPGroups;         // [PG] packed weights consumed (one arrival per expanding warp per chunk)
    uint64_t* bar_accum = bar_pfree + kMaxPGroups;        // every issuing thread's MMAs have completed
    uint64_t* bar_zero = bar_accum + 1;                // the accumulators are zero (one arrival per expanding warp)
    uint64_t* bar_meta = bar_zero + 1;                 // per-sequence scale and sum are in shared memory
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(bars) + ((8 * UmmaSmem::n_bars + 15) & ~15));   // 16-byte aligned
    float* s_inv = reinterpret_cast<float*>(tmem_slot + 4);   // [kMaxN] m/31 of this CTA's sequences
    int* s_sum = reinterpret_cast<int*>(s_inv + kMaxN);       // [kMaxN] sum_k a_k

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { UT(0); UTG(10); }
#ifdef TZ_UMMA_CHECK
    uint32_t dyn_bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    const unsigned char* smem_end = smem_raw + dyn_bytes;
    UCHK(reinterpret_cast<const unsigned char*>(s_sum + kMaxN) <= smem_end, 7, reinterpret_cast<const unsigned char*>(s_sum + kMaxN) - smem_raw, dyn_bytes);
#endif
    constexpr bool glu = EPI == TENZO_EPI_RELU2_GLU;
    const int tile = blockIdx.x, seq0 = blockIdx.y * L.n_box;
    const int blk0 = glu ? tile : 2 * tile;
    const int blk1 = glu ? tile + L.units : (2 * tile + 1 < a.n_blocks ? 2 * tile + 1 : -1);
    const int ksplit = CLUSTER ? L.ksplit : 1;
    const int split = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;         // cluster = the CTAs with this tile's blockIdx.z = 0..ksplit-1
    const int all_chunks = a.K / kKc;
    const int ks_shift = 31 - __clz(ksplit);                                        // (a power of two; a division would be on the way of the first copies)
    const int c_begin = split * all_chunks >> ks_shift;                             // this CTA's chunks of K: never empty (all_chunks >= ksplit)
    const int n_chunks = ((split + 1) * all_chunks >> ks_shift) - c_begin;

    const size_t blk_bytes = (size_t)(a.K / 2) * 32;
    const int n_groups = (n_chunks + kPGroup - 1) / kPGroup;
    auto request_group = [&](int g, int slot) {            // packed weights of chunks kPGroup*g .. kPGroup*g + kPGroup-1, both row blocks
        const int chunks = min(kPGroup, n_chunks - g * kPGroup);
        const unsigned bytes = (unsigned)chunks * (kPBytes / 2);
        unsigned char* sP = pring + (size_t)slot * kPGroup * kPBytes;
        if (!UCHK(sP + 2 * kPGroup * (kPBytes / 2) <= reinterpret_cast<unsigned char*>(bars) && slot < PG && chunks > 0, 1, sP - smem_raw, g)) return;
        mbar_expect_tx(&bar_p[slot], blk1 >= 0 ? 2 * bytes : bytes);
        const size_t k_off = (size_t)(c_begin + g * kPGroup) * (kPBytes / 2);
        bulk_g2s(sP, a.w + (size_t)blk0 * blk_bytes + k_off, bytes, &bar_p[slot]);
        if (blk1 >= 0) bulk_g2s(sP + kPGroup * (kPBytes / 2), a.w + (size_t)blk1 * blk_bytes + k_off, bytes, &bar_p[slot]);
    };
    if (warp == 0 && lane < PG) {
        // The weights depend on no earlier kernel and their latency is the longest in the prologue: ask for the first
        // groups before anything else, one lane per group (an mbarrier operation or a bulk-copy issue costs its thread
        // over a hundred cycles; the other barriers are initialised by another warp meanwhile).
        mbar_init(&bar_p[lane], 1);
        mbar_init_fence();
        if (lane < n_groups) request_group(lane, lane);
        if (lane == 0) UT(2);
    } else if (warp == 2) {
        if (lane < R) {
            mbar_init(&bar_full[lane], 5);             // four expanding warps + the expect_tx of the warp that requests the activation tile
            mbar_init(&bar_empty[lane], 1);
        } else if (lane >= 16 && lane < 16 + kMaxPGroups) {
            mbar_init(&bar_pfree[lane - 16], 4 * kExpandGroups * (b_ahead ? 2 : 1));   // one arrival per expanding warp per iteration
        } else if (lane == 24) {
            mbar_init(bar_accum, kMmaThreads);
        } else if (lane == 25) {
            mbar_init(bar_zero, 4 * kExpandGroups);
        } else if (lane == 26) {
            mbar_init(bar_meta, 1);
        }
        mbar_init_fence();
    } else if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp >= 3) l2_prefetch_slice(a.prefetch, a.prefetch_bytes);       // the next kernel's weights
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    if (tid == 0) UT(1);
    bool timed_out = false, epi_ok = false;
    const int mma_t = warp == 1 ? 0 : warp - (1 + 4 * kExpandGroups);        // issuing thread 0..3: warp 1 and the three warps after the expand warps

    if (warp == 0) {
        if (lane == 0) {
            // ---- producer: the remaining groups of packed weights, each as soon as its ring half is free -------
            RingPos at = {0, 1};
            for (int gp = PG; gp < n_groups; ++gp) {
                if (!mbar_spin_bounded(&bar_pfree[at.slot], (unsigned)(at.round - 1) & 1u)) { timed_out = true; break; }
                request_group(gp, at.slot);
                at.step(1, PG);
            }
        } else {
            // ---- per-sequence epilogue operands (quantiser outputs) ---------------------------------------
            if (a.use_pdl) {
                pdl_wait();
                pdl_launch_dependents();                         // after the own wait: see act_quant_kernel
            }
            for (int i = lane - 1; i < N; i += 31) {
                const int seq = seq0 + i;
                s_inv[i] = seq < a.batch ? __ldcg(L.inv + seq) : 0.0f;
                s_sum[i] = seq < a.batch ? __ldcg(L.sum_a + seq) : 0;
            }
            __syncwarp(0xfffffffeu);
            if (lane == 1) mbar_arrive(bar_meta);
        }
    } else if (warp == 1 || warp >= 2 + 4 * kExpandGroups) {
        // ---- MMA issue: thread t takes chunks t, t + 4, ... ---------------------------------------------------
        if (lane == 0) {
            // c = s32, a = u8, b = s8, both K-major, N at bit 17 (>>3), M at bit 24 (>>4)
            const uint32_t idesc = (2u << 4) | (0u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
            // With fewer activation slots than code slots (four) a thread also requests its chunks' tiles: the slot is its own,
            // and the tile after next is due when the MMAs it has just issued have completed.
            auto request_tile = [&](int j, int s) {
                if (UCHK(ring + (size_t)(mma_t + 1) * slot_bytes <= pring, 2, mma_t, j)) {
                    mbar_expect_tx(&bar_full[s], (unsigned)slot_bytes);
                    tma_load_2d(ring + (size_t)mma_t * slot_bytes, &amap, (c_begin + j) * kKc, seq0, &bar_full[s]);
                }
            };
            RingPos at = {mma_t, 0};
            if (b_ahead && mma_t < n_chunks) {
                if (a.use_pdl) pdl_wait();
                request_tile(mma_t, mma_t);
            }
            if (mma_t < n_chunks && !mbar_spin_bounded(bar_zero, 0u)) timed_out = true;
            for (int j = mma_t; j < n_chunks && !timed_out; j += kMmaThreads) {
                const int s = at.slot, sb = b_ahead ? mma_t : s;
                const unsigned parity = (unsigned)at.round & 1u;
                at.step(kMmaThreads, R);
                UC(j, 4);
                if (!mbar_spin_bounded(&bar_full[s], parity)) { timed_out = true; break; }
                tc_fence_after();
                UC(j, 5);
                const uint32_t ta = tmem_base + tmem_a0 + (uint32_t)(32 * s);
                const uint64_t db = umma_desc_sw128(smem_addr(ring + (size_t)sb * slot_bytes));
                if (UCHK(tmem_a0 + 32 * s + 32 <= (uint32_t)kTmemCols && s < R && ring + (size_t)(sb + 1) * slot_bytes <= pring, 5, s, j))
#pragma unroll
                for (int k4 = 0; k4 < kKc / 32; ++k4)
                    umma_i8_ta(tmem_base, ta + (uint32_t)(8 * k4), db + (uint64_t)(2 * k4), idesc, 1u);
                umma_commit(&bar_empty[s]);
                UC(j, 6);
                if (b_ahead && j + kMmaThreads < n_chunks) {
                    if (!mbar_spin_bounded(&bar_empty[s], parity)) { timed_out = true; break; }
                    request_tile(j + kMmaThreads, at.slot);
                }
            }
            umma_commit(bar_accum);
        }
    } else {
        // ---- expand the 2-bit codes into tensor memory ----------------------------------------------------------
        // Quarter q = warp & 3 owns TMEM lanes 32q..32q+31 = row block q >> 1, nibble half q & 1. Thread 4g + t holds
        // lanes g + 8*jj (jj = 0..3) = rows 4g + jj of the half = the four bytes of packed word g of a column pair, and
        // the columns 8n + 2t, 8n + 2t + 1 = column pairs 16n + 4t .. 16n + 4t + 3. The four words of a (thread, n) are
        // fetched in the order u ^ t so that a warp's request covers 32 banks. A column is made of two words: their
        // bytes, and of each byte the even column's code in the lower half, the odd column's in the upper, where they lie
        // (1 and 4 times the code for the nibbles of the first 32 rows, 16 and 64 times for the second; the even columns'
        // activations carry a four, and the epilogue shifts the sums back). The order of K that comes of it is the one the
        // quantiser writes (mma_word): one permute and one mask a column, where shifting the codes down and putting the
        // columns in order took two to four more of a pipe that takes one in two cycles. (Quantiser and product, 12 sequences: 13824 x 2560 with
        // GLU 15.4 -> 13.9 us, 28672 x 4096 33.1 -> 29.2; 256 sequences: 23.8 -> 22.5 and 52.7 -> 48.6.)
        const int q = warp & 3, grp = (warp - 2) >> 2;
        const int blk = q >> 1, hi = q & 1, g = lane >> 2, t = lane & 3;
        const bool have = blk == 0 || blk1 >= 0;
        const uint32_t codes = hi ? 0xC0C03030u : 0x0C0C0303u;
        int woff[4];                                           // word offsets of the four loads inside a 16-column-pair set
#pragma unroll
        for (int u = 0; u < 4; ++u) woff[u] = (4 * t + (u ^ t)) * 8 + g;
        // An iteration costs a warp about two thousand cycles whatever it expands (a poll of a barrier that has long
        // completed is 300 cycles, a tensor-memory store 500 until it has landed), so where the activation tiles have as many
        // slots it takes two chunks, j and j + 4: one poll for both slots (the same thread issues both chunks' MMAs in order, so the
        // later one's completion implies the earlier one's), one for the weights (both lie in the same group of eight),
        // the two polls on different lanes, one wait for the four stores.
        const int cpi = b_ahead ? 1 : 2;
        // While the first weights are on their way: zero the accumulators (the groups alternate 16-column blocks).
        for (int c0 = 16 * grp; c0 < N; c0 += 16 * kExpandGroups) tmem_zero16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_zero);
        int seen_group = -1;
        RingPos next = {grp, 0}, weights = {0, 0};           // of the iteration's first chunk and of its group of packed weights
        for (int it = 0, j0 = grp; j0 < n_chunks; ++it, j0 += kExpandGroups * cpi) {
            const int n_here = (cpi == 2 && j0 + kExpandGroups < n_chunks) ? 2 : 1;
            const int pg = j0 / kPGroup;
            if (pg != seen_group && pg > 0) weights.step(1, PG);
            const int ps = weights.slot;
            RingPos at[2] = {next, next};
            at[1].step(kExpandGroups, R);
            next.step(kExpandGroups * cpi, R);
            bool ok = true;
            if (lane == 0 && q == 0) { UC(j0, 0); if (n_here == 2) UC(j0 + kExpandGroups, 0); }
            {   // lane 0 waits for the slot, lane 1 for the weights: the same code for both, or one would wait after the other
                const RingPos last = n_here == 2 ? at[1] : at[0];
                uint64_t* bar = lane == 0 ? &bar_empty[last.slot] : &bar_p[ps];
                const int round = lane == 0 ? last.round - 1 : weights.round;
                if (lane == 0 ? round >= 0 : lane == 1 && pg != seen_group) ok = mbar_spin_bounded(bar, (unsigned)round & 1u);
            }
            seen_group = pg;
            ok = __all_sync(0xffffffffu, ok);
            __syncwarp();                                   // what lanes 0 and 1 acquired is visible to the whole warp
            if (j0 == 0 && tid == 64) UT(6);
            if (!ok) { timed_out = true; break; }
            tc_fence_after();
            if (lane == 0 && q == 0) { UC(j0, 1); if (n_here == 2) UC(j0 + kExpandGroups, 1); }
            // The group's warps take turns requesting the activation tiles. They come from the previous kernel, so in the
            // first iteration the request (and the wait for that kernel) is left until the chunks have been expanded:
            // the weights depend on nothing, and the previous kernel runs about as long as the first round of expansion.
            auto request_tiles = [&]() {
                for (int c = 0; c < n_here; ++c) {
                    const int j = j0 + kExpandGroups * c, s = c ? at[1].slot : at[0].slot;
                    if (!b_ahead && lane == 0 && ((it * cpi + c) & 3) == q) {
                        if (UCHK(s < R && ring + (size_t)(s + 1) * slot_bytes <= pring, 2, s, j)) {
                            mbar_expect_tx(&bar_full[s], (unsigned)slot_bytes);
                            tma_load_2d(ring + (size_t)s * slot_bytes, &amap, (c_begin + j) * kKc, seq0, &bar_full[s]);
                        }
                    }
                }
            };
            const bool request_last = it == 0 && a.use_pdl;
            if (!request_last) request_tiles();
            for (int c = 0; c < n_here; ++c) {
                const int j = j0 + kExpandGroups * c, s = c ? at[1].slot : at[0].slot;
                const uint32_t* sP = reinterpret_cast<const uint32_t*>(pring + (size_t)ps * kPGroup * kPBytes + (size_t)blk * kPGroup * (kPBytes / 2) +
                                                                       (size_t)(j % kPGroup) * (kPBytes / 2));
                uint32_t W[16];
                const bool sp_ok = UCHK(reinterpret_cast<const unsigned char*>(sP) >= pring && reinterpret_cast<const unsigned char*>(sP + 512) <= reinterpret_cast<unsigned char*>(bars), 3,
                                        reinterpret_cast<const unsigned char*>(sP) - smem_raw, j);
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int u = 0; u < 4; ++u) W[4 * n + u] = (have && sp_ok) ? sP[n * 128 + woff[u]] : 0u;
                uint32_t lo[16], up[16];                       // registers of the two stores: lanes 0-15 (jj = 0, 1) and 16-31 (jj = 2, 3)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj) {           // byte jj of two words, twice, and its codes left where they are
                        uint32_t* dst = (jj < 2 ? lo : up) + 4 * n + 2 * (jj & 1);
                        dst[0] = prmt(W[4 * n], W[4 * n + 1], 0x4040u + 0x1111u * jj) & codes;
                        dst[1] = prmt(W[4 * n + 2], W[4 * n + 3], 0x4040u + 0x1111u * jj) & codes;
                    }
                const uint32_t ta = tmem_base + tmem_a0 + (uint32_t)(32 * s) + ((uint32_t)(32 * q) << 16);
                if (UCHK(tmem_a0 + 32 * s + 32 <= (uint32_t)kTmemCols && (tmem_base & 0xffffu) == 0u, 4, tmem_a0 + 32 * s, tmem_base)) {
                    tmem_st_16x256b_x4(ta, lo);
                    tmem_st_16x256b_x4(ta + (16u << 16), up);
                }
            }
            if (lane == 0 && q == 0) { UC(j0, 2); if (n_here == 2) UC(j0 + kExpandGroups, 2); }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_pfree[ps]);       // every lane's packed words have been loaded and used
            if (request_last && !b_ahead) {
                if (lane == 0) pdl_wait();
                request_tiles();
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane < n_here) mbar_arrive(&bar_full[lane ? at[1].slot : at[0].slot]);
            if (lane == 0 && q == 0) { UC(j0, 3); if (n_here == 2) UC(j0 + kExpandGroups, 3); }
        }
        // ---- all of this CTA's MMAs have completed; in a cluster it parks its partial tile [N][128 TMEM lanes] int32
        //      (the columns its peers will reduce) in the ring memory the pipeline no longer needs -----------------
        if (a.use_pdl) pdl_wait();                           // the residual rows come from an earlier kernel (long done by now)
        bool ok = true;
        if (lane == 0) ok = !timed_out && mbar_spin_bounded(bar_meta, 0u) && mbar_spin_bounded(bar_accum, 0u);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();
        if (!ok) timed_out = true;
        tc_fence_after();
        if (tid == 64) UT(7);
        epi_ok = ok;
        if (CLUSTER) {
            const int m = 32 * q + lane;
            int* s_part = reinterpret_cast<int*>(ring);
            for (int c0 = 16 * grp; c0 < N; c0 += 16 * kExpandGroups) {
                uint32_t r[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) r[i] = 0u;
                if (ok) tmem_ld16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, r);
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    if ((((c0 + i) >> 2) & (ksplit - 1)) != split)                                              // (this CTA's own units stay in tensor memory)
                        *reinterpret_cast<uint4*>(s_part + (c0 + i) * 128 + 4 * m) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
            }
        }
    }
    if (CLUSTER) cg::this_cluster().sync();                  // every CTA's partial tile is in place
    if (warp >= 2 && warp < 2 + 4 * kExpandGroups) {
        // ---- epilogue: every group, alternate column units; TMEM lane -> weight row through the quarter's permutation ----
        const bool ok = epi_ok;
        const int q = warp & 3, grp = (warp - 2) >> 2;
        const int m = 32 * q + lane;                         // TMEM lane
        const int rblk = q >> 1, rr = 32 * (q & 1) + 4 * (lane & 7) + (lane >> 3), row = 64 * rblk + rr;
        const int block = rblk ? blk1 : blk0;
        const int shift = q & 1 ? 6 : 2;                     // the sums are 4 and 64 times the products (exactly)
        const float wscale = block >= 0 ? umma_seg_scale(a, block) : 0.0f;
        // Output columns [sequences][128 rows] (GLU: [..][64]) are assembled in shared memory the pipeline no longer
        // needs - the rings, which are contiguous; with a cluster behind the partial tile the peers are reading - and
        // leave unit by unit through TMA stores: rows of 512 (256) contiguous bytes per sequence, clipped at the
        // matrix edge by the tensor map. GLU: the up half parks its values and the gate half its ReLU^2 side by side, then
        // the group multiplies them in place. Space: N*512 bytes without a cluster (at least four slots), N*512 plus 512 per
        // own column with one (a rank owns at most every other unit), which the two rings hold for every N.
        // A unit is 32 sequences, 16 up to 64 and four with a cluster or up to 32, so that all groups of all ranks have some: with units
        // of sixteen, 64 sequences on four ranks were one group's work in each, twelve one group's of one rank (quantiser and product,
        // 2560 x 6912: 64 sequences 17.2 -> 15.2 us, 12 sequences 16.1 -> 14.1, 256 25.7 -> 22.9).
        constexpr int row_floats = glu ? 64 : 128;
        float* s_out = reinterpret_cast<float*>(ring + (CLUSTER ? (size_t)N * 512 : 0));            // behind the partial tile [N][128] int32
        float* s_glu = s_out + (size_t)(CLUSTER ? 4 * ((N / 4 + 1) / 2) : N) * 64;                   // behind the GLU output columns (a rank owns at most every other unit)
        const bool leader = lane == 0 && q == 0;
        const uint32_t t_lane = tmem_base + ((uint32_t)(32 * q) << 16);
        auto send = [&](float* unit_out, float* unit_glu, int cols, int c0) {      // a unit assembled by the group's four warps
            if (glu) {
                // gate and up halves of the unit are both in shared memory: out = ReLU(gate)^2 * up, four floats at a time
                named_barrier_sync(1 + grp, 128);
                float4* o4 = reinterpret_cast<float4*>(unit_out);
                const float4* g4 = reinterpret_cast<const float4*>(unit_glu);
                for (int i = 32 * q + lane; i < cols * 16; i += 128) {
                    float4 o = o4[i];
                    const float4 u = g4[i];
                    o.x *= u.x; o.y *= u.y; o.z *= u.z; o.w *= u.w;             // :1619
                    o4[i] = o;
                }
            }
            // the unit is complete in shared memory: hand it to the TMA and go on with the next one
            fence_proxy_async_smem();
            named_barrier_sync(1 + grp, 128);
            if (leader && ok && seq0 + c0 < a.batch &&
                UCHK(reinterpret_cast<unsigned char*>(unit_out) + L.store_cols * row_floats * 4 <= reinterpret_cast<unsigned char*>(bars), 6,
                     reinterpret_cast<unsigned char*>(unit_out) - smem_raw, c0)) {             // else nothing but padding
                asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
                             ::"l"(&omap), "r"((glu ? tile : blk0) * 64), "r"(seq0 + c0), "r"(smem_addr(unit_out)) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        };
        if (CLUSTER || L.store_cols == 4) {
#pragma unroll 1
            for (int k = grp;; k += kExpandGroups) {
                const int c0 = 4 * (CLUSTER ? split + ksplit * k : k);
                if (c0 >= N || seq0 + c0 >= a.batch) break;
                uint32_t r[4] = {0u, 0u, 0u, 0u};
                if (ok) {
                    tmem_ld4_nowait(t_lane + (uint32_t)c0, r);
                    tmem_wait_ld();
                }
                if (CLUSTER) {
                    // the peers' partials over distributed shared memory, every load issued before the first is used
                    uint4 part[8];
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        const bool use_p = p < ksplit && p != split;
                        const int* peer = cg::this_cluster().map_shared_rank(reinterpret_cast<int*>(ring), use_p ? p : split);
                        part[p] = use_p ? *reinterpret_cast<const uint4*>(peer + c0 * 128 + 4 * m) : make_uint4(0u, 0u, 0u, 0u);
                    }
#pragma unroll
                    for (int p = 0; p < 8; ++p) { r[0] += part[p].x; r[1] += part[p].y; r[2] += part[p].z; r[3] += part[p].w; }
                }
                float* unit_out = s_out + (size_t)4 * k * row_floats;
                float* unit_glu = s_glu + (size_t)4 * k * 64;
                umma_epilogue_block<EPI, 4>(a, r, s_inv, s_sum, wscale, shift, c0, seq0, block, rr, row, rblk == 1, unit_out, unit_glu, ok);
                send(unit_out, unit_glu, 4, c0);
            }
        } else {
#pragma unroll 1
            for (int c0 = L.store_cols * grp; c0 < N; c0 += L.store_cols * kExpandGroups) {
                const bool two = L.store_cols == 32 && c0 + 16 < N;
                uint32_t r0[16], r1[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) r0[i] = r1[i] = 0u;
                if (ok) {
                    tmem_ld16_nowait(t_lane + (uint32_t)c0, r0);
                    if (two) tmem_ld16_nowait(t_lane + (uint32_t)(c0 + 16), r1);
                    tmem_wait_ld();
                }
                float* unit_out = s_out + (size_t)c0 * row_floats;
                float* unit_glu = s_glu + (size_t)c0 * 64;
                umma_epilogue_block<EPI, 16>(a, r0, s_inv, s_sum, wscale, shift, c0, seq0, block, rr, row, rblk == 1, unit_out, unit_glu, ok);
                if (two)
                    umma_epilogue_block<EPI, 16>(a, r1, s_inv, s_sum, wscale, shift, c0 + 16, seq0, block, rr, row, rblk == 1, unit_out + 16 * row_floats,
                                                 unit_glu + 16 * 64, ok);
                send(unit_out, unit_glu, two ? 32 : 16, c0);
            }
        }
        if (tid == 64) UT(8);
        if (leader) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");     // the tiles have left shared memory
        if (tid == 64) UT(9);
    }
    if (CLUSTER) cg::this_cluster().sync();                  // every peer has read this CTA's partial tile: it may exit
    if (timed_out) atomicExch(&g_umma_timeouts, 1);
    tc_fence_before();
    if (__syncthreads_or(timed_out ? 1 : 0)) {
        // A role gave up: copies it no longer waits for may still be on their way into this CTA's shared memory, and
        // MMAs it issued may still be running. Give them a bounded time (about 100 us; a copy lands within a few) before
        // the memory and the tensor-memory columns go back to the SM.
        const long long t_end = clock64() + 200000;
        while (clock64() < t_end) __nanosleep(1000);
        __syncthreads();
    }
    if (tid == 0) UTG(11);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

bool tl1_umma_applicable(const tenzo_tl1_gemv_args& a) {
    return a.batch >= kUmmaMinBatch && a.K % kKc == 0 && a.K >= kKc && a.out_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
}

// Sequences a CTA holds (a multiple of 16) and CTAs of a cluster that split one tile's K range. Fewer sequences a CTA use SMs that
// few row tiles leave idle as a split of K does, for the expansion of the weights once more a tile of sequences but without an exchange: a
// cluster's partial tiles move at some 14 bytes a cycle and SM (2560 x 2560 at 256 sequences over clusters of four: 98 KB into each
// CTA, 6900 cycles of 21000). The candidates' costs are compared in units of 10 ns: a CTA's start, its chunks, its
// sequences' epilogue, the exchange; rounds of CTAs, which overlap in part; and launching them. Clusters that do not fit the
// SMs at once (GPCs hold whole ones only) are a round more. The constants were fitted to 1049 timed pairs of quantiser and product, 16 to 1536
// sequences, 12 matrices: the choice is 0.6 % from the best of a size on average, and on none slower than what was taken before (up to
// 256 sequences a CTA and as large a cluster as the SMs hold). In us, before and now: 3840 x 2560 at 96 sequences 10.8 and 9.1, 256 14.8 and
// 11.8, 384 17.2 and 12.6; 2560 x 2560 at 256 15.2 and 12.2, 512 21.0 and 15.8; 2560 x 6912 at 256 20.5 and 18.5; 13824 x 2560 GLU at 384
// 29.7 and 26.1; 4096 x 14336 at 320 46.6 and 41.4. Up to 64 sequences a CTA holds them all and the cluster is as large as the SMs allow,
// the best within 3 % but for 3840 x 2560 at 64 (9.1; 8.6 in two tiles of sequences). TENZO_UMMA_KSPLIT = 1, 2, 4 or 8 overrides the cluster's size (measurement aid).
struct UmmaShape { int n_box, ksplit; };
static UmmaShape pick_umma_shape(int units, int n_chunks, int batch, int epilogue) {
    static const int forced = [] {
        const char* e = std::getenv("TENZO_UMMA_KSPLIT");
        const int v = e ? std::atoi(e) : 0;
        return v == 1 || v == 2 || v == 4 || v == 8 ? v : 0;
    }();
    static const int n_sm = [] {                             // (both set by one thread while others wait)
        int dev = 0, n = 0;
        return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
    }();
    if (batch <= 64) {                                       // one CTA, or the largest cluster that fits
        UmmaShape one = {(batch + 15) & ~15, 1};
        if (forced) one.ksplit = forced <= n_chunks ? forced : 1;
        else while (one.ksplit < 8 && units * one.ksplit * 2 <= n_sm && n_chunks / (one.ksplit * 2) >= 4) one.ksplit *= 2;
        return one;
    }
    UmmaShape best = {0, 1};
    float best_cost = 0.0f;
    const float per_sm = 1.0f / (float)n_sm;
    for (int tiles = (batch + kMaxN - 1) / kMaxN, last = 0;; ++tiles) {
        const int even = ((batch + tiles - 1) / tiles + 15) & ~15;
        if (even < 32) break;
        if (even == last) continue;
        last = even;
        // An odd multiple of 16 among several tiles is stored in units of 16 sequences, others in units of 32 (store_cols), by four groups of warps in
        // turn: 208 and 240 take four rounds where 224 and 256 take two, and where a unit also loads residuals or joins gate and up, a round costs more than 16
        // sequences do (us, residual and GLU, 208 and 224: 13824 x 2560 GLU at 385 sequences 28.0 and 27.5, 14208 x 5760 at 416 53.2 and 51.9, 2560 x 6912 at 1345
        // 47.5 and 46.9; 240 and 256: 14208 x 5760 at 480 61.9 and 59.5, 13824 x 2560 GLU at 1200 61.6 and 61.1, 4096 x 4096 at 960 31.7 and 32.0;
        // plain stores 14208 x 5760 at 480 46.0 and 47.9). One round more, 80 to 176, does not (176 and 192: 13824 x 2560 GLU at 673 sequences 39.5 and 39.4, 2560 x
        // 2560 at 1200 22.0 and 22.7).
        const int padded = tiles > 1 && epilogue != TENZO_EPI_STORE && (even & 31) && (even + 63) / 64 > (even + 127) / 128 + 1 ? even + 16 : even;
        const int ctas_even = units * ((batch + even - 1) / even);
        for (int k = forced ? (forced <= n_chunks ? forced : 1) : 1;; k *= 2) {
            const int n = k == 1 ? padded : even;                // (clusters store in units of four)
            const int ctas = n == even ? ctas_even : units * ((batch + n - 1) / n);
            if (!forced && k > 1 && (k > 8 || n_chunks < 4 * k || ctas * k > n_sm)) break;
            const int fit = k == 8 ? n_sm - n_sm * 3 / 16 : k == 4 ? n_sm - n_sm / 9 : n_sm;
            const float rounds = ctas * k <= fit ? 1.0f : k > 1 ? 2.0f : (float)(int)((float)(ctas + n_sm - 1) * per_sm);
            const float one = 88.0f + 26.0f * (float)((n_chunks + k - 1) / k) + 3.62f * (float)n +
                              (k > 1 ? 156.0f + 0.55f * (float)(n * (k - 1)) / (float)k : 0.0f) + (k == 8 ? 38.0f : 0.0f);
            const float cost = (0.41f + 0.59f * rounds) * one + 1.61f * (float)(ctas * k);
            if (!best.n_box || cost < best_cost) { best = {n, k}; best_cost = cost; }
            if (forced) break;
        }
        // (more CTAs than SMs already, and each tile more is a round more: a call outside a graph waits for this)
        if (even <= 32 || (best.n_box && ctas_even > 16 * n_sm)) break;
    }
    return best;
}

// a8 [batch][K] int8 in the order of act_quant_kernel's a_mma (16-byte aligned), inv [batch], sum_a [batch] already produced on `st`.
int launch_tl1_umma(const tenzo_tl1_gemv_args& a, const int8_t* a8, const float* inv, const int* sum_a, cudaStream_t st) {
    UmmaLaunch L;
    L.a = a;
    L.inv = inv;
    L.sum_a = sum_a;
    const bool glu = a.epilogue == TENZO_EPI_RELU2_GLU;
    L.units = glu ? a.n_blocks / 2 : (a.n_blocks + 1) / 2;
    const UmmaShape shape = pick_umma_shape(L.units, a.K / kKc, a.batch, a.epilogue);
    L.n_box = shape.n_box;
    L.ksplit = shape.ksplit;
    L.n_slots = UmmaSmem::a_slots_for(L.n_box);
    L.b_slots = UmmaSmem::b_slots_for(L.n_box);
    if (L.b_slots > 4) L.n_slots = L.b_slots;                      // (enough of them: requested by the warps that expand the codes, two chunks at a time)
    L.n_pgroups = UmmaSmem::pgroups_for(L.n_box);
    const int seq_tiles = (a.batch + L.n_box - 1) / L.n_box;
    // (A store is not to reach into the next tile's sequences.)
    L.store_cols = L.ksplit > 1 || L.n_box <= 32 ? 4 : L.n_box <= 64 || (seq_tiles > 1 && (L.n_box & 31)) ? 16 : 32;
    CUtensorMap amap, omap;
    // activations [batch][K] int8: B-operand tiles {128 bytes of K, n_box sequences}, 128-byte swizzle
    if (int rc = encode_2d(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, a8, (uint64_t)a.K, (uint64_t)a.batch, (uint64_t)a.K, kKc, (uint32_t)L.n_box,
                           CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    // output [batch][n_out] fp32: store units {128 (GLU: 64) rows of the weight matrix, 32, 16 or 4 sequences}
    const uint64_t n_out = (uint64_t)(glu ? a.n_blocks / 2 : a.n_blocks) * 64;
    if (int rc = encode_2d(&omap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.out, n_out, (uint64_t)a.batch, (uint64_t)a.out_stride * 4, glu ? 64u : 128u,
                           (uint32_t)L.store_cols, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
    const size_t smem = UmmaSmem::bytes(L.n_box);
    using Kernel = void (*)(const UmmaLaunch, const CUtensorMap, const CUtensorMap);
    const bool cl = L.ksplit > 1;
    Kernel kernel = a.epilogue == TENZO_EPI_RELU2_GLU   ? (cl ? tl1_umma_kernel<TENZO_EPI_RELU2_GLU, true> : tl1_umma_kernel<TENZO_EPI_RELU2_GLU, false>)
                    : a.epilogue == TENZO_EPI_RESIDUAL ? (cl ? tl1_umma_kernel<TENZO_EPI_RESIDUAL, true> : tl1_umma_kernel<TENZO_EPI_RESIDUAL, false>)
                                                       : (cl ? tl1_umma_kernel<TENZO_EPI_STORE, true> : tl1_umma_kernel<TENZO_EPI_STORE, false>);
    cudaError_t e = allow_smem(kernel, kMaxSmem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.units, (unsigned)seq_tiles, (unsigned)L.ksplit);
    cfg.blockDim = dim3(kUmmaThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (L.ksplit > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = 1;
        attr[n_attr].val.clusterDim.y = 1;
        attr[n_attr].val.clusterDim.z = (unsigned)L.ksplit;
        ++n_attr;
    }
    if (a.use_pdl) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    e = cudaLaunchKernelEx(&cfg, kernel, L, amap, omap);
    return e == cudaSuccess ? 0 : (int)e;
}


const int* tl1_umma_timeouts_flag() {
    void* p = nullptr;
    return cudaGetSymbolAddress(&p, g_umma_timeouts) == cudaSuccess ? static_cast<const int*>(p) : nullptr;
}
int tl1_umma_take_timeouts() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_umma_timeouts, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_umma_timeouts, &zero, sizeof zero);
    return v;
}

}  // namespace tz

#ifdef TZ_UMMA_CHECK
extern "C" __attribute__((visibility("default"))) int tenzo_check_umma(unsigned long long* out) {
    return (int)cudaMemcpyFromSymbol(out, tz::g_umma_check, sizeof(unsigned long long) * 4);
}
#endif
#ifdef TZ_UMMA_TRACE
extern "C" __attribute__((visibility("default"))) int tenzo_trace_umma(long long* out) {
    return (int)cudaMemcpyFromSymbol(out, tz::g_umma_trace, sizeof(long long) * 160 * 16);
}
extern "C" __attribute__((visibility("default"))) int tenzo_trace_umma_chunks(long long* out) {
    return (int)cudaMemcpyFromSymbol(out, tz::g_umma_chunks, sizeof(long long) * 64 * 8);
}
#endif

extern "C" int tenzo_cuda_tl1_gemm_layout(int batch, int* slots, int* weight_groups, size_t* smem_bytes, size_t* epilogue_bytes) {
    if (batch < tz::kUmmaMinBatch) return -1;                    // the tensor-core path does not apply
    const int per_cta = batch < tz::kMaxN ? batch : tz::kMaxN, n_box = (per_cta + 15) & ~15;
    if (slots) *slots = tz::UmmaSmem::b_slots_for(n_box);
    if (weight_groups) *weight_groups = tz::UmmaSmem::pgroups_for(n_box);
    if (smem_bytes) *smem_bytes = tz::UmmaSmem::bytes(n_box);
    // without a cluster: the output columns [n_box][128] fp32 (GLU: [n_box][64] twice); with one: behind the partial tile
    // [n_box][128] int32, the columns of the units a rank owns (at most every other four sequences)
    if (epilogue_bytes) *epilogue_bytes = (size_t)n_box * 512 + (size_t)4 * ((n_box / 4 + 1) / 2) * 512;
    return 0;
}

static tz::UmmaShape gemm_shape(int n_blocks, int K, int batch, int epilogue) {
    if (n_blocks <= 0 || K < tz::kKc || K % tz::kKc || batch < tz::kUmmaMinBatch) return {0, 0};       // the tensor-core path does not apply
    const int units = epilogue == TENZO_EPI_RELU2_GLU ? n_blocks / 2 : (n_blocks + 1) / 2;
    return tz::pick_umma_shape(units, K / tz::kKc, batch, epilogue);
}
extern "C" int tenzo_cuda_tl1_gemm_ksplit(int n_blocks, int K, int batch, int epilogue) { return gemm_shape(n_blocks, K, batch, epilogue).ksplit; }
extern "C" int tenzo_cuda_tl1_gemm_sequences(int n_blocks, int K, int batch, int epilogue) { return gemm_shape(n_blocks, K, batch, epilogue).n_box; }
