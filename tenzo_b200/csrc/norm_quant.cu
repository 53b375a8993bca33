// Standalone fused RMSNorm + per-token absmax quantiser (both flavours the reference uses).
//
// qmax = 31 : the quantiser half of build_lut — floor 1e-6, q = round(y*(31/m)), scale m/31
//             (src/runtime/TenzoEngine.cpp:27-42 of the reference).
// qmax = 127: compute_logits' quantiser — floor 1e-8, s = amax/127, q = clamp(round(y*(1/s)))
//             (:1666-1678).
// The GEMV and LM-head kernels carry the same code in their prologues; this entry exists for the
// backend class's executeRMSNorm and for checking the quantiser on its own.
#include "common.cuh"
#include "attn_common.cuh"
#include "../../include/tenzo_kernels.h"

namespace tz {

constexpr int kNqThreads = 256;

__global__ void __launch_bounds__(kNqThreads) rmsnorm_quant_kernel(
    const float* __restrict__ x, const float* __restrict__ norm_w, int do_norm, float eps, int dim, int qmax,
    int x_stride, float* y_out, int8_t* q_out, float* scale_out) {
    extern __shared__ float s_y[];            // dim floats + 32 scratch
    float* s_f = s_y + dim;
    const int tid = threadIdx.x, seq = blockIdx.x;
    const float* xs = x + (size_t)seq * x_stride;

    for (int i = tid; i < dim; i += kNqThreads) s_y[i] = xs[i];
    float m = 0.0f;
    if (do_norm) {
        __syncthreads();
        const float ss = sumsq_reference_order(s_y, dim, s_f);
        const float inv_rms = rms_inv(ss, dim, eps);
        for (int i = tid; i < dim; i += kNqThreads) {
            const float y = rms_apply(s_y[i], inv_rms, norm_w, i);
            s_y[i] = y;
            m = fmaxf(m, fabsf(y));
        }
    } else {
        for (int i = tid; i < dim; i += kNqThreads) m = fmaxf(m, fabsf(s_y[i]));
    }
    if (y_out)
        for (int i = tid; i < dim; i += kNqThreads) y_out[(size_t)seq * dim + i] = s_y[i];
    if (!q_out && !scale_out) return;
    m = block_max_nonneg(m, s_f);      // m: running maximum of |y| from 0
    if (qmax == 31) {
        m = fmaxf(m, 1e-6f);
        const float to_q = 31.0f / m;
        if (q_out)
            for (int i = tid; i < dim; i += kNqThreads)
                q_out[(size_t)seq * dim + i] = (int8_t)(int)roundf(s_y[i] * to_q);
        if (scale_out && tid == 0) scale_out[seq] = m / 31.0f;
    } else {
        m = fmaxf(m, 1e-8f);
        const float s = m / 127.0f, inv = 1.0f / s;
        if (q_out)
            for (int i = tid; i < dim; i += kNqThreads)
                q_out[(size_t)seq * dim + i] = (int8_t)(int)fminf(fmaxf(roundf(s_y[i] * inv), -128.0f), 127.0f);
        if (scale_out && tid == 0) scale_out[seq] = s;
    }
}

// Batched front half of the TL1 GEMM: per sequence RMSNorm + absmax(31) quantiser, written as the
// packed tensor-core B fragments tl1_mma_kernel consumes: words[seq][set][t][0] holds 4*a for the
// even columns of column pairs 16*set + 4*i + t (byte i = 0..3), words[seq][set][t][1] the odd
// columns unscaled; columns beyond K are zero. inv[seq] = max|y|/31. `words` may be null (tensor-core GEMM
// path: it takes the int8 matrix a_mma [batch][K] and sum_out[seq] = sum_k a_k instead). a_out, where asked for: the plain
// int8 matrix.
#ifdef TZ_AQ_TRACE
__device__ long long g_aq_trace[8];
#define AQT(i) do { if (blockIdx.x == 0 && threadIdx.x == 0) g_aq_trace[i] = clock64(); } while (0)
#else
#define AQT(i) ((void)0)
#endif

// Row stride of the squares in chain-major order: a chain of K/8 a row, the rows of elements 4i .. 4i + 3 and of their
// neighbours' in different banks.
__host__ __device__ __forceinline__ int squares_stride(int K) { return (((K >> 3) + 3) & ~3) + 4; }

// a_mma: every four elements 4i .. 4i + 3 are one word, the even ones times four (124 at most) in its lower half and the odd ones
// in its upper half, for words i with bit 1 set in reversed order, and words i with bit 2 set change places in pairs:
// the order in which tl1_umma_kernel's expanding threads come by the codes.
__device__ __forceinline__ uint32_t mma_word(int i, int q0, int q1, int q2, int q3) {
    const uint32_t b0 = (uint8_t)(4 * q0), b1 = (uint8_t)(4 * q2), b2 = (uint8_t)q1, b3 = (uint8_t)q3;
    return (i >> 1) & 1 ? b1 | b0 << 8 | b3 << 16 | b2 << 24 : b0 | b1 << 8 | b2 << 16 | b3 << 24;
}
__device__ __forceinline__ int mma_place(int i) { return i ^ ((i >> 2) & 1); }

// A thread holds kAqVec 16-byte pieces of the row in registers (launch_act_quant picks threads and pieces by K; longer rows
// go through shared memory).
// kAqResident: CTAs an SM must hold. With one the norm's weights are loaded ahead of the wait for the previous
// kernel and held in registers as well, for the latency of few rows; with more they are loaded when they are used.
template <int kAqThreads, int kAqVec, int kAqResident>
__global__ void __launch_bounds__(kAqThreads, kAqResident) act_quant_kernel(
    const float* x, const float* __restrict__ norm_w, int do_norm, float eps, int K, int x_stride,
    uint32_t* words, float* inv, int8_t* a_out, int8_t* a_mma, int* sum_out, int use_pdl) {
    extern __shared__ __align__(16) float s_y[];   // K floats (or eight padded rows of K/8 squares) + 32 scratch
    const int stride = squares_stride(K);
    float* s_f = s_y + (8 * stride > K ? 8 * stride : K);
    const int tid = threadIdx.x, seq = blockIdx.x;
    AQT(0);
    const float* xs = x + (size_t)seq * x_stride;
    // The whole row in registers as 16-byte loads, all in flight at once; shared memory is only touched where another
    // thread needs the value (the sum of squares in reference order, the packed fragments of the mma.sync path), instead
    // of four passes over a staged copy.
    const bool vec = (K & 3) == 0 && K <= 4 * kAqVec * kAqThreads && (x_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                     (!norm_w || (reinterpret_cast<uintptr_t>(norm_w) & 15) == 0) && (!a_out || (reinterpret_cast<uintptr_t>(a_out) & 3) == 0);
    if (vec) {
        const int k4 = K >> 2;
        float4 w4[kAqVec], v[kAqVec];
        const bool has_w = do_norm && norm_w;
        if (kAqResident == 1 && has_w) {                // model constants: no need to wait for the previous kernel
#pragma unroll
            for (int r = 0; r < kAqVec; ++r) {
                const int i = tid + r * kAqThreads;
                w4[r] = i < k4 ? __ldg(reinterpret_cast<const float4*>(norm_w) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        // Chains of whole 16-byte pieces. For the other multiples of eight they gain nothing: the elements behind the last piece are
        // added load by load (quantiser and product of 128 rows, in place and by chains: K = 2568 8.66 and 8.74 us at two sequences,
        // 21.1 and 21.3 at 256; K = 6920 11.40 and 11.19, 28.37 and 28.30; K = 14344 17.53 and 17.51, 45.77 and 45.82).
        const bool chains = (K & 31) == 0;
        // The GEMM that consumes this kernel's output starts now: its prologue (tensor-memory allocation, the first weight
        // copies, expanding the first chunks) takes as long as the rest of this kernel; it waits for this grid before it
        // touches the activations. Not before this kernel's own wait: kernels further down the chain would come in as well
        // and take the places of the ones whose turn it is (12 sequences, 4 steps: 11.04 ms, with both triggers here 10.70).
        if (use_pdl) {
            pdl_wait();
            pdl_launch_dependents();
        }
        AQT(1);
#pragma unroll
        for (int r = 0; r < kAqVec; ++r) {
            const int i = tid + r * kAqThreads;
            v[r] = i < k4 ? __ldcg(reinterpret_cast<const float4*>(xs) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float m = 0.0f;
        if (do_norm) {
            float ss;
            if (chains) {
                // squares chain-major (element e in row e & 7, column e >> 3); a lane a chain
#pragma unroll
                for (int r = 0; r < kAqVec; ++r) {
                    const int i = tid + r * kAqThreads;
                    if (i < k4) {
                        float* d = s_y + (4 * (i & 1)) * stride + (i >> 1);      // element 4i + c: row (4i + c) & 7, column (4i + c) >> 3
                        d[0] = __fmul_rn(v[r].x, v[r].x);
                        d[stride] = __fmul_rn(v[r].y, v[r].y);
                        d[2 * stride] = __fmul_rn(v[r].z, v[r].z);
                        d[3 * stride] = __fmul_rn(v[r].w, v[r].w);
                    }
                }
                __syncthreads();
                AQT(2);
                if (tid < 8) s_f[tid] = sequential_sum(s_y + tid * stride, K >> 3);
                __syncthreads();
                ss = s_f[0];
#pragma unroll
                for (int j = 1; j < 8; ++j) ss = __fadd_rn(ss, s_f[j]);        // lanes added left to right, from lane 0
            } else {
#pragma unroll
                for (int r = 0; r < kAqVec; ++r) {
                    const int i = tid + r * kAqThreads;
                    if (i < k4) reinterpret_cast<float4*>(s_y)[i] = v[r];
                }
                __syncthreads();
                AQT(2);
                ss = sumsq_reference_order(s_y, K, s_f);
            }
            AQT(3);
            const float inv_rms = rms_inv(ss, K, eps);
#pragma unroll
            for (int r = 0; r < kAqVec; ++r) {          // y = (x * inv_rms) * w, left to right (rms_apply)
                v[r].x *= inv_rms; v[r].y *= inv_rms; v[r].z *= inv_rms; v[r].w *= inv_rms;
                if (kAqResident > 1 && has_w) {
                    const int i = tid + r * kAqThreads;
                    w4[r] = i < k4 ? __ldg(reinterpret_cast<const float4*>(norm_w) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                if (has_w) { v[r].x *= w4[r].x; v[r].y *= w4[r].y; v[r].z *= w4[r].z; v[r].w *= w4[r].w; }
            }
        }
#pragma unroll
        for (int r = 0; r < kAqVec; ++r) m = fmaxf(fmaxf(m, fmaxf(fabsf(v[r].x), fabsf(v[r].y))), fmaxf(fabsf(v[r].z), fabsf(v[r].w)));
        int* s_i = reinterpret_cast<int*>(s_f + 31);
        if (tid == 0) *s_i = 0;                          // (the maximum's barriers come before the sum)
        m = fmaxf(block_max_nonneg(m, s_f), 1e-6f);      // TenzoEngine.cpp:28-32
        AQT(4);
        const float to_q = 31.0f / m;             // :34
        if (tid == 0) inv[seq] = m / 31.0f;       // :35
        if (words) {                              // the packed fragments gather arbitrary columns: through shared memory
            __syncthreads();
#pragma unroll
            for (int r = 0; r < kAqVec; ++r) {
                const int i = tid + r * kAqThreads;
                if (i < k4) reinterpret_cast<float4*>(s_y)[i] = v[r];
            }
            __syncthreads();
            const int nsets = ((K >> 1) + 15) / 16;
            for (int wd = tid; wd < nsets * 8; wd += kAqThreads) {
                const int s = wd >> 3, tt = (wd >> 1) & 3, odd = wd & 1;
                uint32_t word = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int col = 2 * (16 * s + 4 * i + tt) + odd;
                    const int q = col < K ? (int)roundf(s_y[col] * to_q) : 0;   // :41-42
                    word |= (uint32_t)(uint8_t)(int8_t)(odd ? q : 4 * q) << (8 * i);
                }
                words[(size_t)seq * nsets * 8 + wd] = word;
            }
        }
        if (a_out || a_mma || sum_out) {
            int part = 0;
#pragma unroll
            for (int r = 0; r < kAqVec; ++r) {
                const int i = tid + r * kAqThreads;
                const int q0 = (int)roundf(v[r].x * to_q), q1 = (int)roundf(v[r].y * to_q), q2 = (int)roundf(v[r].z * to_q), q3 = (int)roundf(v[r].w * to_q);
                if (i < k4) {
                    if (a_out)
                        reinterpret_cast<uint32_t*>(a_out + (size_t)seq * K)[i] =
                            (uint32_t)(uint8_t)(int8_t)q0 | ((uint32_t)(uint8_t)(int8_t)q1 << 8) | ((uint32_t)(uint8_t)(int8_t)q2 << 16) | ((uint32_t)(uint8_t)(int8_t)q3 << 24);
                    if (a_mma) reinterpret_cast<uint32_t*>(a_mma + (size_t)seq * K)[mma_place(i)] = mma_word(i, q0, q1, q2, q3);
                    part += q0 + q1 + q2 + q3;
                }
            }
            if (sum_out) {                        // sum_k a_k, for kernels that multiply by the unsigned codes w+1
                part = __reduce_add_sync(0xffffffffu, part);
                if ((tid & 31) == 0) atomicAdd(s_i, part);
                __syncthreads();
                if (tid == 0) sum_out[seq] = *s_i;
            }
        }
        AQT(5);
        return;
    }
    // rows that are longer, or not aligned for 16-byte loads: element by element through shared memory
    if (use_pdl) pdl_wait();
    for (int i = tid; i < K; i += kAqThreads) s_y[i] = __ldcg(xs + i);
    __syncthreads();
    float m = 0.0f;
    if (do_norm) {
        const float ss = sumsq_reference_order(s_y, K, s_f);
        const float inv_rms = rms_inv(ss, K, eps);
        for (int i = tid; i < K; i += kAqThreads) {
            const float y = rms_apply(s_y[i], inv_rms, norm_w, i);
            s_y[i] = y;
            m = fmaxf(m, fabsf(y));
        }
    } else {
        for (int i = tid; i < K; i += kAqThreads) m = fmaxf(m, fabsf(s_y[i]));
    }
    m = fmaxf(block_max_nonneg(m, s_f), 1e-6f);      // TenzoEngine.cpp:28-32
    const float to_q = 31.0f / m;             // :34
    const int nsets = ((K >> 1) + 15) / 16;
    for (int wd = tid; words && wd < nsets * 8; wd += kAqThreads) {
        const int s = wd >> 3, tt = (wd >> 1) & 3, odd = wd & 1;
        uint32_t word = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int col = 2 * (16 * s + 4 * i + tt) + odd;
            const int q = col < K ? (int)roundf(s_y[col] * to_q) : 0;   // :41-42
            word |= (uint32_t)(uint8_t)(int8_t)(odd ? q : 4 * q) << (8 * i);
        }
        words[(size_t)seq * nsets * 8 + wd] = word;
    }
    if (tid == 0) inv[seq] = m / 31.0f;       // :35
    if (a_out || sum_out) {
        int part = 0;
        for (int i = tid; i < K; i += kAqThreads) {
            const int q = (int)roundf(s_y[i] * to_q);
            if (a_out) a_out[(size_t)seq * K + i] = (int8_t)q;
            part += q;
        }
        for (int i = tid; a_mma && i < K >> 2; i += kAqThreads) {
            const float* y = s_y + 4 * i;
            reinterpret_cast<uint32_t*>(a_mma + (size_t)seq * K)[mma_place(i)] =
                mma_word(i, (int)roundf(y[0] * to_q), (int)roundf(y[1] * to_q), (int)roundf(y[2] * to_q), (int)roundf(y[3] * to_q));
        }
        if (sum_out) {                        // sum_k a_k, for kernels that multiply by the unsigned codes w+1
            int* s_i = reinterpret_cast<int*>(s_f);
            __syncthreads();
            if (tid == 0) s_i[0] = 0;
            __syncthreads();
            part = __reduce_add_sync(0xffffffffu, part);
            if ((tid & 31) == 0) atomicAdd(&s_i[0], part);
            __syncthreads();
            if (tid == 0) sum_out[seq] = s_i[0];
        }
    }
}

cudaError_t launch_act_quant(const float* x, const float* norm_w, int do_norm, float eps, int K, int batch, int x_stride,
                             uint32_t* words, float* inv, int8_t* a_out, int8_t* a_mma, int* sum_out, int use_pdl, cudaStream_t st) {
    const int rows = 8 * squares_stride(K);
    const size_t smem = (size_t)((rows > K ? rows : K) + 32) * sizeof(float);
    // 16-byte pieces a thread: as few as the row needs (registers: 1536 rows of 2560 in 21 us with seven, 13 with three), 512
    // threads for rows above 7168 (14336 went through shared memory element by element: 17 us, now 10)
    // From 4097 elements on the registers with the weights leave room for two CTAs an SM (one of 512 threads), and more rows than that
    // would come in rounds of a chain of additions each: then twice as many without them (1536 rows: 6912 elements 31.0 -> 22.0 us, 14336 92.7 -> 62.5;
    // 512 rows 11.3 -> 9.4 and 32.3 -> 21.2; at 256 rows of 6912 no difference; shorter rows gain nothing: 512 of 2560 4.8 -> 5.6).
    const bool many = batch > 148 * (K <= 7168 ? 2 : 1);
    auto kernel = K <= 3072   ? act_quant_kernel<256, 3, 1>
                  : K <= 4096 ? act_quant_kernel<256, 4, 1>
                  : K <= 7168 ? (many ? act_quant_kernel<256, 7, 4> : act_quant_kernel<256, 7, 1>)
                              : (many ? act_quant_kernel<512, 7, 2> : act_quant_kernel<512, 7, 1>);
    const int threads = K <= 7168 ? 256 : 512;
    if (smem > 48 * 1024) {
        cudaError_t ea = allow_smem(kernel, 96 * 1024);
        if (ea != cudaSuccess) return ea;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)batch, 1, 1);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, x, norm_w, do_norm, eps, K, x_stride, words, inv, a_out, a_mma, sum_out, use_pdl);
}

}  // namespace tz

#ifdef TZ_AQ_TRACE
extern "C" __attribute__((visibility("default"))) int tenzo_trace_act_quant(long long* out) {
    return (int)cudaMemcpyFromSymbol(out, tz::g_aq_trace, sizeof(long long) * 8);
}
#endif

extern "C" int tenzo_cuda_rmsnorm_quant(const float* x, const float* norm_w, int do_norm, float eps, int dim,
                                        int qmax, int batch, int x_stride, float* y_out, int8_t* q_out,
                                        float* scale_out, void* stream) {
    if (!x || dim <= 0 || batch <= 0 || (qmax != 31 && qmax != 127)) return -1;
    if (dim > 16384) return -5;
    const size_t smem = (size_t)(dim + 32) * sizeof(float);
    if (smem > 48 * 1024) {
        cudaError_t ea = tz::allow_smem(tz::rmsnorm_quant_kernel, 80 * 1024);
        if (ea != cudaSuccess) return (int)ea;
    }
    tz::rmsnorm_quant_kernel<<<batch, tz::kNqThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        x, norm_w, do_norm, eps, dim, qmax, x_stride, y_out, q_out, scale_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}
