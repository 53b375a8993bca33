// Pieces shared by the tcgen05 kernels (tl1_umma.cu, lm_head_umma.cu) and, the last, by the attention kernels: mbarrier / proxy / tensor-memory
// helpers, the shared-memory operand descriptor for K-major tiles with the 128-byte swizzle, the
// kind::i8 MMA issue, and the host-side tensor-map encoder (driver entry point fetched through the
// runtime, so the library does not link against libcuda).
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace tz {

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar)) : "memory");
}
// K-major operand tile, 128-byte swizzle: rows 128 bytes apart, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// The same MMA with the A operand (M x K, one row per lane, four K-bytes per 32-bit column) read from tensor memory:
// only B crosses shared memory, which is what bounds the shared-memory form (measured, M128 K32: 169 cycles at N = 256
// and 94 at N <= 64 with both operands in shared memory; 129 and 47 with A in tensor memory).
__device__ __forceinline__ void umma_i8_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// Sixteen lanes x 32 columns from sixteen registers per thread. Thread T = 4g + t holds, in register 4n + 2u + w, the
// cell (lane g + 8u, column 8n + 2t + w) of the window that starts at taddr (checked against the hardware by writing
// thread and register numbers and reading them back with the 32x32b shape).
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// Zeros in 16 columns of the warp's 32 lanes.
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(0u) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Tensor maps through the driver entry point, fetched once by way of the runtime.
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static inline TensorMapEncodeFn tensor_map_encoder() {
    static const TensorMapEncodeFn encode = []() -> TensorMapEncodeFn {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) return nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(fn);
    }();
    return encode;
}

// One tensor map of `rank` dimensions. The encoder wants a current context, and a host thread that has made no runtime call
// yet has none: cudaSetDevice makes the device's primary context the thread's (also while a stream is captured).
static inline int encode_tensor_map(CUtensorMap* out, CUtensorMapDataType type, cuuint32_t rank, const void* base, const cuuint64_t* dims,
                                    const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (!encode) return -4;
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    auto run = [&] {
        return encode(out, type, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    if (run() == CUDA_SUCCESS) return 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) return -4;
    return run() == CUDA_SUCCESS ? 0 : -4;
}

// 2-D row-major tensor map: `inner` elements per row, `rows` rows `row_stride_bytes` apart, box {box_inner, box_rows}.
static inline int encode_2d(CUtensorMap* out, CUtensorMapDataType type, const void* base, uint64_t inner, uint64_t rows, uint64_t row_stride_bytes,
                     uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows};
    return encode_tensor_map(out, type, 2, base, dims, strides, box, swizzle);
}

// 3-D byte tensor {inner, rows, planes}, rows `inner` bytes apart, planes `plane_stride` bytes apart, box {box_inner, box_rows, 1}.
static inline int encode_3d_bytes(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint64_t planes, uint64_t plane_stride,
                                  uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
    const cuuint64_t dims[3] = {inner, rows, planes};
    const cuuint64_t strides[2] = {inner, plane_stride};
    const cuuint32_t box[3] = {box_inner, box_rows, 1u};
    return encode_tensor_map(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, swizzle);
}

}  // namespace tz
