// What the prefill kernels share: wrappers of the TMA, tcgen05 and tensor-memory instructions, matrix
// fragment loads, and the encoding of tensor maps.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "mb_device.cuh"

namespace mb {
namespace prefill {

constexpr int kTileK = 64;  // bf16 elements = one 128-byte swizzle row

__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Two floats to a bf16 pair in one instruction (same bits as two cvt.rn.bf16.f32, checked over
// every finite float): the attention's softmax warps and the GEMM epilogue are bound by the
// instructions they issue, and packing was four of them per pair.
__device__ __forceinline__ unsigned int pack_bf16_pair(float lo, float hi) {
    unsigned int packed;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(hi), "f"(lo));
    return packed;
}

// ---------------------------------------------------------------------------------------
// tcgen05 / TMA wrappers
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst_smem, const CUtensorMap* map, int x, int y,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst_smem)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
// A wait of the whole warp, whose result the compiler knows to be the same in all lanes.
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long* bar, unsigned int parity,
                                               volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abort_flag)) != 0;
}
__device__ __forceinline__ void tma_load_blocks(void* dst_smem, const CUtensorMap* map, int row, int block,
                                                unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst_smem)),
        "l"(map), "r"(0), "r"(row), "r"(block), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_heads(void* dst_smem, const CUtensorMap* map, int row, int half, int head,
                                               int block, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_u32(dst_smem)),
        "l"(map), "r"(0), "r"(row), "r"(half), "r"(head), "r"(block), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(unsigned int* slot_smem, unsigned int columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(slot_smem)),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned int base, unsigned int columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// The mbarrier gets one arrival once every tcgen05.mma this thread issued before has finished.
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}
// D[tmem] (+)= A[smem] . B[smem]^T, bf16 operands, fp32 accumulate, M = 64 or 128 (idesc).
__device__ __forceinline__ void umma_bf16(unsigned int tmem_d, unsigned long long desc_a,
                                          unsigned long long desc_b, unsigned int idesc,
                                          unsigned int accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Shared-memory operand descriptor: K-major tile of 128-byte rows, 128-byte swizzle, groups of
// 8 rows 1024 bytes apart (the layout TMA writes with CU_TENSOR_MAP_SWIZZLE_128B).
__device__ __forceinline__ unsigned long long umma_desc(unsigned int smem_addr) {
    unsigned long long d = 0;
    d |= static_cast<unsigned long long>((smem_addr & 0x3ffffu) >> 4);  // start address
    d |= 1ull << 16;                                                     // leading byte offset (unused)
    d |= static_cast<unsigned long long>(1024 >> 4) << 32;               // stride byte offset
    d |= 1ull << 46;                                                     // descriptor version
    d |= 2ull << 61;                                                     // SWIZZLE_128B
    return d;
}
// 32 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_load32(unsigned int taddr, float (&v)[32]) {
    unsigned int r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_load16(unsigned int taddr, float (&v)[16]) {
    unsigned int r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void ldmatrix_x4(unsigned int (&r)[4], const void* smem_ptr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(smem_ptr)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned int (&r)[4], const void* smem_ptr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(smem_ptr)));
}
__device__ __forceinline__ void cp_async_16(void* dst_smem, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)), "l"(src)
                 : "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) ==
                cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// [rows, K] bf16 row-major, boxes of `box_rows` x 64 elements, 128-byte swizzle, zero fill
// outside the tensor.
inline bool make_map(CUtensorMap* map, unsigned long long base, int rows, int K, int box_rows) {
    EncodeTiledFn fn = encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kTileK), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, reinterpret_cast<void*>(base), dims,
              strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same matrix as [K / 64] blocks of [rows, 64], K a multiple of 64: one copy brings `blocks` of them, one
// after the other.
inline bool make_block_map(CUtensorMap* map, unsigned long long base, int rows, int K, int box_rows, int blocks) {
    EncodeTiledFn fn = encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {kTileK, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(K / kTileK)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(K) * 2, kTileK * 2};
    const cuuint32_t box[3] = {kTileK, static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(blocks)};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, reinterpret_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A projection to heads, [heads, 2, D / 2, K]: boxes of `box_rows` rows out of one half of the head dimension, of
// several heads where box_rows is a multiple of D / 2.
inline bool make_head_map(CUtensorMap* map, unsigned long long base, int heads, int D, int K, int box_rows,
                          int blocks) {
    EncodeTiledFn fn = encode_tiled();
    if (fn == nullptr) return false;
    const int half = D / 2, in_half = box_rows < half ? box_rows : half;
    const cuuint64_t dims[5] = {kTileK, static_cast<cuuint64_t>(half), 2, static_cast<cuuint64_t>(heads),
                                static_cast<cuuint64_t>(K / kTileK)};
    const cuuint64_t row = static_cast<cuuint64_t>(K) * 2;
    const cuuint64_t strides[4] = {row, row * half, row * D, kTileK * 2};
    const cuuint32_t box[5] = {kTileK, static_cast<cuuint32_t>(in_half), 1, static_cast<cuuint32_t>(box_rows / in_half),
                               static_cast<cuuint32_t>(blocks)};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, reinterpret_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace prefill
}  // namespace mb
