// What the tcgen05 kernels share: tile constants, descriptors, TMA tile loads,
// fences, and the host's tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "tma_pipe.cuh"

namespace mbem {

constexpr int TC_BM = 128;            // rows per CTA (the MMA's M)
constexpr int TC_BK = 64;             // K per stage: one 128-byte swizzle row of BF16
constexpr int TC_STAGES = 4;
constexpr int TC_THREADS = 192;
constexpr uint32_t TC_WAIT_LIMIT = 1u << 24;

// tcgen05 shared-memory matrix descriptor, K-major operand with 128-byte
// swizzle: start address, leading-dimension offset (unused for this layout),
// stride between 8-row groups (1024 bytes), descriptor version 1, swizzle
// mode 2 (128B).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(16u >> 4) << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t f16_idesc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_addr(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// BF16 row-major (rows x cols) at ld elements, box (64 cols x box_rows), 128B
// swizzle (tc_gemm.cu; the encoder is looked up on first use)
int tc_make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_rows);
// the same with a box of 32 columns and the 64B swizzle
int tc_make_map32(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_rows);
// the device flag that a tensor-core wait that ran out sets (tc_gemm_check)
int* tc_error_flag();

}  // namespace mbem
