// The block solver's product with the three-term BF16 split on the tensor cores
// (sm_103a): Y^T = (A_hi X_hi + A_hi X_lo + A_lo X_hi)^T for up to 256 right-hand
// sides, as partial sums.
//
// A plain GEMM over the three-fold K (tc_gemm.cu) loads A_hi and X_hi twice: 48 KB
// of operands for every four MMAs, and the copies into shared memory bound it (113
// bytes a clock an SM, 0.62 of the tensor pipe). Here a stage holds 32 columns of
// all four panels (48 KB) for six MMAs, two thirds of the traffic. The (row tile,
// K block) units are dealt to the SMs in equal runs, so no SM waits for a last
// wave; a run's pieces of a tile go to partial sums that the Arnoldi step adds in
// order, and a second TMEM accumulator takes the next 16 units while the epilogue
// adds the first in registers. 20,736 x 20,736 x 256, three terms: 0.47 ms against 0.56.
#include <algorithm>

#include "tc_common.cuh"

namespace mbem {

constexpr int B3_BK = 32;                // 64-byte rows, 64-byte swizzle
constexpr int B3_STAGES = 4;
constexpr int B3_THREADS = 320;         // eight epilogue warps, producer, issuer
// Units that an accumulator takes: 512 columns, 96 MMA steps. The tensor core's FP32 sums
// come out low, so their error grows with the steps: over whole tiles (3,888 steps at
// 20,736 columns) 1.8e-7 rms and -4.4e-5 of the sum on average for a block of slip
// patterns, 0.57e-7 and -1.4e-5 with the K split of tc_gemm.cu, 0.07e-7 and -1.8e-6 with
// the pieces' sums rounded to nearest (the three terms alone: 1.4e-8). No slower.
constexpr int B3_CHUNK = 16;

// as sw128_desc for 64-byte rows: 512 bytes between 8-row groups, swizzle mode 4 (64B)
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(16u >> 4) << 16;
    d |= (uint64_t)(512u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

struct B3Maps {
    CUtensorMap a_hi, a_lo, x_hi, x_lo;
};

template <int BN>
__global__ void __launch_bounds__(B3_THREADS, 1)
tc_block3_kernel(const __grid_constant__ B3Maps maps, int64_t M, int kb, int per, int total, int n_rhs,
                 float* __restrict__ P, int* __restrict__ error) {
    constexpr int A_BYTES = TC_BM * B3_BK * 2, B_BYTES = BN * B3_BK * 2, STAGE = 2 * (A_BYTES + B_BYTES);
    constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
    constexpr int COLS = BN < 32 ? BN : BN / 2, EPI = 4 * BN / COLS;     // columns an epilogue warp, epilogue warps
    extern __shared__ __align__(1024) uint8_t b3_smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)b3_smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[B3_STAGES], empty[B3_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u0 = (int)blockIdx.x * per, u1 = min(u0 + per, total);
    if (threadIdx.x == 0) {
        for (int s = 0; s < B3_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], EPI);
        }
        mbar_init_fence();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;

    if (warp == 8 && lane == 0) {
        for (int u = u0; u < u1; u++) {
            const uint32_t g = (uint32_t)(u - u0);
            const int s = g % B3_STAGES;
            if (!mbar_wait(&empty[s], ((g / B3_STAGES) & 1u) ^ 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
            uint8_t* st = smem + s * STAGE;
            const int x = (u % kb) * B3_BK, y = (u / kb) * TC_BM;
            mbar_arrive_expect_tx(&full[s], STAGE);
            tma_load_2d(st, &maps.a_hi, x, y, &full[s]);
            tma_load_2d(st + 2 * A_BYTES, &maps.x_hi, x, 0, &full[s]);
            tma_load_2d(st + A_BYTES, &maps.a_lo, x, y, &full[s]);
            tma_load_2d(st + 2 * A_BYTES + B_BYTES, &maps.x_lo, x, 0, &full[s]);
        }
        // the last copies have landed before the CTA can end
        const uint32_t n = (uint32_t)(u1 - u0);
        for (uint32_t h = n > B3_STAGES ? n - B3_STAGES : 0; h < n; h++)
            if (!mbar_wait(&full[h % B3_STAGES], (h / B3_STAGES) & 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
    } else if (warp == 9 && lane == 0) {
        constexpr uint32_t idesc = f16_idesc(TC_BM, BN);
        uint32_t c = 0;
        int in = 0;
        for (int u = u0; u < u1; u++) {
            const uint32_t g = (uint32_t)(u - u0);
            // an accumulator takes B3_CHUNK units from the run's first of the tile on
            if (u % kb == 0) in = 0;
            const bool first = in == 0, last = in == B3_CHUNK - 1 || u == u1 - 1 || (u + 1) % kb == 0;
            in = last ? 0 : in + 1;
            const uint32_t d = tmem + (c & 1u) * BN;
            if (first) {
                if (!mbar_wait(&acc_empty[c & 1u], ((c >> 1) & 1u) ^ 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
                tc_fence_after();
            }
            const int s = g % B3_STAGES;
            if (!mbar_wait(&full[s], (g / B3_STAGES) & 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
            tc_fence_after();
            const uint32_t a0 = smem_addr(smem + s * STAGE), b0 = a0 + 2 * A_BYTES;
#pragma unroll
            for (int t = 0; t < 3; t++) {          // hi hi, hi lo, lo hi
                const uint32_t at = a0 + (t == 2 ? A_BYTES : 0), bt = b0 + (t == 1 ? B_BYTES : 0);
#pragma unroll
                for (int k = 0; k < B3_BK / 16; k++) {
                    const uint64_t ad = sw64_desc(at + k * 32), bd = sw64_desc(bt + k * 32);
                    const uint32_t add = (!first || t > 0 || k > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                        "l"(ad), "l"(bd), "r"(idesc), "r"(add)
                        : "memory");
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_addr(&empty[s]))
                         : "memory");
            if (last) {
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_addr(&acc_full[c & 1u]))
                             : "memory");
                c++;
            }
        }
    } else if (warp < EPI) {
        // warp w: TMEM lanes 32 (w % 4) .., columns (w / 4) COLS ..
        const int col0 = (warp >> 2) * COLS;
        const uint32_t ta = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)col0;
        uint32_t c = 0;
        for (int u = u0; u < u1;) {
            const int tile = u / kb, end = min(u1, (tile + 1) * kb);
            const int part = (int)blockIdx.x - tile * kb / per;      // this run's place among the tile's
            float acc[COLS];
#pragma unroll
            for (int i = 0; i < COLS; i++) acc[i] = 0.0f;
#pragma unroll 1
            for (; u < end; u += B3_CHUNK, c++) {
                if (!mbar_wait(&acc_full[c & 1u], (c >> 1) & 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
                tc_fence_after();
#pragma unroll
                for (int q = 0; q < COLS; q += 16) {
                    uint32_t v[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                        "%12, %13, %14, %15}, [%16];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                          "=r"(v[14]), "=r"(v[15])
                        : "r"(ta + (c & 1u) * BN + (uint32_t)q));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; i++) acc[q + i] += __uint_as_float(v[i]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[c & 1u]);
            }
            u = end;
            const int64_t row = (int64_t)tile * TC_BM + 32 * (warp & 3) + lane;
            if (row < M) {
                float* out = P + ((int64_t)part * n_rhs + col0) * M + row;
#pragma unroll
                for (int i = 0; i < COLS; i++)
                    if (col0 + i < n_rhs) out[(int64_t)i * M] = acc[i];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        // every MMA has completed: the epilogue has read each accumulator
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

template <int BN>
static int launch_block3(const B3Maps& maps, int64_t M, int kb, int per, int total, int n_rhs, float* P, int* err,
                         cudaStream_t st) {
    const size_t smem = (size_t)B3_STAGES * 2 * (TC_BM + BN) * B3_BK * 2 + 1024;
    cudaFuncSetAttribute(tc_block3_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    tc_block3_kernel<BN><<<(unsigned)ceil_div(total, per), B3_THREADS, smem, st>>>(maps, M, kb, per, total, n_rhs, P, err);
    return launch_status("tc_block3_kernel");
}

}  // namespace mbem

extern "C" int mbem_gemm_bf16x3_t_parts(const void* A, int64_t lda, int64_t lo_a, const void* Xt, int64_t ldx,
                                        int64_t lo_x, int64_t M, int64_t K, int n_rhs, float* work, size_t work_bytes,
                                        int* kb_out, int* per_out, void* stream) {
    using namespace mbem;
    MBEM_REQUIRE(M >= 1 && K >= 1 && n_rhs >= 1 && n_rhs <= 256, MBEM_ERR_ARG,
                 "bad GEMM sizes (M=%lld, K=%lld, n_rhs=%d; n_rhs <= 256)", (long long)M, (long long)K, n_rhs);
    MBEM_REQUIRE(A && Xt && work && kb_out && per_out && lo_a >= K && lo_x >= K && lda >= lo_a + K && ldx >= lo_x + K,
                 MBEM_ERR_ARG, "bad GEMM pointers/strides");
    MBEM_REQUIRE(lda % 8 == 0 && ldx % 8 == 0 && lo_a % 8 == 0 && lo_x % 8 == 0 && (uintptr_t)A % 16 == 0 &&
                     (uintptr_t)Xt % 16 == 0,
                 MBEM_ERR_ARG, "TMA needs 16-byte aligned bases, panels and row strides (multiples of 8)");
    const int64_t kb64 = ceil_div(K, B3_BK), units = kb64 * ceil_div(M, TC_BM);
    MBEM_REQUIRE(units < (int64_t)1 << 30, MBEM_ERR_SIZE, "GEMM of %lld x %lld", (long long)M, (long long)K);
    int sms = 152, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int kb = (int)kb64, total = (int)units;
    // equal runs, of at least 32 blocks (a run's partial sums cost about eight),
    // and no more parts a tile than the workspace holds
    const int64_t slice = M * n_rhs * (int64_t)sizeof(float);
    int per = std::max((int)ceil_div(total, sms), std::min(32, kb));
    const int64_t room = (int64_t)(work_bytes / (size_t)slice);
    MBEM_REQUIRE(room >= 2, MBEM_ERR_SIZE, "GEMM workspace too small for two parts");
    // a tile of kb blocks meets at most (kb - 2) / per + 2 runs
    while ((kb - 2) / per + 2 > room) per++;
    int* err = tc_error_flag();
    MBEM_REQUIRE(err != nullptr, MBEM_ERR_CUDA, "no device error flag");
    const int bn = n_rhs <= 16 ? 16 : n_rhs <= 32 ? 32 : n_rhs <= 64 ? 64 : n_rhs <= 128 ? 128 : 256;
    B3Maps m;
    int e;
    const uint16_t *a = static_cast<const uint16_t*>(A), *x = static_cast<const uint16_t*>(Xt);
    if ((e = tc_make_map32(&m.a_hi, a, M, K, lda, TC_BM))) return e;
    if ((e = tc_make_map32(&m.a_lo, a + lo_a, M, K, lda, TC_BM))) return e;
    if ((e = tc_make_map32(&m.x_hi, x, n_rhs, K, ldx, bn))) return e;
    if ((e = tc_make_map32(&m.x_lo, x + lo_x, n_rhs, K, ldx, bn))) return e;
    *kb_out = kb;
    *per_out = per;
    cudaStream_t st = (cudaStream_t)stream;
    switch (bn) {
        case 16: return launch_block3<16>(m, M, kb, per, total, n_rhs, work, err, st);
        case 32: return launch_block3<32>(m, M, kb, per, total, n_rhs, work, err, st);
        case 64: return launch_block3<64>(m, M, kb, per, total, n_rhs, work, err, st);
        case 128: return launch_block3<128>(m, M, kb, per, total, n_rhs, work, err, st);
        default: return launch_block3<256>(m, M, kb, per, total, n_rhs, work, err, st);
    }
}
