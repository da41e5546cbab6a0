// The far-field residual of a block of right-hand sides, R = B - A X, as exact
// tensor-core products of fixed-point digits (sm_103a).
//
// A refinement residual has to be right to about 2^-48 of |A| |X| while A X
// cancels B, so no FP32 accumulation of rounded products will do. Every row of A
// and every right-hand side is scaled by a power of two into [-1, 1] and cut into
// six signed digits of eight bits, integers in [-128, 128], which BF16 holds
// exactly (48 bits: every bit of an FP32 entry down to 2^-24 of its row's
// largest). A product of two digits is at most 2^14 and 256 of them sum to at
// most 2^22, so the tensor core's FP32 accumulator is exact over 256 columns; the
// epilogue adds it to 32-bit integers (exact up to 131,072 columns) while the next
// 256 run into a second accumulator. The 21 digit products of order p + q <= 5
// are combined in FP64; what the cut leaves out is below 2^-48 of
// max|A_i| max|X_r| a term. (Error-free splitting for matrix products: Ozaki,
// Ogita, Oishi, Rump, Numer. Algorithms 59, 2012.)
//
// Bound by the tensor pipe and the L2 traffic of its operands: 20,736 unknowns x
// 256 right-hand sides 5.2 ms (splitting 1.5 ms, 21 products 3.5 ms at 1.33 PFLOP/s, 0.69 of the measured bf16 rate,
// combination 0.1 ms), against 49 ms for a double-float product on the FP32
// pipe (eleven instructions a term at 70 % of its issue slots).
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "tc_common.cuh"

namespace mbem {

constexpr int EX_D = 6;                       // digits
constexpr int EX_PAIRS = EX_D * (EX_D + 1) / 2;
constexpr int EX_CHUNK = 4;                   // K blocks an accumulator takes: 256 columns, 2^22
constexpr int EX_STAGES = 4;
constexpr int EX_THREADS = 320;               // eight epilogue warps, producer, issuer
constexpr int EX_NONFINITE = INT_MIN;         // exponent of a row that holds an Inf or NaN

// digits of v in [-1, 1] as BF16 bit patterns
__device__ __forceinline__ void digits_f32(float v, uint16_t d[EX_D]) {
    float r = v * 128.0f;
#pragma unroll
    for (int p = 0; p < EX_D; p++) {
        const float t = rintf(r);
        d[p] = (uint16_t)(__float_as_uint(t) >> 16);       // |t| <= 128: eight bits
        r = (r - t) * 256.0f;                              // exact
    }
}
__device__ __forceinline__ void digits_f64(double v, uint16_t d[EX_D]) {
    double r = v * 128.0;
#pragma unroll
    for (int p = 0; p < EX_D; p++) {
        const double t = rint(r);
        d[p] = (uint16_t)(__float_as_uint((float)t) >> 16);
        r = (r - t) * 256.0;
    }
}

__device__ __forceinline__ double ex_block_max(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double m = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) m = fmax(m, red[w]);
    return m;
}
// the exponent e with 2^e >= m, and 2^-e as two factors (either may be subnormal's)
__device__ __forceinline__ int ex_exponent(double m, bool finite) {
    if (!finite) return EX_NONFINITE;
    if (!(m > 0.0)) return 0;
    int e;
    frexp(m, &e);
    return e;
}

// Rows row0 .. row0 + n_rows of A (columns col0 .. col0 + cols) as digits
// D[p][row][ld], zero from cols to ld; a block a row, its exponent in ex.
template <bool VEC>
__global__ void __launch_bounds__(256)
ex_split_rows_kernel(const float* __restrict__ A, int64_t lda, int64_t cols, int64_t rows_pad, int64_t ld,
                     uint16_t* __restrict__ D, int* __restrict__ ex) {
    __shared__ double red[8];
    const int64_t row = blockIdx.x;
    const float* a = A + row * lda;
    float m = 0.0f;
    bool ok = true;
    if (VEC) {
        for (int64_t c = 4 * threadIdx.x; c + 3 < cols; c += 1024) {
            const float4 v = *reinterpret_cast<const float4*>(a + c);
            m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
            ok = ok && isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w);
        }
        for (int64_t c = cols / 4 * 4 + threadIdx.x; c < cols; c += 256) {
            m = fmaxf(m, fabsf(a[c]));
            ok = ok && isfinite(a[c]);
        }
    } else {
        for (int64_t c = threadIdx.x; c < cols; c += 256) {
            m = fmaxf(m, fabsf(a[c]));
            ok = ok && isfinite(a[c]);
        }
    }
    const bool finite = __syncthreads_and(ok);
    const int e = ex_exponent(ex_block_max((double)m, red), finite);
    if (threadIdx.x == 0) ex[row] = e;
    const int e1 = finite ? -(e / 2) : 0, e2 = finite ? -e - e1 : 0;
    const float f1 = finite ? ldexpf(1.0f, e1) : 0.0f, f2 = finite ? ldexpf(1.0f, e2) : 0.0f;
    for (int64_t c = 4 * threadIdx.x; c < ld; c += 1024) {
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (finite) {
            if (VEC && c + 3 < cols) {
                const float4 q = *reinterpret_cast<const float4*>(a + c);
                v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
            } else {
                for (int i = 0; i < 4; i++) v[i] = c + i < cols ? a[c + i] : 0.0f;
            }
        }
        uint16_t d[4][EX_D];
#pragma unroll
        for (int i = 0; i < 4; i++) digits_f32(v[i] * f1 * f2, d[i]);
#pragma unroll
        for (int p = 0; p < EX_D; p++)
            *reinterpret_cast<ushort4*>(D + ((int64_t)p * rows_pad + row) * ld + c) =
                make_ushort4(d[0][p], d[1][p], d[2][p], d[3][p]);
    }
}

// the right-hand sides, D[q][r][ld] for r < n_rhs (of rhs_pad); a block each
__global__ void __launch_bounds__(256)
ex_split_rhs_kernel(const double* __restrict__ X, int64_t ldx, int64_t cols, int rhs_pad, int64_t ld,
                    uint16_t* __restrict__ D, int* __restrict__ ex) {
    __shared__ double red[8];
    const int64_t r = blockIdx.x;
    const double* x = X + r * ldx;
    double m = 0.0;
    bool ok = true;
    for (int64_t c = threadIdx.x; c < cols; c += 256) {
        m = fmax(m, fabs(x[c]));
        ok = ok && isfinite(x[c]);
    }
    const bool finite = __syncthreads_and(ok);
    const int e = ex_exponent(ex_block_max(m, red), finite);
    if (threadIdx.x == 0) ex[r] = e;
    const int e1 = finite ? -(e / 2) : 0, e2 = finite ? -e - e1 : 0;
    const double f1 = finite ? ldexp(1.0, e1) : 0.0, f2 = finite ? ldexp(1.0, e2) : 0.0;
    for (int64_t c = threadIdx.x; c < ld; c += 256) {
        uint16_t d[EX_D];
        digits_f64(finite && c < cols ? x[c] * f1 * f2 : 0.0, d);
#pragma unroll
        for (int q = 0; q < EX_D; q++) D[((int64_t)q * rhs_pad + r) * ld + c] = d[q];
    }
}

// ---------------------------------------------------------------------------
// the digit products: a persistent CTA an SM over (row tile, digit pair) items;
// P[pair][rhs][row] = sum_k A_p[row, k] X_q[rhs, k] as exact 32-bit integers.
// Items of one row tile follow one another, so that the CTAs at work share its
// digit panels in L2 (X's panels, 64 MB at 20,736 x 256, stay there).
// ---------------------------------------------------------------------------
template <int COLS>
__device__ __forceinline__ void ex_tmem_add(uint32_t ta, uint32_t* acc) {
    // v + 1.5 x 2^23 holds the integer v in its low bits; the constant's bits
    // are taken off once at the end
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(ta + (uint32_t)c));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; i++) acc[c + i] += __float_as_uint(__fadd_rn(__uint_as_float(v[i]), 12582912.0f));
    }
}

template <int BN>
__global__ void __launch_bounds__(EX_THREADS, 1)
tc_exact_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapX, int64_t rows,
                int64_t rows_pad, int kb_total, int n_rhs, int items, int32_t* __restrict__ P, int* __restrict__ error) {
    constexpr int A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2, STAGE = A_BYTES + B_BYTES;
    constexpr uint32_t TMEM_COLS = 2 * BN;      // BN in 32 .. 256: a power of two of at least 64
    constexpr int HALF = BN / 2;
    extern __shared__ __align__(1024) uint8_t ex_smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)ex_smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[EX_STAGES], empty[EX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < EX_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 8);
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
    const int chunks = (kb_total + EX_CHUNK - 1) / EX_CHUNK;
    auto pair_of = [](int i, int& p, int& q) {
        p = 0;
        while (i >= EX_D - p) i -= EX_D - p++;
        q = i;
    };

    if (warp == 8 && lane == 0) {
        uint32_t g = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            int p, q;
            pair_of(it % EX_PAIRS, p, q);
            const int ya = (int)(p * rows_pad + (int64_t)(it / EX_PAIRS) * TC_BM), yx = q * BN;
            for (int kb = 0; kb < kb_total; kb++, g++) {
                const int s = g % EX_STAGES;
                if (!mbar_wait(&empty[s], ((g / EX_STAGES) & 1u) ^ 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
                uint8_t* st = smem + s * STAGE;
                mbar_arrive_expect_tx(&full[s], STAGE);
                tma_load_2d(st, &mapA, kb * TC_BK, ya, &full[s]);
                tma_load_2d(st + A_BYTES, &mapX, kb * TC_BK, yx, &full[s]);
            }
        }
        // the last copies have landed before the CTA can end
        for (uint32_t h = g > EX_STAGES ? g - EX_STAGES : 0; h < g; h++)
            if (!mbar_wait(&full[h % EX_STAGES], (h / EX_STAGES) & 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
    } else if (warp == 9 && lane == 0) {
        constexpr uint32_t idesc = f16_idesc(TC_BM, BN);
        uint32_t g = 0, c = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x)
            for (int kb = 0; kb < kb_total; kb++, g++) {
                const int in = kb % EX_CHUNK;
                const uint32_t d = tmem + (c & 1u) * BN;
                if (in == 0) {
                    if (!mbar_wait(&acc_empty[c & 1u], ((c >> 1) & 1u) ^ 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
                    tc_fence_after();
                }
                const int s = g % EX_STAGES;
                if (!mbar_wait(&full[s], (g / EX_STAGES) & 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
                tc_fence_after();
                const uint32_t a0 = smem_addr(smem + s * STAGE), b0 = a0 + A_BYTES;
#pragma unroll
                for (int k = 0; k < TC_BK / 16; k++) {
                    const uint64_t ad = sw128_desc(a0 + k * 32), bd = sw128_desc(b0 + k * 32);
                    const uint32_t add = (in > 0 || k > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                        "l"(ad), "l"(bd), "r"(idesc), "r"(add)
                        : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_addr(&empty[s]))
                             : "memory");
                if (in == EX_CHUNK - 1 || kb == kb_total - 1) {
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                     smem_addr(&acc_full[c & 1u]))
                                 : "memory");
                    c++;
                }
            }
    } else if (warp < 8) {
        // warp w: TMEM lanes 32 (w % 4) .., columns (w / 4) BN / 2 ..
        const uint32_t col0 = (uint32_t)(warp >> 2) * HALF;
        const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
        uint32_t c = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            uint32_t acc[HALF];
#pragma unroll
            for (int i = 0; i < HALF; i++) acc[i] = 0u;
#pragma unroll 1
            for (int h = 0; h < chunks; h++, c++) {
                if (!mbar_wait(&acc_full[c & 1u], (c >> 1) & 1u, TC_WAIT_LIMIT)) atomicExch(error, 1);
                tc_fence_after();
                ex_tmem_add<HALF>(tmem + lanes + (c & 1u) * BN + col0, acc);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[c & 1u]);
            }
            const int64_t row = (int64_t)(it / EX_PAIRS) * TC_BM + 32 * (warp & 3) + lane;
            const uint32_t off = (uint32_t)chunks * 0x4B400000u;
            if (row < rows) {
                int32_t* out = P + ((int64_t)(it % EX_PAIRS) * n_rhs + col0) * rows_pad + row;
#pragma unroll
                for (int i = 0; i < HALF; i++)
                    if ((int)col0 + i < n_rhs) out[(int64_t)i * rows_pad] = (int32_t)(acc[i] - off);
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

// R[r, row] = (first ? B : R)[r, row] - 2^(ea + ex - 14) sum_o 2^(-8 o) sum_{p + q = o} P
__global__ void __launch_bounds__(256)
ex_combine_kernel(const int32_t* __restrict__ P, int64_t rows, int64_t rows_pad, int n_rhs, const int* __restrict__ ea,
                  const int* __restrict__ exr, const double* __restrict__ B, int64_t n, int64_t row0, int first,
                  double* __restrict__ R) {
    const int64_t row = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int r = blockIdx.y;
    if (row >= rows) return;
    int64_t s[EX_D];
#pragma unroll
    for (int o = 0; o < EX_D; o++) s[o] = 0;
    const int32_t* p0 = P + (int64_t)r * rows_pad + row;
    int i = 0;
#pragma unroll
    for (int p = 0; p < EX_D; p++)
#pragma unroll
        for (int q = 0; q < EX_D - p; q++, i++) s[p + q] += p0[(int64_t)i * n_rhs * rows_pad];
    // pairs of orders are exact integers below 2^43
    const double y = (double)(s[0] * 256 + s[1]) + (double)(s[2] * 256 + s[3]) * 0x1p-16 +
                     (double)(s[4] * 256 + s[5]) * 0x1p-32;
    const int e1 = ea[row], e2 = exr[r];
    const double v = (e1 == EX_NONFINITE || e2 == EX_NONFINITE) ? nan("") : scalbn(y, e1 + e2 - 14 - 8);
    const int64_t o = (int64_t)r * n + row0 + row;
    R[o] = (first ? B[o] : R[o]) - v;
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
constexpr int64_t EX_SEGMENT = 65536;             // columns at a time: the sums stay below 2^30
constexpr int64_t EX_PIECE_BYTES = (int64_t)6 << 30;

struct ExPlan {
    int64_t ld, rows, rhs_pad, rhs;               // per column segment and row chunk
    size_t digits_a, digits_x, products, total;
};
static ExPlan ex_plan(int64_t k, int64_t n) {
    ExPlan p;
    p.ld = ceil_div(std::min(n, EX_SEGMENT), TC_BK) * TC_BK;
    p.rhs = std::min<int64_t>(k, 256);
    p.rhs_pad = p.rhs <= 32 ? 32 : p.rhs <= 64 ? 64 : p.rhs <= 128 ? 128 : 256;
    const int64_t most = std::max<int64_t>(EX_PIECE_BYTES / (2 * EX_D * p.ld) / TC_BM * TC_BM, TC_BM);
    p.rows = std::min(ceil_div(n, TC_BM) * TC_BM, most);
    p.digits_a = (size_t)(2 * EX_D * p.rows * p.ld);
    p.digits_x = (size_t)(2 * EX_D * p.rhs_pad * p.ld);
    p.products = (size_t)(4 * EX_PAIRS * p.rhs * p.rows);
    p.total = 1024 + p.digits_a + p.digits_x + p.products + 8 * (size_t)(p.rows + p.rhs_pad);
    return p;
}
size_t exact_residual_workspace(int64_t k, int64_t n) { return ex_plan(k, n).total; }

template <int BN>
static void launch_exact(const CUtensorMap& ma, const CUtensorMap& mx, int64_t rows, int64_t rows_pad, int kb, int n_rhs,
                         int sms, int32_t* P, int* err, cudaStream_t st) {
    const size_t smem = (size_t)EX_STAGES * (TC_BM * TC_BK * 2 + BN * TC_BK * 2) + 1024;
    cudaFuncSetAttribute(tc_exact_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int items = (int)(ceil_div(rows, TC_BM) * EX_PAIRS);
    tc_exact_kernel<BN><<<(unsigned)std::min(items, sms), EX_THREADS, smem, st>>>(ma, mx, rows, rows_pad, kb, n_rhs,
                                                                                  items, P, err);
}

// R = B - A X for k right-hand sides (rows of B, X, R, n each); A is n x n FP32 at lda
int exact_residual(const float* A, int64_t lda, int64_t n, const double* B, const double* X, int64_t k, double* R,
                   void* work, size_t work_bytes, cudaStream_t st) {
    const ExPlan pl = ex_plan(k, n);
    MBEM_REQUIRE(work && work_bytes >= pl.total, MBEM_ERR_SIZE, "batched residual workspace too small");
    int* err = tc_error_flag();
    MBEM_REQUIRE(err != nullptr, MBEM_ERR_CUDA, "no device error flag");
    int sms = 152, dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    uint8_t* w = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(work) + 1023) & ~(uintptr_t)1023);
    uint16_t* da = reinterpret_cast<uint16_t*>(w);
    uint16_t* dx = reinterpret_cast<uint16_t*>(w + pl.digits_a);
    int32_t* P = reinterpret_cast<int32_t*>(w + pl.digits_a + pl.digits_x);
    int* ea = reinterpret_cast<int*>(w + pl.digits_a + pl.digits_x + pl.products);
    int* exr = ea + pl.rows;
    const bool vec = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
    for (int64_t r0 = 0; r0 < k; r0 += 256) {
        const int nr = (int)std::min<int64_t>(256, k - r0);
        const int bn = nr <= 32 ? 32 : nr <= 64 ? 64 : nr <= 128 ? 128 : 256;
        for (int64_t c0 = 0; c0 < n; c0 += EX_SEGMENT) {
            const int64_t nc = std::min(EX_SEGMENT, n - c0), ld = ceil_div(nc, TC_BK) * TC_BK;
            ex_split_rhs_kernel<<<(unsigned)nr, 256, 0, st>>>(X + r0 * n + c0, n, nc, bn, ld, dx, exr);
            CUtensorMap ma, mx;
            int e = tc_make_map(&mx, dx, (int64_t)EX_D * bn, ld, ld, bn);
            if (e) return e;
            for (int64_t row0 = 0; row0 < n; row0 += pl.rows) {
                const int64_t rows = std::min(pl.rows, n - row0), pad = ceil_div(rows, TC_BM) * TC_BM;
                const float* a = A + row0 * lda + c0;
                if (vec) ex_split_rows_kernel<true><<<(unsigned)rows, 256, 0, st>>>(a, lda, nc, pad, ld, da, ea);
                else ex_split_rows_kernel<false><<<(unsigned)rows, 256, 0, st>>>(a, lda, nc, pad, ld, da, ea);
                if ((e = tc_make_map(&ma, da, (int64_t)EX_D * pad, ld, ld, TC_BM))) return e;
                const int kb = (int)(ld / TC_BK);
                switch (bn) {
                    case 32: launch_exact<32>(ma, mx, rows, pad, kb, nr, sms, P, err, st); break;
                    case 64: launch_exact<64>(ma, mx, rows, pad, kb, nr, sms, P, err, st); break;
                    case 128: launch_exact<128>(ma, mx, rows, pad, kb, nr, sms, P, err, st); break;
                    default: launch_exact<256>(ma, mx, rows, pad, kb, nr, sms, P, err, st); break;
                }
                ex_combine_kernel<<<dim3((unsigned)ceil_div(rows, 256), (unsigned)nr), 256, 0, st>>>(
                    P, rows, pad, nr, ea, exr, B + r0 * n, n, row0, c0 == 0, R + r0 * n);
                count_launches(3);
                if ((e = launch_status("exact_residual", 0))) return e;
            }
            count_launches(1);
        }
    }
    return MBEM_OK;
}

}  // namespace mbem
