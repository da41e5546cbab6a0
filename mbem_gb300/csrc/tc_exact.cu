// The far-field residual of a block of right-hand sides, R = B - A X, as exact
// tensor-core products of fixed-point digits (sm_103a).
//
// A refinement residual has to be right to about 2^-48 of |A| |X| while A X
// cancels B, so no FP32 accumulation of rounded products will do. A is scaled by
// powers of two, a row by r_i and then a column by c_j <= 1 (its largest entry of
// the scaled rows), X by the inverse column scales and one a right-hand side, all into
// [-1, 1]: systems with traction unknowns hold columns of 1 / mu beside unknowns of mu,
// which one scale a row and one a right-hand side would cut away. Both are cut into
// signed digits of eight bits, integers in [-128, 128], which BF16 holds exactly.
// A product of two digits is at most 2^14 and 256 of them sum to at
// most 2^22, so the tensor core's FP32 accumulator is exact over 256 columns; the
// epilogue adds it to 32-bit integers (exact up to 131,072 columns) while the next
// 256 run into a second accumulator. The digit products of order p + q <= o
// are combined; what is left out is below (o + 2) 2^(-8 (o + 1)) of the scales a term
// (o + 1 products of the next order a bit over half a unit each, both last digits
// rounded): 7 x 2^-48 for o = 5. (Error-free splitting for matrix products: Ozaki,
// Ogita, Oishi, Rump, Numer. Algorithms 59, 2012.)
//
// The order is 5 (six digits, 21 products) where the entries of each scaled right-hand side lie
// close to its largest one, and grows by one for every eight bits that they lie below
// (ex_rhs_scale_kernel decides on the device): with o = 5 alone, one entry 10^4 times
// the others cost the other rows a factor of 60 against the double-float product.
// Against it (FP32 pairs, every entry with its own exponent) the errors are smaller
// or equal for X of up to 14 decades, mu up to 3e10 and blocks of two materials
// (emulated, 2,592 unknowns, largest and rms error relative to |A| |X|: balanced
// random X 2e-16 | 4e-17 against 4e-13 | 4e-14; one entry 10^8 times the others
// 3e-16 | 5e-17 against 7e-12 | 7e-13).
//
// Bound by the tensor pipe and the L2 traffic of its operands: 20,736 unknowns x
// 256 right-hand sides 5.85 ms (row and column scales 0.53 ms, digits 1.4, 21 products
// 3.6 ms at 1.29 PFLOP/s, 0.68 of the measured bf16 rate, combination 0.2 ms; 5.17 ms
// with one scale a row), against 49 ms for a double-float product on the FP32
// pipe (eleven instructions a term at 70 % of its issue slots).
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "tc_common.cuh"

namespace mbem {

constexpr int EX_ORDER = 5, EX_ORDER_MAX = 11;     // least and largest order of the digit products
constexpr int EX_DA = 8;                      // most digits of A: 64 bits, FP32 entries whole down to 2^-40 of the scales
constexpr int EX_DX = EX_ORDER_MAX + 1;       // most digits of X
// digits of A and digit products at order o
__host__ __device__ constexpr int ex_digits_a(int o) { return o + 1 < EX_DA ? o + 1 : EX_DA; }
__host__ __device__ constexpr int ex_pairs(int o) {
    const int d = ex_digits_a(o);
    return d * (o + 1) - d * (d - 1) / 2;
}
constexpr int EX_CHUNK = 4;                   // K blocks an accumulator takes: 256 columns, 2^22
constexpr int EX_STAGES = 4;
constexpr int EX_THREADS = 320;               // eight epilogue warps, producer, issuer
constexpr int EX_NONFINITE = INT_MIN;         // exponent of a row that holds an Inf or NaN
constexpr int EX_DEAD = -(1 << 20);           // exponent of a column without an entry

// the exponent e of |v| = f 2^e, f in [1/2, 1), from the bits of a finite |v| > 0 (a subnormal
// FP32 entry counts as 2^-127)
__device__ __forceinline__ int ex_exp(int bits) { return (bits >> 23) - 126; }
__device__ __forceinline__ int ex_exp(double v) {
    const int e = (__double2hiint(v) >> 20) & 2047;
    if (e > 0) return e - 1022;
    int q;
    frexp(v, &q);
    return q;
}

// the exponents r_i of the rows of A (n columns at lda): EX_NONFINITE with an Inf or NaN,
// 0 without an entry; a block a row
template <bool VEC>
__global__ void __launch_bounds__(256)
ex_row_scale_kernel(const float* __restrict__ A, int64_t lda, int64_t cols, int* __restrict__ ex) {
    __shared__ int red[8];
    const int64_t row = blockIdx.x;
    const float* a = A + row * lda;
    int m = 0;                                 // largest |a| as bits: an order on them, Inf and NaN above all
    const int64_t c4 = VEC ? cols / 4 * 4 : 0;
    for (int64_t c = 4 * threadIdx.x; c < c4; c += 1024) {
        const float4 v = *reinterpret_cast<const float4*>(a + c);
        m = max(max(m, __float_as_int(fabsf(v.x))), __float_as_int(fabsf(v.y)));
        m = max(max(m, __float_as_int(fabsf(v.z))), __float_as_int(fabsf(v.w)));
    }
    for (int64_t c = c4 + threadIdx.x; c < cols; c += 256) m = max(m, __float_as_int(fabsf(a[c])));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) m = max(m, red[w]);
        ex[row] = m >= 0x7f800000 ? EX_NONFINITE : m == 0 ? 0 : ex_exp(m);
    }
}

// cmax[j] = the largest exponent of column j of the scaled rows as exponent - EX_DEAD (0: none),
// by atomics: a block EX_CROWS rows of 1,024 columns, a thread four of them. The row that
// has its largest entry in column j leaves it at 0, so a scaled row's largest entry stays
// in [1/2, 1).
constexpr int EX_CROWS = 64;
template <bool VEC>
__global__ void __launch_bounds__(256)
ex_col_scale_kernel(const float* __restrict__ A, int64_t lda, int64_t rows, int64_t cols, const int* __restrict__ ex,
                    int* __restrict__ cmax) {
    __shared__ int er[EX_CROWS];
    const int64_t c = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4, r0 = (int64_t)blockIdx.y * EX_CROWS;
    const int nr = (int)lmin(EX_CROWS, rows - r0);
    if ((int)threadIdx.x < nr) er[threadIdx.x] = ex[r0 + threadIdx.x];
    __syncthreads();
    if (c >= cols) return;
    const float* a = A + r0 * lda + c;
    const int nc = (int)lmin(4, cols - c);
    // an entry's bits less its row's exponent: their top is the scaled entry's exponent
    constexpr int NONE = INT_MIN;
    int m[4] = {NONE, NONE, NONE, NONE};
#pragma unroll 8
    for (int i = 0; i < nr; i++) {
        float v[4];
        if (VEC && nc == 4) {
            const float4 q = *reinterpret_cast<const float4*>(a + i * lda);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = u < nc ? a[i * lda + u] : 0.0f;
        }
        const int e = er[i];
        if (e == EX_NONFINITE) continue;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int b = __float_as_int(fabsf(v[u]));
            m[u] = max(m[u], b ? b - e * (1 << 23) : NONE);
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (m[u] != NONE) atomicMax(&cmax[c + u], ex_exp(m[u]) - EX_DEAD);
}

// Exponents of the right-hand sides' largest entries under the column scales, and the order
// that they need: an entry's error goes with the largest one, so the digits go on as
// far as most entries lie below it (mean and standard deviation of their exponents;
// 3 bits for smooth and 5 for random X), and half a bit
// a factor of two in the columns that the double-float sum's error grows by. Six
// digits are then no worse than it up to some 8 bits (a random X with one entry 10
// times its largest: 7.3 bits, rms error 4e-14 against 3e-14; 10^3 times, 13 bits, 1e-12 against
// 5e-14). A block a right-hand side; *extra is raised to the largest order - EX_ORDER.
__global__ void __launch_bounds__(256)
ex_rhs_scale_kernel(const double* __restrict__ X, int64_t ldx, int64_t cols, const int* __restrict__ cmax,
                    float few, int* __restrict__ ex, int* __restrict__ extra) {
    __shared__ int rm[8];
    __shared__ long long rs[8][3];
    const int64_t r = blockIdx.x;
    const double* x = X + r * ldx;
    int m = INT_MIN;
    long long s[3] = {0, 0, 0};                // entries, their exponents' sum and sum of squares
    bool ok = true;
    for (int64_t c = threadIdx.x; c < cols; c += 256) {
        const double v = x[c];
        ok = ok && isfinite(v);
        if (!isfinite(v) || v == 0.0 || cmax[c] == 0) continue;
        const int e = ex_exp(v) + cmax[c] + EX_DEAD;
        m = max(m, e);
        s[0]++;
        s[1] += e;
        s[2] += (long long)e * e;
    }
    const bool finite = __syncthreads_and(ok);
    m = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
    if ((threadIdx.x & 31) == 0) {
        rm[threadIdx.x >> 5] = m;
        for (int k = 0; k < 3; k++) rs[threadIdx.x >> 5][k] = s[k];
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; w++) {
        m = max(m, rm[w]);
        for (int k = 0; k < 3; k++) s[k] += rs[w][k];
    }
    ex[r] = !finite ? EX_NONFINITE : s[0] == 0 ? 0 : m;
    if (!finite || s[0] == 0) return;
    const float mean = (float)((double)s[1] / (double)s[0]);
    const float sd = sqrtf(fmaxf((float)((double)s[2] / (double)s[0] - (double)mean * mean), 0.0f));
    const float need = ((float)m - mean + sd + few - 8.0f) / 8.0f;
    const int o = need > 0.0f ? (int)ceilf(fminf(need, (float)(EX_ORDER_MAX - EX_ORDER))) : 0;
    if (o > 0) atomicMax(extra, o);
}

// Rows of A under both scales as digits D[p][row][ld], p < ex_digits_a(order), zero from
// cols to ld; a block a row
template <bool VEC>
__global__ void __launch_bounds__(256)
ex_split_rows_kernel(const float* __restrict__ A, int64_t lda, int64_t cols, int64_t rows_pad, int64_t ld,
                     const int* __restrict__ ex, const int* __restrict__ cmax, const int* __restrict__ extra,
                     uint16_t* __restrict__ D) {
    const int64_t row = blockIdx.x;
    const float* a = A + row * lda;
    const int e = ex[row], nd = ex_digits_a(EX_ORDER + *extra);
    const bool finite = e != EX_NONFINITE;
    for (int64_t c = 4 * threadIdx.x; c < ld; c += 1024) {
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        int k[4] = {0, 0, 0, 0};
        if (finite) {
            if (c + 3 < cols) {
                if (VEC) {
                    const float4 q = *reinterpret_cast<const float4*>(a + c);
                    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++) v[i] = a[c + i];
                }
                const int4 q = *reinterpret_cast<const int4*>(cmax + c);
                k[0] = q.x; k[1] = q.y; k[2] = q.z; k[3] = q.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (c + i < cols) {
                        v[i] = a[c + i];
                        k[i] = cmax[c + i];
                    }
            }
        }
        float r[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // 2^s as two factors: |v| 2^s <= 1, and what s below -250 leaves has no digit
            const int s = min(max(-(k[i] + EX_DEAD) - e, -250), 250), h = s >> 1;
            r[i] = k[i] ? v[i] * __int_as_float((127 + h) << 23) * __int_as_float((127 + s - h) << 23) * 128.0f : 0.0f;
        }
#pragma unroll
        for (int p = 0; p < EX_DA; p++) {
            if (p >= nd) break;
            uint16_t d[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float t = rintf(r[i]);
                d[i] = (uint16_t)(__float_as_uint(t) >> 16);       // |t| <= 128: eight bits
                r[i] = (r[i] - t) * 256.0f;                        // exact
            }
            *reinterpret_cast<ushort4*>(D + ((int64_t)p * rows_pad + row) * ld + c) = make_ushort4(d[0], d[1], d[2], d[3]);
        }
    }
}

// the right-hand sides, D[q][r][ld] for r < n_rhs (of rhs_pad), q <= order; a block each
__global__ void __launch_bounds__(256)
ex_split_rhs_kernel(const double* __restrict__ X, int64_t ldx, int64_t cols, int rhs_pad, int64_t ld,
                    const int* __restrict__ ex, const int* __restrict__ cmax, const int* __restrict__ extra,
                    uint16_t* __restrict__ D) {
    const int64_t r = blockIdx.x;
    const double* x = X + r * ldx;
    const int e = ex[r], nd = EX_ORDER + 1 + *extra;
    const bool finite = e != EX_NONFINITE;
    for (int64_t c = threadIdx.x; c < ld; c += 256) {
        double v = finite && c < cols && cmax[c] ? x[c] : 0.0;
        if (v != 0.0) v = scalbn(v, cmax[c] + EX_DEAD - e + 7);
        for (int q = 0; q < nd; q++) {
            const double t = rint(v);
            D[((int64_t)q * rhs_pad + r) * ld + c] = (uint16_t)(__float_as_uint((float)t) >> 16);
            v = (v - t) * 256.0;
        }
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
                int64_t rows_pad, int kb_total, int n_rhs, const int* __restrict__ extra, int32_t* __restrict__ P,
                int* __restrict__ error) {
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
    const int order = EX_ORDER + *extra, pairs = ex_pairs(order), items = (int)(rows_pad / TC_BM) * pairs;
    auto pair_of = [order](int i, int& p, int& q) {
        p = 0;
        while (i > order - p) i -= order + 1 - p++;
        q = i;
    };

    if (warp == 8 && lane == 0) {
        uint32_t g = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            int p, q;
            pair_of(it % pairs, p, q);
            const int ya = (int)(p * rows_pad + (int64_t)(it / pairs) * TC_BM), yx = q * BN;
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
            const int64_t row = (int64_t)(it / pairs) * TC_BM + 32 * (warp & 3) + lane;
            const uint32_t off = (uint32_t)chunks * 0x4B400000u;
            if (row < rows) {
                int32_t* out = P + ((int64_t)(it % pairs) * n_rhs + col0) * rows_pad + row;
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
                  const int* __restrict__ exr, const int* __restrict__ extra, const double* __restrict__ B, int64_t n,
                  int64_t row0, int first, double* __restrict__ R) {
    const int64_t row = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int r = blockIdx.y;
    if (row >= rows) return;
    const int order = EX_ORDER + *extra, nd = ex_digits_a(order);
    int64_t s[EX_DX];
#pragma unroll
    for (int o = 0; o < EX_DX; o++) s[o] = 0;
    const int32_t* p0 = P + (int64_t)r * rows_pad + row;
    const int64_t step = (int64_t)n_rhs * rows_pad;
#pragma unroll
    for (int p = 0; p < EX_DA; p++) {
        if (p >= nd) break;
#pragma unroll
        for (int q = 0; q < EX_DX - p; q++)
            if (p + q <= order) {
                s[p + q] += *p0;
                p0 += step;
            }
    }
    // four orders are exact integers: at most eight products of 2^30 each, times 2^24
    double y = 0.0;
#pragma unroll
    for (int o = EX_DX - 4; o >= 0; o -= 4)
        y = y * 0x1p-32 + (double)(((s[o] * 256 + s[o + 1]) * 256 + s[o + 2]) * 256 + s[o + 3]);
    const int e1 = ea[row], e2 = exr[r];
    const double v = (e1 == EX_NONFINITE || e2 == EX_NONFINITE) ? nan("") : scalbn(y, e1 + e2 - 14 - 24);
    const int64_t o = (int64_t)r * n + row0 + row;
    R[o] = (first ? B[o] : R[o]) - v;
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
constexpr int64_t EX_SEGMENT = 65536;             // columns at a time: the sums stay below 2^30
constexpr int64_t EX_PIECE_BYTES = (int64_t)2 << 30;

struct ExPlan {
    int64_t ld, rows, rhs_pad, rhs;               // per column segment and row chunk
    size_t digits_a, digits_x, products, exponents, total;
    int sms;
};
static ExPlan ex_plan(int64_t k, int64_t n) {
    ExPlan p;
    p.sms = 152;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&p.sms, cudaDevAttrMultiProcessorCount, dev);
    p.ld = ceil_div(std::min(n, EX_SEGMENT), TC_BK) * TC_BK;
    p.rhs = std::min<int64_t>(k, 256);
    p.rhs_pad = p.rhs <= 32 ? 32 : p.rhs <= 64 ? 64 : p.rhs <= 128 ? 128 : 256;
    // The row tiles of a piece: of those whose digits fit EX_PIECE_BYTES the number with the
    // fewest rounds of items over the SMs (a piece costs about half a round more)
    const int64_t tiles = ceil_div(n, TC_BM), pairs = ex_pairs(EX_ORDER);
    const int64_t most = std::max<int64_t>(1, std::min(tiles, EX_PIECE_BYTES / (2 * EX_DA * p.ld * TC_BM)));
    double cost = 1e300;
    int64_t best = most;
    for (int64_t t = most; t > most / 2; t--) {
        const int64_t whole = tiles / t, rest = tiles % t;
        const double c = (double)(whole * ceil_div(t * pairs, p.sms) + ceil_div(rest * pairs, p.sms)) +
                         0.5 * (double)(whole + (rest > 0));
        if (c < cost) {
            cost = c;
            best = t;
        }
    }
    p.rows = best * TC_BM;
    p.digits_a = (size_t)(2 * EX_DA * p.rows * p.ld);
    p.digits_x = (size_t)(2 * EX_DX * p.rhs_pad * p.ld);
    p.products = (size_t)(4 * ex_pairs(EX_ORDER_MAX) * p.rhs * p.rows);
    p.exponents = 4 * (size_t)(p.ld + 4 + n + p.rhs_pad);          // columns, the order, rows, right-hand sides
    p.total = 1024 + p.digits_a + p.digits_x + p.products + p.exponents;
    p.total = (p.total + 7) / 8 * 8;
    return p;
}
size_t exact_residual_workspace(int64_t k, int64_t n) { return ex_plan(k, n).total; }

template <int BN>
static void launch_exact(const CUtensorMap& ma, const CUtensorMap& mx, int64_t rows, int64_t rows_pad, int kb, int n_rhs,
                         int sms, const int* extra, int32_t* P, int* err, cudaStream_t st) {
    const size_t smem = (size_t)EX_STAGES * (TC_BM * TC_BK * 2 + BN * TC_BK * 2) + 1024;
    cudaFuncSetAttribute(tc_exact_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int items = (int)(ceil_div(rows, TC_BM) * ex_pairs(EX_ORDER));       // at least
    tc_exact_kernel<BN><<<(unsigned)std::min(items, sms), EX_THREADS, smem, st>>>(ma, mx, rows, rows_pad, kb, n_rhs,
                                                                                  extra, P, err);
}

// R = B - A X for k right-hand sides (rows of B, X, R, n each); A is n x n FP32 at lda
int exact_residual(const float* A, int64_t lda, int64_t n, const double* B, const double* X, int64_t k, double* R,
                   void* work, size_t work_bytes, cudaStream_t st) {
    const ExPlan pl = ex_plan(k, n);
    MBEM_REQUIRE(work && work_bytes >= pl.total, MBEM_ERR_SIZE, "batched residual workspace too small");
    int* err = tc_error_flag();
    MBEM_REQUIRE(err != nullptr, MBEM_ERR_CUDA, "no device error flag");
    uint8_t* w = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(work) + 1023) & ~(uintptr_t)1023);
    uint16_t* da = reinterpret_cast<uint16_t*>(w);
    uint16_t* dx = reinterpret_cast<uint16_t*>(w + pl.digits_a);
    int32_t* P = reinterpret_cast<int32_t*>(w + pl.digits_a + pl.digits_x);
    int* cmax = reinterpret_cast<int*>(w + pl.digits_a + pl.digits_x + pl.products);
    int* extra = cmax + pl.ld;
    int* ea = extra + 4;
    int* exr = ea + n;
    const bool vec = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
    const float few = n < 32768 ? 0.5f * log2f(32768.0f / (float)n) : 0.0f;
    for (int64_t r0 = 0; r0 < k; r0 += 256) {
        const int nr = (int)std::min<int64_t>(256, k - r0);
        const int bn = nr <= 32 ? 32 : nr <= 64 ? 64 : nr <= 128 ? 128 : 256;
        for (int64_t c0 = 0; c0 < n; c0 += EX_SEGMENT) {
            const int64_t nc = std::min(EX_SEGMENT, n - c0), ld = ceil_div(nc, TC_BK) * TC_BK;
            cudaMemsetAsync(cmax, 0, sizeof(int) * (size_t)(pl.ld + 4), st);
            if (vec) ex_row_scale_kernel<true><<<(unsigned)n, 256, 0, st>>>(A + c0, lda, nc, ea);
            else ex_row_scale_kernel<false><<<(unsigned)n, 256, 0, st>>>(A + c0, lda, nc, ea);
            const dim3 cgrid((unsigned)ceil_div(nc, 1024), (unsigned)ceil_div(n, EX_CROWS));
            if (vec) ex_col_scale_kernel<true><<<cgrid, 256, 0, st>>>(A + c0, lda, n, nc, ea, cmax);
            else ex_col_scale_kernel<false><<<cgrid, 256, 0, st>>>(A + c0, lda, n, nc, ea, cmax);
            ex_rhs_scale_kernel<<<(unsigned)nr, 256, 0, st>>>(X + r0 * n + c0, n, nc, cmax, few, exr, extra);
            ex_split_rhs_kernel<<<(unsigned)nr, 256, 0, st>>>(X + r0 * n + c0, n, nc, bn, ld, exr, cmax, extra, dx);
            CUtensorMap ma, mx;
            int e = tc_make_map(&mx, dx, (int64_t)EX_DX * bn, ld, ld, bn);
            if (e) return e;
            for (int64_t row0 = 0; row0 < n; row0 += pl.rows) {
                const int64_t rows = std::min(pl.rows, n - row0), pad = ceil_div(rows, TC_BM) * TC_BM;
                const float* a = A + row0 * lda + c0;
                if (vec) ex_split_rows_kernel<true><<<(unsigned)rows, 256, 0, st>>>(a, lda, nc, pad, ld, ea + row0, cmax, extra, da);
                else ex_split_rows_kernel<false><<<(unsigned)rows, 256, 0, st>>>(a, lda, nc, pad, ld, ea + row0, cmax, extra, da);
                if ((e = tc_make_map(&ma, da, (int64_t)EX_DA * pad, ld, ld, TC_BM))) return e;
                const int kb = (int)(ld / TC_BK);
                switch (bn) {
                    case 32: launch_exact<32>(ma, mx, rows, pad, kb, nr, pl.sms, extra, P, err, st); break;
                    case 64: launch_exact<64>(ma, mx, rows, pad, kb, nr, pl.sms, extra, P, err, st); break;
                    case 128: launch_exact<128>(ma, mx, rows, pad, kb, nr, pl.sms, extra, P, err, st); break;
                    default: launch_exact<256>(ma, mx, rows, pad, kb, nr, pl.sms, extra, P, err, st); break;
                }
                ex_combine_kernel<<<dim3((unsigned)ceil_div(rows, 256), (unsigned)nr), 256, 0, st>>>(
                    P, rows, pad, nr, ea + row0, exr, extra, B + r0 * n, n, row0, c0 == 0, R + r0 * n);
                count_launches(3);
                if ((e = launch_status("exact_residual", 0))) return e;
            }
            count_launches(4);
        }
    }
    return MBEM_OK;
}

}  // namespace mbem
