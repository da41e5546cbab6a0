// One Arnoldi step of k independent Krylov iterations after their shared GEMM,
// one launch: the sum of the GEMM's K splits, the projection, two passes of
// classical Gram-Schmidt, the norm, the next basis vector with its BF16 operand,
// and the right-hand side's Givens rotation (sm_103a).
//
// A cluster holds a right-hand side: its vector stays in shared memory from the
// GEMM's output to the next basis vector, so a step reads the basis four times
// (once from L1) and nothing else more than once (eleven launches before, the subtractions bound
// by FP64 conversions and each vector through memory seven times). Sums over the
// vector are FP32 products in eight chains a lane (at most n / (256 C) terms
// each for C blocks a cluster, as few as one thread's before) added in FP64; the
// subtractions carry a double-float (TwoProd, TwoSum) and round to FP32 once, as
// the FP64 ones did.
// 20,736 unknowns x 256 right-hand sides, 11 basis vectors on average: 223 us
// a step (275 with four readings from L2, 0.90 ms before, the GEMM's 0.48 ms apart).
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include <cuda_bf16.h>

#include "common.cuh"
#include "dfloat.cuh"

namespace mbem {

namespace cg = cooperative_groups;

constexpr int AR_T = 256;
constexpr int AR_SLICE = 27000;                // floats of a slice: two blocks an SM
constexpr size_t AR_SMEM = 220 * 1024;         // most shared memory a block takes

// sums a step takes: its basis vectors, or the projection's three means
__host__ __device__ constexpr int ar_vectors(int m) { return m < 4 ? 4 : m; }

struct ArnoldiArgs {
    const float* P;          // GEMM partial sums [split][k][n]
    int splits;              // their number, or with kb > 0 a row tile's own: the runs of `per` units that its
    int kb, per;             // kb units (128 rows) meet (tc_block.cu)
    int64_t split_stride;
    float* V;                // basis [m + 1][k][n]
    int j, m;
    int64_t k, n, slice;
    URanges ur;
    uint16_t* Vbf;           // next GEMM operand, row stride ldbf, panels at 0, ldp, 2 ldp: [hi], [hi | lo] (the
    int64_t ldbf, ldp;       // three-term product's) or [hi | lo | hi] (of one GEMM over a three-fold K)
    int panels;
    double *H, *cs, *sn, *g; // [(i m + j) k + r], [i k + r] x 3
    const double* beta;      // |r0|
    double rtol;
    int* left;               // right-hand sides above rtol
};

__device__ __forceinline__ void ar_two_sum(float& h, float& l, float p) {
    const float t = __fadd_rn(h, p);
    const float b = __fsub_rn(t, h);
    l = __fadd_rn(l, __fadd_rn(__fsub_rn(h, __fsub_rn(t, b)), __fsub_rn(p, b)));
    h = t;
}
__device__ __forceinline__ double ar_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// part[0 .. cnt) of every block of the cluster summed in rank order into full
__device__ __forceinline__ void ar_cluster_sum(cg::cluster_group& cl, double* part, double* full, int cnt) {
    cl.sync();
    const int ranks = (int)cl.num_blocks();
    for (int i = threadIdx.x; i < cnt; i += AR_T) {
        double s = 0.0;
        for (int r = 0; r < ranks; r++) s += cl.map_shared_rank(part, r)[i];
        full[i] = s;
    }
    cl.sync();      // part may be written again; full is seen by the block
}

// part[i] = V_i . w over the slice, a warp a vector at a time
template <bool VEC>
__device__ __forceinline__ void ar_dots(const float* __restrict__ V, int64_t stride, const float* w, int len, int cnt,
                                        double* part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = warp; i < cnt; i += AR_T / 32) {
        const float* v = V + i * stride;
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (VEC) {
            int t = 4 * lane;
            for (; t + 128 < len; t += 256) {
                const float4 a = *reinterpret_cast<const float4*>(v + t), b = *reinterpret_cast<const float4*>(v + t + 128);
                const float4 x = *reinterpret_cast<const float4*>(w + t), y = *reinterpret_cast<const float4*>(w + t + 128);
                s[0] = fmaf(a.x, x.x, s[0]); s[1] = fmaf(a.y, x.y, s[1]);
                s[2] = fmaf(a.z, x.z, s[2]); s[3] = fmaf(a.w, x.w, s[3]);
                s[4] = fmaf(b.x, y.x, s[4]); s[5] = fmaf(b.y, y.y, s[5]);
                s[6] = fmaf(b.z, y.z, s[6]); s[7] = fmaf(b.w, y.w, s[7]);
            }
            if (t < len) {
                const float4 a = *reinterpret_cast<const float4*>(v + t), x = *reinterpret_cast<const float4*>(w + t);
                s[0] = fmaf(a.x, x.x, s[0]); s[1] = fmaf(a.y, x.y, s[1]);
                s[2] = fmaf(a.z, x.z, s[2]); s[3] = fmaf(a.w, x.w, s[3]);
            }
        } else {
            int q = 0;
            for (int t = lane; t < len; t += 32, q = (q + 1) & 7) {
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (c == q) s[c] = fmaf(v[t], w[t], s[c]);
            }
        }
        double d = 0.0;
#pragma unroll
        for (int c = 0; c < 8; c++) d += (double)s[c];
        d = ar_warp_sum(d);
        if (lane == 0) part[i] = d;
    }
}

// w -= sum_i h_i V_i over the slice
template <bool VEC>
__device__ __forceinline__ void ar_subtract(const float* __restrict__ V, int64_t stride, float* w, int len, int cnt,
                                            const F2* h) {
    if (VEC) {
        for (int t = 4 * threadIdx.x; t < len; t += 4 * AR_T) {
            float4 x = *reinterpret_cast<float4*>(w + t);
            float lo[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
            for (int i = 0; i < cnt; i++) {
                const float4 a = *reinterpret_cast<const float4*>(V + i * stride + t);
                const F2 c = h[i];
                df_acc(x.x, lo[0], a.x, c.hi, c.lo);
                df_acc(x.y, lo[1], a.y, c.hi, c.lo);
                df_acc(x.z, lo[2], a.z, c.hi, c.lo);
                df_acc(x.w, lo[3], a.w, c.hi, c.lo);
            }
            x.x = __fadd_rn(x.x, lo[0]); x.y = __fadd_rn(x.y, lo[1]);
            x.z = __fadd_rn(x.z, lo[2]); x.w = __fadd_rn(x.w, lo[3]);
            *reinterpret_cast<float4*>(w + t) = x;
        }
    } else {
        for (int t = threadIdx.x; t < len; t += AR_T) {
            float x = w[t], lo = 0.0f;
#pragma unroll 4
            for (int i = 0; i < cnt; i++) df_acc(x, lo, V[i * stride + t], h[i].hi, h[i].lo);
            w[t] = __fadd_rn(x, lo);
        }
    }
}

// w -= sum_i h_i V_i and part[i] = V_i . w, a piece of 4 AR_T entries after the other:
// the second reading of a piece's basis entries finds them in L1 (the basis came from
// L2 four times a step, three times now). The sums are ar_dots'. At most AR_FUSED vectors.
constexpr int AR_FUSED = 3 * AR_T / 32;
__device__ __forceinline__ void ar_subtract_dots(const float* __restrict__ V, int64_t stride, float* w, int len, int cnt,
                                                 const F2* h, double* part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float s[3][8];
#pragma unroll
    for (int v = 0; v < 3; v++)
#pragma unroll
        for (int c = 0; c < 8; c++) s[v][c] = 0.0f;
    for (int p = 0; p < len; p += 4 * AR_T) {
        const int lim = min(4 * AR_T, len - p);
        ar_subtract<true>(V + p, stride, w + p, lim, cnt, h);
        __syncthreads();
#pragma unroll
        for (int v = 0; v < 3; v++) {
            const int i = warp + v * (AR_T / 32);
            if (i >= cnt) break;
            const float* vi = V + i * stride + p;
            int t = 4 * lane;
            for (; t + 128 < lim; t += 256) {
                const float4 a = *reinterpret_cast<const float4*>(vi + t), b = *reinterpret_cast<const float4*>(vi + t + 128);
                const float4 x = *reinterpret_cast<const float4*>(w + p + t), y = *reinterpret_cast<const float4*>(w + p + t + 128);
                s[v][0] = fmaf(a.x, x.x, s[v][0]); s[v][1] = fmaf(a.y, x.y, s[v][1]);
                s[v][2] = fmaf(a.z, x.z, s[v][2]); s[v][3] = fmaf(a.w, x.w, s[v][3]);
                s[v][4] = fmaf(b.x, y.x, s[v][4]); s[v][5] = fmaf(b.y, y.y, s[v][5]);
                s[v][6] = fmaf(b.z, y.z, s[v][6]); s[v][7] = fmaf(b.w, y.w, s[v][7]);
            }
            if (t < lim) {
                const float4 a = *reinterpret_cast<const float4*>(vi + t), x = *reinterpret_cast<const float4*>(w + p + t);
                s[v][0] = fmaf(a.x, x.x, s[v][0]); s[v][1] = fmaf(a.y, x.y, s[v][1]);
                s[v][2] = fmaf(a.z, x.z, s[v][2]); s[v][3] = fmaf(a.w, x.w, s[v][3]);
            }
        }
    }
#pragma unroll
    for (int v = 0; v < 3; v++) {
        const int i = warp + v * (AR_T / 32);
        if (i >= cnt) break;
        double d = 0.0;
#pragma unroll
        for (int c = 0; c < 8; c++) d += (double)s[v][c];
        d = ar_warp_sum(d);
        if (lane == 0) part[i] = d;
    }
}

__device__ __forceinline__ int ar_parts(const ArnoldiArgs& a, int64_t t) {
    if (a.kb == 0) return a.splits;
    const int tile = (int)(t >> 7);
    return ((tile + 1) * a.kb - 1) / a.per - tile * a.kb / a.per + 1;
}

template <bool VEC>
__global__ void __launch_bounds__(AR_T) batch_arnoldi_kernel(ArnoldiArgs a) {
    extern __shared__ __align__(16) float ar_w[];
    __shared__ double red[AR_T / 32][3];
    // the slice, then partial and full sums and the column (ar_vectors() each)
    double* part = reinterpret_cast<double*>(ar_w + a.slice);
    double* full = part + ar_vectors(a.m);
    double* h1 = full + ar_vectors(a.m);
    F2* hc = reinterpret_cast<F2*>(h1 + ar_vectors(a.m));
    cg::cluster_group cl = cg::this_cluster();
    const int64_t r = blockIdx.x / cl.num_blocks();
    const int rank = (int)cl.block_rank();
    const int64_t t0 = rank * a.slice;
    const int len = (int)lmax(0, lmin(a.slice, a.n - t0));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cnt = a.j + 1;
    const int64_t stride = a.k * a.n;
    const float* V = a.V + r * a.n + t0;
    float* w = ar_w;
    // the product
    const float* p = a.P + r * a.n + t0;
    if (VEC) {
        for (int t = 4 * threadIdx.x; t < len; t += 4 * AR_T) {
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const int parts = ar_parts(a, t0 + t);
            for (int s = 0; s < parts; s++) {
                const float4 q = *reinterpret_cast<const float4*>(p + s * a.split_stride + t);
                x.x += q.x; x.y += q.y; x.z += q.z; x.w += q.w;
            }
            *reinterpret_cast<float4*>(w + t) = x;
        }
    } else {
        for (int t = threadIdx.x; t < len; t += AR_T) {
            float x = 0.0f;
            const int parts = ar_parts(a, t0 + t);
            for (int s = 0; s < parts; s++) x += p[s * a.split_stride + t];
            w[t] = x;
        }
    }
    __syncthreads();
    // rigid translations: the mean of each component over the u-ranges
    if (a.ur.n > 0) {
        float sh[3] = {0, 0, 0}, sl[3] = {0, 0, 0};
        int64_t nodes = 0;
        for (int q = 0; q < a.ur.n; q++) {
            nodes += a.ur.len[q] / 3;
            const int64_t lo = lmax(a.ur.off[q], t0), hi = lmin(a.ur.off[q] + a.ur.len[q], t0 + len);
            for (int64_t t = lo + threadIdx.x; t < hi; t += AR_T) {
                const int c = (int)((t - a.ur.off[q]) % 3);
                const float x = w[t - t0];
                if (c == 0) ar_two_sum(sh[0], sl[0], x);
                else if (c == 1) ar_two_sum(sh[1], sl[1], x);
                else ar_two_sum(sh[2], sl[2], x);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double s = ar_warp_sum((double)sh[c] + (double)sl[c]);
            if (lane == 0) red[warp][c] = s;
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            double s = 0.0;
            for (int v = 0; v < AR_T / 32; v++) s += red[v][threadIdx.x];
            part[threadIdx.x] = s;
        }
        ar_cluster_sum(cl, part, full, 3);
        // three threads divide: an FP64 instruction of all eight warps takes 128 cycles of the SM
        if (threadIdx.x < 3) hc[threadIdx.x] = split_d(nodes > 0 ? full[threadIdx.x] / (double)nodes : 0.0);
        __syncthreads();
        const F2 mean[3] = {hc[0], hc[1], hc[2]};
        for (int q = 0; q < a.ur.n; q++) {
            const int64_t lo = lmax(a.ur.off[q], t0), hi = lmin(a.ur.off[q] + a.ur.len[q], t0 + len);
            for (int64_t t = lo + threadIdx.x; t < hi; t += AR_T) {
                const int c = (int)((t - a.ur.off[q]) % 3);
                const F2 mc = c == 0 ? mean[0] : c == 1 ? mean[1] : mean[2];
                float x = w[t - t0], l = -mc.lo;
                ar_two_sum(x, l, -mc.hi);
                w[t - t0] = __fadd_rn(x, l);
            }
        }
        __syncthreads();
    }
    // classical Gram-Schmidt, twice
    const bool fused = VEC && cnt <= AR_FUSED;
    for (int pass = 0; pass < 2; pass++) {
        if (pass == 0 || !fused) ar_dots<VEC>(V, stride, w, len, cnt, part);
        ar_cluster_sum(cl, part, full, cnt);
        for (int i = threadIdx.x; i < cnt; i += AR_T) {
            h1[i] = pass ? h1[i] + full[i] : full[i];
            hc[i] = split_d(-full[i]);
        }
        __syncthreads();
        if (pass == 0 && fused) ar_subtract_dots(V, stride, w, len, cnt, hc, part);
        else ar_subtract<VEC>(V, stride, w, len, cnt, hc);
        __syncthreads();
    }
    // the norm
    {
        float sh = 0.0f, sl = 0.0f;
        for (int t = threadIdx.x; t < len; t += AR_T) df_acc(sh, sl, w[t], w[t], 0.0f);
        const double s = ar_warp_sum((double)sh + (double)sl);
        if (lane == 0) red[warp][0] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            double v = 0.0;
            for (int q = 0; q < AR_T / 32; q++) v += red[q][0];
            part[0] = v;
        }
        ar_cluster_sum(cl, part, full, 1);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double nrm = sqrt(full[0]);
        full[0] = nrm;
        hc[0] = split_d(nrm > 0.0 ? 1.0 / nrm : 0.0);
    }
    __syncthreads();
    // the next basis vector and its operand
    const F2 inv = hc[0];
    float* vn = a.V + ((int64_t)(a.j + 1) * a.k + r) * a.n + t0;
    uint16_t* vb = a.Vbf + r * a.ldbf + t0;
    for (int t = threadIdx.x; t < len; t += AR_T) {
        const float v = fmaf(w[t], inv.hi, w[t] * inv.lo);
        vn[t] = v;
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        const uint16_t hb = __bfloat16_as_ushort(h);
        vb[t] = hb;
        if (a.panels > 1) vb[a.ldp + t] = __bfloat16_as_ushort(__float2bfloat16_rn(v - __bfloat162float(h)));
        if (a.panels > 2) vb[2 * a.ldp + t] = hb;
    }
    // the column's rotations, by one thread of the right-hand side
    if (rank == 0 && threadIdx.x == 0) {
        const int j = a.j;
        const double nrm = full[0];
        double col = h1[0];
        for (int i = 0; i < j; i++) {
            const double c = a.cs[i * a.k + r], s = a.sn[i * a.k + r], x = h1[i + 1];
            a.H[((int64_t)i * a.m + j) * a.k + r] = c * col + s * x;
            col = -s * col + c * x;
        }
        const double den = hypot(col, nrm);
        const double c = den > 0.0 ? fabs(col) / den : 1.0;
        const double s = den > 0.0 ? (col >= 0.0 ? 1.0 : -1.0) * nrm / den : 0.0;
        a.cs[j * a.k + r] = c;
        a.sn[j * a.k + r] = s;
        a.H[((int64_t)j * a.m + j) * a.k + r] = c * col + s * nrm;
        const double gj = a.g[j * a.k + r];
        const double gn = -s * gj;
        a.g[j * a.k + r] = c * gj;
        a.g[(j + 1) * a.k + r] = gn;
        const double b = a.beta[r];
        const double rel = b > 0.0 ? fabs(gn) / b : 0.0;
        if (!(rel < a.rtol)) atomicAdd(a.left, 1);
    }
}

// Y[i k + r] of the upper triangular H (cnt columns) and g; a zero pivot gives zero
__global__ void batch_backsolve_kernel(const double* __restrict__ H, const double* __restrict__ g, int m, int cnt,
                                       int64_t k, double* __restrict__ Y) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= k) return;
    for (int i = cnt - 1; i >= 0; i--) {
        double s = 0.0;
        for (int l = i + 1; l < cnt; l++) s += H[((int64_t)i * m + l) * k + r] * Y[l * k + r];
        const double d = H[((int64_t)i * m + i) * k + r];
        Y[i * k + r] = d != 0.0 ? (g[i * k + r] - s) / d : 0.0;
    }
}

}  // namespace mbem

using namespace mbem;

extern "C" {

int mbem_batch_arnoldi(const float* P, int splits, int kb, int per, int64_t split_stride, float* V, int j, int m, int64_t k, int64_t n,
                       const int64_t* u_ranges, int n_u_ranges, uint16_t* Vbf, int64_t ldbf, int64_t ldp, int panels,
                       double* H, double* cs, double* sn, double* g, const double* beta, double rtol, int* left,
                       void* stream) {
    MBEM_REQUIRE(P && V && Vbf && H && cs && sn && g && beta && left && k >= 1 && n >= 1, MBEM_ERR_ARG,
                 "bad batched Arnoldi arguments");
    MBEM_REQUIRE(kb == 0 ? splits >= 1 : kb > 0 && per > 0, MBEM_ERR_ARG, "bad batched Arnoldi partial sums");
    MBEM_REQUIRE(j >= 0 && j < m, MBEM_ERR_ARG, "batched Arnoldi: step %d of %d", j, m);
    MBEM_REQUIRE(panels >= 1 && panels <= 3 && ldp >= n && ldbf >= panels * ldp && split_stride >= (kb > 0 || splits > 1 ? k * n : 0),
                 MBEM_ERR_ARG, "bad batched Arnoldi strides");
    ArnoldiArgs a;
    int e = make_ranges(u_ranges, n_u_ranges, a.ur);
    if (e) return e;
    a.P = P; a.splits = splits; a.kb = kb; a.per = per; a.split_stride = split_stride; a.V = V; a.j = j; a.m = m; a.k = k; a.n = n;
    a.Vbf = Vbf; a.ldbf = ldbf; a.ldp = ldp; a.panels = panels; a.H = H; a.cs = cs; a.sn = sn; a.g = g; a.beta = beta;
    a.rtol = rtol; a.left = left;
    // blocks a cluster: a slice fits twice an SM, and there are two blocks an SM
    int ranks = 1;
    while (ranks < 8 && (ceil_div(n, ranks) > AR_SLICE || k * ranks < 2 * 152) && n / (2 * ranks) >= 1024) ranks *= 2;
    a.slice = ceil_div(ceil_div(n, ranks), 4) * 4;
    const size_t smem = (size_t)a.slice * sizeof(float) + (size_t)ar_vectors(m) * (3 * sizeof(double) + sizeof(F2));
    MBEM_REQUIRE(smem <= AR_SMEM, MBEM_ERR_SIZE, "batched Arnoldi: %d vectors of %lld entries", m, (long long)n);
    const bool vec = n % 4 == 0 && split_stride % 4 == 0 && ((uintptr_t)P | (uintptr_t)V) % 16 == 0;
    auto kernel = vec ? batch_arnoldi_kernel<true> : batch_arnoldi_kernel<false>;
    // the limit is the kernel's, shared by all host threads: always its largest
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AR_SMEM);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(k * ranks));
    cfg.blockDim = dim3(AR_T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ranks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t ce = cudaLaunchKernelEx(&cfg, kernel, a);
    if (ce != cudaSuccess) return set_error(MBEM_ERR_CUDA, "batch_arnoldi_kernel: %s", cudaGetErrorString(ce));
    return launch_status("batch_arnoldi_kernel");
}

int mbem_batch_backsolve(const double* H, const double* g, int m, int cnt, int64_t k, double* Y, void* stream) {
    MBEM_REQUIRE(H && g && Y && cnt >= 1 && cnt <= m && k >= 1, MBEM_ERR_ARG, "bad batched back substitution");
    batch_backsolve_kernel<<<(unsigned)ceil_div(k, 32), 32, 0, (cudaStream_t)stream>>>(H, g, m, cnt, k, Y);
    return launch_status("batch_backsolve_kernel");
}

}  // extern "C"
