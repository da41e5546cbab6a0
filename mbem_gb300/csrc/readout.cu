// Mixed-precision stress readout of a nodal (P0/P1/P2) slip density at many
// points: the elastic stress (DD minus the exact eigenstress,
// evaluate.py:383-407 with subtract_anelastic) of every source at every
// observer, FP32 quadrature for the far pairs and the FP64 nodal machinery
// (nodal.cu) for the near ones.
//
// Far pairs: sum_q w_q H(x - y_q) s(y_q), s(y_q) = sum_k N_k(y_q) d_k, H the
// mollified point kernel of the DD stress (tri_kernels.py:901-964 with every
// moment replaced by its integrand) minus the eigenstress integrand
// (15 eps^4 / 8 pi) / R^7 C:sym(s n) (tri_kernels.py:1206-1214). Collapsed
// Gauss rules of 3 x 3, 5 x 5 and 8 x 8 points for D / L above 12, above 6
// and below (D = sqrt(|x - c|^2 + eps^2), L the longest edge). The offset
// x - c is formed in double-float and each point adds its FP32 offset from
// the centroid, so FP32 sees lengths of the size of the pair, not of the
// coordinates; a source's quadrature sum is FP32, the sum over sources FP64.
// Near pairs: D below near_factor * max(eps, L); listed per observer in
// source order (a count pass, a scan, a fill), evaluated in FP64, and added
// per observer in list order. Every sum runs in a fixed order.
#include <cooperative_groups.h>
#include <math.h>

#include <mutex>

#include "common.cuh"
#include "point_stress.cuh"

namespace mbem {

namespace cg = cooperative_groups;

constexpr int RO_Q0 = 9, RO_Q1 = 25, RO_Q2 = 64;
constexpr int RO_Q = RO_Q0 + RO_Q1 + RO_Q2;
constexpr int RO_HDR = 16;                    // c_hi[3], c_lo[3], n[3], eps, L, rnear2, pad
constexpr int RO_REC = RO_HDR + 8 * RO_Q;     // + per point: offset[3], weight, slip[3], pad
constexpr int RO_THREADS = 128;
constexpr int RO_TILE = 4;                    // sources staged in shared memory at a time, two tiles in turn
// Observers a block: halved down to 32 while there are fewer blocks than twelve rounds
// of resident ones (whole readout, 128 | 64 | 32 observers a block: 5,000 observers 4.3 |
// - | 3.2 ms, 20,000 7.5 | 6.7 | 6.3 ms, 100,000 22.8 | 22.1 | 22.3 ms).
constexpr int64_t RO_BLOCKS = 12 * 5 * 152;
constexpr int RO_RANKS = 8;                   // blocks of a cluster: they share the sources of their observers

__constant__ double c_ro_lam[RO_Q][3];
__constant__ double c_ro_w[RO_Q];

static std::mutex g_ro_mutex;
static bool g_ro_ready[64] = {false};

static void gauss_legendre_ro(int n, double* x, double* w) {
    for (int i = 0; i < n; i++) {
        double z = cos(MBEM_PI * (i + 0.75) / (n + 0.5));
        for (int it = 0; it < 100; it++) {
            double p0 = 1.0, p1 = z;
            for (int k = 2; k <= n; k++) {
                const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            const double dz = p1 / (n * (z * p1 - p0) / (z * z - 1.0));
            z -= dz;
            if (fabs(dz) < 1e-16) break;
        }
        double p0 = 1.0, p1 = z;
        for (int k = 2; k <= n; k++) {
            const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
            p0 = p1;
            p1 = p2;
        }
        const double dp = n * (z * p1 - p0) / (z * z - 1.0);
        x[i] = z;
        w[i] = 2.0 / ((1.0 - z * z) * dp * dp);
    }
}

static int ro_rules() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return set_error(MBEM_ERR_CUDA, "no current CUDA device for the readout rules");
    std::lock_guard<std::mutex> lock(g_ro_mutex);
    if (g_ro_ready[dev]) return MBEM_OK;
    static double lam[RO_Q][3], w[RO_Q];
    int q = 0;
    for (int n : {3, 5, 8}) {
        double g[8], gw[8];
        gauss_legendre_ro(n, g, gw);
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++) {
                const double gi = 0.5 * (g[i] + 1.0), gj = 0.5 * (g[j] + 1.0);
                lam[q][0] = 1.0 - gi - gj * (1.0 - gi);
                lam[q][1] = gi;
                lam[q][2] = gj * (1.0 - gi);
                w[q] = (0.5 * gw[i]) * (0.5 * gw[j]) * (1.0 - gi);
                q++;
            }
    }
    cudaError_t e = cudaMemcpyToSymbol(c_ro_lam, lam, sizeof(lam));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_ro_w, w, sizeof(w));
    if (e != cudaSuccess) return set_error(MBEM_ERR_CUDA, "readout rules: %s", cudaGetErrorString(e));
    g_ro_ready[dev] = true;
    return MBEM_OK;
}

struct Lattice {
    int order, K;
    int a[6][3];
};

// per-source record: centroid (double-float), normal, eps, L, near radius^2,
// and the three rules' points (offset from the centroid, weight x 2 area,
// interpolated slip)
// A thread a (source, point), the header by point 0's: 98 points a thread took
// 1.03 ms for 2,048 sources on 16 blocks, 0.12 ms now.
__global__ void readout_prep_kernel(const double* __restrict__ tv, const double* __restrict__ normals,
                                    const double* __restrict__ eps, const double* __restrict__ density,
                                    int64_t n_src, Lattice lat, double near_factor, float* __restrict__ rec) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n_src * RO_Q) return;
    const int64_t s = id / RO_Q;
    const int q = (int)(id - s * RO_Q);
    const double* v = tv + 9 * s;
    float* r = rec + s * RO_REC;
    double c[3];
    for (int k = 0; k < 3; k++) c[k] = ((v[k] + v[3 + k]) + v[6 + k]) / 3.0;
    if (q == 0) {
        for (int k = 0; k < 3; k++) {
            const float hi = (float)c[k];
            r[k] = hi;
            r[3 + k] = (float)(c[k] - (double)hi);
            r[6 + k] = (float)normals[3 * s + k];
        }
        double L = 0.0;
        for (int e = 0; e < 3; e++) {
            const int e2 = (e + 1) % 3;
            const double dx = v[3 * e2] - v[3 * e], dy = v[3 * e2 + 1] - v[3 * e + 1], dz = v[3 * e2 + 2] - v[3 * e + 2];
            L = fmax(L, sqrt(dx * dx + dy * dy + dz * dz));
        }
        const double ep = eps[s];
        const double rn = near_factor * fmax(ep, L);
        r[9] = (float)ep;
        r[10] = (float)L;
        r[11] = (float)(rn * rn);
        for (int k = 12; k < RO_HDR; k++) r[k] = 0.0f;
    }
    const double e1x = v[3] - v[0], e1y = v[4] - v[1], e1z = v[5] - v[2];
    const double e2x = v[6] - v[0], e2y = v[7] - v[1], e2z = v[8] - v[2];
    const double cx = e1y * e2z - e1z * e2y, cy = e1z * e2x - e1x * e2z, cz = e1x * e2y - e1y * e2x;
    const double area2 = sqrt(cx * cx + cy * cy + cz * cz);
    const double l0 = c_ro_lam[q][0], l1 = c_ro_lam[q][1], l2 = c_ro_lam[q][2];
    const double lam3[3] = {l0, l1, l2};
    float* pq = r + RO_HDR + 8 * q;
    for (int k = 0; k < 3; k++) pq[k] = (float)(((l0 * v[k] + l1 * v[3 + k]) + l2 * v[6 + k]) - c[k]);
    pq[3] = (float)(c_ro_w[q] * area2);
    double sl[3] = {0.0, 0.0, 0.0};
    for (int kk = 0; kk < lat.K; kk++) {
        double N = 1.0;
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < lat.a[kk][i]; j++) N *= (lat.order * lam3[i] - j) / (j + 1);
        const double* d = density + 3 * (lat.K * s + kk);
        sl[0] += N * d[0];
        sl[1] += N * d[1];
        sl[2] += N * d[2];
    }
    pq[4] = (float)sl[0];
    pq[5] = (float)sl[1];
    pq[6] = (float)sl[2];
    pq[7] = 0.0f;
}

// |x - c| in double-float, as FP32 components
__device__ __forceinline__ void df_offset(const double* x, const float* r, float d[3]) {
    for (int k = 0; k < 3; k++) {
        const float xh = (float)x[k];
        const float xl = (float)(x[k] - (double)xh);
        d[k] = __fadd_rn(__fsub_rn(xh, r[k]), __fsub_rn(xl, r[3 + k]));
    }
}

// the one near test (count and fill must agree exactly: no contraction)
__device__ __forceinline__ float pair_d2(const float d[3], float eps) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])), __fmul_rn(d[2], d[2])),
                     __fmul_rn(eps, eps));
}

// The near pairs of each observer: their number, or (FILL) the pairs themselves in
// source order. Headers are staged in shared memory: read in place (one a source, all
// lanes) the count took 0.59 ms for 100,000 observers x 2,048 sources, 0.18 ms now.
constexpr int RO_HTILE = 128;
template <bool FILL>
__global__ void __launch_bounds__(RO_THREADS)
readout_pairs_kernel(const double* __restrict__ x, int64_t n_obs, const float* __restrict__ rec, int64_t n_src,
                     int64_t* __restrict__ counts, const int64_t* __restrict__ rowptr,
                     int64_t* __restrict__ pair_obs, int32_t* __restrict__ pair_src) {
    __shared__ __align__(16) float hdr[RO_HTILE][12];
    const int64_t f = (int64_t)blockIdx.x * RO_THREADS + threadIdx.x;
    const bool live = f < n_obs;
    double xo[3] = {0.0, 0.0, 0.0};
    if (live)
        for (int k = 0; k < 3; k++) xo[k] = x[3 * f + k];
    int64_t slot = FILL && live ? rowptr[f] : 0;
    const int64_t slot_end = FILL && live ? rowptr[f + 1] : 0;
    for (int64_t s0 = 0; s0 < n_src; s0 += RO_HTILE) {
        const int ns = (int)lmin(RO_HTILE, n_src - s0);
        __syncthreads();
        for (int t = threadIdx.x; t < 3 * ns; t += RO_THREADS)
            *reinterpret_cast<float4*>(&hdr[t / 3][4 * (t % 3)]) =
                *reinterpret_cast<const float4*>(rec + (s0 + t / 3) * RO_REC + 4 * (t % 3));
        __syncthreads();
        if (!live) continue;
        for (int t = 0; t < ns; t++) {
            float d[3];
            df_offset(xo, hdr[t], d);
            if (pair_d2(d, hdr[t][9]) <= hdr[t][11]) {
                if (FILL && slot < slot_end) {
                    pair_obs[slot] = f;
                    pair_src[slot] = (int32_t)(s0 + t);
                }
                slot++;
            }
        }
    }
    if (!FILL && live) counts[f] = slot;
}

// rowptr = the exclusive scan of counts, one block, four entries a thread at a time
// (a strided run a thread took 110 us for 100,000 observers, 83 us now)
__global__ void __launch_bounds__(1024) ro_scan_kernel(const int64_t* __restrict__ counts, int64_t n,
                                                       int64_t* __restrict__ rowptr) {
    __shared__ int64_t wsum[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int64_t base = 0, next[4];
#pragma unroll
    for (int k = 0; k < 4; k++) next[k] = 4 * t + k < n ? counts[4 * t + k] : 0;
    for (int64_t i0 = 0; i0 < n; i0 += 4096) {
        const int64_t i = i0 + 4 * t;
        int64_t v[4], run = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = run;
            run += next[k];
            next[k] = i + 4096 + k < n ? counts[i + 4096 + k] : 0;
        }
        int64_t s = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (lane == 31) wsum[warp] = s;
        __syncthreads();
        int64_t w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        const int64_t before = __shfl_sync(0xffffffffu, w, max(warp - 1, 0));
        const int64_t all = __shfl_sync(0xffffffffu, w, 31);
        const int64_t off = base + (warp > 0 ? before : 0) + (s - run);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (i + k < n) rowptr[i + k] = off + v[k];
        base += all;
        __syncthreads();
    }
    if (t == 0) rowptr[n] = base;
}

__device__ __forceinline__ void ro_cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// Far pairs by quadrature; sources staged RO_TILE at a time in shared memory; with
// EIG the eigenstress of the far pairs goes to eig_out as well. Bound by the FP32 pipe
// (some 150 operations a point, 9 to 64 points a pair). Neighbouring observers take
// the same rule and so cost up to seven times others: a thread an observer for all
// 2,048 sources left half of the SMs idle at the end (22.5 ms for 100,000 observers,
// 17.1 ms now). A cluster's blocks take every RO_RANKS-th tile of their observers'
// sources, and where the observers are few a block's threads share them too; the
// FP64 sums are added in rank, then group order through distributed shared memory.
template <bool EIG>
__global__ void __launch_bounds__(RO_THREADS, 5)
readout_far_kernel(const double* __restrict__ x, int64_t n_obs, const float* __restrict__ rec, int64_t n_src,
                   RoMat mat, int ob, double alpha, int accumulate, double* __restrict__ out,
                   double* __restrict__ eig_out) {
    constexpr int NS = EIG ? 12 : 6;
    __shared__ __align__(16) float tile[2][RO_TILE * RO_REC];
    static_assert(sizeof(tile) >= NS * RO_THREADS * sizeof(double), "the sums reuse the tiles");
    cg::cluster_group cl = cg::this_cluster();
    const int ranks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    // ob observers a block: with fewer than its threads, groups share each tile
    const int groups = RO_THREADS / ob, group = (int)threadIdx.x / ob;
    const int64_t f0 = (int64_t)(blockIdx.x / ranks) * ob;
    const int64_t f = f0 + (int)threadIdx.x % ob;
    const bool live = f < n_obs;
    double xo[3] = {0.0, 0.0, 0.0};
    if (live)
        for (int k = 0; k < 3; k++) xo[k] = x[3 * f + k];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    double acc_e[6] = {0, 0, 0, 0, 0, 0};
    const int64_t step = (int64_t)ranks * RO_TILE;
    auto load = [&](int64_t s0, int b) {
        const int n4 = (int)lmax(0, lmin(RO_TILE, n_src - s0)) * (RO_REC / 4);
        const float4* src4 = reinterpret_cast<const float4*>(rec + s0 * RO_REC);
        float4* dst4 = reinterpret_cast<float4*>(tile[b]);
        for (int t = threadIdx.x; t < n4; t += RO_THREADS) ro_cp16(dst4 + t, src4 + t);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load((int64_t)rank * RO_TILE, 0);
    int b = 0;
    for (int64_t s0 = (int64_t)rank * RO_TILE; s0 < n_src; s0 += step, b ^= 1) {
        const int ns = (int)lmin(RO_TILE, n_src - s0);
        load(s0 + step, b ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        if (live)
            for (int t = group; t < ns; t += groups) {
                const float* r = tile[b] + t * RO_REC;
                float dc[3];
                df_offset(xo, r, dc);
                const float eps2 = r[9] * r[9];
                const float D2 = pair_d2(dc, r[9]);
                if (D2 <= r[11]) continue;                    // a near pair
                const float L2 = r[10] * r[10];
                int q0, q1;
                if (D2 > 144.0f * L2) { q0 = 0; q1 = RO_Q0; }
                else if (D2 > 36.0f * L2) { q0 = RO_Q0; q1 = RO_Q0 + RO_Q1; }
                else { q0 = RO_Q0 + RO_Q1; q1 = RO_Q; }
                const float nv[3] = {r[6], r[7], r[8]};
                float sym[6] = {0, 0, 0, 0, 0, 0};
                float sym_e[6] = {0, 0, 0, 0, 0, 0};
                for (int q = q0; q < q1; q++) {
                    const float4* pq = reinterpret_cast<const float4*>(r + RO_HDR + 8 * q);
                    const float4 o = pq[0], p = pq[1];
                    const float d[3] = {dc[0] - o.x, dc[1] - o.y, dc[2] - o.z};
                    const float u[3] = {p.x, p.y, p.z};
                    point_stress<EIG>(d, u, nv, o.w, eps2, mat, sym, sym_e);
                }
#pragma unroll
                for (int k = 0; k < 6; k++) acc[k] += (double)sym[k];
                if (EIG) {
#pragma unroll
                    for (int k = 0; k < 6; k++) acc_e[k] += (double)sym_e[k];
                }
            }
        __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    double* sums = reinterpret_cast<double*>(&tile[0][0]);
#pragma unroll
    for (int k = 0; k < 6; k++) {
        sums[k * RO_THREADS + threadIdx.x] = acc[k];
        if (EIG) sums[(6 + k) * RO_THREADS + threadIdx.x] = acc_e[k];
    }
    cl.sync();
    // each block finishes its share of the observers
    const int per = ob / ranks;
    const int t = rank * per + (int)threadIdx.x;
    if ((int)threadIdx.x < per && f0 + t < n_obs) {
        double s[NS];
#pragma unroll
        for (int k = 0; k < NS; k++) s[k] = 0.0;
        for (int r = 0; r < ranks; r++) {
            const double* p = cl.map_shared_rank(sums, r) + t;
            for (int g = 0; g < groups; g++, p += ob)
#pragma unroll
                for (int k = 0; k < NS; k++) s[k] += p[k * RO_THREADS];
        }
        constexpr int ix[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
        double* o = out + 9 * (f0 + t);
#pragma unroll
        for (int k = 0; k < 9; k++) o[k] = accumulate ? o[k] + alpha * s[ix[k]] : alpha * s[ix[k]];
        if (EIG) {
            double* oe = eig_out + 9 * (f0 + t);
#pragma unroll
            for (int k = 0; k < 9; k++) oe[k] = accumulate ? oe[k] + alpha * s[6 + ix[k]] : alpha * s[6 + ix[k]];
        }
    }
    cl.sync();      // the others' sums stay until every block has read them
}

template <bool EIG>
static int launch_far(const double* x, int64_t n_obs, const float* rec, int64_t n_src, const RoMat& m, double alpha,
                      int accumulate, double* out, double* eig_out, cudaStream_t st) {
    int ranks = RO_RANKS;
    while (ranks > 1 && n_src <= (int64_t)(ranks / 2) * RO_TILE) ranks /= 2;
    int ob = RO_THREADS;
    while (ob > 32 && ceil_div(n_obs, ob) * ranks < RO_BLOCKS) ob /= 2;
    const int64_t grid = ceil_div(n_obs, ob) * ranks;
    MBEM_REQUIRE(grid < INT32_MAX, MBEM_ERR_SIZE, "too many observers (%lld)", (long long)n_obs);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(RO_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ranks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t ce = cudaLaunchKernelEx(&cfg, readout_far_kernel<EIG>, x, n_obs, rec, n_src, m, ob, alpha,
                                              accumulate, out, eig_out);
    if (ce != cudaSuccess) return set_error(MBEM_ERR_CUDA, "readout_far_kernel: %s", cudaGetErrorString(ce));
    return launch_status("readout_far_kernel");
}

// out[f] += alpha * sum of its near pairs' stresses, in list order
__global__ void readout_near_add_kernel(const int64_t* __restrict__ rowptr, int64_t n_obs,
                                        const double* __restrict__ pair_out, double alpha, double* __restrict__ out) {
    const int64_t f = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (f >= n_obs) return;
    double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t p = rowptr[f]; p < rowptr[f + 1]; p++)
        for (int k = 0; k < 9; k++) s[k] += pair_out[9 * p + k];
    for (int k = 0; k < 9; k++) out[9 * f + k] += alpha * s[k];
}

static Lattice lattice_of(int order) {
    Lattice L;
    memset(&L, 0, sizeof(L));
    L.order = order;
    L.K = (order + 1) * (order + 2) / 2;
    if (order == 0) return L;
    int k = 0;
    for (int v = 0; v < 3; v++) {
        L.a[k][v] = order;
        k++;
    }
    const int ij[3][2] = {{0, 1}, {1, 2}, {2, 0}};
    for (int e = 0; e < 3; e++)
        for (int s = 1; s < order; s++) {
            L.a[k][ij[e][0]] = order - s;
            L.a[k][ij[e][1]] = s;
            k++;
        }
    return L;
}

}  // namespace mbem

using namespace mbem;

extern "C" {

size_t mbem_readout_record_bytes(int64_t n_src) { return (size_t)n_src * RO_REC * sizeof(float); }

int mbem_readout_prepare(const double* x, int64_t n_obs, const double* tri_verts, const double* normals,
                         const double* eps, int64_t n_src, const double* density, int order, double near_factor,
                         float* records, int64_t* counts, int64_t* rowptr, int64_t* n_near, void* stream) {
    MBEM_REQUIRE(n_obs >= 0 && n_src >= 0 && order >= 0 && order <= 2 && near_factor > 0.0, MBEM_ERR_ARG,
                 "bad readout sizes");
    MBEM_REQUIRE((n_obs == 0 || (x && rowptr)) && (n_src == 0 || (tri_verts && normals && eps && density && records)) &&
                     n_near,
                 MBEM_ERR_ARG, "NULL readout arrays");
    MBEM_REQUIRE(n_src < INT32_MAX, MBEM_ERR_SIZE, "too many sources");
    int e = ro_rules();
    if (e) return e;
    cudaStream_t st = (cudaStream_t)stream;
    if (n_src > 0) {
        readout_prep_kernel<<<(unsigned)ceil_div(n_src * RO_Q, 128), 128, 0, st>>>(
            tri_verts, normals, eps, density, n_src, lattice_of(order), near_factor, records);
        if ((e = launch_status("readout_prep_kernel"))) return e;
    }
    if (n_obs == 0) {
        cudaMemsetAsync(rowptr, 0, sizeof(int64_t), st);
        *n_near = 0;
        return launch_status("readout memset", 0);
    }
    MBEM_REQUIRE(counts != nullptr, MBEM_ERR_ARG, "NULL counts");
    readout_pairs_kernel<false><<<(unsigned)ceil_div(n_obs, RO_THREADS), RO_THREADS, 0, st>>>(
        x, n_obs, records, n_src, counts, nullptr, nullptr, nullptr);
    if ((e = launch_status("readout_pairs_kernel"))) return e;
    ro_scan_kernel<<<1, 1024, 0, st>>>(counts, n_obs, rowptr);
    if ((e = launch_status("ro_scan_kernel"))) return e;
    cudaMemcpyAsync(n_near, rowptr + n_obs, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return launch_status("readout sync", 0);
    return MBEM_OK;
}

int mbem_readout_evaluate(const double* x, int64_t n_obs, const double* tri_verts, const double* normals,
                          const double* eps, int64_t n_src, const double* density, double mu, double lam, int order,
                          const float* records, const int64_t* rowptr, int64_t n_near, int64_t* pair_obs,
                          int32_t* pair_src, double* pair_out, double alpha, int accumulate, double* out,
                          void* stream) {
    return mbem_readout_evaluate_parts(x, n_obs, tri_verts, normals, eps, n_src, density, mu, lam, order, records,
                                       rowptr, n_near, pair_obs, pair_src, pair_out, nullptr, alpha, accumulate, out,
                                       nullptr, stream);
}

int mbem_readout_evaluate_parts(const double* x, int64_t n_obs, const double* tri_verts, const double* normals,
                                const double* eps, int64_t n_src, const double* density, double mu, double lam,
                                int order, const float* records, const int64_t* rowptr, int64_t n_near,
                                int64_t* pair_obs, int32_t* pair_src, double* pair_out, double* pair_eig,
                                double alpha, int accumulate, double* out, double* eig_out, void* stream) {
    MBEM_REQUIRE(n_obs >= 0 && n_src >= 0 && n_near >= 0 && mu > 0.0 && lam + mu > 0.0, MBEM_ERR_ARG,
                 "bad readout arguments");
    MBEM_REQUIRE(n_obs == 0 || (x && rowptr && out), MBEM_ERR_ARG, "NULL readout arrays");
    MBEM_REQUIRE(n_near == 0 || (pair_obs && pair_src && pair_out), MBEM_ERR_ARG, "NULL near-pair arrays");
    MBEM_REQUIRE(!eig_out || n_near == 0 || pair_eig, MBEM_ERR_ARG, "the eigenstress needs its near-pair array");
    if (n_obs == 0) return MBEM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const RoMat m = make_romat(mu, lam);
    int e = eig_out ? launch_far<true>(x, n_obs, records, n_src, m, alpha, accumulate, out, eig_out, st)
                    : launch_far<false>(x, n_obs, records, n_src, m, alpha, accumulate, out, nullptr, st);
    if (e) return e;
    if (n_near == 0) return MBEM_OK;
    readout_pairs_kernel<true><<<(unsigned)ceil_div(n_obs, RO_THREADS), RO_THREADS, 0, st>>>(
        x, n_obs, records, n_src, nullptr, rowptr, pair_obs, pair_src);
    if ((e = launch_status("readout_pairs_kernel"))) return e;
    if ((e = nodal_pairs_stress(x, tri_verts, normals, eps, density, mu, lam, order, pair_obs, pair_src, n_near,
                                pair_out, st, eig_out ? pair_eig : nullptr)))
        return e;
    readout_near_add_kernel<<<(unsigned)ceil_div(n_obs, 256), 256, 0, st>>>(rowptr, n_obs, pair_out, alpha, out);
    if ((e = launch_status("readout_near_add_kernel"))) return e;
    if (!eig_out) return MBEM_OK;
    readout_near_add_kernel<<<(unsigned)ceil_div(n_obs, 256), 256, 0, st>>>(rowptr, n_obs, pair_eig, alpha, eig_out);
    return launch_status("readout_near_add_kernel");
}

}  // extern "C"
