// Nodal (P1/P2) contractions, FP64 (sm_103a): displacement and stress of a
// nodal density at observers, and the stress of listed pairs; the pair
// arithmetic is nodal_pair.cuh's.
//
// The sources are split over the blocks of a cluster and over the slices of a
// block: a few observers still fill the part, each partial sum has one owner
// and the sums are added in slice, then rank order through distributed shared
// memory (deterministic, no workspace). Bound by the FP64 pipe: the stress of a
// 16 x 16 P2 fault at 2,000 observers went from 266 to 5.97 ms (4.85 with far rules off by up
// to 2e-14, nd_far_rule).
#include <cooperative_groups.h>

#include "contract_split.cuh"
#include "nodal_launch.cuh"

namespace mbem {

namespace cg = cooperative_groups;

constexpr int NC_TILE = 32, NC_OBS = 16;              // sources a tile, most observers a block
constexpr int NC_T = 0, NC_U = 1, NC_STRESS = 2;      // kinds: T, U, 2 + MBEM_STRESS_*

template <int P>
struct NodalTile {
    NodalRec g;
    NodalDen<P> d;
};

template <int P, int KIND>
__device__ __forceinline__ void contract_pair(const NodalTile<P>& t, const double* x, const NodalArgs& a,
                                              const TCoef& tc, const SMat& m, double* acc) {
    if (KIND == NC_T) pair_t_contract<P>(t.g, t.d, x, tc, acc);
    else if (KIND == NC_U) pair_u_contract<P>(t.g, t.d, x, a.c, acc);
    else if (KIND == NC_STRESS + MBEM_STRESS_KELVIN) pair_kelvin_contract<P>(t.g, t.d, x, m, acc);
    else if (KIND == NC_STRESS + MBEM_STRESS_EIGEN) pair_eig_contract<P>(t.g, t.d, x, m, acc);
    else pair_dd_contract<P>(t.g, t.d, x, m, a.which == MBEM_STRESS_ELASTIC, acc, nullptr);
}

// ob observers a block, the source tiles dealt over the cluster's blocks. A
// tile's pairs are evaluated in the queue's order, each into its own place, and
// added to their observers in source order.
template <int P, int KIND>
__global__ void __launch_bounds__(ND_THREADS) nodal_contract_kernel(NodalArgs a, int ob) {
    extern __shared__ __align__(16) unsigned char nd_smem[];
    constexpr int NO = KIND <= NC_U ? 3 : 6;
    constexpr int FAR = KIND == NC_T ? NF_T : KIND == NC_U ? NF_U : KIND == NC_STRESS + MBEM_STRESS_KELVIN ? NF_S
                        : KIND == NC_STRESS + MBEM_STRESS_EIGEN ? NF_E : NF_H;
    __shared__ PairQueue queue;
    __shared__ double sum[NC_OBS * NO];
    __shared__ double xs[NC_OBS][3];
    NodalTile<P>* tile = reinterpret_cast<NodalTile<P>*>(nd_smem);
    double* val = reinterpret_cast<double*>(nd_smem + NC_TILE * sizeof(NodalTile<P>));     // (pair, NO)
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
    const int64_t f0 = (int64_t)(blockIdx.x / ranks) * ob;
    const int nf = (int)lmin(ob, a.n_field_pts - f0);
    for (int i = threadIdx.x; i < 3 * nf; i += ND_THREADS) xs[i / 3][i % 3] = a.x_field[3 * f0 + i];
    for (int i = threadIdx.x; i < nf * NO; i += ND_THREADS) sum[i] = 0.0;
    const TCoef tc = t_coef(a.c);
    const SMat m = stress_mat(a.mu, a.lam);
    constexpr int K = nd_nodes(P);
    for (int64_t s0 = (int64_t)rank * NC_TILE; s0 < a.n_src; s0 += (int64_t)ranks * NC_TILE) {
        const int ns = (int)lmin(NC_TILE, a.n_src - s0), total = ns * nf;
        __syncthreads();
        for (int t = threadIdx.x; t < ns; t += ND_THREADS) {
            const int64_t s = s0 + t;
            nodal_rec(a.tri_verts + 9 * s, a.normals ? a.normals + 3 * s : nullptr, a.eps[s], tile[t].g);
            nodal_den<P>(tile[t].g, a.density + 3 * K * s, tile[t].d);
        }
        __syncthreads();
        queue_pairs(queue, total, [&](int p) { return pair_class<P, FAR>(tile[p / nf].g, xs[p % nf]); });
        int p;
#pragma unroll 1
        while (queue_next(queue, total, p)) {
            if (p < 0) continue;
            const NodalTile<P>& T = tile[p / nf];
            double acc[NO];
#pragma unroll
            for (int i = 0; i < NO; i++) acc[i] = 0.0;
            if (T.g.ok && !T.d.zero) contract_pair<P, KIND>(T, xs[p % nf], a, tc, m, acc);
#pragma unroll
            for (int i = 0; i < NO; i++) val[p * NO + i] = acc[i];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nf * NO; i += ND_THREADS) {
            double v = sum[i];
            for (int t = 0; t < ns; t++) v += val[t * nf * NO + i];
            sum[i] = v;
        }
    }
    cluster.sync();
    if (rank == 0) {
        const int ix[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
        constexpr int NW = KIND <= NC_U ? 3 : 9;
        for (int i = threadIdx.x; i < nf * NO; i += ND_THREADS) {
            double v = sum[i];
            for (int r = 1; r < ranks; r++) v += *cluster.map_shared_rank(&sum[i], r);
            sum[i] = v;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nf * NW; i += ND_THREADS) {
            double* o = a.out + NW * f0 + i;
            const double v = a.alpha * sum[(i / NW) * NO + (NW == 3 ? i % NW : ix[i % NW])];
            *o = a.accumulate ? *o + v : v;
        }
    }
    cluster.sync();      // the partial sums stay until rank 0 has read them
}

// Listed (observer, source) pairs of a readout: the FP64 elastic stress
// (DD minus eigen) of the source's nodal slip density at the observer, nine
// components per pair; the mixed-precision readout sends its near pairs here.
template <int P>
__global__ void __launch_bounds__(ND_THREADS)
nodal_pairs_stress_kernel(NodalArgs a, const int64_t* __restrict__ pair_obs, const int32_t* __restrict__ pair_src,
                          int64_t n_pairs, double* __restrict__ out, double* __restrict__ out_eig) {
    const int64_t p = (int64_t)blockIdx.x * ND_THREADS + threadIdx.x;
    if (p >= n_pairs) return;
    const int64_t f = pair_obs[p], s = pair_src[p];
    double v[6] = {0, 0, 0, 0, 0, 0}, e[6] = {0, 0, 0, 0, 0, 0};
    NodalTile<P> t;
    nodal_rec(a.tri_verts + 9 * s, a.normals + 3 * s, a.eps[s], t.g);
    if (t.g.ok) {
        nodal_den<P>(t.g, a.density + 3 * nd_nodes(P) * s, t.d);
        if (!t.d.zero)
            pair_dd_contract<P>(t.g, t.d, a.x_field + 3 * f, stress_mat(a.mu, a.lam), true, v, out_eig ? e : nullptr);
    }
    const int ix[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
#pragma unroll
    for (int i = 0; i < 9; i++) out[9 * p + i] = v[ix[i]];
    if (out_eig)
#pragma unroll
        for (int i = 0; i < 9; i++) out_eig[9 * p + i] = e[ix[i]];
}

int nodal_pairs_stress(const double* x, const double* tv, const double* normals, const double* eps,
                       const double* density, double mu, double lam, int order, const int64_t* pair_obs,
                       const int32_t* pair_src, int64_t n_pairs, double* out, cudaStream_t st, double* out_eig) {
    MBEM_REQUIRE(order >= 0 && order <= 2, MBEM_ERR_ARG, "order must be 0, 1 or 2");
    int e = nodal_rules_ready();
    if (e) return e;
    if (n_pairs == 0) return MBEM_OK;
    NodalArgs a;
    memset(&a, 0, sizeof(a));
    a.x_field = x; a.tri_verts = tv; a.normals = normals; a.eps = eps; a.density = density;
    a.mu = mu; a.lam = lam;
    const unsigned grid = (unsigned)ceil_div(n_pairs, ND_THREADS);
    if (order == 0) nodal_pairs_stress_kernel<0><<<grid, ND_THREADS, 0, st>>>(a, pair_obs, pair_src, n_pairs, out, out_eig);
    else if (order == 1) nodal_pairs_stress_kernel<1><<<grid, ND_THREADS, 0, st>>>(a, pair_obs, pair_src, n_pairs, out, out_eig);
    else nodal_pairs_stress_kernel<2><<<grid, ND_THREADS, 0, st>>>(a, pair_obs, pair_src, n_pairs, out, out_eig);
    return launch_status("nodal_pairs_stress_kernel");
}

template <int P>
static constexpr size_t contract_smem(int kind, int ob) {
    return NC_TILE * (sizeof(NodalTile<P>) + (size_t)ob * (kind <= NC_U ? 3 : 6) * sizeof(double));
}

template <int P, typename Kernel>
static cudaError_t launch_contract_kernel(const cudaLaunchConfig_t& cfg, Kernel k, int kind, const NodalArgs& a, int ob) {
    // up to 47 KB of dynamic beside 3 KB of static shared memory (P2): four blocks an SM.
    // The limit is the kernel's, shared by all host threads: always its largest.
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)contract_smem<P>(kind, NC_OBS));
    return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, k, a, ob);
}

template <int P>
static cudaError_t launch_nodal_contract(int kind, const NodalArgs& a, unsigned grid, int ranks, int ob,
                                         cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(ND_THREADS);
    cfg.dynamicSmemBytes = contract_smem<P>(kind, ob);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ranks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    static_assert(NC_TILE * NC_OBS <= ND_TILE_PAIRS, "a tile's pairs fit its queue");
    switch (kind) {
        case NC_T: return launch_contract_kernel<P>(cfg, nodal_contract_kernel<P, NC_T>, kind, a, ob);
        case NC_U: return launch_contract_kernel<P>(cfg, nodal_contract_kernel<P, NC_U>, kind, a, ob);
        case NC_STRESS + MBEM_STRESS_KELVIN:
            return launch_contract_kernel<P>(cfg, nodal_contract_kernel<P, NC_STRESS + MBEM_STRESS_KELVIN>, kind, a, ob);
        case NC_STRESS + MBEM_STRESS_EIGEN:
            return launch_contract_kernel<P>(cfg, nodal_contract_kernel<P, NC_STRESS + MBEM_STRESS_EIGEN>, kind, a, ob);
        default:
            return launch_contract_kernel<P>(cfg, nodal_contract_kernel<P, NC_STRESS + MBEM_STRESS_DD>, kind, a, ob);
    }
}

int nodal_contract(int kind, const double* x, int64_t nf, const double* tv, const double* normals,
                   const double* eps, int64_t ns, const double* density, const double* coeffs, double mu,
                   double lam, int order, double alpha, int accumulate, double* out, void* stream) {
    MBEM_REQUIRE(order == 1 || order == 2, MBEM_ERR_ARG, "nodal order must be 1 or 2");
    int e = nodal_rules_ready();
    if (e) return e;
    NodalArgs a;
    memset(&a, 0, sizeof(a));
    a.x_field = x; a.n_field_pts = nf; a.tri_verts = tv; a.normals = normals; a.eps = eps; a.n_src = ns;
    a.density = density;
    for (int i = 0; i < 6; i++) a.c[i] = (coeffs && i < (kind == 0 ? 6 : 3)) ? coeffs[i] : 0.0;
    a.mu = kind >= NC_STRESS ? mu : 1.0;
    a.lam = kind >= NC_STRESS ? lam : 1.0;
    a.which = kind >= NC_STRESS ? kind - NC_STRESS : 0;
    a.alpha = alpha; a.accumulate = accumulate; a.out = out;
    if (nf == 0) return MBEM_OK;
    const ConSplit sp = contract_split(nf, ns, ND_THREADS, NC_OBS, NC_TILE, order == 1 ? 1200.0 : 2200.0, 600.0);
    const int ob = sp.ob, ranks = sp.ranks;
    const int64_t grid = ceil_div(nf, ob) * ranks;
    MBEM_REQUIRE(grid < (int64_t)1 << 31, MBEM_ERR_SIZE, "too many observers (%lld)", (long long)nf);
    const cudaError_t ce = order == 1 ? launch_nodal_contract<1>(kind, a, (unsigned)grid, ranks, ob, (cudaStream_t)stream)
                                      : launch_nodal_contract<2>(kind, a, (unsigned)grid, ranks, ob, (cudaStream_t)stream);
    if (ce != cudaSuccess) return set_error(MBEM_ERR_CUDA, "nodal_contract_kernel: %s", cudaGetErrorString(ce));
    return launch_status("nodal_contract_kernel");
}

}  // namespace mbem
