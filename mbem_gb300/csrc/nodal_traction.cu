// Nodal traction rows (P0/P1/P2), FP64 (sm_103a): the stress per unit nodal
// density dotted with the field point's normal, columns scattered through an
// ids table (tri_nodal.py:1176-1227); the pair arithmetic is nodal_pair.cuh's.
// Entries are added atomically: a shared-node ids table maps several sources
// onto one column (the element-major table maps each entry once, so its result
// does not depend on the order of the adds).
//
// Bound by the FP64 pipe. 288 points x 6,144 P0 sources ("slip"): 70.2 ms with
// run-time tables in local memory and 144 / 64 far points, 4.26 ms now.
#include "nodal_launch.cuh"

namespace mbem {

// rows 3f .. 3f + 2 of one pair
template <int P, int F>
__device__ __forceinline__ void traction_pair(const NodalArgs& a, const NodalRec& g, int64_t f, int64_t s,
                                              const SMat& m, bool eig) {
    constexpr int K = nd_nodes(P);
    if (!g.ok) return;
    pair_traction<P, F>(g, a.x_field + 3 * f, a.n_field + 3 * f, m, eig, [&](int k, const double T[3][3]) {
        const int64_t id = a.ids ? a.ids[s * K + k] : s * K + k;
        if (id < 0 || id >= a.n_cols) return;        // outside the block: never written
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) atomicAdd(&a.out[(3 * f + i) * a.ld + 3 * id + j], a.alpha * T[i][j]);
    });
}

template <int P, int F>
__global__ void __launch_bounds__(ND_THREADS) nodal_traction_kernel(NodalArgs a, int sb, int fb) {
    extern __shared__ __align__(16) unsigned char nd_smem[];
    __shared__ PairQueue queue;
    NodalRec* recs = reinterpret_cast<NodalRec*>(nd_smem);
    const int64_t s0 = (int64_t)blockIdx.x * sb;
    const int ns = (int)lmin(sb, a.n_src - s0);
    load_recs(a, s0, ns, recs);
    __syncthreads();
    const SMat m = stress_mat(a.mu, a.lam);
    for (int64_t f0 = (int64_t)blockIdx.y * fb; f0 < a.n_field_pts; f0 += (int64_t)gridDim.y * fb) {
        const int nf = (int)lmin(fb, a.n_field_pts - f0), total = ns * nf;
        queue_pairs(queue, total, [&](int p) {
            const int t = p / nf;
            return pair_class<P, F>(recs[t], a.x_field + 3 * (f0 + (p - t * nf)));
        });
        int p;
#pragma unroll 1
        while (queue_next(queue, total, p)) {
            if (p < 0) continue;
            const int t = p / nf;
            traction_pair<P, F>(a, recs[t], f0 + (p - t * nf), s0 + t, m, a.which == TR_SLIP);
        }
        __syncthreads();      // the queue is read until every warp is here
    }
}

// listed pairs of an order-0 source patch
template <int F>
__global__ void __launch_bounds__(ND_THREADS) traction_pairs_kernel(NodalArgs a) {
    const int64_t q = (int64_t)blockIdx.x * ND_THREADS + threadIdx.x;
    if (q >= a.n_pairs) return;
    const int64_t f = pair_row(a.pair_rowptr, a.n_field_pts, q), s = a.pair_cols[q];
    NodalRec g;
    nodal_rec(a.tri_verts + 9 * s, a.normals ? a.normals + 3 * s : nullptr, a.eps[s], g);
    traction_pair<0, F>(a, g, f, s, stress_mat(a.mu, a.lam), a.which == TR_SLIP);
}

template <int P>
static void launch_traction(const NodalArgs& a, const PairTiles& t, cudaStream_t st) {
    // slip and total share the DD tables (tri_nodal.py:1367 _TRACTION_KINDS)
    if (a.which == TR_FORCE) nodal_traction_kernel<P, NF_S><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb);
    else if (a.which == TR_EIGEN) nodal_traction_kernel<P, NF_E><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb);
    else nodal_traction_kernel<P, NF_H><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb);
}

// FP64 traction blocks of listed (field point, source) pairs of an order-0
// source patch (the near pairs of the mixed operator's traction rows), added
// into out at column 3 s + j: the per-pair code of mbem_traction_matrix.
int traction_pairs(const double* x_field, const double* n_field, int64_t n_pts, const double* tri_verts,
                   const double* normals, const double* eps, int64_t n_src, double mu, double lam, int which,
                   double alpha, const int64_t* rowptr, const int64_t* cols, int64_t nnz, double* out, int64_t ld,
                   cudaStream_t st) {
    int e = nodal_rules_ready();
    if (e) return e;
    NodalArgs a;
    memset(&a, 0, sizeof(a));
    a.x_field = x_field; a.n_field = n_field; a.n_field_pts = n_pts; a.tri_verts = tri_verts;
    a.normals = normals; a.eps = eps; a.n_src = n_src; a.n_cols = n_src;
    a.mu = mu; a.lam = lam; a.alpha = alpha; a.which = which; a.out = out; a.ld = ld;
    a.pair_rowptr = rowptr; a.pair_cols = cols; a.n_pairs = nnz;
    if (nnz == 0) return MBEM_OK;
    const unsigned grid = (unsigned)ceil_div(nnz, ND_THREADS);
    if (which == TR_FORCE) traction_pairs_kernel<NF_S><<<grid, ND_THREADS, 0, st>>>(a);
    else if (which == TR_EIGEN) traction_pairs_kernel<NF_E><<<grid, ND_THREADS, 0, st>>>(a);
    else traction_pairs_kernel<NF_H><<<grid, ND_THREADS, 0, st>>>(a);
    return launch_status("traction_pairs_kernel");
}

}  // namespace mbem

extern "C" int mbem_traction_matrix(const double* x_field, const double* n_field, int64_t n_pts,
                                    const double* tri_verts, const double* normals, const double* eps,
                                    int64_t n_src, const int64_t* ids, int64_t n_cols, double mu, double lam,
                                    int order, int which, double alpha, double* out, int64_t ld_out,
                                    void* stream) {
    using namespace mbem;
    MBEM_REQUIRE(order >= 0 && order <= 2, MBEM_ERR_ARG, "order must be 0, 1 or 2 (got %d)", order);
    MBEM_REQUIRE(which >= 0 && which <= 3, MBEM_ERR_ARG, "which must be 0..3 (got %d)", which);
    MBEM_REQUIRE(n_pts >= 0 && n_src >= 0 && n_cols >= 0 && ld_out >= 3 * n_cols, MBEM_ERR_ARG,
                 "bad traction shape");
    MBEM_REQUIRE(n_src == 0 || (tri_verts && (normals || which == 1) && eps && ids), MBEM_ERR_ARG,
                 "NULL source arrays");
    MBEM_REQUIRE(n_pts == 0 || (x_field && n_field && out), MBEM_ERR_ARG, "NULL field arrays");
    MBEM_REQUIRE(mu > 0.0 && lam + mu > 0.0, MBEM_ERR_ARG, "material (mu=%g, lam=%g)", mu, lam);
    int e = nodal_rules_ready();
    if (e) return e;
    NodalArgs a;
    memset(&a, 0, sizeof(a));
    a.x_field = x_field; a.n_field = n_field; a.n_field_pts = n_pts; a.tri_verts = tri_verts;
    a.normals = normals; a.eps = eps; a.n_src = n_src; a.ids = ids; a.n_cols = n_cols;
    a.mu = mu; a.lam = lam; a.alpha = alpha; a.which = which; a.out = out; a.ld = ld_out;
    if (n_pts == 0 || n_src == 0) return MBEM_OK;
    const PairTiles t = pair_tiles(n_pts, n_src);
    cudaStream_t st = (cudaStream_t)stream;
    if (order == 0) launch_traction<0>(a, t, st);
    else if (order == 1) launch_traction<1>(a, t, st);
    else launch_traction<2>(a, t, st);
    return launch_status("nodal_traction_kernel");
}
