// Nodal (Lagrange P1/P2) kernel matrices and listed near blocks, FP64 (sm_103a);
// the pair arithmetic is nodal_pair.cuh's. A block holds the records of a few
// sources in shared memory (frame, edges, shape coefficients: made once per
// block) and its threads take (field point, source) pairs of them.
//
// Bound by the FP64 pipe. Against one thread per pair with run-time degrees and
// tables in local memory (the 32-term series and about 12 KB a thread before),
// the 8-per-face cube's P1 T block (1.77e6 pairs) went from 63.2 to 4.1 ms,
// a ragged P2 U block (1,001 x 333) from 26.9 to 1.4 ms.
#include "nodal_launch.cuh"

namespace mbem {

enum { ND_T = 0, ND_U = 1, ND_TBASIS = 2, ND_UBASIS = 3 };

template <int P, int KIND>
__global__ void __launch_bounds__(ND_THREADS) nodal_matrix_kernel(NodalArgs a, int sb, int fb) {
    extern __shared__ __align__(16) unsigned char nd_smem[];
    __shared__ PairQueue queue;
    NodalRec* recs = reinterpret_cast<NodalRec*>(nd_smem);
    constexpr int K = nd_nodes(P), FAR = KIND == ND_T || KIND == ND_UBASIS ? NF_T : KIND == ND_U ? NF_U : NF_H;
    const int64_t s0 = (int64_t)blockIdx.x * sb;
    const int ns = (int)lmin(sb, a.n_src - s0);
    load_recs(a, s0, ns, recs);
    __syncthreads();
    const TCoef tc = t_coef(a.c);
    for (int64_t f0 = (int64_t)blockIdx.y * fb; f0 < a.n_field_pts; f0 += (int64_t)gridDim.y * fb) {
        const int nf = (int)lmin(fb, a.n_field_pts - f0), total = ns * nf;
        queue_pairs(queue, total, [&](int p) {
            const int t = p / nf;
            return pair_class<P, FAR>(recs[t], a.x_field + 3 * (f0 + (p - t * nf)));
        });
        int p;
#pragma unroll 1
        while (queue_next(queue, total, p)) {
            if (p < 0) continue;
            const int t = p / nf;
            const int64_t f = f0 + (p - t * nf), s = s0 + t;
            const NodalRec& g = recs[t];
            double* row = a.out + 3 * f * a.ld + 3 * K * s;
            const double* x = a.x_field + 3 * f;
            if (KIND == ND_T) {
                auto put = [&](int k, const double G[3][3]) {
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            double* q = row + i * a.ld + 3 * k + j;
                            const double v = a.alpha * G[i][j];
                            *q = a.accumulate ? *q + v : v;
                        }
                };
                const double zero[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
                if (g.ok) pair_t_block<P>(g, x, tc, put);
                else
                    for (int k = 0; k < K; k++) put(k, zero);
            } else if (KIND == ND_U) {
                auto put = [&](int k, double I1, double I3, const double* G) {
                    const double d = a.c[0] * I1 + a.c[1] * g.eps2 * I3;
                    const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) {
                            double* q = row + i * a.ld + 3 * k + j;
                            const double v = a.alpha * (G[ix[i][j]] + (i == j ? d : 0.0));
                            *q = a.accumulate ? *q + v : v;
                        }
                };
                const double zero[6] = {0, 0, 0, 0, 0, 0};
                if (g.ok) pair_u<P, FAR>(g, x, a.c[2], put);
                else
                    for (int k = 0; k < K; k++) put(k, 0.0, 0.0, zero);
            } else if (KIND == ND_TBASIS) {
                auto put = [&](int k, const double blk[6][3][3]) {
                    for (int b = 0; b < 6; b++)
                        for (int i = 0; i < 3; i++)
                            for (int j = 0; j < 3; j++) row[b * a.plane + i * a.ld + 3 * k + j] = blk[b][i][j];
                };
                if (g.ok) {
                    pair_t_basis<P>(g, x, put);
                } else {
                    const double zero[6][3][3] = {};
                    for (int k = 0; k < K; k++) put(k, zero);
                }
            } else {
                auto put = [&](int k, double I1, double I3, const double* G) {
                    const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
                    for (int i = 0; i < 3; i++)
                        for (int j = 0; j < 3; j++) {
                            double* q = row + i * a.ld + 3 * k + j;
                            q[0] = (i == j) ? I1 : 0.0;
                            q[a.plane] = (i == j) ? g.eps2 * I3 : 0.0;
                            q[2 * a.plane] = G[ix[i][j]];
                        }
                };
                const double zero[6] = {0, 0, 0, 0, 0, 0};
                if (g.ok) pair_u<P, FAR>(g, x, 1.0, put);
                else
                    for (int k = 0; k < K; k++) put(k, 0.0, 0.0, zero);
            }
        }
        __syncthreads();      // the queue is read until every warp is here
    }
}

// The FP64 nodal blocks of listed near pairs (the mixed operator's near
// field at order 1/2): pair q = (field point f, source s) from a CSR by field
// point; node k's 3x3 block goes to vals[(K q + k) * 9], the layout of the
// node-level near list (columns K s + k).
template <int P, int KIND>
__global__ void __launch_bounds__(ND_THREADS) nodal_near_eval_kernel(NodalArgs a, double* __restrict__ vals) {
    const int64_t q = (int64_t)blockIdx.x * ND_THREADS + threadIdx.x;
    if (q >= a.n_pairs) return;
    constexpr int K = nd_nodes(P);
    const int64_t f = pair_row(a.pair_rowptr, a.n_field_pts, q), s = a.pair_cols[q];
    NodalRec g;
    nodal_rec(a.tri_verts + 9 * s, a.normals ? a.normals + 3 * s : nullptr, a.eps[s], g);
    double* o = vals + 9 * K * q;
    if (!g.ok) {
        for (int e = 0; e < 9 * K; e++) o[e] = 0.0;
        return;
    }
    const double* x = a.x_field + 3 * f;
    if (KIND == ND_T) {
        pair_t_block<P>(g, x, t_coef(a.c), [&](int k, const double G[3][3]) {
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) o[9 * k + 3 * i + j] = a.alpha * G[i][j];
        });
    } else {
        pair_u<P, NF_U>(g, x, a.c[2], [&](int k, double I1, double I3, const double* G) {
            const double d = a.c[0] * I1 + a.c[1] * g.eps2 * I3;
            const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) o[9 * k + 3 * i + j] = a.alpha * (G[ix[i][j]] + (i == j ? d : 0.0));
        });
    }
}

template <int P>
static void launch_nodal_matrix(int kind, const NodalArgs& a, const PairTiles& t, cudaStream_t st) {
    switch (kind) {
        case ND_T: nodal_matrix_kernel<P, ND_T><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb); break;
        case ND_U: nodal_matrix_kernel<P, ND_U><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb); break;
        case ND_TBASIS: nodal_matrix_kernel<P, ND_TBASIS><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb); break;
        default: nodal_matrix_kernel<P, ND_UBASIS><<<t.grid, ND_THREADS, t.smem, st>>>(a, t.sb, t.fb); break;
    }
}

int nodal_matrix(int kind, const double* x, int64_t nf, const double* tv, const double* normals,
                 const double* eps, int64_t ns, const double* coeffs, int order, double alpha, int accumulate,
                 double* out, int64_t ld, void* stream) {
    MBEM_REQUIRE(order == 1 || order == 2, MBEM_ERR_ARG, "nodal order must be 1 or 2");
    int e = nodal_rules_ready();
    if (e) return e;
    const int K = nd_nodes(order);
    NodalArgs a;
    memset(&a, 0, sizeof(a));
    a.x_field = x; a.n_field_pts = nf; a.tri_verts = tv; a.normals = normals; a.eps = eps; a.n_src = ns;
    const int nc = (kind == 0) ? 6 : (kind == 1 ? 3 : 0);
    for (int i = 0; i < 6; i++) a.c[i] = (coeffs && i < nc) ? coeffs[i] : 0.0;
    a.alpha = alpha; a.accumulate = accumulate; a.out = out;
    a.ld = (kind >= 2) ? 3 * K * ns : ld;
    a.plane = 3 * nf * 3 * K * ns;
    MBEM_REQUIRE(kind >= 2 || ld >= 3 * K * ns, MBEM_ERR_ARG, "ld_out %lld < 3*K*n_src", (long long)ld);
    if (nf * ns == 0) return MBEM_OK;
    const PairTiles t = pair_tiles(nf, ns);
    if (order == 1) launch_nodal_matrix<1>(kind, a, t, (cudaStream_t)stream);
    else launch_nodal_matrix<2>(kind, a, t, (cudaStream_t)stream);
    return launch_status("nodal_matrix_kernel");
}

// *flag = 1 where a triangle's height over its longest edge is not above `limit`: the
// host asks before each nodal call, and copying the vertices back to judge them there
// took 150 us for 333 triangles.
__global__ void shape_screen_kernel(const double* __restrict__ tv, int64_t n, double limit, int* flag) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double* v = tv + 9 * s;
    double e0[3], e1[3], e2[3];
    for (int k = 0; k < 3; k++) {
        e0[k] = v[3 + k] - v[k];
        e1[k] = v[6 + k] - v[3 + k];
        e2[k] = v[k] - v[6 + k];
    }
    const double l0 = e0[0] * e0[0] + e0[1] * e0[1] + e0[2] * e0[2], l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2],
                 l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
    const double L2 = fmax(fmax(l0, l1), l2);
    const double c0 = e0[1] * e2[2] - e0[2] * e2[1], c1 = e0[2] * e2[0] - e0[0] * e2[2],
                 c2 = e0[0] * e2[1] - e0[1] * e2[0];
    const double area2 = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
    if (!(area2 >= limit * (1.0 + 1e-9) * L2) || !(L2 > 0.0)) *flag = 1;
}

}  // namespace mbem

extern "C" int mbem_shape_screen(const double* tri_verts, int64_t n, double limit, int* suspect, void* stream) {
    using namespace mbem;
    MBEM_REQUIRE(suspect && n >= 0 && (n == 0 || tri_verts), MBEM_ERR_ARG, "bad shape screen arguments");
    *suspect = 0;
    if (n == 0) return MBEM_OK;
    // one pinned word a host thread, for the thread's life: the kernel writes it directly
    struct Flag {
        int* p = nullptr;
        ~Flag() {
            if (p) cudaFreeHost(p);
        }
    };
    thread_local Flag flag;
    if (!flag.p && cudaHostAlloc(reinterpret_cast<void**>(&flag.p), sizeof(int),
                                 cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        flag.p = nullptr;
        return set_error(MBEM_ERR_CUDA, "shape screen: %s", cudaGetErrorString(cudaGetLastError()));
    }
    MBEM_REQUIRE(ceil_div(n, 128) < INT32_MAX, MBEM_ERR_SIZE, "too many triangles");
    *flag.p = 0;
    shape_screen_kernel<<<(unsigned)ceil_div(n, 128), 128, 0, (cudaStream_t)stream>>>(tri_verts, n, limit, flag.p);
    const int e = launch_status("shape_screen_kernel");
    if (cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess) return launch_status("shape screen sync", 0);
    if (e) return e;
    *suspect = *(volatile int*)flag.p;
    return MBEM_OK;
}

extern "C" int mbem_near_eval_nodal(int kernel, int order, const double* x_field, int64_t n_field,
                                    const double* tri_verts, const double* normals, const double* eps,
                                    const int64_t* rowptr, const int64_t* cols, int64_t nnz, const double* coeffs,
                                    double alpha, double* vals, void* stream) {
    using namespace mbem;
    MBEM_REQUIRE(kernel == 0 || kernel == 1, MBEM_ERR_ARG, "kernel must be 0 (T) or 1 (U)");
    MBEM_REQUIRE(order == 1 || order == 2, MBEM_ERR_ARG, "nodal order must be 1 or 2 (order 0: mbem_near_eval)");
    MBEM_REQUIRE(kernel == 1 || normals, MBEM_ERR_ARG, "normals is NULL");
    MBEM_REQUIRE(coeffs && n_field >= 0 && nnz >= 0 && (nnz == 0 || (rowptr && cols && vals)), MBEM_ERR_ARG,
                 "bad nodal near-eval args");
    if (nnz == 0) return MBEM_OK;
    int e = nodal_rules_ready();
    if (e) return e;
    NodalArgs a;
    memset(&a, 0, sizeof(a));
    a.x_field = x_field; a.n_field_pts = n_field; a.tri_verts = tri_verts; a.eps = eps;
    a.normals = kernel == 0 ? normals : nullptr;
    const int nc = kernel == 0 ? 6 : 3;
    for (int i = 0; i < 6; i++) a.c[i] = i < nc ? coeffs[i] : 0.0;
    a.alpha = alpha;
    a.pair_rowptr = rowptr; a.pair_cols = cols; a.n_pairs = nnz;
    const unsigned grid = (unsigned)ceil_div(nnz, ND_THREADS);
    cudaStream_t st = (cudaStream_t)stream;
    if (kernel == 0) {
        if (order == 1) nodal_near_eval_kernel<1, ND_T><<<grid, ND_THREADS, 0, st>>>(a, vals);
        else nodal_near_eval_kernel<2, ND_T><<<grid, ND_THREADS, 0, st>>>(a, vals);
    } else {
        if (order == 1) nodal_near_eval_kernel<1, ND_U><<<grid, ND_THREADS, 0, st>>>(a, vals);
        else nodal_near_eval_kernel<2, ND_U><<<grid, ND_THREADS, 0, st>>>(a, vals);
    }
    return launch_status("nodal_near_eval_kernel");
}
