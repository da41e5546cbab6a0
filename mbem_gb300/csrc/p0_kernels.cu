// P0 kernel matrices and matrix-free contractions, FP64 (sm_103a).
//
// Both are bound by the FP64 pipe (a warp instruction takes 16 cycles of an SM).
// Matrices: one thread per source triangle, its frame in registers, a tile of
// observers per block read as broadcasts; the tile is the one that shares the
// work out best (matrix_tile). Each warp writes 32 consecutive 3-column blocks
// of a row, i.e. 768 contiguous bytes per output row.
// Contractions: one thread per observer and slice of the sources; tiles of
// source records in shared memory, dealt over the slices of a block and the
// blocks of a cluster, whose partial sums are added in slice, then rank order
// through distributed shared memory (deterministic, no workspace).
//
// Measured: T block 128 x 128 347 -> 22.5 us (8 blocks of 16 observers a thread
// before), 1,728 x 1,728 3.38 -> 1.89 ms (590 FP64 instructions a pair before, some 330
// now; 2.41 with the library's logarithm, atan2 and division);
// T displacement of 6,912 sources at 48 stations 9.98 -> 0.375 ms (6 blocks
// before); elastic stress of 1,856 sources at 4,096 points 17.4 -> 8.7 ms.
#include <cooperative_groups.h>
#include <string.h>

#include <algorithm>

#include "contract_split.cuh"
#include "p0_pair.cuh"

namespace mbem {

namespace cg = cooperative_groups;

constexpr int MAT_THREADS = 64;
constexpr int N_SM = 152;

enum MatKind { MAT_T_DIRECT = 0, MAT_U_DIRECT = 1, MAT_T_BASIS = 2, MAT_U_BASIS = 3 };

struct MatArgs {
    const double* x_field;
    int64_t n_field;
    const double* tri_verts;
    const double* normals;
    const double* eps;
    int64_t n_src;
    double c[6];
    double alpha;
    int accumulate;
    double* out;
    int64_t ld;          // leading dimension (row stride) of `out`
    int64_t plane;       // stride between basis planes (basis kinds)
    int tile;            // observers a block takes at a time
};

template <int KIND>
__global__ void __launch_bounds__(MAT_THREADS) p0_matrix_kernel(MatArgs a) {
    const int64_t s = (int64_t)blockIdx.x * MAT_THREADS + threadIdx.x;
    if (s >= a.n_src) return;
    SrcP0 src;
    double nrm[3] = {0.0, 0.0, 0.0};
    src_setup(a.tri_verts + 9 * s, a.eps[s], src);
    if (KIND == MAT_T_DIRECT || KIND == MAT_T_BASIS) {
        nrm[0] = a.normals[3 * s]; nrm[1] = a.normals[3 * s + 1]; nrm[2] = a.normals[3 * s + 2];
        src_normal(src, nrm);
    }
    const TCoef tc = t_coef(a.c);
    for (int64_t f0 = (int64_t)blockIdx.y * a.tile; f0 < a.n_field; f0 += (int64_t)gridDim.y * a.tile) {
        const int64_t f1 = lmin(f0 + a.tile, a.n_field);
#pragma unroll 1
        for (int64_t f = f0; f < f1; f++) {
            const double ox = a.x_field[3 * f], oy = a.x_field[3 * f + 1], oz = a.x_field[3 * f + 2];
            if (KIND == MAT_T_DIRECT || KIND == MAT_U_DIRECT) {
                double blk[3][3];
                if (src.ok) {
                    PairP0 p;
                    pair_setup(src, ox, oy, oz, p);
                    if (KIND == MAT_T_DIRECT) {
                        t_pair(src, nrm, p, tc, blk);
                    } else {
                        UMoments m;
                        u_moments(src, p, m);
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = 0; j < 3; j++)
                                blk[i][j] = a.c[2] * m.T2[i][j] +
                                            (i == j ? a.c[0] * m.I1 + a.c[1] * src.eps2 * m.I3 : 0.0);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) blk[i][j] = 0.0;
                }
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    double* row = a.out + (3 * f + i) * a.ld + 3 * s;
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        double v = a.alpha * blk[i][j];
                        row[j] = a.accumulate ? row[j] + v : v;
                    }
                }
            } else if (KIND == MAT_T_BASIS) {
                double blk[6][3][3];
                if (src.ok) {
                    PairP0 p;
                    pair_setup(src, ox, oy, oz, p);
                    TMoments m;
                    t_moments(src, nrm, p, m);
                    t_basis_blocks(m, nrm, src.eps2, blk);
                } else {
                    for (int b = 0; b < 6; b++)
                        for (int i = 0; i < 3; i++)
                            for (int j = 0; j < 3; j++) blk[b][i][j] = 0.0;
                }
#pragma unroll
                for (int b = 0; b < 6; b++)
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++)
                            a.out[b * a.plane + (3 * f + i) * a.ld + 3 * s + j] = blk[b][i][j];
            } else {  // MAT_U_BASIS
                double I1 = 0.0, I3 = 0.0, T2[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
                if (src.ok) {
                    PairP0 p;
                    pair_setup(src, ox, oy, oz, p);
                    UMoments m;
                    u_moments(src, p, m);
                    I1 = m.I1;
                    I3 = m.I3;
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int j = 0; j < 3; j++) T2[i][j] = m.T2[i][j];
                }
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        const int64_t idx = (3 * f + i) * a.ld + 3 * s + j;
                        a.out[idx] = (i == j) ? I1 : 0.0;
                        a.out[a.plane + idx] = (i == j) ? src.eps2 * I3 : 0.0;
                        a.out[2 * a.plane + idx] = T2[i][j];
                    }
            }
        }
    }
}

// Observers a block: a tile of t costs a warp 200 + 400 t FP64 instructions (a source's frame
// and its pairs; 250 and 330 with the short functions of dp_math.cuh, whose ratio
// would take another tile, by one to three, in a fifth of the sizes from 40 to 30,000 and the
// same one for blocks of 128, 1,728 and 5,184 squared, the sizes measured) and the part
// the warps of its fullest SM; below about five warps an SM the pipe waits.
static int matrix_tile(int64_t nf, int64_t ns) {
    int best = 16;
    double cost = 1e300;
    for (int t = 1; t <= 16; t++) {
        const int64_t blocks = ceil_div(ns, MAT_THREADS) * ceil_div(nf, t);
        const int64_t rounds = ceil_div(blocks, N_SM);
        // beyond a few rounds the blocks even out
        const double r = rounds > 6 ? (double)blocks / N_SM + 0.5 : rounds < 3 ? 2.5 : (double)rounds;
        const double c = r * (200.0 + 400.0 * t);
        if (c < cost) {
            cost = c;
            best = t;
        }
    }
    return best;
}

// ---------------------------------------------------------------------------
// Contractions: out[f] (+)= alpha * sum_s K(x_f, s) density_s
// ---------------------------------------------------------------------------
enum ConKind {
    CON_T_DISP = 0,
    CON_U_DISP = 1,
    CON_DD_STRESS = 2,
    CON_KELVIN_STRESS = 3,
    CON_EIGENSTRESS = 4,
    CON_ELASTIC_STRESS = 5,   // dd stress minus eigenstress, one pass
};

struct ConArgs {
    const double* x_field;
    int64_t n_field;
    const double* tri_verts;
    const double* normals;
    const double* eps;
    const double* density;
    int64_t n_src;
    double c[6];
    double mu, lam;
    double alpha;
    int accumulate;
    double* out;
    int ob;          // observers a block; its threads / ob slices
};

struct SrcTile {
    SrcP0 g;
    double n[3];     // source normal as passed
    double d[3];     // density
    double dl[3];    // density in the source frame
    bool live;       // non-degenerate and non-zero density
};

// DD stress of a normal off the frame's, minus the eigenstress with eig
static __device__ __noinline__ void dd_pair_general(const SrcTile& T, const PairP0& p, const SMat& m, bool dd, bool eig,
                                                    double out[6]) {
    StressMoments M;
    stress_moments<true>(T.g, p, M);
    double nl[3], loc[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    to_frame(T.g, T.n, nl);
    if (dd) dd_stress_local(M, nl, T.dl, m.mu, m.lam, m.C1, m.c34, m.blob * T.g.eps2, loc);
    const double sgn = dd ? -1.0 : 1.0;
    const double phi = eig ? sgn * m.phi * T.g.eps2 * T.g.eps2 * M.M7[0][0] : 0.0;
    const double ns = nl[0] * T.dl[0] + nl[1] * T.dl[1] + nl[2] * T.dl[2];
    const int ia[6] = {0, 1, 2, 0, 0, 1}, ib[6] = {0, 1, 2, 1, 2, 2};
    for (int t = 0; t < 6; t++) {
        const int i = ia[t], j = ib[t];
        out[t] += loc[i][j] + phi * ((i == j ? m.lam * ns : 0.0) + m.mu * (T.dl[i] * nl[j] + nl[i] * T.dl[j]));
    }
}

// one pair, added to acc: displacement (global), or stress 00 11 22 01 02 12 (global)
template <int KIND>
__device__ __forceinline__ void contract_pair(const SrcTile& T, const double x[3], const ConArgs& a, const TCoef& tc,
                                              const SMat& sm, double* acc) {
    const SrcP0& g = T.g;
    PairP0 p;
    pair_setup(g, x[0], x[1], x[2], p);
    if (KIND == CON_T_DISP) {
        double blk[3][3];
        t_pair(g, T.n, p, tc, blk);
#pragma unroll
        for (int i = 0; i < 3; i++) acc[i] += blk[i][0] * T.d[0] + blk[i][1] * T.d[1] + blk[i][2] * T.d[2];
    } else if (KIND == CON_U_DISP) {
        UMoments m;
        u_moments(g, p, m);
        const double dg = a.c[0] * m.I1 + a.c[1] * g.eps2 * m.I3;
#pragma unroll
        for (int i = 0; i < 3; i++)
            acc[i] += dg * T.d[i] + a.c[2] * (m.T2[i][0] * T.d[0] + m.T2[i][1] * T.d[1] + m.T2[i][2] * T.d[2]);
    } else {
        double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, G[6];
        if (KIND == CON_KELVIN_STRESS) {
            StressMoments M;
            stress_moments<false>(g, p, M);
            double loc[3][3];
            kelvin_stress_local(M, T.dl, a.mu, a.lam, sm.C1, sm.c34, 3.0 * sm.blob * g.eps2, loc);
            v[0] = loc[0][0]; v[1] = loc[1][1]; v[2] = loc[2][2];
            v[3] = loc[0][1]; v[4] = loc[0][2]; v[5] = loc[1][2];
        } else if (!g.aligned) {
            dd_pair_general(T, p, sm, KIND != CON_EIGENSTRESS, KIND != CON_DD_STRESS, v);
        } else {
            double m3[1], m5[6], m7[10];
            dd_moments(g, p, m3, m5, m7);
            if (KIND == CON_EIGENSTRESS) {
                // phi C : sym(s n), n = sn e3
                const double ph = g.sn * sm.phi * g.eps2 * g.eps2 * m7[0];
                v[0] = v[1] = ph * sm.lam * T.dl[2];
                v[2] = ph * (sm.lam + 2.0 * sm.mu) * T.dl[2];
                v[4] = ph * sm.mu * T.dl[0];
                v[5] = ph * sm.mu * T.dl[1];
            } else {
                constexpr bool E = KIND == CON_ELASTIC_STRESS;
                const double w[3] = {g.sn * T.dl[0], g.sn * T.dl[1], g.sn * T.dl[2]};
                dd_slip(m3, m5, m7, p.z, g.eps2, sm, E, w, v);
            }
        }
        rotate_six(g, v, G);
#pragma unroll
        for (int t = 0; t < 6; t++) acc[t] += G[t];
    }
}

template <int KIND, int CON_THREADS, int SRC_TILE>
__global__ void __launch_bounds__(CON_THREADS) p0_contract_kernel(ConArgs a) {
    constexpr int NO = KIND >= CON_DD_STRESS ? 6 : 3;
    __shared__ SrcTile tile[SRC_TILE];
    __shared__ double red[CON_THREADS][NO], part[8][CON_THREADS / 16 * NO];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
    const int ob = a.ob, slices = CON_THREADS / ob;
    const int lane = threadIdx.x % ob, slice = threadIdx.x / ob;
    const int64_t f = (int64_t)(blockIdx.x / ranks) * ob + lane;
    const bool active = f < a.n_field && slice < slices;
    double x[3] = {0.0, 0.0, 0.0};
    if (active) {
        x[0] = a.x_field[3 * f];
        x[1] = a.x_field[3 * f + 1];
        x[2] = a.x_field[3 * f + 2];
    }
    const TCoef tc = t_coef(a.c);
    const SMat sm = stress_mat(KIND >= CON_DD_STRESS ? a.mu : 1.0, KIND >= CON_DD_STRESS ? a.lam : 1.0);
    double acc[NO];
#pragma unroll
    for (int i = 0; i < NO; i++) acc[i] = 0.0;
    for (int64_t s0 = (int64_t)rank * SRC_TILE; s0 < a.n_src; s0 += (int64_t)ranks * SRC_TILE) {
        const int ns = (int)lmin(SRC_TILE, a.n_src - s0);
        __syncthreads();
        if ((int)threadIdx.x < ns) {
            const int64_t s = s0 + threadIdx.x;
            SrcTile& T = tile[threadIdx.x];
            src_setup(a.tri_verts + 9 * s, a.eps[s], T.g);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                T.n[k] = (KIND == CON_U_DISP || KIND == CON_KELVIN_STRESS) ? 0.0 : a.normals[3 * s + k];
                T.d[k] = a.density[3 * s + k];
            }
            src_normal(T.g, T.n);
            to_frame(T.g, T.d, T.dl);
            T.live = T.g.ok && !(T.d[0] == 0.0 && T.d[1] == 0.0 && T.d[2] == 0.0);
            if (KIND == CON_EIGENSTRESS && !(T.g.eps > 0.0)) T.live = false;
        }
        __syncthreads();
        if (!active) continue;
#pragma unroll 1
        for (int t = slice; t < ns; t += slices)
            if (tile[t].live) contract_pair<KIND>(tile[t], x, a, tc, sm, acc);
    }
#pragma unroll
    for (int i = 0; i < NO; i++) red[threadIdx.x][i] = acc[i];
    __syncthreads();
    // the slices' sums, where there are many of them eight runs first
    if (slices >= 16) {
        const int items = ob * NO;
        for (int it = threadIdx.x; it < 8 * items; it += CON_THREADS) {
            const int g = it / items, r = it - g * items;
            double v = 0.0;
            for (int k = g; k < slices; k += 8) v += red[k * ob + r / NO][r % NO];
            part[g][r] = v;
        }
        __syncthreads();
        for (int r = threadIdx.x; r < items; r += CON_THREADS) {
            double v = part[0][r];
#pragma unroll
            for (int g = 1; g < 8; g++) v += part[g][r];
            red[r / NO][r % NO] = v;
        }
    } else {
        for (int r = threadIdx.x; r < ob * NO; r += CON_THREADS) {
            double v = red[r / NO][r % NO];
            for (int k = 1; k < slices; k++) v += red[k * ob + r / NO][r % NO];
            red[r / NO][r % NO] = v;
        }
    }
    cluster.sync();
    if (rank == 0 && slice == 0 && active) {
#pragma unroll
        for (int i = 0; i < NO; i++) acc[i] = red[lane][i];
        for (int r = 1; r < ranks; r++) {
            const double* other = cluster.map_shared_rank(&red[lane][0], r);
#pragma unroll
            for (int i = 0; i < NO; i++) acc[i] += other[i];
        }
        const int ix[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
        constexpr int NW = NO == 3 ? 3 : 9;
        double* o = a.out + NW * f;
#pragma unroll
        for (int i = 0; i < NW; i++) {
            const double v = a.alpha * acc[NW == 3 ? i : ix[i]];
            o[i] = a.accumulate ? o[i] + v : v;
        }
    }
    cluster.sync();      // the partial sums stay until rank 0 has read them
}

// A warp alone takes some 5 us for a tile's records and 12 us for a pair, whatever the
// tile's size, so few observers want large tiles: up to CON_FEW of them one observer a
// block of 128 threads with 128 sources a tile (6,912 sources at 1 to 19 observers:
// 480 us with 64 threads and tiles of 32, 150 with these; at 48 observers 507 and 370).
// Above, contract_split's blocks of observers with 64 threads and tiles of 32. The two meet
// at 76 observers, half an SM's share each (6,912 sources, T displacement | elastic
// stress, one observer a block against contract_split's: 48: 375 | 530 and 517 | 687 us, 70: 500 | 687 and
// 517 | 688, 76: 624 | 860 and 627 | 895, 80: 629 | 880 and 629 | 896, 90: 735 | 1,020 and
// 629 | 896, 200: 1,425 | 2,045 and 1,100 | 1,654; 1,000 sources: 76: 98 | 140 and 99 | 141,
// 90: 115 | 163 and 100 | 141).
constexpr int64_t CON_FEW = 76;

template <int KIND>
static cudaError_t launch_con(const ConArgs& a, bool few, int64_t grid, int ranks, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(few ? 128 : 64);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ranks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return few ? cudaLaunchKernelEx(&cfg, p0_contract_kernel<KIND, 128, 128>, a)
               : cudaLaunchKernelEx(&cfg, p0_contract_kernel<KIND, 64, 32>, a);
}

static int check_common(const double* x, int64_t nf, const double* tv, const double* eps, int64_t ns,
                        int order) {
    MBEM_REQUIRE(nf >= 0 && ns >= 0, MBEM_ERR_ARG, "negative size (n_field=%lld, n_src=%lld)",
                 (long long)nf, (long long)ns);
    MBEM_REQUIRE(order == 0 || order == 1 || order == 2, MBEM_ERR_ARG,
                 "order must be 0, 1 or 2 (got %d)", order);
    MBEM_REQUIRE(nf == 0 || x != nullptr, MBEM_ERR_ARG, "x_field is NULL");
    MBEM_REQUIRE(ns == 0 || (tv != nullptr && eps != nullptr), MBEM_ERR_ARG, "tri_verts/eps is NULL");
    return MBEM_OK;
}

int launch_matrix(int kind, const double* x, int64_t nf, const double* tv, const double* normals,
                  const double* eps, int64_t ns, const double* c, int nc, double alpha, int accumulate,
                  double* out, int64_t ld, int64_t plane, cudaStream_t st) {
    MatArgs a;
    a.x_field = x; a.n_field = nf; a.tri_verts = tv; a.normals = normals; a.eps = eps; a.n_src = ns;
    for (int i = 0; i < 6; i++) a.c[i] = (c && i < nc) ? c[i] : 0.0;
    a.alpha = alpha; a.accumulate = accumulate; a.out = out; a.ld = ld; a.plane = plane;
    if (nf == 0 || ns == 0) return MBEM_OK;
    a.tile = matrix_tile(nf, ns);
    dim3 grid((unsigned)ceil_div(ns, MAT_THREADS), (unsigned)lmin(ceil_div(nf, a.tile), 65535));
    switch (kind) {
        case MAT_T_DIRECT: p0_matrix_kernel<MAT_T_DIRECT><<<grid, MAT_THREADS, 0, st>>>(a); break;
        case MAT_U_DIRECT: p0_matrix_kernel<MAT_U_DIRECT><<<grid, MAT_THREADS, 0, st>>>(a); break;
        case MAT_T_BASIS: p0_matrix_kernel<MAT_T_BASIS><<<grid, MAT_THREADS, 0, st>>>(a); break;
        default: p0_matrix_kernel<MAT_U_BASIS><<<grid, MAT_THREADS, 0, st>>>(a); break;
    }
    return launch_status("p0_matrix_kernel");
}

int launch_contract(int kind, const double* x, int64_t nf, const double* tv, const double* normals,
                    const double* eps, int64_t ns, const double* density, const double* c, int nc,
                    double mu, double lam, double alpha, int accumulate, double* out, cudaStream_t st) {
    ConArgs a;
    a.x_field = x; a.n_field = nf; a.tri_verts = tv; a.normals = normals; a.eps = eps;
    a.density = density; a.n_src = ns;
    for (int i = 0; i < 6; i++) a.c[i] = (c && i < nc) ? c[i] : 0.0;
    a.mu = mu; a.lam = lam; a.alpha = alpha; a.accumulate = accumulate; a.out = out;
    if (nf == 0) return MBEM_OK;
    const bool few = nf <= CON_FEW;
    ConSplit sp = {1, 8};
    if (few)
        while (sp.ranks > 1 && (int64_t)128 * (sp.ranks / 2) >= ns) sp.ranks /= 2;      // no idle half
    else
        sp = contract_split(nf, ns, 64, 64, 32, kind >= CON_DD_STRESS ? 500 : 400, 250);
    a.ob = sp.ob;
    const int64_t grid = ceil_div(nf, sp.ob) * sp.ranks;
    MBEM_REQUIRE(grid < (int64_t)1 << 31, MBEM_ERR_SIZE, "too many observers (%lld)", (long long)nf);
    cudaError_t e;
    switch (kind) {
        case CON_T_DISP: e = launch_con<CON_T_DISP>(a, few, grid, sp.ranks, st); break;
        case CON_U_DISP: e = launch_con<CON_U_DISP>(a, few, grid, sp.ranks, st); break;
        case CON_DD_STRESS: e = launch_con<CON_DD_STRESS>(a, few, grid, sp.ranks, st); break;
        case CON_KELVIN_STRESS: e = launch_con<CON_KELVIN_STRESS>(a, few, grid, sp.ranks, st); break;
        case CON_EIGENSTRESS: e = launch_con<CON_EIGENSTRESS>(a, few, grid, sp.ranks, st); break;
        default: e = launch_con<CON_ELASTIC_STRESS>(a, few, grid, sp.ranks, st); break;
    }
    if (e != cudaSuccess) return set_error(MBEM_ERR_CUDA, "p0_contract_kernel: %s", cudaGetErrorString(e));
    return launch_status("p0_contract_kernel");
}

}  // namespace mbem

using namespace mbem;

extern "C" {

int mbem_t_matrix_direct(const double* x_field, int64_t n_field, const double* tri_verts,
                         const double* normals, const double* eps, int64_t n_src, const double* coeffs,
                         int order, double alpha, int accumulate, double* out, int64_t ld_out,
                         void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    MBEM_REQUIRE(coeffs != nullptr, MBEM_ERR_ARG, "coeffs is NULL");
    MBEM_REQUIRE(n_src == 0 || normals != nullptr, MBEM_ERR_ARG, "normals is NULL");
    if (order != 0)
        return mbem::nodal_matrix(0, x_field, n_field, tri_verts, normals, eps, n_src, coeffs, order, alpha,
                                 accumulate, out, ld_out, stream);
    MBEM_REQUIRE(ld_out >= 3 * n_src, MBEM_ERR_ARG, "ld_out %lld < 3*n_src", (long long)ld_out);
    return launch_matrix(MAT_T_DIRECT, x_field, n_field, tri_verts, normals, eps, n_src, coeffs, 6, alpha,
                         accumulate, out, ld_out, 0, (cudaStream_t)stream);
}

int mbem_u_matrix_direct(const double* x_field, int64_t n_field, const double* tri_verts, const double* eps,
                         int64_t n_src, const double* coeffs, int order, double alpha, int accumulate,
                         double* out, int64_t ld_out, void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    MBEM_REQUIRE(coeffs != nullptr, MBEM_ERR_ARG, "coeffs is NULL");
    if (order != 0)
        return mbem::nodal_matrix(1, x_field, n_field, tri_verts, nullptr, eps, n_src, coeffs, order, alpha,
                                 accumulate, out, ld_out, stream);
    MBEM_REQUIRE(ld_out >= 3 * n_src, MBEM_ERR_ARG, "ld_out %lld < 3*n_src", (long long)ld_out);
    return launch_matrix(MAT_U_DIRECT, x_field, n_field, tri_verts, nullptr, eps, n_src, coeffs, 3, alpha,
                         accumulate, out, ld_out, 0, (cudaStream_t)stream);
}

int mbem_t_basis_matrices(const double* x_field, int64_t n_field, const double* tri_verts,
                          const double* normals, const double* eps, int64_t n_src, int order, double* out,
                          void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    MBEM_REQUIRE(n_src == 0 || normals != nullptr, MBEM_ERR_ARG, "normals is NULL");
    if (order != 0)
        return mbem::nodal_matrix(2, x_field, n_field, tri_verts, normals, eps, n_src, nullptr, order, 1.0, 0,
                                 out, 0, stream);
    return launch_matrix(MAT_T_BASIS, x_field, n_field, tri_verts, normals, eps, n_src, nullptr, 0, 1.0, 0,
                         out, 3 * n_src, 9 * n_field * n_src, (cudaStream_t)stream);
}

int mbem_u_basis_matrices(const double* x_field, int64_t n_field, const double* tri_verts, const double* eps,
                          int64_t n_src, int order, double* out, void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    if (order != 0)
        return mbem::nodal_matrix(3, x_field, n_field, tri_verts, nullptr, eps, n_src, nullptr, order, 1.0, 0,
                                 out, 0, stream);
    return launch_matrix(MAT_U_BASIS, x_field, n_field, tri_verts, nullptr, eps, n_src, nullptr, 0, 1.0, 0,
                         out, 3 * n_src, 9 * n_field * n_src, (cudaStream_t)stream);
}

int mbem_t_disp_contract(const double* x_field, int64_t n_field, const double* tri_verts,
                         const double* normals, const double* eps, int64_t n_src, const double* density,
                         const double* coeffs, int order, double alpha, int accumulate, double* out,
                         void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    MBEM_REQUIRE(coeffs != nullptr && (n_src == 0 || (normals && density)), MBEM_ERR_ARG,
                 "coeffs/normals/density is NULL");
    if (order != 0)
        return mbem::nodal_contract(0, x_field, n_field, tri_verts, normals, eps, n_src, density, coeffs, 0.0,
                                   0.0, order, alpha, accumulate, out, stream);
    return launch_contract(CON_T_DISP, x_field, n_field, tri_verts, normals, eps, n_src, density, coeffs, 6,
                           0.0, 0.0, alpha, accumulate, out, (cudaStream_t)stream);
}

int mbem_u_disp_contract(const double* x_field, int64_t n_field, const double* tri_verts, const double* eps,
                         int64_t n_src, const double* density, const double* coeffs, int order, double alpha,
                         int accumulate, double* out, void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    MBEM_REQUIRE(coeffs != nullptr && (n_src == 0 || density), MBEM_ERR_ARG, "coeffs/density is NULL");
    if (order != 0)
        return mbem::nodal_contract(1, x_field, n_field, tri_verts, nullptr, eps, n_src, density, coeffs, 0.0,
                                   0.0, order, alpha, accumulate, out, stream);
    return launch_contract(CON_U_DISP, x_field, n_field, tri_verts, nullptr, eps, n_src, density, coeffs, 3,
                           0.0, 0.0, alpha, accumulate, out, (cudaStream_t)stream);
}

int mbem_stress_contract(int kind, const double* x_field, int64_t n_field, const double* tri_verts,
                         const double* normals, const double* eps, int64_t n_src, const double* density,
                         double mu, double lam, int order, double alpha, int accumulate, double* out,
                         void* stream) {
    int st = check_common(x_field, n_field, tri_verts, eps, n_src, order);
    if (st) return st;
    MBEM_REQUIRE(kind >= MBEM_STRESS_DD && kind <= MBEM_STRESS_ELASTIC, MBEM_ERR_ARG,
                 "unknown stress kind %d", kind);
    MBEM_REQUIRE(n_src == 0 || density, MBEM_ERR_ARG, "density is NULL");
    MBEM_REQUIRE(kind == MBEM_STRESS_KELVIN || n_src == 0 || normals, MBEM_ERR_ARG, "normals is NULL");
    MBEM_REQUIRE(mu > 0.0 && lam + mu > 0.0, MBEM_ERR_ARG, "material (mu=%g, lam=%g) is not admissible", mu,
                 lam);
    if (order != 0)
        return mbem::nodal_contract(2 + kind, x_field, n_field, tri_verts, normals, eps, n_src, density,
                                   nullptr, mu, lam, order, alpha, accumulate, out, stream);
    return launch_contract(CON_DD_STRESS + kind, x_field, n_field, tri_verts, normals, eps, n_src, density,
                           nullptr, 0, mu, lam, alpha, accumulate, out, (cudaStream_t)stream);
}

}  // extern "C"
