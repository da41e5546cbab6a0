// What the nodal kernels' translation units share: the rule tables, the launch
// arguments and the split of (field point, source) pairs over blocks.
#pragma once
#include <math.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "nodal_pair.cuh"

namespace mbem {

constexpr int ND_THREADS = 64;       // 255 registers a thread: four blocks an SM
constexpr int ND_SLOTS = 152 * 4;    // resident blocks of the part

static inline void nd_gauss_legendre(int n, double* x, double* w) {
    for (int i = 0; i < n; i++) {
        double z = cos(MBEM_PI * (i + 0.75) / (n + 0.5)), dp = 0.0;
        for (int it = 0; it < 100; it++) {
            double p0 = 1.0, p1 = z;
            for (int k = 2; k <= n; k++) {
                const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            dp = n * (z * p1 - p0) / (z * z - 1.0);
            const double dz = p1 / dp;
            z -= dz;
            if (fabs(dz) < 1e-16) break;
        }
        double p0 = 1.0, p1 = z;
        for (int k = 2; k <= n; k++) {
            const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
            p0 = p1;
            p1 = p2;
        }
        dp = n * (z * p1 - p0) / (z * z - 1.0);
        x[i] = z;
        w[i] = 2.0 / ((1.0 - z * z) * dp * dp);
    }
}

static inline NodalRules nd_make_rules() {
    NodalRules r;
    int k = 0;
    for (int n : {8, 10, 12, 16}) {
        double x[16], w[16];
        nd_gauss_legendre(n, x, w);
        for (int i = 0; i < n / 2; i++, k++) {     // decreasing nodes: the positive half first
            r.ex[k] = x[i];
            r.ew[k] = w[i];
        }
    }
    k = 0;
    for (int n = 4; n <= 7; n++) {
        double x[7], w[7];
        nd_gauss_legendre(n, x, w);
        for (int i = 0; i < n; i++, k++) {
            r.fx[k] = 0.5 * (x[i] + 1.0);
            r.fw[k] = 0.5 * w[i];
        }
    }
    return r;
}

#ifdef __CUDACC__
// The rules in this translation unit's constant memory of the current device, once per device.
static int nodal_rules_ready() {
    static std::mutex mutex;
    static bool ready[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return set_error(MBEM_ERR_CUDA, "no current CUDA device for the nodal rules");
    std::lock_guard<std::mutex> lock(mutex);
    if (ready[dev]) return MBEM_OK;
    static const NodalRules r = nd_make_rules();
    const cudaError_t e = cudaMemcpyToSymbol(c_nd, &r, sizeof(r));
    if (e != cudaSuccess) return set_error(MBEM_ERR_CUDA, "nodal rules: %s", cudaGetErrorString(e));
    ready[dev] = true;
    return MBEM_OK;
}
#endif

struct NodalArgs {
    const double* x_field;
    const double* n_field;
    int64_t n_field_pts;
    const double* tri_verts;
    const double* normals;
    const double* eps;
    int64_t n_src;
    const double* density;
    const int64_t* ids;
    int64_t n_cols;
    double c[6];
    double mu, lam, alpha;
    int accumulate, which;
    double* out;
    int64_t ld;
    int64_t plane;
    const int64_t* pair_rowptr;   // listed pairs: field point f's sources are
    const int64_t* pair_cols;     // pair_cols[pair_rowptr[f] .. pair_rowptr[f + 1])
    int64_t n_pairs;
};

// Blocks of sb sources x fb field points. A block is as large as leaves four
// rounds of resident blocks, so that the last round is short and each source's
// record is made few times.
struct PairTiles {
    int sb, fb;
    dim3 grid;
    size_t smem;
};
constexpr int ND_TILE_PAIRS = 1024;      // most pairs a tile holds
static inline PairTiles pair_tiles(int64_t nf, int64_t ns) {
    PairTiles t;
    t.fb = (int)std::min<int64_t>(nf, ND_THREADS);
    const int64_t want = std::max<int64_t>(1, nf * ns / ((int64_t)ND_THREADS * ND_SLOTS * 4));
    const int64_t full = ceil_div(ND_THREADS, t.fb);
    t.sb = (int)std::min<int64_t>(std::min<int64_t>(std::max(full, want * ND_THREADS / t.fb), std::max<int64_t>(full, 16)), ns);
    t.grid = dim3((unsigned)ceil_div(ns, t.sb), (unsigned)std::min<int64_t>(ceil_div(nf, t.fb), 65535));
    t.smem = (size_t)t.sb * sizeof(NodalRec);
    return t;
}

#ifdef __CUDACC__
__device__ __forceinline__ void load_recs(const NodalArgs& a, int64_t s0, int ns, NodalRec* recs) {
    for (int t = threadIdx.x; t < ns; t += blockDim.x) {
        const int64_t s = s0 + t;
        nodal_rec(a.tri_verts + 9 * s, a.normals ? a.normals + 3 * s : nullptr, a.eps[s], recs[t]);
    }
}

// A tile's pairs ordered by what they cost: beside the element, near, and the
// far rules. A warp that mixes closed forms and quadratures runs both (45 to 69 %
// of the lanes were at work in the P2 and traction kernels), so the block lists
// its pairs by class and its warps take 32 at a time, whichever is free next.
constexpr int ND_CLASSES = 5;
struct PairQueue {
    int count[ND_CLASSES], next;
    uint16_t list[ND_TILE_PAIRS];
};
template <int P>
__device__ __forceinline__ int pair_class(const NodalRec& g, const double* x) {
    const double dx = x[0] - g.c[0], dy = x[1] - g.c[1], dz = x[2] - g.c[2];
    const float q = (float)(dx * dx + dy * dy + dz * dz + g.eps2) / (float)g.L2;      // a hint: the pair decides again
    if (q <= 4.0f) return 0;
    if (q <= (float)(ND_D_STAR * ND_D_STAR)) return 1;
    return 9 - nd_far_n<P>(q, 1.0);      // n = 7 .. 5 (and 4 with 5)
}
// queues `total` pairs (at most ND_TILE_PAIRS); cls(p) is called once a pair.
// All threads of the block call it; it ends with a barrier.
template <class Cls>
__device__ __forceinline__ void queue_pairs(PairQueue& q, int total, Cls&& cls) {
    if (threadIdx.x < ND_CLASSES) q.count[threadIdx.x] = 0;
    if (threadIdx.x == 0) q.next = 0;
    __syncthreads();
    uint64_t kept = 0;                   // 3 bits a pair, ND_TILE_PAIRS / ND_THREADS = 16 pairs
    int i = 0;
    for (int p = threadIdx.x; p < total; p += ND_THREADS, i++) {
        const int c = min(cls(p), ND_CLASSES - 1);
        kept |= (uint64_t)c << (3 * i);
        atomicAdd(&q.count[c], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int c = ND_CLASSES - 1; c >= 0; c--) {      // the dearest first
            const int n = q.count[c];
            q.count[c] = run;
            run += n;
        }
    }
    __syncthreads();
    i = 0;
    for (int p = threadIdx.x; p < total; p += ND_THREADS, i++)
        q.list[atomicAdd(&q.count[(kept >> (3 * i)) & 7], 1)] = (uint16_t)p;
    __syncthreads();
}
// the next pair of this lane's warp's 32, or -1; ends when all are taken. The
// whole warp calls it together.
__device__ __forceinline__ bool queue_next(PairQueue& q, int total, int& p) {
    int base = 0;
    const int lane = threadIdx.x & 31;
    if (lane == 0) base = atomicAdd(&q.next, 32);
    base = __shfl_sync(0xffffffffu, base, 0);
    p = base + lane < total ? (int)q.list[base + lane] : -1;
    return base < total;
}

// field point of listed pair q
__device__ __forceinline__ int64_t pair_row(const int64_t* __restrict__ rowptr, int64_t n, int64_t q) {
    int64_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (rowptr[mid] <= q) lo = mid;
        else hi = mid;
    }
    return lo;
}
#endif

}  // namespace mbem
