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

// Fully symmetric rules on the triangle, one line an orbit: points, weight (of a
// unit sum), and two barycentric coordinates of a point of it. Degrees 6, 8, 9,
// 10, 12 and 14 with 12, 16, 19, 25, 33 and 42 points, the orbit counts of Dunavant, Int. J. Numer.
// Meth. Eng. 21 (1985); the values solve the moment equations (invariants
// e2^i e3^j of the barycentric coordinates) by Newton's method in 50 digits.
struct NdOrbit {
    int n;
    double w, a, b;
};
static const NdOrbit ND_ORBITS[ND_FAR_RULES][10] = {
    {{3, 0.1167862757263793660252896, 0.2492867451709104212916386, 0.2492867451709104212916386},
     {3, 0.05084490637020681692093681, 0.0630890144915022283403316, 0.0630890144915022283403316},
     {6, 0.08285107561837357519355346, 0.6365024991213986472301426, 0.05314504984481694735324967}},
    {{1, 0.1443156076777871682510911, 1.0 / 3.0, 1.0 / 3.0},
     {3, 0.03245849762319808031092593, 0.05054722831703097545842355, 0.05054722831703097545842355},
     {3, 0.0950916342672846247938961, 0.4592925882927231560288155, 0.4592925882927231560288155},
     {3, 0.1032173705347182502817916, 0.1705693077517602066222935, 0.1705693077517602066222935},
     {6, 0.02723031417443499426484469, 0.008394777409957605337213835, 0.2631128296346381134217858}},
    {{1, 0.09713579628279883381924198, 1.0 / 3.0, 1.0 / 3.0},
     {3, 0.07782754100477427931673936, 0.4370895914929366372699304, 0.4370895914929366372699304},
     {3, 0.0255776756586980312616788, 0.04472951339445270986510659, 0.04472951339445270986510659},
     {3, 0.03133470022713907053685483, 0.4896825191987376277837069, 0.4896825191987376277837069},
     {3, 0.07964773892721025303289177, 0.1882035356190327302409613, 0.1882035356190327302409613},
     {6, 0.04328353937728937728937729, 0.7411985987844980206900799, 0.2219629891607656956751025}},
    {{1, 0.08174332914628596642811868, 1.0 / 3.0, 1.0 / 3.0},
     {3, 0.04595796360474472801378791, 0.1421611010565643850921621, 0.1421611010565643850921621},
     {3, 0.01335296881314956627557298, 0.03205537321694351293098459, 0.03205537321694351293098459},
     {6, 0.06390490639642404543289873, 0.1481328857838205504978068, 0.5300541189273440282770957},
     {6, 0.03418464816295942862869158, 0.02961988948872976763383627, 0.3691467818278109869114208},
     {6, 0.02529775770728838438904279, 0.8079306009228790650799499, 0.02836766533993843925043576}},
    {{3, 0.02573106644045533541779092, 0.4882173897738048825646621, 0.4882173897738048825646621},
     {3, 0.04369254453803840213545726, 0.4397243922944602729797366, 0.4397243922944602729797366},
     {3, 0.06285822421788510035427051, 0.2712103850121159223459513, 0.2712103850121159223459513},
     {3, 0.0347961129307089429893284, 0.1275761455415859246738963, 0.1275761455415859246738963},
     {3, 0.006166261051559017233866484, 0.02131735045321037024685698, 0.02131735045321037024685698},
     {6, 0.0403715577663809295178287, 0.2757132696855141939747963, 0.6089432357797878068561924},
     {6, 0.02235677320230344571183908, 0.2813255809899395482481307, 0.6958360867878034221416355},
     {6, 0.0173162311086588923716421, 0.1162519159075971412413541, 0.8580140335440726305905366}},
    {{3, 0.02188358136942889064084495, 0.488963910362178638677376, 0.488963910362178638677376},
     {3, 0.03278835354412535064131098, 0.4176447193404539225094408, 0.4176447193404539225094408},
     {3, 0.05177410450729158631478491, 0.2734775283088386597549443, 0.2734775283088386597549443},
     {3, 0.04216258873699301753823044, 0.1772055324125434369566107, 0.1772055324125434369566107},
     {3, 0.01443369966977666760170992, 0.06179988309087260126747883, 0.06179988309087260126747883},
     {3, 0.004923403602400081681826024, 0.0193909612487010481782501, 0.0193909612487010481782501},
     {6, 0.02466575321256367396287525, 0.1722666878213555783752896, 0.7706085547749964825890333},
     {6, 0.03857151078706068322848903, 0.3368614597963450017440552, 0.5702222908466831734976962},
     {6, 0.01443630811353384049608869, 0.2983728821362577529708315, 0.6869801678080878373586272},
     {6, 0.005010228838500671769860093, 0.118974497696956845398182, 0.8797571713701711295145716}}};

static inline NodalRules nd_make_rules() {
    NodalRules r;
    int k = 0;
    for (int n : {7, 8, 9, 10, 12, 16}) {
        double x[16], w[16];
        nd_gauss_legendre(n, x, w);
        for (int i = 0; i < n; i++, k++) {
            if (2 * i + 1 == n) x[i] = 0.0;
            r.ex[k] = x[i];
            double f = w[i];
            for (int p = 0; p < 6; p++, f *= x[i]) r.ew[k][p] = f;
        }
    }
    k = 0;
    for (int d = 0; d < ND_FAR_RULES; d++)
        for (const NdOrbit& o : ND_ORBITS[d]) {
            const double c = 1.0 - o.a - o.b;
            const double p[6][2] = {{o.a, o.b}, {c, o.a}, {o.b, c}, {o.b, o.a}, {o.a, c}, {c, o.b}};
            for (int i = 0; i < o.n; i++, k++) {
                const double l1 = p[i][0], l2 = p[i][1], l0 = 1.0 - l1 - l2, w = 0.5 * o.w;
                r.fl[k][0] = l1; r.fl[k][1] = l2; r.fl[k][2] = w;
                const double l[3] = {l0, l1, l2};
                for (int v = 0; v < 3; v++) {
                    r.fn[k][v] = w * l[v];
                    r.fn[k][3 + v] = w * l[v] * (2.0 * l[v] - 1.0);
                    r.fn[k][6 + v] = 4.0 * w * l[v] * l[(v + 1) % 3];
                }
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
constexpr int ND_CLASSES = 2 + ND_FAR_RULES;
struct PairQueue {
    int count[ND_CLASSES], next;
    uint16_t list[ND_TILE_PAIRS];
};
static_assert(ND_CLASSES <= 8, "queue_pairs keeps three bits a pair");
template <int P, int F>
__device__ __forceinline__ int pair_class(const NodalRec& g, const double* x) {
    const double dx = x[0] - g.c[0], dy = x[1] - g.c[1], dz = x[2] - g.c[2];
    const float q = (float)(dx * dx + dy * dy + dz * dz + g.eps2) / (float)g.L2;      // a hint: the pair decides again
    if (q <= 4.0f) return 0;
    if (q <= (float)(ND_D_STAR * ND_D_STAR)) return 1;
    return 2 + nd_far_rule<P, F>(q, 1.0);
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
        const int c = cls(p);
        kept |= (uint64_t)c << (3 * i);
        atomicAdd(&q.count[c], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int c = 0; c < ND_CLASSES; c++) {
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
