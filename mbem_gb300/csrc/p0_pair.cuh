// FP64 device code for one (observer, P0 source triangle) pair of the
// mollified Kelvin kernels.
//
// The mathematics is the reference's (src/mbem/kernels/tri_kernels.py): the
// observer is lifted to h = sqrt(z^2 + eps^2) over the source plane, the 2-D
// area moments M_n[a,b] = int xi1^a xi2^b / R^n come from the solid angle
// (I3 = -Omega/h) and the divergence-theorem recursion over the three edges,
// and every kernel is a contraction of those moments. The GPU formulation
// differs in what it materialises:
//
//  * all per-source quantities (frame, in-plane vertices, edge tangents,
//    twice the area) are computed once per source and kept in registers;
//  * the lifted-point solid angle uses the in-plane triple product
//    r1.(r2 x r3) = -h * (twice the signed area), exact for the lifted point;
//  * the vertex distances R_k = sqrt(|p_k|^2 + h^2) are shared by the solid
//    angle and the six edge endpoints (the reference recomputes them);
//  * the T-kernel block needs only V3, V5, the trace t_i = T3[i,m,m] and
//    W = T3 . n, so the rank-3 tensor is never built; the stress kernels are
//    contracted with the density in the source frame before rotating back.
// All of these are exact rewrites; results agree with the reference to a
// few ulps of the moments involved.
#pragma once

#include "common.cuh"
#include "dp_math.cuh"

namespace mbem {

struct SrcP0 {
    double v0[3];
    double ex[3], ey[3], nh[3];
    double Px1, Px2, Py1, Py2;   // in-plane coordinates of vertices 1, 2 (vertex 0 at origin)
    double tx[3], ty[3];         // unit in-plane edge tangents, edge e = (e, e+1)
    double area2;                // twice the signed in-plane area
    double eps, eps2;
    bool ok;                     // false for a degenerate triangle (zero block)
    bool edge_ok[3];
    double sn;                   // +-1: the source normal along the frame's (src_normal)
    bool aligned;
};

// A unit source normal along the frame's, to the rounding of both (every mesh),
// takes the forms without the other two components.
__device__ __forceinline__ void src_normal(SrcP0& s, const double* __restrict__ n) {
    const double a = n[0] * s.ex[0] + n[1] * s.ex[1] + n[2] * s.ex[2];
    const double b = n[0] * s.ey[0] + n[1] * s.ey[1] + n[2] * s.ey[2];
    const double c = n[0] * s.nh[0] + n[1] * s.nh[1] + n[2] * s.nh[2];
    s.sn = c < 0.0 ? -1.0 : 1.0;
    s.aligned = fabs(a) < 1e-15 && fabs(b) < 1e-15 && fabs(fabs(c) - 1.0) < 1e-15;
}

// Frame of a source triangle (tri_kernels.py:137-153) and its per-source
// constants. `tv` points at 9 doubles (vertex-major).
__device__ __forceinline__ void src_setup(const double* __restrict__ tv, double eps, SrcP0& s) {
    double e1x = tv[3] - tv[0], e1y = tv[4] - tv[1], e1z = tv[5] - tv[2];
    double e2x = tv[6] - tv[0], e2y = tv[7] - tv[1], e2z = tv[8] - tv[2];
    double cx = e1y * e2z - e1z * e2y;
    double cy = e1z * e2x - e1x * e2z;
    double cz = e1x * e2y - e1y * e2x;
    double a2 = sqrt(cx * cx + cy * cy + cz * cz);
    s.ok = a2 >= 1e-30;
    s.eps = eps;
    s.eps2 = eps * eps;
    s.v0[0] = tv[0]; s.v0[1] = tv[1]; s.v0[2] = tv[2];
    if (!s.ok) {
        // never used: the caller writes a zero block
        for (int k = 0; k < 3; k++) {
            s.ex[k] = s.ey[k] = s.nh[k] = 0.0;
            s.tx[k] = s.ty[k] = 0.0;
            s.edge_ok[k] = false;
        }
        s.Px1 = s.Px2 = s.Py1 = s.Py2 = s.area2 = 0.0;
        return;
    }
    double ia = 1.0 / a2;
    s.nh[0] = cx * ia; s.nh[1] = cy * ia; s.nh[2] = cz * ia;
    double e1n = sqrt(e1x * e1x + e1y * e1y + e1z * e1z);
    double ie = 1.0 / e1n;
    s.ex[0] = e1x * ie; s.ex[1] = e1y * ie; s.ex[2] = e1z * ie;
    s.ey[0] = s.nh[1] * s.ex[2] - s.nh[2] * s.ex[1];
    s.ey[1] = s.nh[2] * s.ex[0] - s.nh[0] * s.ex[2];
    s.ey[2] = s.nh[0] * s.ex[1] - s.nh[1] * s.ex[0];
    s.Px1 = e1x * s.ex[0] + e1y * s.ex[1] + e1z * s.ex[2];
    s.Py1 = e1x * s.ey[0] + e1y * s.ey[1] + e1z * s.ey[2];
    s.Px2 = e2x * s.ex[0] + e2y * s.ex[1] + e2z * s.ex[2];
    s.Py2 = e2x * s.ey[0] + e2y * s.ey[1] + e2z * s.ey[2];
    s.area2 = s.Px1 * s.Py2 - s.Px2 * s.Py1;
    const double Px[3] = {0.0, s.Px1, s.Px2};
    const double Py[3] = {0.0, s.Py1, s.Py2};
#pragma unroll
    for (int e = 0; e < 3; e++) {
        int b = (e + 1) % 3;
        double evx = Px[b] - Px[e], evy = Py[b] - Py[e];
        double L = sqrt(evx * evx + evy * evy);
        s.edge_ok[e] = L > 1e-30;
        double iL = s.edge_ok[e] ? 1.0 / L : 0.0;
        s.tx[e] = evx * iL;
        s.ty[e] = evy * iL;
    }
}

// ---------------------------------------------------------------------------
// forms in the source frame, shared by the P0 pair and the nodal tables
// ---------------------------------------------------------------------------
// index of the moment [a, b] in a table ordered by degree a + b, then b
__host__ __device__ constexpr int nd_tri(int a, int b) { return (a + b) * (a + b + 1) / 2 + b; }

template <class Frame>
__device__ __forceinline__ void rotate_full(const Frame& g, const double B[3][3], double G[3][3]) {
    double Y[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int j = 0; j < 3; j++) Y[a][j] = B[a][0] * g.ex[j] + B[a][1] * g.ey[j] + B[a][2] * g.nh[j];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) G[i][j] = g.ex[i] * Y[0][j] + g.ey[i] * Y[1][j] + g.nh[i] * Y[2][j];
}
// symmetric L (00 11 22 01 02 12) to the global frame, same layout
template <class Frame>
__device__ __forceinline__ void rotate_six(const Frame& g, const double L[6], double G[6]) {
    const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
    double Y[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            Y[a][j] = L[ix[a][0]] * g.ex[j] + L[ix[a][1]] * g.ey[j] + L[ix[a][2]] * g.nh[j];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) G[ix[i][j]] = g.ex[i] * Y[0][j] + g.ey[i] * Y[1][j] + g.nh[i] * Y[2][j];
}
template <class Frame>
__device__ __forceinline__ void to_frame(const Frame& g, const double* v, double l[3]) {
    l[0] = v[0] * g.ex[0] + v[1] * g.ex[1] + v[2] * g.ex[2];
    l[1] = v[0] * g.ey[0] + v[1] * g.ey[1] + v[2] * g.ey[2];
    l[2] = v[0] * g.nh[0] + v[1] * g.nh[1] + v[2] * g.nh[2];
}

// Coefficients of the combined T block. |d|^2 = R^2 - eps^2 turns
// t_i = int d_i |d|^2 / R^5 into V3_i - eps^2 V5_i, so with b_i = cb V3_i + ce6 V5_i
//   out = n_j (c3 V3_i + c5 V5_i) + n_i b_j + w6 W_ij + d_ij n.b
// (c5 and ce6 times eps^2).
struct TCoef {
    double c3, c5, cb, ce6, w6;
};
__host__ __device__ __forceinline__ TCoef t_coef(const double c[6]) {
    TCoef t;
    t.c3 = c[0] + c[1] + 2.0 * c[4];
    t.c5 = c[2] + 3.0 * c[1];
    t.cb = c[3] + c[4];
    t.ce6 = c[5];
    t.w6 = -6.0 * c[4];
    return t;
}

// The T block in the source frame for the normal s e3, from the moments
// i3, a3 = (1,0), b3 = (0,1) of n = 3 and i5 .. c02 of n = 5.
__device__ __forceinline__ void t_local(double i3, double a3, double b3, double i5, double a5, double b5, double c20,
                                        double c11, double c02, double z, double eps2, const TCoef& c, double s,
                                        double B[3][3]) {
    const double k3 = s * c.c3, k5 = s * c.c5 * eps2, kb = s * c.cb, k6 = s * c.ce6 * eps2, kw = s * c.w6 * z;
    const double zi3 = z * i3, zi5 = z * i5, kz = kw * z;
    const double be2 = kb * zi3 + k6 * zi5;
    const double v0 = -(kz * a5), v1 = -(kz * b5);
    B[0][0] = kw * c20 + be2;
    B[1][1] = kw * c02 + be2;
    B[0][1] = B[1][0] = kw * c11;
    B[0][2] = v0 - (k3 * a3 + k5 * a5);
    B[1][2] = v1 - (k3 * b3 + k5 * b5);
    B[2][0] = v0 - (kb * a3 + k6 * a5);
    B[2][1] = v1 - (kb * b3 + k6 * b5);
    B[2][2] = kz * zi5 + (k3 * zi3 + k5 * zi5) + 2.0 * be2;
}

// material constants of the stress forms
struct SMat {
    double mu, lam, C1, c34;
    double k3a;        // 3 c34 - 9
    double x1;         // 3 c34 - 18
    double blob;       // 2 (1 - nu), times eps^2: cblob
    double phi;        // 15 / (8 pi), times eps^4
};
__host__ __device__ inline SMat stress_mat(double mu, double lam) {
    SMat m;
    const double nu = lam / (2.0 * (lam + mu));
    m.mu = mu;
    m.lam = lam;
    m.C1 = 1.0 / (16.0 * MBEM_PI * mu * (1.0 - nu));
    m.c34 = 3.0 - 4.0 * nu;
    m.k3a = 3.0 * m.c34 - 9.0;
    m.x1 = 3.0 * m.c34 - 18.0;
    m.blob = 2.0 * (1.0 - nu);
    m.phi = 15.0 / (8.0 * MBEM_PI);
    return m;
}

// Stress (00 11 22 01 02 12, source frame, normal +e3) of slip along e_K with
// the moment set (m3[0]; m5 to degree 2; m7 to degree 3), times w and added:
// the DD stress of tri_kernels.py:900-964 for that normal and slip, and with
// EIG the eigenstress (tri_kernels.py:1206-1214) taken off.
template <int K>
__device__ __forceinline__ void dd_unit(const double* m3, const double* m5, const double* m7, double z, double eps2,
                                        const SMat& m, bool eig, double w, double out[6]) {
#define A5(a, b) m5[nd_tri(a, b)]
#define A7(a, b) m7[nd_tri(a, b)]
    const double cb = m.blob * eps2;
    const double z2 = z * z;
    const double I3 = m3[0], I5 = A5(0, 0), I7 = A7(0, 0);
    const double phi = eig ? m.phi * eps2 * eps2 * I7 : 0.0;
    if (K < 2) {
        // u: the slip axis, v: the other in-plane axis; d = (-xi, z)
#define U5(a, b) (K == 0 ? A5(a, b) : A5(b, a))
#define U7(a, b) (K == 0 ? A7(a, b) : A7(b, a))
        const double T5u3 = -z * U5(1, 0), T5v3 = -z * U5(0, 1), T533 = z2 * I5;
        const double zu = -z * U7(1, 0), zv = -z * U7(0, 1), z33 = z2 * I7;
        const double c15 = 15.0 * cb;
        const double Fu3 = m.k3a * T5u3 + c15 * zu;
        const double Fv3 = m.k3a * T5v3 + c15 * zv;
        const double Fuv = m.k3a * U5(1, 1) + c15 * U7(1, 1);
        const double Fuu33 = m.k3a * (U5(2, 0) + T533) + c15 * (U7(2, 0) + z33);
        const double q0 = -z * U7(3, 0), q1 = -z * U7(1, 2), q2 = z2 * zu;        // T4 uuu3, vvu3, 33u3
        const double q3 = -z * U7(2, 1), q4 = z2 * U7(2, 0), q5 = z2 * U7(1, 1);  // uvu3, u3u3, v3u3
        // sum_r T4_rru3 = T5_u3 - eps^2 T7_u3
        const double tr = 2.0 * Fu3 + 12.0 * T5u3 - 30.0 * eps2 * zu;
        const double t = m.lam * tr;
        const double base = -12.0 * T5u3;
        const double sA = 2.0 * ((1.0 - m.c34) * I3 - 3.0 * cb * I5);
        const double suu = t + m.mu * (base + 2.0 * Fu3 + 60.0 * q0);
        const double svv = t + m.mu * (base + 60.0 * q1);
        const double s33 = t + m.mu * (base + 2.0 * Fu3 + 60.0 * q2);
        const double suv = Fv3 + 60.0 * q3, su3 = sA + Fuu33 + 60.0 * q4, sv3 = Fuv + 60.0 * q5;
        // sigma = -C1 mu (lam tr delta + mu (Y + Y^T))
        const double gm = -m.C1 * w * m.mu;
        out[K] += gm * suu;
        out[1 - K] += gm * svv;
        out[2] += gm * s33;
        const double g2 = gm * m.mu;
        out[3] += g2 * suv;
        out[K == 0 ? 4 : 5] += g2 * su3 - (m.mu * w) * phi;
        out[K == 0 ? 5 : 4] += g2 * sv3;
#undef U5
#undef U7
    } else {
        const double T00 = A5(2, 0), T11 = A5(0, 2), T01 = A5(1, 1), T02 = -z * A5(1, 0), T12 = -z * A5(0, 1),
                     T22 = z2 * I5;
        const double S00 = A7(2, 0), S11 = A7(0, 2), S01 = A7(1, 1), S02 = -z * A7(1, 0), S12 = -z * A7(0, 1),
                     S22 = z2 * I7;
        const double trT = I3 - eps2 * I5, trS = I5 - eps2 * I7;
        // T4_rt33, and t4c_rt = int d_r d_t |d|^2 / R^7 = T5_rt - eps^2 T7_rt
        const double Q00 = z2 * S00, Q11 = z2 * S11, Q01 = z2 * S01, Q02 = z2 * S02, Q12 = z2 * S12, Q22 = z2 * S22;
        const double C22 = T22 - eps2 * S22;
        const double c15 = 15.0 * cb;
        const double xd = (4.0 - m.c34) * I3 - 3.0 * trT - 3.0 * cb * I5;
        const double trX = 3.0 * xd + m.x1 * trT + 15.0 * (trT - eps2 * trS) + c15 * trS;
        const double F02 = m.k3a * T02 + c15 * S02, F12 = m.k3a * T12 + c15 * S12, F22 = m.k3a * T22 + c15 * S22;
        const double A = (1.0 - m.c34) * I3 - 3.0 * cb * I5;
        const double trY = 2.0 * A + 6.0 * I3 + 2.0 * F22 - 18.0 * T22 - 6.0 * trT + 30.0 * C22;
        const double trB = m.lam * trX + m.mu * trY;
        const double yd = 4.0 * I3 - 12.0 * T22;
        // X = xd delta + x1 T + 15 C + c15 S with 15 C = 15 T - 15 eps^2 S ; Y + Y^T = yd delta - 12 T + 60 Q + (e3, F terms) + 4 A e3 e3
        const double l2 = 2.0 * m.lam, mu = m.mu;
        const double xt = m.x1 + 15.0, xs = c15 - 15.0 * eps2;
        const double diag = m.lam * trB + mu * (l2 * xd + mu * yd);
        const double gw = -m.C1 * w;
        const double ep = phi * w;
        out[0] += gw * (diag + mu * (l2 * (xt * T00 + xs * S00) + mu * (60.0 * Q00 - 12.0 * T00))) -
                  ep * m.lam;
        out[1] += gw * (diag + mu * (l2 * (xt * T11 + xs * S11) + mu * (60.0 * Q11 - 12.0 * T11))) -
                  ep * m.lam;
        out[2] += gw * (diag + mu * (l2 * (xt * T22 + xs * S22) +
                                     mu * (60.0 * Q22 - 12.0 * T22 + 4.0 * (F22 + A)))) -
                  ep * (m.lam + 2.0 * mu);
        out[3] += gw * mu * (l2 * (xt * T01 + xs * S01) + mu * (60.0 * Q01 - 12.0 * T01));
        out[4] += gw * mu * (l2 * (xt * T02 + xs * S02) + mu * (60.0 * Q02 - 12.0 * T02 + 2.0 * F02));
        out[5] += gw * mu * (l2 * (xt * T12 + xs * S12) + mu * (60.0 * Q12 - 12.0 * T12 + 2.0 * F12));
    }
#undef A5
#undef A7
}

// The same for a slip w (source frame) in one go: the in-plane components meet in
// sums along the slip, and the normal one's T5 and T7 terms share their factors, some
// 90 operations less than three dd_unit.
__device__ __forceinline__ void dd_slip(const double* m3, const double* m5, const double* m7, double z, double eps2,
                                        const SMat& m, bool eig, const double w[3], double out[6]) {
#define A5(a, b) m5[nd_tri(a, b)]
#define A7(a, b) m7[nd_tri(a, b)]
    const double cb = m.blob * eps2, c15 = 15.0 * cb, z2 = z * z, mu = m.mu, lam = m.lam;
    const double I3 = m3[0], I5 = A5(0, 0), I7 = A7(0, 0);
    const double T02 = -z * A5(1, 0), T12 = -z * A5(0, 1), T22 = z2 * I5;
    const double S02 = -z * A7(1, 0), S12 = -z * A7(0, 1), S22 = z2 * I7;
    const double F02 = m.k3a * T02 + c15 * S02, F12 = m.k3a * T12 + c15 * S12, F22 = m.k3a * T22 + c15 * S22;
    const double A = (1.0 - m.c34) * I3 - 3.0 * cb * I5;
    const double gm = -m.C1 * mu;
    // in-plane slip
    const double Ts = w[0] * T02 + w[1] * T12, Ss = w[0] * S02 + w[1] * S12, Fs2 = 2.0 * (w[0] * F02 + w[1] * F12);
    const double iso = lam * (Fs2 + 12.0 * Ts - 30.0 * eps2 * Ss) - 12.0 * mu * Ts;
    const double z60 = 60.0 * z, zz = z60 * z, cz = c15 + zz;
    const double g = 2.0 * A + F22, P = m.k3a * A5(1, 1) + cz * A7(1, 1);
    const double s00 = iso + mu * (2.0 * w[0] * F02 - z60 * (w[0] * A7(3, 0) + w[1] * A7(2, 1)));
    const double s11 = iso + mu * (2.0 * w[1] * F12 - z60 * (w[0] * A7(1, 2) + w[1] * A7(0, 3)));
    const double s22 = iso + mu * (Fs2 + zz * Ss);
    const double s01 = w[0] * F12 + w[1] * F02 - z60 * (w[0] * A7(2, 1) + w[1] * A7(1, 2));
    const double s02 = w[0] * (g + m.k3a * A5(2, 0) + cz * A7(2, 0)) + w[1] * P;
    const double s12 = w[1] * (g + m.k3a * A5(0, 2) + cz * A7(0, 2)) + w[0] * P;
    // normal slip: l2 (xt T + xs S) + mu (60 z^2 S - 12 T) and the e3 terms
    const double trT = I3 - eps2 * I5, trS = I5 - eps2 * I7, C22 = T22 - eps2 * S22;
    const double xd = (4.0 - m.c34) * I3 - 3.0 * trT - 3.0 * cb * I5;
    const double trX = 3.0 * xd + m.x1 * trT + 15.0 * (trT - eps2 * trS) + c15 * trS;
    const double trY = 2.0 * A + 6.0 * I3 + 2.0 * F22 - 18.0 * T22 - 6.0 * trT + 30.0 * C22;
    const double yd = 4.0 * I3 - 12.0 * T22, l2 = 2.0 * lam;
    const double diag = lam * (lam * trX + mu * trY) + mu * (l2 * xd + mu * yd);
    const double kt = l2 * (m.x1 + 15.0) - 12.0 * mu, ks = l2 * (c15 - 15.0 * eps2) + mu * zz;
    const double gw = -m.C1 * w[2], gwm = gw * mu;
    const double gm2 = gm * mu;
    out[0] += gm * s00 + gw * diag + gwm * (kt * A5(2, 0) + ks * A7(2, 0));
    out[1] += gm * s11 + gw * diag + gwm * (kt * A5(0, 2) + ks * A7(0, 2));
    out[2] += gm * s22 + gw * diag + gwm * (kt * T22 + ks * S22 + 4.0 * mu * (F22 + A));
    out[3] += gm2 * s01 + gwm * (kt * A5(1, 1) + ks * A7(1, 1));
    out[4] += gm2 * s02 + gwm * (kt * T02 + ks * S02 + 2.0 * mu * F02);
    out[5] += gm2 * s12 + gwm * (kt * T12 + ks * S12 + 2.0 * mu * F12);
    if (eig) {
        const double phi = m.phi * eps2 * eps2 * I7, pl = phi * lam * w[2], pm = phi * mu;
        out[0] -= pl;
        out[1] -= pl;
        out[2] -= pl + 2.0 * pm * w[2];
        out[4] -= pm * w[0];
        out[5] -= pm * w[1];
    }
#undef A5
#undef A7
}

// Pair geometry shared by all kernels: height, lift, projected vertices,
// vertex distances and I3 = -Omega / h (tri_kernels.py:257-273).
struct PairP0 {
    double z, h2, h, ih2;        // ih2 = 1 / h^2
    double px[3], py[3];
    double R[3], iR[3];
    double I3;
};

// FP64 work is the cost of every pair (the FP64 pipe is 1/64 of FP32 on
// this part), so reciprocals come from rsqrt (R and 1/R from one call) and
// from shared divisions.
__device__ __forceinline__ void pair_setup(const SrcP0& s, double ox, double oy, double oz, PairP0& p) {
    double dx = ox - s.v0[0], dy = oy - s.v0[1], dz = oz - s.v0[2];
    p.z = dx * s.nh[0] + dy * s.nh[1] + dz * s.nh[2];
    double qx = dx * s.ex[0] + dy * s.ex[1] + dz * s.ex[2];
    double qy = dx * s.ey[0] + dy * s.ey[1] + dz * s.ey[2];
    p.h2 = p.z * p.z + s.eps2;
    const double ih = rsqrt(p.h2);
    p.h = p.h2 * ih;
    p.ih2 = ih * ih;
    p.px[0] = -qx;          p.py[0] = -qy;
    p.px[1] = s.Px1 - qx;   p.py[1] = s.Py1 - qy;
    p.px[2] = s.Px2 - qx;   p.py[2] = s.Py2 - qy;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double r2 = p.px[k] * p.px[k] + p.py[k] * p.py[k] + p.h2;
        p.iR[k] = rsqrt(r2);
        p.R[k] = r2 * p.iR[k];
    }
    // van Oosterom at the lifted point, in the source frame: r_k = (px, py, -h)
    double d01 = p.px[0] * p.px[1] + p.py[0] * p.py[1] + p.h2;
    double d12 = p.px[1] * p.px[2] + p.py[1] * p.py[2] + p.h2;
    double d02 = p.px[0] * p.px[2] + p.py[0] * p.py[2] + p.h2;
    double numer = -p.h * s.area2;
    double denom = p.R[0] * p.R[1] * p.R[2] + p.R[2] * d01 + p.R[0] * d12 + p.R[1] * d02;
    double omega = 2.0 * angle64(numer, denom);
    p.I3 = -omega * ih;
}

// Per-edge primitive differences at orders 1 and 3 (tri_kernels.py:54-76,
// :298-302): J1 = log(u + R), K1 = R, J3 = u / (rho^2 R), K3 = -1/R.
struct EdgeP0 {
    double nx, ny, tx, ty, dp, ua, ub, rho2, ir2;
    double dJ1, dK1, dJ3, dK3, dL3;
};

// x, or 1e-300 for a zero, by integer operations
__device__ __forceinline__ double not_zero(double x) {
    return __double2hiint(x) == 0 ? 1e-300 : x;
}

// All three edges at once: dJ1 = log((u_b + R_b) / (u_a + R_a)) takes one
// log per edge.
__device__ __forceinline__ void edges_setup(const SrcP0& s, const PairP0& p, EdgeP0 g[3]) {
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const int a = e, b = (e + 1) % 3;
        g[e].tx = s.tx[e]; g[e].ty = s.ty[e];
        g[e].nx = g[e].ty; g[e].ny = -g[e].tx;
        g[e].dp = p.px[a] * g[e].nx + p.py[a] * g[e].ny;
        g[e].ua = p.px[a] * g[e].tx + p.py[a] * g[e].ty;
        g[e].ub = p.px[b] * g[e].tx + p.py[b] * g[e].ty;
        g[e].rho2 = s.edge_ok[e] ? g[e].dp * g[e].dp + p.h2 : 1.0;
        const double num = s.edge_ok[e] ? not_zero(g[e].ub + p.R[b]) : 1.0;
        const double den = s.edge_ok[e] ? not_zero(g[e].ua + p.R[a]) : 1.0;
        g[e].dK1 = p.R[b] - p.R[a];
        g[e].dK3 = p.iR[a] - p.iR[b];
        // rho2 < 1e-60, compared as integers off the FP64 pipe
        g[e].ir2 = __double_as_longlong(g[e].rho2) < __double_as_longlong(1e-60) ? 0.0 : rcp64(g[e].rho2);
        g[e].dJ1 = log64(num * rcp64(den));
        g[e].dJ3 = (g[e].ub * p.iR[b] - g[e].ua * p.iR[a]) * g[e].ir2;
        g[e].dL3 = g[e].dJ1 - g[e].rho2 * g[e].dJ3;
    }
}

// ---------------------------------------------------------------------------
// T kernel (slip -> displacement): the combined 3x3 block
//   out_ij = sum_b c_b B_b,ij,  B = [N[P1], N[P2], N[P3], R[P1], R[P2], R[P3]]
// (tri_kernels.py:251-427 with the coefficients of basis.py:58-72).
// With V3, V5 (first moments), t_i = sum_m T3[i,m,m] and W_ij = T3[i,j,.].n:
//   N1 = n_j V3_i          R1 = d_ij n.V3 + n_i V3_j
//   N2 = n_j (4 V3_i - 3 t_i)
//   R2 = n_i V3_j + 2 n_j V3_i + d_ij n.V3 - 6 W_ij
//   N3 = eps^2 n_j V5_i    R3 = eps^2 (d_ij n.V5 + n_i V5_j)
// ---------------------------------------------------------------------------
struct TMoments {
    double V3[3], V5[3], W[3][3];   // global frame
};

// T-kernel moments V3, V5, t, W (global frame) from the 2-D moments of the
// source frame (ex, ey, nh); shared by the P0 pair and the nodal tables.
struct TScal {
    double z, I3, I5, m10_3, m01_3, m10_5, m01_5, m20_5, m11_5, m02_5, m30_5, m21_5, m12_5, m03_5;
};

__device__ __forceinline__ void t_from_scal(const double* ex, const double* ey, const double* nh,
                                            const double* __restrict__ nrm, const TScal& q, TMoments& m) {
    const double z = q.z, I3 = q.I3, I5 = q.I5;
    const double m10_3 = q.m10_3, m01_3 = q.m01_3, m10_5 = q.m10_5, m01_5 = q.m01_5;
    const double m20_5 = q.m20_5, m11_5 = q.m11_5, m02_5 = q.m02_5;
    const double m30_5 = q.m30_5, m21_5 = q.m21_5, m12_5 = q.m12_5, m03_5 = q.m03_5;
    // local frame (ex, ey, nh): d = (-xi1, -xi2, z)
    const double V3l[3] = {-m10_3, -m01_3, z * I3};
    const double V5l[3] = {-m10_5, -m01_5, z * I5};
    const double z2 = z * z;
    // T3 in the local frame, T[a][b][c] = (-1)^(#0+#1) z^(#2) M5(#0,#1)
    const double T000 = -m30_5, T001 = -m21_5, T002 = z * m20_5, T011 = -m12_5,
                 T012 = z * m11_5, T022 = -z2 * m10_5, T111 = -m03_5, T112 = z * m02_5,
                 T122 = -z2 * m01_5, T222 = z2 * z * I5;
    // local normal of the source normal passed in (may differ from nh)
    const double nl0 = nrm[0] * ex[0] + nrm[1] * ex[1] + nrm[2] * ex[2];
    const double nl1 = nrm[0] * ey[0] + nrm[1] * ey[1] + nrm[2] * ey[2];
    const double nl2 = nrm[0] * nh[0] + nrm[1] * nh[1] + nrm[2] * nh[2];
    double Wl[3][3];
    Wl[0][0] = T000 * nl0 + T001 * nl1 + T002 * nl2;
    Wl[0][1] = T001 * nl0 + T011 * nl1 + T012 * nl2;
    Wl[0][2] = T002 * nl0 + T012 * nl1 + T022 * nl2;
    Wl[1][1] = T011 * nl0 + T111 * nl1 + T112 * nl2;
    Wl[1][2] = T012 * nl0 + T112 * nl1 + T122 * nl2;
    Wl[2][2] = T022 * nl0 + T122 * nl1 + T222 * nl2;
    Wl[1][0] = Wl[0][1]; Wl[2][0] = Wl[0][2]; Wl[2][1] = Wl[1][2];
    // rotate to the global frame: v = Q^T v_l, W = Q^T W_l Q (Q rows ex, ey, nh)
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double qi[3] = {ex[i], ey[i], nh[i]};
        m.V3[i] = qi[0] * V3l[0] + qi[1] * V3l[1] + qi[2] * V3l[2];
        m.V5[i] = qi[0] * V5l[0] + qi[1] * V5l[1] + qi[2] * V5l[2];
    }
    double Y[3][3];  // Y = W_l Q  (3x3 local-by-global)
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            Y[a][j] = Wl[a][0] * ex[j] + Wl[a][1] * ey[j] + Wl[a][2] * nh[j];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
            double w = ex[i] * Y[0][j] + ey[i] * Y[1][j] + nh[i] * Y[2][j];
            m.W[i][j] = w;
            m.W[j][i] = w;
        }
}


// the 2-D moments of any normal (to degree 3 at n = 5)
__device__ __forceinline__ void t_moments(const SrcP0& s, const double* __restrict__ nrm,
                                          const PairP0& p, TMoments& m) {
    double BN1_001 = 0, BN2_001 = 0, BD003 = 0, BN1_003 = 0, BN2_003 = 0, BN1_103 = 0,
           BN1_013 = 0, BN2_013 = 0, BN1_203 = 0, BN1_113 = 0, BN1_023 = 0, BN2_023 = 0;
    EdgeP0 G[3];
    edges_setup(s, p, G);
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (!s.edge_ok[e]) continue;
        const EdgeP0& g = G[e];
        double A = g.dp * g.nx, B = g.dp * g.ny;
        double v10 = A * g.dJ3 + g.tx * g.dK3;
        double v01 = B * g.dJ3 + g.ty * g.dK3;
        double v20 = A * A * g.dJ3 + 2.0 * A * g.tx * g.dK3 + g.tx * g.tx * g.dL3;
        double v11 = A * B * g.dJ3 + (A * g.ty + B * g.tx) * g.dK3 + g.tx * g.ty * g.dL3;
        double v02 = B * B * g.dJ3 + 2.0 * B * g.ty * g.dK3 + g.ty * g.ty * g.dL3;
        BN1_001 += g.nx * g.dJ1; BN2_001 += g.ny * g.dJ1;
        BD003 += g.dp * g.dJ3;
        BN1_003 += g.nx * g.dJ3; BN2_003 += g.ny * g.dJ3;
        BN1_103 += g.nx * v10;
        BN1_013 += g.nx * v01; BN2_013 += g.ny * v01;
        BN1_203 += g.nx * v20;
        BN1_113 += g.nx * v11;
        BN1_023 += g.nx * v02; BN2_023 += g.ny * v02;
    }
    const double I3 = p.I3, z = p.z;
    const double I5 = (BD003 + I3) * p.ih2 * (1.0 / 3.0);
    const double third = 1.0 / 3.0;
    const double m10_3 = -BN1_001, m01_3 = -BN2_001;
    const double m10_5 = -BN1_003 * third, m01_5 = -BN2_003 * third;
    const double m20_5 = (I3 - BN1_103) * third, m11_5 = -BN1_013 * third;
    const double m02_5 = (I3 - BN2_013) * third;
    const double m30_5 = (2.0 * m10_3 - BN1_203) * third, m21_5 = (m01_3 - BN1_113) * third;
    const double m12_5 = -BN1_023 * third, m03_5 = (2.0 * m01_3 - BN2_023) * third;
    TScal q{z, I3, I5, m10_3, m01_3, m10_5, m01_5, m20_5, m11_5, m02_5, m30_5, m21_5, m12_5, m03_5};
    t_from_scal(s.ex, s.ey, s.nh, nrm, q, m);
}

// Combined T block of any normal.
__device__ __forceinline__ void t_block(const TMoments& m, const double* __restrict__ n, const TCoef& c, double eps2,
                                        double out[3][3]) {
    const double nV3 = n[0] * m.V3[0] + n[1] * m.V3[1] + n[2] * m.V3[2];
    const double nV5 = n[0] * m.V5[0] + n[1] * m.V5[1] + n[2] * m.V5[2];
    const double c5 = c.c5 * eps2, ce6 = c.ce6 * eps2;
    const double gam = c.cb * nV3 + ce6 * nV5;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double al = c.c3 * m.V3[i] + c5 * m.V5[i];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double bej = c.cb * m.V3[j] + ce6 * m.V5[j];
            out[i][j] = n[j] * al + n[i] * bej + c.w6 * m.W[i][j] + (i == j ? gam : 0.0);
        }
    }
}

// The T block of one pair (src_normal has been called). For the frame's normal
// W = T3 . e3 needs n = 5 to degree 2 only and t follows from V3 and V5, so the
// edges carry four sums less of degree 2 and no third row: about 330 FP64
// instructions a pair where the general moments take 520.
static __device__ __noinline__ void t_pair_general(const SrcP0& s, const double* nrm, const PairP0& p, const TCoef& c,
                                                   double out[3][3]) {
    TMoments m;
    t_moments(s, nrm, p, m);
    t_block(m, nrm, c, s.eps2, out);
}
__device__ __forceinline__ void t_pair(const SrcP0& s, const double* __restrict__ nrm, const PairP0& p, const TCoef& c,
                                       double out[3][3]) {
    if (!s.aligned) {
        t_pair_general(s, nrm, p, c, out);
        return;
    }
    EdgeP0 G[3];
    edges_setup(s, p, G);
    // (nx, ny) = (ty, -tx): with a = dp dJ3 the sums of nx v10 and ny v01 add up to that of a
    double x1 = 0, y1 = 0, d3 = 0, x3 = 0, y3 = 0, x10 = 0, x01 = 0;
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (!s.edge_ok[e]) continue;
        const EdgeP0& g = G[e];
        const double a = g.dp * g.dJ3;
        const double v10 = g.nx * a + g.tx * g.dK3, v01 = g.ny * a + g.ty * g.dK3;
        x1 += g.nx * g.dJ1; y1 += g.ny * g.dJ1;
        d3 += a;
        x3 += g.nx * g.dJ3; y3 += g.ny * g.dJ3;
        x10 += g.nx * v10;
        x01 += g.nx * v01;
    }
    const double y01 = d3 - x10;
    const double th = 1.0 / 3.0, I3 = p.I3;
    double B[3][3];
    t_local(I3, -x1, -y1, (d3 + I3) * p.ih2 * th, -x3 * th, -y3 * th, (I3 - x10) * th, -x01 * th, (I3 - y01) * th, p.z,
            s.eps2, c, s.sn, B);
    rotate_full(s, B, out);
}

// The six basis blocks separately (t_basis_matrices, tri_kernels.py:473-492).
__device__ __forceinline__ void t_basis_blocks(const TMoments& m, const double* __restrict__ n,
                                               double eps2, double out[6][3][3]) {
    const double nV3 = n[0] * m.V3[0] + n[1] * m.V3[1] + n[2] * m.V3[2];
    const double nV5 = n[0] * m.V5[0] + n[1] * m.V5[1] + n[2] * m.V5[2];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double d = (i == j) ? 1.0 : 0.0;
            out[0][i][j] = n[j] * m.V3[i];
            out[1][i][j] = n[j] * (m.V3[i] + 3.0 * eps2 * m.V5[i]);      // 4 V3 - 3 t
            out[2][i][j] = eps2 * n[j] * m.V5[i];
            out[3][i][j] = d * nV3 + n[i] * m.V3[j];
            out[4][i][j] = n[i] * m.V3[j] + 2.0 * n[j] * m.V3[i] + d * nV3 - 6.0 * m.W[i][j];
            out[5][i][j] = eps2 * (d * nV5 + n[i] * m.V5[j]);
        }
}

// ---------------------------------------------------------------------------
// U kernel (force -> displacement) basis [I1 d, eps^2 I3 d, T2[3]]
// (tri_kernels.py:161-243).
// ---------------------------------------------------------------------------
struct UMoments {
    double I1, I3, T2[3][3];   // T2 in the global frame
};

__device__ __forceinline__ void u_moments(const SrcP0& s, const PairP0& p, UMoments& m) {
    double BD001 = 0, BN1_001 = 0, BN2_001 = 0, BN1_101 = 0, BN1_011 = 0, BN2_011 = 0;
    EdgeP0 G[3];
    edges_setup(s, p, G);
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (!s.edge_ok[e]) continue;
        const double tx = G[e].tx, ty = G[e].ty, nx = G[e].nx, ny = G[e].ny;
        const double dp = G[e].dp;
        const double dJ1 = G[e].dJ1;
        const double dK1 = G[e].dK1;
        const double v10 = dp * nx * dJ1 + tx * dK1;
        const double v01 = dp * ny * dJ1 + ty * dK1;
        BD001 += dp * dJ1;
        BN1_001 += nx * dJ1; BN2_001 += ny * dJ1;
        BN1_101 += nx * v10;
        BN1_011 += nx * v01; BN2_011 += ny * v01;
    }
    const double I3 = p.I3, z = p.z;
    const double I1 = BD001 - p.h2 * I3;
    const double m10 = -BN1_001, m01 = -BN2_001;
    const double m20 = I1 - BN1_101, m11 = -BN1_011, m02 = I1 - BN2_011;
    // local T2: [0][0]=m20 [0][1]=m11 [1][1]=m02 [0][2]=-z m10 [1][2]=-z m01 [2][2]=z^2 I3
    const double L00 = m20, L01 = m11, L11 = m02, L02 = -z * m10, L12 = -z * m01, L22 = z * z * I3;
    double Y[3][3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        Y[0][j] = L00 * s.ex[j] + L01 * s.ey[j] + L02 * s.nh[j];
        Y[1][j] = L01 * s.ex[j] + L11 * s.ey[j] + L12 * s.nh[j];
        Y[2][j] = L02 * s.ex[j] + L12 * s.ey[j] + L22 * s.nh[j];
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
            double w = s.ex[i] * Y[0][j] + s.ey[i] * Y[1][j] + s.nh[i] * Y[2][j];
            m.T2[i][j] = w;
            m.T2[j][i] = w;
        }
    m.I1 = I1;
    m.I3 = I3;
}

// ---------------------------------------------------------------------------
// Stress moments up to n = 7 (tri_kernels.py:656-769), in the source frame.
// M3: I3, m10, m01.  M5: a+b <= 3.  M7: a+b <= 4 (only when NEED7).
// ---------------------------------------------------------------------------
struct StressMoments {
    double z;
    double I3, m3_10, m3_01;
    double M5[4][4];   // [a][b], a+b <= 3
    double M7[5][5];   // [a][b], a+b <= 4
};

// polynomial coefficients in u of (A + tx u)^a (B + ty u)^b, a+b <= 3
template <int a, int b>
__device__ __forceinline__ void edge_poly(double A, double B, double tx, double ty, double c[4]) {
    double pa[4] = {1.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < a; i++) {
        double q[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            q[k] += pa[k] * A;
            q[k + 1] += pa[k] * tx;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) pa[k] = q[k];
    }
#pragma unroll
    for (int i = 0; i < b; i++) {
        double q[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            q[k] += pa[k] * B;
            q[k + 1] += pa[k] * ty;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) pa[k] = q[k];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) c[k] = pa[k];
}

template <int a, int b>
__device__ __forceinline__ double edge_int(double A, double B, double tx, double ty,
                                           double D0, double D1, double D2, double D3) {
    double c[4];
    edge_poly<a, b>(A, B, tx, ty, c);
    double r = c[0] * D0;
    if (a + b >= 1) r += c[1] * D1;
    if (a + b >= 2) r += c[2] * D2;
    if (a + b >= 3) r += c[3] * D3;
    return r;
}

template <bool NEED7>
__device__ __forceinline__ void stress_moments(const SrcP0& s, const PairP0& p, StressMoments& M) {
    double BN1m1 = 0, BN2m1 = 0, BD003 = 0, BD005 = 0;
    // m = 3 edge sums (a+b <= 2): bn1 for 00,10,01,20,11,02 ; bn2 for 00,01,02
    double b3_1_00 = 0, b3_1_10 = 0, b3_1_01 = 0, b3_1_20 = 0, b3_1_11 = 0, b3_1_02 = 0;
    double b3_2_00 = 0, b3_2_01 = 0, b3_2_02 = 0;
    // m = 5 edge sums (a+b <= 3)
    double b5_1_00 = 0, b5_1_10 = 0, b5_1_01 = 0, b5_1_20 = 0, b5_1_11 = 0, b5_1_02 = 0,
           b5_1_30 = 0, b5_1_21 = 0, b5_1_12 = 0, b5_1_03 = 0;
    double b5_2_00 = 0, b5_2_01 = 0, b5_2_02 = 0, b5_2_03 = 0;
    EdgeP0 G[3];
    edges_setup(s, p, G);
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (!s.edge_ok[e]) continue;
        const EdgeP0& g = G[e];
        const double A = g.dp * g.nx, B = g.dp * g.ny;
        BN1m1 += g.nx * g.dJ1; BN2m1 += g.ny * g.dJ1;
        double v;
        v = g.dJ3;                                                            // (0,0)
        b3_1_00 += g.nx * v; b3_2_00 += g.ny * v; BD003 += g.dp * v;
        v = edge_int<1, 0>(A, B, g.tx, g.ty, g.dJ3, g.dK3, g.dL3, 0.0); b3_1_10 += g.nx * v;
        v = edge_int<0, 1>(A, B, g.tx, g.ty, g.dJ3, g.dK3, g.dL3, 0.0);
        b3_1_01 += g.nx * v; b3_2_01 += g.ny * v;
        v = edge_int<2, 0>(A, B, g.tx, g.ty, g.dJ3, g.dK3, g.dL3, 0.0); b3_1_20 += g.nx * v;
        v = edge_int<1, 1>(A, B, g.tx, g.ty, g.dJ3, g.dK3, g.dL3, 0.0); b3_1_11 += g.nx * v;
        v = edge_int<0, 2>(A, B, g.tx, g.ty, g.dJ3, g.dK3, g.dL3, 0.0);
        b3_1_02 += g.nx * v; b3_2_02 += g.ny * v;
        if (NEED7) {
            const int a = e, b = (e + 1) % 3;
            const double ua = g.ua, ub = g.ub;
            // J5 = u (3 rho^2 + 2 u^2) / (3 rho^4 R^3), K5 = -1 / (3 R^3)
            double dJ5 = 0.0;
            if (g.rho2 >= 1e-60) {
                const double ir2 = g.ir2;
                const double ia3 = p.iR[a] * p.iR[a] * p.iR[a];
                const double ib3 = p.iR[b] * p.iR[b] * p.iR[b];
                dJ5 = (ub * (3.0 * g.rho2 + 2.0 * ub * ub) * ib3 -
                       ua * (3.0 * g.rho2 + 2.0 * ua * ua) * ia3) * (ir2 * ir2 * (1.0 / 3.0));
            }
            const double dK5 = (p.iR[a] * p.iR[a] * p.iR[a] - p.iR[b] * p.iR[b] * p.iR[b]) * (1.0 / 3.0);
            const double dL5 = g.dJ3 - g.rho2 * dJ5;
            const double dM5 = g.dK3 - g.rho2 * dK5;
            v = dJ5;
            b5_1_00 += g.nx * v; b5_2_00 += g.ny * v; BD005 += g.dp * v;
            v = edge_int<1, 0>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5); b5_1_10 += g.nx * v;
            v = edge_int<0, 1>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5);
            b5_1_01 += g.nx * v; b5_2_01 += g.ny * v;
            v = edge_int<2, 0>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5); b5_1_20 += g.nx * v;
            v = edge_int<1, 1>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5); b5_1_11 += g.nx * v;
            v = edge_int<0, 2>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5);
            b5_1_02 += g.nx * v; b5_2_02 += g.ny * v;
            v = edge_int<3, 0>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5); b5_1_30 += g.nx * v;
            v = edge_int<2, 1>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5); b5_1_21 += g.nx * v;
            v = edge_int<1, 2>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5); b5_1_12 += g.nx * v;
            v = edge_int<0, 3>(A, B, g.tx, g.ty, dJ5, dK5, dL5, dM5);
            b5_1_03 += g.nx * v; b5_2_03 += g.ny * v;
        }
    }
    const double I3 = p.I3, h2 = p.h2;
    const double third = 1.0 / 3.0, fifth = 0.2;
    const double I5 = (h2 > 1e-60) ? (BD003 + I3) * p.ih2 * third : 0.0;
    M.z = p.z;
    M.I3 = I3;
    M.m3_10 = -BN1m1;
    M.m3_01 = -BN2m1;
    M.M5[0][0] = I5;
    M.M5[1][0] = -b3_1_00 * third;
    M.M5[0][1] = -b3_2_00 * third;
    M.M5[2][0] = (I3 - b3_1_10) * third;
    M.M5[1][1] = -b3_1_01 * third;
    M.M5[0][2] = (I3 - b3_2_01) * third;
    M.M5[3][0] = (2.0 * M.m3_10 - b3_1_20) * third;
    M.M5[2][1] = (M.m3_01 - b3_1_11) * third;
    M.M5[1][2] = -b3_1_02 * third;
    M.M5[0][3] = (2.0 * M.m3_01 - b3_2_02) * third;
    if (NEED7) {
        const double I7 = (h2 > 1e-60) ? (BD005 + 3.0 * I5) * p.ih2 * fifth : 0.0;
        M.M7[0][0] = I7;
        M.M7[1][0] = -b5_1_00 * fifth;
        M.M7[0][1] = -b5_2_00 * fifth;
        M.M7[2][0] = (I5 - b5_1_10) * fifth;
        M.M7[1][1] = -b5_1_01 * fifth;
        M.M7[0][2] = (I5 - b5_2_01) * fifth;
        M.M7[3][0] = (2.0 * M.M5[1][0] - b5_1_20) * fifth;
        M.M7[2][1] = (M.M5[0][1] - b5_1_11) * fifth;
        M.M7[1][2] = -b5_1_02 * fifth;
        M.M7[0][3] = (2.0 * M.M5[0][1] - b5_2_02) * fifth;
        M.M7[4][0] = (3.0 * M.M5[2][0] - b5_1_30) * fifth;
        M.M7[3][1] = (2.0 * M.M5[1][1] - b5_1_21) * fifth;
        M.M7[2][2] = (M.M5[0][2] - b5_1_12) * fifth;
        M.M7[1][3] = -b5_1_03 * fifth;
        M.M7[0][4] = (3.0 * M.M5[0][2] - b5_2_03) * fifth;
    }
}

// The moments the stress of slip on the frame's normal reads (dd_unit): I3, n = 5
// to degree 2, n = 7 to degree 3, in nd_tri order. No edge log enters.
__device__ __forceinline__ void dd_moments(const SrcP0& s, const PairP0& p, double m3[1], double m5[6],
                                           double m7[10]) {
    double d3 = 0, d5 = 0, x3[3] = {0, 0, 0}, y3[2] = {0, 0}, x5[6] = {0, 0, 0, 0, 0, 0}, y5[3] = {0, 0, 0};
    EdgeP0 G[3];
    edges_setup(s, p, G);
    double i3[3];
#pragma unroll
    for (int k = 0; k < 3; k++) i3[k] = p.iR[k] * p.iR[k] * p.iR[k];
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (!s.edge_ok[e]) continue;
        const EdgeP0& g = G[e];
        const int a = e, b = (e + 1) % 3;
        const double A = g.dp * g.nx, B = g.dp * g.ny;
        const double ia3 = i3[a], ib3 = i3[b];
        // J5 = u (3 rho^2 + 2 u^2) / (3 rho^4 R^3), K5 = -1 / (3 R^3)
        const double r3 = 3.0 * g.rho2;
        const double J = (g.ub * (r3 + 2.0 * g.ub * g.ub) * ib3 - g.ua * (r3 + 2.0 * g.ua * g.ua) * ia3) *
                         (g.ir2 * g.ir2 * (1.0 / 3.0));
        const double K = (ia3 - ib3) * (1.0 / 3.0), L = g.dJ3 - g.rho2 * J;
        const double v10 = A * g.dJ3 + g.tx * g.dK3, v01 = B * g.dJ3 + g.ty * g.dK3;
        d3 += g.dp * g.dJ3;
        x3[0] += g.nx * g.dJ3; y3[0] += g.ny * g.dJ3;
        x3[1] += g.nx * v10;
        x3[2] += g.nx * v01; y3[1] += g.ny * v01;
        const double a0 = A * J + g.tx * K, a1 = A * K + g.tx * L, b0 = B * J + g.ty * K, b1 = B * K + g.ty * L;
        const double v02 = B * b0 + g.ty * b1;
        d5 += g.dp * J;
        x5[0] += g.nx * J; y5[0] += g.ny * J;
        x5[1] += g.nx * a0;
        x5[2] += g.nx * b0; y5[1] += g.ny * b0;
        x5[3] += g.nx * (A * a0 + g.tx * a1);
        x5[4] += g.nx * (B * a0 + g.ty * a1);
        x5[5] += g.nx * v02; y5[2] += g.ny * v02;
    }
    const double I3 = p.I3, th = 1.0 / 3.0, f = 0.2;
    const double I5 = (p.h2 > 1e-60) ? (d3 + I3) * p.ih2 * th : 0.0;
    m3[0] = I3;
    m5[0] = I5;
    m5[1] = -x3[0] * th;
    m5[2] = -y3[0] * th;
    m5[3] = (I3 - x3[1]) * th;
    m5[4] = -x3[2] * th;
    m5[5] = (I3 - y3[1]) * th;
    m7[0] = (p.h2 > 1e-60) ? (d5 + 3.0 * I5) * p.ih2 * f : 0.0;
    m7[1] = -x5[0] * f;
    m7[2] = -y5[0] * f;
    m7[3] = (I5 - x5[1]) * f;
    m7[4] = -x5[2] * f;
    m7[5] = (I5 - y5[1]) * f;
    m7[6] = (2.0 * m5[1] - x5[3]) * f;
    m7[7] = (m5[2] - x5[4]) * f;
    m7[8] = -x5[5] * f;
    m7[9] = (2.0 * m5[2] - y5[2]) * f;
}

// Local-frame moment tensors of d = (-xi1, -xi2, z): component c counts
// toward a (c = 0), b (c = 1) or the z power (c = 2).
template <int N>
__device__ __forceinline__ double sgnz(double z) {
    double r = 1.0;
#pragma unroll
    for (int i = 0; i < N; i++) r *= z;
    return r;
}

__device__ __forceinline__ void cnt2(int i, int j, int& a, int& b) {
    a = (i == 0) + (j == 0);
    b = (i == 1) + (j == 1);
}

// Rotation of a symmetric local tensor to the global frame.
__device__ __forceinline__ void rotate_sym(const SrcP0& s, const double L[3][3], double G[3][3]) {
    double Y[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int j = 0; j < 3; j++) Y[a][j] = L[a][0] * s.ex[j] + L[a][1] * s.ey[j] + L[a][2] * s.nh[j];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
            double w = s.ex[i] * Y[0][j] + s.ey[i] * Y[1][j] + s.nh[i] * Y[2][j];
            G[i][j] = w;
            G[j][i] = w;
        }
}

__device__ __forceinline__ void to_local(const SrcP0& s, const double* v, double l[3]) {
    l[0] = v[0] * s.ex[0] + v[1] * s.ex[1] + v[2] * s.ex[2];
    l[1] = v[0] * s.ey[0] + v[1] * s.ey[1] + v[2] * s.ey[2];
    l[2] = v[0] * s.nh[0] + v[1] * s.nh[1] + v[2] * s.nh[2];
}

// Local moment value for index counts (a of xi1, b of xi2, c of z) with sign
// (-1)^(a+b) and z^c.
#define MBEM_T2L(M, a, b, c, z) (((((a) + (b)) & 1) ? -1.0 : 1.0) * sgnz<(c)>(z) * (M)[(a)][(b)])

// Slip -> total stress contracted with a density (local frame in, local
// frame symmetric out): sigma_l[m][n] = H[m,n,k] s_k for the source frame
// (tri_kernels.py:900-964, contracted analytically).
__device__ __forceinline__ void dd_stress_local(const StressMoments& M, const double nl[3],
                                                const double sl[3], double mu, double lam,
                                                double C1, double c34, double cblob,
                                                double out[3][3]) {
    const double z = M.z;
    const double I3 = M.I3, I5 = M.M5[0][0];
    // T2_5, T2_7 local
    double T5[3][3], T7[3][3];
    T5[0][0] = MBEM_T2L(M.M5, 2, 0, 0, z); T5[0][1] = MBEM_T2L(M.M5, 1, 1, 0, z);
    T5[1][1] = MBEM_T2L(M.M5, 0, 2, 0, z); T5[0][2] = MBEM_T2L(M.M5, 1, 0, 1, z);
    T5[1][2] = MBEM_T2L(M.M5, 0, 1, 1, z); T5[2][2] = MBEM_T2L(M.M5, 0, 0, 2, z);
    T7[0][0] = MBEM_T2L(M.M7, 2, 0, 0, z); T7[0][1] = MBEM_T2L(M.M7, 1, 1, 0, z);
    T7[1][1] = MBEM_T2L(M.M7, 0, 2, 0, z); T7[0][2] = MBEM_T2L(M.M7, 1, 0, 1, z);
    T7[1][2] = MBEM_T2L(M.M7, 0, 1, 1, z); T7[2][2] = MBEM_T2L(M.M7, 0, 0, 2, z);
    T5[1][0] = T5[0][1]; T5[2][0] = T5[0][2]; T5[2][1] = T5[1][2];
    T7[1][0] = T7[0][1]; T7[2][0] = T7[0][2]; T7[2][1] = T7[1][2];
    // T4_7 distinct values by (a, b) counts, c = 4 - a - b
    double T4v[5][5];
#pragma unroll
    for (int a = 0; a <= 4; a++)
#pragma unroll
        for (int b = 0; a + b <= 4; b++) {
            const int c = 4 - a - b;
            double zc = 1.0;
            for (int i = 0; i < c; i++) zc *= z;
            T4v[a][b] = (((a + b) & 1) ? -1.0 : 1.0) * zc * M.M7[a][b];
        }
    const double ns = nl[0] * sl[0] + nl[1] * sl[1] + nl[2] * sl[2];
    double u[3], w[3], u7[3], w7[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        u[r] = T5[r][0] * nl[0] + T5[r][1] * nl[1] + T5[r][2] * nl[2];
        w[r] = T5[r][0] * sl[0] + T5[r][1] * sl[1] + T5[r][2] * sl[2];
        u7[r] = T7[r][0] * nl[0] + T7[r][1] * nl[1] + T7[r][2] * nl[2];
        w7[r] = T7[r][0] * sl[0] + T7[r][1] * sl[1] + T7[r][2] * sl[2];
    }
    const double su = sl[0] * u[0] + sl[1] * u[1] + sl[2] * u[2];
    const double trT5 = T5[0][0] + T5[1][1] + T5[2][2];
    // symmetric products S_pq = sl_p n_q + n_p sl_q
    double S[3][3];
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
        for (int q = 0; q < 3; q++) S[p][q] = sl[p] * nl[q] + nl[p] * sl[q];
    double Bs[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int t = 0; t < 3; t++) {
            // T4 contractions: sum_pq T4[r,t,p,q] S_pq / 2 * 2 (= Q4(sl,n)+Q4(n,sl))
            double q4 = 0.0, t4c = 0.0;
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const int a = (r == 0) + (t == 0) + (p == 0) + (q == 0);
                    const int b = (r == 1) + (t == 1) + (p == 1) + (q == 1);
                    const double tv = T4v[a][b];
                    q4 += tv * S[p][q];
                    if (p == q) t4c += tv;
                }
            const double drt = (r == t) ? 1.0 : 0.0;
            const double X = (4.0 - c34) * I3 * drt + (3.0 * c34 - 18.0) * T5[r][t] -
                             3.0 * trT5 * drt + 15.0 * t4c + cblob * (15.0 * T7[r][t] - 3.0 * I5 * drt);
            const double Ysum = I3 * (1.0 - c34) * S[r][t] + 2.0 * drt * ns * I3 +
                                3.0 * (c34 - 1.0) * (sl[r] * u[t] + nl[r] * w[t]) -
                                6.0 * (sl[t] * u[r] + nl[t] * w[r]) - 6.0 * drt * su -
                                6.0 * ns * T5[r][t] + 15.0 * q4 +
                                cblob * (-3.0 * I5 * S[r][t] + 15.0 * (sl[r] * u7[t] + nl[r] * w7[t]));
            Bs[r][t] = C1 * (lam * ns * X + mu * Ysum);
        }
    const double trB = Bs[0][0] + Bs[1][1] + Bs[2][2];
#pragma unroll
    for (int m = 0; m < 3; m++)
#pragma unroll
        for (int n = m; n < 3; n++) {
            const double v = -((m == n ? lam * trB : 0.0) + mu * (Bs[m][n] + Bs[n][m]));
            out[m][n] = v;
            out[n][m] = v;
        }
}

// Force -> stress contracted with a force density, local frame
// (tri_kernels.py:857-897 contracted analytically).
__device__ __forceinline__ void kelvin_stress_local(const StressMoments& M, const double fl[3],
                                                    double mu, double lam, double C1, double c34,
                                                    double cbdg, double out[3][3]) {
    const double z = M.z;
    const double V3[3] = {-M.m3_10, -M.m3_01, z * M.I3};
    const double V5[3] = {-M.M5[1][0], -M.M5[0][1], z * M.M5[0][0]};
    // T3 local from M5: T[a][b][c] by counts
    double T3v[4][4];
#pragma unroll
    for (int a = 0; a <= 3; a++)
#pragma unroll
        for (int b = 0; a + b <= 3; b++) {
            const int c = 3 - a - b;
            double zc = 1.0;
            for (int i = 0; i < c; i++) zc *= z;
            T3v[a][b] = (((a + b) & 1) ? -1.0 : 1.0) * zc * M.M5[a][b];
        }
    double Tf[3][3];   // (T3 f)_ij
    double tvec[3];    // t_k = sum_i T3[i,k,i]
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const int a = (i == 0) + (j == 0) + (k == 0);
                const int b = (i == 1) + (j == 1) + (k == 1);
                acc += T3v[a][b] * fl[k];
            }
            Tf[i][j] = acc;
        }
        double acc = 0.0;
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const int a = 2 * (m == 0) + (i == 0);
            const int b = 2 * (m == 1) + (i == 1);
            acc += T3v[a][b];
        }
        tvec[i] = acc;
    }
    const double fV3 = fl[0] * V3[0] + fl[1] * V3[1] + fl[2] * V3[2];
    const double fV5 = fl[0] * V5[0] + fl[1] * V5[1] + fl[2] * V5[2];
    const double ft = fl[0] * tvec[0] + fl[1] * tvec[1] + fl[2] * tvec[2];
    const double tau = C1 * ((4.0 - c34) * fV3 - 3.0 * ft - cbdg * fV5);
    double Gf[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            Gf[i][j] = C1 * (-c34 * fl[i] * V3[j] + (i == j ? fV3 : 0.0) + fl[j] * V3[i] -
                             3.0 * Tf[i][j] - cbdg * fl[i] * V5[j]);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
            const double v = (i == j ? lam * tau : 0.0) + mu * (Gf[i][j] + Gf[j][i]);
            out[i][j] = v;
            out[j][i] = v;
        }
}

}  // namespace mbem
