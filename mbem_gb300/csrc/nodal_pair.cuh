// FP64 device code for one (observer, nodal P0/P1/P2 source triangle) pair.
//
// The mathematics is the reference's (src/mbem/kernels/tri_nodal.py:262-708):
// the raw moments M_n[a,b] = int_T xi1^a xi2^b / R^n dS (xi about the foot of
// the observer in the source's plane, n = -1 .. 7) come from the solid angle
// and the divergence-theorem recursion over the edge primitives
// int u^k / R^m du; beyond NODAL_D_STAR longest edges the smooth integrand is
// summed by a collapsed Gauss-Legendre rule instead.
//
// FP64 instructions are the cost of every pair here (one warp instruction
// takes 16 cycles of an SM's FP64 pipe, 60 issue slots of anything else), so
// the code is written to need few of them:
//  * order and kernel family are template parameters: every degree is known,
//    every table is in registers, no entry is formed that no kernel reads;
//  * everything that depends on the source alone is in one record per source;
//  * an edge evaluates one row of primitives, int u^k / R^m for the highest m,
//    by an n-point Gauss rule whose n follows from the ellipse on which the
//    integrand is analytic (a = (R_a + R_b) / L_e is its semi-axis; n = 7 at
//    a >= 26, 8 at 15, 9 at 9.3, 10 at 6.6, 12 at 3.9, 16 at 2.2 keep the
//    truncation below 1e-16 of int |u|^k / R^m), and the lower rows from it
//    (R^2 is a polynomial in u). The rule has no cancellation, so it replaces
//    both 32-term series (small |u| always has a >= 2.23) and, away from the
//    edge, the closed form; a large-|u| interval with a < 2.2 is summed in
//    pieces of ratio 2.5. Only what is left, an edge the observer is beside at
//    less than about its length, takes the closed form. The powers are of the
//    rule's own abscissa (tabulated with its weights), the edge's midpoint the
//    origin of the chain below;
//  * (A + t u)^a (B + t' u)^b integrates by a chain of two-term combinations;
//  * the far quadratures are fully symmetric rules of 12 to 42 points (degrees 6,
//    8, 9, 10, 12, 14), each from the distance on where it is off by less than 2e-16;
//  * a nodal matrix block is assembled from the blocks of the shifted moments
//    (one per monomial of the shape functions) instead of from one table per
//    node, and a contraction folds the density's polynomial into the moments;
//  * a source normal along the frame's (every mesh) drops the terms of the
//    other two components; any other normal takes the general forms.
#pragma once

#include "p0_pair.cuh"

namespace mbem {

// T, U, DD stress, eigenstress, Kelvin stress; TG and HG: T and DD for any source
// normal. For the frame's normal the trace identities |d|^2 = R^2 - eps^2 leave T
// with n = 5 to degree 2 (3 in general) and DD with n = 7 to degree 3 (4).
enum NodalFam { NF_T, NF_U, NF_H, NF_E, NF_S, NF_TG, NF_HG };

constexpr int ND_MAXK = 6;
constexpr double ND_D_STAR = 10.0;

__host__ __device__ constexpr int nd_nodes(int p) { return (p + 1) * (p + 2) / 2; }
__host__ __device__ constexpr int nd_max(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int nd_len(int d) { return d < 0 ? 1 : (d + 1) * (d + 2) / 2; }
__host__ __device__ constexpr int nd_edge(int d) { return d < 0 ? -1 : nd_max(d - 1, 0); }

// Moment degrees d_n of order P and family F (what the kernel reads plus the
// closure under the recursion and its seeds), and the edge degrees they need.
template <int P, int F>
struct NDeg {
    static constexpr bool H = F == NF_H || F == NF_HG;
    static constexpr int d7 = F == NF_H ? 3 + P : F == NF_HG ? 4 + P : F == NF_E ? P : -1;
    static constexpr int d5 = H ? 2 + P : F == NF_E ? 0 : F == NF_U ? -1 : F == NF_T ? 2 + P : 3 + P;
    static constexpr int d3 = H ? P : F == NF_E ? 0 : F == NF_U ? 2 + P : 1 + P;
    static constexpr int d1 = H ? (P >= 2 ? P - 2 : -1) : F == NF_E ? -1 : F == NF_U ? P : P - 1;
    static constexpr int dm1 = (F == NF_U && P == 2) ? 0 : -1;
    static constexpr int e5 = nd_edge(d7);
    static constexpr int e3 = nd_max(nd_edge(d5), d5 >= 0 ? 0 : -1);
    static constexpr int e1 = nd_max(d3 >= 1 ? d3 - 1 : -1, d1 >= 0 ? 0 : -1);
    static constexpr int em1 = nd_max(d1 >= 1 ? d1 - 1 : -1, dm1 >= 0 ? 0 : -1);
    static constexpr int top = e5 >= 0 ? 5 : e3 >= 0 ? 3 : 1;
    static constexpr int k5 = e5 < 0 ? -1 : nd_max(e5, nd_max(e3 >= 0 ? e3 + 2 : -1, e1 >= 0 ? e1 + 4 : -1));
    static constexpr int k3 = e3 < 0 ? -1 : nd_max(e3, nd_max(e1 >= 0 ? e1 + 2 : -1, em1 >= 0 ? em1 + 4 : -1));
    static constexpr int k1 = e1 < 0 ? -1 : nd_max(e1, em1 >= 0 ? em1 + 2 : -1);
    static constexpr int ktop = top == 5 ? k5 : top == 3 ? k3 : k1;
};

// The edge rules (n = 7, 8, 9, 10, 12, 16): abscissae and weights times their
// powers 0 .. 5; the last one's plain form also sums pieces. The far rules
// (12, 16, 19, 25, 33 and 42 points): barycentric l1, l2, the weight (sum 1/2) and the
// weight times the shape functions of P1 (3) and P2 (6).
constexpr int ND_EDGE_Q = 7 + 8 + 9 + 10 + 12 + 16;
constexpr int ND_FAR_Q = 12 + 16 + 19 + 25 + 33 + 42;
struct NodalRules {
    double ex[ND_EDGE_Q], ew[ND_EDGE_Q][6];
    double fl[ND_FAR_Q][3], fn[ND_FAR_Q][9];
};
#ifndef MBEM_ND_RULES
static __constant__ NodalRules c_nd;       // one copy per translation unit (nodal_rules_ready)
#define MBEM_ND_RULES c_nd
#endif

// The far rule, 0 .. 5 for 42, 33, 25, 19, 16, 12 points. Each is taken from the distance (in
// longest edges) on where its truncation is below 2e-16 of the pair's largest entry, a tenth of
// what the rounding of the sums leaves: against 196 points in 80-bit arithmetic over 1,200 random and slender triangles and
// directions, along edges and medians among them, eps from 0 to D, and 4 % farther out. The
// kernels differ by their highest power of 1 / R: U, T and Kelvin stress, DD stress, eigenstress.
// (With one line for all of them the P2 stress was off by 2e-14 at 10 longest edges and the
// P2 eigenstress by 8e-13; the lines for 5e-17 take another 12 % of the traction rows' time
// and 7 % of the P2 stress's.)
constexpr int ND_FAR_RULES = 6;
__host__ __device__ constexpr double nd_far_at(int P, int F, int k) {
    constexpr double never = 1e30;
    constexpr double at[3][4][ND_FAR_RULES - 1] = {
        {{0, 0, 0, 15.5, 33}, {0, 0, 13, 21.5, 49.5}, {0, 0, 16.5, 24.5, 69.5}, {0, 13.5, 22.5, 33, 94}},
        {{0, 0, 13.5, 24, 70.5}, {0, 11, 18.5, 33, 115}, {0, 13.5, 24.5, 40, 149}, {10.7, 18.7, 34, 54.5, 215}},
        {{0, 0, 20.2, 42.5, 187}, {0, 15, 30, 60.5, 315}, {0, 19.2, 40.7, 76, 435}, {13.8, 26.5, 53.5, 97, never}}};
    const double d = at[P][F == NF_U ? 0 : F == NF_E ? 3 : F == NF_H || F == NF_HG ? 2 : 1][k];
    return d * d;
}
template <int P, int F>
__device__ __forceinline__ int nd_far_rule(double D2, double L2) {
    constexpr double a0 = nd_far_at(P, F, 0), a1 = nd_far_at(P, F, 1), a2 = nd_far_at(P, F, 2), a3 = nd_far_at(P, F, 3),
                     a4 = nd_far_at(P, F, 4);
    if (D2 > a2 * L2) return D2 > a4 * L2 ? 5 : D2 > a3 * L2 ? 4 : 3;
    return a1 == 0.0 || D2 > a1 * L2 ? 2 : a0 == 0.0 || D2 > a0 * L2 ? 1 : 0;
}
// first and last + 1 point of rule r
__device__ __forceinline__ int nd_far_first(int r) {
    return r == 0 ? 105 : r == 1 ? 72 : r == 2 ? 47 : r == 3 ? 28 : r == 4 ? 12 : 0;
}
__device__ __forceinline__ int nd_far_last(int r) {
    return r == 0 ? 147 : r == 1 ? 105 : r == 2 ? 72 : r == 3 ? 47 : r == 4 ? 28 : 12;
}

// ---------------------------------------------------------------------------
// per-source record
// ---------------------------------------------------------------------------
struct NodalRec {
    double c[3], ex[3], ey[3], nh[3];
    double p2[3][2];          // vertices in the centroid frame
    double tx[3], ty[3], Le[3], iLe[3];
    double abc[3][3];         // lam_k(eta) = A_k + B_k eta1 + C_k eta2
    double area2s, area2;     // twice the area, in plane (signed) and in space
    double L2;                // longest edge squared
    double eps, eps2;
    double n[3], nl[3];       // the normal passed in, global and in the frame
    double s;                 // +-1 when it is along the frame's
    // slim: height below a tenth of the longest edge. The shape polynomials of
    // P2 about the foot then cancel by (distance / height)^2.
    bool ok, aligned, slim;
};

static __device__ __noinline__ void nodal_rec(const double* __restrict__ tv, const double* __restrict__ nrm, double eps,
                                 NodalRec& g) {
    SrcP0 s0;
    src_setup(tv, eps, s0);
    g.ok = s0.ok;
    g.eps = eps;
    g.eps2 = eps * eps;
    for (int k = 0; k < 3; k++) {
        g.ex[k] = s0.ex[k]; g.ey[k] = s0.ey[k]; g.nh[k] = s0.nh[k];
        g.c[k] = ((tv[k] + tv[3 + k]) + tv[6 + k]) / 3.0;
        g.n[k] = nrm ? nrm[k] : 0.0;
    }
    for (int k = 0; k < 3; k++) {
        const double dx = tv[3 * k] - g.c[0], dy = tv[3 * k + 1] - g.c[1], dz = tv[3 * k + 2] - g.c[2];
        g.p2[k][0] = dx * g.ex[0] + dy * g.ex[1] + dz * g.ex[2];
        g.p2[k][1] = dx * g.ey[0] + dy * g.ey[1] + dz * g.ey[2];
    }
    const double (*p)[2] = g.p2;
    g.L2 = 0.0;
    for (int k = 0; k < 3; k++) {
        const int b = (k + 1) % 3;
        const double dx = tv[3 * b] - tv[3 * k], dy = tv[3 * b + 1] - tv[3 * k + 1], dz = tv[3 * b + 2] - tv[3 * k + 2];
        g.L2 = fmax(g.L2, dx * dx + dy * dy + dz * dz);
        const double ux = p[b][0] - p[k][0], uy = p[b][1] - p[k][1];
        const double Le = sqrt(ux * ux + uy * uy);
        g.Le[k] = Le;
        g.iLe[k] = 1.0 / Le;
        g.tx[k] = ux / Le;
        g.ty[k] = uy / Le;
    }
    const double e1x = tv[3] - tv[0], e1y = tv[4] - tv[1], e1z = tv[5] - tv[2];
    const double e2x = tv[6] - tv[0], e2y = tv[7] - tv[1], e2z = tv[8] - tv[2];
    const double cx = e1y * e2z - e1z * e2y, cy = e1z * e2x - e1x * e2z, cz = e1x * e2y - e1y * e2x;
    g.area2 = sqrt(cx * cx + cy * cy + cz * cz);
    const double den = (p[1][0] - p[0][0]) * (p[2][1] - p[0][1]) - (p[1][1] - p[0][1]) * (p[2][0] - p[0][0]);
    g.area2s = den;
    for (int k = 0; k < 3; k++) {
        const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
        const double x1 = p[k1][0], y1 = p[k1][1], x2 = p[k2][0], y2 = p[k2][1];
        g.abc[k][0] = (x1 * y2 - y1 * x2) / den;
        g.abc[k][1] = (y1 - y2) / den;
        g.abc[k][2] = (x2 - x1) / den;
    }
    g.nl[0] = g.n[0] * g.ex[0] + g.n[1] * g.ex[1] + g.n[2] * g.ex[2];
    g.nl[1] = g.n[0] * g.ey[0] + g.n[1] * g.ey[1] + g.n[2] * g.ey[2];
    g.nl[2] = g.n[0] * g.nh[0] + g.n[1] * g.nh[1] + g.n[2] * g.nh[2];
    // a unit normal along the frame's, to the rounding of both
    g.s = g.nl[2] < 0.0 ? -1.0 : 1.0;
    g.slim = g.area2 < 0.1 * g.L2;
    g.aligned = fabs(g.nl[0]) < 1e-15 && fabs(g.nl[1]) < 1e-15 && fabs(fabs(g.nl[2]) - 1.0) < 1e-15;
}

// The observer in the source's frame.
struct NodalObs {
    double z, X1, X2, h2, D2;
};
__device__ __forceinline__ NodalObs nodal_obs(const NodalRec& g, const double* x) {
    const double dx = x[0] - g.c[0], dy = x[1] - g.c[1], dz = x[2] - g.c[2];
    NodalObs o;
    o.z = dx * g.nh[0] + dy * g.nh[1] + dz * g.nh[2];
    o.X1 = dx * g.ex[0] + dy * g.ex[1] + dz * g.ex[2];
    o.X2 = dx * g.ey[0] + dy * g.ey[1] + dz * g.ey[2];
    o.h2 = o.z * o.z + g.eps2;
    o.D2 = (dx * dx + dy * dy + dz * dz) + g.eps2;
    return o;
}
__device__ __forceinline__ bool nodal_is_far(const NodalRec& g, const NodalObs& o) {
    return o.D2 > (ND_D_STAR * ND_D_STAR) * g.L2;
}

// ---------------------------------------------------------------------------
// edge primitives
// ---------------------------------------------------------------------------
template <int P, int F>
struct EdgePrim {
    typedef NDeg<P, F> G;
    // int v^k / R^m dv with u = off + step v, step included on use
    double p5[nd_max(G::k5, 0) + 1], p3[nd_max(G::k3, 0) + 1], p1[nd_max(G::k1, 0) + 1], pm1[nd_max(G::em1, 0) + 1];
    double off, step;
};

// s[k] = sum_q w_q x_q^k / R^TOP at u_q = uc + hl x_q
template <int TOP, int KT>
__device__ __forceinline__ void edge_gauss(double uc, double hl, double rho2, int q0, int q1, double s[KT + 1]) {
#pragma unroll
    for (int k = 0; k <= KT; k++) s[k] = 0.0;
#pragma unroll 2
    for (int q = q0; q < q1; q++) {
        const double u = uc + hl * MBEM_ND_RULES.ex[q];
        double f;
        if constexpr (TOP == 1) f = rsqrt(u * u + rho2);
        else f = inv_pow64<TOP>(u * u + rho2);
#pragma unroll
        for (int k = 0; k <= KT; k++) s[k] += f * MBEM_ND_RULES.ew[q][k];
    }
}
// acc[k] += int u^k / R^TOP over a piece of the edge (n = 16)
template <int TOP, int KT>
__device__ __noinline__ void edge_piece(double uc, double hl, double rho2, double acc[KT + 1]) {
#pragma unroll 1
    for (int q = ND_EDGE_Q - 16; q < ND_EDGE_Q; q++) {
        const double u = uc + hl * MBEM_ND_RULES.ex[q];
        const double iR = rsqrt(u * u + rho2);
        double f = hl * MBEM_ND_RULES.ew[q][0] * iR;
        for (int m = 1; m < TOP; m += 2) f *= iR * iR;
        acc[0] += f;
#pragma unroll
        for (int k = 1; k <= KT; k++) {
            f *= u;
            acc[k] += f;
        }
    }
}

// conjugate closed-form differences (tri_nodal.py:346-382) and the upward
// recursion P_m[k] = P_{m-2}[k-2] - rho^2 P_m[k-2]
template <int P, int F>
__device__ __noinline__ void edge_closed(double ua, double ub, double Le, double rho2, EdgePrim<P, F>& E) {
    typedef NDeg<P, F> G;
    const double ra2 = ua * ua + rho2, rb2 = ub * ub + rho2;
    const double Ra = sqrt(ra2), Rb = sqrt(rb2);
    const double us = ua + ub;
    const double dR = Le * us / (Ra + Rb);
    // J1: log of a quotient, as log1p of the part that the same-signed terms leave
    const bool pos = ua >= 0.0, neg = ub <= 0.0;
    const double num = pos ? Le + dR : neg ? Le - dR : (ub + Rb) * (Ra - ua) - rho2;
    const double den = pos ? ua + Ra : neg ? Rb - ub : rho2;
    const double dJ1 = log1p(num / den);
    const double RaRb = Ra * Rb;
    const double dJ3 = (ua * ub > 0.0) ? (Le * us) / (RaRb * (ub * Ra + ua * Rb)) : (ub / Rb - ua / Ra) / rho2;
    const double S3 = (Rb * Rb + RaRb) + Ra * Ra;
    if (G::e1 >= 0 || G::k1 >= 0) {
        E.p1[0] = dJ1;
        if (G::k1 >= 1) E.p1[1] = dR;
    }
    if (G::em1 >= 0) {
        const double duR = 0.5 * Le * (Ra + Rb) + 0.5 * us * dR;
        E.pm1[0] = 0.5 * (duR + rho2 * dJ1);
        if (G::em1 >= 1) E.pm1[1] = dR * S3 / 3.0;
    }
    double p1l[nd_max(G::k5 - 4, nd_max(G::k3 - 2, 0)) + 2];     // row 1 as far as the rows above use it
    p1l[0] = dJ1;
    p1l[1] = dR;
    if (G::e3 >= 0) {
        E.p3[0] = dJ3;
        if (G::k3 >= 1) E.p3[1] = dR / RaRb;
    }
    if (G::e5 >= 0) {
        const double duRm = ub / (rb2 * Rb) - ua / (ra2 * Ra);
        E.p5[0] = (duRm + 2.0 * dJ3) / (3.0 * rho2);
        if (G::k5 >= 1) E.p5[1] = dR * S3 / (3.0 * (RaRb * RaRb * RaRb));
    }
#pragma unroll
    for (int k = 2; k <= 5; k++) {
        if (G::top > 1 && k <= nd_max(G::k5 - 4, G::k3 - 2)) {
            // row 1 beyond its first two: only P = 2 stress and displacement, from row -1
            const double duR = 0.5 * Le * (Ra + Rb) + 0.5 * us * dR;
            const double m1 = k == 2 ? 0.5 * (duR + rho2 * dJ1) : dR * S3 / 3.0;
            p1l[k] = m1 - rho2 * p1l[k - 2];
        }
        if (G::top == 1 && k <= G::e1) E.p1[k] = E.pm1[k - 2] - rho2 * E.p1[k - 2];
        if (G::top > 1 && k <= G::k1) E.p1[k] = p1l[k];
        if (k <= G::k3) E.p3[k] = p1l[k - 2] - rho2 * E.p3[k - 2];
        if (k <= G::k5) E.p5[k] = E.p3[k - 2] - rho2 * E.p5[k - 2];
    }
}

// |u| from umin >= 2 rho up, in pieces of ratio 2.5; an odd power keeps the sign of u
template <int P, int F>
__device__ __noinline__ void edge_pieces(double ua, double ub, double rho2, EdgePrim<P, F>& E) {
    typedef NDeg<P, F> G;
    double t[G::ktop + 1];
#pragma unroll
    for (int k = 0; k <= G::ktop; k++) t[k] = 0.0;
    const double b = fmax(fabs(ua), fabs(ub));
    double t0 = fmin(fabs(ua), fabs(ub));
#pragma unroll 1
    while (t0 < b) {
        double t1 = 2.5 * t0;
        if (!(t1 < b)) t1 = b;
        edge_piece<G::top, G::ktop>(0.5 * (t0 + t1), 0.5 * (t1 - t0), rho2, t);
        t0 = t1;
    }
    if (ua < 0.0)
#pragma unroll
        for (int k = 1; k <= G::ktop; k += 2) t[k] = -t[k];
    // lower rows: u^k / R^(m-2) = u^(k+2) / R^m + rho^2 u^k / R^m
#pragma unroll
    for (int k = 0; k <= G::k5; k++) E.p5[k] = t[k];
#pragma unroll
    for (int k = 0; k <= G::k3; k++) E.p3[k] = G::top == 5 ? t[k + 2 <= G::ktop ? k + 2 : 0] + rho2 * t[k] : t[k];
#pragma unroll
    for (int k = 0; k <= G::k1; k++)
        E.p1[k] = G::top > 1 ? E.p3[k + 2 <= G::k3 ? k + 2 : 0] + rho2 * E.p3[k <= G::k3 ? k : 0] : t[k];
#pragma unroll
    for (int k = 0; k <= G::em1; k++) E.pm1[k] = E.p1[k + 2 <= G::k1 ? k + 2 : 0] + rho2 * E.p1[k];
}

// The primitives of one edge, u in [ua, ub] (ub - ua = Le), rho^2 = R^2 - u^2.
template <int P, int F>
__device__ __forceinline__ void edge_primitives(double ua, double ub, double Le, double iLe, double RaRb_sum,
                                                double rho2, EdgePrim<P, F>& E) {
    typedef NDeg<P, F> G;
    const double a = RaRb_sum * iLe;
    const double umin = fmin(fabs(ua), fabs(ub));
    if (a >= 2.2) {
        const double uc = 0.5 * (ua + ub), hl = 0.5 * Le;
        // offsets 0, 7, 15, 24, 34, 46 of n = 7, 8, 9, 10, 12, 16
        const int q0 = a >= 26.0 ? 0 : a >= 15.0 ? 7 : a >= 9.3 ? 15 : a >= 6.6 ? 24 : a >= 3.9 ? 34 : 46;
        const int q1 = a >= 26.0 ? 7 : a >= 15.0 ? 15 : a >= 9.3 ? 24 : a >= 6.6 ? 34 : a >= 3.9 ? 46 : 62;
        double t[G::ktop + 1];
        edge_gauss<G::top, G::ktop>(uc, hl, rho2, q0, q1, t);
        E.off = uc;
        E.step = hl;
        // lower rows: R^2 = hl^2 x^2 + 2 uc hl x + (uc^2 + rho^2)
        const double r0 = uc * uc + rho2, r1 = Le * uc, r2 = hl * hl;
#pragma unroll
        for (int k = 0; k <= G::k5; k++) E.p5[k] = t[k];
#pragma unroll
        for (int k = 0; k <= G::k3; k++)
            E.p3[k] = G::top == 5 ? (r0 * t[k] + r1 * t[k + 1 <= G::ktop ? k + 1 : 0]) + r2 * t[k + 2 <= G::ktop ? k + 2 : 0]
                                  : t[k];
#pragma unroll
        for (int k = 0; k <= G::k1; k++)
            E.p1[k] = G::top > 1 ? (r0 * E.p3[k <= G::k3 ? k : 0] + r1 * E.p3[k + 1 <= G::k3 ? k + 1 : 0]) +
                                       r2 * E.p3[k + 2 <= G::k3 ? k + 2 : 0]
                                 : t[k];
#pragma unroll
        for (int k = 0; k <= G::em1; k++)
            E.pm1[k] = (r0 * E.p1[k] + r1 * E.p1[k + 1 <= G::k1 ? k + 1 : 0]) + r2 * E.p1[k + 2 <= G::k1 ? k + 2 : 0];
        return;
    }
    E.off = 0.0;
    E.step = 1.0;
    if (ua * ub > 0.0 && umin * umin >= 4.0 * rho2) {
        edge_pieces<P, F>(ua, ub, rho2, E);
    } else {
        edge_closed<P, F>(ua, ub, Le, rho2, E);
    }
}

// bn1[a,b] += c1 int (A + tx u)^a (B + ty u)^b / R^m, bn2[b] += c2 (a = 0), a + b <= D
template <int D, int N>
__device__ __forceinline__ void edge_chain(const double (&p)[N], double A, double B, double tx, double ty, double c1,
                                           double c2, double* bn1, double* bn2) {
    double va[D + 1];
#pragma unroll
    for (int k = 0; k <= D; k++) va[k] = p[k];
#pragma unroll
    for (int a = 0; a <= D; a++) {
        double vb[D + 1];
#pragma unroll
        for (int k = 0; k <= D - a; k++) vb[k] = va[k];
#pragma unroll
        for (int b = 0; b <= D - a; b++) {
            bn1[nd_tri(a, b)] += c1 * vb[0];
            if (a == 0) bn2[b] += c2 * vb[0];
#pragma unroll
            for (int k = 0; k < D - a - b; k++) vb[k] = B * vb[k] + ty * vb[k + 1];
        }
#pragma unroll
        for (int k = 0; k < D - a; k++) va[k] = A * va[k] + tx * va[k + 1];
    }
}

// ---------------------------------------------------------------------------
// raw moments about the foot (tri_nodal.py:519-619)
// ---------------------------------------------------------------------------
template <int P, int F>
struct NMom {
    typedef NDeg<P, F> G;
    double m7[nd_len(G::d7)], m5[nd_len(G::d5)], m3[nd_len(G::d3)], m1[nd_len(G::d1)], mm1[1];
};

// M[a,b] (a + b = 1 .. D) from the row below: ML of degree >= D - 2
template <int D, int DL>
__device__ __forceinline__ void moment_row(double* M, const double* ML, const double* bn1, const double* bn2,
                                           double inv) {
#pragma unroll
    for (int q = 1; q <= D; q++)
#pragma unroll
        for (int b = 0; b <= q; b++) {
            const int a = q - b;
            double v;
            if (a >= 1) {
                v = -bn1[nd_tri(a - 1, b)];
                if (a >= 2) v += (a - 1) * ML[nd_tri(a - 2, b)];
            } else {
                v = -bn2[b - 1];
                if (b >= 2) v += (b - 1) * ML[nd_tri(0, b - 2)];
            }
            M[nd_tri(a, b)] = v * inv;
        }
}

template <int P, int F>
__device__ __forceinline__ void nodal_moments(const NodalRec& g, const NodalObs& o, NMom<P, F>& M) {
    typedef NDeg<P, F> G;
    const double h2 = o.h2;
    const double ih = rsqrt(h2), h = h2 * ih;
    double px[3], py[3], R[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        px[k] = g.p2[k][0] - o.X1;
        py[k] = g.p2[k][1] - o.X2;
        const double r2 = px[k] * px[k] + py[k] * py[k] + h2;
        R[k] = r2 * rsqrt(r2);
    }
    // I3 from the solid angle of the lifted point
    const double d01 = px[0] * px[1] + py[0] * py[1] + h2;
    const double d12 = px[1] * px[2] + py[1] * py[2] + h2;
    const double d02 = px[0] * px[2] + py[0] * py[2] + h2;
    // (the P2 kernels keep the library's: the short one took their stress at 512 sources x
    // 2,000 points from 4.9 to 5.6 ms, P1 matrices from 4.3 to 4.1 with the edges' powers)
    const double num = -h * g.area2s, den = R[0] * R[1] * R[2] + R[2] * d01 + R[0] * d12 + R[1] * d02;
    const double I3 = -2.0 * (P < 2 ? angle64(num, den) : atan2(num, den)) * ih;

    constexpr int e5 = G::e5, e3 = G::e3, e1 = G::e1, em1 = G::em1;
    double b5[nd_len(e5)], c5[nd_max(e5, 0) + 1], b3[nd_len(e3)], c3[nd_max(e3, 0) + 1], b1[nd_len(e1)],
        c1v[nd_max(e1, 0) + 1], bm[nd_len(em1)], cm[nd_max(em1, 0) + 1];
#pragma unroll
    for (int i = 0; i < nd_len(e5); i++) b5[i] = 0.0;
#pragma unroll
    for (int i = 0; i < nd_len(e3); i++) b3[i] = 0.0;
#pragma unroll
    for (int i = 0; i < nd_len(e1); i++) b1[i] = 0.0;
#pragma unroll
    for (int i = 0; i < nd_len(em1); i++) bm[i] = 0.0;
#pragma unroll
    for (int i = 0; i <= e5; i++) c5[i] = 0.0;
#pragma unroll
    for (int i = 0; i <= e3; i++) c3[i] = 0.0;
#pragma unroll
    for (int i = 0; i <= e1; i++) c1v[i] = 0.0;
#pragma unroll
    for (int i = 0; i <= em1; i++) cm[i] = 0.0;
    double bd5 = 0.0, bd3 = 0.0, bd1 = 0.0, bdm = 0.0;
#pragma unroll 1
    for (int e = 0; e < 3; e++) {
        const double pax = e == 0 ? px[0] : e == 1 ? px[1] : px[2], pay = e == 0 ? py[0] : e == 1 ? py[1] : py[2];
        const double pbx = e == 0 ? px[1] : e == 1 ? px[2] : px[0], pby = e == 0 ? py[1] : e == 1 ? py[2] : py[0];
        const double Rs = e == 0 ? R[0] + R[1] : e == 1 ? R[1] + R[2] : R[2] + R[0];
        const double tx = g.tx[e], ty = g.ty[e];
        const double n1 = ty, n2 = -tx;
        const double dp = pax * n1 + pay * n2;
        const double ua = pax * tx + pay * ty, ub = pbx * tx + pby * ty;
        const double rho2 = dp * dp + h2;
        EdgePrim<P, F> E;
        edge_primitives<P, F>(ua, ub, g.Le[e], g.iLe[e], Rs, rho2, E);
        // the point of the edge at v: (A + sx v, B + sy v)
        const double A = dp * n1 + E.off * tx, B = dp * n2 + E.off * ty;
        const double sx = E.step * tx, sy = E.step * ty;
        const double m1 = E.step * n1, m2 = E.step * n2, ds = E.step * dp;
        if (e5 >= 0) {
            bd5 += ds * E.p5[0];
            if (G::d7 >= 1) edge_chain<nd_max(e5, 0)>(E.p5, A, B, sx, sy, m1, m2, b5, c5);
        }
        if (e3 >= 0) {
            bd3 += ds * E.p3[0];
            if (G::d5 >= 1) edge_chain<nd_max(e3, 0)>(E.p3, A, B, sx, sy, m1, m2, b3, c3);
        }
        if (e1 >= 0) {
            bd1 += ds * E.p1[0];
            if (G::d3 >= 1) edge_chain<nd_max(e1, 0)>(E.p1, A, B, sx, sy, m1, m2, b1, c1v);
        }
        if (em1 >= 0) {
            bdm += ds * E.pm1[0];
            if (G::d1 >= 1) edge_chain<nd_max(em1, 0)>(E.pm1, A, B, sx, sy, m1, m2, bm, cm);
        }
    }
    const double ih2 = ih * ih;
    M.m3[0] = I3;
    if (G::d5 >= 0) M.m5[0] = (bd3 + I3) * ih2 * (1.0 / 3.0);
    if (G::d7 >= 0) M.m7[0] = (bd5 + 3.0 * M.m5[0]) * ih2 * 0.2;
    if (G::d1 >= 0) M.m1[0] = bd1 - h2 * I3;
    if (G::dm1 >= 0) M.mm1[0] = (bdm + h2 * M.m1[0]) * (1.0 / 3.0);
    if (G::d1 >= 1) moment_row<nd_max(G::d1, 0), G::dm1>(M.m1, M.mm1, bm, cm, -1.0);
    if (G::d3 >= 1) moment_row<nd_max(G::d3, 0), G::d1>(M.m3, M.m1, b1, c1v, 1.0);
    if (G::d5 >= 1) moment_row<nd_max(G::d5, 0), G::d3>(M.m5, M.m3, b3, c3, 1.0 / 3.0);
    if (G::d7 >= 1) moment_row<nd_max(G::d7, 0), G::d5>(M.m7, M.m5, b5, c5, 0.2);
}

// ---------------------------------------------------------------------------
// shape functions
// ---------------------------------------------------------------------------
// Coefficients of N_k about the foot on the monomials 1, xi1, xi2, xi1^2,
// xi1 xi2, xi2^2 (index nd_tri); l[i] = lam_i at the foot.
template <int P>
__device__ __forceinline__ void shape_about_foot(const NodalRec& g, const double l[3], int k, double C[nd_nodes(P)]) {
    if (P == 0) {
        C[0] = 1.0;
    } else if (P == 1) {
        C[0] = l[k];
        C[1] = g.abc[k][1];
        C[2] = g.abc[k][2];
    } else if (k < 3) {
        const double B = g.abc[k][1], Cc = g.abc[k][2];
        const double q = 4.0 * l[k] - 1.0;
        C[0] = l[k] * (2.0 * l[k] - 1.0);
        C[1] = B * q;
        C[2] = Cc * q;
        C[3] = 2.0 * B * B;
        C[4] = 4.0 * B * Cc;
        C[5] = 2.0 * Cc * Cc;
    } else {
        const int i = k - 3, j = i == 2 ? 0 : i + 1;
        const double Bi = 4.0 * g.abc[i][1], Ci = 4.0 * g.abc[i][2], li = 4.0 * l[i];
        const double Bj = g.abc[j][1], Cj = g.abc[j][2], lj = l[j];
        C[0] = li * lj;
        C[1] = li * Bj + Bi * lj;
        C[2] = li * Cj + Ci * lj;
        C[3] = Bi * Bj;
        C[4] = Bi * Cj + Ci * Bj;
        C[5] = Ci * Cj;
    }
}
__device__ __forceinline__ void lam_at_foot(const NodalRec& g, const NodalObs& o, double l[3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) l[i] = (g.abc[i][0] + o.X1 * g.abc[i][1]) + o.X2 * g.abc[i][2];
}
// W[a,b] (a + b <= D) = sum over monomials C[ap,bp] M[a + ap, b + bp]
template <int P, int D>
__device__ __forceinline__ void weight_moments(const double* M, const double* C, double* W) {
#pragma unroll
    for (int q = 0; q <= D; q++)
#pragma unroll
        for (int b = 0; b <= q; b++) {
            double acc = C[0] * M[nd_tri(q - b, b)];
#pragma unroll
            for (int t = 1; t <= P; t++)
#pragma unroll
                for (int bp = 0; bp <= t; bp++)
                    acc += C[nd_tri(t - bp, bp)] * M[nd_tri(q - b + t - bp, b + bp)];
            W[nd_tri(q - b, b)] = acc;
        }
}

// The per-node weighted tables of a near pair, for what the fast forms do not
// take: a normal off the frame's, and slim P2 sources, whose weights cancel so
// far that all kernels have to read the same bits (one out-of-line function,
// compiled alike everywhere, instead of one inlined copy a kernel).
template <int P>
struct NodeTab {
    double w1[nd_nodes(P)], w3[nd_nodes(P)][6], w5[nd_nodes(P)][10], w7[nd_nodes(P)][15];
};
template <int P, int F>
__device__ __noinline__ void node_tables(const NodalRec& g, const double* x, NodeTab<P>& W) {
    const NodalObs o = nodal_obs(g, x);
    NMom<P, F> M;
    nodal_moments<P, F>(g, o, M);
    double l[3];
    lam_at_foot(g, o, l);
#pragma unroll 1
    for (int k = 0; k < nd_nodes(P); k++) {
        double C[nd_nodes(P)];
        shape_about_foot<P>(g, l, k, C);
        if constexpr (F == NF_U) {
            weight_moments<P, 0>(M.m1, C, &W.w1[k]);
            weight_moments<P, 2>(M.m3, C, W.w3[k]);
        } else if constexpr (F == NF_TG || F == NF_S) {
            weight_moments<P, 1>(M.m3, C, W.w3[k]);
            weight_moments<P, 3>(M.m5, C, W.w5[k]);
        } else if constexpr (F == NF_HG) {
            weight_moments<P, 0>(M.m3, C, W.w3[k]);
            weight_moments<P, 2>(M.m5, C, W.w5[k]);
            weight_moments<P, 4>(M.m7, C, W.w7[k]);
        } else {
            weight_moments<P, 0>(M.m7, C, W.w7[k]);
        }
    }
}
template <int P>
__device__ __forceinline__ bool node_by_node(const NodalRec& g) { return P == 2 && g.slim; }

// ---------------------------------------------------------------------------
// local forms (source frame)
// ---------------------------------------------------------------------------
// The T block (source frame, normal s e3) of the moments shifted by (SA, SB).
template <int SA, int SB>
__device__ __forceinline__ void t_local_shift(const double* m3, const double* m5, double z, double eps2,
                                              const TCoef& c, double s, double B[3][3]) {
#define M3_(a, b) m3[nd_tri((a) + SA, (b) + SB)]
#define M5_(a, b) m5[nd_tri((a) + SA, (b) + SB)]
    t_local(M3_(0, 0), M3_(1, 0), M3_(0, 1), M5_(0, 0), M5_(1, 0), M5_(0, 1), M5_(2, 0), M5_(1, 1), M5_(0, 2), z, eps2,
            c, s, B);
#undef M3_
#undef M5_
}

// column j of the T block (source frame, any normal nl) of one moment set
template <int J>
__device__ __forceinline__ void t_local_col(const double* m3, const double* m5, double z, double eps2,
                                            const TCoef& c, const double nl[3], double out[3]) {
    const double z2 = z * z;
    const double V3[3] = {-m3[1], -m3[2], z * m3[0]};
    const double V5[3] = {-m5[1], -m5[2], z * m5[0]};
    const double T000 = -m5[nd_tri(3, 0)], T001 = -m5[nd_tri(2, 1)], T002 = z * m5[nd_tri(2, 0)],
                 T011 = -m5[nd_tri(1, 2)], T012 = z * m5[nd_tri(1, 1)], T022 = -z2 * m5[nd_tri(1, 0)],
                 T111 = -m5[nd_tri(0, 3)], T112 = z * m5[nd_tri(0, 2)], T122 = -z2 * m5[nd_tri(0, 1)],
                 T222 = z2 * z * m5[0];
    const double c5 = c.c5 * eps2, ce6 = c.ce6 * eps2;
    // T3[i][J][.] . nl
    double W[3];
    if (J == 0) {
        W[0] = T000 * nl[0] + T001 * nl[1] + T002 * nl[2];
        W[1] = T001 * nl[0] + T011 * nl[1] + T012 * nl[2];
        W[2] = T002 * nl[0] + T012 * nl[1] + T022 * nl[2];
    } else if (J == 1) {
        W[0] = T001 * nl[0] + T011 * nl[1] + T012 * nl[2];
        W[1] = T011 * nl[0] + T111 * nl[1] + T112 * nl[2];
        W[2] = T012 * nl[0] + T112 * nl[1] + T122 * nl[2];
    } else {
        W[0] = T002 * nl[0] + T012 * nl[1] + T022 * nl[2];
        W[1] = T012 * nl[0] + T112 * nl[1] + T122 * nl[2];
        W[2] = T022 * nl[0] + T122 * nl[1] + T222 * nl[2];
    }
    double be[3];
#pragma unroll
    for (int i = 0; i < 3; i++) be[i] = c.cb * V3[i] + ce6 * V5[i];
    const double gam = nl[0] * be[0] + nl[1] * be[1] + nl[2] * be[2];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double al = c.c3 * V3[i] + c5 * V5[i];
        out[i] += nl[J] * al + nl[i] * be[J] + c.w6 * W[i] + (i == J ? gam : 0.0);
    }
}

// the same for any normal nl and a slip sl (source frame) through the general
// contraction; m5 to degree 2, m7 to degree 4
static __device__ __noinline__ void dd_general(const double* m3, const double* m5, const double* m7, double z, double eps2,
                                        const SMat& m, const double nl[3], const double sl[3], bool eig,
                                        double out[6]) {
    StressMoments S;
    S.z = z;
    S.I3 = m3[0];
    S.m3_10 = S.m3_01 = 0.0;
    for (int a = 0; a < 4; a++)
        for (int b = 0; b < 4; b++) S.M5[a][b] = a + b <= 2 ? m5[nd_tri(a, b)] : 0.0;
    for (int a = 0; a < 5; a++)
        for (int b = 0; b < 5; b++) S.M7[a][b] = a + b <= 4 ? m7[nd_tri(a, b)] : 0.0;
    double loc[3][3];
    dd_stress_local(S, nl, sl, m.mu, m.lam, m.C1, m.c34, m.blob * eps2, loc);
    const double phi = eig ? m.phi * eps2 * eps2 * m7[0] : 0.0;
    const double ns = nl[0] * sl[0] + nl[1] * sl[1] + nl[2] * sl[2];
    const int ia[6] = {0, 1, 2, 0, 0, 1}, ib[6] = {0, 1, 2, 1, 2, 2};
    for (int t = 0; t < 6; t++) {
        const int i = ia[t], j = ib[t];
        out[t] += loc[i][j] - phi * ((i == j ? m.lam * ns : 0.0) + m.mu * (sl[i] * nl[j] + nl[i] * sl[j]));
    }
}

// Kelvin stress (source frame) of a force fl with the moments m3, m5
__device__ __forceinline__ void kelvin_six(const double* m3, const double* m5, double z, double eps2, const SMat& m,
                                           const double fl[3], double out[6]) {
    StressMoments S;
    S.z = z;
    S.I3 = m3[0];
    S.m3_10 = m3[1];
    S.m3_01 = m3[2];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) S.M5[a][b] = a + b <= 3 ? m5[nd_tri(a, b <= 3 - a ? b : 0)] : 0.0;
    double loc[3][3];
    kelvin_stress_local(S, fl, m.mu, m.lam, m.C1, m.c34, 3.0 * m.blob * eps2, loc);
    out[0] += loc[0][0]; out[1] += loc[1][1]; out[2] += loc[2][2];
    out[3] += loc[0][1]; out[4] += loc[0][2]; out[5] += loc[1][2];
}

// ---------------------------------------------------------------------------
// far quadrature: fn(xi1, xi2, R^2, q) at every point q; sums are times 2 area
// ---------------------------------------------------------------------------
template <class Fn>
__device__ __forceinline__ void far_points(const NodalRec& g, const NodalObs& o, int rule, Fn&& fn) {
    const double e1x = g.p2[1][0] - g.p2[0][0], e1y = g.p2[1][1] - g.p2[0][1];
    const double e2x = g.p2[2][0] - g.p2[0][0], e2y = g.p2[2][1] - g.p2[0][1];
    const double ox = g.p2[0][0] - o.X1, oy = g.p2[0][1] - o.X2;
    const int q1 = nd_far_last(rule);
#pragma unroll 1
    for (int q = nd_far_first(rule); q < q1; q++) {
        const double l1 = MBEM_ND_RULES.fl[q][0], l2 = MBEM_ND_RULES.fl[q][1];
        const double xi1 = ox + l1 * e1x + l2 * e2x, xi2 = oy + l1 * e1y + l2 * e2y;
        fn(xi1, xi2, xi1 * xi1 + xi2 * xi2 + o.h2, q);
    }
}
// weight of point q times the shape function of node k
template <int P>
__device__ __forceinline__ double far_wn(int q, int k) {
    return P == 0 ? MBEM_ND_RULES.fl[q][2] : MBEM_ND_RULES.fn[q][(P == 2 ? 3 : 0) + k];
}

// ---------------------------------------------------------------------------
// matrix blocks: put(k, G) receives node k's 3 x 3 block (global frame)
// ---------------------------------------------------------------------------
// T block (source frame) of one moment set and any normal
__device__ __forceinline__ void t_general(const double* W3, const double* W5, double z, const NodalRec& g,
                                          const TCoef& c, double T[3][3]) {
    double col[3][3];
#pragma unroll
    for (int j = 0; j < 3; j++) col[j][0] = col[j][1] = col[j][2] = 0.0;
    t_local_col<0>(W3, W5, z, g.eps2, c, g.nl, col[0]);
    t_local_col<1>(W3, W5, z, g.eps2, c, g.nl, col[1]);
    t_local_col<2>(W3, W5, z, g.eps2, c, g.nl, col[2]);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) T[i][j] = col[j][i];
}

// The far T blocks of a normal off the frame's.
template <int P, class Put>
__device__ __noinline__ void far_t_general(const NodalRec& g, const double* x, const TCoef& c, Put&& put) {
    constexpr int K = nd_nodes(P);
    const NodalObs o = nodal_obs(g, x);
    double W3[K][3], W5[K][10];
    for (int k = 0; k < K; k++) {
        for (int t = 0; t < 3; t++) W3[k][t] = 0.0;
        for (int t = 0; t < 10; t++) W5[k][t] = 0.0;
    }
    far_points(g, o, nd_far_rule<P, NF_T>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
        const double iR = rsqrt(R2), iR2 = iR * iR;
        const double a = iR * iR2, b = a * iR2;
        const double x11 = xi1 * xi1, x22 = xi2 * xi2;
        const double p[10] = {1.0, xi1, xi2, x11, xi1 * xi2, x22, x11 * xi1, x11 * xi2, x22 * xi1, x22 * xi2};
        for (int k = 0; k < K; k++) {
            const double w = g.area2 * far_wn<P>(q, k), wa = w * a, wb = w * b;
            for (int t = 0; t < 3; t++) W3[k][t] += wa * p[t];
            for (int t = 0; t < 10; t++) W5[k][t] += wb * p[t];
        }
    });
    for (int k = 0; k < K; k++) {
        double T[3][3], G[3][3];
        t_general(W3[k], W5[k], o.z, g, c, T);
        rotate_full(g, T, G);
        put(k, G);
    }
}

template <int P, class Put>
__device__ __forceinline__ void pair_t_block(const NodalRec& g, const double* x, const TCoef& c, Put&& put) {
    constexpr int K = nd_nodes(P);
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z;
    if (nodal_is_far(g, o)) {
        if (!g.aligned) {
            far_t_general<P>(g, x, c, put);
            return;
        }
        // per node: n = 3 and n = 5 to degree 2 but (0, 2), which (2, 0) leaves of I3 - h^2 I5
        double acc[K][8];
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int t = 0; t < 8; t++) acc[k][t] = 0.0;
        far_points(g, o, nd_far_rule<P, NF_T>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
            const double iR = rsqrt(R2), iR2 = iR * iR;
            const double a = iR * iR2, b = a * iR2;
            const double b1 = b * xi1, b2 = b * xi2;
            const double p[8] = {a, a * xi1, a * xi2, b, b1, b2, b1 * xi1, b1 * xi2};
#pragma unroll
            for (int k = 0; k < K; k++) {
                const double w = far_wn<P>(q, k);
#pragma unroll
                for (int t = 0; t < 8; t++) acc[k][t] += w * p[t];
            }
        });
#pragma unroll
        for (int k = 0; k < K; k++) {
            const double* m = acc[k];
            double T[3][3], G[3][3];
            t_local(m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7], m[0] - o.h2 * m[3] - m[6], z, g.eps2, c,
                    g.s * g.area2, T);
            rotate_full(g, T, G);
            put(k, G);
        }
        return;
    }
    if (!g.aligned || node_by_node<P>(g)) {
        NodeTab<P> W;
        node_tables<P, NF_TG>(g, x, W);
#pragma unroll 1
        for (int k = 0; k < K; k++) {
            double T[3][3], G[3][3];
            t_general(W.w3[k], W.w5[k], z, g, c, T);
            rotate_full(g, T, G);
            put(k, G);
        }
        return;
    }
    NMom<P, NF_T> M;
    nodal_moments<P, NF_T>(g, o, M);
    double l[3];
    lam_at_foot(g, o, l);
    // the block of every shifted moment set, then the shape coefficients
    double B[nd_nodes(P)][3][3];
#define MBEM_ND_SHIFT(sa, sb)                                                                        \
{                                                                                                \
    double T[3][3];                                                                              \
    t_local_shift<sa, sb>(M.m3, M.m5, z, g.eps2, c, g.s, T);                                     \
    rotate_full(g, T, B[nd_tri(sa, sb)]);                                                        \
}
    MBEM_ND_SHIFT(0, 0)
    if constexpr (P >= 1) {
        MBEM_ND_SHIFT(1, 0)
        MBEM_ND_SHIFT(0, 1)
    }
    if constexpr (P >= 2) {
        MBEM_ND_SHIFT(2, 0)
        MBEM_ND_SHIFT(1, 1)
        MBEM_ND_SHIFT(0, 2)
    }
#undef MBEM_ND_SHIFT
#pragma unroll
    for (int k = 0; k < K; k++) {
        double C[K], G[3][3];
        shape_about_foot<P>(g, l, k, C);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                double v = C[0] * B[0][i][j];
#pragma unroll
                for (int t = 1; t < K; t++) v += C[t] * B[t][i][j];
                G[i][j] = v;
            }
        put(k, G);
    }
}

// The six T basis blocks of node k: put(k, blocks).
template <int P, class Put>
__device__ __forceinline__ void pair_t_basis(const NodalRec& g, const double* x, Put&& put) {
    constexpr int K = nd_nodes(P);
    const NodalObs o = nodal_obs(g, x);
    double W3[K][3], W5[K][10];
    if (nodal_is_far(g, o)) {
        for (int k = 0; k < K; k++) {
            for (int t = 0; t < 3; t++) W3[k][t] = 0.0;
            for (int t = 0; t < 10; t++) W5[k][t] = 0.0;
        }
        far_points(g, o, nd_far_rule<P, NF_H>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
            const double iR = rsqrt(R2), iR2 = iR * iR;
            const double a = iR * iR2, b = a * iR2;
            const double x11 = xi1 * xi1, x22 = xi2 * xi2;
            const double p[10] = {1.0, xi1, xi2, x11, xi1 * xi2, x22, x11 * xi1, x11 * xi2, x22 * xi1, x22 * xi2};
            for (int k = 0; k < K; k++) {
                const double w = g.area2 * far_wn<P>(q, k), wa = w * a, wb = w * b;
                for (int t = 0; t < 3; t++) W3[k][t] += wa * p[t];
                for (int t = 0; t < 10; t++) W5[k][t] += wb * p[t];
            }
        });
    } else {
        NMom<P, NF_TG> M;
        nodal_moments<P, NF_TG>(g, o, M);
        double l[3];
        lam_at_foot(g, o, l);
#pragma unroll
        for (int k = 0; k < K; k++) {
            double C[K];
            shape_about_foot<P>(g, l, k, C);
            weight_moments<P, 1>(M.m3, C, W3[k]);
            weight_moments<P, 3>(M.m5, C, W5[k]);
        }
    }
#pragma unroll 1
    for (int k = 0; k < K; k++) {
        TScal q;
        q.z = o.z;
        q.I3 = W3[k][0]; q.m10_3 = W3[k][1]; q.m01_3 = W3[k][2];
        q.I5 = W5[k][0]; q.m10_5 = W5[k][1]; q.m01_5 = W5[k][2];
        q.m20_5 = W5[k][3]; q.m11_5 = W5[k][4]; q.m02_5 = W5[k][5];
        q.m30_5 = W5[k][6]; q.m21_5 = W5[k][7]; q.m12_5 = W5[k][8]; q.m03_5 = W5[k][9];
        TMoments m;
        t_from_scal(g.ex, g.ey, g.nh, g.n, q, m);
        double blk[6][3][3];
        t_basis_blocks(m, g.n, g.eps2, blk);
        put(k, blk);
    }
}

// U: put(k, I1, I3, T2) with T2 = int N_k d d / R^3 as 00 11 22 01 02 12
// (global frame) times c2, I1 = int N_k / R and I3 = int N_k / R^3. F: the far rules' family
// (the blocks by themselves: I3 falls off as the T kernel does)
template <int P, int F, class Put>
__device__ __forceinline__ void pair_u(const NodalRec& g, const double* x, double c2, Put&& put) {
    constexpr int K = nd_nodes(P);
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z;
    double A[K][8];        // per monomial (near) or node (far): T2 and I1, I3
    if (nodal_is_far(g, o)) {
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int t = 0; t < 8; t++) A[k][t] = 0.0;
        far_points(g, o, nd_far_rule<P, F>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
            const double iR = rsqrt(R2), iR2 = iR * iR;
            const double a = iR * iR2;
            const double v0 = a * xi1, v1 = a * xi2;
            // (0, 2) is what (2, 0) leaves of I1 - h^2 I3
            const double p[6] = {iR, a, v0, v1, v0 * xi1, v0 * xi2};
#pragma unroll
            for (int k = 0; k < K; k++) {
                const double w = far_wn<P>(q, k);
#pragma unroll
                for (int t = 0; t < 6; t++) A[k][t] += w * p[t];
            }
        });
        const double f = c2 * g.area2;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const double* p = A[k];
            const double L[6] = {f * p[4], f * (p[0] - o.h2 * p[1] - p[4]), f * (z * z) * p[1],
                                 f * p[5], -f * z * p[2],                    -f * z * p[3]};
            double G[6];
            rotate_six(g, L, G);
            put(k, g.area2 * p[0], g.area2 * p[1], G);
        }
        return;
    }
    NMom<P, NF_U> M;
    nodal_moments<P, NF_U>(g, o, M);
    double l[3];
    lam_at_foot(g, o, l);
#define MBEM_ND_SHIFT(sa, sb)                                                                                       \
    {                                                                                                               \
        const double L[6] = {c2 * M.m3[nd_tri(2 + sa, sb)], c2 * M.m3[nd_tri(sa, 2 + sb)],                          \
                             c2 * (z * z) * M.m3[nd_tri(sa, sb)], c2 * M.m3[nd_tri(1 + sa, 1 + sb)],                \
                             -c2 * z * M.m3[nd_tri(1 + sa, sb)], -c2 * z * M.m3[nd_tri(sa, 1 + sb)]};               \
        rotate_six(g, L, A[nd_tri(sa, sb)]);                                                                        \
        A[nd_tri(sa, sb)][6] = M.m1[nd_tri(sa, sb)];                                                                \
        A[nd_tri(sa, sb)][7] = M.m3[nd_tri(sa, sb)];                                                                \
    }
    MBEM_ND_SHIFT(0, 0)
    if constexpr (P >= 1) {
        MBEM_ND_SHIFT(1, 0)
        MBEM_ND_SHIFT(0, 1)
    }
    if constexpr (P >= 2) {
        MBEM_ND_SHIFT(2, 0)
        MBEM_ND_SHIFT(1, 1)
        MBEM_ND_SHIFT(0, 2)
    }
#undef MBEM_ND_SHIFT
#pragma unroll
    for (int k = 0; k < K; k++) {
        double C[K], G[8];
        shape_about_foot<P>(g, l, k, C);
#pragma unroll
        for (int t = 0; t < 8; t++) {
            double v = C[0] * A[0][t];
#pragma unroll
            for (int q = 1; q < K; q++) v += C[q] * A[q][t];
            G[t] = v;
        }
        put(k, G[6], G[7], G);
    }
}

// ---------------------------------------------------------------------------
// contractions: the density as a polynomial per frame component
// ---------------------------------------------------------------------------
template <int P>
struct NodalDen {
    double f[3][nd_nodes(P)];      // about the centroid, on 1, eta1, eta2, eta1^2, eta1 eta2, eta2^2
    double node[nd_nodes(P)][3];   // the nodal values (frame)
    bool zero;
};
template <int P>
__device__ inline void nodal_den(const NodalRec& g, const double* __restrict__ d, NodalDen<P>& D) {
    constexpr int K = nd_nodes(P);
    const double l[3] = {g.abc[0][0], g.abc[1][0], g.abc[2][0]};
    D.zero = true;
    for (int j = 0; j < 3; j++)
        for (int t = 0; t < K; t++) D.f[j][t] = 0.0;
    for (int k = 0; k < K; k++) {
        double C[K], dl[3];
        shape_about_foot<P>(g, l, k, C);
        to_frame(g, d + 3 * k, dl);
        for (int j = 0; j < 3; j++) {
            D.node[k][j] = dl[j];
            D.zero = D.zero && d[3 * k + j] == 0.0;
            for (int t = 0; t < K; t++) D.f[j][t] += C[t] * dl[j];
        }
    }
}
// the same polynomial about the foot (X1, X2)
template <int P>
__device__ __forceinline__ void den_at_foot(const double* f, double X1, double X2, double* q) {
    if (P == 0) {
        q[0] = f[0];
    } else if (P == 1) {
        q[0] = f[0] + f[1] * X1 + f[2] * X2;
        q[1] = f[1];
        q[2] = f[2];
    } else {
        const double a = f[1] + f[3] * X1 + f[4] * X2, b = f[2] + f[5] * X2;
        q[0] = f[0] + a * X1 + b * X2;
        q[1] = a + f[3] * X1;
        q[2] = b + f[4] * X1 + f[5] * X2;
        q[3] = f[3];
        q[4] = f[4];
        q[5] = f[5];
    }
}
// Far pairs take the density from its nodal values and the rule's weighted shape functions:
// u = w sum_k N_k d_k at point q. (From the polynomial about the centroid at the point's
// coordinates, which lose D / L of their digits about the foot, the displacement of slender
// triangles was off by 1e-12 at 30 longest edges.)
template <int P>
__device__ __forceinline__ void far_density(const NodalDen<P>& D, int q, double u[3]) {
    const double w0 = far_wn<P>(q, 0);
#pragma unroll
    for (int j = 0; j < 3; j++) u[j] = w0 * D.node[0][j];
#pragma unroll
    for (int k = 1; k < nd_nodes(P); k++) {
        const double w = far_wn<P>(q, k);
#pragma unroll
        for (int j = 0; j < 3; j++) u[j] += w * D.node[k][j];
    }
}

// far displacement of a slip density on a normal off the frame's (source frame)
template <int P>
__device__ __noinline__ void far_t_contract_general(const NodalRec& g, const NodalDen<P>& D, const double* x,
                                                    const TCoef& c, double v[3]) {
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z, c5 = c.c5 * g.eps2, ce6 = c.ce6 * g.eps2;
    const double n0 = g.nl[0], n1 = g.nl[1], n2 = g.nl[2];
    far_points(g, o, nd_far_rule<P, NF_T>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
        double u[3];
        far_density<P>(D, q, u);
        const double u0 = u[0], u1 = u[1], u2 = u[2];
        const double iR = rsqrt(R2), iR2 = iR * iR;
        const double a = g.area2 * iR * iR2, b = a * iR2;
        const double pa = c.c3 * a + c5 * b, pb = c.cb * a + ce6 * b;
        const double d0 = -xi1, d1 = -xi2;
        const double dn = d0 * n0 + d1 * n1 + z * n2, du = d0 * u0 + d1 * u1 + z * u2;
        const double un = u0 * n0 + u1 * n1 + u2 * n2;
        // (n.u) pa d + n pb (d.u) - 6 c5 b (d.n)(d.u) d + pb (d.n) u
        const double s = un * pa + c.w6 * b * dn * du, t = pb * du, r = pb * dn;
        v[0] += s * d0 + t * n0 + r * u0;
        v[1] += s * d1 + t * n1 + r * u1;
        v[2] += s * z + t * n2 + r * u2;
    });
}

// displacement of a slip density, added to acc (global)
template <int P>
__device__ __forceinline__ void pair_t_contract(const NodalRec& g, const NodalDen<P>& D, const double* x,
                                                const TCoef& c, double acc[3]) {
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z;
    double v[3] = {0.0, 0.0, 0.0};
    if (nodal_is_far(g, o)) {
        if (!g.aligned) {
            far_t_contract_general<P>(g, D, x, c, v);
        } else {
            // normal s e3: s [ q d + pb z u + e3 sum pb (d.u) ], q = pa u3 + w6 z b (d.u)
            const double c5 = c.c5 * g.eps2, ce6 = c.ce6 * g.eps2, wz = c.w6 * z;
            double s0 = 0.0, s1 = 0.0, sq = 0.0, sd = 0.0, t0 = 0.0, t1 = 0.0, t2 = 0.0;
            far_points(g, o, nd_far_rule<P, NF_T>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
                double u[3];
                far_density<P>(D, q, u);
                const double u0 = u[0], u1 = u[1], u2 = u[2];
                const double iR = rsqrt(R2), iR2 = iR * iR;
                const double a = iR * iR2, b = a * iR2;
                const double pa = c.c3 * a + c5 * b, pb = c.cb * a + ce6 * b;
                const double du = z * u2 - (xi1 * u0 + xi2 * u1);
                const double r = pa * u2 + (wz * b) * du;
                s0 += r * xi1;
                s1 += r * xi2;
                sq += r;
                sd += pb * du;
                t0 += pb * u0;
                t1 += pb * u1;
                t2 += pb * u2;
            });
            const double sa = g.s * g.area2;
            v[0] = sa * (z * t0 - s0);
            v[1] = sa * (z * t1 - s1);
            v[2] = sa * (z * (t2 + sq) + sd);
        }
    } else if (!g.aligned || node_by_node<P>(g)) {
        NodeTab<P> W;
        node_tables<P, NF_TG>(g, x, W);
#pragma unroll 1
        for (int k = 0; k < nd_nodes(P); k++) {
            double q[3][3];
#pragma unroll
            for (int j = 0; j < 3; j++) q[j][0] = q[j][1] = q[j][2] = 0.0;
            t_local_col<0>(W.w3[k], W.w5[k], z, g.eps2, c, g.nl, q[0]);
            t_local_col<1>(W.w3[k], W.w5[k], z, g.eps2, c, g.nl, q[1]);
            t_local_col<2>(W.w3[k], W.w5[k], z, g.eps2, c, g.nl, q[2]);
            const double* d = D.node[k];
#pragma unroll
            for (int i = 0; i < 3; i++) v[i] += q[0][i] * d[0] + q[1][i] * d[1] + q[2][i] * d[2];
        }
    } else {
        NMom<P, NF_T> M;
        nodal_moments<P, NF_T>(g, o, M);
#define MBEM_ND_COL(j)                                                \
    {                                                                 \
        double C[nd_nodes(P)], W3[3], W5[6], B[3][3];                 \
        den_at_foot<P>(D.f[j], o.X1, o.X2, C);                        \
        weight_moments<P, 1>(M.m3, C, W3);                            \
        weight_moments<P, 2>(M.m5, C, W5);                            \
        t_local_shift<0, 0>(W3, W5, z, g.eps2, c, g.s, B);            \
        v[0] += B[0][j];                                              \
        v[1] += B[1][j];                                              \
        v[2] += B[2][j];                                              \
    }
        MBEM_ND_COL(0)
        MBEM_ND_COL(1)
        MBEM_ND_COL(2)
#undef MBEM_ND_COL
    }
#pragma unroll
    for (int i = 0; i < 3; i++) acc[i] += g.ex[i] * v[0] + g.ey[i] * v[1] + g.nh[i] * v[2];
}

// displacement of a force density: c[0] I1 + c[1] eps^2 I3 on the diagonal, c[2] T2
template <int P>
__device__ __forceinline__ void pair_u_contract(const NodalRec& g, const NodalDen<P>& D, const double* x,
                                                const double c[3], double acc[3]) {
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z;
    const double ce = c[1] * g.eps2;
    double v[3] = {0.0, 0.0, 0.0};
    if (nodal_is_far(g, o)) {
        far_points(g, o, nd_far_rule<P, NF_U>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
            double u[3];
            far_density<P>(D, q, u);
            const double u0 = u[0], u1 = u[1], u2 = u[2];
            const double iR = rsqrt(R2), iR2 = iR * iR;
            const double a = iR * iR2;
            const double dg = c[0] * iR + ce * a, s = a * (z * u2 - (xi1 * u0 + xi2 * u1));
            v[0] += dg * u0 - (c[2] * s) * xi1;
            v[1] += dg * u1 - (c[2] * s) * xi2;
            v[2] += dg * u2 + (c[2] * s) * z;
        });
#pragma unroll
        for (int i = 0; i < 3; i++) v[i] *= g.area2;
    } else if (node_by_node<P>(g)) {
        NodeTab<P> W;
        node_tables<P, NF_U>(g, x, W);
#pragma unroll 1
        for (int k = 0; k < nd_nodes(P); k++) {
            const double* d = D.node[k];
            const double* w = W.w3[k];
            const double dg = c[0] * W.w1[k] + ce * w[0];
            v[0] += dg * d[0] + c[2] * (w[3] * d[0] + w[4] * d[1] - z * w[1] * d[2]);
            v[1] += dg * d[1] + c[2] * (w[4] * d[0] + w[5] * d[1] - z * w[2] * d[2]);
            v[2] += dg * d[2] + c[2] * z * (z * w[0] * d[2] - w[1] * d[0] - w[2] * d[1]);
        }
    } else {
        NMom<P, NF_U> M;
        nodal_moments<P, NF_U>(g, o, M);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double C[nd_nodes(P)], W1[1], W3[6];
            den_at_foot<P>(D.f[j], o.X1, o.X2, C);
            weight_moments<P, 0>(M.m1, C, W1);
            weight_moments<P, 2>(M.m3, C, W3);
            const double L[3][3] = {{W3[3], W3[4], -z * W3[1]},
                                    {W3[4], W3[5], -z * W3[2]},
                                    {-z * W3[1], -z * W3[2], z * z * W3[0]}};
#pragma unroll
            for (int i = 0; i < 3; i++) v[i] += c[2] * L[i][j] + (i == j ? c[0] * W1[0] + ce * W3[0] : 0.0);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; i++) acc[i] += g.ex[i] * v[0] + g.ey[i] * v[1] + g.nh[i] * v[2];
}

// eigenstress phi C : sym(s n) of I7 = int s / R^7 (source frame)
__device__ __forceinline__ void eig_six(const SMat& m, double eps2, const double nl[3], const double I7[3],
                                        double e[6]) {
    const double phi = m.phi * eps2 * eps2;
    const double un = nl[0] * I7[0] + nl[1] * I7[1] + nl[2] * I7[2];
    const int ia[6] = {0, 1, 2, 0, 0, 1}, ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int t = 0; t < 6; t++) {
        const int i = ia[t], j = ib[t];
        e[t] = phi * ((i == j ? m.lam * un : 0.0) + m.mu * (I7[i] * nl[j] + nl[i] * I7[j]));
    }
}

// Far DD stress and I7 = int u / R^7 for the normal s e3 (source frame): with a,
// b, c = w / R^3, 5, 7, d = (-xi, z) and |d|^2 = R^2 - eps^2 every term is one of
// f d d (f as below), G (z u + (d.u) e3) d, A u, and scalars in u3 and d.u, so the
// sums are of those and the stress is formed once.
template <int P>
__device__ __forceinline__ void far_dd_frame(const NodalRec& g, const NodalDen<P>& D, const NodalObs& o, int rule,
                                             const SMat& m, double v[6], double I7[3]) {
    const double z = o.z, e = g.eps2, cb = m.blob * e, c15 = 15.0 * cb, ce = 15.0 * (cb - e);
    const double lam = m.lam, mu = m.mu, xt = m.x1 + 15.0;
    // f = u3 (kb b + kc c) + kd c (d.u)
    const double kb = 2.0 * lam * xt - 12.0 * mu, kc = 2.0 * lam * ce, kd = 60.0 * mu * z;
    double S00 = 0, S01 = 0, S11 = 0, f0s = 0, f1s = 0, fs = 0, au[3] = {0, 0, 0}, bu[3] = {0, 0, 0}, cu[3] = {0, 0, 0};
    double bd = 0, cd = 0, V0 = 0, V1 = 0, W0[3] = {0, 0, 0}, W1[3] = {0, 0, 0};
    far_points(g, o, rule, [&](double xi1, double xi2, double R2, int q) {
        double u[3];
        far_density<P>(D, q, u);
        const double iR = rsqrt(R2), iR2 = iR * iR;
        const double a = iR * iR2, b = a * iR2, c = b * iR2;
        const double du = z * u[2] - (xi1 * u[0] + xi2 * u[1]);
        const double bq = b * du, cq = c * du;
        const double f = u[2] * (kb * b + kc * c) + kd * cq;
        const double f0 = f * xi1, f1 = f * xi2;
        S00 += f0 * xi1;
        S01 += f0 * xi2;
        S11 += f1 * xi2;
        f0s += f0;
        f1s += f1;
        fs += f;
        bd += bq;
        cd += cq;
        const double ge = m.k3a * bq + c15 * cq, G = m.k3a * b + c15 * c;
        V0 += ge * xi1;
        V1 += ge * xi2;
#pragma unroll
        for (int i = 0; i < 3; i++) {
            au[i] += a * u[i];
            bu[i] += b * u[i];
            cu[i] += c * u[i];
            const double gu = G * u[i];
            W0[i] += gu * xi1;
            W1[i] += gu * xi2;
        }
    });
    const double A0 = 1.0 - m.c34, B0 = 3.0 * (e - cb), l2 = 2.0 * lam, m2 = 2.0 * mu;
    // lam tr Bs + the delta part of Bs + Bs^T, over C1
    const double ka = lam * lam * (3.0 * A0 + xt) + 2.0 * lam * mu * A0 + mu * (l2 * A0 + 2.0 * m2);
    const double kb3 = lam * lam * (3.0 * B0 - e * xt + ce) + lam * mu * 6.0 * (e - cb) + mu * l2 * B0;
    const double kc3 = -lam * lam * e * ce;
    const double pb = lam * mu * (12.0 + 2.0 * m.k3a) - 6.0 * mu * m2, pc = 2.0 * lam * mu * ce;
    const double su = ka * au[2] + kb3 * bu[2] + kc3 * cu[2] + z * (pb * bd + pc * cd);
    // Q = A u; W[j] = sum G d_j u (times z below), V = sum G (d.u) d
    double Q[3], W2[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        Q[i] = A0 * au[i] - 3.0 * cb * bu[i];
        W2[i] = z * (m.k3a * bu[i] + c15 * cu[i]);
        W0[i] = -W0[i];
        W1[i] = -W1[i];
    }
    const double V2 = z * (m.k3a * bd + c15 * cd);
    const double s = -m.C1 * g.s * g.area2;
    v[0] = s * (mu * (S00 + mu * (2.0 * z * W0[0])) + su);
    v[1] = s * (mu * (S11 + mu * (2.0 * z * W1[1])) + su);
    v[2] = s * (mu * (z * z * fs + mu * (4.0 * Q[2] + 2.0 * (z * W2[2] + V2))) + su);
    v[3] = s * mu * (S01 + mu * z * (W0[1] + W1[0]));
    v[4] = s * mu * (mu * (2.0 * Q[0] + z * (W0[2] + W2[0]) - V0) - z * f0s);
    v[5] = s * mu * (mu * (2.0 * Q[1] + z * (W1[2] + W2[1]) - V1) - z * f1s);
#pragma unroll
    for (int i = 0; i < 3; i++) I7[i] = g.area2 * cu[i];
}

// the same for any normal
template <int P>
__device__ __noinline__ void far_dd_general(const NodalRec& g, const NodalDen<P>& D, const double* x, int rule,
                                            const SMat& m, double v[6], double I7[3]) {
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z, e2 = g.eps2;
    const double n0 = g.nl[0], n1 = g.nl[1], n2 = g.nl[2];
    const double cb = m.blob * e2;
    // sums of the point form: DD = e d d + g (w d + d w) + a (u n + n u) + delta s
    double S[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, V[3] = {0.0, 0.0, 0.0}, su = 0.0, Q[3] = {0.0, 0.0, 0.0};
    double W[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    const double l2 = 2.0 * m.lam, mu2 = 2.0 * m.mu;
    far_points(g, o, rule, [&](double xi1, double xi2, double R2, int q) {
        double u[3];
        far_density<P>(D, q, u);
        const double iR = rsqrt(R2), iR2 = iR * iR;
        const double a = g.area2 * iR * iR2, b = a * iR2, c = b * iR2;
        const double dd = R2 - e2;
        const double d[3] = {-xi1, -xi2, z};
        const double dn = d[0] * n0 + d[1] * n1 + z * n2, du = d[0] * u[0] + d[1] * u[1] + z * u[2];
        const double un = u[0] * n0 + u[1] * n1 + u[2] * n2;
        const double db = dd + cb;
        const double X0 = (4.0 - m.c34) * a - 3.0 * db * b;
        const double X1 = m.x1 * b + 15.0 * db * c;
        const double A1 = (1.0 - m.c34) * a - 3.0 * cb * b;
        const double p = du * dn;
        const double S0 = 2.0 * un * a - 6.0 * p * b;
        const double G = m.k3a * b + 15.0 * cb * c;
        const double E = 30.0 * p * c - 6.0 * un * b;
        const double ux = un * X1;
        // Bs + Bs^T = delta (l2 un X0 + mu2 S0) + (l2 un X1 + mu2 E) d d + mu (2 A1 sym + G (w d + d w)), w = dn u + du n
        const double f = l2 * ux + mu2 * E;
        S[0] += f * d[0] * d[0]; S[1] += f * d[1] * d[1]; S[2] += f * z * z;
        S[3] += f * d[0] * d[1]; S[4] += f * d[0] * z; S[5] += f * d[1] * z;
        const double trX = 3.0 * (un * X0) + ux * dd;
        const double trS = 2.0 * (A1 * un) + 3.0 * S0 + 2.0 * (G * p) + E * dd;
        su += m.lam * (m.lam * trX + m.mu * trS) + m.mu * (l2 * (un * X0) + mu2 * S0);
        for (int i = 0; i < 3; i++) {
            Q[i] += A1 * u[i];
            V[i] += G * du * d[i];
            I7[i] += c * u[i];
            for (int j = 0; j < 3; j++) W[i][j] += G * dn * d[i] * u[j];
        }
    });
    const double nl[3] = {n0, n1, n2};
    const int ia[6] = {0, 1, 2, 0, 0, 1}, ib[6] = {0, 1, 2, 1, 2, 2};
    for (int t = 0; t < 6; t++) {
        const int i = ia[t], j = ib[t];
        const double sym = Q[i] * nl[j] + nl[i] * Q[j];
        const double wd = W[i][j] + W[j][i] + V[i] * nl[j] + nl[i] * V[j];
        v[t] = -m.C1 * (m.mu * (S[t] + m.mu * (2.0 * sym + wd)) + (i == j ? su : 0.0));
    }
}

// stress of a slip density (DD, minus the eigenstress with EIG) added to acc (00 11 22 01 02 12, global); with
// acc_e the eigenstress alone is added there
template <int P>
__device__ __forceinline__ void pair_dd_contract(const NodalRec& g, const NodalDen<P>& D, const double* x,
                                                 const SMat& m, bool eig, double acc[6], double* acc_e) {
    const NodalObs o = nodal_obs(g, x);
    const double z = o.z, e2 = g.eps2;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double I7[3] = {0.0, 0.0, 0.0};          // int u / R^7
    const double n0 = g.nl[0], n1 = g.nl[1], n2 = g.nl[2];
    if (nodal_is_far(g, o)) {
        const int rule = acc_e ? nd_far_rule<P, NF_E>(o.D2, g.L2) : nd_far_rule<P, NF_H>(o.D2, g.L2);
        if (g.aligned) far_dd_frame<P>(g, D, o, rule, m, v, I7);
        else far_dd_general<P>(g, D, x, rule, m, v, I7);
        if (eig) {
            const double nl[3] = {n0, n1, n2};
            double e[6];
            eig_six(m, e2, nl, I7, e);
#pragma unroll
            for (int t = 0; t < 6; t++) v[t] -= e[t];
        }
    } else {
        if (!g.aligned || node_by_node<P>(g)) {
            NodeTab<P> W;
            node_tables<P, NF_HG>(g, x, W);
#pragma unroll 1
            for (int k = 0; k < nd_nodes(P); k++) {
                const double* sl = D.node[k];
                dd_general(W.w3[k], W.w5[k], W.w7[k], z, e2, m, g.nl, sl, eig, v);
#pragma unroll
                for (int j = 0; j < 3; j++) I7[j] += W.w7[k][0] * sl[j];
            }
        } else {
            NMom<P, NF_H> M;
            nodal_moments<P, NF_H>(g, o, M);
#define MBEM_ND_COL(j)                                              \
    {                                                               \
        double C[nd_nodes(P)], W3[1], W5[6], W7[10];                \
        den_at_foot<P>(D.f[j], o.X1, o.X2, C);                      \
        weight_moments<P, 0>(M.m3, C, W3);                          \
        weight_moments<P, 2>(M.m5, C, W5);                          \
        weight_moments<P, 3>(M.m7, C, W7);                          \
        I7[j] = W7[0];                                              \
        dd_unit<j>(W3, W5, W7, z, e2, m, eig, g.s, v);              \
    }
            MBEM_ND_COL(0)
            MBEM_ND_COL(1)
            MBEM_ND_COL(2)
#undef MBEM_ND_COL
        }
    }
    if (acc_e) {
        const double nl[3] = {n0, n1, n2};
        double e[6], G[6];
        eig_six(m, e2, nl, I7, e);
        rotate_six(g, e, G);
        for (int t = 0; t < 6; t++) acc_e[t] += G[t];
    }
    double G[6];
    rotate_six(g, v, G);
#pragma unroll
    for (int t = 0; t < 6; t++) acc[t] += G[t];
}

// eigenstress of a slip density
template <int P>
__device__ __forceinline__ void pair_eig_contract(const NodalRec& g, const NodalDen<P>& D, const double* x,
                                                  const SMat& m, double acc[6]) {
    const NodalObs o = nodal_obs(g, x);
    double I7[3] = {0.0, 0.0, 0.0};
    if (nodal_is_far(g, o)) {
        far_points(g, o, nd_far_rule<P, NF_E>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
            double u[3];
            far_density<P>(D, q, u);
            const double iR = rsqrt(R2), iR2 = iR * iR;
            const double c = iR * (iR2 * iR2) * iR2;
#pragma unroll
            for (int j = 0; j < 3; j++) I7[j] += c * u[j];
        });
#pragma unroll
        for (int j = 0; j < 3; j++) I7[j] *= g.area2;
    } else if (node_by_node<P>(g)) {
        NodeTab<P> W;
        node_tables<P, NF_E>(g, x, W);
#pragma unroll 1
        for (int k = 0; k < nd_nodes(P); k++)
#pragma unroll
            for (int j = 0; j < 3; j++) I7[j] += W.w7[k][0] * D.node[k][j];
    } else {
        NMom<P, NF_E> M;
        nodal_moments<P, NF_E>(g, o, M);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double C[nd_nodes(P)];
            den_at_foot<P>(D.f[j], o.X1, o.X2, C);
            weight_moments<P, 0>(M.m7, C, &I7[j]);
        }
    }
    double e[6], G[6];
    eig_six(m, g.eps2, g.nl, I7, e);
    rotate_six(g, e, G);
#pragma unroll
    for (int t = 0; t < 6; t++) acc[t] += G[t];
}

// the moments m3 (degree 1) and m5 (degree 3) of a density component by quadrature
template <int P>
__device__ __forceinline__ void far_s_moments(const NodalRec& g, const NodalObs& o, const NodalDen<P>& D,
                                              double W3[3][3], double W5[3][10]) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
#pragma unroll
        for (int t = 0; t < 3; t++) W3[j][t] = 0.0;
#pragma unroll
        for (int t = 0; t < 10; t++) W5[j][t] = 0.0;
    }
    far_points(g, o, nd_far_rule<P, NF_S>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q) {
        double u[3];
        far_density<P>(D, q, u);
        const double iR = rsqrt(R2), iR2 = iR * iR;
        const double a = g.area2 * iR * iR2, b = a * iR2;
        const double x11 = xi1 * xi1, x12 = xi1 * xi2, x22 = xi2 * xi2;
        const double p[10] = {1.0, xi1, xi2, x11, x12, x22, x11 * xi1, x11 * xi2, x22 * xi1, x22 * xi2};
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double ua = u[j] * a, ub = u[j] * b;
#pragma unroll
            for (int t = 0; t < 3; t++) W3[j][t] += ua * p[t];
#pragma unroll
            for (int t = 0; t < 10; t++) W5[j][t] += ub * p[t];
        }
    });
}

// Kelvin stress of a force density
template <int P>
__device__ __forceinline__ void pair_kelvin_contract(const NodalRec& g, const NodalDen<P>& D, const double* x,
                                                     const SMat& m, double acc[6]) {
    const NodalObs o = nodal_obs(g, x);
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, G[6];
    if (nodal_is_far(g, o)) {
        double W3[3][3], W5[3][10];
        far_s_moments<P>(g, o, D, W3, W5);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double fl[3] = {j == 0 ? 1.0 : 0.0, j == 1 ? 1.0 : 0.0, j == 2 ? 1.0 : 0.0};
            kelvin_six(W3[j], W5[j], o.z, g.eps2, m, fl, v);
        }
    } else if (node_by_node<P>(g)) {
        NodeTab<P> W;
        node_tables<P, NF_S>(g, x, W);
#pragma unroll 1
        for (int k = 0; k < nd_nodes(P); k++)
            kelvin_six(W.w3[k], W.w5[k], o.z, g.eps2, m, D.node[k], v);
    } else {
        NMom<P, NF_S> M;
        nodal_moments<P, NF_S>(g, o, M);
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double C[nd_nodes(P)], W3[3], W5[10];
            den_at_foot<P>(D.f[j], o.X1, o.X2, C);
            weight_moments<P, 1>(M.m3, C, W3);
            weight_moments<P, 3>(M.m5, C, W5);
            const double fl[3] = {j == 0 ? 1.0 : 0.0, j == 1 ? 1.0 : 0.0, j == 2 ? 1.0 : 0.0};
            kelvin_six(W3, W5, o.z, g.eps2, m, fl, v);
        }
    }
    rotate_six(g, v, G);
#pragma unroll
    for (int t = 0; t < 6; t++) acc[t] += G[t];
}

// ---------------------------------------------------------------------------
// traction rows: put(k, T), T[i][j] = n_f . sigma(e_j density of node k)_i
// ---------------------------------------------------------------------------
enum { TR_SLIP = 0, TR_FORCE = 1, TR_EIGEN = 2, TR_TOTAL = 3 };

template <int F>
__device__ __forceinline__ void traction_block(const NodalRec& g, double z, const SMat& m, bool eig,
                                               const double nf[3], const double* W3, const double* W5,
                                               const double* W7, double T[3][3]) {
    // nf in the frame; columns: density along the frame's axes
    double L[3][3];
    const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#define MBEM_ND_COL(j)                                                                                           \
    {                                                                                                            \
        double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};                                                            \
        const double sl[3] = {j == 0 ? 1.0 : 0.0, j == 1 ? 1.0 : 0.0, j == 2 ? 1.0 : 0.0};                       \
        if (F == NF_S) {                                                                                         \
            kelvin_six(W3, W5, z, g.eps2, m, sl, v);                                                             \
        } else if (F == NF_E) {                                                                                  \
            const double ph = m.phi * g.eps2 * g.eps2 * W7[0];                                                   \
            const double lu = m.lam * g.nl[j];                                                                   \
            v[0] = ph * (lu + 2.0 * m.mu * sl[0] * g.nl[0]);                                                     \
            v[1] = ph * (lu + 2.0 * m.mu * sl[1] * g.nl[1]);                                                     \
            v[2] = ph * (lu + 2.0 * m.mu * sl[2] * g.nl[2]);                                                     \
            v[3] = ph * m.mu * (sl[0] * g.nl[1] + g.nl[0] * sl[1]);                                              \
            v[4] = ph * m.mu * (sl[0] * g.nl[2] + g.nl[0] * sl[2]);                                              \
            v[5] = ph * m.mu * (sl[1] * g.nl[2] + g.nl[1] * sl[2]);                                              \
        } else if (F == NF_H) {                                                                                  \
            dd_unit<j>(W3, W5, W7, z, g.eps2, m, eig, g.s, v);                                                   \
        } else {                                                                                                 \
            dd_general(W3, W5, W7, z, g.eps2, m, g.nl, sl, eig, v);                                              \
        }                                                                                                        \
        _Pragma("unroll") for (int i = 0; i < 3; i++) L[i][j] =                                                  \
            v[ix[i][0]] * nf[0] + v[ix[i][1]] * nf[1] + v[ix[i][2]] * nf[2];                                     \
    }
    MBEM_ND_COL(0)
    MBEM_ND_COL(1)
    MBEM_ND_COL(2)
#undef MBEM_ND_COL
    rotate_full(g, L, T);
}

// F as in NodalFam: NF_H for a source normal along the frame's, NF_HG for any
template <int P, int F, class Put>
__device__ __forceinline__ void pair_traction_fam(const NodalRec& g, const double* x, const double* nfg, const SMat& m,
                                                  bool eig, Put&& put) {
    constexpr int K = nd_nodes(P);
    const NodalObs o = nodal_obs(g, x);
    double nf[3];
    to_frame(g, nfg, nf);
    constexpr int D3 = F == NF_S ? 1 : 0, D5 = F == NF_S ? 3 : 2, D7 = F == NF_E ? 0 : F == NF_H ? 3 : 4;
    if (nodal_is_far(g, o)) {
        double W3[K][3], W5[K][10], W7[K][15];
#pragma unroll
        for (int k = 0; k < K; k++) {
#pragma unroll
            for (int t = 0; t < 3; t++) W3[k][t] = 0.0;
#pragma unroll
            for (int t = 0; t < 10; t++) W5[k][t] = 0.0;
#pragma unroll
            for (int t = 0; t < 15; t++) W7[k][t] = 0.0;
        }
        far_points(g, o, nd_far_rule<P, F>(o.D2, g.L2), [&](double xi1, double xi2, double R2, int q0) {
            const double iR = rsqrt(R2), iR2 = iR * iR;
            const double a = iR * iR2, b = a * iR2, c = b * iR2;
            double p[15];
            p[0] = 1.0; p[1] = xi1; p[2] = xi2;
#pragma unroll
            for (int q = 2; q <= 4; q++) {
                p[nd_tri(q, 0)] = p[nd_tri(q - 1, 0)] * xi1;
#pragma unroll
                for (int t = 1; t <= q; t++) p[nd_tri(q - t, t)] = p[nd_tri(q - t, t - 1)] * xi2;
            }
#pragma unroll
            for (int k = 0; k < K; k++) {
                const double w = g.area2 * far_wn<P>(q0, k);
                const double na = w * a, nb = w * b, nc = w * c;
                if (F != NF_E) {
                    W3[k][0] += na;
#pragma unroll
                    for (int t = 1; t < nd_len(D3); t++) W3[k][t] += na * p[t];
                    W5[k][0] += nb;
#pragma unroll
                    for (int t = 1; t < nd_len(D5); t++) W5[k][t] += nb * p[t];
                }
                if (F != NF_S) {
                    W7[k][0] += nc;
#pragma unroll
                    for (int t = 1; t < nd_len(D7); t++) W7[k][t] += nc * p[t];
                }
            }
        });
#pragma unroll 1
        for (int k = 0; k < K; k++) {
            double T[3][3];
            traction_block<F>(g, o.z, m, eig, nf, W3[k], W5[k], W7[k], T);
            put(k, T);
        }
        return;
    }
    NMom<P, F> M;
    nodal_moments<P, F>(g, o, M);
    double l[3];
    lam_at_foot(g, o, l);
#pragma unroll 1
    for (int k = 0; k < K; k++) {
        double C[K], W3[3], W5[10], W7[15], T[3][3];
        shape_about_foot<P>(g, l, k, C);
        if constexpr (F != NF_E) {
            weight_moments<P, D3>(M.m3, C, W3);
            weight_moments<P, D5>(M.m5, C, W5);
        }
        if constexpr (F != NF_S) weight_moments<P, D7>(M.m7, C, W7);
        traction_block<F>(g, o.z, m, eig, nf, W3, W5, W7, T);
        put(k, T);
    }
}
template <int P, class Put>
static __device__ __noinline__ void pair_traction_general(const NodalRec& g, const double* x, const double* nfg,
                                                          const SMat& m, bool eig, Put&& put) {
    pair_traction_fam<P, NF_HG>(g, x, nfg, m, eig, put);
}
template <int P, int F, class Put>
__device__ __forceinline__ void pair_traction(const NodalRec& g, const double* x, const double* nfg, const SMat& m,
                                              bool eig, Put&& put) {
    if (F == NF_H && !g.aligned) pair_traction_general<P>(g, x, nfg, m, eig, put);
    else pair_traction_fam<P, F>(g, x, nfg, m, eig, put);
}

}  // namespace mbem
