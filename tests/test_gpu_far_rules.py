"""The nodal kernels' far quadratures against 196 points in extended precision, just beyond
the distances where a coarser rule takes over.

A rule's truncation is below 1e-16 of the pair's largest entry where it is used, so what is left is rounding:
some 40 roundings of 2^-53 to an entry, R's once for each of up to seven powers: 5e-15 of the
pair's largest entry. The eigenstress, which falls off fastest, is held to its own largest entry.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
I3 = np.eye(3)
SIX = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))


def _rule(n=14):
    x, w = np.polynomial.legendre.leggauss(n)
    x = x.astype(LD)
    for _ in range(2):                                    # Newton's step to extended precision
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
        d = n * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / d
    w = 2 / ((1 - x * x) * d * d)
    g, w = (x + 1) / 2, w / 2
    a, b = np.repeat(g, n), np.tile(g, n)
    return np.stack([1 - a - b * (1 - a), a, b * (1 - a)], 1), np.repeat(w, n) * np.tile(w, n) * (1 - a)


def _shapes(lam, order):
    if order == 0:
        return np.ones_like(lam[:, :1])
    return lam if order == 1 else np.concatenate([lam * (2 * lam - 1), 4 * lam * np.roll(lam, -1, 1)], 1)


def _integrand(kind, d, n, e2):
    """(q, 3, 3) blocks of U and T, (q, 3, 6) stresses by slip direction; mu = lam = 1, nu = 1/4."""
    c1, dd = 1 / (12 * LD(np.pi)), (d * d).sum(-1)
    ir = 1 / np.sqrt(dd + e2)
    a, b, c = ir ** 3, ir ** 5, ir ** 7
    outer = d[:, :, None] * d[:, None, :]
    if kind == "U":
        return (2 * c1 * ir + e2 * a / (8 * LD(np.pi)))[:, None, None] * I3 + (c1 * a)[:, None, None] * outer
    dn = d @ n
    if kind == "T":
        al = d * (-2 * a + 3 * dd * b + LD(4.5) * e2 * b)[:, None]
        nd = n[None, :, None] * d[:, None, :]
        dI = dn[:, None, None] * I3
        out = al[:, :, None] * n + (2 * a + LD(4.5) * e2 * b)[:, None, None] * (nd + dI)
        out = out - a[:, None, None] * (nd + 2 * d[:, :, None] * n + dI)
        return c1 * (out + (6 * b * dn)[:, None, None] * outer)
    phi = 15 / (8 * LD(np.pi)) * e2 * e2 * c
    out = np.zeros((d.shape[0], 3, 6), LD)
    for j in range(3):
        u, du, un = I3[j], d[:, j], n[j]
        blob = LD(1.5) * e2
        x0, x1 = 2 * a - 3 * (dd + blob) * b, -12 * b + 15 * (dd + blob) * c
        a1, s0 = -a - 3 * blob * b, 2 * un * a - 6 * du * dn * b
        g, ee = -3 * b + 15 * blob * c, 30 * du * dn * c - 6 * un * b
        w = dn[:, None] * u + du[:, None] * n
        tr = c1 * (un * (3 * x0 + x1 * dd) + 2 * a1 * un + 3 * s0 + 2 * g * du * dn + ee * dd)
        for t, (i, k) in enumerate(SIX):
            sym = u[i] * n[k] + n[i] * u[k]
            eig = phi * (un * (i == k) + sym)
            if kind == "eigen":
                out[:, j, t] = eig
                continue
            dik = d[:, i] * d[:, k]
            bb = 2 * un * x1 * dik + 2 * a1 * sym + g * (w[:, i] * d[:, k] + d[:, i] * w[:, k]) + 2 * ee * dik
            if i == k:
                bb = bb + 2 * un * x0 + 2 * s0
            out[:, j, t] = -(i == k) * tr - c1 * bb - eig
    return out


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("dist", [10.01, 11.01, 12.51, 16.02, 18.02, 24.02, 30.02, 42.05, 55.1, 90.1, 120.2, 250.5])
def test_far_pairs(gpu, order, dist):
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_nodal as tn
    rng = np.random.default_rng(int(100 * dist) + order)
    lam, w = _rule()
    N = w[:, None] * _shapes(lam, order)
    K = N.shape[1]
    worst = {}
    for s in range(4):
        tv = np.array([[0, 0, 0], [1, 0, 0], [rng.uniform(0, 1), rng.uniform(0.2, 0.7), 0]])
        tv = (tv - tv.mean(0)) @ np.linalg.qr(rng.normal(size=(3, 3)))[0]
        L = np.linalg.norm(tv - np.roll(tv, 1, 0), axis=1).max()
        cr = np.cross(tv[1] - tv[0], tv[2] - tv[0])
        n = cr / np.linalg.norm(cr)
        eps = (0.05, 0.5, 3.0, 0.9 * dist)[s] * L
        x = rng.normal(size=(16, 3))
        x[:3] = tv - np.roll(tv, 1, 0)                   # along the edges
        x *= np.sqrt((dist * L) ** 2 - eps ** 2) / np.linalg.norm(x, axis=1, keepdims=True)
        got = {}
        if order:
            got["T"] = tn.t_matrix_direct(x, tv[None], n[None], np.array([eps]), *kb.t_coeffs(1.0, 1.0), order=order)
            got["U"] = tn.u_matrix_direct(x, tv[None], np.array([eps]), *kb.u_coeffs(1.0, 1.0), order=order)
        ids = np.arange(K).reshape(1, K)
        for which in ("slip", "eigen"):
            t = tn.traction_matrix(np.repeat(x, 3, 0), np.tile(I3, (len(x), 1)), tv[None], n[None], np.array([eps]), ids, K,
                                   1.0, 1.0, order, which)
            got[which] = t.reshape(len(x), 3, 3, K, 3)   # observer, field normal, component, node, slip
        y, A2 = lam @ tv.astype(LD), np.sqrt((np.cross(*(tv[1:] - tv[0]).astype(LD)) ** 2).sum())
        for f in range(len(x)):
            for kind in got:
                v = A2 * np.einsum("qk,qij->kij", N, _integrand(kind, x[f].astype(LD) - y, n.astype(LD), LD(eps) ** 2))
                if kind in "TU":
                    g = got[kind].reshape(len(x), 3, K, 3)[f].transpose(1, 0, 2)
                else:
                    v = v[:, :, [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(K, 3, 3, 3)      # node, slip, stress
                    g = got[kind][f].transpose(2, 3, 0, 1)
                worst[kind] = max(worst.get(kind, 0.0), float(np.abs(g - v).max() / np.abs(v).max()))
    assert all(e < 5e-15 for e in worst.values()), worst


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("height", [0.01, 0.05, 0.5])
@pytest.mark.parametrize("dist", [10.5, 14.0, 30.0, 200.0])
def test_far_contractions(gpu, order, height, dist):
    """A contraction of one far source against its matrix blocks times the density, slender
    sources among them: both round some 40 times, 5e-15 of the sum of magnitudes each."""
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_nodal as tn
    rng = np.random.default_rng(int(1000 * height + dist) + order)
    K = (order + 1) * (order + 2) // 2
    tv = np.array([[0, 0, 0], [1, 0, 0], [0.3, height, 0]])
    tv = ((tv - tv.mean(0)) @ np.linalg.qr(rng.normal(size=(3, 3)))[0])[None]
    cr = np.cross(tv[0, 1] - tv[0, 0], tv[0, 2] - tv[0, 0])
    n, eps = (cr / np.linalg.norm(cr))[None], np.array([0.2])
    x = rng.normal(size=(40, 3))
    x[:3] = tv[0] - np.roll(tv[0], 1, 0)
    x *= dist / np.linalg.norm(x, axis=1, keepdims=True)
    d = rng.normal(size=(K, 3))
    t, u = kb.t_coeffs(1.0, 1.0), kb.u_coeffs(1.0, 1.0)
    ids = np.arange(K).reshape(1, K)
    rows = [(tn.t_disp_contract(x, tv, n, eps, d, *t, order), tn.t_matrix_direct(x, tv, n, eps, *t, order=order)),
            (tn.u_disp_contract(x, tv, eps, d, *u, order), tn.u_matrix_direct(x, tv, eps, *u, order=order))]
    for which, got in (("slip", tn.elastic_stress_contract(x, tv, n, eps, d, 1.0, 1.0, order)),
                       ("eigen", tn.eigenstress_contract(x, tv, n, eps, d, 1.0, 1.0, order)),
                       ("force", tn.kelvin_stress_contract(x, tv, eps, d, 1.0, 1.0, order))):
        rows.append((got, tn.traction_matrix(np.repeat(x, 3, 0), np.tile(I3, (len(x), 1)), tv, n, eps, ids, K, 1.0, 1.0,
                                             order, which)))
    for got, M in rows:
        err = np.abs(got.reshape(-1) - M @ d.reshape(-1))
        size = (np.abs(M) @ np.abs(d.reshape(-1))).reshape(len(x), -1).max(1)       # of the observer
        assert np.all(err.reshape(len(x), -1) <= 1e-14 * size[:, None]), float((err.reshape(len(x), -1) / size[:, None]).max())
