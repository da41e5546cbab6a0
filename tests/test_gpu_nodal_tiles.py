"""The nodal kernels' splits and branches: ragged tiles, the cluster split of a
contraction, and the two normal branches (along the frame's, any other).

Reference: the same driver on one source at a time (its values are held to the
golden vectors in test_gpu_nodal.py), and the kernels' linearity in the normal.
A pair's arithmetic does not depend on its tile, so matrices agree to the bit;
a contraction adds the same pair values in another order, 1e-13 of the sum of
magnitudes (600 terms x 2^-53). The normal branches round differently, by the
shape polynomials' cancellation (D / L)^2 <= 100 of some 30 roundings: 1e-12.
"""

import numpy as np
import pytest
import torch

from mbem_gb300 import mesh as M

pytestmark = pytest.mark.gpu


def _case(ns, nf, order, seed=0):
    rng = np.random.default_rng(seed)
    n = int(np.ceil(np.sqrt(ns / 2)))
    m = M.centre_fault(n)
    tv = m.tri_verts()[:ns]
    nrm = m.normals_and_areas()[0][:ns]
    # observers from on the fault (every edge regime) to beyond 60 longest edges
    x = rng.uniform(-1, 1, size=(nf, 3)) * 10.0 ** rng.uniform(-2, 1.2, size=(nf, 1))
    K = (order + 1) * (order + 2) // 2
    return x, tv, nrm, np.full(ns, 0.5 / n), rng.normal(size=(K * ns, 3))


@pytest.fixture(scope="module")
def drivers(gpu):
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_nodal as tn
    return tn, kb


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("nf,ns", [(1, 1), (1, 70), (63, 3), (64, 17), (65, 16), (300, 33)])
def test_matrix_tiles(drivers, order, nf, ns):
    tn, kb = drivers
    x, tv, n, e, _ = _case(ns, nf, order)
    c, u = kb.t_coeffs(1.0, 1.0), kb.u_coeffs(1.0, 1.0)
    T = tn.t_matrix_direct(x, tv, n, e, *c, order=order)
    U = tn.u_matrix_direct(x, tv, e, *u, order=order)
    K = (order + 1) * (order + 2) // 2
    for s in {0, ns // 2, ns - 1}:
        sl = slice(3 * K * s, 3 * K * (s + 1))
        assert np.array_equal(T[:, sl], tn.t_matrix_direct(x, tv[s:s + 1], n[s:s + 1], e[s:s + 1], *c, order=order))
        assert np.array_equal(U[:, sl], tn.u_matrix_direct(x, tv[s:s + 1], e[s:s + 1], *u, order=order))


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("nf,ns", [(1, 1), (3, 15), (5, 17), (64, 129), (65, 600), (400, 40)])
def test_contraction_splits(drivers, order, nf, ns):
    tn, kb = drivers
    x, tv, n, e, d = _case(ns, nf, order, 1)
    K = (order + 1) * (order + 2) // 2
    d[:K] = 0.0                                       # a source without slip is left out
    kinds = [lambda *a, **k: tn.t_disp_contract(*a[:5], *kb.t_coeffs(1.0, 1.0), **k),
             lambda *a, **k: tn.u_disp_contract(a[0], a[1], a[3], a[4], *kb.u_coeffs(1.0, 1.0), **k),
             lambda *a, **k: tn.dd_stress_contract(*a[:5], 1.0, 1.0, **k),
             lambda *a, **k: tn.kelvin_stress_contract(a[0], a[1], a[3], a[4], 1.0, 1.0, **k),
             lambda *a, **k: tn.eigenstress_contract(*a[:5], 1.0, 1.0, **k),
             lambda *a, **k: tn.elastic_stress_contract(*a[:5], 1.0, 1.0, **k)]
    for f in kinds:
        got = f(x, tv, n, e, d, order=order)
        parts = [f(x, tv[s:s + 1], n[s:s + 1], e[s:s + 1], d[K * s:K * (s + 1)], order=order) for s in range(ns)]
        want, mag = sum(parts), sum(np.abs(p) for p in parts)
        assert np.all(np.abs(got - want) <= 1e-13 * mag + 1e-300)
        out = torch.from_numpy(np.ones_like(want)).cuda()
        f(*(torch.from_numpy(v).cuda() for v in (x, tv, n, e, d)), order=order, out=out, alpha=-2.0, accumulate=True)
        assert np.all(np.abs(out.cpu().numpy() - (1.0 - 2.0 * got)) <= 1e-13 * (1.0 + 2.0 * mag))


@pytest.mark.parametrize("order", [0, 1, 2])
def test_normal_branches(drivers, order):
    """A reversed normal, and normals off the frame's whose mean is it."""
    tn, kb = drivers
    x, tv, n, e, d = _case(24, 200, order, 2)
    nf = np.random.default_rng(3).normal(size=x.shape)
    ids = kb.identity_ids(order, len(tv))
    off = 0.3 * (tv[:, 1] - tv[:, 0]) / np.linalg.norm(tv[:, 1] - tv[:, 0], axis=1)[:, None]
    kinds = [lambda m: tn.elastic_stress_contract(x, tv, m, e, d, 1.0, 1.3, order=order),
             lambda m: tn.traction_matrix(x, nf, tv, m, e, ids, ids.size, 1.0, 1.3, order, "slip")]
    if order:
        kinds += [lambda m: tn.t_matrix_direct(x, tv, m, e, *kb.t_coeffs(1.0, 1.3), order=order),
                  lambda m: tn.t_disp_contract(x, tv, m, e, d, *kb.t_coeffs(1.0, 1.3), order=order)]
    for f in kinds:
        a, b, c = f(n), f(-n), 0.5 * (f(n + off) + f(n - off))
        scale = np.abs(a).max()
        assert np.abs(a + b).max() <= 1e-12 * scale
        assert np.abs(a - c).max() <= 1e-12 * scale


# the device's screen refuses what the host's test refuses, at both sides of the limit
# and for triangles without a length
@pytest.mark.parametrize("height, ok", [(0.5, True), (1.0000001, True), (1.0, True), (0.9999999, False), (0.0, False)])
@pytest.mark.parametrize("n", [1, 129])
def test_needles_refused_on_device(gpu, height, ok, n):
    from mbem_gb300 import defaults
    from mbem_gb300.kernels import tri_nodal as tn
    h = height if height == 0.5 else height * defaults.NODAL_MIN_HEIGHT_OVER_L
    tv = np.tile(np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.0, 0.8, 0.0]]), (n, 1, 1))
    tv[-1] = [[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.5, h, 0.0]]
    for v in (tv, torch.from_numpy(tv).cuda()):
        try:
            tn._check_shape(v)
            accepted = True
        except ValueError:
            accepted = False
        # at the limit itself the host's rounding decides for both
        assert accepted == ok or height == 1.0
    a = [True, True]
    for i, v in enumerate((tv, torch.from_numpy(tv).cuda())):
        try:
            tn._check_shape(v)
        except ValueError:
            a[i] = False
    assert a[0] == a[1]


# The P1 T block does not depend on the unit of length: by powers of two the same numbers
# to a few ulps of the largest (1e-11 as for the P0 blocks), also where the distances'
# fifth powers leave the range of the short ones (lengths above 2^192).
@pytest.mark.parametrize("k", [-40, 60, 195])
def test_nodal_block_in_any_unit(gpu, k):
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_nodal as tn
    m = M.centre_fault(4)
    x = np.random.default_rng(3).uniform(-1, 1, size=(50, 3))
    tv, n, e = m.tri_verts(), m.normals_and_areas()[0], np.full(m.tri_verts().shape[0], 0.05)
    c, s = kb.t_coeffs(1.0, 1.3), 2.0 ** k
    ref = tn.t_matrix_direct(x, tv, n, e, *c, order=1)
    got = tn.t_matrix_direct(x * s, tv * s, n, e * s, *c, order=1)
    assert np.abs(got - ref).max() < 1e-11 * np.abs(ref).max()
