"""The P0 kernels' splits and branches: observer tiles of the matrices, the
cluster split of the contractions, and a source normal along the frame's or not.

Reference: the C oracle. Tolerance: some 30 roundings of 2^-53 a moment times the
moments' cancellation (D / L)^2 <= 300 here, 1e-12 of the largest value, and ten
times that for sums whose terms (random densities) cancel.
"""

import numpy as np
import pytest

from mbem_gb300 import mesh as M

pytestmark = pytest.mark.gpu
TOL = 1e-11


def _case(ns, nf, seed=0):
    rng = np.random.default_rng(seed)
    n = int(np.ceil(np.sqrt(ns / 2)))
    m = M.centre_fault(n)
    x = rng.uniform(-1, 1, size=(nf, 3))
    return x, m.tri_verts()[:ns], m.normals_and_areas()[0][:ns], np.full(ns, 0.5 / n), rng.normal(size=(ns, 3))


def _err(a, b):
    return np.abs(np.asarray(a) - b).max() / np.abs(b).max()


@pytest.mark.parametrize("branch", ["frame", "reversed", "other"])
@pytest.mark.parametrize("nf,ns", [(1, 1), (1, 600), (2, 33), (63, 64), (65, 31), (500, 129)])
def test_against_the_oracle(gpu, oracle, nf, ns, branch):
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_kernels as tk
    x, tv, n, e, d = _case(ns, nf)
    if ns > 2:
        d[1] = 0.0                                  # a source without density is left out
    if branch == "reversed":
        n = -n
    elif branch == "other":
        n = n + 0.3 * np.random.default_rng(1).normal(size=n.shape)
    mu, lam = 1.0, 1.3
    c, u = kb.t_coeffs(mu, lam), kb.u_coeffs(mu, lam)
    assert _err(tk.t_matrix_direct(x, tv, n, e, *c), oracle.matrix("t", x, tv, n, e, c)) < TOL
    assert _err(tk.u_matrix_direct(x, tv, e, *u), oracle.matrix("u", x, tv, n, e, u)) < TOL
    assert _err(tk.t_disp_contract(x, tv, n, e, d, *c), oracle.contract("t_disp", x, tv, n, e, d, c)) < TOL
    assert _err(tk.u_disp_contract(x, tv, e, d, *u), oracle.contract("u_disp", x, tv, n, e, d, u)) < TOL
    for name, got in (("dd", tk.dd_stress_contract(x, tv, n, e, d, mu, lam)),
                      ("kelvin", tk.kelvin_stress_contract(x, tv, e, d, mu, lam)),
                      ("eigen", tk.eigenstress_contract(x, tv, n, e, d, mu, lam))):
        assert _err(got, oracle.contract(name, x, tv, n, e, d, mu=mu, lam=lam)) < TOL


# one observer a block and whole blocks of them, tiles of 128 sources with remainders
# over one to eight blocks a cluster
@pytest.mark.parametrize("nf,ns", [(1, 128), (3, 129), (19, 1025), (76, 513), (77, 513)])
def test_few_observers(gpu, oracle, nf, ns):
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_kernels as tk
    x, tv, n, e, d = _case(ns, nf, seed=nf)
    c = kb.t_coeffs(1.0, 1.3)
    assert _err(tk.t_disp_contract(x, tv, n, e, d, *c), oracle.contract("t_disp", x, tv, n, e, d, c)) < TOL
    assert _err(tk.dd_stress_contract(x, tv, n, e, d, 1.0, 1.3),
                oracle.contract("dd", x, tv, n, e, d, mu=1.0, lam=1.3)) < TOL


# The T block does not depend on the unit of length: by powers of two it is the same
# numbers to a few ulps (the file's bound) wherever the element's frame exists. Areas
# below 1e-30 count as degenerate, and areas whose squares overflow have no frame:
# zero blocks for both.
@pytest.mark.parametrize("k", [-60, 0, 60, 330])
def test_block_in_any_unit(gpu, k):
    from mbem_gb300.kernels import basis as kb
    from mbem_gb300.kernels import tri_kernels as tk
    x, tv, n, e, _ = _case(40, 60)
    c, s = kb.t_coeffs(1.0, 1.3), 2.0 ** k
    got = tk.t_matrix_direct(x * s, tv * s, n, e * s, *c)
    if k in (-60, 330):
        assert not got.any()
    else:
        assert _err(got, tk.t_matrix_direct(x, tv, n, e, *c)) < TOL
