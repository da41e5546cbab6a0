"""The exact digit products of the block residual (tc_exact.cu) against 80-bit
sums on the host.

Bound: the five digit products of order 6 that are left out are at most 2^14 in
units of 2^-62, and the last digit of either factor is rounded at half of 2^-47
of its scale, so a term is off by at most (5 + 2) 2^-48 of max|A_i| max|X_r|
(powers of two at most twice the largest entries: times 4); the FP64 result and
the subtraction from B round at 2^-53 of |B| + |y|.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _residual(A, B, X, ld=None):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    from mbem_gb300.la.mixed import MixedOperator
    n = A.shape[0]
    ld = (n + 3) // 4 * 4 if ld is None else ld
    A32 = torch.zeros((n, ld), dtype=torch.float32, device="cuda")[:, :n]
    A32.copy_(torch.from_numpy(A))
    op = MixedOperator(A32, [])
    b, x = torch.from_numpy(B).cuda(), torch.from_numpy(X).cuda()
    R = torch.empty_like(b)
    k = B.shape[0]
    need = nat.lib().mbem_batch_residual_workspace_size(k, n)
    work = torch.full((need // 8,), float("nan"), dtype=torch.float64, device="cuda")
    s = op.struct()
    nat.call("mbem_batch_residual_mixed", ctypes.byref(s), ptr(b), ptr(x), k, ptr(R), ptr(work), need,
             stream_handle())
    nat.call("mbem_gemm_bf16_check", stream_handle())
    return R.cpu().numpy()


def _check(A, B, X, **kw):
    got = _residual(A, B, X, **kw)
    y = X.astype(np.longdouble) @ A.T.astype(np.longdouble)
    term = np.abs(X).max(axis=1)[:, None] * np.abs(A).max(axis=1)[None, :]
    tol = 4 * 7 * 2.0 ** -48 * A.shape[0] * term + 2.0 ** -52 * (np.abs(B) + np.abs(y).astype(float))
    err = np.abs((B.astype(np.longdouble) - y - got).astype(float))
    assert np.all(err <= tol), float((err / np.maximum(tol, 1e-300)).max())


@pytest.mark.parametrize("n,k", [(1, 1), (63, 3), (128, 32), (129, 33), (333, 64), (700, 129), (515, 257)])
def test_against_extended_precision(gpu, n, k):
    rng = np.random.default_rng(n)
    # entries over six decades in a row, rows and right-hand sides over many more
    A = (rng.normal(size=(n, n)) * 10.0 ** rng.uniform(-6, 0, size=(n, n)) *
         10.0 ** rng.uniform(-12, 12, size=(n, 1))).astype(np.float32)
    X = rng.normal(size=(k, n)) * 10.0 ** rng.uniform(-100, 100, size=(k, 1))
    B = (X @ A.T.astype(float)) * (1.0 + 1e-9 * rng.normal(size=(k, n)))
    A[0] = 0.0
    X[-1] = 0.0
    _check(A, B, X)


@pytest.mark.parametrize("a,x", [(1.0, 1.0), (-1.0, 1.0), (0.99999994, 1.0 - 2.0 ** -53), (0.50000006, -0.4999999999)])
def test_largest_digit_sums(gpu, a, x):
    """Every product of a digit pair at its largest, of one sign."""
    A = np.full((300, 300), a, dtype=np.float32)
    _check(A, np.zeros((40, 300)), np.full((40, 300), x))


def test_unaligned_rows(gpu):
    rng = np.random.default_rng(5)
    A = rng.normal(size=(201, 201)).astype(np.float32)
    X = rng.normal(size=(5, 201))
    _check(A, rng.normal(size=(5, 201)), X, ld=203)


def test_nonfinite_rows_give_nan(gpu):
    rng = np.random.default_rng(6)
    A = rng.normal(size=(150, 150)).astype(np.float32)
    X = rng.normal(size=(4, 150))
    A[7, 3], A[9, 0] = np.inf, np.nan
    X[2, 149] = np.nan
    R = _residual(A, np.zeros((4, 150)), X)
    bad = np.zeros((4, 150), bool)
    bad[:, [7, 9]] = True
    bad[2] = True
    assert np.array_equal(np.isnan(R), bad)
