"""The block residual's digits where columns, unknowns or entries differ by many decades.

Columns against each other: with A_ij = G_ij s_j and X_rj = Y_rj / s_j every term is that of
(G, Y), so the bound is the balanced one of test_gpu_exact_residual.py, doubled for the
column scales, which are powers of two: 56 2^-48 n max_j(|G_ij| / C_j) max_j(C_j |Y_rj|),
C_j = max_i |G_ij|. Entries of a right-hand side against each other: an error of at most
n 2^-48 of |A| |X|, what FP32 pairs keep (the low part of each product rounds at 2^-48 of
it, and the low sum at 2^-24 of 2^-24 of the sum a step). Both with the FP64 rounding
of |B| + |y|.
"""

import numpy as np
import pytest
from test_gpu_exact_residual import _residual

pytestmark = pytest.mark.gpu


def _error(A, X):
    B = X @ A.T.astype(float)
    got = _residual(A, B, X)
    y = X.astype(np.longdouble) @ A.T.astype(np.longdouble)
    err = np.abs((B.astype(np.longdouble) - y - got).astype(float))
    return np.maximum(err - 2.0 ** -52 * (np.abs(B) + np.abs(y).astype(float)), 0.0)


@pytest.mark.parametrize("n,k", [(63, 3), (700, 129)])
@pytest.mark.parametrize("scales", ["decades", 1e-4, 1e-6, 1 / 3e10])
def test_columns_over_decades(gpu, n, k, scales):
    rng = np.random.default_rng(n)
    G, Y = rng.normal(size=(n, n)).astype(np.float32), rng.normal(size=(k, n))
    s = 10.0 ** rng.uniform(-10, 0, size=n) if scales == "decades" else np.where(rng.random(n) < 0.5, scales, 1.0)
    s = 2.0 ** np.round(np.log2(s))                  # exact in FP32 and FP64
    C = np.abs(G).max(axis=0)
    term = (C * np.abs(Y)).max(axis=1)[:, None] * (np.abs(G) / C).max(axis=1)[None, :]
    err = _error((G * s).astype(np.float32), Y / s)
    assert np.all(err <= 56 * 2.0 ** -48 * n * term), float((err / term).max())


def test_unknowns_missing_from_some_right_hand_sides(gpu):
    """Displacement and traction columns (1 and 1 / mu); right-hand sides with both unknowns,
    with one of them alone, and with a traction far below mu."""
    rng = np.random.default_rng(11)
    n, mu = 500, 2.0 ** 35
    G, Y = rng.normal(size=(n, n)).astype(np.float32), rng.normal(size=(12, n))
    t = rng.random(n) < 0.5
    A = np.where(t[None], G / np.float32(mu), G).astype(np.float32)
    X = np.where(t[None], Y * mu, Y)
    X[:3, t], X[3:6, ~t] = 0.0, 0.0
    X[6:9, t] *= 1e-3
    err = _error(A, X)
    size = np.abs(X) @ np.abs(A).T.astype(float)
    assert np.all(err <= n * 2.0 ** -48 * size), float((err / size).max())


@pytest.mark.parametrize("n", [300, 1500])
@pytest.mark.parametrize("spread", ["one 1e2", "one 1e4", "one 1e8", "one 1e14", "six decades", "block 1e-12"])
def test_entries_of_a_right_hand_side(gpu, n, spread):
    rng = np.random.default_rng(n)
    A = (rng.normal(size=(n, n)) * 10.0 ** rng.uniform(-3, 0, size=(n, n))).astype(np.float32)
    X = rng.normal(size=(5, n))
    kind, value = spread.split()
    if kind == "one":
        X[np.arange(5), rng.integers(0, n, 5)] *= float(value)
    elif kind == "block":                            # two bodies of one system, one hardly moved
        b = np.arange(n) < n // 2
        A[b[:, None] != b[None, :]] = 0.0
        X[:, b] *= float(value)
    else:
        X *= 10.0 ** rng.uniform(-6, 0, size=X.shape)
    err = _error(A, X)
    size = np.abs(X) @ np.abs(A).T.astype(float)
    assert np.all(err <= n * 2.0 ** -48 * size), float((err / size).max())
