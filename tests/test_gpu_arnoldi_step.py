"""The FP64 product and the Arnoldi step of the single right-hand side solve at the
edges of their launches, against a modified Gram-Schmidt GMRES of plain FP64."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, cols", [(1, 1), (3, 65), (2431, 64), (2432, 131), (2435, 130), (5184, 33)])
def test_product_rows(gpu, rows, cols):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cuda").manual_seed(rows)
    A = torch.randn((rows, cols + cols % 2), generator=g, dtype=torch.float64, device="cuda")
    x = torch.randn(cols, generator=g, dtype=torch.float64, device="cuda")
    y = torch.randn(rows, generator=g, dtype=torch.float64, device="cuda")
    ref = -0.5 * (A[:, :cols] * x).sum(1) + 2.0 * y
    bound = 0.5 * (A[:, :cols] * x).abs().sum(1) + 2.0 * y.abs()
    nat.call("mbem_dgemv", ptr(A), A.stride(0), rows, cols, ptr(x), -0.5, 2.0, ptr(y), stream_handle())
    assert bool(((y - ref).abs() <= (cols + 3) * 2.0 ** -52 * bound).all())


def _gmres(A, b, P, rtol, restart):
    n = b.numel()
    x = torch.zeros_like(b)
    b = P(b)
    bn, hist, res = b.norm().item(), [], 1.0
    while res >= rtol and len(hist) < 200:
        r = b - P(A @ P(x))
        beta = r.norm().item()
        V, H = [r / beta], np.zeros((restart + 1, restart))
        for j in range(restart):
            w = P(A @ P(V[j]))
            for _ in range(2):
                for i in range(j + 1):
                    c = torch.dot(V[i], w).item()
                    H[i, j] += c
                    w = w - c * V[i]
            H[j + 1, j] = w.norm().item()
            e1 = np.zeros(j + 2)
            e1[0] = beta
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e1, rcond=None)[0]
            res = np.linalg.norm(e1 - H[:j + 2, :j + 1] @ y) / bn
            hist.append(res)
            if res < rtol or H[j + 1, j] == 0.0:
                break
            V.append(w / H[j + 1, j])
        for i, c in enumerate(y):
            x = x + c * V[i]
    return P(x), hist


# 16 blocks' slices with and without remainder, blocks without a slice, more vectors
# than a block has warps, and both sides of the largest vector of one launch
@pytest.mark.parametrize("n, restart", [(2, 5), (17, 30), (301, 20), (5184, 40), (32768, 6), (32769, 6)])
@pytest.mark.parametrize("ranges", [False, True])
def test_gmres_steps(gpu, n, restart, ranges):
    from mbem_gb300.la.solver import fgmres_dense
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), generator=g, dtype=torch.float64, device="cuda")
    A.mul_(1.0 / n ** 0.5)
    A.diagonal().add_(3.0)
    b = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    ur = []
    if ranges and n >= 17:
        ur = [(0, 3 * (n // 9)), (3 * (n // 6) + 1, 3 * (n // 12))]

    def P(v):
        if not ur:
            return v
        out = v.clone()
        M = sum(l for _, l in ur) // 3
        for k in range(3):
            mean = sum(v[o + k:o + l:3].sum() for o, l in ur) / M
            for o, l in ur:
                out[o + k:o + l:3] -= mean
        return out

    x, rep = fgmres_dense(A, b, rtol=1e-9, restart=restart, u_ranges=ur)
    xr, hist = _gmres(A, b, P, 1e-9, restart)
    # the operator's condition is below 4: residual estimates and solution agree
    # to rounding times the number of steps
    assert rep.converged and rep.iterations == len(hist)
    assert np.abs(np.asarray(rep.residual_history) - hist).max() < 1e-12
    assert float((x - xr).abs().max()) < 1e-12 * float(xr.abs().max()) * 10
