"""One fused step of the batched Arnoldi iteration and its back substitution
against the same algebra in FP64 torch.

Vectors are FP32: basis, column and norm agree to 1e-5 relative (as the single
vector kernels), and the new basis vector is orthogonal to the others to
1e-5 (two Gram-Schmidt passes; n roundings of 2^-24 in chains of at most 100).
The rotations are FP64: 1e-12 of the column's norm.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,splits,terms", [(12, 1, 1, 1), (1003, 7, 3, 3), (1024, 256, 2, 3), (5001, 3, 1, 3),
                                              (60000, 2, 7, 1)])
@pytest.mark.parametrize("deflate", [False, True])
def test_steps(gpu, n, k, splits, terms, deflate):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cuda").manual_seed(n + k)
    dev = "cuda"
    m, ldp = 70, (n + 7) // 8 * 8
    steps = min(4, n - 1)
    ranges = np.array([0, n // 6 * 3, n // 6 * 3 + 1, (n // 2 - 1) // 3 * 3] if deflate else [], dtype=np.int64)
    rp = ranges.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    V = torch.zeros((m + 1, k, n), device=dev)
    v0 = torch.randn((k, n), generator=g, device=dev, dtype=torch.float64)
    V[0] = (v0 / v0.norm(dim=1, keepdim=True)).float()
    Vbf = torch.zeros((k, terms * ldp), dtype=torch.bfloat16, device=dev)
    H = torch.zeros((m, m, k), dtype=torch.float64, device=dev)
    cs, sn = (torch.zeros((m, k), dtype=torch.float64, device=dev) for _ in range(2))
    gv = torch.zeros((m + 1, k), dtype=torch.float64, device=dev)
    beta = torch.rand(k, generator=g, device=dev, dtype=torch.float64) + 1.0
    gv[0] = beta
    left = torch.zeros(m, dtype=torch.int32, device=dev)
    for j in range(steps):
        P = torch.randn((splits, k, n), generator=g, device=dev) * 10.0 ** (j - 2)
        nat.call("mbem_batch_arnoldi", ptr(P), splits, 0, 0, n * k, ptr(V), j, m, k, n, rp, len(ranges) // 2, ptr(Vbf),
                 Vbf.stride(0), ldp, terms, ptr(H), ptr(cs), ptr(sn), ptr(gv), ptr(beta), 1e-3, ptr(left[j:]),
                 stream_handle())
        w = P.double().sum(dim=0)
        if deflate:
            parts = ranges.reshape(-1, 2)
            mean = [torch.cat([w[:, a + c:a + b:3] for a, b in parts], dim=1).mean(dim=1) for c in range(3)]
            for a, b in parts:
                for c in range(3):
                    w[:, a + c:a + b:3] -= mean[c][:, None]
        scale = w.norm(dim=1)
        h = torch.zeros((j + 1, k), dtype=torch.float64, device=dev)
        for _ in range(2):
            d = torch.einsum("ikn,kn->ik", V[:j + 1].double(), w)
            w = w - torch.einsum("ik,ikn->kn", d, V[:j + 1].double())
            h += d
        nrm = w.norm(dim=1)
        v = V[j + 1].double()
        assert float(((v * nrm[:, None] - w).norm(dim=1) / scale).max()) < 1e-5
        assert float(torch.einsum("ikn,kn->ik", V[:j + 1].double(), v).abs().max()) < 1e-5
        hi = V[j + 1].to(torch.bfloat16)
        assert torch.equal(Vbf[:, :n], hi)
        if terms == 3:
            assert torch.equal(Vbf[:, ldp:ldp + n], (V[j + 1] - hi.float()).to(torch.bfloat16))
            assert torch.equal(Vbf[:, 2 * ldp:2 * ldp + n], hi)
        # the rotated column has the column's norm, and the rotations reproduce it
        col = torch.cat([h, nrm[None]])
        for i in range(j):
            a, b = col[i].clone(), col[i + 1].clone()
            col[i], col[i + 1] = cs[i] * a + sn[i] * b, -sn[i] * a + cs[i] * b
        size = torch.cat([h, nrm[None]]).norm(dim=0)
        assert float(((cs[j] * cs[j] + sn[j] * sn[j]) - 1).abs().max()) < 1e-12
        assert float(((-sn[j] * col[j] + cs[j] * col[j + 1]).abs() / size).max()) < 1e-5
        col[j] = cs[j] * col[j] + sn[j] * col[j + 1]
        assert float(((H[:j + 1, j] - col[:j + 1]).abs() / size).max()) < 1e-5
        rel = gv[j + 1].abs() / beta
        assert int(left[j]) == int((~(rel < 1e-3)).sum())
    Y = torch.empty((steps, k), dtype=torch.float64, device=dev)
    nat.call("mbem_batch_backsolve", ptr(H), ptr(gv), m, steps, k, ptr(Y), stream_handle())
    back = torch.einsum("ilk,lk->ik", torch.triu(H[:steps, :steps].permute(2, 0, 1)).permute(1, 2, 0), Y)
    assert float((back - gv[:steps]).abs().max() / beta.max()) < 1e-10


# one vector a warp, two, three, and more than the piecewise pass takes; whole and
# partial pieces of 1,024 entries. The file's bound: 1e-5.
@pytest.mark.parametrize("j", [7, 8, 23, 24])
@pytest.mark.parametrize("n", [1024, 4100, 20736])
def test_many_vectors(gpu, n, j):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cuda").manual_seed(n + j)
    k, m, ldp, dev = 3, 30, (n + 7) // 8 * 8, "cuda"
    V = torch.zeros((m + 1, k, n), device=dev)
    for r in range(k):
        q = torch.linalg.qr(torch.randn((n, j + 1), generator=g, device=dev, dtype=torch.float64))[0]
        V[:j + 1, r] = q.T.float()
    P = torch.randn((1, k, n), generator=g, device=dev)
    Vbf = torch.zeros((k, ldp), dtype=torch.bfloat16, device=dev)
    H = torch.zeros((m, m, k), dtype=torch.float64, device=dev)
    cs, sn = torch.ones((m, k), dtype=torch.float64, device=dev), torch.zeros((m, k), dtype=torch.float64, device=dev)
    gv, beta = torch.ones((m + 1, k), dtype=torch.float64, device=dev), torch.ones(k, dtype=torch.float64, device=dev)
    left = torch.zeros(1, dtype=torch.int32, device=dev)
    nat.call("mbem_batch_arnoldi", ptr(P), 1, 0, 0, n * k, ptr(V), j, m, k, n, None, 0, ptr(Vbf), Vbf.stride(0), ldp, 1,
             ptr(H), ptr(cs), ptr(sn), ptr(gv), ptr(beta), 1e-3, ptr(left), stream_handle())
    w, h = P[0].double(), 0.0
    for _ in range(2):
        d = torch.einsum("ikn,kn->ik", V[:j + 1].double(), w)
        w, h = w - torch.einsum("ik,ikn->kn", d, V[:j + 1].double()), h + d
    size = P[0].double().norm(dim=1)
    v = V[j + 1].double()
    assert float(((v * w.norm(dim=1)[:, None] - w).norm(dim=1) / size).max()) < 1e-5
    assert float(torch.einsum("ikn,kn->ik", V[:j + 1].double(), v).abs().max()) < 1e-5
    assert float(((H[:j, j] - h[:j]).abs() / size).max()) < 1e-5
