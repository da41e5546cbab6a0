"""The block solver's products as partial sums.

Three terms: an accumulator takes 96 MMA steps of 16 products, each of which rounds the running
FP32 sum by at most 2^-23 of it, and the pieces are added to nearest: 96 2^-23 of the
sum of magnitudes and 2^-24 of it a piece. Operands of one sign show what a
longer chain leaves. One term (the plain product's K splits): FP32 accumulation, 2^-24 of the sum of
magnitudes a step of 16 products and a split.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,n", [(152 * 128, 12288, 24), (1000, 511, 200), (300, 1025, 16)])
def test_three_terms_of_one_sign(gpu, M, K, n):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cuda").manual_seed(K)
    ld = (K + 7) // 8 * 8
    A = torch.rand((M, 2 * ld), generator=g, device="cuda").to(torch.bfloat16)
    X = torch.rand((n, 2 * ld), generator=g, device="cuda").to(torch.bfloat16)
    need = nat.lib().mbem_gemm_bf16_workspace_size(M, n)
    work = torch.full((need // 4,), float("nan"), device="cuda")
    kb, per = ctypes.c_int(0), ctypes.c_int(0)
    nat.call("mbem_gemm_bf16x3_t_parts", ptr(A), A.stride(0), ld, ptr(X), X.stride(0), ld, M, K, n, ptr(work), need,
             ctypes.byref(kb), ctypes.byref(per), stream_handle())
    nat.call("mbem_gemm_bf16_check", stream_handle())
    kb, per = kb.value, per.value
    P = work[:(work.numel() // (n * M)) * n * M].view(-1, n, M)
    xh, xl = X[:, :K].double(), X[:, ld:ld + K].double()
    for t in sorted({0, (M - 1) // 256, (M - 1) // 128}):
        parts = ((t + 1) * kb - 1) // per - t * kb // per + 1
        rows = slice(128 * t, min(M, 128 * (t + 1)))
        y = P[:parts, :, rows].double().sum(dim=0)
        ah, al = A[rows, :K].double(), A[rows, ld:ld + K].double()
        ref = xh @ ah.T + xl @ ah.T + xh @ al.T
        err = float(((y - ref).abs() / ref).max())
        assert err <= 96 * 2.0 ** -23 + (3 * K / 1536 + 2) * 2.0 ** -24, err


@pytest.mark.parametrize("M,K,n", [(1, 1, 1), (129, 1000, 40), (3000, 3001, 256)])
def test_one_term_in_parts(gpu, M, K, n):
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cuda").manual_seed(M + K)
    ld = (K + 7) // 8 * 8
    A = torch.randn((M, ld), generator=g, device="cuda").to(torch.bfloat16)
    X = torch.randn((n, ld), generator=g, device="cuda").to(torch.bfloat16)
    need = nat.lib().mbem_gemm_bf16_workspace_size(M, n)
    work = torch.full((need // 4,), float("nan"), device="cuda")
    splits = ctypes.c_int(0)
    nat.call("mbem_gemm_bf16_t_parts", ptr(A), A.stride(0), ptr(X), X.stride(0), M, K, n, ptr(work), need,
             ctypes.byref(splits), stream_handle())
    nat.call("mbem_gemm_bf16_check", stream_handle())
    y = work[:splits.value * n * M].view(-1, n, M).double().sum(dim=0)
    a, x = A[:, :K].double(), X[:, :K].double()
    mag = x.abs() @ a.abs().T
    assert bool(((y - x @ a.T).abs() <= 2.0 ** -24 * (K / 16 + 16 + splits.value) * mag).all())


def test_one_term_solver(gpu):
    """The BF16 operator alone as the inner one: more refinement steps, the same solution. Both
    meet 1e-9 of the right-hand sides; the deflated 8-per-face system turns that into at
    most 1e-6 of the solution."""
    from mbem_gb300.backends.dense import DenseBackend
    from mbem_gb300.cases import cube_fault_model, gaussian_slips
    from mbem_gb300.la.multirhs import BlockSolver, slip_rhs
    from mbem_gb300.model import generate_system
    model, eps = cube_fault_model(8, 6)
    asm = DenseBackend(jump="calibrated", deflate=True, precision="mixed").assemble(generate_system(model), eps)
    fault = model.regions[0].faults[0]
    B = slip_rhs(asm, fault, gaussian_slips(fault, 5, 0.3, 2))
    X = []
    for terms in (1, 3):
        x, rep = BlockSolver(asm, terms=terms).solve(B, rtol=1e-9)
        assert rep.converged and np.all(rep.true_relres < 1e-9)
        X.append(x)
    assert float((X[0] - X[1]).norm() / X[1].norm()) < 1e-6


@pytest.mark.parametrize("n", [1003, 1024])
def test_operand_panels(gpu, n):
    """The next product's operand is [hi], [hi | lo] or [hi | lo | hi] of one and the same vector."""
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    k, m, ldp, dev = 3, 2, (n + 7) // 8 * 8, "cuda"
    P = torch.randn((1, k, n), device=dev)
    V0 = torch.nn.functional.normalize(torch.randn((k, n), device=dev), dim=1)
    seen = []
    for panels in (1, 2, 3):
        V = torch.zeros((m + 1, k, n), device=dev)
        V[0] = V0
        Vbf = torch.zeros((k, panels * ldp), dtype=torch.bfloat16, device=dev)
        H = torch.zeros((m, m, k), dtype=torch.float64, device=dev)
        cs, sn = (torch.zeros((m, k), dtype=torch.float64, device=dev) for _ in range(2))
        g, beta = torch.ones((m + 1, k), dtype=torch.float64, device=dev), torch.ones(k, dtype=torch.float64, device=dev)
        left = torch.zeros(1, dtype=torch.int32, device=dev)
        nat.call("mbem_batch_arnoldi", ptr(P), 1, 0, 0, n * k, ptr(V), 0, m, k, n, None, 0, ptr(Vbf), Vbf.stride(0), ldp,
                 panels, ptr(H), ptr(cs), ptr(sn), ptr(g), ptr(beta), 1e-3, ptr(left), stream_handle())
        hi = V[1].to(torch.bfloat16)
        lo = (V[1] - hi.float()).to(torch.bfloat16)
        seen.append(V[1])
        for p, want in enumerate((hi, lo, hi)[:panels]):
            assert torch.equal(Vbf[:, p * ldp:p * ldp + n], want)
    assert torch.equal(seen[0], seen[1]) and torch.equal(seen[0], seen[2])


def test_two_panels_are_held(gpu):
    from mbem_gb300.backends.dense import DenseBackend
    from mbem_gb300.cases import cube_fault_model
    from mbem_gb300.la.multirhs import BlockSolver
    from mbem_gb300.model import generate_system
    model, eps = cube_fault_model(4, 2)
    asm = DenseBackend(jump="calibrated", deflate=True, precision="mixed").assemble(generate_system(model), eps)
    for terms, panels in ((1, 1), (3, 2)):
        bs = BlockSolver(asm, terms=terms)
        assert bs.A16.shape == (bs.n, panels * bs.ldp)
        if terms == 3:
            A = asm.op.dense64()
            A16 = bs.A16[:, :bs.n].double() + bs.A16[:, bs.ldp:bs.ldp + bs.n].double()
            assert float((A16 - A).abs().max() / A.abs().max()) < 2.0 ** -16


