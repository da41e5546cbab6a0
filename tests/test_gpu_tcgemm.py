"""The tcgen05 multi-RHS GEMM against torch's FP32 product of the same BF16
operands. Tolerance: 1e-5 of the largest output entry (both accumulate in
FP32; the summation orders differ), 3e-5 for K = 4096."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(A, Xt):
    return A.float() @ Xt.float().T


@pytest.mark.parametrize("M,K,n", [(128, 64, 16), (300, 200, 37), (256, 1000, 256), (129, 72, 64), (64, 8, 5)])
def test_gemm_bf16_small(gpu, M, K, n):
    from mbem_gb300.la.multirhs import gemm_bf16, gemm_check
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + K + n)
    A = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    Xt = torch.randn((n, K), generator=g, device="cuda").to(torch.bfloat16)
    Y = gemm_bf16(A, Xt)
    gemm_check()
    R = _ref(A, Xt)
    assert float((Y - R).abs().max() / R.abs().max()) < 1e-5


def test_gemm_bf16_large_and_strided(gpu):
    from mbem_gb300.la.multirhs import gemm_bf16, gemm_check
    g = torch.Generator(device="cuda").manual_seed(7)
    big = torch.randn((4100, 4104), generator=g, device="cuda").to(torch.bfloat16)
    A = big[:4096, :4096]                          # lda = 4104
    Xt = torch.randn((256, 4096), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((4096, 260), 7.0, device="cuda")
    gemm_bf16(A, Xt, out=out[:, :256])
    gemm_check()
    R = _ref(A, Xt)
    assert float((out[:, :256] - R).abs().max() / R.abs().max()) < 3e-5
    assert torch.all(out[:, 256:] == 7.0)


@pytest.mark.parametrize("M,K,n", [(1000, 4096, 256), (20736, 1024, 64), (200, 640, 16)])
def test_gemm_split_k(gpu, M, K, n):
    """The K-split product (partial sums in slice order) equals the product."""
    from mbem_gb300.la.multirhs import gemm_bf16_t, gemm_check
    g = torch.Generator(device="cuda").manual_seed(M + K + n)
    A = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    Xt = torch.randn((n, K), generator=g, device="cuda").to(torch.bfloat16)
    out = torch.empty((n, M), device="cuda")
    gemm_bf16_t(A, Xt, K, out, split=True)
    gemm_check()
    ref = (A.float() @ Xt.float().T).T
    assert float((out - ref).abs().max() / ref.abs().max()) < 3e-5


@pytest.mark.parametrize("M,N,K", [(300, 7, 384), (1000, 64, 384), (936, 64, 384), (520, 130, 384), (200, 256, 192),
                                   (777, 33, 64), (128, 16, 384), (1500, 300, 384)])
def test_gemm_sub_update(gpu, M, N, K):
    """C -= A Bt^T (the LU update) against FP64 products of the same BF16
    operands: FP32 accumulation, tolerance 1e-5 of max|A Bt^T|; rows and
    columns outside C untouched."""
    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cpu").manual_seed(M + N)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    Bt = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    ldc = N + 5
    C0 = torch.randn(M + 3, ldc, generator=g).cuda()
    C = C0.clone()
    nat.call("mbem_gemm_bf16_sub", ptr(A), A.stride(0), ptr(Bt), Bt.stride(0), M, N, K, ptr(C), ldc, stream_handle())
    torch.cuda.synchronize()
    P = A.double() @ Bt.double().T
    ref = C0.double().clone()
    ref[:M, :N] -= P
    err = float((C.double() - ref).abs().max() / P.abs().max())
    assert err < 1e-5, err
    assert torch.equal(C[M:], C0[M:]) and torch.equal(C[:, N:], C0[:, N:])


@pytest.mark.parametrize("M,K,n", [(1, 1, 1), (127, 33, 16), (128, 32, 17), (129, 1000, 40), (700, 1001, 128),
                                   (1025, 500, 256), (5000, 3001, 100)])
def test_three_term_product_in_parts(gpu, M, K, n):
    """The runs' partial sums, added tile by tile, against the FP32 products of
    the same BF16 panels: FP32 accumulation in another order, 2^-24 times the sum
    of magnitudes times the chains (K / 16 products, three terms)."""
    import ctypes

    from mbem_gb300 import _native as nat
    from mbem_gb300._device import ptr, stream_handle
    g = torch.Generator(device="cuda").manual_seed(M + K)
    ld = (K + 7) // 8 * 8
    A = torch.randn((M, 3 * ld), generator=g, device="cuda").to(torch.bfloat16)
    X = torch.randn((n, 3 * ld), generator=g, device="cuda").to(torch.bfloat16)
    need = nat.lib().mbem_gemm_bf16_workspace_size(M, n)
    work = torch.full((need // 4,), float("nan"), device="cuda")
    kb, per = ctypes.c_int(0), ctypes.c_int(0)
    nat.call("mbem_gemm_bf16x3_t_parts", ptr(A), A.stride(0), 2 * ld, ptr(X), X.stride(0), ld, M, K, n, ptr(work),
             need, ctypes.byref(kb), ctypes.byref(per), stream_handle())
    nat.call("mbem_gemm_bf16_check", stream_handle())
    kb, per = kb.value, per.value
    P = work[:(work.numel() // (n * M)) * n * M].view(-1, n, M)
    Y = torch.empty((n, M), device="cuda", dtype=torch.float64)
    for t in range((M + 127) // 128):
        parts = ((t + 1) * kb - 1) // per - t * kb // per + 1
        rows = slice(128 * t, min(M, 128 * (t + 1)))
        Y[:, rows] = P[:parts, :, rows].double().sum(dim=0)
    ah, al = A[:, :K].double(), A[:, 2 * ld:2 * ld + K].double()
    xh, xl = X[:, :K].double(), X[:, ld:ld + K].double()
    ref = xh @ ah.T + xl @ ah.T + xh @ al.T
    mag = xh.abs() @ ah.abs().T + xl.abs() @ ah.abs().T + xh.abs() @ al.abs().T
    assert bool(((Y - ref).abs() <= 2.0 ** -24 * (3 * K / 16 + 16) * mag).all())
