"""Many right-hand sides: the tensor-core product Y = A X (``mbem_gemm_bf16``)
that replaces one matvec per right-hand side by one GEMM per iteration.

The reference solves many right-hand sides by one LU factorisation and its
triangular solves (src/mbem/la/lu.py:110-258, the refinement product at
:210); here the operator stays in HBM once as BF16 and every product over
the whole block of right-hand sides reads it once.
"""

from __future__ import annotations

import torch

from .. import _native as nat
from .._device import ptr, stream_handle

MAX_RHS = 256


def gemm_bf16(A: torch.Tensor, Xt: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """Y (M, n) FP32 = A (M, K) @ Xt (n, K)^T for BF16 CUDA tensors with
    unit column stride; n <= 256 (larger blocks: call per 256 columns)."""
    if A.dtype != torch.bfloat16 or Xt.dtype != torch.bfloat16 or not A.is_cuda:
        raise ValueError("A and Xt must be bfloat16 CUDA tensors")
    if A.stride(1) != 1 or Xt.stride(1) != 1 or A.shape[1] != Xt.shape[1]:
        raise ValueError("A (M, K) and Xt (n, K) need unit column strides and one K")
    M, K = A.shape
    n = Xt.shape[0]
    if not 1 <= n <= MAX_RHS:
        raise ValueError(f"1..{MAX_RHS} right-hand sides per product (got {n})")
    Y = out if out is not None else torch.empty((M, n), dtype=torch.float32, device=A.device)
    nat.call("mbem_gemm_bf16", ptr(A), A.stride(0), ptr(Xt), Xt.stride(0), M, K, n, ptr(Y), Y.stride(0),
             stream_handle())
    return Y


def gemm_check():
    """Synchronises and raises if a tensor-core pipeline wait gave up."""
    nat.call("mbem_gemm_bf16_check", stream_handle())


_split_work = {}


def gemm_bf16_t(A: torch.Tensor, Xt: torch.Tensor, K: int, out: torch.Tensor, split: bool = True) -> torch.Tensor:
    """out (n, M) FP32 = (A[:, :K] @ Xt[:, :K]^T)^T, out's rows at out.stride(0);
    with ``split`` K is divided over the SMs when the row tiles alone
    would leave them unevenly loaded."""
    M = A.shape[0]
    n = Xt.shape[0]
    if not split:
        nat.call("mbem_gemm_bf16_t", ptr(A), A.stride(0), ptr(Xt), Xt.stride(0), M, K, n, ptr(out),
                 out.stride(0), stream_handle())
        return out
    need = nat.lib().mbem_gemm_bf16_workspace_size(M, n)
    key = (A.device.index, need)
    work = _split_work.get(key)
    if work is None:
        work = torch.empty(need // 4, dtype=torch.float32, device=A.device)
        _split_work.clear()
        _split_work[key] = work
    nat.call("mbem_gemm_bf16_t_split", ptr(A), A.stride(0), ptr(Xt), Xt.stride(0), M, K, n, ptr(out),
             out.stride(0), ptr(work), need, stream_handle())
    return out


# ---------------------------------------------------------------------------
# a block of right-hand sides: batched GMRES on the BF16 tensor-core
# operator inside FP64-accurate iterative refinement
# ---------------------------------------------------------------------------
import ctypes  # noqa: E402
from dataclasses import dataclass, field  # noqa: E402

import numpy as np  # noqa: E402


@dataclass
class BlockReport:
    converged: bool
    outer: int                        # refinement steps
    inner_iterations: list = field(default_factory=list)   # batched GMRES iterations per step
    true_relres: np.ndarray = None    # per right-hand side |b - A x| / |b|
    gemm_ms: float = 0.0              # tensor-core GEMM time
    residual_ms: float = 0.0          # FP64-accurate residuals
    inner_ms: float = 0.0             # batched GMRES (GEMM included)

    def __str__(self):
        worst = float(np.max(self.true_relres)) if self.true_relres is not None else float("nan")
        return (f"block solve {'converged' if self.converged else 'NOT CONVERGED'}: {self.outer} refinement steps, "
                f"inner {self.inner_iterations}, worst relres {worst:.3e}")


def _pad8(n: int) -> int:
    return (n + 7) // 8 * 8


class BlockSolver:
    """Solves A X = B for up to 256 right-hand sides at once.

    The refinement loop computes the residual R = P (B - A X) with the
    accurate operator (the mixed operator's FP32 far field by exact digit
    products and its FP64 near blocks, or the FP64 dense matrix), and
    corrects X by batched GMRES on the BF16 copy of the operator, whose
    every step is one tensor-core GEMM over the whole block. P removes the
    rigid translations of the u-slots of a deflated system."""

    def __init__(self, asm, inner_restart: int = 30, inner_rtol: float = 3e-5, terms: int = 3):
        """``terms``: 1 = the operator in BF16 (relative error ~2^-9 per
        product: about five refinement steps to 1e-8); 3 = A and the Krylov
        vectors each split into BF16 high and low parts, A_hi V_hi + A_hi
        V_lo + A_lo V_hi in one product (error ~2^-16: two
        refinement steps)."""
        if terms not in (1, 3):
            raise ValueError("terms must be 1 or 3")
        self.terms = terms
        self.asm = asm
        self.op = asm.op
        self.A = asm.A
        if self.op is None and self.A is None:
            raise ValueError("the assembled system holds no operator")
        dev = (self.A if self.A is not None else self.op.A32).device
        self.device = dev
        self.n = n = int(asm.b.shape[0])
        self.ldp = _pad8(n)
        # A16 = [A_hi | A_lo] (terms 3) or A_hi, each panel ldp wide
        self.panels = 2 if terms == 3 else 1
        self.A16 = torch.zeros((n, self.panels * self.ldp), dtype=torch.bfloat16, device=dev)
        hi = self.A16[:, :self.ldp]
        lo = self.A16[:, self.ldp:] if terms == 3 else None
        st = stream_handle()
        ld16 = self.A16.stride(0)
        if self.op is not None:
            s = self.op.struct()
            nat.call("mbem_mixed_to_bf16x2", ctypes.byref(s), ptr(hi), ptr(lo) if lo is not None else None, ld16, st)
        elif lo is not None:
            nat.call("mbem_to_bf16x2", ptr(self.A), 1, self.A.stride(0), n, n, ptr(hi), ptr(lo), ld16, st)
        else:
            nat.call("mbem_to_bf16", ptr(self.A), 1, self.A.stride(0), n, n, ptr(hi), ld16, st)
        rng = np.ascontiguousarray(np.asarray(asm.u_ranges(), dtype=np.int64).reshape(-1))
        self._ranges = rng
        self.inner_restart = inner_restart
        self.inner_rtol = inner_rtol

    # -- pieces ---------------------------------------------------------
    def project(self, X: torch.Tensor):
        if self._ranges.size == 0:
            return X
        is64 = 1 if X.dtype == torch.float64 else 0
        nat.call("mbem_batch_project", ptr(X), is64, X.shape[0], X.shape[1],
                 self._ranges.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), len(self._ranges) // 2,
                 stream_handle())
        return X

    def residual(self, B: torch.Tensor, X: torch.Tensor) -> torch.Tensor:
        """P (B - A X) for (k, n) FP64 blocks with the accurate operator."""
        k = B.shape[0]
        R = torch.empty_like(B)
        if self.op is not None:
            need = nat.lib().mbem_batch_residual_workspace_size(k, self.n)
            work = torch.empty(need // 8, dtype=torch.float64, device=self.device)
            s = self.op.struct()
            nat.call("mbem_batch_residual_mixed", ctypes.byref(s), ptr(B), ptr(X), k, ptr(R), ptr(work), need,
                     stream_handle())
        else:
            Y = torch.empty((self.n, k), dtype=torch.float64, device=self.device)
            Xc = X.T.contiguous()
            nat.call("mbem_dgemm_multi", ptr(self.A), self.A.stride(0), self.n, self.n, ptr(Xc), k, ptr(Y),
                     stream_handle())
            R = B - Y.T
        return self.project(R)

    def product_workspace(self, k: int) -> torch.Tensor:
        return torch.empty(nat.lib().mbem_gemm_bf16_workspace_size(self.n, k) // 4, dtype=torch.float32,
                           device=self.device)

    def product_parts(self, Vbf: torch.Tensor, work: torch.Tensor):
        """A16's product with the BF16 vectors of ``Vbf`` (k, panels ldp) as
        partial sums in ``work``: (splits, kb, per), what
        ``mbem_batch_arnoldi`` adds them up by."""
        k, ld, st = Vbf.shape[0], self.ldp, stream_handle()
        parts, kb, per = ctypes.c_int(0), ctypes.c_int(0), ctypes.c_int(0)
        if self.terms == 3:
            nat.call("mbem_gemm_bf16x3_t_parts", ptr(self.A16), self.A16.stride(0), ld, ptr(Vbf), Vbf.stride(0), ld,
                     self.n, self.n, k, ptr(work), 4 * work.numel(), ctypes.byref(kb), ctypes.byref(per), st)
        else:
            nat.call("mbem_gemm_bf16_t_parts", ptr(self.A16), self.A16.stride(0), ptr(Vbf), Vbf.stride(0), self.n, ld,
                     k, ptr(work), 4 * work.numel(), ctypes.byref(parts), st)
        return parts.value, kb.value, per.value

    def inner_gmres(self, R: torch.Tensor, m: int, rtol: float):
        """D (k, n) FP64 with |R - A16 D| small for every row, by batched
        GMRES(m) on the BF16 operator; returns (D, iterations, gemm_ms)."""
        k, n = R.shape
        dev = self.device
        st = stream_handle()
        ld = self.ldp
        V = torch.empty((m + 1, k, n), dtype=torch.float32, device=dev)
        # the GEMM operand [V_hi | V_lo] (or V_hi); its padding stays zero
        Vbf = torch.zeros((k, self.panels * ld), dtype=torch.bfloat16, device=dev)
        beta = torch.empty(k, dtype=torch.float64, device=dev)
        nat.call("mbem_batch_normalize", ptr(R), 1, k, n, ptr(beta), ptr(V[0]), None, st)
        vh = V[0].to(torch.bfloat16)
        Vbf[:, :n] = vh
        if self.panels == 2:
            Vbf[:, ld:ld + n] = (V[0] - vh.float()).to(torch.bfloat16)
        H = torch.zeros((m, m, k), dtype=torch.float64, device=dev)
        rot = torch.zeros((2, m, k), dtype=torch.float64, device=dev)
        g = torch.zeros((m + 1, k), dtype=torch.float64, device=dev)
        g[0] = beta
        left = torch.zeros(m, dtype=torch.int32, device=dev)
        work = self.product_workspace(k)
        ranges = self._ranges.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
        events = []
        jdone = 0
        for j in range(m):
            ev = (torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
            ev[0].record()
            parts, kb, per = self.product_parts(Vbf, work)
            ev[1].record()
            events.append(ev)
            nat.call("mbem_batch_arnoldi", ptr(work), parts, kb, per, n * k, ptr(V), j, m, k, n, ranges,
                     len(self._ranges) // 2, ptr(Vbf), Vbf.stride(0), ld, self.panels, ptr(H), ptr(rot[0]), ptr(rot[1]),
                     ptr(g), ptr(beta), float(rtol), ptr(left[j:]), st)
            jdone = j + 1
            if int(left[j]) == 0:
                break
        Y = torch.empty((jdone, k), dtype=torch.float64, device=dev)
        nat.call("mbem_batch_backsolve", ptr(H), ptr(g), m, jdone, k, ptr(Y), st)
        D = torch.zeros((k, n), dtype=torch.float64, device=dev)
        nat.call("mbem_batch_update", ptr(D), ptr(V), jdone, ptr(Y), k, n, st)
        return D, jdone, sum(a.elapsed_time(b) for a, b in events)

    # -- the solve ------------------------------------------------------
    def solve(self, B: torch.Tensor, rtol: float = 1e-8, max_outer: int = 12):
        """X (k, n) FP64 for B (k, n) FP64 on the device, and a BlockReport."""
        B = self.project(B.to(dtype=torch.float64, device=self.device).contiguous().clone())
        k = B.shape[0]
        if not 1 <= k <= MAX_RHS:
            raise ValueError(f"1..{MAX_RHS} right-hand sides per block (got {k})")
        bnorm = torch.linalg.vector_norm(B, dim=1).cpu().numpy()
        X = torch.zeros_like(B)
        rep = BlockReport(converged=False, outer=0)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        rep.residual_ms = 0.0
        rep.inner_ms = 0.0
        for outer in range(max_outer + 1):
            ev[0].record()
            R = B.clone() if outer == 0 else self.residual(B, X)     # X = 0: R = P B
            ev[1].record()
            ev[1].synchronize()
            rep.residual_ms += ev[0].elapsed_time(ev[1])
            rel = torch.linalg.vector_norm(R, dim=1).cpu().numpy() / np.where(bnorm > 0, bnorm, 1.0)
            rep.true_relres = rel
            if np.all(rel < rtol) or outer == max_outer:
                rep.converged = bool(np.all(rel < rtol))
                break
            ev[0].record()
            D, its, ms = self.inner_gmres(R, self.inner_restart, self.inner_rtol)
            ev[1].record()
            ev[1].synchronize()
            rep.inner_ms += ev[0].elapsed_time(ev[1])
            rep.inner_iterations.append(its)
            rep.gemm_ms += ms
            X += D
            self.project(X)
            rep.outer = outer + 1
        gemm_check()
        return X, rep


def slip_rhs(asm, fault, slips) -> torch.Tensor:
    """B (k, n) FP64: the right-hand sides of k slip patterns (k, n_dofs, 3)
    on a prescribed-slip fault, every other datum of the system zero. Each
    RHS term of the fault (equations.py:296-309: scale -sigma times the T
    block) is assembled once in FP64 and applied to all patterns at once."""
    from ..kernels import KERNEL_T
    from ..kernels import basis as kb
    from ..kernels import tri_nodal as tn
    slips = np.asarray(slips, float)
    k = slips.shape[0]
    dev = asm.b.device
    B = torch.zeros((k, asm.b.shape[0]), dtype=torch.float64, device=dev)
    S = torch.from_numpy(np.ascontiguousarray(slips.reshape(k, -1).T)).to(dev)     # (3 n_src, k)
    held = asm._arrays
    if held is None:
        asm._arrays = asm._arrays_in if asm._arrays_in is not None else {}
    for rt in asm.system.rhs_terms:
        if rt.source_patch is not fault:
            continue
        if rt.kernel != KERNEL_T:
            raise NotImplementedError("slip right-hand sides through the T kernel only")
        mat = asm.materials[rt.region.name]
        f = asm._patch_arrays(rt.field_patch)
        s = asm._patch_arrays(rt.source_patch)
        c = kb.t_coeffs(mat.mu, mat.lam)
        T = tn.t_matrix_direct(f["coll"], s["tv"], s["normals"], s["eps"], *c, order=rt.source_patch.order)
        Y = torch.empty((T.shape[0], k), dtype=torch.float64, device=dev)
        nat.call("mbem_dgemm_multi", ptr(T), T.stride(0), T.shape[0], T.shape[1], ptr(S), k, ptr(Y),
                 stream_handle())
        B[:, rt.row.offset:rt.row.stop] += rt.scale * Y.T
    asm._arrays = held
    return B
