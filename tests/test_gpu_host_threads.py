"""Kernels whose shared memory goes with the call, launched from two host threads with a large and a
small call: each call finds the limit that it needs, whatever the other has set. The
threads are native ones (Python's take turns)."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <atomic>
#include <thread>
#include <vector>
#include "mbem_gb300.h"

struct Arnoldi { const float* P; float* V; int64_t k, n; uint16_t* Vbf; double *H, *cs, *sn, *g, *beta; int* left; };
struct Stress { const double* x; int64_t nf; const double *tv, *n, *eps, *d; double* out; };

template <class Call> static int both(int repeats, Call a, Call b, int (*wait)()) {
    std::atomic<int> worst{0}, ready{0};
    auto loop = [&](Call& c) {
        ready++;
        while (ready < 2) {}
        for (int i = 0; i < repeats; i++) {
            const int e = c();
            if (e) worst = e;
            if (i % 100 == 99) wait();
        }
    };
    std::thread t([&] { loop(a); });
    loop(b);
    t.join();
    return worst;
}
struct CallArnoldi {
    Arnoldi* a;
    int operator()() { return mbem_batch_arnoldi(a->P, 1, 0, 0, a->k * a->n, a->V, 0, 4, a->k, a->n, nullptr, 0, a->Vbf,
        (a->n + 7) / 8 * 8, (a->n + 7) / 8 * 8, 1, a->H, a->cs, a->sn, a->g, a->beta, 1e-3, a->left, nullptr); }
};
struct CallStress {
    Stress* a;
    int operator()() { return mbem_stress_contract(3, a->x, a->nf, a->tv, a->n, a->eps, 3, a->d, 1.0, 1.0, 2, 1.0, 0,
                                                   a->out, nullptr); }
};
static int wait_gemm() { return mbem_gemm_bf16_check(nullptr); }
extern "C" int arnoldi(int repeats, Arnoldi* a, Arnoldi* b) { return both(repeats, CallArnoldi{a}, CallArnoldi{b}, wait_gemm); }
extern "C" int stress(int repeats, Stress* a, Stress* b) { return both(repeats, CallStress{a}, CallStress{b}, wait_gemm); }
"""


@pytest.fixture(scope="module")
def threads(tmp_path_factory):
    from mbem_gb300 import build as B
    from mbem_gb300 import _native as nat
    nat.lib()
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("threads")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-I", os.path.join(ROOT, "include"),
                    str(d / "t.cpp"), "-o", str(d / "t.so"), "-L", B.LIBDIR, "-l:" + B.LIBNAME,
                    "-Wl,-rpath," + B.LIBDIR], check=True)
    return ctypes.CDLL(str(d / "t.so"))


def _struct(*values):
    """C layout of the tensors' pointers and the integers, and what keeps them alive."""
    raw = (ctypes.c_int64 * len(values))(*[v.data_ptr() if isinstance(v, torch.Tensor) else v for v in values])
    return raw, values


def test_nodal_contractions(gpu, threads):
    rng = np.random.default_rng(0)
    tv = torch.from_numpy(np.eye(3)[None] + rng.normal(size=(3, 1, 3))).cuda()
    n = torch.nn.functional.normalize(torch.ones((3, 3), dtype=torch.float64, device="cuda"), dim=1)
    eps = torch.full((3,), 0.1, dtype=torch.float64, device="cuda")
    d = torch.zeros((18, 3), dtype=torch.float64, device="cuda")

    def args(nf):
        x = torch.randn((nf, 3), dtype=torch.float64, device="cuda")
        return _struct(x, nf, tv, n, eps, d, torch.empty((nf, 9), dtype=torch.float64, device="cuda"))
    # sixteen observers a block (47 KB beside the static tables) against one
    big, small = args(20000), args(1)
    assert threads.stress(20000, big[0], small[0]) == 0


def test_batched_arnoldi(gpu, threads):
    dev, k, m = "cuda", 2, 4

    def args(n):
        ldp = (n + 7) // 8 * 8
        f = dict(dtype=torch.float64, device=dev)
        return _struct(torch.randn((1, k, n), device=dev), torch.randn((m + 1, k, n), device=dev), k, n,
                       torch.zeros((k, ldp), dtype=torch.bfloat16, device=dev), torch.zeros((m, m, k), **f),
                       torch.ones((m, k), **f), torch.zeros((m, k), **f), torch.ones((m + 1, k), **f),
                       torch.ones(k, **f), torch.zeros(1, dtype=torch.int32, device=dev))
    big, small = args(120_000), args(64)
    assert threads.arnoldi(20000, big[0], small[0]) == 0
