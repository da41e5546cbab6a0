"""Performance cases: the work a user of the framework has it do, through its public entry points.

The dense boundary-element path is measured at each of its layers and as whole calls:

* ``matrix``    a block of the collocation matrix (T or U kernel, P0 / P1 / P2 densities), FP64;
* ``traction``  the traction rows of a FAULT_TRACTION fault over a boundary (P0), FP64;
* ``disp``      displacement of a slip density at a list of stations, FP64;
* ``stress``    the eigenstress-subtracted stress of a slip density at observers, FP64;
* ``readout``   the same stress at many observers in mixed precision;
* ``solve``     a cube with an embedded fault assembled and solved (FP64, or the mixed operator with the
                learned preconditioner inside its BF16 inner solve);
* ``block``     many slip right-hand sides solved at once on a kept mixed operator.

Sizes are those of the repository's benchmark, tests and profiles (cube grids of 8 to 48 per face, faults of 8 to 32
per side, 256 slip patterns, a 64 x 64 readout grid, 100,000 readout points), odd ones beside them.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from mbem_gb300 import mesh as M
from mbem_gb300.backends.dense import DenseBackend
from mbem_gb300.cases import gaussian_slips
from mbem_gb300.evaluate import evaluate_stress
from mbem_gb300.kernels import basis as kb
from mbem_gb300.kernels import tri_nodal as tn
from mbem_gb300.la.multirhs import BlockSolver, slip_rhs
from mbem_gb300.model import BCType, Patch, Region, RegionModel, generate_system

SIDE = 4.0                       # cube side; faults have side 1
NODES = {0: 1, 1: 3, 2: 6}       # Lagrange nodes per triangle by order


def listed():
    return [
        # the self block of a small fault, 8 x 8 squares: the smallest call, where launches and idle SMs count
        dict(name="t_p0_fault8", kind="matrix", kernel="T", order=0, surface="fault", ns=128, nf=0),
        # the self block of the 12-per-face cube: the FP64 assembly's main kernel at an ordinary size
        dict(name="t_p0_cube12", kind="matrix", kernel="T", order=0, surface="cube", ns=1728, nf=0),
        # the P1 self block of the 8-per-face cube (2,304 collocation points)
        dict(name="t_p1_cube8", kind="matrix", kernel="T", order=1, surface="cube", ns=768, nf=0),
        # a P2 single-layer block at a ragged size: 1,001 field points over part of a fault
        dict(name="u_p2_ragged", kind="matrix", kernel="U", order=2, surface="fault", ns=333, nf=1001),
        # the traction rows of a 12 x 12 fault (288 points) over a boundary of 6,144 triangles
        dict(name="traction_p0", kind="traction", ns=6144, nf=288),
        # displacement at a network of 48 stations from a density on the 24-per-face cube
        dict(name="disp_stations", kind="disp", order=0, surface="cube", ns=6912, nf=48),
        # stress on a 64 x 64 grid inside the solved 12-per-face cube with an 8 x 8 fault
        dict(name="stress_grid64", kind="grid", n_face=12, n_fault=8, nf=4096),
        # the parity readout of a P2 fault (16 x 16) at 2,000 observers, FP64
        dict(name="stress_p2", kind="stress", order=2, surface="fault", ns=512, nf=2000),
        # the mixed readout of a P2 fault (32 x 32) at 100,000 observers, a tenth of them at the fault
        dict(name="readout_p2", kind="readout", order=2, ns=2048, nf=100_000),
        # the plain dense system of the 12-per-face cube, assembled and solved to 1e-10 in FP64
        dict(name="solve_fp64_cube12", kind="solve", precision="fp64", n_face=12, n_fault=8),
        # 256 smooth random slip patterns on the kept 24-per-face operator
        dict(name="block_cube24", kind="block", n_face=24, n_fault=16, nrhs=256),
        # the 82,944-unknown mixed system with the learned preconditioner: the whole call from host arrays
        dict(name="solve_mixed_cube48", kind="solve", precision="mixed", n_face=48, n_fault=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matrix", "matrix", "matrix", "traction", "disp", "stress", "stress", "grid", "readout",
                       "solve", "block"])
    if kind == "matrix":
        order = rng.choice([0, 1, 2])
        ns = _log(rng, 40, (1728, 768, 333)[order])
        nf = _log(rng, 40, (1728, 2304, 2000)[order])
        return dict(kind=kind, kernel=rng.choice(["T", "U"]), order=order, surface=rng.choice(["cube", "fault"]),
                    ns=ns, nf=nf)
    if kind == "traction":
        return dict(kind=kind, ns=_log(rng, 200, 6144), nf=_log(rng, 30, 288))
    if kind == "disp":
        order = rng.choice([0, 0, 1, 2])
        return dict(kind=kind, order=order, surface=rng.choice(["cube", "fault"]),
                    ns=_log(rng, 100, (6912, 1500, 600)[order]), nf=_log(rng, 5, 500))
    if kind == "stress":
        order = rng.choice([0, 1, 2])
        return dict(kind=kind, order=order, surface=rng.choice(["cube", "fault"]),
                    ns=_log(rng, 60, (1728, 768, 512)[order]), nf=_log(rng, 40, 2000))
    if kind == "grid":
        return dict(kind=kind, n_face=rng.randint(6, 12), n_fault=rng.randint(4, 8), nf=_log(rng, 200, 4096))
    if kind == "readout":
        return dict(kind=kind, order=rng.choice([0, 1, 2]), ns=_log(rng, 200, 2048), nf=_log(rng, 5_000, 100_000))
    if kind == "solve":
        precision = rng.choice(["fp64", "mixed"])
        n = rng.randint(6, 12) if precision == "fp64" else _log(rng, 12, 47)
        return dict(kind=kind, precision=precision, n_face=n, n_fault=max(4, (2 * n) // 3))
    return dict(kind=kind, n_face=rng.randint(10, 23), n_fault=rng.randint(6, 16), nrhs=_log(rng, 16, 256))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return q


def _turned(mesh, Q):
    mesh.vertices = np.ascontiguousarray(mesh.vertices @ Q.T)
    return mesh


def _surface(case, rng):
    """The first ``ns`` triangles of the smallest cube or fault that has them, turned by a random rotation:
    (tri_verts, normals, eps, rotation); eps is half the grid spacing."""
    ns = case["ns"]
    if case.get("surface", "cube") == "cube":
        n = math.ceil(math.sqrt(ns / 12))
        mesh, h = M.cube(n, SIDE), SIDE / n
    else:
        n = math.ceil(math.sqrt(ns / 2))
        mesh, h = M.centre_fault(n), 1.0 / n
    Q = _rotation(rng)
    mesh = _turned(mesh, Q)
    nrm, _ = mesh.normals_and_areas()
    return mesh.tri_verts()[:ns], nrm[:ns], np.full(ns, 0.5 * h), Q


def _cuda(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _model(case, rng):
    """The cube with an embedded fault through the region-model API, turned, under a random uniform slip."""
    Q = _rotation(rng)
    n = case["n_face"]
    cube = Patch("cube", _turned(M.cube(n, SIDE), Q), BCType.FREE_TRACTION)
    slip = Q @ np.array([1.0, 0.3 * rng.normal(), 0.0])[[0, 2, 1]]       # along strike, with some dip
    fault = Patch("fault", _turned(M.centre_fault(case["n_fault"]), Q), BCType.FAULT, value=slip)
    region = Region("body", M.ElasticMaterial(mu=1.0, lam=1.0), [cube], np.zeros(3), faults=[fault])
    return RegionModel([region]), 0.5 * SIDE / n, Q, slip


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("matrix", "disp", "stress", "traction"):
        tv, nrm, eps, Q = _surface(case, rng)
        order, nf = case.get("order", 0), case["nf"]
        st = dict(case=case)
        if kind == "matrix" and nf == 0:         # the self block: the surface's own collocation points
            x = _collocation(tv, order)
        elif kind == "traction":                 # points and normals of a small fault inside the cube
            f = _turned(M.centre_fault(math.ceil(math.sqrt(nf / 2))), Q)
            x = f.centroids()[:nf]
            st["nx"] = _cuda(f.normals_and_areas()[0][:nf])[0]
        else:                                    # points of the body
            x = rng.uniform(-1.0, 1.0, size=(nf, 3)) @ Q.T
        st["x"], st["tv"], st["n"], st["eps"] = _cuda(x, tv, nrm, eps)
        st["ids"] = np.arange(case["ns"], dtype=np.int64).reshape(-1, 1)
        if kind in ("disp", "stress"):
            st["d"] = _cuda(rng.normal(size=(NODES[order] * case["ns"], 3)))[0]
        return st
    if kind == "readout":
        n = math.ceil(math.sqrt(case["ns"] / 2))
        fault = M.centre_fault(n)
        tv, ns, nf = fault.tri_verts()[:case["ns"]], case["ns"], case["nf"]
        nrm = fault.normals_and_areas()[0][:ns]
        eps = 0.07 * float(np.linalg.norm(tv[:, [1, 2, 0]] - tv, axis=2).mean(axis=1).min())
        x = rng.uniform(-1.0, 1.0, size=(nf, 3))
        x[:nf // 10, 1] = rng.uniform(-2 * eps, 2 * eps, size=nf // 10)
        d = rng.normal(size=(NODES[case["order"]] * ns, 3))
        x, tv, nrm, eps, d = _cuda(x, tv, nrm, np.full(ns, eps), d)
        return dict(case=case, x=x, tv=tv, n=nrm, eps=eps, d=d)
    model, eps, Q, _ = _model(case, rng)
    if kind == "solve":
        return dict(case=case, model=model, eps=eps)
    if kind == "grid":
        # a grid of the plane y = 0.1 as a tensor on the device, the boundary displacement a smooth field
        n = math.ceil(math.sqrt(case["nf"]))
        g = (np.arange(n) + 0.5) / n * SIDE - 0.5 * SIDE
        X, Z = np.meshgrid(g, g, indexing="xy")
        pts = np.column_stack([X.ravel(), np.full(X.size, 0.1), Z.ravel()])[:case["nf"]] @ Q.T
        cube = model.regions[0].patches[0]
        return dict(case=case, model=model, eps=eps, solution={"u:cube": _smooth(cube.mesh.centroids(), rng)},
                    points=_cuda(pts)[0])
    be = DenseBackend(jump="calibrated", deflate=True, precision="mixed")
    asm = be.assemble(generate_system(model), eps)
    fault = model.regions[0].faults[0]
    slips = gaussian_slips(fault, case["nrhs"], 0.3, int(rng.integers(1 << 30)))
    return dict(case=case, solver=BlockSolver(asm), B=slip_rhs(asm, fault, slips))


def _smooth(c, rng):
    k, ph = rng.normal(size=(3, 3)), rng.uniform(0, 6.28, size=3)
    return 0.1 * np.sin(c @ k.T + ph)


def _collocation(tv, order):
    """Collocation points: the centroid at order 0, else the Lagrange nodes half-way to the centroid."""
    lam = {0: np.full((1, 3), 1.0 / 3.0), 1: np.eye(3),
           2: np.vstack([np.eye(3), [[0.5, 0.5, 0], [0, 0.5, 0.5], [0.5, 0, 0.5]]])}[order]
    if order:
        lam = 0.5 * lam + 0.5 / 3.0
    return np.einsum("kv,svc->skc", lam, tv).reshape(-1, 3)


def run(state):
    case = state["case"]
    kind, order = case["kind"], case.get("order", 0)
    if kind == "matrix":
        if case["kernel"] == "T":
            return tn.t_matrix_direct(state["x"], state["tv"], state["n"], state["eps"], *kb.t_coeffs(1.0, 1.0),
                                      order)
        return tn.u_matrix_direct(state["x"], state["tv"], state["eps"], *kb.u_coeffs(1.0, 1.0), order)
    if kind == "traction":
        return tn.traction_matrix(state["x"], state["nx"], state["tv"], state["n"], state["eps"], state["ids"],
                                  case["ns"], 1.0, 1.0, 0, "slip")
    if kind == "disp":
        return tn.t_disp_contract(state["x"], state["tv"], state["n"], state["eps"], state["d"],
                                  *kb.t_coeffs(1.0, 1.0), order)
    if kind == "stress":
        return tn.elastic_stress_contract(state["x"], state["tv"], state["n"], state["eps"], state["d"], 1.0, 1.0,
                                          order)
    if kind == "readout":
        return tn.elastic_stress_readout(state["x"], state["tv"], state["n"], state["eps"], state["d"], 1.0, 1.0,
                                         order)
    if kind == "grid":
        return evaluate_stress(state["model"], "body", state["solution"], state["points"], state["eps"])
    if kind == "solve":
        mixed = case["precision"] == "mixed"
        be = DenseBackend(jump="calibrated", deflate=True, precision=case["precision"],
                          precond="bf16_learned" if mixed else None)
        asm = be.assemble(generate_system(state["model"]), state["eps"])
        u = asm.solve()["u:cube"]
        # the FP64 system is small enough to be kept; the mixed one is held for the solve alone
        return {"u": u, "b": asm.b} if mixed else {"u": u, "b": asm.b, "A": asm.A}
    return state["solver"].solve(state["B"], rtol=1e-10)[0]


def work(case):
    """Bytes of the inputs and outputs, and the FLOPs of the closed forms (about 600 for a P0 T block, 300 for a U
    block, 1,000 for a stress pair and as much again for the higher moments of each order)."""
    kind, order = case["kind"], case.get("order", 0)
    K = NODES[order]
    if kind in ("matrix", "traction", "disp", "stress", "readout"):
        ns, nf = case["ns"], case["nf"]
        if kind == "matrix" and nf == 0:
            nf = K * ns
        n_in = 8 * (3 * nf + 13 * ns)
        pairs = nf * ns
        if kind == "matrix":
            return {"bytes": n_in + 8 * 9 * K * pairs,
                    "flops": pairs * (1 + order) * (600 if case["kernel"] == "T" else 300)}
        if kind == "traction":
            return {"bytes": n_in + 8 * 9 * pairs, "flops": 1500 * pairs}
        out = 3 if kind == "disp" else 9
        return {"bytes": n_in + 8 * (3 * K * ns + out * nf),
                "flops": pairs * (1 + order) * (600 if kind == "disp" else 1000)}
    ns = 12 * case["n_face"] ** 2
    nq = 2 * case["n_fault"] ** 2
    if kind == "grid":
        return {"bytes": 8 * (12 * case["nf"] + 16 * (ns + nq)), "flops": 1000 * case["nf"] * (ns + nq)}
    n = 3 * ns
    if kind == "block":
        # one read of the operator, the right-hand sides and solutions; ten products
        return {"bytes": 4 * n * n + 16 * n * case["nrhs"], "flops": 20 * n * n * case["nrhs"]}
    if case["precision"] == "fp64":
        return {"bytes": 8 * n * n, "flops": 600 * ns * (ns + nq) + 50 * n * n}
    return {"bytes": 6 * n * n, "flops": 300 * ns * (ns + nq) + 30 * n * n}


# ---------------------------------------------------------------------------
# the same values by adaptive quadrature of the mollified kernels in 64 bits
# ---------------------------------------------------------------------------
def _rule(n, split=0):
    """Collapsed Gauss rule of n x n points on each of 4^split equal sub-triangles: (barycentric (q, 3), weights
    that sum to 1/2)."""
    g, w = np.polynomial.legendre.leggauss(n)
    g, w = 0.5 * (g + 1), 0.5 * w
    a = np.repeat(g, n)
    b = np.tile(g, n) * (1 - a)
    w = np.repeat(w, n) * np.tile(w, n) * (1 - a)
    lam = np.column_stack([1 - a - b, a, b])
    for _ in range(split):
        h = 0.5 * np.eye(3)
        m = [np.vstack([np.eye(3)[i], h[i] + h[(i + 1) % 3], h[i] + h[(i + 2) % 3]]) for i in range(3)]
        m.append(np.vstack([h[0] + h[1], h[1] + h[2], h[2] + h[0]]))
        lam, w = np.vstack([lam @ t for t in m]), np.concatenate([0.25 * w] * 4)
    return _cuda(lam, w)


def _shapes(lam, order):
    if order == 0:
        return torch.ones_like(lam[:, :1])
    if order == 1:
        return lam
    return torch.cat([lam * (2 * lam - 1), 4 * lam * lam.roll(-1, 1)], 1)


def _unit(d):
    return torch.eye(3, dtype=d.dtype, device=d.device)


def _point_block(kernel, d, nrm, e2):
    """The (..., 3, 3) displacement kernel at offsets d (P, q, 3) for mu = lam = 1, nu = 1/4."""
    c1 = 1 / (16 * math.pi * 0.75)
    dd = (d * d).sum(-1)
    ir = (dd + e2[:, None]) ** -0.5
    I, outer = _unit(d), d[..., :, None] * d[..., None, :]
    if kernel == "U":
        diag = 2 * c1 * ir + e2[:, None] * ir ** 3 / (8 * math.pi)
        return diag[..., None, None] * I + c1 * (ir ** 3)[..., None, None] * outer
    a, b = ir ** 3, ir ** 5
    n = nrm[:, None, :].expand_as(d)
    dn = (d * n).sum(-1)
    al = d * ((2 - 4) * a + 3 * dd * b + 4.5 * e2[:, None] * b)[..., None]
    nd, dn_ = n[..., :, None] * d[..., None, :], al[..., :, None] * n[..., None, :]
    r1 = 2 * a + 4.5 * e2[:, None] * b
    out = dn_ + r1[..., None, None] * (nd + dn[..., None, None] * I)
    r2 = nd + 2 * d[..., :, None] * n[..., None, :] + dn[..., None, None] * I
    return c1 * (out - a[..., None, None] * r2 + (6 * b * dn)[..., None, None] * outer)


def _point_stress(d, u, nrm, e2):
    """Elastic stress (..., 6: xx yy zz xy xz yz) of a point dislocation u on normal nrm, mu = lam = 1, nu = 1/4:
    the double-layer stress of the mollified kernel minus its eigenstress."""
    c1 = 1 / (16 * math.pi * 0.75)
    v = nrm[:, None, :]
    e = e2[:, None]
    dd = (d * d).sum(-1)
    ir2 = 1 / (dd + e)
    a = ir2 ** 1.5
    b, c = a * ir2, a * ir2 * ir2
    du, dv, uv = (d * u).sum(-1), (d * v).sum(-1), (u * v).sum(-1)
    blob = 1.5 * e
    x0, x1 = 2 * a - 3 * (dd + blob) * b, -12 * b + 15 * (dd + blob) * c
    a1 = -a - 3 * blob * b
    s0 = 2 * uv * a - 6 * du * dv * b
    g = 3 * b + 15 * blob * c - 6 * b
    ee = 30 * du * dv * c - 6 * uv * b
    w = dv[..., None] * u + du[..., None] * v
    trx = 3 * x0 + x1 * dd
    trs = 2 * a1 * uv + 3 * s0 + g * 2 * du * dv + ee * dd
    trb = c1 * (uv * trx + trs)
    phi = 15 / (8 * math.pi) * e * e * c
    out = []
    for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
        sym = u[..., i] * v[..., j] + v[..., i] * u[..., j]
        dij = d[..., i] * d[..., j]
        bb = uv * x1 * dij * 2 + 2 * a1 * sym + g * (w[..., i] * d[..., j] + d[..., i] * w[..., j]) + 2 * ee * dij
        if i == j:
            bb = bb + 2 * uv * x0 + 2 * s0
            out.append(-trb - c1 * bb - phi * (uv + sym))
        else:
            out.append(-c1 * bb - phi * sym)
    return torch.stack(out, -1)


_FULL = [0, 3, 4, 3, 1, 5, 4, 5, 2]


def _by_class(x, tv, eps, rows):
    """Index pairs (f, s) of the field points ``rows`` and every source, by the rule that resolves them."""
    L = (tv - tv.roll(1, 1)).norm(dim=2).max(1).values
    D = torch.cdist(x[rows.start:rows.stop], tv.mean(1), compute_mode="donot_use_mm_for_euclid_dist") / L
    near = max(2, math.ceil(math.log2(float((L / eps).max()) / 1.2)))
    for lo, hi, n, split in ((0, 1.3, 10, near), (1.3, 3, 10, 1), (3, 7, 9, 0), (7, 1e9, 7, 0)):
        f, s = torch.nonzero((D >= lo) & (D < hi), as_tuple=True)
        lam, w = _rule(n, split)
        step = max(1, 3_000_000 // lam.shape[0])
        for k in range(0, f.shape[0], step):
            yield f[k:k + step] + rows.start, s[k:k + step], lam, w


def _rows(nf, ns):
    step = max(1, 20_000_000 // max(ns, 1))
    return [range(k, min(nf, k + step)) for k in range(0, nf, step)]


def _areas2(tv):
    return torch.linalg.cross(tv[:, 1] - tv[:, 0], tv[:, 2] - tv[:, 0]).norm(dim=1)


def _matrix(kernel, x, tv, nrm, eps, order):
    nf, ns, K = x.shape[0], tv.shape[0], NODES[order]
    out = torch.zeros((nf, 3, ns, K, 3), dtype=torch.float64, device=x.device)
    A2 = _areas2(tv)
    for rows in _rows(nf, ns):
        for f, s, lam, w in _by_class(x, tv, eps, rows):
            d = x[f][:, None, :] - torch.einsum("qv,pvc->pqc", lam, tv[s])
            blk = _point_block(kernel, d, nrm[s], eps[s] ** 2)
            blk = torch.einsum("qk,pqij->pikj", w[:, None] * _shapes(lam, order), blk)
            out[f, :, s] = blk * A2[s][:, None, None, None]
    return out.reshape(3 * nf, 3 * K * ns)


def _contract(what, x, tv, nrm, eps, dens, order):
    nf, ns, K = x.shape[0], tv.shape[0], NODES[order]
    out = torch.zeros((nf, 3 if what == "disp" else 6), dtype=torch.float64, device=x.device)
    A2, dens = _areas2(tv), dens.reshape(ns, K, 3)
    for rows in _rows(nf, ns):
        for f, s, lam, w in _by_class(x, tv, eps, rows):
            d = x[f][:, None, :] - torch.einsum("qv,pvc->pqc", lam, tv[s])
            u = torch.einsum("qk,pkc->pqc", _shapes(lam, order), dens[s])
            if what == "disp":
                v = torch.einsum("pqij,pqj->pqi", _point_block("T", d, nrm[s], eps[s] ** 2), u)
            else:
                v = _point_stress(d, u, nrm[s], eps[s] ** 2)
            out.index_add_(0, f, torch.einsum("q,pqc->pc", w, v) * A2[s][:, None])
    return out if what == "disp" else out[:, _FULL].reshape(nf, 3, 3)


def _traction(x, nx, tv, nrm, eps):
    nf, ns = x.shape[0], tv.shape[0]
    out = torch.zeros((nf, 3, ns, 3), dtype=torch.float64, device=x.device)
    A2 = _areas2(tv)
    for rows in _rows(nf, ns):
        for f, s, lam, w in _by_class(x, tv, eps, rows):
            d = x[f][:, None, :] - torch.einsum("qv,pvc->pqc", lam, tv[s])
            for j in range(3):
                u = torch.zeros_like(d)
                u[..., j] = 1.0
                sg = torch.einsum("q,pqc->pc", w, _point_stress(d, u, nrm[s], eps[s] ** 2)) * A2[s][:, None]
                out[f, :, s, j] = torch.einsum("pic,pc->pi", sg[:, _FULL].reshape(-1, 3, 3), nx[f])
    return out.reshape(3 * nf, 3 * ns)


def _system(case, seed, slips=None):
    """The calibrated system of the model and its deflated solution(s): (A, b, u)."""
    rng = np.random.default_rng(seed)
    model, eps, _, slip = _model(case, rng)
    cube, fault = model.regions[0].patches[0].mesh, model.regions[0].faults[0].mesh
    tv, nrm, ftv, fn = _cuda(cube.tri_verts(), cube.normals_and_areas()[0], fault.tri_verts(),
                             fault.normals_and_areas()[0])
    x, n = tv.mean(1), tv.shape[0]
    e = torch.full((n,), eps, dtype=torch.float64, device=x.device)
    ef = e[:1].expand(ftv.shape[0]).contiguous()
    A = _matrix("T", x, tv, nrm, e, 0)
    C = -A.view(n, 3, n, 3).sum(2)
    i = torch.arange(n, device=x.device)
    A.view(n, 3, n, 3)[i, :, i, :] += C
    d = _cuda(slip)[0].expand(ftv.shape[0], 3).contiguous()
    b = _contract("disp", x, ftv, fn, ef, d, 0).reshape(-1)     # scale -sigma of a fault: +1
    P = torch.zeros((3 * n, 3), dtype=torch.float64, device=x.device)
    for k in range(3):
        P[k::3, k] = n ** -0.5
    S = torch.cat([torch.cat([A, P], 1), torch.cat([P.T, torch.zeros_like(P[:3])], 1)])
    u = torch.linalg.solve(S, torch.cat([b, b.new_zeros(3)]))[:3 * n].reshape(n, 3)
    return A, b, u


def exact(case, seed):
    kind, order = case["kind"], case.get("order", 0)
    if kind == "solve":
        if case["n_face"] > 20:                 # a dense solve in 64 bits of over 15,000 unknowns takes too long
            return None
        A, b, u = _system(case, seed)
        return {"u": u, "b": b} if case["precision"] == "mixed" else {"u": u, "b": b, "A": A}
    if kind == "block":                         # the operator it is given is the mixed one, to 1e-7
        return None
    st = prepare(case, seed)
    if kind == "grid":
        region = st["model"].regions[0]
        cube, fault = region.patches[0].mesh, region.faults[0].mesh
        tot = 0.0
        for mesh, dens, sign in ((cube, st["solution"]["u:cube"], -1.0),
                                 (fault, region.faults[0].value_array(), 1.0)):
            tv, nrm, d = _cuda(mesh.tri_verts(), mesh.normals_and_areas()[0], np.asarray(dens, float))
            e = torch.full((tv.shape[0],), st["eps"], dtype=torch.float64, device=tv.device)
            tot = tot + sign * _contract("stress", st["points"], tv, nrm, e, d, 0)
        return tot
    x, tv, nrm, eps = st["x"], st["tv"], st["n"], st["eps"]
    if kind == "matrix":
        return _matrix(case["kernel"], x, tv, nrm, eps, order)
    if kind == "traction":
        return _traction(x, st["nx"], tv, nrm, eps)
    return _contract("disp" if kind == "disp" else "stress", x, tv, nrm, eps, st["d"], order)
