"""The work a program gives this backend, as cases to be timed.

Every case goes through the package's public entry points (the LinAlg layer,
the batched Generate hook, post-processing, the learned correction) as a
resolution's ``Operation { Generate[A]; Solve[A]; ... }`` does, on the seeded
problems of ``getdp_gb300.workloads`` with the sizes of the repository's own
configurations, tests and benchmark.  What a program keeps between calls (the
element tables on the device, A, b, x, the solver's parameters, a pinned
buffer for the result) is made by ``prepare``; what it asks for on each call
is in ``run``.

Iterative solves stop at a residual small enough that the solution itself,
not the path of the iteration, is what two runs have in common; the edge
problem stops at its configuration's 1e-8, since the nearly singular operator
lets no residual fall below some 4e-9, and the mixed elasticity solves at 1e-9,
ten times above where their FP32 inner iteration stalls.
"""
from __future__ import annotations

import ctypes
import dataclasses
import functools
import math
import os

import numpy as np
import torch

from getdp_gb300 import _lib
from getdp_gb300 import generate as G
from getdp_gb300 import learned as LR
from getdp_gb300 import linalg as LA
from getdp_gb300 import post as P
from getdp_gb300 import workloads as W

_WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(LR.__file__)), "weights",
                        "mpnn_nl2d_256_twolevel.npy")


def listed():
    return [
        # a template-sized 2D magnetostatic problem (Generate + ILU(0)-GMRES):
        # every launch and host step counts
        {"name": "magnet_24", "kind": "magnet", "n": 24, "tol": 1e-12},
        # configuration 1: 2D P1 magnetostatics, 65,025 unknowns
        {"name": "magnet_256", "kind": "magnet", "n": 256, "tol": 1e-12},
        # an unchanged program's path: scalar entries in element order, merged
        # by AssembleMatrix, then the product GetResidual needs
        {"name": "entries_300", "kind": "entries", "n": 300},
        # 3D P2 elasticity, small and odd, plain FP64 CG
        {"name": "elastic_11_f64", "kind": "elastic", "n": 11, "precision": 0, "tol": 1e-11},
        # the same, mid-sized, mixed precision
        {"name": "elastic_24_mixed", "kind": "elastic", "n": 24, "precision": 1, "tol": 1e-9},
        # configuration 2: 48^3 cells, 2.7 M unknowns, 229 M entries, mixed
        {"name": "elastic_48_mixed", "kind": "elastic", "n": 48, "precision": 1, "tol": 1e-9},
        # configuration 3: 3D edge elements, FGMRES with the FP32 factor, the
        # flux density on every element
        {"name": "curlcurl_40", "kind": "curlcurl", "n": 40, "precision": 1, "tol": 1e-8},
        # configuration 4: a sweep of complex eddy-current problems of uneven
        # size and frequency, one Generate and one batched solve
        {"name": "sweep_64", "kind": "sweep", "problems": 64, "n_min": 32, "n_max": 160,
         "tol": 1e-12},
        # configuration 5: one Newton step at 1 M unknowns with the two-level
        # preconditioner
        {"name": "newton_1024", "kind": "newton", "n": 1024, "cells": 32, "tol": 1e-12},
        # a trial of the relaxation: Generate at a state, then GetResidual
        {"name": "residual_513", "kind": "residual", "n": 513},
        # a Newton step's solve with the learned correction in the cycle
        {"name": "learned_256", "kind": "learned", "n": 256, "cells": 32, "tol": 1e-11},
        # training of that correction: one system's loss and gradient
        {"name": "train_129", "kind": "train", "n": 129},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["magnet", "magnet", "entries", "elastic", "elastic", "curlcurl", "sweep",
                       "newton", "residual", "learned", "train"])
    if kind == "magnet":
        return {"kind": kind, "n": log_int(24, 400), "tol": 1e-12}
    if kind == "elastic":
        prec = rng.choice([0, 1])
        return {"kind": kind, "n": log_int(5, 24 if prec == 0 else 44), "precision": prec,
                "tol": 1e-11 if prec == 0 else 1e-9}
    if kind == "curlcurl":
        return {"kind": kind, "n": log_int(8, 40), "precision": rng.choice([0, 1]),
                "tol": 1e-8}
    if kind == "sweep":
        lo = rng.randint(12, 48)
        return {"kind": kind, "problems": log_int(4, 48), "n_min": lo,
                "n_max": lo + rng.randint(16, 110), "tol": 1e-12}
    if kind == "newton":
        n = log_int(160, 1024)
        return {"kind": kind, "n": n, "cells": rng.randint(16, min(n // 8, 40)), "tol": 1e-12}
    if kind == "learned":
        n = log_int(128, 320)
        return {"kind": kind, "n": n, "cells": rng.randint(12, n // 8), "tol": 1e-11}
    return {"kind": kind, "n": {"entries": log_int(30, 400), "residual": log_int(40, 1024),
                                "train": log_int(32, 256)}[kind]}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

class _HostMemory:
    """Page-locked host memory, freed when the last array on it goes."""

    def __init__(self, n: int):
        self.h = ctypes.c_void_p()
        _lib.check(_lib.load().gb300_host_alloc(8 * n, ctypes.byref(self.h)))

    def __del__(self):
        try:
            _lib.load().gb300_host_free(self.h)
        except Exception:
            pass


class Pinned:
    """A page-locked array the results are read into."""

    def __init__(self, n: int):
        m = _HostMemory(n)
        buf = (ctypes.c_double * n).from_address(m.h.value)
        buf.owner = m  # the array keeps buf, and buf the memory
        self.a = np.frombuffer(buf, np.float64)

    def read(self, v: LA.gVector) -> np.ndarray:
        _lib.check(_lib.load().gb300_vector_get(v.h, self.a.ctypes.data_as(ctypes.c_void_p)))
        return self.a


@functools.lru_cache(maxsize=3)
def _cube(kind: str, n: int):
    """The 3D meshes do not depend on the seed, only the materials do."""
    p = W.elasticity_p2(n) if kind == "elastic" else W.curlcurl_edge(n)
    return p, W.dofmap_for(p)


def _problem(c, seed):
    k = c["kind"]
    if k in ("magnet", "entries"):
        p = W.magnetostatics_2d(c["n"], seed=seed % 100003)
        return p, W.dofmap_for(p)
    if k in ("newton", "residual", "learned", "train"):
        p = W.nonlinear_2d(c["n"], seed=seed % 100003)
        return p, W.dofmap_for(p)
    p, dm = _cube(k, c["n"])
    rng = np.random.default_rng(seed)
    if k == "elastic":  # lognormal E, as the generator draws it
        coef = 200.0e9 * np.exp(0.5 * rng.standard_normal(len(p.coef)))
        return dataclasses.replace(p, coef=coef), dm
    # materials and coil current vary from problem to problem
    mu_r = math.exp(rng.uniform(math.log(200.0), math.log(1000.0)))
    coef = np.where(p.mesh.region == 2, 1.0 / (mu_r * W.MU0), 1.0 / W.MU0)
    return dataclasses.replace(p, coef=coef, source=p.source * rng.uniform(0.5, 2.0)), dm


def _sweep(c, seed):
    # the meshes' sizes belong to the case; their nodes, conductors and
    # frequencies to the seed
    rng = np.random.default_rng(c["problems"])
    sizes = rng.integers(c["n_min"], c["n_max"] + 1, size=c["problems"])
    return [W.eddy_2d(int(n), seed=int(seed % 100003) * 1009 + k) for k, n in enumerate(sizes)]


def _unknown_nodes(p, dm):
    node = np.empty(dm.n_dof, np.int64)
    m = dm.elem_dofs >= 0
    node[dm.elem_dofs[m]] = p.mesh.elems[m]
    return p.mesh.nodes[node]


def _state(p, dm, seed):
    """A Newton iterate: a smooth a_z whose flux density reaches 1-2 T, where
    the saturating law is far from linear."""
    xy = _unknown_nodes(p, dm)
    rng = np.random.default_rng(seed + 17)
    amp, ph = rng.uniform(0.2, 0.4), rng.uniform(0.0, 6.0)
    return amp * np.sin(np.pi * xy[:, 0]) * np.sin(np.pi * xy[:, 1]) * \
        (1.0 + 0.3 * np.sin(9.0 * xy[:, 0] + 5.0 * xy[:, 1] + ph))


def _triplets(p, dm):
    """Element matrices as a program adds them entry by entry (order of
    GetDP's loop: element, row, column), fixed unknowns left out."""
    x = p.mesh.nodes[p.mesh.elems][:, :, :2]
    g, area = _p1(x)
    ke = np.einsum("eac,ebc->eab", g, g) * (p.coef * area)[:, None, None]
    d = dm.elem_dofs.astype(np.int64)
    i = np.broadcast_to(d[:, :, None], ke.shape)
    j = np.broadcast_to(d[:, None, :], ke.shape)
    m = (i >= 0) & (j >= 0)
    return i[m].astype(np.int32), j[m].astype(np.int32), ke[m]


def _solver(alg, prec, krylov, c, n_iter=20000):
    S = LA.LinAlg_CreateSolver(None)
    for k, v in (("Algorithm", alg), ("Preconditioner", prec), ("Krylov_Size", krylov),
                 ("Renumbering_Technique", 1), ("Nb_Iter_Max", n_iter),
                 ("Precision", c.get("precision", 0))):
        S.set(k, v)
    S["stopping_test"] = c["tol"]
    return S


def prepare(case, seed):
    c, k = dict(case), case["kind"]
    s = {"case": c}
    if k == "sweep":
        bt = W.concat_problems(_sweep(c, seed))
        p, dm = bt.problem, bt.dofmap
        s["offsets"] = bt.offsets
    else:
        p, dm = _problem(c, seed)
    n = dm.n_dof
    s["A"] = LA.gMatrix(n)
    s["out"] = Pinned(n)
    if k == "entries":
        s["ijv"] = _triplets(p, dm)
        s["v"], s["y"] = LA.gVector(n), LA.gVector(n)
        s["v"].set(np.random.default_rng(seed).standard_normal(n))
        return s
    s["terms"] = G.DeviceTerms(p, dm)
    s["b"], s["x"] = LA.gVector(n), LA.gVector(n)
    if k == "magnet":
        s["S"] = _solver(8, 6, 50, c)
    elif k == "elastic":
        s["S"] = _solver(1, 0, 50, c, 200000)
        s["S"].set("Scaling", 1)
    elif k == "curlcurl":
        s["S"] = _solver(9, 6, 40, c)
    elif k == "sweep":
        s["S"] = _solver(8, 6, 40, c)
    else:  # the Newton loop's calls: a state, the pattern of the first Generate
        s["state"] = LA.gVector(n)
        s["state"].set(_state(p, dm, seed))
        G.generate(s["A"], s["b"], s["terms"].batch, pattern=True, solution=s["state"])
        if k in ("newton", "learned"):
            s["A"].set_aggregates(*W.cell_aggregates(p, dm, c["cells"]))
        if k == "newton":
            s["S"] = _solver(8, 21, 50, c)
        elif k == "learned":
            s["S"] = _solver(9, 22, 50, {**c, "precision": 1})
        if k in ("learned", "train"):
            s["net"] = LR.MPNN(seed=1)
            s["net"].set_params(np.load(_WEIGHTS))
        if k == "train":  # r1 = A e1, as the training samples have it
            s["e1"], s["r1"] = LA.gVector(n), LA.gVector(n)
            s["e1"].set(np.random.default_rng(seed + 5).standard_normal(n))
            LA.LinAlg_ProdMatrixVector(s["A"], s["e1"], s["r1"])
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def _converged(info):
    if info["status"] != 0:
        raise RuntimeError(f"solve: status {info['status']} after {info['iterations']} steps, "
                           f"residual {info['true_residual'] / info['rhs_norm']:.3e}")


def run(s):
    k, A = s["case"]["kind"], s["A"]
    if k == "entries":
        _lib.check(_lib.load().gb300_matrix_reset(A.h))  # ZeroMatrix of a Generate
        A.add_coo(*s["ijv"])
        LA.LinAlg_AssembleMatrix(A)
        LA.LinAlg_ProdMatrixVector(A, s["v"], s["y"])
        return s["out"].read(s["y"])
    if k == "train":
        loss, grad = s["net"].loss_grad(A, s["r1"], s["e1"], want_grad=True)
        return {"loss": np.float32(loss), "grad": grad}
    b, x, batch = s["b"], s["x"], s["terms"].batch
    if k == "residual":
        G.generate(A, b, batch, pattern=False, solution=s["state"])
        norm = ctypes.c_double()
        _lib.check(_lib.load().gb300_residual_noalloc(A.h, s["state"].h, b.h, x.h,
                                                      ctypes.byref(norm)))
        return {"r": s["out"].read(x), "norm": norm.value}
    if k == "sweep":
        G.generate(A, b, batch)
        for info in LA.LinAlg_SolveBatch(A, b, s["S"], x, s["offsets"]):
            _converged(info)
        return s["out"].read(x)
    if k in ("newton", "learned"):
        G.generate(A, b, batch, pattern=False, solution=s["state"])
        if k == "learned":
            s["net"].infer(A)
    else:
        G.generate(A, b, batch)
    _converged(LA.LinAlg_Solve(A, b, s["S"], x))
    if k == "curlcurl":
        # the vector potential is unique up to a gradient the 1e-6 mass term
        # barely weighs; the flux density is the result
        return P.curl_on_elements(batch, x)
    return s["out"].read(x)


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _krylov(n, nnz, steps, value=8, sweeps=1, basis=25, flexible=False):
    """Per step: the matrix and `sweeps` factors once, half a restart's basis
    read for the projections, a handful of vectors."""
    nbytes = steps * (nnz * (8 + 4) + sweeps * nnz * (value + 4) + 8 * n * (2 * basis + 6))
    flops = steps * (2 * nnz + 2 * sweeps * nnz + 4 * basis * n)
    return nbytes, flops


def work(case):
    k, n = case["kind"], case.get("n", 0)
    if k == "sweep":
        b = f = 0.0
        mid = 0.5 * (case["n_min"] + case["n_max"])
        nd = 2 * (mid - 1) ** 2
        kb, kf = _krylov(nd, 9 * nd, 3.6 * mid, basis=20)
        el = 2 * mid * mid
        b = case["problems"] * (kb + el * 100 + 9 * nd * 12)
        f = case["problems"] * (kf + el * 300)
        return {"bytes": b, "flops": f}
    if k == "elastic":
        ne, nodes = 6 * n ** 3, 8.0 * n ** 3 + 3.0 * n * n
        blocks = 28.2 * nodes
        steps = 70 * n
        val = 4 if case["precision"] else 8
        per = blocks * (9 * val + 4) + 14 * 3 * nodes * val
        return {"bytes": steps * per + ne * 160 + blocks * 9 * 12,
                "flops": steps * (18 * blocks + 10 * 3 * nodes) + ne * 10970}
    if k == "curlcurl":
        ne, nd = 6 * n ** 3, 7.0 * n ** 3 - 9.0 * n * n
        kb, kf = _krylov(nd, 15.5 * nd, 10 * n, 4 if case["precision"] else 8, basis=20)
        return {"bytes": kb + ne * 190 + 16 * nd * 12 + 24 * ne, "flops": kf + ne * 900}
    nd, ne = (n - 1.0) ** 2, 2.0 * n * n
    gen_b, gen_f = ne * 56 + 7 * nd * 12 + 8 * nd, ne * 150
    if k == "entries":
        return {"bytes": 9 * ne * 16 + 7 * nd * 12 * 2 + 16 * nd, "flops": 9 * ne + 14 * nd}
    if k == "residual":
        return {"bytes": gen_b + 7 * nd * 12 + 24 * nd, "flops": gen_f + 16 * nd}
    if k == "train":  # three layers of width 32, forward and backward
        return {"bytes": nd * 32 * 4 * 24 + 7 * nd * 12 * 4,
                "flops": 3 * 3 * 2 * nd * 64 * 32 + 6 * 7 * nd * 64}
    if k == "magnet":
        kb, kf = _krylov(nd, 7 * nd, 3 * n)
    else:  # two smoothings and two residuals per two-level step
        kb, kf = _krylov(nd, 7 * nd, 130 if k == "newton" else 110, 8 if k == "newton" else 4,
                         4 if k == "newton" else 8)
        if k == "learned":
            gen_b += nd * 32 * 4 * 8
            gen_f += 3 * 2 * nd * 64 * 32
    return {"bytes": gen_b + kb, "flops": gen_f + kf}


# --------------------------------------------------------------------------
# the same results in plain 64-bit arithmetic
# --------------------------------------------------------------------------

def _p1(x):
    """Gradients (e, 3, 2) of the barycentric functions and areas."""
    e1, e2 = x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]
    det = e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]
    g1 = np.stack([e2[:, 1], -e2[:, 0]], 1) / det[:, None]
    g2 = np.stack([-e1[:, 1], e1[:, 0]], 1) / det[:, None]
    return np.stack([-g1 - g2, g1, g2], 1), 0.5 * np.abs(det)


class _Elements:
    """sum_e P_e^T K_e P_e as an operator: element matrices (ne, m, m) on
    element -> unknown tables (-1: fixed)."""

    def __init__(self, ke, dofs, n):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n = n
        self.ke = torch.as_tensor(ke, device=dev)
        d = torch.as_tensor(np.ascontiguousarray(dofs), device=dev).long()
        self.m = (d >= 0)
        self.d = torch.where(self.m, d, n)
        self.flat = self.d.reshape(-1)
        self.diag = self.scatter(torch.diagonal(self.ke, dim1=1, dim2=2))

    def scatter(self, fe):
        out = torch.zeros(self.n + 1, dtype=fe.dtype, device=fe.device)
        return out.index_add_(0, self.flat, fe.reshape(-1))[:self.n]

    def __call__(self, x):
        xe = torch.cat([x, x.new_zeros(1)])[self.d]
        return self.scatter(torch.bmm(self.ke, xe.unsqueeze(2)).squeeze(2))

    def solve(self, b, rtol=1e-14, most=60000):
        """Conjugate gradients with the diagonal, without conjugation for a
        complex symmetric operator, restarted on the true residual."""
        x = torch.zeros_like(b)
        inv, left, last = 1.0 / self.diag, most, math.inf
        b0 = float(torch.linalg.vector_norm(b))
        for _ in range(6):
            r = b - self(x)
            now = float(torch.linalg.vector_norm(r))
            if now <= rtol * b0 or now > 0.3 * last or left <= 0:
                break
            last = now
            d = torch.zeros_like(b)
            z = inv * r
            p = z.clone()
            rz = (r * z).sum()
            for it in range(left):
                q = self(p)
                a = rz / (p * q).sum()
                d += a * p
                r -= a * q
                if it % 50 == 49 and float(torch.linalg.vector_norm(r)) <= max(
                        1e-7 * now, 0.3 * rtol * b0):
                    break
                z = inv * r
                new = (r * z).sum()
                p = z + (new / rz) * p
                rz = new
            left -= it + 1
            x = x + d
        return x


def _elastic_exact(c, seed):
    p, dm = _problem(c, seed)
    x = p.mesh.nodes[p.mesh.elems[:, :4]]
    J = np.stack([x[:, 1] - x[:, 0], x[:, 2] - x[:, 0], x[:, 3] - x[:, 0]], 1)
    vol = np.linalg.det(J) / 6.0
    gl = np.linalg.inv(J).transpose(0, 2, 1)  # rows: gradients of l1, l2, l3
    gl = np.concatenate([-gl.sum(1, keepdims=True), gl], 1)  # (e, 4, 3)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gl = torch.as_tensor(gl, device=dev)
    nu = p.params["poisson"]
    E = torch.as_tensor(p.coef, device=dev)
    lam, mu = E * nu / (1 + nu) / (1 - 2 * nu), E / 2 / (1 + nu)
    w = torch.as_tensor(np.abs(vol) / 4.0, device=dev)
    a, bq = 0.5854101966249685, 0.1381966011250105
    ne = len(p.coef)
    ke = torch.zeros((ne, 3, 10, 3, 10), dtype=torch.float64, device=dev)
    fe = torch.zeros((ne, 3, 10), dtype=torch.float64, device=dev)
    edges = W.TET10_EDGES
    for q in range(4):
        l = [a if i == q else bq for i in range(4)]
        g = [(4 * l[i] - 1) * gl[:, i] for i in range(4)]
        g += [4 * (l[i] * gl[:, j] + l[j] * gl[:, i]) for i, j in edges]
        g = torch.stack(g, 1)  # (e, 10, 3)
        shp = [l[i] * (2 * l[i] - 1) for i in range(4)] + [4 * l[i] * l[j] for i, j in edges]
        dot = torch.einsum("eac,ebc->eab", g, g)
        for i in range(3):
            ke[:, i, :, i, :] += (w * mu)[:, None, None] * dot
            for j in range(3):
                gi, gj = g[:, :, i], g[:, :, j]
                ke[:, i, :, j, :] += (w * lam)[:, None, None] * gi[:, :, None] * gj[:, None, :]
                ke[:, i, :, j, :] += (w * mu)[:, None, None] * gj[:, :, None] * gi[:, None, :]
        fe[:, 2] += w[:, None] * torch.as_tensor(shp, device=dev, dtype=torch.float64) * \
            (-p.params["rho"] * p.params["g"])
    op = _Elements(ke.reshape(ne, 30, 30), dm.elem_dofs, dm.n_dof)
    return op.solve(op.scatter(fe.reshape(ne, 30)), 1e-13).cpu().numpy()


_EDGE_ENDS = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))


def _curlcurl_exact(c, seed):
    p, dm = _problem(c, seed)
    x = p.mesh.nodes[p.mesh.elems]
    J = np.stack([x[:, 1] - x[:, 0], x[:, 2] - x[:, 0], x[:, 3] - x[:, 0]], 1)
    vol = np.abs(np.linalg.det(J)) / 6.0
    gl = np.linalg.inv(J).transpose(0, 2, 1)
    gl = np.concatenate([-gl.sum(1, keepdims=True), gl], 1)
    sg = dm.elem_sign.astype(np.float64)
    cu = np.stack([2.0 * np.cross(gl[:, i], gl[:, j]) for i, j in _EDGE_ENDS], 1) * sg[:, :, None]
    ke = np.einsum("eac,ebc->eab", cu, cu) * (p.coef * vol)[:, None, None]
    a, bq = 0.5854101966249685, 0.1381966011250105
    fe = np.zeros((len(vol), 6))
    for q in range(4):
        l = [a if i == q else bq for i in range(4)]
        w = np.stack([l[i] * gl[:, j] - l[j] * gl[:, i] for i, j in _EDGE_ENDS], 1) * sg[:, :, None]
        ke += np.einsum("eac,ebc->eab", w, w) * (p.params["reg"] * p.coef * vol / 4)[:, None, None]
        fe += np.einsum("eac,ec->ea", w, p.source) * (vol / 4)[:, None]
    op = _Elements(ke, dm.elem_dofs, dm.n_dof)
    u = op.solve(op.scatter(torch.as_tensor(fe, device=op.ke.device)), 1e-13).cpu().numpy()
    ue = np.where(dm.elem_dofs >= 0, np.append(u, 0.0)[dm.elem_dofs], 0.0)
    return np.einsum("eac,ea->ec", cu, ue)


def _nu(p, b2):
    return p.coef / (1.0 + p.params["k_sat"] * np.exp(-b2 / p.params["b_sat2"]))


def _flat_exact(c, seed):
    """The 2D kinds: P1 triangles."""
    k = c["kind"]
    p, dm = _problem(c, seed)
    g, area = _p1(p.mesh.nodes[p.mesh.elems][:, :, :2])
    dot = np.einsum("eac,ebc->eab", g, g)
    d = dm.elem_dofs
    fe = np.broadcast_to((p.source * area / 3)[:, None], d.shape)
    if k in ("magnet", "entries"):
        op = _Elements(dot * (p.coef * area)[:, None, None], d, dm.n_dof)
        if k == "entries":
            v = np.random.default_rng(seed).standard_normal(dm.n_dof)
            return op(torch.as_tensor(v, device=op.ke.device)).cpu().numpy()
    else:
        a = np.append(_state(p, dm, seed), 0.0)
        ga = np.einsum("ea,eac->ec", np.where(d >= 0, a[d], 0.0), g)  # |{d a}| = |grad a|
        b2 = (ga * ga).sum(1)
        nu = _nu(p, b2)
        t = p.params["k_sat"] * np.exp(-b2 / p.params["b_sat2"])
        dnu = p.coef * t / p.params["b_sat2"] / (1.0 + t) ** 2
        h = np.einsum("eac,ec->ea", g, ga)
        ke = (nu * area)[:, None, None] * dot + \
            (2.0 * dnu * area)[:, None, None] * h[:, :, None] * h[:, None, :]
        op = _Elements(ke, d, dm.n_dof)
        # rhs of the Newton system: dhdb b - nu b + J
        fe = fe + (2.0 * dnu * b2 * area)[:, None] * h
    b = op.scatter(torch.as_tensor(np.ascontiguousarray(fe), device=op.ke.device))
    if k == "residual":
        r = b - op(torch.as_tensor(a[:-1], device=op.ke.device))
        return {"r": r.cpu().numpy(), "norm": float(torch.linalg.vector_norm(r))}
    return op.solve(b).cpu().numpy()


def _sweep_exact(c, seed):
    bt = W.concat_problems(_sweep(c, seed))
    p, dm = bt.problem, bt.dofmap
    g, area = _p1(p.mesh.nodes[p.mesh.elems][:, :, :2])
    mass = (np.ones((3, 3)) + np.eye(3)) / 12.0
    ke = np.einsum("eac,ebc->eab", g, g) * (p.coef * area)[:, None, None] + 0j
    ke += 1j * (p.params["omega_e"] * p.params["sigma"] * area)[:, None, None] * mass
    d = np.where(dm.elem_dofs >= 0, dm.elem_dofs // 2, -1)
    op = _Elements(ke, d, dm.n_dof // 2)
    fe = np.broadcast_to((p.source * area / 3)[:, None] + 0j, d.shape)
    b = op.scatter(torch.as_tensor(np.ascontiguousarray(fe), device=op.ke.device))
    u = op.solve(b, most=12000).cpu().numpy()
    return np.stack([u.real, u.imag], 1).reshape(-1)


def exact(case, seed):
    k = case["kind"]
    if k == "train":
        return None  # a network's gradient, held to its type's bound
    if k == "elastic":
        return _elastic_exact(dict(case), seed)
    if k == "curlcurl":
        return _curlcurl_exact(dict(case), seed)
    return _sweep_exact(dict(case), seed) if k == "sweep" else _flat_exact(dict(case), seed)
