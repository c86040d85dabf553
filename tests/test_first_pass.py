"""What a solve sets up on its first pass over a pattern: the rows of the
pattern at the edge of the two kernels that build them, and the multicolour
order of the fronts against the sequential first fit written out in Python
(through the ILU(0) it gives, applied in numpy)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import _lib
from getdp_gb300 import generate as G
from getdp_gb300 import linalg as LA
from getdp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _fan(k, formulation):
    """k triangles around node 0, which so has 3 k (complex: 6 k) candidates."""
    t = 2 * np.pi * np.arange(k) / k
    nodes = np.zeros((k + 1, 3))
    nodes[1:, 0], nodes[1:, 1] = np.cos(t), np.sin(t)
    ring = np.arange(k)
    elems = np.stack([np.zeros(k), 1 + ring, 1 + (ring + 1) % k], 1).astype(np.int32)
    m = W.Mesh(nodes, W.TRI3, elems, np.ones(k, np.int32), "line2", np.zeros((0, 2), np.int32),
               np.zeros(0, np.int32))
    params = {"sigma": np.where(np.arange(k) % 2, 3.0, 0.0), "freq": 50.0}
    return W.Problem("fan", m, formulation, np.ones(k), np.ones(k), params)


# the warps' kernel takes up to 64 candidates: 21 triangles, 10 complex ones
@pytest.mark.parametrize("formulation,k", [("magnetostatics2d", 3), ("magnetostatics2d", 10),
                                           ("magnetostatics2d", 11), ("magnetostatics2d", 21),
                                           ("magnetostatics2d", 22), ("eddy2d", 5),
                                           ("eddy2d", 10), ("eddy2d", 11)])
def test_pattern_rows(formulation, k):
    p = _fan(k, formulation)
    dm = W.dofmap_for(p)
    terms = G.DeviceTerms(p, dm)
    A, b = LA.gMatrix(dm.n_dof), LA.gVector(dm.n_dof)
    G.generate(A, b, terms.batch)
    ref = set()
    for e, d in enumerate(dm.elem_dofs):
        for i in d:
            for j in d:
                if formulation == "magnetostatics2d":
                    ref.add((i, j))
                    continue
                for h in range(2):
                    ref.add((i + h, j + h))
                    if p.params["sigma"][e]:
                        ref.add((i + h, j + 1 - h))
    ip, ix, _ = A.csr()
    rows = np.repeat(np.arange(dm.n_dof), np.diff(ip))
    assert list(zip(rows.tolist(), ix.tolist())) == sorted((int(i), int(j)) for i, j in ref)


def _patterns(name, rng):
    if name == "random":
        S = sp.random(300, 300, 0.02, random_state=3)
    elif name == "clique":  # more colours than the 64 of one window
        S = sp.block_diag([np.ones((70, 70)), sp.diags([np.ones(29)], [1])])
    elif name == "star":
        S = sp.lil_matrix((200, 200))
        S[100, :] = 1.0
    else:  # isolated vertices among pairs
        S = sp.lil_matrix((97, 97))
        for i in range(0, 90, 3):
            S[i, i + 1] = 1.0
    S = sp.csr_matrix(S)
    S = ((S + S.T) != 0).astype(float).tolil()
    S.setdiag(1.0)
    S = S.tocsr()
    S.data = rng.uniform(-1.0, 1.0, S.nnz)
    A = S + sp.diags(2.0 + np.asarray(abs(S).sum(axis=1)).ravel())
    A = A.tocsr()
    A.sort_indices()
    return A


@pytest.mark.parametrize("name", ["random", "clique", "star", "pairs"])
def test_fronts_are_first_fit_from_the_last_row(name):
    rng = np.random.default_rng(4)
    A = _patterns(name, rng)
    n = A.shape[0]
    colour = np.full(n, -1)
    for i in range(n - 1, -1, -1):
        used = {colour[j] for j in A.indices[A.indptr[i]:A.indptr[i + 1]] if j > i}
        colour[i] = next(c for c in range(n) if c not in used)
    order = np.argsort(colour, kind="stable")  # old row of each new row
    B = A.toarray()[np.ix_(order, order)]
    P = B != 0
    for i in range(1, n):
        for k in range(i):
            if P[i, k]:
                B[i, k] /= B[k, k]
                m = P[i, k + 1:]
                B[i, k + 1:][m] -= B[i, k] * B[k, k + 1:][m]
    v = rng.standard_normal(n)
    y = np.linalg.solve(np.tril(B, -1) + np.eye(n), v[order])
    z = np.empty(n)
    z[order] = np.linalg.solve(np.triu(B), y)
    M, vin, out = LA.gMatrix(n), LA.gVector(n), LA.gVector(n)
    M.set_csr(A.indptr, A.indices, A.data)
    vin.set(v)
    S = LA.LinAlg_CreateSolver(None)
    S.set("Preconditioner", 6)
    S.set("Renumbering_Technique", 1)
    _lib.check(_lib.load().gb300_precond_apply(M.h, ctypes.byref(S.params), vin.h, out.h))
    # dominant rows (|a_ii| > 2 + sum |a_ij|): factors and sweeps are
    # contractions, errors a few hundred roundings at most
    assert np.max(np.abs(out.numpy() - z)) <= 1000 * 1.2e-16 * np.max(np.abs(z)) * 10
