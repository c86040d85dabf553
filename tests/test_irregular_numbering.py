"""The multicolour order of meshes numbered at random, where rounds over all
vertices do the colouring or its first part: the same sequential first fit, from
the last vertex to the first, as in any other numbering.  Checked through the
ILU(0) it gives, written out in Python: dominant rows, so factor and sweeps are
contractions and the difference is some roundings of a few terms a row (the
bound is the one of the fronts' test)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import _lib
from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


def _grid(m):
    T = sp.diags([np.ones(m - 1)] * 2, [-1, 1])
    return sp.kron(sp.identity(m), T) + sp.kron(T, sp.identity(m))


def _first_fit(S):
    """Colours of S's rows (a symmetric pattern with its diagonal)."""
    n = S.shape[0]
    colour = [-1] * n
    ip, ix = S.indptr.tolist(), S.indices.tolist()
    for i in range(n - 1, -1, -1):
        used = {colour[j] for j in ix[ip[i]:ip[i + 1]] if j > i}
        c = 0
        while c in used:
            c += 1
        colour[i] = c
    return np.array(colour)


def _ilu0_solve(B, v):
    B = B.tocsr()
    B.sort_indices()
    ip, ix, n = B.indptr.tolist(), B.indices.tolist(), B.shape[0]
    rows = [dict(zip(ix[ip[i]:ip[i + 1]], B.data[ip[i]:ip[i + 1]].tolist())) for i in range(n)]
    y = v.tolist()
    for i in range(n):
        r = rows[i]
        for k in ix[ip[i]:ip[i + 1]]:
            if k >= i:
                break
            r[k] /= rows[k][k]
            for j, u in rows[k].items():
                if j > k and j in r:
                    r[j] -= r[k] * u
            y[i] -= r[k] * y[k]
    for i in range(n - 1, -1, -1):
        for j, u in rows[i].items():
            if j > i:
                y[i] -= u * y[j]
        y[i] /= rows[i][i]
    return np.array(y)


def _vertices(name, rng):
    if name.startswith("grid"):
        S = _grid(int(name[4:]))
        p = rng.permutation(S.shape[0])
        return S.tocsr()[p][:, p]
    # most of it at random, and a path in order that 32 rounds do not reach the
    # end of: the fronts colour what the rounds leave
    S = _grid(182).tocsr()
    p = rng.permutation(S.shape[0])
    path = sp.diags([np.ones(2999)] * 2, [-1, 1])
    return sp.block_diag([S[p][:, p], path]).tocsr()


# 32,761 vertices take the fronts alone, 33,124 the rounds
@pytest.mark.parametrize("name,bs", [("grid181", 1), ("grid182", 1), ("mixed", 1), ("mixed", 2)])
def test_random_numbering(name, bs):
    rng = np.random.default_rng(len(name) + bs)
    S = _vertices(name, rng)
    S = (S + sp.identity(S.shape[0])).tocsr()
    S.sort_indices()
    colour = _first_fit(S)
    order = np.argsort(colour, kind="stable")
    nv = S.shape[0]
    n = nv * bs
    M = LA.gMatrix(n)
    C = S.tocoo()
    if bs == 1:
        A = S.copy()
        A.data = rng.uniform(-1.0, 1.0, A.nnz)
        A = (A + sp.diags(2.0 + np.asarray(abs(A).sum(axis=1)).ravel())).tocsr()
        A.sort_indices()
        M.set_csr(A.indptr, A.indices, A.data)
    else:  # complex entries: pairs of rows (2 m, 2 m + 1)
        re, im = rng.uniform(-1.0, 1.0, C.nnz), rng.uniform(-1.0, 1.0, C.nnz)
        re[C.row == C.col] += 14.0
        i, j = 2 * C.row, 2 * C.col
        LA.LinAlg_AddComplexInMatrix(re[0], im[0], M, int(i[0]), int(j[0]), int(i[0]) + 1,
                                     int(j[0]) + 1)
        LA.LinAlg_AddComplexInMatrix(0.0, 0.0, M, 0, 0, 1, 1)
        rows = np.concatenate([i[1:], i[1:] + 1, i[1:], i[1:] + 1])
        cols = np.concatenate([j[1:], j[1:] + 1, j[1:] + 1, j[1:]])
        M.add_coo(rows, cols, np.concatenate([re[1:], re[1:], -im[1:], im[1:]]))
        ip, ix, dv = M.csr()
        A = sp.csr_matrix((dv, ix, ip), shape=(n, n))
        order = (order[:, None] * 2 + np.arange(2)).ravel()
    v = rng.standard_normal(n)
    z = np.empty(n)
    z[order] = _ilu0_solve(A[order][:, order], v[order])
    vin, out = LA.gVector(n), LA.gVector(n)
    vin.set(v)
    P = LA.LinAlg_CreateSolver(None)
    P.set("Preconditioner", 6)
    P.set("Renumbering_Technique", 1)
    _lib.check(_lib.load().gb300_precond_apply(M.h, ctypes.byref(P.params), vin.h, out.h))
    assert np.max(np.abs(out.numpy() - z)) <= 1e4 * 1.2e-16 * np.max(np.abs(z))
