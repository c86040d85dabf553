"""The two-level cycle at sizes on both sides of the line (131,072 rows) where
its kernels stop starting early and the prolongation leaves the residual's
kernel: one application against the cycle written out in numpy around the GPU's
own smoother, in GetDP's order and the multicolour order, with and without a
correction in the first and in the second smoothing.

The smoother's applications are the same numbers on both sides.  What differs is
the coarse matrix (fixed point, 2^-51 of max|a| a term), its inverse (an
elimination of 400 rows) and the rounding of residuals and sums; cond(Ac) is
below 300 here, so some 300 * 400 * 1e-16, asserted with a factor of ten."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import _lib
from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[361, 363])
def system(request):
    m = request.param
    rng = np.random.default_rng(m)
    T = sp.diags([np.ones(m - 1)], [1], shape=(m, m))
    U = (sp.kron(sp.identity(m), T) + sp.kron(T, sp.identity(m))).tocsr()
    U.data = -rng.uniform(0.5, 1.0, U.nnz)
    S = U + U.T
    A = (S + sp.diags(0.05 + np.asarray(abs(S).sum(axis=1)).ravel())).tocsr()
    A.sort_indices()
    n, side = m * m, 20
    i = np.arange(n)
    agg = (i // m) * side // m * side + (i % m) * side // m
    nc = side * side
    P = sp.csr_matrix((np.ones(n), (i, agg)), shape=(n, nc))
    Ac = (P.T @ A @ P).toarray()
    assert np.linalg.cond(Ac) < 300
    G = LA.gMatrix(n)
    G.set_csr(A.indptr, A.indices, A.data)
    G.set_aggregates(agg, nc)
    g = 0.02 * rng.standard_normal(A.nnz)
    _lib.check(_lib.load().gb300_matrix_set_correction(
        G.h, g.ctypes.data_as(ctypes.c_void_p), 0))
    return G, A, P, np.linalg.inv(Ac)


# smoothers before and after the coarse step: 6 ILU(0), 20 with the correction
@pytest.mark.parametrize("renumbering", [0, 1])
@pytest.mark.parametrize("prec,pre,post", [(21, 6, 6), (22, 20, 20), (23, 20, 6)])
def test_cycle(system, prec, pre, post, renumbering):
    G, A, P, Aci = system

    def apply(pc, v):
        S = LA.LinAlg_CreateSolver(None)
        S.set("Preconditioner", pc)
        S.set("Renumbering_Technique", renumbering)
        x, z = LA.gVector(G.n), LA.gVector(G.n)
        x.set(v)
        _lib.check(_lib.load().gb300_precond_apply(G.h, ctypes.byref(S.params), x.h, z.h))
        return z.numpy()

    v = np.random.default_rng(prec).standard_normal(G.n)
    z = apply(pre, v)
    z = z + P @ (Aci @ (P.T @ (v - A @ z)))
    z = z + apply(post, v - A @ z)
    got = apply(prec, v)
    assert np.linalg.norm(got - z) <= 10 * 300 * 400 * 1e-16 * np.linalg.norm(z)
