"""The second Gram-Schmidt pass, on systems that take it in most steps of the
first dozen: eight eigenvalues far above the others.  Their part of a product is
most of it and lies in the span of the basis, so one pass leaves an error of some
eps 10^p in the new vector and the basis loses its orthogonality step by step (in
numpy a single pass stagnates at 10^8).  The reference is one cycle written out in
numpy, with the pass repeated when the first removed more than 98 % of the square.

The true residual may exceed the estimate by what forming x from the basis loses:
eps ||A|| ||x||, and ||x|| is about ||b|| here."""
import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu

M = 60


def _cycle(d, b, rtol, keep):
    """One cycle of GMRES on diag(d): its steps (the first residual counts) and
    the true residual of its solution over ||b||."""
    V, H, g = [b / np.linalg.norm(b)], np.zeros((M + 1, M)), np.zeros(M + 1)
    cs, sn = np.zeros(M), np.zeros(M)
    g[0] = np.linalg.norm(b)
    tol = rtol * g[0]
    for k in range(M):
        Q, w = np.array(V), d * V[-1]
        before = w @ w
        h = Q @ w
        w = w - Q.T @ h
        if w @ w < keep * before:
            h2 = Q @ w
            w, h = w - Q.T @ h2, h + h2
        norm = np.linalg.norm(w)
        V.append(w / norm)
        H[:k + 1, k], H[k + 1, k] = h, norm
        for i in range(k):
            a, c = H[i, k], H[i + 1, k]
            H[i, k], H[i + 1, k] = cs[i] * a + sn[i] * c, cs[i] * c - sn[i] * a
        r = np.hypot(H[k, k], norm)
        cs[k], sn[k] = H[k, k] / r, norm / r
        H[k, k], H[k + 1, k] = r, 0.0
        g[k + 1], g[k] = -sn[k] * g[k], cs[k] * g[k]
        if abs(g[k + 1]) <= tol:
            break
    y = np.linalg.solve(np.triu(H[:k + 1, :k + 1]), g[:k + 1])
    x = np.array(V[:k + 1]).T @ y
    return k + 2, np.linalg.norm(b - d * x) / np.linalg.norm(b)


@pytest.mark.parametrize("p,rtol", [(4, 1e-10), (6, 1e-8), (8, 1e-8)])
@pytest.mark.parametrize("form", ["gmres", "fgmres", "cluster", "per-kernel"])
def test_steps_and_residual(form, p, rtol):
    d = np.concatenate([np.logspace(p, p + 1, 8), np.linspace(1, 2, 1592)])
    n = len(d)
    bh = np.random.default_rng(0).standard_normal(n)
    two, res = _cycle(d, bh, rtol, 0.02)
    attainable = 1.1e-16 * 10.0 ** (p + 1)
    assert res <= 1.1 * rtol + attainable
    batch = form in ("cluster", "per-kernel")
    D = sp.diags(np.tile(d, 2) if batch else d).tocsr()
    A, b, x = LA.gMatrix(D.shape[0]), LA.gVector(D.shape[0]), LA.gVector(D.shape[0])
    A.set_csr(D.indptr, D.indices, D.data)
    b.set(np.tile(bh, 2) if batch else bh)
    S = LA.LinAlg_CreateSolver(None)
    for k, v in dict(Algorithm=9 if form == "fgmres" else 8, Preconditioner=0, Krylov_Size=M,
                     Nb_Iter_Max=M, Batch_Kernel=0 if form == "per-kernel" else 4).items():
        S.set(k, v)
    S["stopping_test"] = rtol
    infos = (LA.LinAlg_SolveBatch(A, b, S, x, [0, n, 2 * n]) if batch else
             [LA.LinAlg_Solve(A, b, S, x)])
    for info in infos:
        assert info["status"] == 0 and abs(info["iterations"] - two) <= 2, (info, two)
        assert info["true_residual"] <= (1.1 * rtol + attainable) * info["rhs_norm"], info
