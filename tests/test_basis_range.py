"""GMRES and FGMRES without a preconditioner on s A, s a power of two: the
basis vectors are kept unnormalised, and still every s that leaves ||A x||^2 in
range has to be solved.  Scaling by a power of two rounds nothing, so the
iteration is the one of A itself: its solution of s A x = s b, step counts within
one (a reciprocal root or a division may round otherwise), solutions to the
residual both stop at
(1e-12, times a condition number of at most 3: see the dominant matrices' file,
and times 1e3 for the graded one)."""
import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


def _dominant(m, seed):
    rng = np.random.default_rng(seed)
    T = sp.diags([np.ones(m - 1), np.ones(m - 1)], [-1, 1])
    S = sp.csr_matrix(sp.kron(sp.identity(m), T) + sp.kron(T, sp.identity(m)))
    S.data = rng.uniform(0.2, 1.0, S.nnz) * rng.choice([-1.0, 1.0], S.nnz)
    S = sp.diags(0.5 / np.asarray(abs(S).sum(axis=1)).ravel()) @ S
    A = (S + sp.identity(m * m)).tocsr()
    A.sort_indices()
    return A


def _graded():  # eight outliers: a few steps take the second pass
    return sp.diags(np.concatenate([np.logspace(2, 3, 8), np.linspace(1, 2, 1592)])).tocsr()


def _solve(A, bh, algorithm):
    n = A.shape[0]
    G, b, x = LA.gMatrix(n), LA.gVector(n), LA.gVector(n)
    G.set_csr(A.indptr, A.indices, A.data)
    b.set(bh)
    S = LA.LinAlg_CreateSolver(None)
    for k, v in dict(Algorithm=algorithm, Preconditioner=0, Krylov_Size=30,
                     Nb_Iter_Max=500).items():
        S.set(k, v)
    S["stopping_test"] = 1e-12
    info = LA.LinAlg_Solve(G, b, S, x)
    assert info["status"] == 0 and info["true_residual"] <= 1e-11 * info["rhs_norm"], info
    return info["iterations"], x.numpy()


@pytest.mark.parametrize("algorithm", [8, 9])
@pytest.mark.parametrize("power", [-470, -300, -64, -15, 15, 64, 300, 470])
@pytest.mark.parametrize("kind", ["dominant", "graded"])
def test_scaled_system(kind, power, algorithm):
    A = _dominant(40, 3) if kind == "dominant" else _graded()
    x0 = np.random.default_rng(1).standard_normal(A.shape[0])
    s = 2.0 ** power
    its, x = _solve(A, A @ x0, algorithm)
    its_s, x_s = _solve(A * s, (A @ x0) * s, algorithm)
    assert abs(its_s - its) <= 1, (its_s, its)
    bound = 2 * 1e-12 * (3 if kind == "dominant" else 1000) * np.linalg.norm(A @ x0)
    assert np.linalg.norm(x_s - x) <= bound
