"""CG on the scalar CSR product (any matrix that is not the elasticity
Generate's own), FP64 and mixed, on both sides of the line up to which a step's
kernels start early (65,536 unknowns): its product reads the search direction
that the kernel before it writes, so a stale or early read shows in the steps
and in the solution.

The matrices are symmetric with spectrum in [1 - w, 1 + w], w = 0.999: S is
scaled to D^-1/2 S D^-1/2, of norm at most 1.  The error is therefore at most
1000 times the residual and ||b|| <= 2 ||x||, which bounds it by 2000 times the
relative residual.  Step counts: the recurrences of the two sides differ by
rounding only, which moves the residual by some kappa eps a step, so the step at
which it passes the tolerance differs by one or two."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


def _matrix(n, halfband, seed):
    """Symmetric, unit diagonal, 2 halfband off-diagonals; halfband 0: the
    five-point pattern of a grid."""
    rng = np.random.default_rng(seed)
    if halfband == 0:
        side = int(round(np.sqrt(n)))
        T = sp.diags([np.ones(side - 1)], [1], shape=(side, side))
        U = sp.kron(sp.identity(side), T) + sp.kron(T, sp.identity(side))
    else:
        U = sp.diags([np.ones(n - k) for k in range(1, halfband + 1)],
                     list(range(1, halfband + 1)))
    U = sp.csr_matrix(U)
    U.data = -rng.uniform(0.5, 1.0, U.nnz)
    S = U + U.T
    d = 1.0 / np.sqrt(np.asarray(abs(S).sum(axis=1)).ravel())
    A = (sp.identity(S.shape[0]) + 0.999 * (sp.diags(d) @ S @ sp.diags(d))).tocsr()
    A.sort_indices()
    return A


# 3,025 / 59,536 / 65,536 / 66,049 / 70,225 unknowns; rows of 5, 25, 51, 101 and
# 201 entries take 2, 4, 8, 16 and 32 lanes
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,halfband", [(55 ** 2, 0), (244 ** 2, 0), (256 ** 2, 0),
                                        (257 ** 2, 0), (265 ** 2, 0), (3001, 12), (3001, 25),
                                        (3001, 50), (3001, 100), (1, 0)])
def test_scalar_cg(n, halfband, precision):
    A = _matrix(n, halfband, n + halfband) if n > 1 else sp.identity(1, format="csr") * 2.0
    n = A.shape[0]
    x0 = np.random.default_rng(7).standard_normal(n)
    bh = A @ x0
    G, b, x = LA.gMatrix(n), LA.gVector(n), LA.gVector(n)
    G.set_csr(A.indptr, A.indices, A.data)
    b.set(bh)
    S = LA.LinAlg_CreateSolver(None)
    for k, v in dict(Algorithm=1, Preconditioner=0, Nb_Iter_Max=5000, Precision=precision).items():
        S.set(k, v)
    S["stopping_test"] = 1e-10
    info = LA.LinAlg_Solve(G, b, S, x)
    assert info["status"] == 0, info
    assert info["true_residual"] <= 1.1e-10 * info["rhs_norm"], info
    assert np.linalg.norm(x.numpy() - x0) <= 2000 * 1.1e-10 * np.linalg.norm(x0)
    if precision == 0:
        xo, st, its, _ = oracle.solve(A.indptr, A.indices, A.data, bh, algorithm=oracle.CG,
                                      preconditioner=oracle.NONE, renumbering=0,
                                      nb_iter_max=5000, stopping_test=1e-10)
        assert st == 0 and abs(info["iterations"] - its) <= 3, (info["iterations"], its)
