"""CG on the 3 x 3 block product: one block row to several waves of CTAs, both
sides of the line up to which a step's kernels start early (65,536 vector
entries), FP64 and mixed.

The stopping test bounds the recurrence's residual; the true one drifts from it
by a few eps ||A|| ||x|| a step, far below the factor of ten allowed here.  On
the small systems the solution is compared with a direct solve: the error is at
most kappa times the relative residual, kappa estimated from the matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import generate as G
from getdp_gb300 import linalg as LA
from getdp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 12, 13])
def test_block_cg(n, precision):
    p = W.elasticity_p2(n, seed=n)
    dm = W.dofmap_for(p)
    A, b = G.generate_problem(p, dm)
    x = LA.gVector(dm.n_dof)
    S = LA.LinAlg_CreateSolver(None)
    for k, v in dict(Algorithm=1, Preconditioner=0, Scaling=1, Nb_Iter_Max=100000,
                     Precision=precision).items():
        S.set(k, v)
    S["stopping_test"] = 1e-9
    info = LA.LinAlg_Solve(A, b, S, x)
    assert info["status"] == 0, info
    assert info["true_residual"] <= 1e-8 * info["rhs_norm"], info
    if n > 3:
        return
    indptr, indices, data = A.csr()
    M = sp.csr_matrix((data, indices, indptr), shape=(dm.n_dof, dm.n_dof)).toarray()
    d = 1.0 / np.sqrt(np.abs(np.diag(M)))
    kappa = np.linalg.cond(d[:, None] * M * d)
    ref = np.linalg.solve(M, b.numpy())
    scaled = np.linalg.norm((x.numpy() - ref) / d) / np.linalg.norm(ref / d)
    assert scaled <= 10 * kappa * 1e-9
