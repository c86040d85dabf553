"""A Krylov vector that becomes exactly zero ends GMRES with mgsro's code -1 as
the break-down status -3, at the oracle's step, whatever the number of column
groups and CTAs in flight: A shifts e_s to e_(s-1) and e_0 to zero, so the step
after s + 1 of them has the product zero.  The solution stays zero."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algorithm", [8, 9])
@pytest.mark.parametrize("n,start", [(500, 0), (500, 6), (500, 7), (500, 8), (70000, 15),
                                     (70000, 16), (400000, 25)])
def test_zero_product(n, start, algorithm):
    i = np.arange(n)  # rows (i, i) = 0, (i, i + 1) = 1
    ix = np.stack([i, i + 1], 1).ravel()[:-1]
    dv = np.tile([0.0, 1.0], n)[:-1]
    A = sp.csr_matrix((dv, ix, np.append(2 * i, 2 * n - 1)), shape=(n, n))
    bh = np.zeros(n)
    bh[start] = 1.0
    _, st, its, _ = oracle.solve(A.indptr, A.indices, A.data, bh, algorithm=algorithm,
                                 preconditioner=oracle.NONE, renumbering=0, krylov_size=30,
                                 nb_iter_max=200)
    assert st == -3 and its == start + 2
    G, b, x = LA.gMatrix(n), LA.gVector(n), LA.gVector(n)
    G.set_csr(A.indptr, A.indices, A.data)
    b.set(bh)
    S = LA.LinAlg_CreateSolver(None)
    for k, v in dict(Algorithm=algorithm, Preconditioner=0, Krylov_Size=30,
                     Nb_Iter_Max=200).items():
        S.set(k, v)
    info = LA.LinAlg_Solve(G, b, S, x)
    assert info["status"] == -3 and info["iterations"] == its, info
    assert not x.numpy().any()
