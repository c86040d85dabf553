"""A row's product touches the columns that the row holds and no other: with
entries of x that are NaN or infinite, the rows without those columns come out
as the host's product has them (to the rounding bound of a row's dot product,
1e-13 sum_j |a_ij x_j| for up to some 200 terms of 1.1e-16), the rows with them
not finite.  Row lengths take every number of lanes per row and all remainders."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import _lib
from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("most", [9, 39, 89, 179, 349])  # 2, 4, 8, 16, 32 lanes per row
def test_rows_without_the_bad_column(most, bad):
    n = 1000
    rng = np.random.default_rng(most)
    rows = [np.sort(rng.choice(n, 1 + i % most, replace=False)) for i in range(n)]
    ip = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    M = sp.csr_matrix((rng.standard_normal(ip[-1]), np.concatenate(rows), ip), shape=(n, n))
    xv, bv = rng.standard_normal(n), rng.standard_normal(n)
    xv[0] = bad
    holds = np.zeros(n, bool)
    holds[[i for i, r in enumerate(rows) if r[0] == 0]] = True
    assert 0 < holds.sum() < n
    A, x, y, b = LA.gMatrix(n), LA.gVector(n), LA.gVector(n), LA.gVector(n)
    A.set_csr(M.indptr, M.indices, M.data)
    x.set(xv)
    b.set(bv)
    clean = np.where(np.isfinite(xv), xv, 0.0)
    bound = 1e-13 * (abs(M) @ np.abs(clean) + np.abs(bv))
    LA.LinAlg_ProdMatrixVector(A, x, y)
    for got, ref in ((y.numpy(), M @ clean), (None, bv - M @ clean)):
        if got is None:
            r, nrm = LA.gVector(n), ctypes.c_double()
            _lib.check(_lib.load().gb300_residual_noalloc(A.h, x.h, b.h, r.h, ctypes.byref(nrm)))
            got = r.numpy()
            assert not np.isfinite(nrm.value)
        assert np.all(np.abs(got - ref)[~holds] <= bound[~holds])
        assert not np.any(np.isfinite(got[holds]))
