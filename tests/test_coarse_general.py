"""The coarse inverse of a matrix that is not symmetric: u^T C u and the
two-level cycle against numpy's inverse.  The matrices have a positive definite
symmetric part, so every pivot of an elimination without pivoting is positive.

Forward errors: an elimination without pivoting of a matrix whose symmetric part
dominates is off by ~nc eps cond, as in the tests of the symmetric ones."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from getdp_gb300 import _lib
from getdp_gb300 import linalg as LA

pytestmark = pytest.mark.gpu


def _energy(A, uh):
    u, out = LA.gVector(A.n), ctypes.c_double()
    u.set(uh)
    _lib.check(_lib.load().gb300_matrix_coarse_energy(A.h, u.h, ctypes.byref(out)))
    return out.value


# a single upper or lower entry apart, and the whole matrix; around the blocks
# of 32 and the check's tiles
@pytest.mark.parametrize("nc", [2, 31, 32, 33, 65, 200])
@pytest.mark.parametrize("where", ["all", "first", "last"])
def test_energy_with_a_skew_part(nc, where):
    rng = np.random.default_rng(nc)
    M = rng.standard_normal((nc, nc))
    D = M @ M.T / nc + 0.5 * np.eye(nc)
    if where == "all":
        K = rng.standard_normal((nc, nc))
        D += (K - K.T) / np.sqrt(nc)
    elif where == "first":
        D[1, 0] += 0.2
    else:
        D[nc - 2, nc - 1] += 0.2
    assert np.linalg.eigvalsh((D + D.T) / 2)[0] > 0.1 and np.linalg.cond(D) < 100
    S = sp.csr_matrix(D)
    A = LA.gMatrix(nc)
    A.set_csr(S.indptr, S.indices, S.data)
    A.set_aggregates(rng.permutation(nc), nc)
    uh = rng.standard_normal(nc)
    ref = uh @ np.linalg.solve(D, uh)
    mirrored = uh @ np.linalg.solve(np.tril(D) + np.tril(D, -1).T, uh)
    bound = 200 * 1.1e-16 * 100 * (uh @ uh) / 0.1
    assert abs(_energy(A, uh) - ref) <= bound
    if where == "all":  # (what half of the matrix alone would give is elsewhere)
        assert abs(mirrored - ref) > 1e3 * bound
    # the same matrix made symmetric again takes the other way
    D = (D + D.T) / 2
    S = sp.csr_matrix(D)
    A.set_csr(S.indptr, S.indices, S.data)
    A.set_aggregates(np.arange(nc), nc)
    assert abs(_energy(A, uh) - uh @ np.linalg.solve(D, uh)) <= bound


@pytest.mark.parametrize("renumbering", [0, 1])
def test_cycle_on_a_transport_problem(renumbering):
    m = 40  # -div grad + an upwind transport, structurally symmetric
    T = sp.diags([-1.0, 2.0, -1.0], [-1, 0, 1], shape=(m, m))
    C = sp.diags([-1.0, 1.0], [-1, 0], shape=(m, m))
    E = sp.identity(m)
    Am = (sp.kron(T, E) + sp.kron(E, T) + 0.7 * sp.kron(C, E) + 0.3 * sp.kron(E, C)).tocsr()
    Am.sort_indices()
    n, nc = m * m, 100
    i = np.arange(n)
    agg = (i // m // 4) * 10 + (i % m) // 4
    A = LA.gMatrix(n)
    A.set_csr(Am.indptr, Am.indices, Am.data)
    A.set_aggregates(agg, nc)
    P = sp.csr_matrix((np.ones(n), (i, agg)), shape=(n, nc))
    Aci = np.linalg.inv((P.T @ Am @ P).toarray())

    def apply(prec, v):
        S = LA.LinAlg_CreateSolver(None)
        S.set("Preconditioner", prec)
        S.set("Renumbering_Technique", renumbering)
        vv, z = LA.gVector(n), LA.gVector(n)
        vv.set(v)
        _lib.check(_lib.load().gb300_precond_apply(A.h, ctypes.byref(S.params), vv.h, z.h))
        return z.numpy()

    v = np.random.default_rng(1).standard_normal(n)
    z = apply(6, v)
    z = z + P @ (Aci @ (P.T @ (v - Am @ z)))
    z = z + apply(6, v - Am @ z)
    got = apply(21, v)
    # Ac is summed in fixed point (2^-51 of max|a| a term) and inverted: cond(Ac)
    # is some 100 here, and its error reaches z through contractions
    assert np.linalg.norm(got - z) <= 1e-11 * np.linalg.norm(z)


@pytest.mark.parametrize("bad", [33, 515, 991])
def test_bad_pivot_while_other_tiles_run(bad):
    """The pivot is found by one CTA of an update whose other CTAs are at any
    point of theirs; the next inversion on the same handle starts clean."""
    nc = 1000
    d = np.linspace(1.0, 2.0, nc)
    uh = np.random.default_rng(bad).standard_normal(nc)
    A = LA.gMatrix(nc)
    for value in (-1.0, 1.5):
        d[bad] = value
        S = sp.diags(d).tocsr()
        A.set_csr(S.indptr, S.indices, S.data)
        A.set_aggregates(np.arange(nc), nc)
        if value < 0:
            with pytest.raises(LA.GetDPError, match=f"pivot {bad + 1} of {nc}"):
                _energy(A, uh)
        else:  # (one rounding of the entry's sum, one of its inverse)
            ref = uh @ (uh / d)
            assert abs(_energy(A, uh) - ref) <= nc * 2.3e-16 * ref
