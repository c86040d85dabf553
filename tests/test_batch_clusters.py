"""The batched solve's default cluster size (4, 8 or 16 CTAs by the batch's
size) and its colour sweeps against the per-kernel form: step counts within
one, solutions within the residual the two stop at (1e-12; the systems'
condition numbers are below 1e5, so 1e-7 of the solution, tightened to the
1e-9 the forms' existing comparison asserts)."""
import numpy as np
import pytest

from getdp_gb300 import generate as G
from getdp_gb300 import linalg as LA
from getdp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _solve(A, b, off, kernel, algorithm, precision):
    S = LA.LinAlg_CreateSolver(None)
    for k, v in dict(Algorithm=algorithm, Preconditioner=6, Krylov_Size=40, Nb_Iter_Max=5000,
                     Renumbering_Technique=1, Precision=precision).items():
        S.set(k, v)
    if kernel is not None:
        S.set("Batch_Kernel", kernel)
    S["stopping_test"] = 1e-12
    x = LA.gVector(A.n)
    infos = LA.LinAlg_SolveBatch(A, b, S, x, off)
    return infos, x.numpy()


# largest system 2 (n - 1)^2 rows (complex): 16,562 rows take clusters of 16,
# 8,450 of 8, 450 of 4; real systems (one row per vertex) beside the complex
@pytest.mark.parametrize("kind,sizes", [("eddy", (92, 24)), ("eddy", (66, 9, 31)),
                                        ("eddy", (16, 13)), ("magnet", (130, 33))])
@pytest.mark.parametrize("algorithm,precision", [(8, 0), (9, 1)])
def test_default_clusters_match_the_per_kernel_form(kind, sizes, algorithm, precision):
    make = W.eddy_2d if kind == "eddy" else W.magnetostatics_2d
    bt = W.concat_problems([make(n, seed=40 + n) for n in sizes])
    terms = G.DeviceTerms(bt.problem, bt.dofmap)
    A, b = LA.gMatrix(bt.dofmap.n_dof), LA.gVector(bt.dofmap.n_dof)
    G.generate(A, b, terms.batch)
    i0, x0 = _solve(A, b, bt.offsets, 0, algorithm, precision)
    i1, x1 = _solve(A, b, bt.offsets, None, algorithm, precision)
    for k in range(len(sizes)):
        assert i1[k]["batch_form"] == 1 and i0[k]["batch_form"] == 0
        assert i1[k]["status"] == 0 and i0[k]["status"] == 0, (i1[k], i0[k])
        assert abs(i1[k]["iterations"] - i0[k]["iterations"]) <= 1, (i1[k], i0[k])
        r0, r1 = bt.offsets[k], bt.offsets[k + 1]
        assert np.linalg.norm(x1[r0:r1] - x0[r0:r1]) <= 1e-9 * np.linalg.norm(x0[r0:r1])


def test_a_size_asked_for_is_the_size_used():
    """The sums are split by the cluster's CTAs, so another size rounds otherwise
    and the same one does not: the default takes 16 CTAs for these systems, and
    a size given in Batch_Kernel is kept, the smallest of the default's too."""
    bt = W.concat_problems([W.eddy_2d(n, seed=40 + n) for n in (92, 24)])
    terms = G.DeviceTerms(bt.problem, bt.dofmap)
    A, b = LA.gMatrix(bt.dofmap.n_dof), LA.gVector(bt.dofmap.n_dof)
    G.generate(A, b, terms.batch)
    x = {c: _solve(A, b, bt.offsets, c, 8, 0) for c in (4, 8, 16, -1, None)}
    for infos, _ in x.values():
        assert all(i["batch_form"] == 1 and i["status"] == 0 for i in infos)
    assert np.array_equal(x[None][1], x[16][1]) and np.array_equal(x[-1][1], x[16][1])
    assert not np.array_equal(x[4][1], x[16][1]) and not np.array_equal(x[4][1], x[8][1])
    # asked for again: the same bits
    assert np.array_equal(_solve(A, b, bt.offsets, 4, 8, 0)[1], x[4][1])
