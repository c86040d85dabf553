"""A network used on a matrix of another context than its own, and on after that
context is gone: same correction on both (inference has a fixed order of
operations), buffers grown in between."""
import ctypes

import numpy as np
import pytest

from getdp_gb300 import _lib
from getdp_gb300 import learned as ML
from getdp_gb300 import linalg as LA
from getdp_gb300 import workloads as W
from getdp_gb300.generate import generate_problem

pytestmark = pytest.mark.gpu


def _system(n):
    p = W.nonlinear_2d(n=n, seed=5)
    A, b = generate_problem(p, W.dofmap_for(p))
    return A.csr(), b.numpy()


def _corrected(ctx, csr, v, net):
    """z = M^-1 v with Preconditioner 20 on a matrix of the context ctx."""
    L, check = _lib.load(), _lib.check
    ip, ix, dv = (np.ascontiguousarray(a, t) for a, t in zip(csr, (np.int32, np.int32, float)))
    n = len(ip) - 1
    A, x, z = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    check(L.gb300_matrix_create(ctx, n, ctypes.byref(A)))
    check(L.gb300_vector_create(ctx, n, ctypes.byref(x)))
    check(L.gb300_vector_create(ctx, n, ctypes.byref(z)))
    ptr = lambda a: ctypes.c_void_p(a.ctypes.data)
    check(L.gb300_matrix_set_csr(A, len(dv), ptr(ip), ptr(ix), ptr(dv)))
    check(L.gb300_vector_set(x, ptr(v)))
    check(L.gb300_mpnn_infer(net.h, A))
    S = LA.LinAlg_CreateSolver(None)
    S.set("Preconditioner", 20)
    S.set("Renumbering_Technique", 1)
    check(L.gb300_precond_apply(A, ctypes.byref(S.params), x, z))
    out = np.empty(n)
    check(L.gb300_vector_get(z, ptr(out)))
    for h in (x, z):
        check(L.gb300_vector_destroy(h))
    check(L.gb300_matrix_destroy(A))
    return out


def test_network_outlives_a_matrix_context():
    L = _lib.load()
    small, big = _system(17)[0], _system(33)[0]
    rng = np.random.default_rng(3)
    v, vb = rng.standard_normal(len(small[0]) - 1), rng.standard_normal(len(big[0]) - 1)
    net = ML.MPNN(seed=2)
    w = net.params()
    net.set_params(w + 0.05 * rng.standard_normal(w.shape).astype(np.float32))
    first = _corrected(LA.context(), small, v, net)
    for _ in range(2):
        ctx = ctypes.c_void_p()
        _lib.check(L.gb300_ctx_create(0, ctypes.byref(ctx)))
        assert np.array_equal(_corrected(ctx, small, v, net), first)
        other = ML.MPNN(seed=2)  # its first buffers made for the other context's matrix
        other.set_params(net.params())
        assert np.array_equal(_corrected(ctx, small, v, other), first)
        _lib.check(L.gb300_ctx_destroy(ctx))
        assert np.all(np.isfinite(_corrected(LA.context(), big, vb, other)))  # buffers grow
        assert np.array_equal(_corrected(LA.context(), small, v, other), first)
        del other
