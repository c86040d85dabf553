"""AssembleMatrix of scalar entries: bulk adds staged on the device, mixed with
single ones, on both sides of the 32-entries-per-row rule.  Duplicates are
summed in call order, so every value equals the sequential sum to the bit."""
import numpy as np
import pytest

from getdp_gb300 import linalg as LA
from getdp_gb300._lib import GetDPError

pytestmark = pytest.mark.gpu


def _reference(n, calls):
    acc = {}
    for i, j, v in calls:
        for a, b, x in zip(i.tolist(), j.tolist(), v.tolist()):
            acc[(a, b)] = acc[(a, b)] + x if (a, b) in acc else x
    keys = sorted(acc)
    ip = np.zeros(n + 1, np.int64)
    for a, _ in keys:
        ip[a + 1] += 1
    return np.cumsum(ip), np.array([b for _, b in keys]), np.array([acc[k] for k in keys])


def _entries(rng, n, m, spread):
    i = rng.integers(0, n, m)
    j = np.clip(i + rng.integers(-spread, spread + 1, m), 0, n - 1)
    v = rng.standard_normal(m) * 10.0 ** rng.integers(-8, 9, m)
    return i.astype(np.int32), j.astype(np.int32), v


# entries per row about 20000 / n: 10 (all rows in the warps' kernel), 33 and
# 34 around the rule, 400 (several warps' worth)
@pytest.mark.parametrize("n,spread", [(3000, 4), (620, 3), (50, 30)])
def test_bulk_and_single_adds_keep_the_call_order(n, spread):
    rng = np.random.default_rng(n)
    calls = [_entries(rng, n, 300, spread), _entries(rng, n, 16384, spread),
             _entries(rng, n, 77, spread), _entries(rng, n, 20001, spread)]
    A = LA.gMatrix(n)
    for c in calls:
        A.add_coo(*c)
    LA.LinAlg_AddDoubleInMatrix(0.125, A, 1, 1)
    calls.append((np.array([1]), np.array([1]), np.array([0.125])))
    for got, ref in zip(A.csr(), _reference(n, calls)):
        assert np.array_equal(got, ref)
    # a second assembly adds to the first one's values
    ip, ix, dv = A.csr()
    more = _entries(rng, n, 17000, spread)
    A.add_coo(*more)
    rows = np.repeat(np.arange(n), np.diff(ip))
    ref = _reference(n, [(rows, ix, dv), more])
    for got, r in zip(A.csr(), ref):
        assert np.array_equal(got, r)


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("lengths", [(31, 32), (32, 32), (33, 32)])
def test_row_length_rule_and_unaligned_arrays(shift, lengths):
    n, rng = 600, np.random.default_rng(shift)
    per = np.resize(lengths, n)
    i = np.repeat(np.arange(n), per)
    order = rng.permutation(len(i))
    i = i[order]
    j = rng.integers(0, n, len(i))
    v = rng.standard_normal(len(i))

    def place(a, t):  # the same values at an address `shift` elements off
        b = np.empty(len(a) + 4, t)[shift:shift + len(a)]
        b[:] = a
        return b

    c = place(i, np.int32), place(j, np.int32), place(v, np.float64)
    A = LA.gMatrix(n)
    A.add_coo(*c)
    for got, ref in zip(A.csr(), _reference(n, [c])):
        assert np.array_equal(got, ref)


def test_out_of_range_bulk_add_is_refused_whole():
    n, rng = 500, np.random.default_rng(9)
    A = LA.gMatrix(n)
    good = _entries(rng, n, 20000, 3)
    A.add_coo(*good)
    bad = [a.copy() for a in _entries(rng, n, 20000, 3)]
    bad[0][12345] = n
    bad[1][15000] = -1
    with pytest.raises(GetDPError, match=rf"entry 12345 \({n}, "):
        A.add_coo(*bad)
    for got, ref in zip(A.csr(), _reference(n, [good])):
        assert np.array_equal(got, ref)
