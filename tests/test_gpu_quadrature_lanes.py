"""The quadrature kernel's two forms (a lane or a pair of lanes per node, chosen by the number of
nodes) against the oracle's QL, around the number of nodes where the form changes: odd counts, a last
block that is not full, one step and two, exact zeros on and off the diagonal, and sub-diagonals that
span the range of the fast root and fall outside it.  Every operation is correctly rounded in both
forms, so the deflation order is the oracle's and values agree to 1e-12 relative."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,q", [(1, 40), (1, 1), (3, 2), (33, 17), (9728, 12), (9729, 12), (4097, 64)])
def test_lanes_match_oracle(n, q, oracle_mod):
    from sqminiapp_gb300.capi import lib
    r = np.random.default_rng(n * 100 + q)
    a = 18.0 + 2.0 * r.standard_normal((n, q))
    b = 11.0 + 0.5 * r.random((n, q))
    special = set()
    if n > 30 and q > 4:
        a[5], b[5] = 0.0, 0.0                                   # a node after a breakdown
        b[7, q // 2:] = 0.0
        b[9] = 10.0 ** r.uniform(-30, 2, q)
        b[11, 1:3] = 1e-60                                      # products below the fast root's range
        a[12], b[12] = a[12] * 1e30, b[12] * 1e30               # and above it
        special = {5, 7, 9, 11, 12}
    out = [np.empty((n, q)), np.empty((n, q)), np.empty(n), np.empty(n)]
    dp = ctypes.POINTER(ctypes.c_double)
    st = lib().sq_tridiag_nodes_and_weights(a.ctypes.data_as(dp), b.ctypes.data_as(dp), n, q,
                                            *[x.ctypes.data_as(dp) for x in out], 0)
    assert st == 0
    for i in sorted(special | {0, n // 2, n - 1} | set(r.integers(0, n, 40))):
        lam, w, lo, hi = oracle_mod.ql(a[i], b[i])
        scale = max(1.0, np.max(np.abs(lam)))
        np.testing.assert_allclose(out[0][i], lam, rtol=1e-12, atol=1e-12 * scale)
        np.testing.assert_allclose(out[1][i], w, rtol=1e-12, atol=1e-14)
        assert (out[2][i], out[3][i]) == pytest.approx((lo, hi), rel=1e-12, abs=1e-12 * scale)
