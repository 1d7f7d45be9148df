"""The quadrature's deflation test where |d_m| + |d_(m+1)| overflows or is infinite: as in the oracle's QL
every sub-diagonal then counts as zero, so such a node deflates at once instead of never.  The arithmetic
is the oracle's, operation by operation: equal values, and 1e-12 for the ordinary node beside it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 9731])  # two lanes per node, and one
def test_overflowing_diagonal_deflates(n, oracle_mod):
    from sqminiapp_gb300.capi import lib
    q = 4
    a, b = np.full((n, q), 18.0), np.full((n, q), 11.0)
    a += np.arange(q)
    a[0] = 1.5e308
    b[0] = 1e300
    a[1] = np.inf
    b[1] = np.inf
    out = [np.empty((n, q)), np.empty((n, q)), np.empty(n), np.empty(n)]
    dp = ctypes.POINTER(ctypes.c_double)
    st = lib().sq_tridiag_nodes_and_weights(a.ctypes.data_as(dp), b.ctypes.data_as(dp), n, q,
                                            *[x.ctypes.data_as(dp) for x in out], 0)
    assert st == 0
    for i in (0, 1):
        lam, w, lo, hi = oracle_mod.ql(a[i], b[i])
        np.testing.assert_array_equal(out[0][i], lam)
        np.testing.assert_array_equal(out[1][i], w)
    lam, w, _, _ = oracle_mod.ql(a[2], b[2])
    np.testing.assert_allclose(out[0][2], lam, rtol=1e-12)
    np.testing.assert_allclose(out[1][2], w, rtol=1e-12, atol=1e-14)
