"""The Fermi search of a cell that is empty or nearly so: no electrons at all at a low temperature (the
bisection ends where every occupation underflows), and fillings down to 1e-30, where states more than 45
occupation widths above the level hold the electrons.

Tolerance.  The midpoints are those of a plain bisection in FP64, whose sums differ by their order alone: the
level within 1e-9 (1e-13 relative of a sum with a slope of beta = 1000 per Ha, over a bracket of 50 Ha);
without electrons within the last bits of exp's overflow, 1e-9 as well."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fill", [0.0, 1e-30, 1e-18, 1e-12, 3e-8, 3e-7])
def test_nearly_empty(fill):
    import torch
    from sqminiapp_gb300.capi import lib
    r = np.random.default_rng(17)
    n, q, beta, tol = 2000, 16, 1000.0, 1e-12
    lam = 0.3 + 40.0 * r.random((n, q)) ** 2
    w = r.random((n, q))
    w /= w.sum(1, keepdims=True)
    ne = 2.0 * n * fill
    lo, hi = lam.min() - 1.0, lam.max() + 1.0
    with np.errstate(over="ignore"):
        for _ in range(200):
            mid = 0.5 * (lo + hi)
            if 2 * np.sum(w / (1.0 + np.exp(beta * (lam - mid)))) > ne:
                hi = mid
            else:
                lo = mid
            if hi - lo < tol:
                break
    d = [torch.from_numpy(a).cuda() for a in (lam, w)]
    rho = torch.empty(n, dtype=torch.float64, device="cuda")
    out = np.zeros(4)
    st = lib().sq_fermi_density_energy_noalloc(
        ctypes.c_void_p(d[0].data_ptr()), ctypes.c_void_p(d[1].data_ptr()), ctypes.c_long(n), q,
        ctypes.c_double(beta), ctypes.c_double(ne), ctypes.c_double(0.125), ctypes.c_double(tol), 200,
        ctypes.c_void_p(rho.data_ptr()), out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None)
    assert st == 0
    assert abs(out[0] - 0.5 * (lo + hi)) < 1e-9
