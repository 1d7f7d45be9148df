"""The Fermi search against the plain bisection of every midpoint (numpy, FP64), where it can go
wrong: one node and few, slices that fit the gathered entries and slices that do not (all Ritz values
within one occupation width), steps of a low and a high beta, electron counts at both ends, empty
shells that leave N_e flat, and weights below zero (N_e no longer grows with the level, every midpoint
is evaluated).

Tolerance.  Midpoints and stop rule are the same, so the level differs only where a midpoint lies
within the rounding of N_e (relative 1e-13 of it, divided by the slope): 1e-9 in lf, and 1e-9 relative
in the sums; where N_e is flat to rounding the level is any of the flat part, so only N_e is compared."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _f(beta, lam, lf):
    x = np.clip(beta * (lam - lf), -700.0, 700.0)
    return 1.0 / (1.0 + np.exp(x))


def _bisect(lam, w, beta, ne, tol=1e-12):
    lo, hi = lam.min() - 1.0, lam.max() + 1.0
    for _ in range(400):
        mid = 0.5 * (lo + hi)
        if 2 * np.sum(w * _f(beta, lam, mid)) > ne:
            hi = mid
        else:
            lo = mid
        if hi - lo < tol:
            break
    return 0.5 * (lo + hi)


CASES = [(1, 5, 30.0, 0.5, "band"), (7, 30, 316.0, 0.1, "band"), (513, 40, 316.0, 0.07, "band"),
         (40000, 40, 316.0, 0.05, "band"), (40000, 40, 5.0, 0.3, "band"), (60000, 40, 316.0, 0.5, "point"),
         (3000, 20, 1000.0, 0.999, "band"), (3000, 20, 1000.0, 1e-6, "band"), (2000, 16, 316.0, 0.25, "gap"),
         (500, 12, 316.0, 0.3, "negative")]


@pytest.mark.parametrize("n,q,beta,fill,kind", CASES)
def test_search_equals_bisection(n, q, beta, fill, kind, tmp_path):
    import torch
    from sqminiapp_gb300.capi import lib
    import ctypes
    r = np.random.default_rng(n + q)
    lam = -0.4 + 45.0 * r.random((n, q)) ** 2
    if kind == "point":  # all within one occupation width
        lam = 0.2 + 1e-3 * r.random((n, q))
    if kind == "gap":
        lam = np.where(r.random((n, q)) < 0.25, -0.5 + 0.1 * r.random((n, q)), 3.0 + r.random((n, q)))
    w = r.random((n, q))
    w /= w.sum(1, keepdims=True)
    if kind == "negative":
        w[3, 2] = -0.4
    ne = 2.0 * n * fill
    if kind == "gap":
        ne = 2.0 * np.sum(w * (lam < 1.0))
    dv, tol = 0.125, 1e-12
    d = [torch.from_numpy(a).cuda() for a in (lam, w)]
    rho = torch.empty(n, dtype=torch.float64, device="cuda")
    out = np.zeros(4)
    dp = ctypes.POINTER(ctypes.c_double)
    st = lib().sq_fermi_density_energy_noalloc(
        ctypes.c_void_p(d[0].data_ptr()), ctypes.c_void_p(d[1].data_ptr()), ctypes.c_long(n), q,
        ctypes.c_double(beta), ctypes.c_double(ne), ctypes.c_double(dv), ctypes.c_double(tol), 200,
        ctypes.c_void_p(rho.data_ptr()), out.ctypes.data_as(dp), None)
    assert st == 0
    lf = out[0]
    f = _f(beta, lam, lf)
    total = 2 * np.sum(w * f)
    if kind == "gap":
        assert abs(total - ne) < 1e-9 * ne
    else:
        assert abs(lf - _bisect(lam, w, beta, ne)) < 1e-9
    np.testing.assert_allclose(rho.cpu().numpy(), 2 * np.sum(w * f, axis=1) / dv, rtol=1e-9, atol=1e-12)
    assert out[1] == pytest.approx(2 * np.sum(w * lam * f), rel=1e-9, abs=1e-9)
    with np.errstate(divide="ignore", invalid="ignore"):
        s = np.where((f > 0) & (f < 1), f * np.log(f) + (1 - f) * np.log(1 - f), 0.0)
    assert out[2] == pytest.approx(2 * np.sum(w * s) / beta, rel=1e-7, abs=1e-9)
