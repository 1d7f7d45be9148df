"""Values that are not finite in the Fermi call end where a plain sum over every entry brings them: an
infinite Ritz value (infinity minus infinity) and a weight that is not a number make the band energy NaN;
an infinite weight pulls the level down to where its occupation underflows, and where a coarse tolerance
ends the bisection beyond that (780 occupation widths below it) its term is 0 times infinity: its node's
density is NaN."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(lam, w, beta, ne, tol, dv=0.125):
    import torch
    from sqminiapp_gb300.capi import lib
    n, q = lam.shape
    d = [torch.from_numpy(a).cuda() for a in (lam, w)]
    rho = torch.empty(n, dtype=torch.float64, device="cuda")
    out = np.zeros(4)
    st = lib().sq_fermi_density_energy_noalloc(
        ctypes.c_void_p(d[0].data_ptr()), ctypes.c_void_p(d[1].data_ptr()), ctypes.c_long(n), q,
        ctypes.c_double(beta), ctypes.c_double(ne), ctypes.c_double(dv), ctypes.c_double(tol), 200,
        ctypes.c_void_p(rho.data_ptr()), out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None)
    return st, out, rho.cpu().numpy()


@pytest.mark.parametrize("kind", ["clean", "lambda", "weight", "infinite weight"])
def test_not_finite_values_reach_the_sums(kind):
    r = np.random.default_rng(11)
    n, q, beta = 300, 12, 316.0
    lam = -0.4 + 20.0 * r.random((n, q)) ** 2
    w = r.random((n, q))
    w /= w.sum(1, keepdims=True)
    if kind == "lambda":
        lam[7, 3] = np.inf
    elif kind == "weight":
        w[7, 3] = np.nan
    elif kind == "infinite weight":
        lam[7, 3], w[7, 3] = 10.0, np.inf
    st, out, rho = _call(lam, w, beta, 0.2 * n, 2.0 if kind == "infinite weight" else 1e-12)
    if kind == "clean":
        assert st == 0 and np.all(np.isfinite(out)) and np.all(np.isfinite(rho))
        return
    assert not np.isfinite(out[1])
    if kind == "infinite weight":
        assert beta * (10.0 - out[0]) > 745.2 and np.isnan(rho[7])
        assert np.all(np.isfinite(np.delete(rho, 7)))
