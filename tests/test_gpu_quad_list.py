"""The split-pass kernel's projector list at the sizes where it can go wrong: cubes of fewer planes
than a unit has (3^3), of one plane range per column and of several, with and without pad points in
the last quad, columns dealt to the lanes by bank class and (most nodes of the three smallest) by the
number of units alone, on one CTA and on a pair, and every channel set the Mg pseudopotential gives
(s+p, s+d, p+d).

Tolerance.  The first coefficients of the recurrence against the FP64 oracle: a_k and b_k are sums
over stencil and projector terms of size up to 2 * 18 (h = 0.5), each rounded to FP32 (2^-24), about
50 roundings deep: 50 * 36 * 6e-8 = 1.1e-4 at most, absolute.  The quadrature's moments of order <= 3
relative to max(1, |value|): 1e-4, as in the other parity tests.  Two runs give the same bits (no
atomics, fixed orders)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rcut, h, steps, PSEUDOPOTENTIAL_LOCAL, seed -> cubes of 3, 5, 7, 9, 15, 17, 21, 27, 29, 31 and 33 points
CASES = [(0.8, 0.85, 6, 2, 1), (1.6, 0.85, 10, 1, 2), (2.5, 0.85, 12, 0, 3), (3.4, 0.85, 12, 2, 4),
         (4.2, 0.607, 12, 1, 5), (4.8, 0.607, 12, 2, 6), (5.0, 0.5, 10, 0, 7), (6.5, 0.5, 10, 1, 8),
         (6.5, 0.5, 10, 0, 9), (7.0, 0.5, 10, 2, 10), (7.5, 0.5, 8, 1, 11), (7.0, 0.45, 8, 0, 12)]


@pytest.mark.parametrize("rcut,h,q,lloc,seed", CASES)
def test_list_against_oracle(rcut, h, q, lloc, seed, tmp_path, oracle_mod):
    from sqminiapp_gb300 import LSDFT
    from sqminiapp_gb300.decks import make_fcc_mg_deck
    d, name, _ = make_fcc_mg_deck(str(tmp_path), "c", ncell=1, h=h, rcut=rcut, n_qp=q, disp=0.2,
                                  seed=seed, lloc=lloc)
    o = oracle_mod.Oracle(d, name, faithful=False)
    nodes = np.arange(0, o.n_nodes, max(1, o.n_nodes // 9))
    veff = -0.3 + 0.1 * np.random.default_rng(seed).standard_normal(o.n_nodes)
    ref = o.nodes_and_weights(nodes=nodes, veff=veff, want_ab=True)
    with LSDFT(d, name, faithful=False, precision=32, kernel=2) as eng:
        assert eng.info.kernel_layout & 16
        out = eng.NodesAndWeights_LSSGQ(veff=veff)
        a, b = eng.lanczos_coefficients(eng.n_nodes)
        again = eng.NodesAndWeights_LSSGQ(veff=veff)
    np.testing.assert_allclose(a[nodes, :4], ref["a"][:, :4], rtol=0, atol=1.1e-4)
    np.testing.assert_allclose(b[nodes, :4], ref["b"][:, :4], rtol=0, atol=1.1e-4)
    for k in range(4):
        g = np.sum(out["weights"][nodes] * out["lambda"][nodes] ** k, axis=1)
        e = np.sum(ref["weights"] * ref["lambda"] ** k, axis=1)
        assert np.max(np.abs(g - e) / np.maximum(1.0, np.abs(e))) < 1e-4, k
    for k in out:
        assert np.array_equal(out[k], again[k]), k
