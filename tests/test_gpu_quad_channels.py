"""The split-pass kernel over the channel sets that no Mg deck of this repository has: none at all (a
29^3 cube whose shared memory ends just behind its two vectors).

Tolerance.  As in test_gpu_quad_list: 1.1e-4 on the first coefficients (50 roundings of 2^-24 on terms of up
to 36), 1e-4 relative to max(1, |value|) on the moments of order <= 3."""
import os

import numpy as np
import pytest

from sqminiapp_gb300 import plan_kernel
from sqminiapp_gb300.decks import make_fcc_mg_deck


def _psd(path, lmax):
    """Cuts a pseudopotential file down to the channels 0..lmax."""
    head, *blocks = [b for b in _blocks(open(path).read())]
    keep = [b for b in blocks if not b[0].startswith(("Pseudopotential", "Pseudo-wave")) or _channel(b) <= lmax]
    return "\n".join(head + [line for b in keep for line in b]) + "\n"


def _blocks(text):
    out = [[]]
    for line in text.splitlines():
        if "follows" in line:
            out.append([])
        out[-1].append(line.strip() if "follows" in line else line)
    return out


def _channel(block):
    return int(block[1].split()[0])


# name: (lmax, PSEUDOPOTENTIAL_LOCAL) of every type, ncell, h, rcut, steps, cube, threads
CASES = {"none": ([(0, 0)], 1, 0.5, 7.0, 10, 29, 512)}


def _deck(path, name):
    types, ncell, h, rcut, q, _, _ = CASES[name]
    d, n, _ = make_fcc_mg_deck(str(path), "c", ncell=ncell, h=h, rcut=rcut, n_qp=q, disp=0.2, seed=21, lloc=types[0][1])
    f = os.path.join(d, "pseudopotential", "psd_Mg.pot")
    text = _psd(f, types[0][0])
    with open(f, "w") as out:
        out.write(text)
    return d, n


@pytest.mark.parametrize("name", CASES)
def test_plan(name, tmp_path):
    info = plan_kernel(*_deck(tmp_path, name))
    assert (info.kernel_layout, info.cube[0], info.kernel_threads) == (16, CASES[name][5], CASES[name][6])


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_against_oracle(name, tmp_path, oracle_mod):
    from sqminiapp_gb300 import LSDFT
    d, n = _deck(tmp_path, name)
    o = oracle_mod.Oracle(d, n, faithful=False)
    nodes = np.arange(0, o.n_nodes, max(1, o.n_nodes // 9))
    veff = -0.3 + 0.1 * np.random.default_rng(5).standard_normal(o.n_nodes)
    ref = o.nodes_and_weights(nodes=nodes, veff=veff, want_ab=True)
    o.close()
    with LSDFT(d, n, faithful=False, precision=32) as eng:
        assert eng.info.kernel_layout == 16
        out = eng.NodesAndWeights_LSSGQ(veff=veff)
        a, b = eng.lanczos_coefficients(eng.n_nodes)
    np.testing.assert_allclose(a[nodes, :4], ref["a"][:, :4], rtol=0, atol=1.1e-4)
    np.testing.assert_allclose(b[nodes, :4], ref["b"][:, :4], rtol=0, atol=1.1e-4)
    for k in range(4):
        g = np.sum(out["weights"][nodes] * out["lambda"][nodes] ** k, axis=1)
        e = np.sum(ref["weights"] * ref["lambda"] ** k, axis=1)
        assert np.max(np.abs(g - e) / np.maximum(1.0, np.abs(e))) < 1e-4, k
