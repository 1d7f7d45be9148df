"""The split-pass kernel over the channel sets that no Mg deck of this repository has: none at all (a
29^3 cube whose shared memory ends just behind its two vectors), one channel, s+p+d, two atom types of
different sets (s+p beside s+d, and s+p+d beside p+d+f, all 16 harmonics), and a cell of more atoms in a
cube than the CTA has warps.  The f channel is made from the file's p and d channels.

Tolerance.  As in test_gpu_quad_list: 1.1e-4 on the first coefficients (50 roundings of 2^-24 on terms of up
to 36), 1e-4 relative to max(1, |value|) on the moments of order <= 3."""
import os
import re

import numpy as np
import pytest

from sqminiapp_gb300 import plan_kernel
from sqminiapp_gb300.decks import make_fcc_mg_deck


def _blocks(text):
    out = [[]]
    for line in text.splitlines():
        if "follows" in line:
            out.append([])
        out[-1].append(line.strip() if "follows" in line else line)
    return out


def _numbers(block):
    return [float(t) for line in block[1:] for t in line.split()]


def _psd(path, lmax):
    """A pseudopotential file's text with the channels 0..lmax (3: an f channel, its potential the mean of
    p's and d's, its wave function d's times r)."""
    head, *blocks = _blocks(open(path).read())
    r = next(_numbers(b) for b in blocks if b[0].startswith("Radial"))
    out, p = list(head), None
    for b in blocks:
        lead = 1 if b[0].startswith("Pseudopotential") else 3 if b[0].startswith("Pseudo-wave") else 0
        v = _numbers(b)
        if not lead or v[0] <= lmax:
            out += b
        if lead and v[0] == 1:
            p = v
        if lead and v[0] == 2 and lmax == 3:
            f = [0.5 * (x + y) for x, y in zip(p[1:], v[1:])] if lead == 1 else v[1:3] + [x * y for x, y in zip(v[3:], r)]
            out += [b[0], " ".join("%.12g" % x for x in [3.0] + f)]
    return "\n".join(out) + "\n"


# name: ([(lmax, PSEUDOPOTENTIAL_LOCAL)] of the types, ncell, h, rcut, steps, cube, threads)
CASES = {"none": ([(0, 0)], 1, 0.5, 7.0, 10, 29, 512), "s": ([(1, 1)], 1, 0.607, 4.8, 10, 17, 384),
         "spd": ([(3, 3)], 1, 0.5, 6.0, 10, 25, 384), "sp and sd": ([(2, 2), (2, 1)], 1, 0.607, 4.8, 10, 17, 384),
         "spd and pdf": ([(3, 3), (3, 0)], 1, 0.607, 4.8, 10, 17, 384), "32 atoms": ([(2, 2)], 2, 0.607, 4.8, 10, 17, 192)}


def _deck(path, name):
    types, ncell, h, rcut, q, _, _ = CASES[name]
    d, n, _ = make_fcc_mg_deck(str(path), "c", ncell=ncell, h=h, rcut=rcut, n_qp=q, disp=0.2, seed=21)
    folder = os.path.join(d, "pseudopotential")
    files = []
    for i, (lmax, _) in enumerate(types):
        files.append("psd_%d.pot" % i)
        with open(os.path.join(folder, files[-1]), "w") as f:
            f.write(_psd(os.path.join(folder, "psd_Mg.pot"), lmax))
    inpt = os.path.join(d, "c.inpt")
    text = open(inpt).read()
    text = text.replace("NTYPE: 1", "NTYPE: %d" % len(types))
    text = re.sub("PSEUDOPOTENTIAL_LOCAL: .*", "PSEUDOPOTENTIAL_LOCAL: " + " ".join(str(l) for _, l in types), text)
    text = re.sub("PSEUDOPOTENTIAL_FILE: .*", "PSEUDOPOTENTIAL_FILE: " + " ".join(files), text)
    with open(inpt, "w") as f:
        f.write(text)
    ion = open(os.path.join(d, "c.ion")).read().split("\n")
    atoms = [line for line in ion[3:] if line]
    share = np.array_split(atoms, len(types))
    with open(os.path.join(d, "c.ion"), "w") as f:
        f.write("%d\n\n" % len(atoms) + "".join("Mg 2 %d\n%s\n" % (len(a), "\n".join(a)) for a in share))
    return d, n


@pytest.mark.parametrize("name", CASES)
def test_plan(name, tmp_path):
    info = plan_kernel(*_deck(tmp_path, name))
    assert (info.kernel_layout, info.cube[0], info.kernel_threads) == (16, CASES[name][5], CASES[name][6])
    assert info.n_types == len(CASES[name][0])
    assert info.n_lm == {"none": 0, "s": 1, "spd": 9, "sp and sd": 9, "spd and pdf": 16, "32 atoms": 4}[name]


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
