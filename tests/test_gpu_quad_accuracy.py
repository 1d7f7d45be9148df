"""Accuracy of the split-pass FP32 kernel on single nodes, where no average over nodes hides one that
is off: the quadrature weights of 24 nodes of the 32-atom cell (27^3 cubes, 40 steps), each against the
FP64 oracle, in ascending order of the Ritz values.

Tolerance.  The recurrence restated on the CPU with the kernel's roundings, 144 nodes: relative error
(2-norm) of a node's weights 2.3e-7 root mean square and 5.6e-7 at most; 1e-6 leaves room for another
order of the sums.  With the stencil's constant diagonal inside the FP32 products they were 1.1e-6 and
2.6e-6.  The lowest Ritz value: 8e-8 Ha at most over 120 nodes of other meshes, so 3e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [3, 4])
def test_single_nodes_against_fp64(seed, tmp_path, oracle_mod):
    from sqminiapp_gb300 import LSDFT
    from sqminiapp_gb300.decks import make_fcc_mg_deck
    d, name, _ = make_fcc_mg_deck(str(tmp_path), "c", ncell=2, h=0.5, rcut=6.5, n_qp=40, disp=0.15, seed=seed)
    o = oracle_mod.Oracle(d, name, faithful=False)
    r = np.random.default_rng(seed)
    x = np.arange(34) * (2 * np.pi / 34)
    veff = np.full((34, 34, 34), -0.6)
    for _ in range(40):
        k, a, ph = r.integers(-4, 5, 3), 0.05 * r.standard_normal(), r.uniform(0, 2 * np.pi)
        veff += a * np.cos(k[2] * x[:, None, None] + k[1] * x[None, :, None] + k[0] * x[None, None, :] + ph)
    veff = veff.reshape(-1)
    nodes = np.sort(r.choice(o.n_nodes, 12, replace=False))
    ref = o.nodes_and_weights(nodes=nodes, veff=veff)
    o.close()
    with LSDFT(d, name, faithful=False, precision=32) as eng:
        assert eng.info.kernel_layout & 16
        for i, node in enumerate(nodes):
            out = eng.NodesAndWeights_LSSGQ(veff=veff, node_begin=int(node), node_end=int(node) + 1)
            g, e = np.argsort(out["lambda"][0]), np.argsort(ref["lambda"][i])
            w, we = out["weights"][0][g], ref["weights"][i][e]
            assert np.linalg.norm(w - we) < 1e-6 * np.linalg.norm(we), node
            assert abs(out["lambda"][0][g[0]] - ref["lambda"][i][e[0]]) < 3e-7, node
