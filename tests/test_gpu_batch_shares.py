"""A batch's split of the SMs between cells whose kernels run different numbers of CTAs on an SM: the
plan on the CPU, and on the GPU cells of one, two and three CTAs per SM in one submission (a node is
computed by one CTA without atomics, so the results are those of one call per cell, bit by bit)."""
import ctypes

import numpy as np
import pytest

from sqminiapp_gb300.capi import SQ_BAD_INPUT, lib


def _plan(cost, nodes, ctas, sms):
    n = len(cost)
    out = (ctypes.c_int * n)()
    st = lib().sq_plan_batch((ctypes.c_double * n)(*cost), (ctypes.c_long * n)(*nodes), (ctypes.c_int * n)(*ctas),
                             n, sms, out)
    return st, list(out)


@pytest.mark.parametrize("ctas", [(1, 1), (1, 3), (4, 2)])
def test_equal_work_gets_equal_shares(ctas):
    st, share = _plan([2.0, 2.0], [100000, 100000], ctas, 152)
    assert st == 0 and sum(share) == 152 and abs(share[0] - share[1]) <= 2


def test_shares_follow_cost_and_stop_at_the_nodes():
    st, share = _plan([1.0, 3.0], [40000, 40000], (3, 1), 152)
    assert st == 0 and sum(share) == 152 and abs(share[1] - 114) <= 2
    st, share = _plan([1.0, 1.0], [2, 3], (1, 2), 152)
    assert st == 0 and all(1 <= s <= n for s, n in zip(share, (2, 3)))


def test_bad_input_is_refused():
    for cost, nodes, ctas, sms in (([0.0], [1], [1], 152), ([1.0], [0], [1], 152), ([1.0], [1], [0], 152),
                                   ([1.0, 1.0], [1, 1], [1, 1], 1)):
        assert _plan(cost, nodes, ctas, sms)[0] == SQ_BAD_INPUT


@pytest.mark.gpu
def test_cells_of_several_ctas_per_sm(tmp_path):
    import torch
    from sqminiapp_gb300 import LSDFT, batch_nodes_and_weights
    from sqminiapp_gb300.decks import make_fcc_mg_deck
    cells = []
    for i, (h, rcut) in enumerate([(0.5, 6.0), (0.607, 4.8), (0.85, 3.4)]):  # 25^3, 17^3, 9^3 cubes
        d, name, _ = make_fcc_mg_deck(str(tmp_path / str(i)), "c", ncell=1, h=h, rcut=rcut, n_qp=12, disp=0.2, seed=i)
        cells.append(LSDFT(d, name, precision=32))
    veffs, outs, refs = [], [], []
    for e in cells:
        v = -0.2 + 0.05 * np.random.default_rng(e.n_nodes).standard_normal(e.n_nodes)
        refs.append(e.NodesAndWeights_LSSGQ(veff=v))
        veffs.append(torch.from_numpy(v).cuda())
        outs.append({k: torch.empty(s, dtype=torch.float64, device="cuda") for k, s in
                     (("lambda", (e.n_nodes, e.n_qp)), ("weights", (e.n_nodes, e.n_qp)),
                      ("lambda_min", (e.n_nodes,)), ("lambda_max", (e.n_nodes,)))})
    torch.cuda.synchronize()
    for order in ([0, 1, 2], [2, 1, 0]):  # the second split uses the measured node costs
        batch_nodes_and_weights([cells[i] for i in order], [veffs[i].data_ptr() for i in order], None,
                                [{k: t.data_ptr() for k, t in outs[i].items()} for i in order],
                                torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for o, r in zip(outs, refs):
            for k in r:
                assert np.array_equal(o[k].cpu().numpy(), r[k]), k
            for t in o.values():
                t.zero_()
        torch.cuda.synchronize()
    for e in cells:
        e.close()
