"""The split-pass kernel on meshes of unequal spacings: cubes of more planes than the list's words could
count from the cube's first plane (67), on one CTA and on a pair, of few planes and many rows, and the
kernels for three different spacings, with every channel set the Mg pseudopotential gives.

Tolerance.  As in test_gpu_quad_list: about 50 roundings of 2^-24 on terms of up to twice the stencil's
diagonal D (18 at h = 0.5, more in the direction of the finest spacing), 50 * 2 D * 6e-8 on the first
coefficients; the moments of order <= 3 relative to max(1, |value|) 1e-4 (their third power of D
cancels against the value's own)."""
import re

import numpy as np
import pytest

from sqminiapp_gb300 import plan_kernel
from sqminiapp_gb300.decks import make_fcc_mg_deck

# FD_GRID, rcut, steps, PSEUDOPOTENTIAL_LOCAL, cube, layout (16 one CTA, 48 a pair)
CASES = [((12, 12, 54), 5.2, 10, 2, (17, 17, 69), 16), ((10, 10, 60), 5.2, 10, 1, (15, 15, 75), 16),
         ((13, 13, 66), 5.0, 10, 0, (17, 17, 79), 16), ((6, 6, 120), 4.2, 10, 2, (7, 7, 121), 16),
         ((15, 15, 60), 5.6, 8, 2, (21, 21, 81), 48), ((5, 60, 5), 4.2, 10, 1, (7, 61, 7), 16),
         ((13, 17, 15), 5.0, 10, 0, (17, 21, 19), 16), ((18, 16, 14), 4.5, 10, 2, (21, 19, 17), 16)]
# with one range per row: a thread per column would own 69 planes
ONE_RANGE = ((2, 68, 68), 4.2, 8, 2, (3, 69, 69), 16)


def _deck(path, grid, rcut, q, lloc):
    d, name, _ = make_fcc_mg_deck(str(path), "c", ncell=1, h=0.5, rcut=rcut, n_qp=q, disp=0.2, seed=sum(grid), lloc=lloc)
    f = path / "c.inpt"
    f.write_text(re.sub(r"FD_GRID: .*", "FD_GRID: %d %d %d" % grid, f.read_text()))
    return d, name


def _list_chunks(columns, planes, threads):
    c = max(1, threads // columns)
    while c > 1 and planes // c < 4:
        c -= 1
    return c


@pytest.mark.parametrize("grid,rcut,q,lloc,cube,layout,tile", [c + (0,) for c in CASES] + [ONE_RANGE + (1,)])
def test_plan_and_word_widths(grid, rcut, q, lloc, cube, layout, tile, tmp_path):
    """CPU: the planned kernel, and a unit's first plane within 6 bits of its item's first one."""
    info = plan_kernel(*_deck(tmp_path, grid, rcut, q, lloc), kernel=2, tile=tile)
    assert tuple(info.cube) == cube and info.kernel_layout == layout
    planes = cube[2] if layout == 16 else (cube[2] + 1) // 2
    columns = (cube[0] + 3) // 4 * cube[1]
    chunks = _list_chunks(columns, planes, info.kernel_threads)
    assert columns * chunks <= info.kernel_threads
    for c in range(chunks):
        zb, ze = planes * c // chunks, planes * (c + 1) // chunks
        assert max(ze, zb + 4) - 4 - zb < 64


@pytest.mark.gpu
@pytest.mark.parametrize("grid,rcut,q,lloc,cube,layout,tile", [c + (0,) for c in CASES] + [ONE_RANGE + (1,)])
def test_against_oracle(grid, rcut, q, lloc, cube, layout, tile, tmp_path, oracle_mod):
    from sqminiapp_gb300 import LSDFT
    d, name = _deck(tmp_path, grid, rcut, q, lloc)
    o = oracle_mod.Oracle(d, name, faithful=False)
    nodes = np.arange(0, o.n_nodes, max(1, o.n_nodes // 11))
    veff = -0.3 + 0.1 * np.random.default_rng(q).standard_normal(o.n_nodes)
    ref = o.nodes_and_weights(nodes=nodes, veff=veff, want_ab=True)
    with LSDFT(d, name, faithful=False, precision=32, kernel=2, tile=tile) as eng:
        assert eng.cube == cube and eng.info.kernel_layout == layout
        out = eng.NodesAndWeights_LSSGQ(veff=veff)
        a, b = eng.lanczos_coefficients(eng.n_nodes)
        again = eng.NodesAndWeights_LSSGQ(veff=veff)
        diag = sum(1.4913888888888889 / h ** 2 for h in eng.h)  # sum of 1/p^2, p = 1..6
    tol = 50 * 2 * diag * 6e-8
    np.testing.assert_allclose(a[nodes, :4], ref["a"][:, :4], rtol=0, atol=tol)
    np.testing.assert_allclose(b[nodes, :4], ref["b"][:, :4], rtol=0, atol=tol)
    for k in range(4):
        g = np.sum(out["weights"][nodes] * out["lambda"][nodes] ** k, axis=1)
        e = np.sum(ref["weights"] * ref["lambda"] ** k, axis=1)
        assert np.max(np.abs(g - e) / np.maximum(1.0, np.abs(e))) < 1e-4, k
    for k in out:
        assert np.array_equal(out[k], again[k]), k
