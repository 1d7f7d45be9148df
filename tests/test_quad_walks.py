"""The split-pass kernel's walks through shared memory, restated on the CPU for every accepted cube and
tile: what a thread reads of P lies inside P, with P and U in either place (the 16-warp kernels exchange
them every step) and with nothing behind them that a read beyond could rest on."""
import pytest

O, MAX_THREADS = 6, 512
SMEM_OPTIN = 232448


def plane_floats(ny, pitch):
    return (ny * pitch + 31) // 32 * 32


def cubes():
    for n in range(3, 32, 2):
        yield n, n, n
    yield from [(17, 17, 69), (7, 7, 121), (7, 61, 7), (25, 27, 31), (31, 9, 5)]


def plans():
    for nx, ny, nz in cubes():
        nq = (nx + 3) // 4
        for tile in range(1, 5):
            if nq * max(ny, nz) * tile <= MAX_THREADS and 8 * plane_floats(ny, 4 * nq) * nz < SMEM_OPTIN:
                yield nx, ny, nz, tile


def z_ranges(nz, tile):
    """(first plane, live planes, planes that every lane walks) of pass A's ranges in use."""
    zlen = -(-nz // tile)
    for c in range(tile):
        zb = min(nz, c * zlen)
        if zb < min(nz, zb + zlen):
            yield zb, min(nz, zb + zlen) - zb, zlen


def test_pass_a_reads_stay_in_the_vector():
    beyond = 0
    for nx, ny, nz, tile in plans():
        nq, ps = (nx + 3) // 4, plane_floats(ny, (nx + 3) // 4 * 4)
        alloc = ps * max(nz, 4)
        for zb, live, zlen in z_ranges(nz, tile):
            for i in range(zlen):
                plane = zb + min(i, live - 1)     # of the x neighbours
                assert zb <= plane < nz
                last = (plane * ps + (ny - 1) * 4 * nq + 4 * (nq - 1)) + 3
                assert 0 <= plane * ps and last < alloc
                beyond += (zb + i + 1) * ps > alloc  # a walk that went on would leave the vector
                if i < nz - O - zb:               # the plane that joins the ring
                    assert zb + i + O < nz
    assert beyond
