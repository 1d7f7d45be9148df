"""The split-pass kernel's walks and lists, restated on the CPU for every accepted cube and tile:
  * what a thread reads of P lies inside P, with P and U in either place (the 16-warp kernels exchange
    them every step) and with nothing behind them that a read beyond could rest on;
  * the dealing by bank class (bank_slot) gives every column of pass B and every list item one lane, and a
    quarter of a warp eight classes wherever each class has its share;
  * the list's items cover every quad of the owned planes once, their units and runs fit the words and
    the tensor memory's columns, and the batches of the dealing by number the bound of the planner."""
import numpy as np
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


# ---- dealing by bank class ----
def bank_slot(r, rank, groups, sizes):
    if rank < groups:
        return 8 * rank + r
    m = rank - groups + sum(max(0, sizes[i] - groups) for i in range(r))
    for i in range(8):
        free = max(0, groups - sizes[i])
        if m < free:
            return 8 * (sizes[i] + m) + i
        m -= free
    raise AssertionError("no place")


def block(threads):
    return threads if threads <= 256 else 384 if threads <= 384 else 512


def test_a_quad_has_the_bank_of_its_column():
    for nx, ny, nz in cubes():
        assert plane_floats(ny, (nx + 3) // 4 * 4) % 32 == 0


def test_pass_b_columns_each_get_one_lane():
    for nx, ny, nz, tile in plans():
        nq = (nx + 3) // 4
        ylen = -(-ny // tile)
        cols = [(c, z, q) for c in range(tile) for z in range(nz) for q in range(nq)]
        cls = [(c * ylen * nq + q) & 7 for c, z, q in cols]
        sizes = [cls.count(r) for r in range(8)]

        def of_class(c, r):
            first = (r - c * ylen * nq) & 7
            return (nq - first + 7) >> 3 if first < nq else 0

        assert sizes == [sum(of_class(c, r) for c in range(tile)) * nz for r in range(8)]
        groups = (len(cols) + 31) // 32 * 4
        lanes = set()
        for (c, z, q), r in zip(cols, cls):
            rank = (q >> 3) * nz + z + sum(of_class(i, r) for i in range(c)) * nz
            assert rank < sizes[r]
            lane = bank_slot(r, rank, groups, sizes)
            assert lane < 8 * groups and (rank >= groups or lane & 7 == r)
            lanes.add(lane)
        assert len(lanes) == len(cols)


# ---- the list ----
def list_chunks(columns, planes, threads):
    c = max(1, threads // columns)
    while c > 1 and planes // c < 4:
        c -= 1
    return c


def list_plans():
    for nx, ny, nz, tile in plans():
        nq = (nx + 3) // 4
        yield nx, ny, nz, max(64, 32 * -(-nq * max(ny, nz) * tile // 32))
    for n in (31, 33):  # each CTA of a pair
        yield n, n, (n + 1) // 2, 384
        yield n, n, n // 2, 384


def test_items_cover_the_columns_and_get_one_lane_each():
    rng = np.random.default_rng(1)
    for nx, ny, planes, threads in list_plans():
        nq, t = (nx + 3) // 4, block(threads)
        ncol = nq * ny
        nlc = list_chunks(ncol, planes, t)
        n_item = ncol * nlc
        assert n_item <= t
        for chunk in range(nlc):
            zb, ze = planes * chunk // nlc, planes * (chunk + 1) // nlc
            assert ze > zb and (nlc == 1 or ze - zb >= 4)
            top = max(ze, zb + 4)
            assert top <= max(planes, 4) and top - 4 - zb < 64 and ze - zb <= 127
        assert [planes * c // nlc for c in range(nlc + 1)][::nlc] == [0, planes]
        sizes = [nlc * ((ncol - i + 7) >> 3) for i in range(8)]
        assert sum(sizes) == n_item
        units = rng.integers(0, 9, n_item)
        lanes = set()
        for r in range(8):
            items = [i for i in range(n_item) if i // nlc & 7 == r]
            assert len(items) == sizes[r]
            for rank, i in enumerate(sorted(items, key=lambda i: (-units[i], i))):
                lanes.add(bank_slot(r, rank, t >> 3, sizes))
        assert len(lanes) == n_item and max(lanes) < t


@pytest.mark.parametrize("channels", [2, 3, 4])
@pytest.mark.parametrize("columns", [512, 256, 128])
def test_units_fit_the_tensor_memory(channels, columns):
    per_quarter = columns // (16 * channels + 4)
    rng = np.random.default_rng(columns + channels)
    for _ in range(50):
        w_units = rng.integers(0, 12, rng.integers(2, 17))
        quarter = [0] * 4
        used = [set() for _ in range(4)]
        for w, u in enumerate(w_units):
            q0 = quarter[w & 3]
            for k in range(max(0, min(u, per_quarter - q0))):
                t0, m0 = (q0 + k) * 16 * channels, per_quarter * 16 * channels + (q0 + k) * 4
                for c in list(range(t0, t0 + 16 * channels)) + list(range(m0, m0 + 4)):
                    assert c < columns and c not in used[w & 3]
                    used[w & 3].add(c)
            quarter[w & 3] += u


def test_batches_of_the_dealing_by_number_stay_within_the_bound():
    rng = np.random.default_rng(2)
    for nw in (2, 6, 12, 16):
        for _ in range(100):
            most = int(rng.integers(1, 40))
            units = np.sort(rng.integers(0, most + 1, 32 * nw))[::-1]
            batches = sum(int(units[32 * w]) for w in range(nw))
            assert batches <= int(units.sum()) // 32 + 2 * most + nw + 2
