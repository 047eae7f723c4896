"""Index arithmetic of the plane kernel's split phases (plane.cuh; FP64 grids whose plane does not
fit in shared memory), enumerated on the CPU for every such size: all accesses lie in their buffers,
the column blocks of a plane write each place of the scratch lines once, and the line phase reads and
writes the places that they wrote. The arithmetic between the exchanges is that of the unsplit
kernel, whose numpy model (test_plane_model.py) is run here at these sizes as well."""
import numpy as np
import pytest

from tests.test_plane_model import test_phases_give_the_direct_d_apply as phases
from tests.test_plane_model import test_transform_of_a_real_field_and_back as transforms

SIZES = [160, 176, 192, 208, 224, 240, 256]
T = 8  # columns per tile of a column phase


def split(n):
    r2 = 16
    r1, nq = n // r2, n // 2
    ps2 = n + r1
    assert r1 * r2 == n and r1 <= 16 and nq * ps2 * 16 > 200 * 1024
    tc = 16 if nq % 16 == 0 else 8
    buf = max(2 * n * T, 4 * 512 // 2, 16 * ps2)  # column tiles, partial sums, line pairs
    assert (buf + 3 * n + n // 2) * 16 <= 227 * 1024
    return r1, r2, nq, ps2, tc, buf


@pytest.mark.parametrize("n", SIZES)
def test_column_blocks_and_lines_meet_in_the_scratch_lines(n):
    r1, r2, nq, ps2, tc, buf = split(n)
    nh = nq + 1
    written = np.zeros((nq, n), int)  # the lines of one plane and component
    seen_in = np.zeros((n, nh), int)
    assert nq % tc == 0
    for cb in range(nq // tc):
        # y inverse: R1-point tasks (b, c), inputs G[(R2 a + b) nh + column], into shared memory
        b, c, a = np.meshgrid(np.arange(r2), np.arange(tc), np.arange(r1), indexing="ij")
        col = cb * tc + c
        flat = (r2 * a + b) * nh + col
        assert flat.min() >= 0 and flat.max() < n * nh
        np.add.at(seen_in.reshape(-1), flat, 1)
        place = b * tc + c + a * (r2 * tc)  # task's result k1 = a
        assert place.max() < buf and np.unique(place).size == place.size
        # R2-point tasks (k1, c), pairs of rows into the two lines of a pair
        k1, c, q = np.meshgrid(np.arange(r1), np.arange(tc), np.arange(r2), indexing="ij")
        src = k1 * r2 * tc + c + (q >> 1) * (2 * tc) + (q & 1) * tc
        assert np.array_equal(np.sort(src, axis=None), np.sort(place, axis=None))
        cc = cb * tc + c
        d = np.where(cc == 0, nq, n - cc) - cc
        w = cb * tc + k1 * (r2 // 2) * n + c + (q >> 1) * n + (q & 1) * d
        assert w.min() >= 0 and w.max() < nq * n
        np.add.at(written.reshape(-1), w, 1)
    assert (written == 1).all()
    assert (seen_in[:, :nq] == 1).all() and (seen_in[:, nq] == 0).all()
    # the last plane of the last component ends where the scratch does
    assert ((2 * n + n - 1) * nq + nq - 1) * n + n - 1 == 3 * n * nq * n - 1
    # a pair's line: thread t holds places t + R2 a; its shared row has one gap after R2 places
    t, a = np.meshgrid(np.arange(r2), np.arange(r1), indexing="ij")
    assert np.array_equal(np.sort(t + r2 * a, axis=None), np.arange(n))
    row = t + (r2 + 1) * a
    groups = 8 * (32 // r2)  # of 8 warps: 256 threads
    assert groups == 16 and (groups - 1) * ps2 + row.max() < buf and row.max() < ps2
    k1, k2 = np.meshgrid(np.arange(r1), np.arange(r2), indexing="ij")
    assert np.array_equal(np.sort(k1 * (r2 + 1) + k2, axis=None), np.sort(row, axis=None))
    # the pair's two real lines, every voxel of the plane once
    pr = np.arange(nq)
    y0 = 2 * pr // r2 + r1 * (2 * pr % r2)
    assert np.array_equal(np.sort(np.concatenate([y0, y0 + r1])), np.arange(n))
    assert np.array_equal(np.sort(k1 + r1 * k2, axis=None), np.arange(n))


@pytest.mark.parametrize("n", SIZES)
def test_column_tiles(n):
    r1, r2, nq, ps2, tc, buf = split(n)
    pl = n * (nq + 1)
    tiles = -(-pl // T)
    task = np.arange(2 * T * r2)
    c, ib = task % T, task // T
    i, b = ib // r2, ib % r2
    assert set(i) == {0, 1}
    place = (i * n * T + b * T + c)[:, None] + r2 * T * np.arange(r1)
    assert place.max() < buf and np.unique(place).size == place.size
    task = np.arange(T * r1)
    c, k1 = task % T, task // T
    inner = (k1 * r2 * T + c)[:, None] + T * np.arange(r2)
    assert np.unique(inner).size == inner.size == n * T and inner.max() < n * T
    q = np.arange(tiles * T)
    assert q[q < pl].size == pl  # the last tile's columns past the plane are left out


@pytest.mark.parametrize("n", SIZES[1:])
def test_arithmetic_at_the_split_sizes(n):
    phases(n, False)
    transforms(n)
