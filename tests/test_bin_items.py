"""The work items of the bin tiles (mappings 7 and 8), laid out on the host: every
item stages at least one chunk (an item without any is never seen by the warps
that sum, so its tile would never be written), and the pieces of a tile join
without a gap for every row and both fold cadences. The tables are those whose
small tiles lie beside large ones: few azimuthal sectors with a radial range that
ends inside the detector, a beam near a corner, few inner pixels left by a mask."""
import ctypes as C
import math

import numpy as np
import pytest

from dioptrin_b200 import _native as N


def bin_items(variant, row_ptr, col):
    rp = np.ascontiguousarray(row_ptr, np.int64)
    col = np.ascontiguousarray(col, np.int32)
    n = len(rp) - 1
    counts = np.zeros(5, np.int64)

    def call(*arrays):
        N.check(N.lib().dg_test_bin_items(
            variant, n, rp.ctypes.data, col.ctypes.data, counts.ctypes.data,
            *[a.ctypes.data if a is not None else None for a in arrays]))

    call(*[None] * 5)
    items, rows, tiles, parts, _ = (int(v) for v in counts)
    out = dict(rows=rows, items=np.zeros((items, 4), np.int32),
               first_chunk=np.zeros(tiles + 1, np.int64),
               spans=np.zeros((2, items, rows, 4), np.int32),
               row_part=np.zeros(n + 1, np.int32), part_ids=np.zeros(parts, np.int32))
    call(out["items"], out["first_chunk"], out["spans"] if parts else None, out["row_part"],
         out["part_ids"])
    return out


def check_items(b, n_rows):
    rows, items, first = b["rows"], b["items"], b["first_chunk"]
    assert np.all(items[:, 3] >= 1), "items without chunks"
    tile = items[:, 0] // rows
    assert np.array_equal(items[:, 0], tile * rows)
    assert np.array_equal(items[:, 1], np.minimum(rows, n_rows - items[:, 0]))
    assert np.all(items[:, 2] >= first[tile]) and np.all(items[:, 2] + items[:, 3] <= first[tile + 1])
    if not len(b["part_ids"]):  # whole tiles, one item each
        assert np.array_equal(np.sort(tile), np.arange(len(first) - 1))
        assert np.array_equal(items[:, 3], np.diff(first)[tile])
        return 0
    pieces = np.bincount(tile, minlength=len(first) - 1)
    assert np.all(pieces >= 1)
    assert np.array_equal(np.diff(b["row_part"]), pieces[np.arange(n_rows) // rows])
    for r in range(n_rows):
        ids = b["part_ids"][b["row_part"][r]:b["row_part"][r + 1]]
        mine = ids // rows
        assert np.all(ids % rows == r % rows) and np.all(tile[mine] == r // rows)
        assert len(set(mine)) == len(mine)
        n_chunks = int(first[r // rows + 1] - first[r // rows])
        if len(mine) == 1:  # an uncut tile
            assert items[mine[0], 3] == n_chunks
        for cadence in range(2):
            at = (0, 0)
            for i in mine:
                c0, p0, c1, p1 = (int(v) for v in b["spans"][cadence, i, r % rows])
                if len(mine) == 1:
                    assert (c0, p0) == (0, 0) and c1 >= n_chunks
                    at = (n_chunks, 0)
                    continue
                if (c0, p0) >= (c1, p1):
                    continue  # the row has no work in this piece
                base = int(items[i, 2] - first[r // rows])
                assert (base + c0, p0) == at
                assert c0 >= 0 and c1 + (p1 > 0) <= items[i, 3]  # in the chunks it stages
                at = (base + c1, p1)
            assert at == (n_chunks, 0)
    return int(pieces.max())


def sectors(oracle, shape, method, bins, azimuthal):
    """Few sectors, the beam at the centre, a radial range that ends inside."""
    px, dist = 172e-6, 0.2
    p = oracle.poni(pixel1=px, pixel2=px, distance=dist, poni1=0.5 * shape[0] * px,
                    poni2=0.5 * shape[1] * px, wavelength=1e-10)
    g = oracle.grid2d_for(p, *shape, method, bins, azimuthal, n_ss=2,
                          radial_range=(1e-4, math.atan(0.48 * shape[1] * px / dist)))
    return oracle.build_2d(p, *shape, method, g, n_ss=2)


def corner_beam(oracle, shape, off, bins):
    px = 172e-6
    p = oracle.poni(pixel1=px, pixel2=px, distance=0.2, poni1=off * px, poni2=off * px,
                    wavelength=1e-10)
    return oracle.build_ps1d(p, *shape, bins)


@pytest.mark.parametrize("variant,shape,method,bins,azimuthal", [
    (8, (1043, 981), "pixel_split", 496, 4),
    (8, (1043, 981), "pixel_split", 368, 2),
    (8, (2167, 2070), "counting", 500, 8),
    (7, (2167, 2070), "counting", 1000, 4),
])
def test_few_sectors(oracle, variant, shape, method, bins, azimuthal):
    t = sectors(oracle, shape, method, bins, azimuthal)
    assert check_items(bin_items(variant, t.row_ptr, t.col), t.n_rows) > 1


@pytest.mark.parametrize("variant", [7, 8])
@pytest.mark.parametrize("shape,off,bins", [
    ((701, 899), 10, 50), ((701, 899), 30, 50), ((1043, 981), 10, 82), ((1043, 981), 60, 82)])
def test_beam_near_a_corner(oracle, variant, shape, off, bins):
    t = corner_beam(oracle, shape, off, bins)
    assert check_items(bin_items(variant, t.row_ptr, t.col), t.n_rows) > 1


@pytest.mark.parametrize("variant", [7, 8])
@pytest.mark.parametrize("left", [0.0, 0.002, 0.01])
def test_few_inner_pixels_left(oracle, variant, left):
    """A mask that leaves a small share of the first tile's pixels, or none."""
    t = corner_beam(oracle, (1043, 981), 500.3, 100)
    rng = np.random.default_rng(3)
    rows = 24 if variant == 7 else 16
    mask = np.zeros(1043 * 981, np.uint8)
    inner = np.unique(t.col[:t.row_ptr[rows]])
    mask[inner[rng.random(inner.size) >= left]] = 1
    t = oracle.compact(t, mask)
    assert check_items(bin_items(variant, t.row_ptr, t.col), t.n_rows) > 1


def test_small_tables():
    """Whole tiles, rows without entries, one row."""
    for rp in ([0, 1], [0, 0, 0, 5, 5], np.arange(0, 100)):
        rp = np.array(rp, np.int64)
        for variant in (7, 8):
            assert check_items(bin_items(variant, rp, np.arange(rp[-1])), len(rp) - 1) == 0
    with pytest.raises(ValueError, match="7 and 8"):
        bin_items(3, np.array([0, 1]), np.array([0]))
