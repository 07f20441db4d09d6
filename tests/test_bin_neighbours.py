"""Neighbouring bin tiles that are cut alike and claimed side by side: two in a table
of few chunks, four in one of more than 22,750 (mapping 8)."""
import numpy as np
import pytest

from test_bin_items import bin_items, check_items

DCAP, ROWS = 160, 16


@pytest.mark.parametrize("groups,near", [(1, 2), (8, 4)])
def test_neighbours_are_cut_alike(groups, near):
    chunks = [1000, 700, 600, 650] * groups  # per tile; each pixel in one row
    lengths = np.repeat(np.array(chunks) * DCAP // ROWS, ROWS)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    col = np.concatenate([np.arange(r, n * DCAP, ROWS) for n in chunks for r in range(ROWS)])
    b = bin_items(8, rp, col)
    check_items(b, len(rp) - 1)
    assert b["first_chunk"][-1] == sum(chunks)
    tile = b["items"][:, 0] // ROWS
    pieces = np.bincount(tile).reshape(-1, near)
    assert np.all(pieces == pieces[:, :1])  # alike within a group
    cap = min(max(sum(chunks) // 350, 64), 96)
    want = [-(-max(chunks[i:i + near]) // cap) for i in range(0, len(chunks), near)]
    assert list(pieces[:, 0]) == want
    # a group's first pieces are claimed one after the other
    assert len(set(tile[:near] // near)) == 1 and len(set(tile[:near])) == near
