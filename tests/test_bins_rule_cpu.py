"""When a prepared matrix takes the two-pass SpMV: sizes, evenness of the rows, value type."""

import pytest
import torch

from flagsparse_b200 import bins

M = 1 << 20


@pytest.mark.parametrize("nnz,rows,longest,size,lanes,want", [
    (16 * M, M, 16, 4, True, 2 * M),             # even rows from 2^24 entries on
    (16 * M - 1, M, 16, 4, True, None),
    (16 * M, M, 40, 4, True, 2 * M),             # Poisson(16) over a million rows
    (5 * M // 2, M, 64, 4, True, M),             # uneven rows earlier
    (5 * M // 2 - 1, M, 64, 4, True, None),
    (16 * M, M, 16, 8, True, 120 * M),           # float64: an x that L2 does not hold
    (8 * M, M, 16, 8, True, None),
    (4 * M, 2 * M, 63, 8, True, M),              # float64, uneven rows of two entries on lanes
    (4 * M, 2 * M, 63, 8, False, None),
])
def test_span(nnz, rows, longest, size, lanes, want):
    assert bins.min_span(nnz, rows, longest, size, lanes) == want


@pytest.mark.parametrize("nnz,rows,longest,want", [
    (16 * M, M, 16, 1 << 16),
    (10 * M, 30 * M, 30, 1 << 16),               # mostly empty rows, 427 blocks by entries
    (16 * M, 64 * M, 9, 1 << 17),                # a quarter of an entry per row: 98 k rows in a block by entries are not cut
    (3 * M, 512 * M, 9, 1 << 20),
])
def test_rows_of_a_block(nnz, rows, longest, want):
    step, most = bins.cuts(nnz, rows, longest, 24576)
    assert step == 24576 - longest + 1 and most == want


@pytest.mark.parametrize("begin,n_rows,most,want", [
    ([0], 5, 10, [0, 5]),
    ([0, 10, 20], 30, 10, [0, 10, 20, 30]),                  # as long as allowed: not cut
    ([0, 10, 21], 30, 10, [0, 10, 15, 21, 30]),
    ([3, 4, 4, 40], 70, 10, [0, 4, 13, 22, 31, 40, 50, 60, 70]),      # leading rows, an empty block, runs of empty rows
    ([0, 80], 70, 100, [0, 70]),                             # nothing starts that far behind
])
def test_rows_cut(begin, n_rows, most, want):
    assert bins._cut_rows(torch.tensor(begin), n_rows, most).tolist() == want
