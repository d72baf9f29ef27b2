"""When a prepared matrix takes the two-pass SpMV: sizes, evenness of the rows, value type."""

import pytest

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
