"""Where the longest row sends an SpMV from lanes per row to tiles.  Host logic only."""

import pytest

from flagsparse_b200 import spmv_csr as M


@pytest.mark.parametrize("size", [2, 8, 16])
def test_stored_types(size):
    # (rows, entries) -> longest row that still goes to lanes per row: a floor, a multiple of the mean, a share of the entries
    for n_rows, nnz, line in ((4096, 1 << 16, 288), (1000, 200000, 1664), (0, 0, 288),
                              (2000000, 40000000, {2: 288, 8: 1142, 16: 2222}[size])):
        assert not M._uneven_rows(n_rows, nnz, line, size) and M._uneven_rows(n_rows, nnz, line + 1, size)
