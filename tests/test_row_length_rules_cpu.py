"""Where the longest row sends an SpMV from lanes per row to tiles.  Host logic only."""

import pytest

from flagsparse_b200 import _lib, spmv_csr as M


@pytest.mark.parametrize("size", [2, 8, 16])
def test_stored_types(size):
    # (rows, entries) -> longest row that still goes to lanes per row
    for n_rows, nnz, half, c64, c128 in ((4096, 1 << 16, 288, 288, 288), (1000, 200000, 1664, 2304, 2304), (0, 0, 288, 144, 144),
                                         (500000, 12000000, 288, 685, 1333), (2000000, 40000000, 288, 1142, 2222)):
        line = {2: half, 8: c64, 16: c128}[size]
        assert not M._uneven_rows(n_rows, nnz, line, size) and M._uneven_rows(n_rows, nnz, line + 1, size)


@pytest.mark.parametrize("size,line", [(4, 256), (8, 64)])
def test_small_matrices_of_native_types(size, line):
    for n_rows, mean in ((2000, 4), (4096, 16), (4096, 48)):
        longest = 8 * mean + line
        assert M._select_spmv_algo(n_rows, n_rows * mean, longest, size) == _lib.FSB_SPMV_VECTOR
        assert M._select_spmv_algo(n_rows, n_rows * mean, longest + 1, size) == _lib.FSB_SPMV_STREAM
