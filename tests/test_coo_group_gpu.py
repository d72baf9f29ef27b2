"""fsb_coo_group: triples grouped by row against numpy's stable sorts -- sizes around a tile and a digit, every id and value
width, hot rows, ids out of range."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import coo
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("by_column", [False, True])
@pytest.mark.parametrize("nnz,n_rows,n_cols,vdt,rt,ct", [
    (1, 1, 1, "float32", "int64", "int64"), (33, 2, 5, "float64", "int32", "int64"), (4095, 512, 3, "float16", "int64", "int32"),
    (4096, 513, 1 << 20, "complex128", "int32", "int32"), (4097, 300000, 700, "complex64", "int64", "int64"),
    (100003, 77, 100001, "float32", "int32", "int64"), (300001, 1 << 27, 1 << 19, "float64", "int64", "int32"),
])
def test_against_stable_sorts(cuda, fsb_lib, nnz, n_rows, n_cols, vdt, rt, ct, by_column):
    rng = np.random.default_rng(nnz)
    row, col = rng.integers(0, n_rows, nnz), rng.integers(0, n_cols, nnz)
    row[rng.random(nnz) < 0.3] = n_rows // 2                              # a hot row
    row[-1], col[0] = n_rows - 1, n_cols - 1
    val = np.arange(nnz).astype(vdt)                                      # tells equal ids apart
    g = coo._group(dev(val), dev(row.astype(rt)), dev(col.astype(ct)), n_rows, n_cols, by_column)
    order = np.lexsort((col, row)) if by_column else np.argsort(row, kind="stable")
    assert np.array_equal(g.row.cpu().numpy(), row[order]) and np.array_equal(g.col.cpu().numpy(), col[order])
    assert np.array_equal(g.data.cpu().numpy(), val[order])
    lens = np.bincount(row, minlength=n_rows)
    ptr = g.indptr.cpu().numpy()
    assert ptr[0] == 0 and np.array_equal(np.diff(ptr), lens)
    s = g.stats
    assert (s.ptr_first, s.ptr_last, s.n_decreasing, s.min_index, s.max_index) == (0, nnz, 0, col.min(), col.max())
    assert (g.min_row, g.max_row, s.max_row_nnz, s.n_empty_rows) == (row.min(), row.max(), lens.max(), (lens == 0).sum())
    assert s.n_long_rows == (lens > max(64, 32 * -(-nnz // n_rows))).sum()


@pytest.mark.parametrize("nnz", [2047, 2048, 2049, (3 << 20) - 1, 3 << 20, (3 << 20) + 1])
def test_tiles_of_both_sizes(cuda, fsb_lib, nnz):
    rng = np.random.default_rng(nnz)
    row, col = rng.integers(0, 3000, nnz), rng.integers(0, 50000, nnz)
    for by_column in (False, True):
        g = coo._group(dev(np.arange(nnz).astype(np.float64)), dev(row), dev(col.astype(np.int32)), 3000, 50000, by_column)
        order = np.lexsort((col, row)) if by_column else np.argsort(row, kind="stable")
        assert np.array_equal(g.data.cpu().numpy(), order) and np.array_equal(g.col.cpu().numpy(), col[order])
        assert np.array_equal(np.diff(g.indptr.cpu().numpy()), np.bincount(row, minlength=3000))


@pytest.mark.parametrize("bad_row,bad_col,message", [(-1, 0, "row"), (50, 0, "row"), (2**40, 0, "row"), (0, -5, "col"),
                                                     (0, 60, "col"), (-1, 60, "row")])
def test_ids_out_of_range_are_refused(cuda, fsb_lib, bad_row, bad_col, message):
    row, col = np.arange(5000) % 50, np.arange(5000) % 60
    row[4321], col[1234] = bad_row, bad_col
    triple = (dev(np.ones(5000, dtype=np.float32)), dev(row), dev(col))
    B = torch.ones((60, 8), device=cuda)
    with pytest.raises(IndexError, match=message):
        fs.flagsparse_spmm_coo(*triple, B, (50, 60))
    with pytest.raises(IndexError, match=message):
        fs.flagsparse_spmv_coo(*triple, B[:, 0].contiguous(), (50, 60))
    with pytest.raises(IndexError, match=message):
        fs.prepare_spmv_coo(*triple, (50, 60), sort_by_row=False)
    torch.cuda.synchronize()
