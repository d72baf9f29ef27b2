"""The tiled kernels at the sizes where they can go wrong: rows around the length from which a block shares them, around
a tile and over several tiles, every value type, widths that take one or several accesses per lane, arrays that start
off a 16-byte boundary.  Reference: the product of the stored values in complex128."""

import numpy as np
import pytest
import scipy.sparse as sp
import torch

import flagsparse_b200 as fs
from helpers import handmade_csr

pytestmark = pytest.mark.gpu

DTYPES = (torch.float32, torch.float64, torch.float16, torch.bfloat16, torch.complex64, torch.complex128)
# unit roundoff of the sums and of the stored result
SUM_U = {torch.float16: 2.0 ** -24, torch.bfloat16: 2.0 ** -24, torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53,
         torch.complex64: 2.0 ** -24, torch.complex128: 2.0 ** -53}
STORE_U = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}
LENS = {
    "shared": [64, 65, 0, 128, 129, 1, 256, 257, 0, 0, 63, 40, 500],
    "tiles": [1023, 1, 1024, 0, 1025, 2047, 2048, 2049, 0, 7],
    "crossing": [5000, 0, 0, 300, 3, 9000, 0],
    "one": [4097],
    "empty_ends": [0] * 3000 + [700, 0, 70] + [0] * 3000,
}


def _values(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(-1, 1, shape)
    if dtype.is_complex:
        v = v + 1j * rng.uniform(-1, 1, shape)
    return torch.from_numpy(v).to(dtype)


def _check(got, vals, i, p, n_cols, operand, dtype):
    a = sp.csr_matrix((vals.cpu().to(torch.complex128).numpy(), i, p), shape=(len(p) - 1, n_cols))
    o = operand.cpu().to(torch.complex128).numpy()
    ref, mag = np.asarray(a @ o), np.asarray(abs(a) @ np.abs(o))
    n = np.diff(p).reshape((-1,) + (1,) * (ref.ndim - 1))
    # a sum of n products in any order: (n + 1) u |A||B|, times 4 for the four products of a complex one
    bound = (4 if dtype.is_complex else 1) * (n + 1) * SUM_U[dtype] * mag
    if dtype in STORE_U:
        bound = bound * (1 + STORE_U[dtype]) + STORE_U[dtype] * np.abs(ref) + (2.0 ** -25 if dtype == torch.float16 else 0)
    err = np.abs(got.cpu().to(torch.complex128).numpy() - ref)
    assert got.dtype == dtype and np.all(err <= bound * 1.0001), float((err - bound).max())


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
@pytest.mark.parametrize("name", sorted(LENS))
def test_spmm_rows_shared_by_a_block(cuda, fsb_lib, dtype, name):
    n_cols = 12000
    _, i, p = handmade_csr(3, LENS[name], n_cols)
    vals = _values(int(p[-1]), dtype, 4)
    d, ti, tp = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda)
    for n_dense in (1, 8, 33, 40, 101, 128, 200):
        B = _values((n_cols, n_dense), dtype, n_dense)
        C = fs.flagsparse_spmm_csr(d, ti, tp, B.to(cuda), (len(p) - 1, n_cols))
        _check(C, vals, i, p, n_cols, B, dtype)
        # the same columns as part of wider rows: narrower accesses, the same order of additions
        wide = torch.zeros((n_cols, n_dense + 3), dtype=dtype, device=cuda)
        wide[:, 1:n_dense + 1] = B.to(cuda)
        assert torch.equal(fs.flagsparse_spmm_csr(d, ti, tp, wide[:, 1:n_dense + 1], (len(p) - 1, n_cols)), C)
        # 64-bit column indices and row pointers
        assert torch.equal(fs.flagsparse_spmm_csr(d, ti.long(), tp.long(), B.to(cuda), (len(p) - 1, n_cols)), C)


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
@pytest.mark.parametrize("name", sorted(LENS) + ["even"])
def test_spmv_of_even_and_uneven_rows(cuda, fsb_lib, dtype, name):
    n_cols = 12000
    lens = [17, 16, 15, 18, 20, 3, 0, 31] * 300 + [5] if name == "even" else LENS[name]
    _, i, p = handmade_csr(5, lens, n_cols)
    vals, x = _values(int(p[-1]), dtype, 6), _values(n_cols, dtype, 7)
    d, ti, tp, tx = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), x.to(cuda)
    shape = (len(p) - 1, n_cols)
    y = fs.flagsparse_spmv_csr(d, ti, tp, tx, shape)
    _check(y, vals, i, p, n_cols, x, dtype)
    assert torch.equal(fs.flagsparse_spmv_csr(d, ti.long(), tp.long(), tx, shape), y)
    # arrays that start one element behind a boundary
    off = lambda t: torch.cat([t[:1], t])[1:]                                        # noqa: E731
    _check(fs.flagsparse_spmv_csr(off(d), off(ti), off(tp), off(tx), shape), vals, i, p, n_cols, x, dtype)
    prep = fs.prepare_spmv_csr(d, ti, tp, shape)
    y2 = fs.flagsparse_spmv_csr(x=tx, prepared=prep)
    _check(y2, vals, i, p, n_cols, x, dtype)
    assert torch.equal(fs.flagsparse_spmv_csr(x=tx, prepared=prep), y2)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.complex64], ids=str)
def test_out_may_be_the_operand(cuda, fsb_lib, dtype):
    n = 900
    _, i, p = handmade_csr(8, [3, 40, 0, 7, 500, 1] * 150, n)
    d, ti, tp = _values(int(p[-1]), dtype, 1).to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda)
    x, B = _values(n, dtype, 2).to(cuda), _values((n, 12), dtype, 3).to(cuda)
    y, C = fs.flagsparse_spmv_csr(d, ti, tp, x, (n, n)), fs.flagsparse_spmm_csr(d, ti, tp, B, (n, n))
    assert torch.equal(fs.flagsparse_spmv_csr(d, ti, tp, x, (n, n), out=x), y) and torch.equal(x, y)
    assert torch.equal(fs.flagsparse_spmm_csr(d, ti, tp, B, (n, n), out=B), C) and torch.equal(B, C)


def test_long_row_hint_keeps_the_accumulating_form(cuda, fsb_lib, monkeypatch):
    """C += A B over column panels of A (FSB_SPMM_PANELS) with rows that a block shares."""
    n_cols = 12000
    _, i, p = handmade_csr(9, LENS["tiles"] + LENS["shared"], n_cols)
    vals = _values(int(p[-1]), torch.float32, 1)
    B = _values((n_cols, 48), torch.float32, 2)
    monkeypatch.setenv("FSB_SPMM_PANELS", "3")
    prep = fs.prepare_spmm_csr_opt(vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda),
                                   (len(p) - 1, n_cols))
    _check(fs.flagsparse_spmm_csr_opt(B=B.to(cuda), prepared=prep), vals, i, p, n_cols, B, torch.float32)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.complex128], ids=str)
def test_spmm_rows_over_many_tiles(cuda, fsb_lib, dtype):
    """Rows that cross 7 to 25 tiles of 1024, where their partial sums are taken eight at a time and one by one."""
    n_cols = 30000
    for lens in ([3, 7 * 1024, 5, 8 * 1024, 1, 9 * 1024 + 1, 0, 16 * 1024], [17 * 1024 - 3, 2, 25 * 1024, 40]):
        _, i, p = handmade_csr(3, lens, n_cols)
        vals = _values(int(p[-1]), dtype, 4)
        for n_dense in (1, 33, 40):
            B = _values((n_cols, n_dense), dtype, n_dense)
            C = fs.flagsparse_spmm_csr(vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), B.to(cuda), (len(p) - 1, n_cols))
            _check(C, vals, i, p, n_cols, B, dtype)


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
def test_spmm_segments_by_length(cuda, fsb_lib, dtype):
    """Tiles with more segments than threads, all of one length but for one row of the matrix, chunks of segments none of which has an
    entry, and lengths around the last bucket; every result twice, as the order inside a bucket is not fixed."""
    n_cols = 700
    rng = np.random.default_rng(1)
    for lens in ([1] * 3000 + [2], [0, 2] * 1500 + [300], [3] * 300 + [0] * 2500 + [3] * 300 + [9], [5] * 700 + [6] * 400 + [8],
                 [int(v) for v in rng.integers(0, 4, 5000)] + [63, 64, 65, 124, 125, 126, 127, 130]):
        _, i, p = handmade_csr(3, lens, n_cols)
        vals = _values(int(p[-1]), dtype, 4)
        d, ti, tp = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda)
        if dtype in (torch.float32, torch.float64):
            assert fs.prepare_spmm_csr_opt(d, ti, tp, (len(p) - 1, n_cols))._uneven     # all of these are taken by length
        for n_dense in (16, 32, 64, 128):
            B = _values((n_cols, n_dense), dtype, n_dense)
            C = fs.flagsparse_spmm_csr(d, ti, tp, B.to(cuda), (len(p) - 1, n_cols))
            _check(C, vals, i, p, n_cols, B, dtype)
            assert torch.equal(fs.flagsparse_spmm_csr(d, ti, tp, B.to(cuda), (len(p) - 1, n_cols)), C)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.complex64, torch.complex128], ids=str)
def test_any_nonzero_long_rows_shares_them(cuda, fsb_lib, dtype):
    """fsb_spmm_csr_stored takes long_rows as yes or no: every value but 0 gives the sums of rows that a block shares."""
    from flagsparse_b200.spmm_csr import _STORED_VTYPE

    n_cols, n_dense = 2000, 24
    _, i, p = handmade_csr(13, [900, 3, 500, 700, 0, 8] * 20, n_cols)
    n = len(p) - 1
    vals, B = _values(int(p[-1]), dtype, 4), _values((n_cols, n_dense), dtype, 5)
    d, ti, tp, tb = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), B.to(cuda)
    vt = _STORED_VTYPE[dtype]
    scratch = torch.empty(fsb_lib.fsb_spmm_stored_scratch_bytes(vt, d.numel(), n_dense), dtype=torch.uint8, device=cuda)
    got = {}
    for yes in (0, 1, 64, 3):
        got[yes] = torch.empty((n, n_dense), dtype=dtype, device=cuda)
        assert fsb_lib.fsb_spmm_csr_stored(vt, 0, d.data_ptr(), ti.data_ptr(), tp.data_ptr(), tb.data_ptr(), n_dense,
                                           got[yes].data_ptr(), n_dense, n, n_cols, n_dense, d.numel(), yes, scratch.data_ptr(),
                                           scratch.numel(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(got[64], got[1]) and torch.equal(got[3], got[1])
    if dtype != torch.float16 and dtype != torch.bfloat16:      # (the rounding of the result hides the order of the sums)
        assert not torch.equal(got[0], got[1])
    _check(got[64], vals, i, p, n_cols, B, dtype)


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
def test_spmm_few_segments_in_a_tile(cuda, fsb_lib, dtype):
    """As many segments as a block has groups (16 or 32), one less, one more: from there on they are taken by length.  Every tile ends
    with a row, and the last one holds a few rows only."""
    n_cols = 700
    for count in (15, 16, 17, 31, 32, 33):
        short = 1024 // count - 3
        tile = [short] * (count - 2) + [1024 - short * (count - 2) - 1, 1]
        lens = tile * 4 + [7, 0, 3, 90]
        _, i, p = handmade_csr(3, lens, n_cols)
        vals = _values(int(p[-1]), dtype, 4)
        d, ti, tp = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda)
        for n_dense in (16, 32, 64, 128):
            B = _values((n_cols, n_dense), dtype, n_dense)
            C = fs.flagsparse_spmm_csr(d, ti, tp, B.to(cuda), (len(p) - 1, n_cols))
            _check(C, vals, i, p, n_cols, B, dtype)
