"""The SpMV kernel that walks neighbouring rows on one SM (from 8192 rows on, of short rows as many as its warps take): every number of
lanes, rows that take one turn and several, shares of even and uneven weight, ends of the arrays, every value type and index
width.  Reference and bound as for the tiled kernels: the product of the stored values in complex128."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from helpers import handmade_csr
from test_stored_types_gpu import DTYPES, _check, _values

pytestmark = pytest.mark.gpu


def _lengths(size):
    """Row lengths that take the kernel, whatever the values of `size` bytes."""
    rng = np.random.default_rng(5)
    most = 125000 if size <= 4 else 63000                      # rows for the warps with two lanes a row
    yield "least", [24 + k % 6 for k in range(8192)] if size != 16 else [60 + k % 6 for k in range(8192)]
    yield "one more", [24 + k % 6 for k in range(8193)] if size != 16 else [60 + k % 6 for k in range(8193)]
    # 2, 2, 4, 8, 16, 32 lanes for four entries at a time, 2, 2, 4, 8, 16, 32 for two (complex128)
    for mean, n in ((1, most), (5, most), (13, most // 2), (27, 16000), (60, 8260), (130, 8330)):
        yield f"mean {mean}", rng.poisson(mean, n)
    yield "several turns", np.where(np.arange(16001) % 97 == 5, 75, 30)
    yield "empty, then rows", np.where(np.arange(30000) < 6000, 0, 30)     # uneven shares: dealt in turn
    yield "long rows first", np.where(np.arange(70003) < 9000, 26, 9)
    yield "last entry", [0] * (most + 20000) + [1]


def _csr(lens, n_cols):
    p = np.zeros(len(lens) + 1, dtype=np.int32)
    np.cumsum(lens, out=p[1:])
    row = np.repeat(np.arange(len(lens)), lens)
    start = np.random.default_rng(7).integers(0, n_cols - 7 * int(max(lens)), len(lens))
    return (start[row] + 7 * (np.arange(int(p[-1])) - p[row])).astype(np.int32), p       # ascending inside a row


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
def test_against_the_stored_values(cuda, fsb_lib, dtype):
    n_cols = 12000
    for name, lens in _lengths(torch.empty(0, dtype=dtype).element_size()):
        i, p = _csr(lens, n_cols)
        vals, x = _values(int(p[-1]), dtype, 4), _values(n_cols, dtype, 5)
        shape = (len(p) - 1, n_cols)
        d, ti, tp, tx = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), x.to(cuda)
        y = fs.flagsparse_spmv_csr(d, ti, tp, tx, shape)
        _check(y, vals, i, p, n_cols, x, dtype)
        for wi, wp in ((ti.long(), tp), (ti, tp.long()), (ti.long(), tp.long())):
            assert torch.equal(fs.flagsparse_spmv_csr(d, wi, wp, tx, shape), y), name
        prep = fs.prepare_spmv_csr(d, ti, tp, shape)
        assert not prep.uneven, name
        assert torch.equal(fs.flagsparse_spmv_csr(x=tx, prepared=prep), y), name
        if vals.numel() > 1:                                    # arrays that start off a 16-byte boundary: lanes per row
            off = torch.cat([d[:1], d])[1:], torch.cat([ti[:1], ti])[1:]
            _check(fs.flagsparse_spmv_csr(*off, tp, tx, shape), vals, i, p, n_cols, x, dtype)


def test_what_neighbours_hold_stays_out(cuda, fsb_lib):
    """Infinite and NaN entries of one row, read along with the rows beside it, and of x, where no entry points."""
    n, length = 9000, 7
    d = torch.ones(n * length, device=cuda)
    d[length * 100:length * 101] = float("inf")
    d[length * 205] = float("nan")
    i = (torch.arange(n * length, device=cuda, dtype=torch.int32) * 3) % 5000
    x = torch.ones(5001, device=cuda)
    x[5000] = float("nan")
    y = fs.flagsparse_spmv_csr(d, i, torch.arange(n + 1, device=cuda, dtype=torch.int32) * length, x, (n, 5001))
    want = torch.full((n,), float(length), device=cuda)
    want[100], want[205] = float("inf"), float("nan")
    assert torch.equal(torch.nan_to_num(y, nan=-1.0), torch.nan_to_num(want, nan=-1.0))


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
def test_longest_row_at_the_line(cuda, fsb_lib, dtype):
    """Either side of the longest row from which rows are spread over all SMs; the two launches give the same sums but for their order."""
    from flagsparse_b200 import spmv_csr

    n_cols, n = 6000, 9000
    lens = [6] * n
    line = spmv_csr._longest_neighbour(n, 6 * n, torch.empty(0, dtype=dtype).element_size())
    for longest in (line, line + 2):                            # the mean grows by less than what moves the line by one
        lens[n // 2] = longest
        _, i, p = handmade_csr(9, lens, n_cols)
        vals, x = _values(int(p[-1]), dtype, 6), _values(n_cols, dtype, 7)
        d, ti, tp, tx = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), x.to(cuda)
        prep = fs.prepare_spmv_csr(d, ti, tp, (n, n_cols))
        assert (prep.uneven != 0) == (longest > line)
        y = fs.flagsparse_spmv_csr(x=tx, prepared=prep)
        _check(y, vals, i, p, n_cols, x, dtype)
        assert torch.equal(fs.flagsparse_spmv_csr(d, ti, tp, tx, (n, n_cols)), y)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=str)
def test_neighbours_stay_on_one_sm_only_where_the_caller_says_even(cuda, fsb_lib, dtype):
    """FSB_SPMV_VECTOR with tuning 0 takes lanes per row, whatever the rows; FSB_SPMV_AUTO without a plan, too."""
    from flagsparse_b200 import _lib
    from flagsparse_b200._common import _VTYPE

    n, n_cols, lanes = 9000, 3000, 4                            # 16 * 2 < 50 + 3, 16 * 4 is not
    _, i, p = handmade_csr(11, [50] * n, n_cols)
    vals, x = _values(int(p[-1]), dtype, 6), _values(n_cols, dtype, 7)
    d, ti, tp, tx = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), x.to(cuda)

    def run(algo, tuning):
        y = torch.full((n,), float("nan"), dtype=dtype, device=cuda)
        assert fsb_lib.fsb_spmv_csr(_VTYPE[dtype], 0, 0, d.data_ptr(), ti.data_ptr(), tp.data_ptr(), tx.data_ptr(), y.data_ptr(), n,
                                    n_cols, d.numel(), algo, tuning, None, None, 0, torch.cuda.current_stream().cuda_stream) == 0
        return y

    spread = run(_lib.FSB_SPMV_VECTOR, lanes)
    assert torch.equal(run(_lib.FSB_SPMV_VECTOR, 0), spread) and torch.equal(run(_lib.FSB_SPMV_AUTO, 0), spread)
    even = run(_lib.FSB_SPMV_VECTOR, 1024)
    assert not torch.equal(even, spread)                        # another order of the sums
    _check(even, vals, i, p, n_cols, x, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=str)
def test_into_several_vectors(cuda, fsb_lib, dtype):
    """The rows kernel with the epilogue that stores every value into the vectors of all GPUs, here two vectors of this one: even
    rows, shares of uneven weight, a row offset; the values are those of the product into one vector."""
    from flagsparse_b200 import _lib
    from flagsparse_b200._common import _VTYPE

    n_cols = 4000
    for lens in ([20 + k % 9 for k in range(8192)], np.where(np.arange(30000) < 6000, 0, 40), [k % 9 for k in range(125000)]):
        _, i, p = handmade_csr(12, [int(v) for v in lens], n_cols)
        vals, x = _values(int(p[-1]), dtype, 6), _values(n_cols, dtype, 7)
        n = len(p) - 1
        d, ti, tp, tx = vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), x.to(cuda)
        y = torch.empty(n, dtype=dtype, device=cuda)
        st = torch.cuda.current_stream().cuda_stream
        args = (_VTYPE[dtype], 0, 0, d.data_ptr(), ti.data_ptr(), tp.data_ptr(), tx.data_ptr())
        assert fsb_lib.fsb_spmv_csr(*args, y.data_ptr(), n, n_cols, d.numel(), _lib.FSB_SPMV_VECTOR, 1024, None, None, 0, st) == 0
        _check(y, vals, i, p, n_cols, x, dtype)
        for tuning in (1024, 0):
            out = [torch.full((n + 20,), 7.0, dtype=dtype, device=cuda) for _ in range(2)]
            peers = torch.tensor([t.data_ptr() for t in out], dtype=torch.int64, device=cuda)
            assert fsb_lib.fsb_spmv_csr_scatter(*args, peers.data_ptr(), 2, 1, 9, n, n_cols, d.numel(), _lib.FSB_SPMV_VECTOR, tuning,
                                                None, None, 0, st) == 0
            for t in out:
                assert bool((t[:9] == 7).all()) and bool((t[9 + n:] == 7).all())
                if tuning:
                    assert torch.equal(t[9:9 + n], y)
                else:
                    _check(t[9:9 + n], vals, i, p, n_cols, x, dtype)


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
def test_enough_rows_for_the_warps(cuda, fsb_lib, dtype):
    """Short rows, 2 and 4 lanes each, either side of the number of rows from which neighbours stay on one SM: 32 rows a warp (values
    of 8 and 16 bytes: 16) with two lanes a row, half as many with four."""
    from flagsparse_b200 import _lib
    from flagsparse_b200._common import _VTYPE

    size = torch.empty(0, dtype=dtype).element_size()
    together, n_cols = (2 if size <= 4 else 1), 500
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    gen = torch.Generator(device="cuda").manual_seed(5)
    for lanes in (2, 4):
        mean = 9 if lanes == 2 else 12               # (float64 and half precisions: rows of 12 are long, whatever their number)
        line = -(-4 * sms * 32 * together * (32 // lanes) // 5)
        for n in (line - 1, line):
            p = torch.arange(n + 1, device=cuda, dtype=torch.int32) * mean
            i = torch.randint(0, n_cols, (n * mean,), device=cuda, generator=gen, dtype=torch.int32)
            d, x = _values(n * mean, dtype, 1).to(cuda), _values(n_cols, dtype, 2).to(cuda)
            y = fs.flagsparse_spmv_csr(d, i, p, x, (n, n_cols))
            wide = torch.complex128 if dtype.is_complex else torch.float64
            prod = (d.to(wide) * x.to(wide)[i.long()]).view(n, mean)
            ref, mag = prod.sum(1), prod.abs().sum(1)
            u = {4: 2.0 ** -24, 8: 2.0 ** -53}[4 if dtype in (torch.float16, torch.bfloat16, torch.float32, torch.complex64) else 8]
            bound = (4 if dtype.is_complex else 1) * (mean + 1) * u * mag
            if size == 2:
                v = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
                bound = bound * (1 + v) + v * ref.abs() + (2.0 ** -25 if dtype == torch.float16 else 0)
            assert bool(((y.to(wide) - ref).abs() <= 1.0001 * bound).all()), n
            assert torch.equal(fs.flagsparse_spmv_csr(x=x, prepared=fs.prepare_spmv_csr(d, i, p, (n, n_cols))), y)
            if dtype in (torch.float32, torch.float64) and lanes == 2:
                spread = torch.empty_like(y)         # two lanes a row, and no neighbours
                assert fsb_lib.fsb_spmv_csr(_VTYPE[dtype], 0, 0, d.data_ptr(), i.data_ptr(), p.data_ptr(), x.data_ptr(), spread.data_ptr(),
                                            n, n_cols, d.numel(), _lib.FSB_SPMV_VECTOR, 2, None, None, 0,
                                            torch.cuda.current_stream().cuda_stream) == 0
                assert torch.equal(y, spread) == (n < line)
