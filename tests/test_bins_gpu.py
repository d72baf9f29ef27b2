"""The two-pass SpMV (csrc/spmv_bins.cu): rows that end on, straddle and fill the slices, blocks and chunks, against the
float64 oracle; the same bits on every call and whatever the chunks; infinities stay in their rows."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import _lib, bins
from gpu_util import dev, env, spmv
from helpers import assert_spmv_ok, handmade_csr

pytestmark = pytest.mark.gpu


def _layout(d, i, p, shape, chunk_cols=None):
    lens = np.diff(p)
    return bins.build_bins_layout(dev(d), dev(i), dev(p), shape[0], shape[1], int(lens.max()), chunk_cols=chunk_cols)


def _product(lay, x, shape, shift=0):
    """y into a vector that starts `shift` elements behind a 256-byte boundary."""
    y = torch.full((shape[0] + shift,), float("nan"), dtype=x.dtype, device=x.device)[shift:]
    bins.launch_bins(lay, x, y, shape[0], shape[1], torch.cuda.current_stream().cuda_stream)
    return y


_LENS = {
    "one entry": [1],
    "empty rows around": [0] * 9 + [3, 0, 0, 1] + [0] * 5,
    "slice edges": [31, 1, 32, 33, 15, 1, 16, 17, 64, 0, 95, 5],
    "rows over many threads": [2000, 1, 0, 3000, 33, 2500] * 9,
    "one block exactly": {4: [512] * 48, 8: [256] * 48},
    "one entry more than a block": {4: [512] * 48 + [1], 8: [256] * 48 + [1]},
    "many blocks, short rows": list(np.random.default_rng(5).integers(0, 12, 30001)),
    "no row ends in a warp": [3001] + [1] * 40,
}


@pytest.mark.parametrize("name", sorted(_LENS))
@pytest.mark.parametrize("vdt,pdt", [("float32", "int32"), ("float64", "int64")])
def test_edges(cuda, fsb_lib, name, vdt, pdt):
    lens = _LENS[name]
    lens = lens[np.dtype(vdt).itemsize] if isinstance(lens, dict) else lens
    n_cols = 3001
    d, i, p = handmade_csr(11, lens, n_cols, value_dtype=vdt, indptr_dtype=pdt, replace=True, sort=False)
    shape = (len(lens), n_cols)
    x = np.random.default_rng(3).uniform(-1, 1, n_cols + 1).astype(vdt)
    want = None
    for chunk_cols, shift in ((None, 0), (400, 1), (3004, 3)):     # one chunk; eight, the last one ragged; x and y off 16 bytes
        lay = _layout(d, i, p, shape, chunk_cols)
        tx = dev(x)[1:] if shift else dev(x[1:])
        y = _product(lay, tx, shape, shift)
        assert_spmv_ok(y.cpu().numpy(), d, i, p, shape, x[1:], what=f"{name} {chunk_cols}")
        assert torch.equal(y, _product(lay, tx, shape))
        want = y if want is None else want
        assert torch.equal(y, want)


def test_a_row_over_two_slices_is_rounded_once(cuda, fsb_lib):
    # the part in the slice where the row ends has 25 bits, and in the second row more than float32 can hold
    big, huge = 2.0**30, 3e38
    d = np.zeros(80, dtype=np.float32)
    d[[0, 1, 32, 33]] = [big, 0.5, -big, 0.25]
    d[[40, 64, 65]] = [-huge, huge, huge]
    i = np.tile(np.arange(40, dtype=np.int32), 2)
    lay = _layout(d, i, np.array([0, 40, 80], dtype=np.int32), (2, 40))
    y = _product(lay, torch.ones(40, device=cuda), (2, 40)).cpu().numpy()
    assert y.tolist() == [0.75, float(np.float32(huge))]


def _two_products(a, b):
    """a * b of float64 values as an unevaluated sum, exact (Dekker)."""
    def halves(v):
        t = v * 134217729.0
        hi = t - (t - v)
        return hi, v - hi

    p, (ah, al), (bh, bl) = a * b, halves(a), halves(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


@pytest.mark.parametrize("length", [2, 4, 16, 60, 700])
@pytest.mark.parametrize("vdt", ["float32", "float64"])
def test_no_less_accurate_than_one_pass(cuda, fsb_lib, vdt, length):
    """Root mean square error of rows of equal length: 1.03 is left for the spread of an rms over 3 * 10^4 rows and more,
    1.1 over the 3000 longest."""
    n_rows, n_cols = max(3000, 200000 // length), 30000
    rng = np.random.default_rng(length)
    i = rng.integers(0, n_cols, n_rows * length).astype(np.int32)
    d, x = rng.uniform(-1, 1, n_rows * length).astype(vdt), rng.uniform(-1, 1, n_cols).astype(vdt)
    p = np.arange(n_rows + 1, dtype=np.int32) * length
    hi, lo = _two_products(d.astype(np.float64), x.astype(np.float64)[i])
    wide = hi.reshape(n_rows, -1).astype(np.longdouble).sum(1) + lo.reshape(n_rows, -1).astype(np.longdouble).sum(1)
    rms = lambda y: float(np.sqrt(np.mean((y.astype(np.longdouble) - wide) ** 2)))  # noqa: E731
    two = rms(_product(_layout(d, i, p, (n_rows, n_cols), 4096), dev(x), (n_rows, n_cols)).cpu().numpy())
    one = min(rms(spmv(d, i, p, (n_rows, n_cols), x, algo=algo)) for algo in ("vector", "stream"))
    assert two <= (1.03 if n_rows >= 3 * 10**4 else 1.1) * one, (two, one)


@pytest.mark.parametrize("vdt", ["float32", "float64"])
def test_infinities_stay_in_their_rows(cuda, fsb_lib, vdt):
    lens = [40, 3, 70, 1, 5] * 300
    d, i, p = handmade_csr(2, lens, 5000, value_dtype=vdt)
    x = np.random.default_rng(1).uniform(0.5, 1, 5000).astype(vdt)
    rows = [0, 2, 601, 1499]
    for r in rows:
        d[p[r]] = np.inf
    d[p[7]], d[p[7] + 1] = np.inf, -np.inf
    y = _product(_layout(d, i, p, (1500, 5000), 1000), dev(x), (1500, 5000)).cpu().numpy()
    assert np.isposinf(y[rows]).all() and np.isnan(y[7])
    rest = np.setdiff1d(np.arange(1500), rows + [7])
    assert np.isfinite(y[rest]).all()
    x[0] = np.nan                       # what fills the packs up has column 0 of its chunk: no row may see it
    y2 = _product(_layout(d, i, p, (1500, 5000), 1000), dev(x), (1500, 5000)).cpu().numpy()
    keep = np.setdiff1d(rest, [r for r in range(1500) if (i[p[r]:p[r + 1]] == 0).any()])
    assert np.array_equal(y2[keep], y[keep])


def test_what_is_left_to_one_pass(cuda, fsb_lib):
    d, i, p = handmade_csr(4, [7000] + [2] * 50, 9000)
    assert _layout(d, i, p, (51, 9000)) is None                        # a row too long for a block
    d, i, p = handmade_csr(4, [4] * 500, 9000)
    assert bins.build_bins_layout(dev(d), dev(i), dev(p), 500, 9000, 4, span=9000 * 4 + 1) is None
    assert bins.build_bins_layout(dev(d), dev(i), dev(p), 500, 9000, 4, span=9000 * 4, chunk_cols=1000) is not None
    # the units are looked at, not only the width of the matrix: a band reaches few chunks
    i = (i % 40).astype(np.int32)
    assert bins.build_bins_layout(dev(d), dev(i), dev(p), 500, 9000, 4, span=9000 * 4, chunk_cols=1000) is None


def test_blocks_of_empty_rows_do_not_count_for_the_reach(cuda, fsb_lib):
    lens = [4] * 500 + [0] * 3 * 10**5
    d, i, p = handmade_csr(4, lens, 9000)
    build = lambda span: bins.build_bins_layout(dev(d), dev(i), dev(p), len(lens), 9000, 4, span=span, chunk_cols=1000)  # noqa: E731
    assert build(9000 * 4) is not None and build(9000 * 4 + 1) is None


@pytest.mark.parametrize("where", ["start", "middle", "end", "rows of one block", "one row more"])
@pytest.mark.parametrize("vdt", ["float32", "float64"])
def test_runs_of_empty_rows_are_shared_by_blocks(cuda, fsb_lib, where, vdt):
    some = list(np.random.default_rng(2).integers(1, 9, 2000))
    empty = {"rows of one block": (1 << 16) - 2000, "one row more": (1 << 16) - 1999}.get(where, 3 * 10**5)
    cut = {"start": 0, "middle": 1000}.get(where, 2000)
    lens = some[:cut] + [0] * empty + some[cut:]
    d, i, p = handmade_csr(5, lens, 7000, value_dtype=vdt)
    shape = (len(lens), 7000)
    x = np.random.default_rng(3).uniform(-1, 1, 7000).astype(vdt)
    lay = _layout(d, i, p, shape, 1000)
    rows = lay.block_start.view(-1, 2)[:, 0].cpu().numpy()
    assert rows[0] == 0 and rows[-1] == shape[0] and 0 < np.diff(rows).min() and np.diff(rows).max() <= 1 << 16
    assert_spmv_ok(_product(lay, dev(x), shape).cpu().numpy(), d, i, p, shape, x, what=where)


def test_prepared_matrix_takes_the_two_passes(cuda, fsb_lib, monkeypatch):
    monkeypatch.setattr(bins, "UNEVEN_MIN_NNZ", 1 << 17)
    monkeypatch.setattr(bins, "UNEVEN_MIN_SPAN", 1 << 10)
    lens = np.random.default_rng(7).integers(0, 9, 60000)
    lens[::5000] = 700
    d, i, p = handmade_csr(8, lens.tolist(), 50000)
    x = np.random.default_rng(9).uniform(-1, 1, 50000).astype(np.float32)
    prep = fs.prepare_spmv_csr(dev(d), dev(i.astype(np.int64)), dev(p), (60000, 50000))
    assert prep.bins is not None and prep.opt_buckets[0]["kind"] == "bins"
    y = fs.flagsparse_spmv_csr(x=dev(x), prepared=prep)
    assert_spmv_ok(y.cpu().numpy(), d, i, p, (60000, 50000), x)
    graph, got = torch.cuda.CUDAGraph(), None
    tx = dev(x)
    with torch.cuda.graph(graph):
        got = fs.flagsparse_spmv_csr(x=tx, prepared=prep)
    graph.replay()
    assert torch.equal(got, y)
    monkeypatch.setenv("FSB_SPMV_BINS", "0")
    assert fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (60000, 50000)).bins is None


@pytest.mark.parametrize("longest,form", [(40, "vector"), (700, "stream")])
def test_memory_that_is_refused_leaves_one_pass(cuda, fsb_lib, monkeypatch, longest, form):
    for name in ("UNEVEN_MIN_NNZ", "UNEVEN_MIN_SPAN"):
        monkeypatch.setattr(bins, name, 1 << 10)
    lens = np.random.default_rng(7).integers(0, 9, 60000)
    lens[::5000] = longest
    d, i, p = handmade_csr(8, lens.tolist(), 50000)
    x = dev(np.random.default_rng(9).uniform(-1, 1, 50000).astype(np.float32))
    with env(FSB_SPMV_ALGO=form):
        want = fs.flagsparse_spmv_csr(x=x, prepared=fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (60000, 50000)))
    prep = fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (60000, 50000))
    assert prep.bins is not None

    def refuse(*args):
        raise torch.OutOfMemoryError

    monkeypatch.setattr(bins, "_between_passes", refuse)
    assert torch.equal(fs.flagsparse_spmv_csr(x=x, prepared=prep), want)
    monkeypatch.setattr(bins, "build_bins_layout", refuse)
    prep = fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (60000, 50000))
    assert prep.bins is None and prep.opt_buckets[0]["kind"] == form
    assert torch.equal(fs.flagsparse_spmv_csr(x=x, prepared=prep), want)


def test_refused_calls(fsb_lib):
    """Argument errors are found on the host, before anything is launched."""
    L = fsb_lib
    one = [1 << 20] * 9
    call = lambda vt=0, chunks=1, width=64, cols=64, packs=1, nbytes=32, rows=1, ptrs=one: L.fsb_spmv_csr_bins(  # noqa: E731
        vt, *ptrs, 1, chunks, width, packs, 1 << 20, nbytes, 1 << 20, 1 << 20, rows, cols, None)
    assert call(vt=_lib.FSB_BF16) == -1 and call(chunks=2) == -1 and call(cols=65) == -1 and call(ptrs=[None] + one[1:]) == -1
    assert call(width=65, cols=65) == -2 and call(packs=2**31) == -2
    assert call(nbytes=31) == -4
    assert call(ptrs=[(1 << 20) + 4] + one[1:]) == -3
