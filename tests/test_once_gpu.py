"""Products straight from CSR arrays through one call that checks, waits and launches: what is refused, uneven rows, index widths,
calls from several threads and streams, a stream that is being captured.  Results are compared with those of a prepared matrix, whose
arrays are checked on their own."""

import threading

import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import _common

pytestmark = pytest.mark.gpu


def _matrix(n, cols, long_row=0, dtype=torch.float32, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    lens = torch.randint(0, 12, (n,), device="cuda", generator=g)
    if long_row:
        lens[n // 2] = long_row
    p = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    p[1:] = torch.cumsum(lens, 0)
    nnz = int(p[-1])
    i = torch.randint(0, cols, (nnz,), device="cuda", generator=g)
    return torch.randn(nnz, device="cuda", generator=g).to(dtype), i, p, (n, cols)


@pytest.mark.parametrize("long_row", [0, 60, 400, 5000])       # even rows, and rows that go to tiles or are shared by a block
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.complex64], ids=str)
def test_same_as_prepared(cuda, fsb_lib, dtype, long_row):
    for n in (1, 300, 9000):
        d, i, p, shape = _matrix(n, 700, long_row, dtype)
        x, B = torch.randn(700, device=cuda).to(dtype), torch.randn(700, 24, device=cuda).to(dtype)
        y = fs.flagsparse_spmv_csr(x=x, prepared=fs.prepare_spmv_csr(d, i.int(), p.int(), shape))
        C = None
        for ii in (i, i.int()):
            for pp in (p, p.int()):
                out = torch.empty_like(y)
                assert torch.equal(fs.flagsparse_spmv_csr(d, ii, pp, x, shape), y)
                assert fs.flagsparse_spmv_csr(d, ii, pp, x, shape, out=out) is out and torch.equal(out, y)
                got = fs.flagsparse_spmm_csr(d, ii, pp, B, shape)
                C = got if C is None else C
                assert torch.equal(got, C) and torch.equal(fs.flagsparse_spmm_csr(d, ii, pp, B, shape, out=torch.empty_like(C)), C)
        if dtype in (torch.float32, torch.float64):
            assert torch.equal(fs.flagsparse_spmm_csr_opt(B=B, prepared=fs.prepare_spmm_csr_opt(d, i.int(), p.int(), shape)), C)


def test_refused_arrays_leave_out_alone(cuda, fsb_lib):
    d, i, p, shape = _matrix(500, 90)
    x, B = torch.randn(90, device=cuda), torch.randn(90, 8, device=cuda)

    def changed(t, at, v):
        t = t.clone()
        t[at] = v
        return t

    bad = [(changed(i, 7, 90), p, IndexError), (changed(i, 0, -1), p, IndexError), (i, changed(p, 0, 1), ValueError),
           (i, changed(p, -1, int(p[-1]) - 1), ValueError), (i, changed(p, 40, int(p[39]) - 1), ValueError)]
    for ii, pp, error in bad:
        for cast in (torch.int32, torch.int64):
            out, outm = torch.full((500,), 3.0, device=cuda), torch.full((500, 8), 3.0, device=cuda)
            with pytest.raises(error):
                fs.flagsparse_spmv_csr(d, ii.to(cast), pp.to(cast), x, shape, out=out)
            with pytest.raises(error):
                fs.flagsparse_spmm_csr(d, ii.to(cast), pp.to(cast), B, shape, out=outm)
            with pytest.raises(error):
                fs.flagsparse_spmm_csr(d, ii.to(cast), pp.to(cast), B, shape)
            with pytest.raises(error):
                fs.prepare_spmv_csr(d, ii.to(cast), pp.to(cast), shape)
            assert bool((out == 3).all()) and bool((outm == 3).all())
    # the counters are as they were: the next matrix is judged by itself
    s = _common._analyze_csr(i, p, 500)
    lens = p[1:] - p[:-1]
    assert (s.ptr_first, s.ptr_last, s.n_decreasing, s.min_index, s.max_index, s.max_row_nnz, s.n_empty_rows, s.n_long_rows) == (
        0, d.numel(), 0, int(i.min()), int(i.max()), int(lens.max()), int((lens == 0).sum()), 0)
    s = _common._analyze_csr(i[:0], p[:1], 0)
    assert (s.min_index, s.max_index, s.max_row_nnz) == (2 ** 63 - 1, -2 ** 63, 0)


def test_threads_and_streams(cuda, fsb_lib):
    cases = [_matrix(2000 + 700 * k, 500 + k, seed=k) for k in range(4)]
    xs = [torch.randn(500 + k, device=cuda) for k in range(4)]
    want = [fs.flagsparse_spmv_csr(*cases[k][:3], xs[k], cases[k][3]) for k in range(4)]
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in range(60):
                j = (k + r) % 4
                if r % 20 == 19:                       # another stream of the same thread
                    with torch.cuda.stream(torch.cuda.Stream()):
                        y = fs.flagsparse_spmv_csr(*cases[j][:3], xs[j], cases[j][3])
                        torch.cuda.current_stream().synchronize()
                else:
                    y = fs.flagsparse_spmv_csr(*cases[j][:3], xs[j], cases[j][3])
                    torch.cuda.current_stream().synchronize()
                if not torch.equal(y, want[j]):
                    wrong.append((k, r))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_not_while_a_stream_is_captured(cuda, fsb_lib):
    d, i, p, shape = _matrix(300, 90)
    x = torch.randn(90, device=cuda)
    want = fs.flagsparse_spmv_csr(d, i, p, x, shape)
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            fs.flagsparse_spmv_csr(d, i, p, x, shape)
    torch.cuda.synchronize()
    assert torch.equal(fs.flagsparse_spmv_csr(d, i, p, x, shape), want)


def test_a_check_after_one_that_was_not_waited_for(cuda, fsb_lib):
    """Words as a call leaves them that returned before its kernel had ended: the next one counts on from that call's ticket."""
    d, i, p, shape = _matrix(300, 90)
    _common._analyze_csr(i, p, 300)
    slot = _common._check_slot(i.device)
    words = slot.host
    words[9] += 3
    last = int(words[9])
    assert int(words[8]) == last - 3
    s = _common._analyze_csr(i, p, 300)
    assert int(words[8]) == int(words[9]) == last + 1 and s.ptr_last == d.numel()
