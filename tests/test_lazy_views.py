"""Operands that carry a conjugation or a negation which torch has not carried out yet (x.conj(), z.conj().imag): the same
results as for their resolved copies, which the kernels read as memory."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from fake_device import fake_cuda
from helpers import handmade_csr

LENS, N_COLS = [3, 0, 40, 7, 12, 1], 50


def _draw(shape, dtype, seed, device="cpu"):
    rng = np.random.default_rng(seed)
    return torch.from_numpy(rng.uniform(-1, 1, shape) + 1j * rng.uniform(-1, 1, shape)).to(dtype).to(device)


def _calls(dtype, device):
    """(name, call of the arguments that may be lazy)"""
    _, i, p = handmade_csr(4, LENS, N_COLS)
    row = torch.from_numpy(np.repeat(np.arange(len(LENS)), LENS)).to(device)
    i, p, shape = torch.from_numpy(i).to(device), torch.from_numpy(p).to(device), (len(LENS), N_COLS)
    n = i.numel()
    v = lambda *s: _draw(s, dtype, len(s), device)  # noqa: E731
    calls = [("spmv", lambda d, x: fs.flagsparse_spmv_csr(d, i, p, x, shape), (v(n), v(N_COLS))),
             ("spmv prepared", lambda d, x: fs.flagsparse_spmv_csr(x=x, prepared=fs.prepare_spmv_csr(d, i, p, shape)),
              (v(n), v(N_COLS))),
             ("spmm", lambda d, b: fs.flagsparse_spmm_csr(d, i, p, b, shape), (v(n), v(N_COLS, 5))),
             ("spmm_coo", lambda d, b: fs.flagsparse_spmm_coo(d, row, i, b, shape), (v(n), v(N_COLS, 5)))]
    return calls, (i, p, row, shape)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128], ids=str)
def test_conjugated_operands_on_the_host_path(dtype, fsb_lib):
    _conjugated(dtype, "cpu")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128], ids=str)
def test_conjugated_operands(cuda, fsb_lib, dtype):
    _conjugated(dtype, cuda)


def _conjugated(dtype, device):
    calls, _ = _calls(dtype, device)
    for name, call, args in calls:
        for k in range(len(args)):
            lazy = [a.conj() if j == k else a for j, a in enumerate(args)]
            assert lazy[k].is_conj() and lazy[k].is_contiguous()
            if device == "cpu":
                with fake_cuda():
                    got, want = call(*lazy), call(*[a.resolve_conj() for a in lazy])
            else:
                got, want = call(*lazy), call(*[a.resolve_conj() for a in lazy])
            assert not torch.equal(want, want.conj().resolve_conj()) and torch.equal(got, want), (name, k)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,part", [(torch.complex64, torch.float32), (torch.complex128, torch.float64)], ids=str)
def test_negated_real_views(cuda, fsb_lib, dtype, part):
    """One column of imaginary parts is a view that needs no copy for its strides; so is a result of one element."""
    calls, (i, p, row, shape) = _calls(dtype, cuda)
    d = torch.rand(i.numel(), dtype=part, device=cuda)
    col = lambda n, s: _draw((n, 1), dtype, s, cuda).conj().imag  # noqa: E731
    B, X, Y = col(N_COLS, 5), col(len(LENS), 6), col(N_COLS, 7)
    assert B.is_neg()
    for call in (lambda b: fs.flagsparse_spmm_csr(d, i, p, b, shape),
                 lambda b: fs.flagsparse_spmm_csr_opt(B=b, prepared=fs.prepare_spmm_csr_opt(d, i, p, shape)),
                 lambda b: fs.flagsparse_spmm_coo(d, row, i, b, shape)):
        assert torch.equal(call(B), call(B.resolve_neg()))
    prep = fs.prepare_sddmm_csr(i, p, shape)
    assert torch.equal(fs.flagsparse_sddmm_csr(x=X, y=Y, prepared=prep),
                       fs.flagsparse_sddmm_csr(x=X.resolve_neg(), y=Y.resolve_neg(), prepared=prep))
    one = torch.ones(2, dtype=torch.int32, device=cuda).cumsum(0).to(torch.int32) - 1      # indptr of a 1 x 1 matrix
    out = torch.zeros(1, dtype=dtype, device=cuda).conj().imag
    assert out.is_neg() and out.is_contiguous()
    v = torch.full((1,), 3, dtype=part, device=cuda)
    fs.flagsparse_spmv_csr(v, one[:1], one, v, (1, 1), out=out)
    assert out.item() == 9
