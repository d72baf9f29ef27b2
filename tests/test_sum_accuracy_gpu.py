"""float16, bfloat16 and complex products against the kernels that keep one group of lanes per whole row and two partial
sums (fsb_spmv_csr_wide, fsb_spmm_csr_wide): the root mean square error against a product in twice the precision is no
larger.  One sided: 1.03 is left for the spread of an rms over 3 * 10^4 elements."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import _lib, widetypes as W

pytestmark = pytest.mark.gpu

VT = {torch.float16: _lib.FSB_F16, torch.bfloat16: _lib.FSB_BF16, torch.complex64: _lib.FSB_C64,
      torch.complex128: _lib.FSB_C128}


def _values(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(-1, 1, shape)
    return torch.from_numpy(v + 1j * rng.uniform(-1, 1, shape) if dtype.is_complex else v).to(dtype)


def _exact(vals, idx, operand, lens):
    """Rows of equal length: sums of the products in numpy's widest type."""
    wide = (lambda t: t.to(torch.complex128).numpy().astype(np.clongdouble)) if vals.is_complex() else \
        (lambda t: t.double().numpy().astype(np.longdouble))
    a, o = wide(vals).reshape(-1, lens), wide(operand)[idx.reshape(-1, lens)]
    return np.einsum("rk,rk...->r...", a, o)


def _rms(got, exact):
    g = got.cpu()
    g = g.to(torch.complex128).numpy() if g.is_complex() else g.double().numpy()
    return float(np.sqrt(np.mean(np.abs(g - exact) ** 2)))


@pytest.mark.parametrize("dtype", W.WIDE_DTYPES, ids=str)
@pytest.mark.parametrize("length", [3, 7, 16, 60, 200, 700])
def test_no_less_accurate_than_two_sums_over_a_row(cuda, fsb_lib, dtype, length):
    n_cols, n_rows = 3000, 6000 if length < 100 else 2000
    st = torch.cuda.current_stream().cuda_stream
    for n_dense, n_rows in ((16, n_rows), (0, 10 * n_rows)):
        idx = np.random.default_rng(length).integers(0, n_cols, n_rows * length).astype(np.int32)
        vals = _values((n_rows * length,), dtype, 1)
        operand = _values((n_cols, n_dense) if n_dense else (n_cols,), dtype, 2)
        exact = _exact(vals, idx, operand, length)
        d, i = vals.to(cuda), torch.from_numpy(idx).to(cuda)
        p = torch.arange(n_rows + 1, dtype=torch.int32, device=cuda) * length
        dense = operand.to(cuda).to(W.dense_dtype(dtype))
        old = torch.empty((n_rows,) + tuple(operand.shape[1:]), dtype=dense.dtype, device=cuda)
        if n_dense:
            new = fs.flagsparse_spmm_csr(d, i, p, operand.to(cuda), (n_rows, n_cols))
            rc = fsb_lib.fsb_spmm_csr_wide(VT[dtype], 0, d.data_ptr(), i.data_ptr(), p.data_ptr(), dense.data_ptr(), n_dense,
                                           old.data_ptr(), n_dense, n_rows, n_cols, n_dense, d.numel(), st)
        else:
            new = fs.flagsparse_spmv_csr(d, i, p, operand.to(cuda), (n_rows, n_cols))
            rc = fsb_lib.fsb_spmv_csr_wide(VT[dtype], 0, d.data_ptr(), i.data_ptr(), p.data_ptr(), dense.data_ptr(),
                                           old.data_ptr(), n_rows, n_cols, d.numel(), st)
        assert rc == 0
        a, b = _rms(new, exact), _rms(old.to(dtype), exact)
        assert a <= 1.03 * b, (n_dense, a, b)


@pytest.mark.parametrize("k", [8, 16, 64, 100, 128])
def test_sddmm_no_less_accurate_than_products_one_by_one(cuda, fsb_lib, k):
    """float32, four elements a lane: the rms error against that of the same sum with the four products added one after the other by fused
    multiply-adds and the lanes added in a tree.  The bound leaves half a percent for the last place in which the model's
    double rounding may differ."""
    n_rows, length, n_cols = 4000, 12, 500
    rng = np.random.default_rng(k)
    i = rng.integers(0, n_cols, n_rows * length).astype(np.int32)
    x, y = rng.uniform(-1, 1, (n_rows, k)).astype(np.float32), rng.uniform(-1, 1, (n_cols, k)).astype(np.float32)
    p = torch.arange(n_rows + 1, device=cuda) * length
    prep = fs.prepare_sddmm_csr(torch.from_numpy(i).to(cuda), p, (n_rows, n_cols))
    out = fs.flagsparse_sddmm_csr(x=torch.from_numpy(x).to(cuda), y=torch.from_numpy(y).to(cuda), prepared=prep).cpu().numpy()
    prod = np.repeat(x.astype(np.float64), length, 0) * y.astype(np.float64)[i]          # exact
    lanes = 1
    while 4 * lanes < k:
        lanes *= 2
    part = np.zeros((len(i), lanes, 4))
    part.reshape(len(i), -1)[:, :k] = prod
    s = np.zeros((len(i), lanes), dtype=np.float32)
    for j in range(4):
        s = (s + part[:, :, j]).astype(np.float32)
    while lanes > 1:
        lanes //= 2
        s = s[:, :lanes] + s[:, lanes:]
    exact = prod.astype(np.longdouble).sum(1)
    rms = lambda v: float(np.sqrt(np.mean((v - exact) ** 2)))  # noqa: E731
    assert rms(out.astype(np.longdouble)) <= 1.005 * rms(s[:, 0].astype(np.longdouble))
