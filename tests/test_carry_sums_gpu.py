"""Rows over many tiles whose partial sums cancel: large ones of opposite sign in tiles far apart, small ones between them.  The
partial sums are added with what each addition loses, so the small ones are all there in the end (a plain sum of doubles at
2^80 has none of them left).  Every product here is exact in the type of the values."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs

pytestmark = pytest.mark.gpu

N = 60000                                     # entries of the row: tiles of at most 4096 put the large ones into tiles of their own


def _row(dtype, plus, minus, rng):
    v = np.zeros(N)
    at = rng.choice(np.arange(9000, N - 9000), 120, replace=False)
    v[at] = 1
    if plus:                                  # the small ones stay out of the tiles of the large ones
        for k in (plus, minus):
            v[max(0, k - 4096):k + 4096] = 0
    want = int(v.sum())
    v[plus], v[minus] = 2.0 ** 80, -2.0 ** 80
    return torch.from_numpy(v).to(dtype), want


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.complex64, torch.complex128], ids=str)
def test_small_partial_sums_survive_large_ones(cuda, fsb_lib, dtype):
    rng = np.random.default_rng(3)
    for plus, minus in ((0, N - 1), (N - 1, 0), (20000, 40000), (13000, 14000 + 8192)):
        v, want = _row(dtype, plus, minus, rng)
        # two rows of the same entries, and short ones around them
        d = torch.cat([torch.ones(5, dtype=dtype), v, torch.ones(3, dtype=dtype), v]).to(cuda)
        p = torch.tensor([0, 5, 5 + N, 8 + N, 8 + 2 * N], dtype=torch.int32, device=cuda)
        i = torch.cat([torch.arange(5), torch.arange(N), torch.arange(3), torch.arange(N)]).int().to(cuda)
        y = torch.tensor([5, want, 3, want], dtype=dtype, device=cuda)
        if dtype in (torch.float32, torch.float64):
            assert torch.equal(fs.flagsparse_spmv_csr(d, i, p, torch.ones(N, dtype=dtype, device=cuda), (4, N)), y)
        for n_dense in (1, 8, 33):
            C = fs.flagsparse_spmm_csr(d, i, p, torch.ones((N, n_dense), dtype=dtype, device=cuda), (4, N))
            assert torch.equal(C, y[:, None].expand(4, n_dense)), (plus, minus, n_dense)
