"""Infinities and NaN in rows that lie inside a tile, cross one tile boundary and cross several: every element of the result
is the infinity, the NaN or the finite number that the plain sum of the products gives."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from gpu_util import env
from helpers import handmade_csr

pytestmark = pytest.mark.gpu

DTYPES = (torch.float32, torch.float64, torch.float16, torch.bfloat16, torch.complex64, torch.complex128)
N_COLS = 9000
# rows 1 .. 5: inside a tile, across one boundary, across several, inside one again, across one
LENS = [900, 40, 1500, 9000, 30, 2600] + [5] * 200
PLANTS = {"inf": [np.inf], "-inf": [-np.inf], "both": [np.inf, -np.inf], "nan": [np.nan], "inf twice": [np.inf, np.inf]}


def _matrix(dtype, plant, at):
    """Rows 1 .. 5 get the planted values, one near their start and one near their end (at 0) or the other way round."""
    vals, i, p = handmade_csr(5, LENS, N_COLS, value_dtype=np.float64)
    if dtype.is_complex:
        vals = vals + 1j * np.random.default_rng(6).uniform(-1, 1, vals.size)
    for r in range(1, 6):
        for k, v in enumerate(PLANTS[plant]):
            vals[p[r] + 2 if (k + at) % 2 == 0 else p[r + 1] - 3] = v
    return torch.from_numpy(vals).to(dtype), i, p


def _operand(shape, dtype):
    v = np.random.default_rng(7).uniform(0.5, 1.5, shape)
    return torch.from_numpy(v + 1j * v[::-1] if dtype.is_complex else v).to(dtype)


def _row_sums(products, p):
    return np.stack([products[a:b].sum(0) for a, b in zip(p[:-1], p[1:])])


def _check(got, vals, i, p, operand):
    """Compares real and imaginary parts by class: NaN, +inf, -inf, finite."""
    with np.errstate(invalid="ignore"):
        a, b = vals.to(torch.complex128).numpy(), operand.to(torch.complex128).numpy()[i]
        a = a.reshape((-1,) + (1,) * (b.ndim - 1))
        parts = [(a.real * b.real - a.imag * b.imag, got.real if got.is_complex() else got)]
        if got.is_complex():
            parts.append((a.real * b.imag + a.imag * b.real, got.imag))
        for products, g in parts:
            want, g = _row_sums(products, p), g.cpu().to(torch.float64).numpy()
            assert np.array_equal(np.isnan(g), np.isnan(want))
            assert np.array_equal(np.where(np.isinf(g), g, 0), np.where(np.isinf(want), want, 0))


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
@pytest.mark.parametrize("plant", sorted(PLANTS))
def test_spmm(cuda, fsb_lib, dtype, plant):
    shape = (len(LENS), N_COLS)
    for at in (0, 1):
        vals, i, p = _matrix(dtype, plant, at)
        args = [t.to(cuda) for t in (vals, torch.from_numpy(i), torch.from_numpy(p))]
        for n_dense in (1, 6):
            B = _operand((N_COLS, n_dense), dtype)
            _check(fs.flagsparse_spmm_csr(*args, B.to(cuda), shape), vals, i, p, B)
            if dtype in (torch.float32, torch.float64):
                prep = fs.prepare_spmm_csr_opt(*args, shape)
                _check(fs.flagsparse_spmm_csr_opt(B=B.to(cuda), prepared=prep), vals, i, p, B)


@pytest.mark.parametrize("dtype", DTYPES, ids=str)
@pytest.mark.parametrize("plant", sorted(PLANTS))
def test_spmv(cuda, fsb_lib, dtype, plant):
    shape = (len(LENS), N_COLS)
    for at in (0, 1):
        vals, i, p = _matrix(dtype, plant, at)
        args = [t.to(cuda) for t in (vals, torch.from_numpy(i), torch.from_numpy(p))]
        x = _operand((N_COLS,), dtype)
        for algo in (None, "vector", "stream") if dtype in (torch.float32, torch.float64) else (None,):
            with env(FSB_SPMV_ALGO=algo):
                _check(fs.flagsparse_spmv_csr(*args, x.to(cuda), shape), vals, i, p, x)
                prep = fs.prepare_spmv_csr(*args, shape)
                _check(fs.flagsparse_spmv_csr(x=x.to(cuda), prepared=prep), vals, i, p, x)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=str)
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_spmv_row_of_many_tiles(cuda, fsb_lib, dtype, value):
    """A row across more tiles than one thread of the fix-up adds up by itself (its warp does, lane by lane)."""
    _, i, p = handmade_csr(8, [7, 150000, 9], 200000)
    x = _operand((200000,), dtype)
    for at in (7, 60000, 150006):
        vals = torch.from_numpy(np.random.default_rng(9).uniform(-1, 1, i.size)).to(dtype)
        vals[at] = value
        y = fs.flagsparse_spmv_csr(vals.to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), x.to(cuda),
                                   (3, 200000))
        _check(y, vals, i, p, x)
