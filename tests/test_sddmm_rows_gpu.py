"""SDDMM where batches of eight entries meet one, two and more rows, for the lane counts and access widths whose kernels
treat them differently.  Bound: a dot product of K terms in any order, (K + 1) u sum |x y|."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from helpers import handmade_csr

pytestmark = pytest.mark.gpu

LENS = {"one": [8] * 40, "two": [5, 11, 8, 7, 9, 4, 12] * 9, "more": [1, 2, 0, 3, 1, 1, 0, 0, 4] * 21, "odd": [13, 0, 6, 1, 2, 30, 3],
        # batches of one row, of two and of more beside each other, in every order that the groups of a warp can meet
        "mixed": ([16, 5, 3, 1, 2, 1, 4, 8, 8, 1, 1, 6, 24, 7, 9, 2, 2, 2, 2] * 5 + [40] * 3 + [1] * 50) * 2}


@pytest.mark.parametrize("dtype,u", [(torch.float32, 2.0 ** -24), (torch.float64, 2.0 ** -53)], ids=str)
@pytest.mark.parametrize("name", sorted(LENS))
def test_batches_over_rows(cuda, fsb_lib, dtype, u, name):
    n_cols = 200
    _, i, p = handmade_csr(2, LENS[name], n_cols)
    n_rows = len(p) - 1
    row = np.repeat(np.arange(n_rows), np.diff(p))
    prep = fs.prepare_sddmm_csr(torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), (n_rows, n_cols))
    for k in (1, 3, 4, 8, 16, 24, 32, 33, 64, 66, 128, 130):
        rng = np.random.default_rng(k)
        x, y = (torch.from_numpy(rng.uniform(-1, 1, (n, k))).to(dtype) for n in (n_rows, n_cols))
        out = fs.flagsparse_sddmm_csr(x=x.to(cuda), y=y.to(cuda), prepared=prep).cpu().double().numpy()
        xd, yd = x.double().numpy()[row], y.double().numpy()[i]
        assert np.all(np.abs(out - (xd * yd).sum(1)) <= (k + 1) * u * 1.0001 * np.abs(xd * yd).sum(1))


@pytest.mark.parametrize("dtype,u", [(torch.float32, 2.0 ** -24), (torch.float64, 2.0 ** -53)], ids=str)
@pytest.mark.parametrize("k", [3, 4, 64, 128])          # a thread, a half warp, a warp per entry, and single elements
def test_ends_of_tiles(cuda, fsb_lib, dtype, u, k):
    """Tiles of 512 to 2048 entries: one less, all, one more, and out in the place of data."""
    rng = np.random.default_rng(k)
    for nnz in (1, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049):
        ptr = np.unique(np.concatenate([[0, nnz], rng.integers(0, nnz + 1, nnz // 7)]))
        col = rng.integers(0, 50, nnz)
        x, y, d = (rng.uniform(-1, 1, s).astype(np.float32) for s in ((len(ptr) - 1, k), (50, k), nnz))
        x, y, d = (torch.from_numpy(v).to(dtype) for v in (x, y, d))
        prep = fs.prepare_sddmm_csr(torch.from_numpy(col.astype(np.int32)).to(cuda), torch.from_numpy(ptr).to(cuda), (len(ptr) - 1, 50))
        out = d.to(cuda)
        fs.flagsparse_sddmm_csr(out, x=x.to(cuda), y=y.to(cuda), alpha=0.5, beta=-2.0, prepared=prep, out=out)
        xd, yd = x.double().numpy()[np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))], y.double().numpy()[col]
        # the dot product's (k + 1) u, and a rounding for beta * data and one for the sum
        bound = (k + 1) * u * 0.5 * np.abs(xd * yd).sum(1) + 2 * u * (0.5 * np.abs((xd * yd).sum(1)) + 2 * np.abs(d.double().numpy()))
        assert np.all(np.abs(out.cpu().double().numpy() - (0.5 * (xd * yd).sum(1) - 2 * d.double().numpy())) <= 1.0001 * bound), nnz


@pytest.mark.parametrize("dtype,u", [(torch.float32, 2.0 ** -24), (torch.float64, 2.0 ** -53)], ids=str)
@pytest.mark.parametrize("name", sorted(LENS))
def test_rows_of_several_steps(cuda, fsb_lib, dtype, u, name):
    """More than one access per lane of a warp: 16-byte accesses (float32 from 132, float64 from 66 on), single elements and pairs, whole
    last steps and short ones, tiles that end in the middle."""
    n_cols = 200
    _, i, p = handmade_csr(2, LENS[name], n_cols)
    n_rows = len(p) - 1
    row = np.repeat(np.arange(n_rows), np.diff(p))
    prep = fs.prepare_sddmm_csr(torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), (n_rows, n_cols))
    for k in (35, 65, 68, 129, 132, 134, 192, 256, 257, 260, 388):
        rng = np.random.default_rng(k)
        x, y = (torch.from_numpy(rng.uniform(-1, 1, (n, k))).to(dtype) for n in (n_rows, n_cols))
        d = torch.from_numpy(rng.uniform(-1, 1, len(i))).to(dtype)
        out = fs.flagsparse_sddmm_csr(d.to(cuda), x=x.to(cuda), y=y.to(cuda), beta=1.0, prepared=prep).cpu().double().numpy()
        xy, dd = x.double().numpy()[row] * y.double().numpy()[i], d.double().numpy()
        bound = (k + 1) * u * np.abs(xy).sum(1) + 2 * u * (np.abs(xy.sum(1)) + np.abs(dd))
        assert np.all(np.abs(out - xy.sum(1) - dd) <= 1.0001 * bound), k


@pytest.mark.parametrize("dtype,u", [(torch.float32, 2.0 ** -24), (torch.float64, 2.0 ** -53)], ids=str)
def test_several_steps_in_the_instance_for_one(cuda, fsb_lib, dtype, u):
    """Numbers of tiles for which rows of several steps take the instance for one: more than three an SM and up to four; single elements
    in more tiles than that (float64: from 14 an SM on), with rows of 12 entries and more."""
    for n_rows, length, k in ((1 << 15, 16, 33), (1 << 16, 11, 35), (1 << 14, 40, 129), (1 << 14, 16, 132), (1 << 14, 16, 260),
                              (1 << 14, 16, 65), (80000, 14, 35), (1 << 13, 16, 260)):
        gen = torch.Generator(device="cuda").manual_seed(k)
        i = torch.randint(0, 500, (n_rows * length,), generator=gen, device=cuda, dtype=torch.int32)
        p = torch.arange(n_rows + 1, device=cuda) * length
        x, y = (torch.empty(n, k, device=cuda, dtype=dtype).uniform_(-1, 1, generator=gen) for n in (n_rows, 500))
        out = fs.flagsparse_sddmm_csr(x=x, y=y, prepared=fs.prepare_sddmm_csr(i, p, (n_rows, 500)))
        for a in range(0, n_rows, 4096):                        # (in parts: the products of all entries would be large)
            some = slice(a * length, min(n_rows, a + 4096) * length)
            xy = x[a:a + 4096].double().repeat_interleave(length, 0) * y.double()[i[some].long()]
            # (the sum that is compared with has roundings of its own)
            assert bool(((out[some].double() - xy.sum(1)).abs() <= ((k + 1) * u + k * 2.0 ** -53) * 1.0001 * xy.abs().sum(1)).all())
