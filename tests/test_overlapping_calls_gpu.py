"""Products on one prepared matrix that overlap in two streams, for the matrices whose calls bring their own scratch."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from helpers import handmade_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.complex64], ids=str)
def test_two_streams_share_a_matrix(cuda, fsb_lib, dtype):
    lens = np.random.default_rng(1).integers(0, 12, 4000)
    lens[::500] = 6000
    _, i, p = handmade_csr(1, lens.tolist(), 9000)
    gen = torch.Generator().manual_seed(2)
    draw = lambda n: torch.randn(n, generator=gen, dtype=torch.complex64 if dtype.is_complex else torch.float32).to(dtype)  # noqa: E731
    prep = fs.prepare_spmv_csr(draw(i.size).to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), (4000, 9000))
    assert prep.tile_row is not None and i.size < 1 << 18
    xs = [draw(9000).to(cuda) for _ in range(2)]
    want = [fs.flagsparse_spmv_csr(x=x, prepared=prep) for x in xs]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(50):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                got[k].append(fs.flagsparse_spmv_csr(x=xs[k], prepared=prep))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[k]) for k in range(2) for y in got[k])
