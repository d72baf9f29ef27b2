"""Products on one prepared matrix that overlap in two streams, for the matrices whose calls bring their own scratch."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import _lib, spmv_csr
from helpers import handmade_csr

pytestmark = pytest.mark.gpu


class _Recorder:
    """The library, noting which scratch every SpMV launch is given (third argument from the end)."""

    def __init__(self, lib):
        self._lib, self.scratch = lib, []

    def __getattr__(self, name):
        entry = getattr(self._lib, name)
        if name not in ("fsb_spmv_csr", "fsb_spmv_csr_stored"):
            return entry

        def launch(*args):
            self.scratch.append(args[-3])
            return entry(*args)

        return launch


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.complex64], ids=str)
def test_two_streams_share_a_matrix(cuda, fsb_lib, monkeypatch, dtype):
    lens = np.random.default_rng(1).integers(0, 12, 4000)
    lens[::500] = 6000
    _, i, p = handmade_csr(1, lens.tolist(), 9000)
    gen = torch.Generator().manual_seed(2)
    draw = lambda n: torch.randn(n, generator=gen, dtype=torch.complex64 if dtype.is_complex else torch.float32).to(dtype)  # noqa: E731
    prep = fs.prepare_spmv_csr(draw(i.size).to(cuda), torch.from_numpy(i).to(cuda), torch.from_numpy(p).to(cuda), (4000, 9000))
    assert prep.tile_row is not None and i.size < 1 << 18
    xs = [draw(9000).to(cuda) for _ in range(2)]
    want = [fs.flagsparse_spmv_csr(x=x, prepared=prep) for x in xs]
    streams, other = [torch.cuda.Stream() for _ in range(2)], torch.cuda.Stream()
    seen = _Recorder(_lib.lib())
    monkeypatch.setattr(spmv_csr._lib, "lib", lambda: seen)
    a = torch.randn(4096, 4096, device=cuda)
    ready = torch.cuda.Event()
    got = [[], []]
    for rounds in (1, 50):                # once so that both streams have their memory, then all at once
        torch.cuda.synchronize()
        if rounds > 1:                    # both streams wait for some tens of milliseconds of other work
            with torch.cuda.stream(other):
                for _ in range(40):
                    a @ a
                ready.record()
            for s in streams:
                s.wait_event(ready)
        for _ in range(rounds):
            for k in range(2):
                with torch.cuda.stream(streams[k]):
                    got[k].append(fs.flagsparse_spmv_csr(x=xs[k], prepared=prep))
    assert not ready.query(), "the calls were not waiting together"
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[k]) for k in range(2) for y in got[k])
    # no scratch is handed to both streams
    assert set(seen.scratch[0::2]).isdisjoint(seen.scratch[1::2]) and None not in seen.scratch
