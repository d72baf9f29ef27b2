"""Two-pass products on one prepared matrix that overlap in two streams: each call brings the memory between its passes."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import _lib, bins
from gpu_util import dev
from helpers import handmade_csr

pytestmark = pytest.mark.gpu


class _Recorder:
    """The library, noting where every two-pass product is told to keep what goes between its passes."""

    def __init__(self, lib):
        self._lib, self.between = lib, []

    def __getattr__(self, name):
        entry = getattr(self._lib, name)
        if name != "fsb_spmv_csr_bins":
            return entry

        def launch(*args):
            self.between.append((args[14], args[15]))
            return entry(*args)

        return launch


def test_two_streams_share_a_matrix(cuda, fsb_lib, monkeypatch):
    monkeypatch.setattr(bins, "UNEVEN_MIN_NNZ", 1 << 16)
    monkeypatch.setattr(bins, "UNEVEN_MIN_SPAN", 1 << 10)
    lens = np.random.default_rng(1).integers(0, 9, 60000)
    lens[::5000] = 700
    d, i, p = handmade_csr(1, lens.tolist(), 50000)
    prep = fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (60000, 50000))
    assert prep.bins is not None
    gen = torch.Generator().manual_seed(2)
    xs = [torch.randn(50000, generator=gen).to(cuda) for _ in range(2)]
    want = [fs.flagsparse_spmv_csr(x=x, prepared=prep) for x in xs]
    streams, other = [torch.cuda.Stream() for _ in range(2)], torch.cuda.Stream()
    seen = _Recorder(_lib.lib())
    monkeypatch.setattr(bins._lib, "lib", lambda: seen)
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
    assert len(seen.between) == 102
    for p0, n0 in set(seen.between[0::2]):
        assert all(p0 + n0 <= p1 or p1 + n1 <= p0 for p1, n1 in set(seen.between[1::2]))
