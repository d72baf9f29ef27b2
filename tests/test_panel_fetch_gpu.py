"""Panel layouts whose slots add straight into accumulators: x fetched by a warp of its own.  Chunks with ragged ends, x off
the 16-byte boundary, more and fewer buffers and warps, many short units: the same bits every time, within the oracle's bound."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import panel as P
from gpu_util import dev, env
from helpers import assert_spmv_ok

pytestmark = pytest.mark.gpu


def _band(n, n_cols, mean, seed):
    """About one entry per row and chunk: `mean` distinct columns anywhere, rows of unequal length."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(mean // 2, 3 * mean // 2, n)
    lens[::97] = 0
    p = np.zeros(n + 1, dtype=np.int32)
    p[1:] = np.cumsum(lens)
    i = np.concatenate([np.sort(rng.choice(n_cols, k, replace=False)) for k in lens]).astype(np.int32)
    return rng.uniform(-1, 1, i.size), i, p


@pytest.mark.parametrize("vdt,buffers,chunk,rounds", [
    ("float32", 2, 32, 4), ("float32", 2, 256, 8), ("float32", 3, 132, 8), ("float32", 8, 128, 16),
    ("float64", 2, 32, 4), ("float64", 4, 132, 8),
])
def test_fetching_warp(cuda, fsb_lib, vdt, buffers, chunk, rounds):
    n, n_cols = 6007, 9001
    d, i, p = _band(n, n_cols, 18, 5)
    d = d.astype(vdt)
    x = np.random.default_rng(6).uniform(-1, 1, n_cols + 3).astype(vdt)
    with env(FSB_SPMV_ALGO="panel", FSB_PANEL_BUFFERS=buffers, FSB_PANEL_CHUNK=chunk, FSB_PANEL_ROUNDS=rounds):
        prep = fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (n, n_cols))
    lay = prep.panel
    assert not lay.flags & (P.FLAG_RUNS | P.FLAG_LONG_RUNS)
    for shift in range(4):
        tx, want = dev(x)[shift:shift + n_cols], None
        for few in (0, P.FLAG_FEW_PIECES):
            lay.flags = (lay.flags & ~P.FLAG_FEW_PIECES) | few
            for _ in range(3):
                y = fs.flagsparse_spmv_csr(x=tx, prepared=prep)
                want = y if want is None else want
                assert torch.equal(y, want)
        prep.check_status()
        assert_spmv_ok(want.cpu().numpy(), d, i, p, (n, n_cols), x[shift:shift + n_cols], what=f"x off by {shift}")


@pytest.mark.parametrize("vdt,few", [("float32", 0), ("float32", P.FLAG_FEW_PIECES), ("float64", P.FLAG_FEW_PIECES)])
def test_more_units_than_a_window(cuda, fsb_lib, vdt, few):
    """The adding warps change their tables of 512 units while the fetching warp runs on: 1251 units a row block."""
    n, n_cols = 6007, 40001
    d, i, p = _band(n, n_cols, 18, 8)
    d = d.astype(vdt)
    x = np.random.default_rng(9).uniform(-1, 1, n_cols).astype(vdt)
    with env(FSB_SPMV_ALGO="panel", FSB_PANEL_CHUNK=32, FSB_PANEL_ROUNDS=4):
        prep = fs.prepare_spmv_csr(dev(d), dev(i), dev(p), (n, n_cols))
    lay = prep.panel
    assert not lay.flags & (P.FLAG_RUNS | P.FLAG_LONG_RUNS) and int((lay.rb_unit_ptr[1:] - lay.rb_unit_ptr[:-1]).max()) > 1024
    lay.flags = (lay.flags & ~P.FLAG_FEW_PIECES) | few
    y = fs.flagsparse_spmv_csr(x=dev(x), prepared=prep)
    prep.check_status()
    assert_spmv_ok(y.cpu().numpy(), d, i, p, (n, n_cols), x, what="three windows of units")
    assert torch.equal(y, fs.flagsparse_spmv_csr(x=dev(x), prepared=prep))


def test_a_wait_that_runs_out_is_reported(cuda, fsb_lib):
    d, i, p = _band(3000, 9000, 18, 7)
    with env(FSB_SPMV_ALGO="panel", FSB_PANEL_CHUNK=128):
        prep = fs.prepare_spmv_csr(dev(d.astype(np.float32)), dev(i), dev(p), (3000, 9000))
    assert not prep.panel.flags & (P.FLAG_RUNS | P.FLAG_LONG_RUNS)
    x = dev(np.ones(9000, dtype=np.float32))
    good = fs.flagsparse_spmv_csr(x=x, prepared=prep)
    prep.panel.flags |= P.FLAG_DEBUG_TIMEOUT
    fs.flagsparse_spmv_csr(x=x, prepared=prep)
    with pytest.raises(RuntimeError, match="wait ran out"):
        prep.check_status()
    prep.panel.flags &= ~P.FLAG_DEBUG_TIMEOUT
    assert torch.equal(fs.flagsparse_spmv_csr(x=x, prepared=prep), good)
    prep.check_status()
