"""Run with FSB_BOUNDS_CHECK=1 (tests/test_bounds_check_bins_gpu.py does, in a child process): layouts of the two-pass SpMV with
one bad number are refused by the checking build of the library, and nothing is launched.

No case depends on the check for its memory safety: every bad number leads to a place inside the arrays and the shared memory
of the kernels, or to nothing at all."""

import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

from flagsparse_b200 import _lib, bins  # noqa: E402
from gpu_util import dev  # noqa: E402
from helpers import assert_spmv_ok, handmade_csr  # noqa: E402


def main():
    L = _lib.lib()
    assert _lib.CHECKING and L.fsb_bounds_check_enabled() == 1, "not the checking build"
    st = torch.cuda.current_stream().cuda_stream
    lens = [3, 0, 40, 700, 1] * 60
    shape = (len(lens), 3001)
    x = np.random.default_rng(1).uniform(-1, 1, shape[1])
    for vdt in ("float32", "float64"):
        d, i, p = handmade_csr(6, lens, shape[1], value_dtype=vdt)
        lay = bins.build_bins_layout(dev(d), dev(i), dev(p), *shape, 700, chunk_cols=400)
        tx = dev(x.astype(vdt))
        y = torch.full((shape[0],), 7.0, dtype=tx.dtype, device=tx.device)

        def product():
            bins.launch_bins(lay, tx, y, *shape, st)
            torch.cuda.synchronize()

        product()
        good = y.clone()
        assert_spmv_ok(good.cpu().numpy(), d, i, p, shape, x.astype(vdt), what=f"{vdt} under the checking build")
        threads, cap = int(L.fsb_spmv_bins_ends()), int(L.fsb_spmv_bins_cap(_lib.FSB_F32 if vdt == "float32" else _lib.FSB_F64))
        n_blocks, last_width = lay.n_blocks, shape[1] - 400 * (lay.n_chunks - 1)
        assert 0 < last_width < 400 and 32 * lay.n_packs % 512 != 0      # room behind the last chunk and the last pack
        cases = [("col", -1, last_width, 1), ("place", 5, lay.n_packs, 8),
                 ("dst", 3, threads + cap, 5), ("chunk_pack", 0, 1, 8), ("block_pack", n_blocks, lay.n_packs - 1, 8),
                 ("block_pack", 0, 1, 8), ("block_start", 2 * n_blocks, shape[0] - 1, 4), ("block_start", 1, 1, 2)]
        if vdt == "float64":
            cases.append(("ends", 0, 1 << 16, 5))        # a slice has 16 entries
        for name, where, bad, kind in cases:
            table = getattr(lay, name).view(-1)
            was = int(table[where])
            table[where] = bad
            y.fill_(7.0)
            try:
                product()
            except IndexError as e:
                assert _lib.BAD_KINDS[kind] in str(e), f"{vdt} {name}: {e}"
            else:
                raise AssertionError(f"{vdt}: {name}[{where}] = {bad} was taken")
            torch.cuda.synchronize()
            assert bool((y == 7.0).all()), "a refused call writes nothing"
            table[where] = was
        product()
        assert torch.equal(y, good)
    print("all cases ok")


if __name__ == "__main__":
    main()
