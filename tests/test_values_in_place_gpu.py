"""Values written into the caller's array after prepare_spmv_csr: the kernels that read the CSR arrays see them."""

import numpy as np
import pytest
import torch

import flagsparse_b200 as fs
from flagsparse_b200 import bins
from gpu_util import dev, env
from helpers import assert_spmv_ok, handmade_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["vector", "stream", "bins"])
@pytest.mark.parametrize("vdt", ["float32", "float64"])
def test_the_next_product_has_the_new_values(cuda, fsb_lib, monkeypatch, form, vdt):
    if form == "bins":
        for name in ("UNEVEN_MIN_NNZ", "UNEVEN_MIN_SPAN", "F64_MIN_SPAN", "EVEN_MIN_NNZ"):
            monkeypatch.setattr(bins, name, 1 << 10)
    rng = np.random.default_rng(3)
    lens = rng.integers(0, 9, 30000)
    lens[::3000] = 700
    d, i, p = handmade_csr(8, lens.tolist(), 40000, value_dtype=vdt)
    x = rng.uniform(-1, 1, 40000).astype(vdt)
    room = torch.empty(d.size + 1, dtype=torch.from_numpy(d).dtype, device=cuda)
    values = room[1:]                                   # off the 16-byte boundary, as a slice of a larger buffer is
    values.copy_(dev(d))
    with env(FSB_SPMV_ALGO=None if form == "bins" else form):
        prep = fs.prepare_spmv_csr(values, dev(i), dev(p), (30000, 40000))
    assert prep.opt_buckets[0]["kind"] == form
    for step in range(3):
        y = fs.flagsparse_spmv_csr(x=dev(x), prepared=prep)
        assert_spmv_ok(y.cpu().numpy(), d, i, p, (30000, 40000), x, what=f"{form}, values {step}")
        d = rng.uniform(-1, 1, d.size).astype(vdt)
        values.copy_(dev(d))
