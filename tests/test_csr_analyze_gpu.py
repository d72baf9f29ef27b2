"""fsb_csr_analyze against torch reductions, at lengths around its 16-byte loads, for every pair of index types, aligned or
not, with negative, decreasing and empty inputs."""

import pytest
import torch

from fake_device import fake_analyze
from flagsparse_b200 import _common

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("itype", [torch.int32, torch.int64], ids=str)
@pytest.mark.parametrize("ptype", [torch.int32, torch.int64], ids=str)
def test_statistics(cuda, fsb_lib, itype, ptype):
    gen = torch.Generator().manual_seed(3)
    for nnz in (0, 1, 2, 3, 4, 5, 7, 1023, 4096, 4099, 300001):
        for n_rows in (0, 1, 255, 1024, 70001):
            idx = torch.randint(-5, 1 << 30, (nnz + 1,), generator=gen).to(itype)
            ptr = torch.randint(0, nnz + 1, (n_rows + 2,), generator=gen).to(ptype)
            if n_rows % 2:
                ptr = ptr.sort().values
            for off in (0, 1):
                i, p = idx.to(cuda)[off:off + nnz], ptr.to(cuda)[off:off + n_rows + 1]
                got, want = _common._analyze_csr(i, p, n_rows), fake_analyze(i.cpu(), p.cpu(), n_rows)
                for name in _common.CsrStats.__slots__:
                    assert getattr(got, name) == max(getattr(want, name), 0 if name == "max_row_nnz" else -2**63), (
                        name, nnz, n_rows, off)
