"""C entry points that plan or analyse before they multiply: a call that is refused is refused before its first launch.  The
addresses below are never read: nothing reaches a device."""

import pytest

from flagsparse_b200 import _lib

BASE = 1 << 20                       # stands for an array: aligned, and not a null pointer
EINVAL, ERANGE, EALIGN, ESCRATCH = -1, -2, -3, -4


def _stored(fsb_lib, **kw):
    a = dict(vtype=_lib.FSB_BF16, ptype=0, data=BASE, indices=BASE, indptr=BASE, B=BASE, ldb=8, C=BASE, ldc=8, n_rows=100,
             n_cols=100, n_dense=8, nnz=5000, long_rows=0, scratch=BASE, bytes=1 << 30, stream=None)
    a.update(kw)
    return fsb_lib.fsb_spmm_csr_stored(*a.values())


@pytest.mark.parametrize("vtype", [_lib.FSB_F16, _lib.FSB_BF16, _lib.FSB_C64, _lib.FSB_C128])
def test_stored_spmm(fsb_lib, vtype):
    size = {_lib.FSB_F16: 2, _lib.FSB_BF16: 2, _lib.FSB_C64: 8, _lib.FSB_C128: 16}[vtype]
    call = lambda **kw: _stored(fsb_lib, vtype=vtype, **kw)  # noqa: E731
    assert call(indptr=BASE + 2) == EALIGN and call(indptr=BASE + 4, ptype=1) == EALIGN
    assert call(indices=BASE + 2) == EALIGN and call(scratch=BASE + 8) == EALIGN
    for name in ("data", "B", "C"):
        assert call(**{name: BASE + size // 2}) == EALIGN
    for name in ("data", "indices", "indptr", "B", "C", "scratch"):
        assert call(**{name: None}) == EINVAL
    assert call(ldb=7) == EINVAL and call(ldc=7) == EINVAL and call(ptype=2) == EINVAL and call(n_cols=-1) == EINVAL
    assert call(nnz=1 << 31) == ERANGE and call(n_rows=(1 << 31) - 1) == ERANGE and call(n_cols=(1 << 31) - 1) == ERANGE
    assert call(n_dense=1 << 24, ldb=1 << 24, ldc=1 << 24) == ERANGE
    wide = (1 << 24) - 1                        # odd, so one column per access: more column tiles than a grid has
    assert call(n_dense=wide, ldb=wide, ldc=wide, bytes=1 << 40) == ERANGE
    assert call(bytes=fsb_lib.fsb_spmm_stored_scratch_bytes(vtype, 5000, 8) - 1) == ESCRATCH
    assert _stored(fsb_lib, vtype=_lib.FSB_F32) == EINVAL


def test_plan_and_analysis(fsb_lib):
    plan = lambda ptype, indptr, out: fsb_lib.fsb_csr_tile_plan(ptype, indptr, 100, 5000, 1024, out, None)  # noqa: E731
    assert plan(0, BASE + 2, BASE) == EALIGN and plan(1, BASE + 4, BASE) == EALIGN and plan(0, BASE, BASE + 2) == EALIGN
    look = lambda itype, ptype, i, p, s: fsb_lib.fsb_csr_analyze(itype, ptype, i, p, 100, 5000, s, None)  # noqa: E731
    assert look(0, 0, BASE + 2, BASE, BASE) == EALIGN and look(1, 0, BASE + 4, BASE, BASE) == EALIGN
    assert look(0, 0, BASE, BASE + 2, BASE) == EALIGN and look(0, 1, BASE, BASE + 4, BASE) == EALIGN
    assert look(0, 0, BASE, BASE, BASE + 4) == EALIGN


def test_no_two_checks_wait_for_the_same_ticket(fsb_lib):
    """Words as a call leaves them that returned before its kernel had ended (ticket 9 on its way, 7 the last that was written):
    the next call, here one that finds no device, moves on to a number of its own."""
    import ctypes

    import torch

    if torch.cuda.is_available():
        pytest.skip("for a machine on which nothing can be launched")
    host = (ctypes.c_int64 * 10)(*[0] * 8, 7, 9)
    for ticket in (10, 11):
        rc = fsb_lib.fsb_csr_check(0, 0, BASE, BASE, 100, 5000, BASE, ctypes.addressof(host), None)
        assert rc > _lib.FSB_CUDA_ERROR_BASE and list(host) == [0] * 8 + [7, ticket]


@pytest.mark.parametrize("vtype", [_lib.FSB_F16, _lib.FSB_BF16, _lib.FSB_C64, _lib.FSB_C128])
def test_hints_are_arguments_of_their_own(fsb_lib, vtype):
    """An index type is an index type: nothing else rides in it; and only hints that there are."""
    for ptype in (1024, 1025):
        assert fsb_lib.fsb_spmv_csr_stored(vtype, ptype, BASE, BASE, BASE, BASE, BASE, 100, 100, 5000, None, None, 0, None) == EINVAL
        assert fsb_lib.fsb_spmv_csr_stored_even(vtype, ptype, BASE, BASE, BASE, BASE, BASE, 100, 100, 5000, None) == EINVAL
    for hints in (1, 16, 32 + 128):
        assert fsb_lib.fsb_spmm_csr_stored_rows(vtype, 0, BASE, BASE, BASE, BASE, 8, BASE, 8, 100, 100, 8, 5000, hints, BASE, 1 << 30,
                                                None) == EINVAL
