"""Dtype tables, limits and tolerances shared by the CSR SpMV / SpMM host code.

Mirrors the conventions of the reference's src/flagsparse/sparse_operations/_common.py:22-31 (dtype
whitelists, int32 index limit) and :76-85 (allclose tolerances).  float32 and float64 values have kernels with plans of
their own; the other four value dtypes of the reference's whitelist run through kernels that read them as they are
stored (widetypes.py), on the entry points where the reference accepts them.
"""

import ctypes
import threading

import torch

from . import _lib

SUPPORTED_VALUE_DTYPES = (torch.float16, torch.bfloat16, torch.float32, torch.float64, torch.complex64,
                          torch.complex128)
SUPPORTED_INDEX_DTYPES = (torch.int32, torch.int64)
_INDEX_LIMIT_INT32 = 2**31 - 1

_VTYPE = {torch.float32: _lib.FSB_F32, torch.float64: _lib.FSB_F64}
_ITYPE = {torch.int32: _lib.FSB_I32, torch.int64: _lib.FSB_I64}


def _check_value_dtype(dtype, what="data"):
    if dtype in SUPPORTED_VALUE_DTYPES:
        return
    raise TypeError(
        f"{what} dtype must be one of: float16, bfloat16, float32, float64, complex64, complex128"
    )


def _tolerance_for_dtype(value_dtype):
    """(atol, rtol) used by the reference's allclose checks (_common.py:76-85)."""
    if value_dtype == torch.float16:
        return 2e-3, 2e-3
    if value_dtype == torch.bfloat16:
        return 1e-1, 1e-1
    if value_dtype in (torch.float32, torch.complex64):
        return 1e-6, 1e-5
    if value_dtype in (torch.float64, torch.complex128):
        return 1e-10, 1e-8
    return 1e-6, 1e-5


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_ptr(device):
    if _raw_stream is not None and device.index is not None:
        return _raw_stream(device.index)         # the handle alone, without a Stream object around it
    return torch.cuda.current_stream(device).cuda_stream


class _Here:
    __slots__ = ()

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


_HERE = _Here()


def _on_device(device):
    """Context in which `device` is the current one: nothing to enter where it already is."""
    return _HERE if torch.cuda.current_device() == device.index else torch.cuda.device(device)


def _resolved(t):
    """t with the conjugation or negation that torch keeps as a flag of the tensor (x.conj(), z.conj().imag) carried out:
    the kernels read the memory, and contiguous() leaves the flag as it is."""
    return t.resolve_conj().resolve_neg() if t.is_conj() or t.is_neg() else t


def _ptr(t):
    return t.data_ptr() if t is not None and t.numel() > 0 else None


class CsrStats:
    """The eight numbers fsb_csr_analyze produces, read back with a single device-to-host copy."""

    __slots__ = ("ptr_first", "ptr_last", "n_decreasing", "min_index", "max_index", "max_row_nnz",
                 "n_empty_rows", "n_long_rows")

    def __init__(self, values):
        (self.ptr_first, self.ptr_last, self.n_decreasing, self.min_index, self.max_index,
         self.max_row_nnz, self.n_empty_rows, self.n_long_rows) = (int(v) for v in values)


class _CheckSlot:
    """What fsb_csr_check needs beside the matrix: counters on the device and page-locked memory for the answer.  One per thread
    and device: a call is over when its answer is there, whichever stream it was enqueued on."""

    __slots__ = ("work", "host", "work_ptr", "host_ptr", "_words")

    def __init__(self, device):
        self.host = torch.zeros(10, dtype=torch.int64, pin_memory=True)
        self.work = torch.zeros(7, dtype=torch.int64, device=device)
        torch.cuda.current_stream(device).synchronize()       # the zeros are there for whatever stream comes next
        self.work_ptr, self.host_ptr = self.work.data_ptr(), self.host.data_ptr()
        self._words = (ctypes.c_int64 * 8).from_address(self.host_ptr)

    def stats(self):
        return CsrStats(self._words)


_thread = threading.local()


def _check_slot(device):
    """This thread's slot for `device`, or None where there can be none (not a GPU; first used while a stream is captured)."""
    slots = getattr(_thread, "slots", None)
    if slots is None:
        slots = _thread.slots = {}
    slot = slots.get(device.index)
    if slot is None and device.type == "cuda" and device.index is not None and not torch.cuda.is_current_stream_capturing():
        slot = slots[device.index] = _CheckSlot(device)
    return slot


def _analyze_csr(indices, indptr, n_rows):
    """One fused device pass over indptr and indices (the reference does six reductions with six host
    syncs, spmv_csr.py:404-427); returns CsrStats."""
    L = _lib.lib()
    dev = indptr.device
    with _on_device(dev):
        slot = _check_slot(dev)
        if slot is not None:
            rc = L.fsb_csr_check(_ITYPE[indices.dtype], _ITYPE[indptr.dtype], _ptr(indices), indptr.data_ptr(), n_rows,
                                 indices.numel(), slot.work_ptr, slot.host_ptr, _stream_ptr(dev))
            if rc != _lib.FSB_CAPTURING:
                _lib.check(rc, "fsb_csr_check")
                return slot.stats()
        stats = torch.empty(8, dtype=torch.int64, device=dev)
        rc = L.fsb_csr_analyze(
            _ITYPE[indices.dtype], _ITYPE[indptr.dtype], _ptr(indices), indptr.data_ptr(),
            n_rows, indices.numel(), stats.data_ptr(), _stream_ptr(dev),
        )
    _lib.check(rc, "fsb_csr_analyze")
    return CsrStats(stats.cpu().tolist())


def _tile_plan(indptr, n_rows, nnz, tile_nnz):
    """int32 tile_row[n_tiles + 1] on the device (see fsb_csr_tile_plan in include/fsb.h)."""
    L = _lib.lib()
    n_tiles = int(L.fsb_csr_num_tiles(nnz, tile_nnz))
    plan = torch.empty(n_tiles + 1, dtype=torch.int32, device=indptr.device)
    with _on_device(indptr.device):
        rc = L.fsb_csr_tile_plan(
            _ITYPE[indptr.dtype], indptr.data_ptr(), n_rows, nnz, tile_nnz, plan.data_ptr(),
            _stream_ptr(indptr.device),
        )
    _lib.check(rc, "fsb_csr_tile_plan")
    return plan


class StatusWord:
    """The word through which a kernel reports that one of its bounded waits ran out, and the host side of it.
    The word lives in pinned host memory that the GPU writes directly (only when a wait does run out), so looking
    at it costs neither a copy nor a synchronisation: every call on the same object polls it, and check() waits
    for the last launch first.  A set word is reset and turned into a RuntimeError, so a product whose kernel gave
    up is never handed on silently."""

    def __init__(self, device):
        device = torch.device(device)
        self._cuda = device.type == "cuda"
        self.word = torch.zeros(1, dtype=torch.int32)
        if self._cuda:
            self.word = self.word.pin_memory()       # page-locked: the same address is valid on the device
        self._event = None
        self._what = None

    def data_ptr(self):
        return self.word.data_ptr()

    def item(self):
        return int(self.word[0])

    def posted(self, what, stream=None):
        """Call right after a launch that may set the word; `stream` is the torch stream of that launch (default:
        the current one)."""
        if not self._cuda:
            return
        if self._event is None:
            self._event = torch.cuda.Event()
        self._event.record(stream or torch.cuda.current_stream())
        self._what = what

    def poll(self):
        """Raise if a launch is known to have failed; never waits for the GPU."""
        if int(self.word[0]) != 0:
            self._raise()

    def check(self):
        """Wait for the last launch and raise if it (or an earlier one) failed."""
        if self._event is not None:
            self._event.synchronize()
        if int(self.word[0]) != 0:
            self._raise()

    def _raise(self):
        code, what = int(self.word[0]), self._what or "a kernel of this matrix"
        self.word.zero_()
        raise RuntimeError(f"{what}: a device-side wait ran out (status {code}); the result of that call is "
                           "incomplete")
