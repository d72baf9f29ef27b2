"""CSR SpMM host code: the reference's entry points over the hand-written sm_100a kernel.

Same names, arguments, defaults, validation order and exception types as the reference's
src/flagsparse/sparse_operations/spmm_csr.py (_prepare_spmm_csr_matrix :197-255,
_prepare_spmm_csr_inputs :258-281, the launch-override checks :284-334, PreparedCsrSpmmOpt
:337-392, prepare_spmm_csr_opt :480-522, flagsparse_spmm_csr :1057-1126, flagsparse_spmm_csr_opt
:1129-1183).  Both entry points run the same nnz-tiled CUDA kernel; the reference's row-length buckets
and its split workspace for rows over 2048 nnz are replaced by the tile plan and per-tile partial rows.
"""

import os
import time

import torch

from . import _lib, widetypes
from ._common import (
    SUPPORTED_INDEX_DTYPES,
    _INDEX_LIMIT_INT32,
    _ITYPE,
    _VTYPE,
    _analyze_csr,
    _check_slot,
    _check_value_dtype,
    _on_device,
    _ptr,
    _resolved,
    StatusWord,
    _stream_ptr,
    _tile_plan,
)

_STORED_VTYPE = {torch.float16: _lib.FSB_F16, torch.bfloat16: _lib.FSB_BF16, torch.complex64: _lib.FSB_C64,
                 torch.complex128: _lib.FSB_C128}
_SPMM_ALGO_NAMES = {"auto": _lib.FSB_SPMM_AUTO, "plain": _lib.FSB_SPMM_PLAIN, "bulk": _lib.FSB_SPMM_BULK}

# A product whose gathers range over more of B than stays in L2 can be split: A into column panels (each panel's
# slice of B at most this many bytes per column tile, so that it is fetched from DRAM about once) and B / C into
# column tiles of one 128-byte line per row; passes after the first add to C.  Off by default (0): on the 2^20-row
# matrix with 16 uniform entries per row every split measured slower than the single pass (width 32: 0.31 ms with
# two panels, 0.43 ms with four, against 0.23 ms) -- a pass over rows of a few entries each is bound by the latency
# of its read-add-write of C, not by the bytes it saves.  FSB_SPMM_PANEL_MB=<MiB> or FSB_SPMM_PANELS=<n> turn it on.
PANEL_BYTES = 0
COL_TILE_BYTES = 128
# A matrix with a row longer than this gets FSB_SPMM_LONG_ROWS (include/fsb.h).  A group that walks a row alone takes about
# 0.06 us per entry (float32) to 0.12 us (half precisions), up to the 1024 of a tile; sharing it costs 1 to 4 % where it
# brings nothing.  One row of 260 / 400 / 1030 entries, alone against shared: 262144 rows of 16, 16 columns, float32: 50 / 57 /
# 93 us against 46 / 41 / 47 us; 4096 rows of 16, 64 columns, bfloat16: 90 / 111 / 190 us against 62 us; 60000 rows of 31, 64
# columns, float64: 67 / 68 / 91 us against 70 us.
LONG_ROW_NNZ = 256
# The same where a lane takes several accesses per entry (odd widths beyond 32), whose shared form has fewer CTAs in flight:
# 262144 rows of 16, 33 columns, one row of 400 / 600 / 1030: float32 88 / 93 / 120 us alone against 98 / 101 / 105 us, float64
# 174 / 176 / 200 us against 218 / 220 / 222 us; 60000 rows of 31: float64 73 / 74 / 91 us against 83 us, bfloat16 138 / 150 / 174 us
# against 144 us.
LONG_ROW_NNZ_SEVERAL = 640
SPAN_WINDOW = 1 << 20        # consecutive entries over which the column span is sampled


def _panel_bytes():
    v = os.environ.get("FSB_SPMM_PANEL_MB")
    return PANEL_BYTES if v is None else int(float(v) * (1 << 20))


class _CsrPart:
    """CSR arrays of one column panel of A (or of all of A) plus the tile plan and scratch the kernel needs."""

    __slots__ = ("data", "kernel_indices", "kernel_indptr", "n_rows", "tile_row", "_scratch")

    def __init__(self, data, kernel_indices, kernel_indptr, n_rows, tile_nnz):
        self.data, self.kernel_indices, self.kernel_indptr, self.n_rows = data, kernel_indices, kernel_indptr, n_rows
        self.tile_row = _tile_plan(kernel_indptr, n_rows, data.numel(), tile_nnz) if data.numel() > 0 and n_rows > 0 \
            else None
        self._scratch = {}

    def scratch_for(self, n_dense):
        buf = self._scratch.get(n_dense)
        if buf is None:
            nbytes = int(_lib.lib().fsb_spmm_csr_scratch_bytes(_VTYPE[self.data.dtype], self.data.numel(), n_dense))
            buf = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=self.data.device)
            self._scratch = {n_dense: buf}  # keep one width at a time
        return buf


def split_by_column_panels(data, indices, indptr, n_rows, n_cols, n_panels):
    """CSR arrays (data, indices, indptr) of the n_panels column panels of A: panel p holds the entries whose
    column lies in [p * w, (p + 1) * w), w = ceil(n_cols / n_panels), in their original order; every panel keeps
    all n_rows rows (rows without entries in a panel are empty there)."""
    w = -(-n_cols // n_panels)
    lens = (indptr[1:] - indptr[:-1]).to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(n_rows, device=data.device), lens)
    panel_of = torch.div(indices.to(torch.int64), w, rounding_mode="floor")
    out = []
    for p in range(n_panels):
        keep = panel_of == p
        counts = torch.bincount(rows[keep], minlength=n_rows)
        ptr = torch.zeros(n_rows + 1, dtype=indptr.dtype, device=data.device)
        ptr[1:] = torch.cumsum(counts, 0).to(indptr.dtype)
        out.append((data[keep].contiguous(), indices[keep].contiguous(), ptr))
    return out


def _prepare_spmm_csr_matrix(data, indices, indptr, shape, narrow=True):
    """Checks of the reference's function of this name (spmm_csr.py:197-255), in its order.  Returns
    (data, kernel_indices, kernel_indptr, n_rows, n_cols, stats); unlike the reference the indptr keeps
    its 32-bit width when it has one (the kernels read either)."""
    if len(shape) != 2:
        raise ValueError("shape must be a 2-tuple: (n_rows, n_cols)")
    if data.ndim != 1 or indices.ndim != 1 or indptr.ndim != 1:
        raise ValueError("data, indices, and indptr must be 1D tensors")
    n_rows, n_cols = int(shape[0]), int(shape[1])
    if n_rows < 0 or n_cols < 0:
        raise ValueError("shape dimensions must be non-negative")
    if indptr.numel() != n_rows + 1:
        raise ValueError(f"indptr length must be n_rows+1={n_rows + 1}, got {indptr.numel()}")
    if data.numel() != indices.numel():
        raise ValueError("data and indices must have the same length (nnz)")
    if not (data.is_cuda and indices.is_cuda and indptr.is_cuda):
        raise ValueError("data, indices, and indptr must be CUDA tensors")
    if indices.device != data.device or indptr.device != data.device:
        raise ValueError("data, indices, and indptr must be on the same CUDA device")
    _check_value_dtype(data.dtype)
    if indices.dtype not in SUPPORTED_INDEX_DTYPES:
        raise TypeError("indices dtype must be torch.int32 or torch.int64")
    if indptr.dtype not in SUPPORTED_INDEX_DTYPES:
        raise TypeError("indptr dtype must be torch.int32 or torch.int64")

    data = _resolved(data).contiguous()
    indices = indices.contiguous()
    indptr = indptr.contiguous()
    nnz = data.numel()
    stats = _analyze_csr(indices, indptr, n_rows)
    if stats.ptr_first != 0:
        raise ValueError("indptr[0] must be 0")
    if stats.ptr_last != nnz:
        raise ValueError(f"indptr[-1] must equal nnz={nnz}, got {stats.ptr_last}")
    if stats.n_decreasing > 0:
        raise ValueError("indptr must be nondecreasing")
    if nnz > 0:
        if stats.min_index < 0 or stats.max_index >= n_cols:
            raise IndexError("indices out of range for n_cols")
        if stats.max_index > _INDEX_LIMIT_INT32:
            raise ValueError("column indices exceed the int32 range supported by the kernel")
    # a product that uses the matrix once (narrow=False) reads 64-bit indices as they are: the kernels take either, and a
    # pass that narrows them moves more than it saves
    keep = indices.dtype == torch.int32 or (not narrow and data.dtype in _VTYPE)
    kernel_indices = indices if keep else indices.to(torch.int32)
    return data, kernel_indices, indptr, n_rows, n_cols, stats


def _check_spmm_dense(B, data, n_cols):
    """Checks on B of the reference's _prepare_spmm_csr_inputs (spmm_csr.py:271-280)."""
    if B.shape[0] != n_cols:
        raise ValueError(f"B.shape[0] must be n_cols={n_cols}, got {B.shape[0]}")
    if not B.is_cuda:
        raise ValueError("B must be a CUDA tensor")
    if B.device != data.device:
        raise ValueError("B must be on the same CUDA device as the sparse matrix")
    if B.dtype != data.dtype:
        raise TypeError("B dtype must match data dtype")
    return _row_major(B)


def _row_major(B):
    """B as the kernel can read it: unit stride along a row, any stride between rows (the reference copies every
    non-contiguous B, spmm_csr.py:280; a row-strided view needs no copy here)."""
    if B.is_neg() or B.is_conj():
        B = _resolved(B)
    if B.shape[1] <= 1 or B.stride(1) == 1:
        if B.shape[0] <= 1 or B.stride(0) >= B.shape[1]:
            return B
    return B.contiguous()


# (dense columns above which the shape applies, lanes, column factor): the launch shapes the reference picks for its
# base SpMM kernel (spmm_csr.py:284-296).  The CUDA kernel does not use them; they only give the defaults against
# which explicit overrides are checked, and the bookkeeping dictionary callers may look at.
_ALG1_SHAPES = ((64, 32, 4), (32, 32, 2), (16, 32, 1), (8, 16, 1), (4, 8, 1))


def _alg1_shape(n_dense_cols):
    for above, lanes, factor in _ALG1_SHAPES:
        if n_dense_cols > above:
            return lanes, factor
    return 4, 1


def _check_launch_overrides(n_dense_cols, max_row_nnz, block_n=None, block_nnz=None, max_segments=None):
    """The two ways a call can be refused for its launch overrides, as in the reference (spmm_csr.py:299-334): a
    non-positive block size or segment count, and a max_segments that cannot hold the longest row.  Returns the
    reference's bookkeeping for the accepted values."""
    lanes, factor = _alg1_shape(n_dense_cols)
    tile_cols = lanes * factor if block_n is None else block_n
    seg_len = lanes if block_nnz is None else block_nnz
    if min(tile_cols, seg_len) <= 0:
        raise ValueError("block_n and block_nnz, when given, must be positive")
    needed = -(-max_row_nnz // seg_len) if max_row_nnz > 0 else 0
    if max_segments is not None:
        if max_segments <= 0:
            raise ValueError("max_segments, when given, must be positive")
        if needed > int(max_segments):
            raise ValueError(f"the longest row needs {needed} segments of {seg_len} entries; max_segments allows "
                             f"{int(max_segments)}")
    return {"block_n": int(tile_cols), "block_nnz": int(seg_len),
            "max_segments": None if max_segments is None else int(max_segments), "required_segments": int(needed),
            "warp_size": int(lanes), "factor": int(factor), "max_row_nnz": int(max_row_nnz),
            "auto_max_segments": max_segments is None}


def _select_spmm_opt_block_n(n_dense_cols):
    """Column-tile table of the reference's opt path (spmm_csr.py:405-414); informational here."""
    for bound in (8, 16, 32, 64):
        if n_dense_cols <= bound:
            return bound
    return 128


_SPLIT_TABLES = {"long_part_rows": (0, torch.int32), "long_part_starts": (0, torch.int64),
                 "long_part_ends": (0, torch.int64), "long_row_ids": (0, torch.int32),
                 "long_row_part_ptr": (1, torch.int64)}


class PreparedCsrSpmmOpt:
    """Cached CSR metadata for repeated SpMM calls on the same sparse matrix.

    Attribute names follow the reference's class (spmm_csr.py:337-392).  `row_buckets` describes the tile
    plan; the `long_*` split tables of the reference stay empty because rows of any length go through the
    same tiles.  Scratch (two partial rows per tile) depends on the width of B and is cached per width:
    calls that share a prepared object must not overlap on the GPU (float16 / bfloat16 / complex values: each
    call brings its own, so they may).
    """

    __slots__ = (
        "data", "kernel_indices", "kernel_indptr", "shape", "n_rows", "n_cols", "max_row_nnz",
        "row_buckets", "supports_opt", "long_part_rows", "long_part_starts", "long_part_ends",
        "long_row_ids", "long_row_part_ptr", "long_row_fallback_only", "stats", "tile_nnz", "tile_row",
        "_scratch", "_status", "_row_lengths", "wide", "_whole", "_panels", "_span", "_once", "_uneven",
    )

    def __init__(self, data, kernel_indices, kernel_indptr, shape, n_rows, n_cols, stats, tile_nnz, tile_row,
                 wide=None):
        self.data = data
        self.kernel_indices = kernel_indices
        self.kernel_indptr = kernel_indptr
        self.shape = (int(shape[0]), int(shape[1]))
        self.n_rows = int(n_rows)
        self.n_cols = int(n_cols)
        self.max_row_nnz = int(stats.max_row_nnz)
        self.stats = stats
        self.tile_nnz = tile_nnz
        self.tile_row = tile_row
        n_tiles = 0 if tile_row is None else tile_row.numel() - 1
        self.row_buckets = [{"kind": "tiles", "tile_nnz": tile_nnz, "n_tiles": n_tiles, "n_rows": self.n_rows}]
        self._scratch = None
        self.supports_opt = data.dtype in (torch.float32, torch.float64)
        self.long_row_fallback_only = False
        self._status = None
        self._row_lengths = None
        self._once = False
        # where rows differ in length, segments that share a warp are picked by length
        self._uneven = _lib.FSB_SPMM_UNEVEN_ROWS if 4 * self.max_row_nnz * self.n_rows > 5 * data.numel() else 0
        self._whole = None       # the matrix as one _CsrPart (shares the tile plan)
        self._panels = {}        # number of column panels -> list of _CsrPart
        self._span = None        # columns spanned by a window of consecutive entries (median over samples)
        # float16 / bfloat16 / complex values: ("native", []) -- the product goes through fsb_spmm_csr_stored_rows
        self.wide = wide

    def __getattr__(self, name):
        # the reference's tables of split rows, always empty here: made when somebody looks at them
        if name in _SPLIT_TABLES:
            n, dtype = _SPLIT_TABLES[name]
            value = torch.zeros(n, dtype=dtype, device=self.data.device)
            setattr(self, name, value)
            return value
        raise AttributeError(f"{type(self).__name__!r} object has no attribute {name!r}")

    @property
    def row_lengths(self):
        if self._row_lengths is None:
            p = self.kernel_indptr.to(torch.int64)
            self._row_lengths = p[1:] - p[:-1] if self.n_rows > 0 else p.new_empty((0,))
        return self._row_lengths

    # -- how a product of a given width is run --------------------------------------------------------------
    def column_span(self):
        """Median number of columns between the smallest and the largest column index inside windows of
        SPAN_WINDOW consecutive entries: about how many rows of B the CTAs running at one time gather from."""
        if self._span is None:
            idx = self.kernel_indices
            nnz = idx.numel()
            if nnz == 0:
                self._span = 0
            else:
                k = max(1, min(64, nnz // SPAN_WINDOW))
                win = min(SPAN_WINDOW, nnz)
                starts = [(nnz - win) * j // max(1, k - 1) if k > 1 else 0 for j in range(k)]
                spans = [int(idx[s0:s0 + win].max()) - int(idx[s0:s0 + win].min()) + 1 for s0 in starts[:8]]
                spans.sort()
                self._span = spans[len(spans) // 2]
        return self._span

    def n_panels_for(self, n_dense):
        """Column panels of A for a product of this width (1 = the matrix as it is)."""
        forced = int(os.environ.get("FSB_SPMM_PANELS", "0"))
        if forced > 0:
            return forced
        limit = _panel_bytes()
        if limit <= 0 or self.tile_row is None:
            return 1
        sv = self.data.element_size()
        row_bytes = min(n_dense * sv, COL_TILE_BYTES)
        if self.column_span() * row_bytes <= limit:
            return 1                                  # the gathers of concurrent CTAs stay within what L2 holds
        return max(1, min(16, -(-self.n_cols * row_bytes // limit)))

    def parts_for(self, n_panels):
        if n_panels == 1:
            if self._whole is None:
                part = _CsrPart.__new__(_CsrPart)
                part.data, part.kernel_indices, part.kernel_indptr = self.data, self.kernel_indices, self.kernel_indptr
                part.n_rows, part.tile_row, part._scratch = self.n_rows, self.tile_row, {}
                self._whole = part
            return [self._whole]
        parts = self._panels.get(n_panels)
        if parts is None:
            triples = split_by_column_panels(self.data, self.kernel_indices, self.kernel_indptr, self.n_rows,
                                             self.n_cols, n_panels)
            parts = [_CsrPart(d, i, p, self.n_rows, self.tile_nnz) for d, i, p in triples]
            self._panels = {n_panels: parts}          # keep one split at a time
        return parts

    def passes_for(self, n_dense):
        """[(part, first column, width, accumulate)]: the launches of one product, in order."""
        n_panels = self.n_panels_for(n_dense)
        parts = self.parts_for(n_panels)
        sv = self.data.element_size()
        tile = n_dense if n_panels == 1 else max(1, COL_TILE_BYTES // sv)
        out = []
        for c0 in range(0, n_dense, tile):
            for k, part in enumerate(parts):
                out.append((part, c0, min(tile, n_dense - c0), k > 0))
        return out

    def launches_per_product(self, n_dense):
        return sum(2 if (part.tile_row is not None and part.tile_row.numel() > 2) else 1
                   for part, _, _, _ in self.passes_for(n_dense))

    def plan_summary(self, n_dense):
        passes = self.passes_for(n_dense)
        return {"column_panels_of_A": self.n_panels_for(n_dense), "column_tiles_of_B": len({c for _, c, _, _ in passes}),
                "passes": len(passes), "column_span": self.column_span(), "panel_bytes_limit": _panel_bytes()}

    def status_word(self):
        if self._status is None:
            self._status = StatusWord(self.data.device)
        return self._status

    def check_status(self):
        """Wait for the last product on this matrix and raise RuntimeError if its kernel gave up on a bounded
        device-side wait (tiles of C are then unwritten).  Every product also looks, without waiting, at how the
        previous one ended."""
        if self._status is not None:
            self._status.check()
        if self.wide is not None:
            for part in self.wide[1]:
                part.check_status()


def prepare_spmm_csr_opt(data, indices, indptr, shape):
    """Analyse a CSR matrix once for repeated SpMM calls (reference: spmm_csr.py:480-522)."""
    return _prepare_spmm(data, indices, indptr, shape, once=False)


def _prepare_spmm(data, indices, indptr, shape, once, known=None):
    """once: for a single product -- 64-bit indices stay, and the tiles are staged by ordinary loads, which have no
    wait that could run out and so need no status word (a page-locked allocation and an event).  known: the statistics of
    arrays that were made here (contiguous, 32-bit column ids): nothing is left to check."""
    if known is None:
        data, kernel_indices, kernel_indptr, n_rows, n_cols, stats = _prepare_spmm_csr_matrix(
            data, indices, indptr, shape, narrow=not once
        )
    else:
        kernel_indices, kernel_indptr, (n_rows, n_cols), stats = indices, indptr, shape, known
    nnz = data.numel()
    if data.dtype in widetypes.WIDE_DTYPES:
        # read as stored by fsb_spmm_csr_stored_rows, which plans its tiles itself: no second copy of the matrix
        return PreparedCsrSpmmOpt(data, kernel_indices, kernel_indptr, shape, n_rows, n_cols, stats, 0, None,
                                  wide=("native", []))
    tile_nnz, tile_row = 0, None
    if nnz > 0 and n_rows > 0:
        tile_nnz = int(_lib.lib().fsb_spmm_tile_nnz(_VTYPE[data.dtype]))
        tile_row = _tile_plan(kernel_indptr, n_rows, nnz, tile_nnz)
    prepared = PreparedCsrSpmmOpt(data, kernel_indices, kernel_indptr, shape, n_rows, n_cols, stats, tile_nnz, tile_row)
    prepared._once = once
    return prepared


def _long_row(n_dense, element_size):
    """Longest row up to which a product of this width does without FSB_SPMM_LONG_ROWS."""
    vw = min(16 // element_size, n_dense & -n_dense)      # widest access that divides a row of B
    several = n_dense > 32 * vw and vw * element_size < 16
    return LONG_ROW_NNZ_SEVERAL if several else LONG_ROW_NNZ


def _shares_long_rows(max_row_nnz, n_dense, element_size):
    """Whether a product of this width gets FSB_SPMM_LONG_ROWS."""
    return max_row_nnz > _long_row(n_dense, element_size)


def _spmm_launch(prepared, B, C):
    """Enqueue C = A B on the current stream.  Stands in for _triton_spmm_csr_impl (spmm_csr.py:525-599)
    and _triton_spmm_csr_impl_opt_prepared (:1033-1055).  One launch of the tiled kernel per pass: the whole
    product, or (column panel of A) x (column tile of B) passes when B is too large to be gathered from L2."""
    L = _lib.lib()
    p = prepared
    dev = p.data.device
    n_dense = int(B.shape[1])
    if p.n_rows == 0 or n_dense == 0:
        return
    algo = _SPMM_ALGO_NAMES.get(os.environ.get("FSB_SPMM_ALGO", "auto").strip().lower(), _lib.FSB_SPMM_AUTO)
    status = None
    if p._once and algo == _lib.FSB_SPMM_AUTO:
        algo = _lib.FSB_SPMM_PLAIN
    else:
        status = p.status_word()
        status.poll()
    sv = B.element_size()
    if p.max_row_nnz > LONG_ROW_NNZ and _shares_long_rows(p.max_row_nnz, n_dense, sv):
        algo |= _lib.FSB_SPMM_LONG_ROWS
    algo |= p._uneven
    vt, it, pt = _VTYPE[p.data.dtype], _ITYPE[p.kernel_indices.dtype], _ITYPE[p.kernel_indptr.dtype]
    ldb, ldc = B.stride(0), C.stride(0)
    stream = _stream_ptr(dev)
    with _on_device(dev):
        for part, c0, width, accumulate in p.passes_for(n_dense):
            scratch = part.scratch_for(width) if part.tile_row is not None else None
            rc = L.fsb_spmm_csr(
                vt, it, pt, _ptr(part.data), _ptr(part.kernel_indices), part.kernel_indptr.data_ptr(),
                B.data_ptr() + c0 * sv, ldb, C.data_ptr() + c0 * sv, ldc, p.n_rows, p.n_cols, width,
                part.data.numel(), algo | (_lib.FSB_SPMM_ACCUMULATE if accumulate else 0),
                None if part.tile_row is None else part.tile_row.data_ptr(),
                None if scratch is None else scratch.data_ptr(), 0 if scratch is None else scratch.numel(),
                None if status is None else status.data_ptr(), stream,
            )
            _lib.check(rc, "fsb_spmm_csr")
    if status is not None:
        status.posted("fsb_spmm_csr")


def _check_out(out, device, shape, dtype, device_msg):
    if not out.is_cuda:
        raise ValueError("out must be a CUDA tensor")
    if out.device != device:
        raise ValueError(device_msg)
    if out.shape != shape or out.dtype != dtype:
        raise ValueError("out shape/dtype must match result")


def _spmm_launch_stored(prepared, B, C):
    """Enqueue C = A B for float16 / bfloat16 / complex values with B and C in the matrix's own type: the tiled kernel,
    which reads 2-byte values as they are and rounds every element of C once.  Stands in for the reference's base launch
    on these types (_triton_spmm_csr_impl, spmm_csr.py:525-599)."""
    p = prepared
    dev = p.data.device
    n_dense, nnz = int(B.shape[1]), p.data.numel()
    if p.n_rows == 0 or n_dense == 0:
        return
    L = _lib.lib()
    vt = _STORED_VTYPE[p.data.dtype]
    scratch = torch.empty(int(L.fsb_spmm_stored_scratch_bytes(vt, nnz, n_dense)), dtype=torch.uint8, device=dev)
    with _on_device(dev):
        rc = L.fsb_spmm_csr_stored_rows(
            vt, _ITYPE[p.kernel_indptr.dtype], _ptr(p.data), _ptr(p.kernel_indices), p.kernel_indptr.data_ptr(),
            _ptr(B), B.stride(0) if B.shape[0] > 1 else n_dense, C.data_ptr(), n_dense, p.n_rows, p.n_cols, n_dense, nnz,
            (_lib.FSB_SPMM_LONG_ROWS if _shares_long_rows(p.max_row_nnz, n_dense, B.element_size()) else 0) | p._uneven,
            scratch.data_ptr(), scratch.numel(), _stream_ptr(dev),
        )
    _lib.check(rc, "fsb_spmm_csr_stored_rows")


def _run_spmm(prepared, B, out, return_time):
    dev, dtype = prepared.data.device, prepared.data.dtype
    shape = (prepared.n_rows, int(B.shape[1]))
    # float16 / bfloat16 / complex products never write into `out` while B is still read: it may be B itself there
    direct = out is not None and out.is_contiguous() and not out.is_neg() and prepared.wide is None
    C = out if direct else torch.empty(shape, dtype=dtype, device=dev)
    t0 = None
    if return_time:
        torch.cuda.synchronize(dev)
        t0 = time.perf_counter()
    if prepared.wide is not None:
        _spmm_launch_stored(prepared, _row_major(B), C)
    else:
        _spmm_launch(prepared, B, C)
    elapsed_ms = None
    if return_time:
        torch.cuda.synchronize(dev)
        elapsed_ms = (time.perf_counter() - t0) * 1000.0
        prepared.check_status()
    if out is not None and not direct:
        out.copy_(C)
        C = out
    if return_time:
        return C, elapsed_ms
    return C


_SPMM_SWITCHES = ("FSB_SPMM_ALGO", "FSB_SPMM_PANELS", "FSB_SPMM_PANEL_MB")


def _spmm_once(data, indices, indptr, B, shape):
    """C = A B straight from the arrays, where every argument is as the kernels read it, by one call that checks the arrays, plans
    the tiles, waits for the answer and enqueues the product.  None where that was not done: the arguments are for the general
    path, which also finds the words for what is wrong with them."""
    if not (isinstance(data, torch.Tensor) and isinstance(indices, torch.Tensor) and isinstance(indptr, torch.Tensor)):
        return None
    dev, dtype = data.device, data.dtype
    if dev.type != "cuda" or indices.device != dev or indptr.device != dev or B.device != dev or B.dtype != dtype:
        return None
    vt, it, pt = _VTYPE.get(dtype), _ITYPE.get(indices.dtype), _ITYPE.get(indptr.dtype)
    if vt is None:
        vt = _STORED_VTYPE.get(dtype)
        if it != _lib.FSB_I32:
            return None
    elif any(name in os.environ for name in _SPMM_SWITCHES):
        return None
    if vt is None or it is None or pt is None or data.ndim != 1 or indices.ndim != 1 or indptr.ndim != 1 or len(shape) != 2:
        return None
    n_rows, n_cols, nnz, n_dense = int(shape[0]), int(shape[1]), data.numel(), int(B.shape[1])
    if not (0 < nnz == indices.numel() and 0 < n_rows == indptr.numel() - 1 and B.shape[0] == n_cols < _INDEX_LIMIT_INT32
            and n_dense > 0):
        return None
    if not (data.is_contiguous() and indices.is_contiguous() and indptr.is_contiguous() and B.is_contiguous()):
        return None
    if data.is_neg() or B.is_neg() or data.is_conj() or B.is_conj():
        return None
    L = _lib.lib()
    with _on_device(dev):
        slot = _check_slot(dev)
        if slot is None:
            return None
        C = torch.empty((n_rows, n_dense), dtype=dtype, device=dev)
        scratch = torch.empty(int(L.fsb_spmm_stored_scratch_bytes(vt, nnz, n_dense)), dtype=torch.uint8, device=dev)
        rc = L.fsb_spmm_csr_once(
            vt, it, pt, data.data_ptr(), indices.data_ptr(), indptr.data_ptr(), B.data_ptr(), n_dense, C.data_ptr(), n_dense, n_rows,
            n_cols, n_dense, nnz, _long_row(n_dense, data.element_size()), scratch.data_ptr(), scratch.numel(), slot.work_ptr,
            slot.host_ptr, _stream_ptr(dev))
    if rc == _lib.FSB_OK:
        return C
    if rc not in (_lib.FSB_NOT_LAUNCHED, _lib.FSB_CAPTURING):
        _lib.check(rc, "fsb_spmm_csr_once")
    return None


def flagsparse_spmm_csr(data, indices, indptr, B, shape, block_n=None, block_nnz=None, max_segments=None,
                        out=None, return_time=False):
    """CSR SpMM: C = A @ B (reference: spmm_csr.py:1057-1126, same arguments and defaults).

    A is given as CSR arrays; B is a dense CUDA tensor of shape (n_cols, n_dense_cols), any strides.
    block_n / block_nnz / max_segments are the reference's Triton launch overrides: validated the same
    way, otherwise unused.  Unlike the reference this call does not synchronise the device unless
    return_time is set.
    """
    if block_n is not None and block_n <= 0:
        raise ValueError("block_n must be positive when provided")
    if block_nnz is not None and block_nnz <= 0:
        raise ValueError("block_nnz must be positive when provided")
    if max_segments is not None and max_segments <= 0:
        raise ValueError("max_segments must be positive when provided")
    if B.ndim != 2:
        raise ValueError("B must be a 2D dense tensor")
    if out is None and not return_time and block_n is None and block_nnz is None and max_segments is None:
        C = _spmm_once(data, indices, indptr, B, shape)
        if C is not None:
            return C
    prepared = _prepare_spmm(data, indices, indptr, shape, once=True)
    B = _check_spmm_dense(B, prepared.data, prepared.n_cols)
    n_dense_cols = int(B.shape[1])
    _check_launch_overrides(n_dense_cols, prepared.max_row_nnz, block_n=block_n, block_nnz=block_nnz,
                                     max_segments=max_segments)
    if out is not None:
        _check_out(out, prepared.data.device, (prepared.n_rows, n_dense_cols), prepared.data.dtype,
                   "out must be on the same CUDA device as the inputs")
    return _run_spmm(prepared, B, out, return_time)


def flagsparse_spmm_csr_opt(data=None, indices=None, indptr=None, B=None, shape=None, prepared=None, out=None,
                            return_time=False):
    """CSR SpMM on a prepared matrix (reference: spmm_csr.py:1129-1183, same arguments and defaults)."""
    if prepared is not None and not isinstance(prepared, PreparedCsrSpmmOpt):
        raise TypeError("prepared must be a PreparedCsrSpmmOpt instance")
    if prepared is None:
        if any(arg is None for arg in (data, indices, indptr, shape)):
            raise ValueError("data, indices, indptr, and shape are required when prepared is not provided")
        prepared = _prepare_spmm(data, indices, indptr, shape, once=True)
    elif shape is not None:
        resolved_shape = (int(shape[0]), int(shape[1]))
        if resolved_shape != prepared.shape:
            raise ValueError(f"shape {resolved_shape} does not match prepared.shape {prepared.shape}")
    if B is None:
        raise ValueError("B is required")
    if not prepared.supports_opt:
        raise TypeError("flagsparse_spmm_csr_opt only supports float32 and float64")
    if not B.is_cuda:
        raise ValueError("B must be a CUDA tensor")
    if B.device != prepared.data.device:
        raise ValueError("B must be on the same CUDA device as sparse matrix data")
    if out is not None:
        _check_out(out, prepared.data.device, (prepared.n_rows, int(B.shape[1])), prepared.data.dtype,
                   "out must be on the same CUDA device as sparse matrix data")
    # checks the reference makes inside its launch helper (:1040-1046)
    if B.dtype != prepared.data.dtype:
        raise TypeError("B dtype must match sparse matrix dtype")
    if B.shape[0] != prepared.n_cols:
        raise ValueError(f"B.shape[0] must be n_cols={prepared.n_cols}, got {B.shape[0]}")
    if B.ndim != 2:
        raise ValueError("B must be a 2D dense tensor")
    return _run_spmm(prepared, _row_major(B), out, return_time)
