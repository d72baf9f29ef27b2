"""CSR SpMV host code: the reference's entry points over hand-written sm_100a kernels.

Same names, arguments, defaults, validation order and exception types as the reference's
src/flagsparse/sparse_operations/spmv_csr.py (PreparedCsrSpmv :9-58, _prepare_spmv_csr_matrix :379-436,
_validate_spmv_x :439-452, prepare_spmv_csr :455-495, flagsparse_spmv_csr :557-610, the COO front-end
:613-758).  What differs is below the boundary: one fused analysis pass instead of six reductions, an
nnz-tile plan instead of row-length buckets, and CUDA kernels (libfsb.so) instead of Triton launches.
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
    _stream_ptr,
    _tile_plan,
)

# matrices below this many nnz are a handful of tiles: the single-launch vector kernel wins on latency
_STREAM_MIN_NNZ = 1 << 18
# the vector kernel gives a row to at most 32 lanes, so it is kept away from very long rows
_VECTOR_MAX_ROW_NNZ = 4096
# "uniform" rows: the longest row is within this factor (plus a small allowance) of the mean row length
_UNIFORM_ROW_FACTOR = 8
_UNIFORM_ROW_SLACK = 64
# The same for matrices of less than _STREAM_MIN_NNZ entries, by bytes per value.  Lanes per row against the stream kernel,
# longest row 120 / 200 / 250 / 300 / 400 / 600: 4096 rows of 16, float32: 10.2 / 10.4 / 11.3 / 12.7 / 16.4 / 22.6 us against 15.1 us,
# float64: 10.3 / 14.4 / 16.4 / 18.5 / 24.6 / 33.9 us; 10000 rows of 24, float32: 10.3 / 12.3 / 13.0 / 14.4 / 18.5 / 24.7 us, float64:
# 12.3 / 16.4 / 18.7 / 22.6 / 28.7 / 39.0 us; 4096 rows of 48, from 600 and from 400 on.
_SMALL_ROW_SLACK = {4: 256, 8: 64}
# regroup banded matrices for the panel kernel (costs a second copy of the entries); FSB_SPMV_PANEL=0 turns it off
_PANEL_ENABLED = os.environ.get("FSB_SPMV_PANEL", "1") != "0"


def _long_rows_enabled():
    """Split the long rows of skewed matrices off to the row-group panel kernel; FSB_SPMV_LONG_ROWS=0 turns it off."""
    return os.environ.get("FSB_SPMV_LONG_ROWS", "1") != "0"


_WIDE_VTYPE = {torch.float16: _lib.FSB_F16, torch.bfloat16: _lib.FSB_BF16, torch.complex64: _lib.FSB_C64,
               torch.complex128: _lib.FSB_C128}
_ALGO_NAMES = {"auto": _lib.FSB_SPMV_AUTO, "vector": _lib.FSB_SPMV_VECTOR, "stream": _lib.FSB_SPMV_STREAM,
               "panel": _lib.FSB_SPMV_PANEL}


def _resolve_block_nnz(max_row_nnz, block_nnz, max_segments):
    """block_nnz / max_segments bookkeeping of the reference (spmv_csr.py:465-475).  The CUDA kernels do
    not use either number; they are kept as attributes of the prepared object."""
    block_nnz_use = block_nnz
    if max_segments is None:
        max_segments_use = max((max_row_nnz + block_nnz_use - 1) // block_nnz_use, 1)
        while max_segments_use > 2048 and block_nnz_use < 65536:
            block_nnz_use *= 2
            max_segments_use = max((max_row_nnz + block_nnz_use - 1) // block_nnz_use, 1)
    else:
        max_segments_use = max_segments
    return block_nnz_use, max_segments_use


def _select_spmv_algo(n_rows, nnz, max_row_nnz, element_size=4):
    """Kernel choice from indptr statistics.  Rows of about equal length (longest row within a small
    factor of the mean) go to the lanes-per-row vector kernel, which needs one launch, no scratch, and leaves
    the whole L1 to the gathers of x; skewed row lengths go to the nnz-tiled stream kernel, whose work per
    CTA does not depend on the row structure.  Small matrices take the vector kernel unless a row is long."""
    forced = os.environ.get("FSB_SPMV_ALGO", "").strip().lower()
    if forced in ("vector", "stream", "panel"):
        return _ALGO_NAMES[forced]
    return _lib.FSB_SPMV_VECTOR if max_row_nnz <= _longest_even(n_rows, nnz, element_size) else _lib.FSB_SPMV_STREAM


def _longest_even(n_rows, nnz, element_size):
    """Longest row of a float32 / float64 matrix up to which its rows are even: one launch of the kernels for such rows against two
    of the stream kernel, until the longest row takes its lanes longer than that."""
    slack = _SMALL_ROW_SLACK[element_size] if nnz < _STREAM_MIN_NNZ else _UNIFORM_ROW_SLACK
    return min(_VECTOR_MAX_ROW_NNZ, int(_UNIFORM_ROW_FACTOR * (nnz / max(n_rows, 1)) + slack))


# Longest row from which the tiled kernel for float16 / bfloat16 / complex values is taken.  A row of n entries takes its L
# lanes about 0.15 n / L us (complex), and twice that while others keep memory busy; the tiled kernel takes a second launch,
# and complex values their way through shared memory: 6 to 15 % of complex64, 25 to 45 % of complex128.  So the line for
# complex values is a number of entries per lane, or a share of all entries where that is more (_UNEVEN_ENTRIES[bytes per
# value], for four lanes).  Lanes per row against tiles, longest row 200 / 300 / 400 / 600 / 1000 / 2000:
# 30000 rows of 16, complex64: 12 / 16 / 19 / 25 / 39 / 74 us against 15 us, complex128: 14 / 18 / 23 / 29 / 47 / 88 us against 15 us,
# bfloat16: 14 / 19 / 22 / 31 / 45 / 81 us against 16 us;
# 500009 rows of 24, complex64: 64 / 64 / 64 / 66 / 82 / 124 us against 74 us, complex128: 80 / 81 / 84 / 83 / 101 / 158 us against
# 113 us, bfloat16: 64 / 69 / 76 / 92 / 119 / 197 us against 60 us;
# 2000000 rows of 20, complex64: 209 / 214 / 213 / 213 / 220 / 272 us against 223 us, complex128: 295 / 305 / 303 / 300 / 302 / 362 us
# against 359 us, bfloat16: 187 / 187 / 187 / 187 / 215 / 290 us against 176 us.
_UNEVEN_MIN = 288
_UNEVEN_PER_LANE = 72
_UNEVEN_ENTRIES = {8: 35000, 16: 18000}


def _longest_even_stored(n_rows, nnz, element_size):
    """The same for float16 / bfloat16 / complex values."""
    mean = nnz / max(n_rows, 1)
    line = _UNIFORM_ROW_FACTOR * mean + _UNIFORM_ROW_SLACK
    if element_size not in _UNEVEN_ENTRIES:
        return int(max(line, _UNEVEN_MIN))
    lanes = 2                            # as stored_launch in csrc/spmv_wide.cu gives them to a row
    while lanes < 32 and 6 * lanes < int(mean) + 3:
        lanes *= 2
    return int(max(line, _UNEVEN_PER_LANE * lanes, nnz / _UNEVEN_ENTRIES[element_size] * lanes / 4))


# Longest row, in means (plus eight entries), up to which neighbouring rows stay on one SM (csrc/spmv_rows.cuh): its warps hold more
# rows together than those of the kernel that spreads the rows over all SMs, and all of them wait for the longest.  600000 rows,
# columns anywhere, Zipf lengths cut off at 4.2 / 7.1 / 11.7 / 20 means, us spread / on one SM: float16 37 / 31, 48 / 41, 62 / 51,
# 31 / 37; float32 35 / 33, 49 / 44, 64 / 53, 29 / 37; float64 41 / 39, 61 / 66, 84 / 92, 33 / 38; complex64 41 / 37, 49 / 58, 62 / 82,
# 29 / 33; complex128 59 / 72, 81 / 100, 104 / 153, 52 / 76.
_NEIGHBOUR_MEANS = {2: 10, 4: 10, 8: 5, 16: 3}


def _longest_neighbour(n_rows, nnz, element_size):
    return _NEIGHBOUR_MEANS[element_size] * nnz // max(n_rows, 1) + 8


def _uneven_rows(n_rows, nnz, max_row_nnz, element_size):
    """Whether the longest row leaves the lanes-per-row kernel for float16 / bfloat16 / complex values waiting for it."""
    return max_row_nnz > _longest_even_stored(n_rows, nnz, element_size)


class PreparedCsrSpmv:
    """Cached CSR metadata for repeated SpMV calls on the same sparse matrix.

    Carries the attributes of the reference's class (spmv_csr.py:9-58) plus the tile plan and scratch of
    the stream kernel.  `opt_buckets` describes the plan (the reference lists row ids per length bucket
    there).  Calls on one prepared matrix may overlap in several streams where each brings the scratch it needs: matrices
    of less than _STREAM_MIN_NNZ entries, float16 / bfloat16 / complex values, the two-pass form (a call that is refused the
    memory between the passes takes one, with the kernel that its rows get without them), and every matrix that takes
    the lanes-per-row or the panel kernel, which need none.  Larger matrices on the stream kernel, and matrices whose long rows
    were split off, own one buffer that their calls share: these calls must not overlap on the GPU.
    """

    __slots__ = (
        "data", "kernel_indices", "kernel_indptr", "shape", "n_rows", "n_cols", "block_nnz",
        "max_segments", "max_row_nnz", "opt_buckets", "supports_opt", "stats", "algo", "tuning",
        "tile_nnz", "tile_row", "scratch", "panel", "long_rows", "wide", "bins", "uneven", "vector_tuning",
    )

    def __init__(self, data, kernel_indices, kernel_indptr, shape, n_rows, n_cols, block_nnz,
                 max_segments, max_row_nnz, stats, algo, tuning, tile_nnz, tile_row, scratch, panel=None,
                 long_rows=None, wide=None, bins=None):
        self.data = data
        self.kernel_indices = kernel_indices
        self.kernel_indptr = kernel_indptr
        self.shape = (int(shape[0]), int(shape[1]))
        self.n_rows = n_rows
        self.n_cols = n_cols
        self.block_nnz = block_nnz
        self.max_segments = max_segments
        self.max_row_nnz = max_row_nnz
        # whether a row is too long for neighbouring rows to stay on one SM
        self.uneven = max_row_nnz > _longest_neighbour(n_rows, data.numel(), data.element_size())
        # what fsb_spmv_csr is told of the rows where FSB_SPMV_VECTOR picks its lanes itself
        self.vector_tuning = 0 if self.uneven else _lib.FSB_SPMV_EVEN_ROWS
        self.supports_opt = data.dtype in (torch.float32, torch.float64)
        self.stats = stats
        self.algo = algo
        self.tuning = tuning
        self.tile_nnz = tile_nnz
        self.tile_row = tile_row
        self.scratch = scratch
        self.panel = panel
        self.long_rows = long_rows   # (prepared short-row part, LongRowLayout) when the long rows were split off
        # float16 / bfloat16 / complex values: ("native", []) -- the product goes through fsb_spmv_csr_stored
        self.wide = wide
        self.bins = bins             # the entries regrouped for the two-pass kernels (bins.py)
        n_tiles = 0 if tile_row is None else tile_row.numel() - 1
        kind = {_lib.FSB_SPMV_STREAM: "stream", _lib.FSB_SPMV_PANEL: "panel"}.get(algo, "vector")
        if bins is not None:
            kind = "bins"
        if long_rows is not None:
            kind = "long-row panel + " + long_rows[0].opt_buckets[0]["kind"]
        self.opt_buckets = [{"kind": kind, "tile_nnz": tile_nnz, "n_tiles": n_tiles, "n_rows": n_rows}]

    def _status_words(self):
        if self.panel is not None:
            yield self.panel.status
        if self.long_rows is not None:
            yield self.long_rows[1].status
            yield from self.long_rows[0]._status_words()

    def check_status(self):
        """Wait for the last product on this matrix and raise RuntimeError if one of its kernels gave up on a
        bounded device-side wait (its rows of y are then incomplete).  Every product also looks, without waiting,
        at how the previous one ended."""
        for word in self._status_words():
            word.check()


def _prepare_spmv_csr_matrix(data, indices, indptr, shape, narrow=True, stats=None):
    """Validate and normalise the CSR arrays; same checks, order and exception types as the reference's
    function of this name (spmv_csr.py:379-436).  narrow=False leaves the indices of float32 / float64 matrices at their
    width (a one-shot product reads them once: the kernels take either, and a pass that narrows them moves more than it
    saves).  stats: what the analysis of these very arrays gave.  Returns (data, kernel_indices, kernel_indptr, n_rows,
    n_cols, stats)."""
    if not (torch.is_tensor(data) and torch.is_tensor(indices) and torch.is_tensor(indptr)):
        raise TypeError("data, indices and indptr have to be torch.Tensor objects")
    if data.ndim != 1 or indices.ndim != 1 or indptr.ndim != 1:
        raise ValueError("data, indices and indptr have to be one-dimensional")
    n_rows, n_cols = int(shape[0]), int(shape[1])
    if indptr.numel() != n_rows + 1:
        raise ValueError(f"indptr has {indptr.numel()} entries, {n_rows} rows need {n_rows + 1}")
    if data.numel() != indices.numel():
        raise ValueError(f"{data.numel()} values but {indices.numel()} column indices")
    if not (data.is_cuda and indices.is_cuda and indptr.is_cuda):
        raise ValueError("data, indices and indptr have to live on a CUDA device")
    _check_value_dtype(data.dtype)
    if indices.dtype not in SUPPORTED_INDEX_DTYPES:
        raise TypeError(f"indices are {indices.dtype}; int32 or int64 is needed")

    data = _resolved(data).contiguous()
    indices = indices.contiguous()
    indptr = indptr.contiguous()
    if indptr.dtype not in SUPPORTED_INDEX_DTYPES:
        # the reference accepts any integer indptr and converts it (:423-425)
        indptr = indptr.to(torch.int64)

    nnz = data.numel()
    if stats is None:
        stats = _analyze_csr(indices, indptr, n_rows)
    if stats.ptr_first != 0:
        raise ValueError("indptr[0] is not 0")
    if stats.ptr_last != nnz:
        raise ValueError(f"indptr[-1] is {stats.ptr_last}, the arrays hold {nnz} entries")
    if stats.n_decreasing > 0:
        raise ValueError("indptr decreases somewhere")
    if nnz > 0:
        if stats.min_index < 0 or stats.max_index >= n_cols:
            raise IndexError(f"column indices span [{stats.min_index}, {stats.max_index}], the matrix has {n_cols} columns")
        if stats.max_index > _INDEX_LIMIT_INT32:
            raise ValueError(f"int64 column index {stats.max_index} exceeds the int32 kernel range")
    if not narrow and data.dtype in _VTYPE:
        return data, indices, indptr, n_rows, n_cols, stats
    # same narrowing as the reference (:422-425): 32-bit column indices always, 32-bit indptr when it fits
    kernel_indices = indices.to(torch.int32) if indices.dtype == torch.int64 else indices
    kernel_indptr = indptr.to(torch.int32) if nnz <= _INDEX_LIMIT_INT32 else indptr.to(torch.int64)
    return data, kernel_indices, kernel_indptr, n_rows, n_cols, stats


def _validate_spmv_x(x, prepared):
    """x against a prepared matrix: the checks of the reference's _validate_spmv_x (spmv_csr.py:439-452) in its
    order, each with the exception type it raises there.  Returns x, contiguous."""
    if not isinstance(x, torch.Tensor):   # None included
        raise TypeError("x has to be a torch.Tensor")
    a = prepared.data
    if x.ndim == 1 and x.dtype == a.dtype and x.numel() == prepared.n_cols and x.device == a.device:
        return (_resolved(x) if x.is_neg() or x.is_conj() else x).contiguous()
    for failed, exc, why in (
        (x.ndim != 1, ValueError, "x has to be one-dimensional"),
        (not x.is_cuda, ValueError, "x has to live on a CUDA device"),
        (x.dtype != a.dtype, TypeError, f"x is {x.dtype}, the matrix holds {a.dtype}"),
        (x.numel() != prepared.n_cols, ValueError, f"x has {x.numel()} elements, the matrix {prepared.n_cols} columns"),
        (x.device != a.device, ValueError, f"x is on {x.device}, the matrix on {a.device}"),
    ):
        if failed:
            raise exc(why)
    return _resolved(x).contiguous()


def prepare_spmv_csr(data, indices, indptr, shape, block_nnz=256, max_segments=None):
    """Analyse a CSR matrix once for repeated SpMV calls (reference: spmv_csr.py:455-495).

    Values written into `data` afterwards are seen by the next product of matrices on the lanes-per-row, the stream and the
    two-pass kernels, which read the array itself (opt_buckets[0]["kind"] "vector", "stream", "bins"); the panel and the
    long-row form keep a copy of the values in their own order, made here: prepare again after a change.  `indices` and
    `indptr` belong to what is prepared and must not change in any form.
    """
    return _prepare_spmv_csr(data, indices, indptr, shape, block_nnz, max_segments, reuse_expected=True)


def _split_long_rows(data, kernel_indices, kernel_indptr, n_rows, n_cols, shape, block_nnz, max_segments):
    """(prepared short-row part, LongRowLayout) for a skewed matrix whose long rows hold a large share of the
    entries, else None."""
    from . import longrows

    nnz = data.numel()
    threshold = longrows.long_row_threshold()
    lens, candidates, cand_nnz = longrows.split_rows(kernel_indptr, n_rows, threshold or longrows.MIN_CANDIDATE_LEN)
    enough = lambda k: k >= longrows.MIN_LONG_NNZ and k >= longrows.MIN_LONG_SHARE * nnz  # noqa: E731
    if not enough(cand_nnz) or cand_nnz > longrows.MAX_CANDIDATE_NNZ:
        return None
    built = longrows.build_long_row_layout(data, kernel_indices, kernel_indptr, lens, candidates, n_cols,
                                           min_unit_entries=0 if threshold else longrows.MIN_UNIT_ENTRIES)
    if built is None or not enough(built[0].nnz):
        return None
    layout, is_long = built
    d_s, i_s, p_s = longrows.short_part(data, kernel_indices, kernel_indptr, lens, is_long)
    short = _prepare_spmv_csr(d_s, i_s, p_s, shape, block_nnz, max_segments, reuse_expected=True, allow_split=False)
    return short, layout


def _prepare_spmv_csr(data, indices, indptr, shape, block_nnz, max_segments, reuse_expected, allow_split=True,
                      known=None, stats=None):
    """known: the statistics of arrays that were made here (contiguous, 32-bit column ids): nothing is left to check.
    reuse_expected=False (a one-shot product) skips the panel regrouping, which costs about as much as a
    hundred products and only pays when the prepared matrix is used again."""
    if known is None:
        data, kernel_indices, kernel_indptr, n_rows, n_cols, stats = _prepare_spmv_csr_matrix(
            data, indices, indptr, shape, narrow=reuse_expected, stats=stats
        )
    else:
        kernel_indices, kernel_indptr, (n_rows, n_cols), stats = indices, indptr, shape, known
    max_row_nnz = stats.max_row_nnz
    block_nnz_use, max_segments_use = _resolve_block_nnz(max_row_nnz, block_nnz, max_segments)
    nnz = data.numel()
    if data.dtype in widetypes.WIDE_DTYPES:
        # float16 / bfloat16 / complex values are read as they are stored by kernels of their own (fsb_spmv_csr_stored):
        # no second copy of the matrix, and a tile plan where the row lengths call for one
        tile_nnz, tile_row = 0, None
        if nnz > 0 and n_rows > 0 and _uneven_rows(n_rows, nnz, max_row_nnz, data.element_size()):
            tile_nnz = int(_lib.lib().fsb_spmv_stored_tile_nnz(_WIDE_VTYPE[data.dtype]))
            tile_row = _tile_plan(kernel_indptr, n_rows, nnz, tile_nnz)
        return PreparedCsrSpmv(
            data=data, kernel_indices=kernel_indices, kernel_indptr=kernel_indptr, shape=shape, n_rows=n_rows,
            n_cols=n_cols, block_nnz=block_nnz_use, max_segments=max_segments_use, max_row_nnz=max_row_nnz,
            stats=stats, algo=_lib.FSB_SPMV_VECTOR if tile_row is None else _lib.FSB_SPMV_STREAM, tuning=0,
            tile_nnz=tile_nnz, tile_row=tile_row, scratch=None, wide=("native", []),
        )
    algo = _select_spmv_algo(n_rows, nnz, max_row_nnz, data.element_size())
    tuning = int(os.environ.get("FSB_SPMV_TUNING", "0"))
    tile_nnz, tile_row, scratch, panel_layout = 0, None, None, None
    # rows of about equal length whose columns stay within a few chunks: regroup once, keep x in shared memory
    want_panel = algo == _lib.FSB_SPMV_PANEL or (
        reuse_expected and algo == _lib.FSB_SPMV_VECTOR and os.environ.get("FSB_SPMV_ALGO", "") == ""
        and _PANEL_ENABLED)
    if want_panel:
        from . import panel

        panel_layout = panel.build_panel_layout(data, kernel_indices, kernel_indptr, n_rows, n_cols, max_row_nnz,
                                                force=algo == _lib.FSB_SPMV_PANEL)
        algo = _lib.FSB_SPMV_PANEL if panel_layout is not None else _lib.FSB_SPMV_VECTOR
    automatic = reuse_expected and os.environ.get("FSB_SPMV_ALGO", "") == ""
    # skewed rows: the long ones leave for the row-group panel kernel, the short ones are a matrix of their own
    long_rows = bins_layout = None
    if algo == _lib.FSB_SPMV_STREAM and allow_split and automatic and _long_rows_enabled():
        long_rows = _split_long_rows(data, kernel_indices, kernel_indptr, n_rows, n_cols, shape, block_nnz,
                                     max_segments)
    # columns all over a long x: two streaming passes instead of a gather per entry
    if algo in (_lib.FSB_SPMV_VECTOR, _lib.FSB_SPMV_STREAM) and long_rows is None and automatic:
        from . import bins

        bins_layout = bins.bins_for(data, kernel_indices, kernel_indptr, n_rows, n_cols, max_row_nnz,
                                    algo == _lib.FSB_SPMV_VECTOR)
    # (with the two-pass form, too: a product that cannot have the memory between the passes takes one)
    if algo == _lib.FSB_SPMV_STREAM and nnz > 0 and n_rows > 0:
        L = _lib.lib()
        vt = _VTYPE[data.dtype]
        tile_nnz = int(L.fsb_spmv_tile_nnz(vt, tuning))
        tile_row = _tile_plan(kernel_indptr, n_rows, nnz, tile_nnz)
        scratch = torch.empty(int(L.fsb_spmv_csr_scratch_bytes(vt, nnz, tuning)), dtype=torch.uint8,
                              device=data.device)
    return PreparedCsrSpmv(
        data=data, kernel_indices=kernel_indices, kernel_indptr=kernel_indptr, shape=shape, n_rows=n_rows,
        n_cols=n_cols, block_nnz=block_nnz_use, max_segments=max_segments_use, max_row_nnz=max_row_nnz,
        stats=stats, algo=algo, tuning=tuning, tile_nnz=tile_nnz, tile_row=tile_row, scratch=scratch,
        panel=panel_layout, long_rows=long_rows, bins=bins_layout,
    )


def _spmv_launch(prepared, x, y):
    """Enqueue y = A x on the current stream of the matrix's device.  Stands in for both of the
    reference's launch helpers (_triton_spmv_csr_impl_opt_prepared :329-376 and
    _triton_spmv_csr_impl_prepared :510-554): float32 and float64 accumulate natively either way."""
    L = _lib.lib()
    p = prepared
    dev = p.data.device
    if p.algo == _lib.FSB_SPMV_PANEL and p.panel is not None:
        from . import panel

        with _on_device(dev):
            panel.launch_panel(p.panel, x, y, p.n_rows, p.n_cols, _stream_ptr(dev))
        return
    if p.long_rows is not None:
        from . import longrows

        short, layout = p.long_rows
        _spmv_launch(short, x, y)      # every row of y; the long rows get zeros here
        with _on_device(dev):
            longrows.launch_long_rows(layout, x, y, p.n_cols, _stream_ptr(dev))
        return
    if p.bins is not None:
        from . import bins

        with _on_device(dev):
            done = bins.launch_bins(p.bins, x, y, p.n_rows, p.n_cols, _stream_ptr(dev), data=p.data)
        if done:
            return
    algo = p.algo if p.tile_row is not None else _lib.FSB_SPMV_VECTOR
    # calls on a small matrix may overlap in several streams, whichever kernel its rows get: scratch of the call's own
    scratch = p.scratch
    if scratch is not None and (p.data.numel() < _STREAM_MIN_NNZ or p.bins is not None):
        scratch = torch.empty_like(scratch)
    lanes = p.tuning & 0xFF
    tuning = p.tuning if algo == _lib.FSB_SPMV_STREAM else (lanes if lanes in (2, 4, 8, 16, 32) else p.vector_tuning)
    with _on_device(dev):
        rc = L.fsb_spmv_csr(
            _VTYPE[p.data.dtype], _ITYPE[p.kernel_indices.dtype], _ITYPE[p.kernel_indptr.dtype],
            _ptr(p.data), _ptr(p.kernel_indices), p.kernel_indptr.data_ptr(), _ptr(x), _ptr(y),
            p.n_rows, p.n_cols, p.data.numel(), algo, tuning,
            None if p.tile_row is None else p.tile_row.data_ptr(),
            None if scratch is None else scratch.data_ptr(),
            0 if scratch is None else scratch.numel(), _stream_ptr(dev),
        )
    _lib.check(rc, "fsb_spmv_csr")


def _spmv_launch_stored(prepared, x, y):
    """Enqueue y = A x for float16 / bfloat16 / complex values with x and y in the matrix's own type.  Stands in for the
    reference's base launch on these types (spmv_csr.py:510-554)."""
    p = prepared
    dev = p.data.device
    if p.n_rows == 0:
        return
    L = _lib.lib()
    scratch = None
    if p.tile_row is not None:       # the call's own: calls on one matrix may overlap in several streams
        scratch = torch.empty(int(L.fsb_spmv_stored_scratch_bytes(_WIDE_VTYPE[p.data.dtype], p.data.numel())),
                              dtype=torch.uint8, device=dev)
    with _on_device(dev):
        args = (_WIDE_VTYPE[p.data.dtype], _ITYPE[p.kernel_indptr.dtype], _ptr(p.data), _ptr(p.kernel_indices),
                p.kernel_indptr.data_ptr(), _ptr(x), _ptr(y), p.n_rows, p.n_cols, p.data.numel())
        if p.tile_row is None and not p.uneven:
            rc = L.fsb_spmv_csr_stored_even(*args, _stream_ptr(dev))
        else:
            rc = L.fsb_spmv_csr_stored(*args, None if p.tile_row is None else p.tile_row.data_ptr(), _ptr(scratch),
                                       0 if scratch is None else scratch.numel(), _stream_ptr(dev))
    _lib.check(rc, "fsb_spmv_csr_stored")


def _spmv_once(data, indices, indptr, x, shape, out):
    """(y, stats): the product straight from the arrays, where every argument is as the kernels read it, by one call that checks the
    arrays, waits for the answer and enqueues the kernel for even rows.  y is None where that was not done: the arguments are for
    the general path, which also finds the words for what is wrong with them (stats None: nothing was looked at)."""
    none = None, None
    if not (isinstance(data, torch.Tensor) and isinstance(indices, torch.Tensor) and isinstance(indptr, torch.Tensor)
            and isinstance(x, torch.Tensor)):
        return none
    dev, dtype = data.device, data.dtype
    if dev.type != "cuda" or indices.device != dev or indptr.device != dev or x.device != dev or x.dtype != dtype:
        return none
    vt, it, pt = _VTYPE.get(dtype), _ITYPE.get(indices.dtype), _ITYPE.get(indptr.dtype)
    stored = vt is None
    if stored:
        vt = _WIDE_VTYPE.get(dtype)
        if out is not None or it != _lib.FSB_I32:
            return none
    elif "FSB_SPMV_ALGO" in os.environ or "FSB_SPMV_TUNING" in os.environ:
        return none
    if vt is None or it is None or pt is None or data.ndim != 1 or indices.ndim != 1 or indptr.ndim != 1 or x.ndim != 1:
        return none
    n_rows, n_cols, nnz = int(shape[0]), int(shape[1]), data.numel()
    if not (0 < nnz == indices.numel() and 0 < n_rows == indptr.numel() - 1 and x.numel() == n_cols < _INDEX_LIMIT_INT32):
        return none
    if not (data.is_contiguous() and indices.is_contiguous() and indptr.is_contiguous() and x.is_contiguous()):
        return none
    if data.is_neg() or x.is_neg() or data.is_conj() or x.is_conj():
        return none
    if out is not None and not (out.device == dev and out.shape == (n_rows,) and out.dtype == dtype and out.is_contiguous()
                                and not out.is_neg()):
        return none
    L = _lib.lib()
    with _on_device(dev):
        slot = _check_slot(dev)
        if slot is None:
            return none
        y = out if out is not None else torch.empty(n_rows, dtype=dtype, device=dev)
        longest = (_longest_even_stored if stored else _longest_even)(n_rows, nnz, data.element_size())
        rc = L.fsb_spmv_csr_once(vt, it, pt, data.data_ptr(), indices.data_ptr(), indptr.data_ptr(), x.data_ptr(), y.data_ptr(),
                                 n_rows, n_cols, nnz, longest, _longest_neighbour(n_rows, nnz, data.element_size()),
                                 slot.work_ptr, slot.host_ptr, _stream_ptr(dev))
    if rc == _lib.FSB_OK:
        return y, None
    if rc == _lib.FSB_NOT_LAUNCHED:
        return None, slot.stats()
    if rc != _lib.FSB_CAPTURING:
        _lib.check(rc, "fsb_spmv_csr_once")
    return none


def flagsparse_spmv_csr(data=None, indices=None, indptr=None, x=None, shape=None, block_nnz=256,
                        max_segments=None, out=None, return_time=False, use_opt=False, prepared=None):
    """CSR SpMV: y = A @ x (reference: spmv_csr.py:557-610, same arguments and defaults).

    data, indices, indptr: CSR arrays; x: dense vector; shape: (n_rows, n_cols).
    prepared: result of prepare_spmv_csr for steady-state calls.  block_nnz, max_segments and use_opt
    select Triton launch shapes in the reference; here they are validated bookkeeping only -- both
    settings of use_opt run the same CUDA kernels.  Returns a new tensor, or `out` when it is given.
    """
    if prepared is None:
        if any(arg is None for arg in (data, indices, indptr, shape)):
            raise ValueError("data, indices, indptr, and shape are required when prepared is not provided")
        stats = None
        if not return_time and block_nnz == 256 and max_segments is None:
            y, stats = _spmv_once(data, indices, indptr, x, shape, out)
            if y is not None:
                return y
        prepared = _prepare_spmv_csr(data, indices, indptr, shape, block_nnz, max_segments, reuse_expected=False, stats=stats)
    x = _validate_spmv_x(x, prepared)
    dev = prepared.data.device
    dtype = prepared.data.dtype
    if out is not None and (out.shape != (prepared.n_rows,) or out.dtype != dtype):
        raise ValueError("out shape/dtype must match result")
    if prepared.wide is not None:
        t0 = None
        if return_time:
            torch.cuda.synchronize(dev)
            t0 = time.perf_counter()
        y = torch.empty(prepared.n_rows, dtype=dtype, device=dev)   # not `out`, which may be x itself
        _spmv_launch_stored(prepared, x, y)
        elapsed_ms = None
        if return_time:
            torch.cuda.synchronize(dev)
            elapsed_ms = (time.perf_counter() - t0) * 1000.0
        if out is not None:
            out.copy_(y)
            y = out
        return (y, elapsed_ms) if return_time else y
    # write straight into `out` when that is safe, else into a fresh vector that is copied over
    direct = out is not None and out.is_cuda and out.device == dev and out.is_contiguous() and not out.is_neg()
    y = out if direct else torch.empty(prepared.n_rows, dtype=dtype, device=dev)
    t0 = None
    if return_time:
        torch.cuda.synchronize(dev)
        t0 = time.perf_counter()
    _spmv_launch(prepared, x, y)
    elapsed_ms = None
    if return_time:
        torch.cuda.synchronize(dev)
        elapsed_ms = (time.perf_counter() - t0) * 1000.0
        prepared.check_status()
    if out is not None and not direct:
        out.copy_(y)
        y = out
    if return_time:
        return y, elapsed_ms
    return y


# ---------------------------------------------------------------------------------------------------
# COO front-end: convert to CSR, then the same kernels (reference: spmv_csr.py:613-758)
# ---------------------------------------------------------------------------------------------------
def coo_to_csr_for_spmv(data, row, col, shape, assume_sorted=False):
    """COO triple -> (values, int32 column indices, int64 row pointer) with the entries in (row, column) order,
    which is what the reference's function of this name returns (spmv_csr.py:623-647).  Entries already in order
    (or declared so) are not touched; otherwise one sort on the combined key.  The row pointer is read off
    the ordered row ids by binary search."""
    n_rows, n_cols = int(shape[0]), int(shape[1])
    dev = data.device
    rows, cols = row.to(torch.int64), col.to(torch.int64)
    if rows.numel() == 0:
        return data, cols.to(torch.int32), torch.zeros(n_rows + 1, dtype=torch.int64, device=dev)
    if not assume_sorted and rows.numel() > 1:
        key = rows * max(1, n_cols) + cols
        if bool((key[1:] < key[:-1]).any()):
            order = torch.argsort(key)     # entries with one (row, column) keep the order torch's default sort gives
            rows, cols, data = rows[order], cols[order], data[order]
        del key
    indptr = torch.searchsorted(rows.contiguous(), torch.arange(n_rows + 1, dtype=torch.int64, device=dev))
    return data, cols.to(torch.int32), indptr


def _check_coo_triple(data, row, col, extra=()):
    names = "data, row, col" + (", x" if extra else "")
    tensors = (data, row, col) + tuple(extra)
    if not all(torch.is_tensor(t) for t in tensors):
        raise TypeError(f"{names} must all be torch.Tensor")
    if not all(t.is_cuda for t in tensors):
        raise ValueError(f"{names} must all be CUDA tensors")
    if any(t.ndim != 1 for t in tensors):
        raise ValueError(f"{names} must all be 1D tensors")


def prepare_spmv_coo_tocsr(data, row, col, shape, block_nnz=256, max_segments=None, assume_sorted=False):
    """One-time COO -> CSR + analysis; use with flagsparse_spmv_coo_tocsr(..., prepared=p)
    (reference :650-684)."""
    _check_coo_triple(data, row, col)
    _check_value_dtype(data.dtype)
    if row.numel() != col.numel() or data.numel() != row.numel():
        raise ValueError("data, row, col must have the same length")
    data_s, indices, indptr = coo_to_csr_for_spmv(data, row, col, shape, assume_sorted=assume_sorted)
    return prepare_spmv_csr(data_s, indices, indptr, shape, block_nnz=block_nnz, max_segments=max_segments)


def flagsparse_spmv_coo_tocsr(data=None, row=None, col=None, x=None, shape=None, block_nnz=256,
                              max_segments=None, out=None, return_time=False, use_opt=True, prepared=None,
                              assume_sorted=False):
    """COO SpMV via CSR conversion: y = A @ x (reference :687-758, same arguments and defaults)."""
    if prepared is not None:
        if x is None:
            raise TypeError("x is required")
        if shape is None:
            shape = prepared.shape
        sh = (int(shape[0]), int(shape[1]))
        if sh != prepared.shape:
            raise ValueError(f"shape {sh} does not match prepared.shape {prepared.shape}")
        return flagsparse_spmv_csr(x=x, shape=shape, block_nnz=block_nnz, max_segments=max_segments, out=out,
                                   return_time=return_time, use_opt=use_opt, prepared=prepared)
    _check_coo_triple(data, row, col, extra=(x,))
    _check_value_dtype(data.dtype)
    if x.dtype != data.dtype:
        raise TypeError("x dtype must match data dtype")
    data_s, indices, indptr = coo_to_csr_for_spmv(data, row, col, shape, assume_sorted=assume_sorted)
    return flagsparse_spmv_csr(data_s, indices, indptr, x, shape, block_nnz=block_nnz,
                               max_segments=max_segments, out=out, return_time=return_time, use_opt=use_opt)
