"""Prepare-time regrouping of a CSR matrix for the two-pass SpMV (csrc/spmv_bins.cu): for matrices whose columns lie all
over a long x and whose rows have nothing to share in a chunk of it.

The reference's prepare step builds row-length buckets (src/flagsparse/sparse_operations/spmv_csr.py:281-327); this one
stores the columns a second time, by (chunk of columns, block of rows), so that the product reads x from shared memory and
everything else in order; the values are read where the caller has them.  One count and one placing kernel, a cumulative sum
over the units between them.
"""

import os

import torch

from . import _lib
from ._common import _ITYPE, _VTYPE

# Where the two passes win, each line with both sides measured (us, one pass against two; columns anywhere unless said).
# Rows of about equal length against the lanes-per-row kernel, float32: 2^27 entries in 33.6 M / 16.8 M / 4.2 M rows: 1326 / 624 /
# 549 against 606 / 530 / 473; 2^24 entries in 4.2 M / 1 M / 0.5 M rows: 92 / 75 / 75 against 75 / 67 / 65; 2^23 entries in 2.1 M /
# 0.5 M rows: 45 / 35 against 43 / 40.
EVEN_MIN_NNZ = 1 << 24
EVEN_MIN_SPAN = 2 << 20
# Uneven rows (the short rows of a skewed matrix, mostly), float32: 107 M entries 1081 against 439; 10.4 M in 2.1 M rows 90 against
# 47; 3.1 M in 0.5 M rows 24.1 against 22.3; 2.7 M in 0.3 M rows 22.0 against 19.8; 2.6 M in 0.25 M rows 20.6 against 20.0.
UNEVEN_MIN_NNZ = 5 << 19
UNEVEN_MIN_SPAN = 1 << 20
# float64 moves 29 bytes an entry instead of 12, so it takes an x that L2 does not hold: 2^27 entries in 33.6 M / 16.8 M / 8.4 M
# rows: 2154 / 1334 / 709 against 1420 / 1135 / 994; uneven, 2^26 entries in 16.8 M / 8.4 M rows: 780 / 465 against 630 / 530.
F64_MIN_SPAN = 120 << 20
# ... or uneven rows of a few entries that would have gone to the lanes-per-row kernel, whose warps wait for their longest row:
# 4.8 M entries in 2.1 M rows 66 against 48, 3.3 M in 1 M rows 41 against 34; by tiles, 2.6 M in 0.5 M rows 23.3 against 29.8.
F64_SHORT_MEAN = 4
# Rows of a block, at most (see cuts): one CTA writes them, and rows without entries count for nothing in the cut by entries.
# float32, one pass against two with no such line / with it: 2^24 rows, 4 entries in every row of the first half 272 against 1499 /
# 175 us; 16 in every one of the last 2^20 rows 207 against 2519 / 119; 10 M entries in the first 2 M of 30 M rows 323 against 4578 /
# 126; with 2^14 / 2^18 instead: 177 / 204, 120 / 121, 128 / 143.  Blocks of fewer rows stay whole: cut at every 2^16th row of the
# matrix, 107 M entries of short rows took 452 instead of 439 us, 27 M in 67 M rows 324 instead of 283.
BLOCK_ROWS = 1 << 16
# Mean entries of a unit below which the packs would mostly be padding; near the line, one pass against two: float32 with 17 entries
# (2^25 in all, 70 M columns) 519 against 218 us, float64 with 8.4 (2^27, 36 M columns) 2177 against 1448.
MIN_UNIT = {4: 16, 8: 8}


def _enabled():
    """FSB_SPMV_BINS=0 keeps the one-pass kernels."""
    return os.environ.get("FSB_SPMV_BINS", "1") != "0"


def min_span(nnz, n_rows, max_row_nnz, element_size, lanes_per_row):
    """Bytes of x that a row block has to reach for the two passes to pay, or None where they never do.  lanes_per_row: the
    matrix would otherwise go to the lanes-per-row kernel."""
    mean = nnz / max(n_rows, 1)
    uneven = max_row_nnz > 2 * mean + 16
    if element_size == 4:
        if nnz >= EVEN_MIN_NNZ and not uneven:
            return EVEN_MIN_SPAN
        return UNEVEN_MIN_SPAN if uneven and nnz >= UNEVEN_MIN_NNZ else None
    if uneven and lanes_per_row and mean <= F64_SHORT_MEAN and nnz >= UNEVEN_MIN_NNZ:
        return UNEVEN_MIN_SPAN
    return F64_MIN_SPAN if nnz >= EVEN_MIN_NNZ else None


def cuts(nnz, n_rows, max_row_nnz, cap):
    """(entries, rows) from one cut of the row blocks to the next: the row in which a cut by entries falls goes to the block
    before it; rows as BLOCK_ROWS says, or twice what a block of a matrix of almost empty rows has on average."""
    step = cap - max_row_nnz + 1
    return step, max(BLOCK_ROWS, 2 * -(-n_rows // max(1024, -(-nnz // step))))


class BinsLayout:
    """Device arrays of the regrouped matrix (include/fsb.h, fsb_spmv_csr_bins)."""

    __slots__ = ("data", "col", "place", "dst", "ends", "chunk_pack", "block_pack", "block_start", "row_slot", "n_blocks",
                 "n_chunks", "chunk_cols", "n_packs")

    def nbytes(self):
        return sum(t.numel() * t.element_size() for t in (self.col, self.place, self.dst, self.ends, self.row_slot,
                                                          self.chunk_pack, self.block_pack, self.block_start))


def _cut_rows(begin, n_rows, most):
    """First rows of the blocks, and n_rows, as int32: those that begin at the rows `begin` (the first at row 0 whatever it
    says), each cut into parts of about as many rows and `most` at most, and nothing for the empty ones."""
    begin = torch.cat((begin.new_zeros(1), begin[1:].clamp(max=n_rows), begin.new_full((1,), n_rows)))
    lens = begin[1:] - begin[:-1]
    parts = (lens + (most - 1)) // most
    block = torch.repeat_interleave(torch.arange(parts.numel(), device=begin.device), parts)      # a sync
    part = torch.arange(block.numel(), device=begin.device) - (torch.cumsum(parts, 0) - parts)[block]
    rows = begin[block] + lens[block] * part // parts[block]
    return torch.cat((rows, begin[-1:])).to(torch.int32)


def _starts(packs):
    """First pack of every unit (and the total) in the order of `packs`, as int32; the total again as a number (a sync)."""
    ends = torch.cumsum(packs.reshape(-1), 0, dtype=torch.int64)
    n = int(ends[-1])
    out = torch.zeros(ends.numel() + 1, dtype=torch.int32, device=packs.device)
    out[1:] = ends
    return out, n


def build_bins_layout(data, indices, indptr, n_rows, n_cols, max_row_nnz, span=0, chunk_cols=None):
    """BinsLayout for float32 / float64 values on the GPU (int32 indices, at least one entry), or None when a row is too long
    for a block, there are too many chunks or entries, or the row blocks reach less than `span` bytes of x on average (whole
    chunks counted: then the gathers of a one-pass kernel are served close to the SM)."""
    L = _lib.lib()
    dev, nnz = data.device, data.numel()
    vt, pt = _VTYPE[data.dtype], _ITYPE[indptr.dtype]
    cap, pack, n_ends = (int(v) for v in (L.fsb_spmv_bins_cap(vt), L.fsb_spmv_bins_pack(vt), L.fsb_spmv_bins_ends()))
    chunk_cols = chunk_cols or int(L.fsb_spmv_bins_chunk_cols(vt))
    n_chunks = -(-n_cols // chunk_cols)
    if max_row_nnz > cap // 4 or n_chunks > int(L.fsb_spmv_bins_max_chunks()) or n_cols * data.element_size() < span:
        return None
    # a block begins at the first row that starts at or behind entry k * step: at most step - 1 + max_row_nnz entries; one of
    # more than `rows` rows is cut into parts of as many rows each
    step, rows = cuts(nnz, n_rows, max_row_nnz, cap)
    n_blocks = -(-nnz // step) + -(-n_rows // rows)            # at most
    if nnz // pack + n_blocks * n_chunks >= 2**31 - 1 or (indptr.dtype == torch.int32 and nnz >= 2**31 - 1 - cap):
        return None
    st = torch.cuda.current_stream(dev).cuda_stream
    with torch.cuda.device(dev):
        block_row = _cut_rows(torch.searchsorted(indptr, torch.arange(-(-nnz // step), device=dev, dtype=indptr.dtype) * step),
                              n_rows, rows)
        n_blocks = block_row.numel() - 1
        counts = torch.empty((n_blocks, n_chunks), dtype=torch.int32, device=dev)
        _lib.check(L.fsb_spmv_bins_count(pt, indices.data_ptr(), indptr.data_ptr(), block_row.data_ptr(), n_blocks, n_chunks,
                                         chunk_cols, n_cols, counts.data_ptr(), st), "fsb_spmv_bins_count")
        start = indptr[block_row.long()].to(torch.int64)
        if span:
            units, blocks = torch.stack((torch.count_nonzero(counts), torch.count_nonzero(start[1:] > start[:-1]))).tolist()  # a sync
            if units * chunk_cols * data.element_size() < span * blocks:       # (blocks of empty rows reach nothing)
                return None
        packs = (counts + (pack - 1)) // pack
        del counts
        unit_block, n_packs = _starts(packs)
        by_chunk, _ = _starts(packs.t())
        del packs
        chunk_pack = by_chunk[::n_blocks].contiguous()
        block_pack = unit_block[::n_chunks].contiguous()
        unit_chunk = by_chunk[:-1].view(n_chunks, n_blocks).t().contiguous()
        del by_chunk
        lay = BinsLayout()
        lay.data = data                       # the caller's own: the product reads the values there
        lay.col = torch.empty(pack * n_packs, dtype=torch.int16, device=dev)
        lay.place = torch.empty(n_packs, dtype=torch.int32, device=dev)
        lay.dst = torch.empty(pack * n_packs, dtype=torch.int16, device=dev)
        lay.ends = torch.empty(n_ends * n_blocks, dtype=torch.int32, device=dev)
        lay.row_slot = torch.empty(n_rows, dtype=torch.int16, device=dev)
        _lib.check(L.fsb_spmv_bins_place(vt, pt, indices.data_ptr(), indptr.data_ptr(), block_row.data_ptr(),
                                         n_blocks, n_chunks, chunk_cols, n_cols, unit_chunk.data_ptr(), unit_block.data_ptr(),
                                         lay.col.data_ptr(), lay.place.data_ptr(), lay.dst.data_ptr(),
                                         lay.ends.data_ptr(), lay.row_slot.data_ptr(), st), "fsb_spmv_bins_place")
        lay.block_start = torch.stack((block_row.to(torch.int64), start), 1)
    lay.chunk_pack, lay.block_pack = chunk_pack, block_pack
    lay.n_blocks, lay.n_chunks, lay.chunk_cols, lay.n_packs = n_blocks, n_chunks, chunk_cols, n_packs
    return lay


def bins_for(data, indices, indptr, n_rows, n_cols, max_row_nnz, lanes_per_row):
    """BinsLayout for a matrix that is multiplied again and again, or None where one pass over its entries is the better way."""
    nnz, sv = data.numel(), data.element_size()
    if not _enabled() or not data.is_cuda or data.device.type != "cuda" or nnz == 0 or n_rows == 0:
        return None
    span = min_span(nnz, n_rows, max_row_nnz, sv, lanes_per_row)
    if span is None:
        return None
    L, vt = _lib.lib(), _VTYPE[data.dtype]
    if int(L.fsb_spmv_bins_cap(vt)) * int(L.fsb_spmv_bins_chunk_cols(vt)) < MIN_UNIT[sv] * n_cols:
        return None
    try:
        return build_bins_layout(data, indices, indptr, n_rows, n_cols, max_row_nnz, span)
    except torch.OutOfMemoryError:       # a one-pass kernel needs none of it
        return None


def _between_passes(layout, device):
    return torch.empty(32 * layout.n_packs, dtype=torch.uint8, device=device)


def launch_bins(layout, x, y, n_rows, n_cols, stream_ptr, data=None):
    """Enqueue the product on the current stream (its handle in stream_ptr).  data: the values, in CSR order, instead of those
    that the layout was made with.  The memory between the passes is the call's own: calls on one matrix may overlap in
    several streams.  False where it is refused: nothing was enqueued then."""
    la = layout
    data = la.data if data is None else data
    try:
        xg = _between_passes(la, data.device)
    except torch.OutOfMemoryError:
        return False
    rc = _lib.lib().fsb_spmv_csr_bins(
        _VTYPE[data.dtype], la.col.data_ptr(), la.place.data_ptr(), la.dst.data_ptr(), la.ends.data_ptr(),
        la.row_slot.data_ptr(), la.chunk_pack.data_ptr(), la.block_pack.data_ptr(), la.block_start.data_ptr(), data.data_ptr(),
        la.n_blocks, la.n_chunks, la.chunk_cols, la.n_packs, xg.data_ptr(), xg.numel(), x.data_ptr(), y.data_ptr(), n_rows,
        n_cols, stream_ptr,
    )
    _lib.check(rc, "fsb_spmv_csr_bins")
    return True
