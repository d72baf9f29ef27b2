"""Workloads of the sparse products, as a user's program runs them: the matrices, the calls, what a call has to move.

A case is a dict: which product ("op"), the matrix (rows, cols, mean entries per row, how the row lengths and columns
are distributed) and its types.  Products:

  spmv        y = A x on a matrix prepared once (iterative solvers, PageRank: the same matrix, many vectors)
  spmv_once   y = A x straight from the CSR arrays (the matrix changes from call to call; checks included)
  spmm        C = A B on a matrix prepared once
  spmm_once   C = A B straight from the CSR arrays
  spmv_coo    y = A x on a COO matrix prepared once
  spmv_coo_once, spmm_coo   straight from the COO triples (edge lists), sorted by row or in any order
  sddmm       dot products of rows of X and Y on a prepared CSR pattern (attention scores of a graph, the gradient of
              an SpMM with respect to the matrix)

Row laws: "exact" (mean entries in every row), "poisson" (mesh and finite-element matrices have rows of about equal
length), "skewed" (Zipf lengths, exponent 2: web and social graphs).  Columns are distinct and sorted inside a row,
uniform over a band of +-band columns around the diagonal, or over all columns where band is 0.  Values, vectors and
dense matrices are uniform in [-1, 1].
"""

import math

import torch

import flagsparse_b200 as fs

_DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32, "f64": torch.float64,
           "c64": torch.complex64, "c128": torch.complex128}
_SIZE = {"f16": 2, "bf16": 2, "f32": 4, "f64": 8, "c64": 8, "c128": 16}
_INDEX = {"i32": torch.int32, "i64": torch.int64}
_TOLERANCE = {"f16": 2e-3, "bf16": 1e-2, "f32": 1e-5, "f64": 1e-13, "c64": 1e-5, "c128": 1e-13}
_LONGEST = 1 << 17


def _case(name, op, dtype, index, law, rows, mean, band=0, cols=0, dense=0, ordered=True, scaled=False):
    c = {"op": op, "dtype": dtype, "index": index, "law": law, "rows": rows, "cols": cols or rows, "mean": mean,
         "band": band, "dense": dense, "ordered": ordered, "scaled": scaled}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small system inside a solver: the time of a call is the time to launch it
        _case("spmv_small", "spmv", "f32", "i32", "exact", 4096, 16),
        # an ordinary finite-element matrix in double precision; the torch default of 64-bit indices; a ragged size
        _case("spmv_mesh_f64", "spmv", "f64", "i64", "poisson", 300007, 27, band=1 << 13),
        # a large banded matrix: the entries stream from memory, the vector stays on the chip
        _case("spmv_banded", "spmv", "f32", "i32", "poisson", 1 << 22, 32, band=1 << 16),
        # a web-like graph: row lengths from 1 to 2^17, columns anywhere
        _case("spmv_graph", "spmv", "f32", "i32", "skewed", 1 << 24, 15),
        # the largest: a wide band, the vector larger than what the caches hold close to a row
        _case("spmv_wide_band", "spmv", "f32", "i32", "poisson", 1 << 24, 32, band=1 << 20),
        # complex amplitudes (wave problems), an operator of ordinary size
        _case("spmv_complex", "spmv", "c64", "i32", "poisson", 500009, 24, band=1 << 14),
        # a matrix that is used once: the checks of the arrays belong to the call
        _case("spmv_once", "spmv_once", "f32", "i64", "poisson", 250007, 12, band=1 << 12),
        # features of a graph multiplied over and over: uniform neighbours, 64 features
        _case("spmm_features", "spmm", "f32", "i32", "exact", 1 << 20, 16, dense=64),
        # a small graph, one product per sampled batch
        _case("spmm_batch", "spmm_once", "f32", "i32", "poisson", 4096, 16, dense=32),
        # half-precision features of a skewed graph
        _case("spmm_half", "spmm_once", "bf16", "i32", "skewed", 200003, 20, dense=128),
        # an edge list in no particular order, an odd number of features
        _case("spmm_edges", "spmm_coo", "f32", "i64", "skewed", 150001, 14, dense=33, ordered=False),
        # edge scores of a graph
        _case("sddmm_edges", "sddmm", "f32", "i32", "poisson", 1 << 19, 16, dense=64),
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng):
    op = rng.choice(["spmv"] * 5 + ["spmv_once"] * 2 + ["spmm"] * 3 + ["spmm_once"] * 2 + ["sddmm"] * 2
                    + ["spmv_coo", "spmv_coo_once", "spmm_coo"])
    narrow = ["f32", "f32", "f64"]                       # what most callers have, and what every product takes
    every = narrow * 2 + ["f16", "bf16", "c64", "c128"]
    dtype = rng.choice(every if op in ("spmv", "spmv_once", "spmm_once") else narrow)
    index = "i32" if op == "sddmm" else rng.choice(["i32", "i64"])
    most = {"spmv": 1 << 27, "spmv_coo": 1 << 22, "spmv_coo_once": 1 << 21, "spmm_coo": 1 << 21,
            "spmv_once": 1 << 24}.get(op, 1 << 24)
    dense = 0
    if op in ("spmm", "spmm_once", "spmm_coo", "sddmm"):
        dense = rng.choice([16, 32, 64, 128]) if rng.random() < 0.5 else _log_uniform(rng, 4, 200)
        most = min(most, (1 << 29) // (dense * max(1, _SIZE[dtype] // 4)))
    mean = _log_uniform(rng, 4, 64)
    nnz = _log_uniform(rng, 1 << 15, most)
    rows = max(512, nnz // mean)
    law = rng.choice(["exact", "poisson", "poisson", "skewed"])
    band, cols = 0, rows
    if law == "poisson" and rng.random() < 0.7:
        band = max(128, _log_uniform(rng, rows // 4096 + 128, rows // 3 + 256))
    elif rng.random() < 0.3:
        cols = max(512, int(rows * rng.uniform(0.3, 2.0)))
    return _case(None, op, dtype, index, law, rows, mean, band, cols, dense, ordered=rng.random() < 0.5,
                 scaled=op == "sddmm" and rng.random() < 0.5)


# ---- inputs -----------------------------------------------------------------------------------------------------
def _row_lengths(case, width, gen):
    n, mean, dev = case["rows"], case["mean"], "cuda"
    longest = max(1, width)
    if case["law"] == "exact":
        return torch.full((n,), min(mean, longest), dtype=torch.int64, device=dev)
    # the same lengths for every seed, in another order: evenly spread quantiles of the law
    u = (torch.randperm(n, device=dev, generator=gen).to(torch.float64) + 0.5) / n
    if case["law"] == "poisson":
        k = torch.arange(mean + 16 * math.isqrt(mean) + 32, dtype=torch.float64, device=dev)
        cdf = torch.cumsum(torch.exp(k * math.log(mean) - mean - torch.lgamma(k + 1)), 0)
        return torch.searchsorted(cdf, u).clamp_(max=longest)
    # Zipf with exponent 2, clipped: length = s / u, s from the wanted mean
    longest = max(4, min(_LONGEST, width // 4))
    s = 1.0
    for _ in range(60):
        s = mean / (1.0 + math.log(max(1.01, longest / s)))
    return torch.round(s / u).to(torch.int64).clamp_(min=1, max=longest)


def _csr(case, gen):
    """(row of every entry, column of every entry, row pointer), 64-bit."""
    n, m, dev = case["rows"], case["cols"], "cuda"
    width = min(m, 2 * case["band"] + 1) if case["band"] else m
    lens = _row_lengths(case, width, gen)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    torch.cumsum(lens, 0, out=ptr[1:])
    nnz = int(ptr[-1])
    every_row = torch.arange(n, device=dev)
    row = torch.repeat_interleave(every_row, lens, output_size=nnz)
    # sorted uniform positions without a sort: running sums of exponential gaps, scaled to the row (whole numbers, so
    # that the sums are the same whatever order they are made in)
    gaps = torch.empty(nnz + n, dtype=torch.float32, device=dev).exponential_(generator=gen).mul_(1 << 20)
    sums = torch.cumsum(gaps.to(torch.int64).add_(1), 0)
    del gaps
    end = sums[ptr[1:] + every_row]
    start = torch.cat([end.new_zeros(1), end[:-1]])
    place = torch.arange(nnz, device=dev)
    pos = sums[place + row]
    del sums
    pos -= start[row]
    pos = pos.to(torch.float64)
    pos /= (end - start)[row]
    free = width - lens                      # distinct columns: a sorted draw from the free places, plus the rank
    pos *= (free + 1)[row]
    col = torch.minimum(pos.to(torch.int64), free[row])
    del pos
    col += place
    del place
    low = (every_row - case["band"]).clamp_(0, m - width) if case["band"] else torch.zeros_like(every_row)
    col += (low - ptr[:-1])[row]
    return row, col, ptr


def _uniform(shape, dtype, gen):
    if dtype.is_complex:
        part = torch.float32 if dtype == torch.complex64 else torch.float64
        return torch.view_as_complex(_uniform(tuple(shape) + (2,), part, gen))
    wide = torch.float64 if dtype == torch.float64 else torch.float32
    return torch.empty(shape, dtype=wide, device="cuda").uniform_(-1, 1, generator=gen).to(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    op, dtype, index = case["op"], _DTYPES[case["dtype"]], _INDEX[case["index"]]
    shape = (case["rows"], case["cols"])
    row, col, ptr = _csr(case, gen)
    data = _uniform((col.numel(),), dtype, gen)
    state = {"op": op, "shape": shape}
    if op == "sddmm":
        state["prepared"] = fs.prepare_sddmm_csr(col.to(index), ptr.to(index), shape, k_hint=case["dense"])
        state["x"] = _uniform((case["rows"], case["dense"]), dtype, gen)
        state["y"] = _uniform((case["cols"], case["dense"]), dtype, gen)
        state["scale"] = {"data": data, "alpha": 0.5, "beta": 1.5} if case["scaled"] else {}
        return state
    state["dense"] = _uniform((case["cols"], case["dense"]) if case["dense"] else (case["cols"],), dtype, gen)
    if "coo" in op:
        if not case["ordered"]:
            order = torch.randperm(col.numel(), device="cuda", generator=gen)
            row, col, data = row[order], col[order], data[order]
        matrix = (data, row.to(index), col.to(index))
    else:
        del row
        matrix = (data, col.to(index), ptr.to(index))
        del col, ptr
    if op == "spmv":
        state["prepared"] = fs.prepare_spmv_csr(*matrix, shape)
    elif op == "spmm":
        state["prepared"] = fs.prepare_spmm_csr_opt(*matrix, shape)
    elif op == "spmv_coo":
        state["prepared"] = fs.prepare_spmv_coo(*matrix, shape)
    else:
        state["matrix"] = matrix
    return state


# ---- one call ---------------------------------------------------------------------------------------------------
def run(state):
    op, shape = state["op"], state["shape"]
    if op == "spmv":
        return fs.flagsparse_spmv_csr(x=state["dense"], prepared=state["prepared"])
    if op == "spmv_once":
        return fs.flagsparse_spmv_csr(*state["matrix"], state["dense"], shape)
    if op == "spmm":
        return fs.flagsparse_spmm_csr_opt(B=state["dense"], prepared=state["prepared"])
    if op == "spmm_once":
        return fs.flagsparse_spmm_csr(*state["matrix"], state["dense"], shape)
    if op == "spmv_coo":
        return fs.flagsparse_spmv_coo(x=state["dense"], prepared=state["prepared"])
    if op == "spmv_coo_once":
        return fs.flagsparse_spmv_coo(*state["matrix"], state["dense"], shape)
    if op == "spmm_coo":
        return fs.flagsparse_spmm_coo(*state["matrix"], state["dense"], shape)
    return fs.flagsparse_sddmm_csr(x=state["x"], y=state["y"], prepared=state["prepared"], **state["scale"])


def work(case):
    """Every array of the call read or written once.  A prepared matrix holds 32-bit column indices and row pointers
    (all of these matrices have fewer than 2^31 entries); the other calls read the index type they are given."""
    op, sv, rows, cols = case["op"], _SIZE[case["dtype"]], case["rows"], case["cols"]
    nnz, dense = rows * case["mean"], max(1, case["dense"])
    si = 8 if case["index"] == "i64" and op not in ("spmv", "spmm", "spmv_coo", "sddmm") else 4
    if op in ("spmv_coo_once", "spmm_coo"):
        matrix = nnz * (sv + 2 * si)
    else:
        matrix = nnz * ((0 if op == "sddmm" else sv) + si) + (rows + 1) * si
    if op == "sddmm":
        moved = matrix + (rows + cols) * dense * sv + nnz * sv * (2 if case["scaled"] else 1)
    else:
        moved = matrix + (rows + cols) * dense * sv
    return {"bytes": moved, "flops": nnz * dense * (8 if case["dtype"] in ("c64", "c128") else 2)}


def tolerance(case):
    """Sums in the value type (in float32 for the half precisions, rounded once at the end: what is left there is the
    last place of the result)."""
    return {"rel": _TOLERANCE[case["dtype"]]}
