// CSR SpMM (C = A B, B and C dense row-major) for sm_100a.
//
// Same tiling as the SpMV stream kernel: the nnz range is cut into tiles of T entries, so a tile of
// `data` and of `indices` is one contiguous, 16-byte aligned block.  A CTA stages its tile in shared
// memory -- with one cp.async.bulk (TMA 1-D bulk copy) per array completing on an mbarrier, or with
// ordinary coalesced loads -- and loads indptr[ra .. rb] as tile-relative offsets.  Then groups of LR
// lanes each take one row segment (VW elements per access of at most 128 bits, LR lanes and NC accesses per
// lane picked by spmm_shape below): the (value, column) pairs come from shared memory as broadcasts, each lane
// gathers its elements of B's row through the read-only path, and the accumulators stay in registers.
// This is CUDA-core work on purpose: the operand is an irregular gather with at most 0.5 flop per byte.
// Rows ending in the tile are written to C with streaming stores; a row continuing into the next tile
// leaves its partial row in carry[t, :], a row that began in an earlier tile leaves it in head[t, :],
// and a second kernel adds them up in a fixed order (deterministic, no atomics).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fsb_common.cuh"

namespace fsb {

constexpr int kMmThreads = 256;
constexpr int kMmTile = 1024;  // nnz per tile
constexpr int kMmMinPiece = 32; // shortest piece of a long segment
constexpr int kMmBuckets = 64;  // of segment lengths: two entries each, the last for all that are longer
constexpr int kWaitSpins = 1 << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
// 1-D bulk copy global -> this CTA's shared memory; src, dst and bytes are multiples of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
// bounded: gives up after kWaitSpins polls and reports it
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t phase) {
  for (int i = 0; i < kWaitSpins; ++i)
    if (mbar_try_wait(bar, phase)) return true;
  return false;
}

// ---- stored value types: what is accumulated, and how a value enters a sum ---------------------------------------
// half precisions are accumulated in float32 and rounded once when a row of C is stored
// chains: partial sums per element of C that the entries of a segment take in turn.  Two for complex values: half as many
// roundings behind one another (complex64, rows of 16 / 60 / 200 entries: one sum with both products fused into it has 1.48 /
// 1.76 / 1.86 times the rms error).  One for the others: float32 / float64 have always had one, and the half precisions have
// no registers for two of their eight sums per lane, which the rounding of the result would hide.
template <typename S>
struct MmOps {
  typedef S Acc;
  static constexpr int chains = 1;
  static __device__ __forceinline__ void fma(Acc& acc, S a, S b) { acc += a * b; }
  static __device__ __forceinline__ Acc add(Acc a, Acc b) { return a + b; }
  static __device__ __forceinline__ Acc widen(S v) { return v; }
  static __device__ __forceinline__ S narrow(Acc v) { return v; }
  static __device__ __forceinline__ Acc zero() { return (Acc)0; }
};
template <>
struct MmOps<__half> {
  typedef float Acc;
  static constexpr int chains = 1;
  static __device__ __forceinline__ void fma(Acc& acc, __half a, __half b) {
    acc = fmaf(__half2float(a), __half2float(b), acc);
  }
  static __device__ __forceinline__ Acc add(Acc a, Acc b) { return a + b; }
  static __device__ __forceinline__ Acc widen(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half narrow(Acc v) { return __float2half_rn(v); }
  static __device__ __forceinline__ Acc zero() { return 0.f; }
};
template <>
struct MmOps<__nv_bfloat16> {
  typedef float Acc;
  static constexpr int chains = 1;
  static __device__ __forceinline__ void fma(Acc& acc, __nv_bfloat16 a, __nv_bfloat16 b) {
    acc = fmaf(__bfloat162float(a), __bfloat162float(b), acc);
  }
  static __device__ __forceinline__ Acc add(Acc a, Acc b) { return a + b; }
  static __device__ __forceinline__ Acc widen(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 narrow(Acc v) { return __float2bfloat16_rn(v); }
  static __device__ __forceinline__ Acc zero() { return 0.f; }
};
template <typename C2>
struct MmComplex {
  typedef C2 Acc;
  static constexpr int chains = 2;
  static __device__ __forceinline__ void fma(Acc& acc, C2 a, C2 b) {
    // the product first, then one rounding at the size of the sum; written out, as what the compiler would fuse differs
    // between the kernels
    acc.x += ::fma(a.x, b.x, -(a.y * b.y));
    acc.y += ::fma(a.x, b.y, a.y * b.x);
  }
  static __device__ __forceinline__ Acc add(Acc a, Acc b) {
    a.x += b.x;
    a.y += b.y;
    return a;
  }
  static __device__ __forceinline__ Acc widen(C2 v) { return v; }
  static __device__ __forceinline__ C2 narrow(Acc v) { return v; }
  static __device__ __forceinline__ Acc zero() {
    Acc z;
    z.x = 0;
    z.y = 0;
    return z;
  }
};
template <> struct MmOps<float2> : MmComplex<float2> {};
template <> struct MmOps<double2> : MmComplex<double2> {};

template <typename S> struct RealOf { typedef S Out; typedef typename MmOps<S>::Acc Acc; static constexpr int parts = 1; };
template <> struct RealOf<float2> { typedef float Out; typedef float Acc; static constexpr int parts = 2; };
template <> struct RealOf<double2> { typedef double Out; typedef double Acc; static constexpr int parts = 2; };

template <int BYTES> struct RawVec;
template <> struct RawVec<2> { typedef unsigned short type; };
template <> struct RawVec<4> { typedef unsigned int type; };
template <> struct RawVec<8> { typedef uint2 type; };
template <> struct RawVec<16> { typedef uint4 type; };

// VW stored values moved as one access of VW * sizeof(S) bytes
template <typename S, int VW>
struct Pack {
  typedef typename RawVec<VW * (int)sizeof(S)>::type Raw;
  Raw raw;
  __device__ __forceinline__ void gather(const S* p) { raw = __ldg(reinterpret_cast<const Raw*>(p)); }
  __device__ __forceinline__ void load_stream(const S* p) { raw = __ldcs(reinterpret_cast<const Raw*>(p)); }
  __device__ __forceinline__ void store_stream(S* p) const { __stcs(reinterpret_cast<Raw*>(p), raw); }
  __device__ __forceinline__ S get(int i) const { return reinterpret_cast<const S*>(&raw)[i]; }
  __device__ __forceinline__ void set(int i, S v) { reinterpret_cast<S*>(&raw)[i] = v; }
};

// Resident CTAs the register budget is set for.  One access per lane: 40 registers hold four gathers of 4-byte values; left
// to itself the compiler fits 32 at times and issues them one after the other (54 columns, 28386 rows of 45 entries, float32:
// 39 us, 37 us).  Four gathers and the sums of 8-byte values take 48 (float64, 60000 rows of 31, 40 / 64 / 128 columns with 40
// registers: 70.6 / 77.8 / 145 us, with 48: 59.6 / 67.7 / 130 us, with 64: 66 / 74 / 146 us), and so do four gathers of eight
// half-precision values with their eight sums (float16, 2^20 rows of 10, 128 columns: 558 us with 40, 454 us; bfloat16, 200003 Zipf
// rows of 20, 128 columns: 157 us, 148 us; both with rows found by their stride in bytes).  Several accesses: 64 (60000 rows of 31, 65
// columns with 80 registers: float32 80.0 us, float64 114 us; with 64: 78.0 us, 98.8 us), four of them 80, which leaves 12 bytes to
// spill where rows are found by their stride in bytes (198 columns: rows of one length 4 % slower than without, others 2 to 10 %
// faster).  With long rows the pieces' arithmetic comes on top (float64, 33 columns, one row of 300 among 60000 of 31: 102 us with
// 128 registers, 82 us with 80, 88 us with 64).
__host__ __device__ constexpr int mm_ctas(int nc, size_t size, bool with_long) {
  if (nc == 1) return size == 16 ? 4 : size == 8 || size == 2 ? 5 : 6;
  if (with_long) return nc == 4 || (nc == 3 && size == 4) ? 2 : 3;
  return nc < 4 ? 4 : 3;
}

// A group of LR lanes takes one segment (the part of a row that lies in the tile) at a time, four gathers of B on their
// way.  LONG: segments of more than 2 * piece entries are left to a second pass: cut into pieces, dealt to all groups of
// the CTA, their partial rows added in shared memory.  Without it the group that meets a long row of a skewed matrix
// walks it alone while the others wait (float32, 300000 rows of Zipf lengths, 3.6 M entries, 128 columns: 402 us, with it
// 266 us; bfloat16, 200003 such rows, 4 M entries, 128 columns, from the CSR arrays, through a kernel of whole rows on
// widened copies of B and C: 8.8 ms, here 219 us).  Handing out equal slices of the tile instead, whatever rows they cross,
// balances as well but pays a row-end test per entry, and an even matrix then loses what a skewed one gains (2^20 rows
// of 16 entries, 64 columns, float32: 615 us against 531 us).  `piece` depends on the number of columns and the value
// type only (not on the alignment, which picks VW and LR), so the order of additions does too.
// BY_LENGTH: the segments of a tile are taken in the order of their lengths, the longest first: two to four groups share a warp, and
// those whose segment is shorter wait for the longest among them (us, in the order of the rows / by length: float32, 32 columns,
// 300000 rows of 5 37 / 33, 262144 Zipf rows of 16 87 / 81; 64 columns, 2^19 rows of 16 231 / 225, Zipf 130 / 123; float64, 32 columns,
// Zipf rows of 12 135 / 121).  Rows of one length lose what the sorting takes (2^20 of 16: 521 / 524), eight groups in a warp gain
// nothing (16 columns: 40.1 / 40.3), one none (float64, 64 columns: 156 / 159), several accesses a lane spill (33 columns, Zipf 91 / 109),
// and complex64 with long rows has no registers left for it (32 columns, Zipf rows: 87381 of 24 67 / 81, 419430 of 5 145 / 185).
// (As an argument of the launch it costs those that do without: 1390783 rows of 9, 16 columns, 108.1 us, 106.7 us as it is.)
// n_dense is covered by LR * NC accesses of VW elements per entry; wider products take column tiles (gridDim.y).
// ACCUM: add to what C holds instead of overwriting it (rows without entries are then left alone) -- the later passes
// of a product that the host code splits into column panels of A.
template <typename S, typename I, int VW, int NC, bool LONG, bool ACCUM, bool BY_LENGTH>
__global__ void __launch_bounds__(kMmThreads, mm_ctas(NC, sizeof(S), LONG))
spmm_tile_kernel(const S* __restrict__ data, const I* __restrict__ idx, const void* __restrict__ ptr, int ptr64,
                 const S* __restrict__ B, int64_t ldb, S* __restrict__ C, int64_t ldc,
                 const int32_t* __restrict__ tile_row, typename MmOps<S>::Acc* __restrict__ carry,
                 typename MmOps<S>::Acc* __restrict__ head, int64_t nnz, int n_dense, int LR, int piece,
                 int use_bulk, int32_t* __restrict__ status) {
  typedef MmOps<S> Ops;
  typedef typename Ops::Acc A;
  constexpr int T = kMmTile;
  constexpr int RC = T;
  constexpr int U = 4;                                    // entries whose gathers are in flight together
  constexpr int PIECES = T / kMmMinPiece + T / (2 * kMmMinPiece);   // most pieces the long segments of a tile have
  __shared__ __align__(128) S s_val[T];
  __shared__ __align__(128) I s_idx[T];
  __shared__ int32_t s_off[RC + 1];
  __shared__ int32_t s_piece_at[LONG ? PIECES : 1];       // a piece: first entry | end << 16
  __shared__ int32_t s_long[LONG ? T / (2 * kMmMinPiece) : 1];   // a long segment: number | first piece << 16
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ int s_head_partial;
  __shared__ int s_failed;
  __shared__ int s_n_long, s_n_pieces;
  __shared__ uint16_t s_order[BY_LENGTH ? RC : 1];        // segments by length
  __shared__ int s_bucket[BY_LENGTH ? kMmBuckets : 1];
  extern __shared__ __align__(16) unsigned char s_parts[];

  const int tid = threadIdx.x;
  const int64_t t = blockIdx.x;
  const int64_t lo = t * (int64_t)T;
  const int cnt = (int)((nnz - lo) < (int64_t)T ? (nnz - lo) : (int64_t)T);
  const int32_t ra = tile_row[t];
  const int32_t rb = tile_row[t + 1];

  // ---- stage the tile -------------------------------------------------------------------------
  const bool bulk = use_bulk && cnt == T;
  if (bulk) {
    if (tid == 0) {
      s_failed = 0;
      mbar_init(&s_bar, 1);
      fence_barrier_init();
    }
    __syncthreads();
    if (tid == 0) {
      mbar_expect_tx(&s_bar, (uint32_t)(T * (sizeof(S) + sizeof(I))));
      bulk_g2s(s_val, data + lo, (uint32_t)(T * sizeof(S)), &s_bar);
      bulk_g2s(s_idx, idx + lo, (uint32_t)(T * sizeof(I)), &s_bar);
    }
  } else {
    for (int e = tid; e < cnt; e += kMmThreads) {
      s_val[e] = ld_stream(data + lo + e);
      s_idx[e] = ld_stream(idx + lo + e);
    }
  }

  // segments: rows ra .. rb-1 end in this tile, segment nrf is the row that continues
  const int nrf = rb - ra;
  const int nseg = nrf + 1;
  const int lane = tid & (LR - 1);
  const int grp = tid / LR;
  const int ngrp = kMmThreads / LR;
  const int width = LR * NC * VW;                          // columns of this column tile
  const int col0 = (int)blockIdx.y * width + lane * VW;    // first column of access 0; access i is LR * VW further on

  // Row c of B: one wide multiply-add from a stride in bytes, and one for the high word, where several accesses per lane, small ones
  // or conversions leave the arithmetic in the way of the gathers (float32, 262144 rows of 16, 33 columns: 102 us, from the stride in
  // elements 112 us; float16, 200003 rows of 20, 70 columns: 132 / 146, 200 columns: 229 / 241; complex64, 32 columns: 81 / 86).  float64
  // and 16-byte gathers of one access lose registers to it (float64, 75 columns: 179 / 161; float32, 64 columns: 256 / 233).
  // ROWS_FIRST: the four rows before the first of their gathers; single floats, one access, left each gather waiting for its own row
  // where few tiles run (5461 rows of 24, 13 / 21 columns: stride in elements 8.6 / 12.3 us, in bytes 9.5 / 13.9, here 8.3 / 11.7; 174762
  // rows of 24, 21 columns: 81.5, 71.7, 66.7).  Others lose to it (float32, 70 columns 2 %, float64, 33 columns 12 %) or do not care.
  // Eight half-precision values at a time, long rows, by length: the same (bfloat16, 128 columns, 419430 Zipf rows of 5: 164 / 147).
  constexpr bool FROM_BYTES = RealOf<S>::parts == 2 || (sizeof(S) == 2 && !(BY_LENGTH && LONG && VW == 8)) ||
                              (sizeof(S) == 4 && VW * (int)sizeof(S) < 16);
  constexpr bool ROWS_FIRST = sizeof(S) == 4 && VW == 1 && NC == 1;
  const char* B0 = reinterpret_cast<const char*>(B + col0);
  const uint64_t row_bytes = (uint64_t)ldb * sizeof(S);
  auto row_of = [&](I c) {
    if constexpr (FROM_BYTES) return reinterpret_cast<const S*>(B0 + (uint64_t)(uint32_t)c * row_bytes);
    else return B + (int64_t)c * ldb + col0;
  };
  auto clear = [](A (&acc)[NC][VW]) {
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < VW; ++j) acc[i][j] = Ops::zero();
  };
  constexpr int CHAINS = Ops::chains;
  // acc += value * row of B for entry p
  auto one = [&](int p, A (&acc)[NC][VW]) {
    const S* row = row_of(s_idx[p]);
    const S v = s_val[p];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      if (i == 0 || col0 + i * LR * VW < n_dense) {
        Pack<S, VW> b;
        b.gather(row + i * LR * VW);
#pragma unroll
        for (int j = 0; j < VW; ++j) Ops::fma(acc[i][j], v, b.get(j));
      }
    }
  };
  // acc = sum over the entries p .. e-1 of value * row of B (acc comes in cleared)
  auto walk = [&](int p, int e, A (&acc)[NC][VW]) {
    A odd[NC][VW];                         // every other entry, where there are two partial sums
    if (CHAINS == 2) clear(odd);
    for (; p + U <= e; p += U) {
      Pack<S, VW> b[U][NC];
      const S* rows[ROWS_FIRST ? U : 1];
      if constexpr (ROWS_FIRST) {
#pragma unroll
        for (int u = 0; u < U; ++u) rows[u] = row_of(s_idx[p + u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const S* row = ROWS_FIRST ? rows[ROWS_FIRST ? u : 0] : row_of(s_idx[p + u]);
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (i == 0 || col0 + i * LR * VW < n_dense) b[u][i].gather(row + i * LR * VW);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const S v = s_val[p + u];
#pragma unroll
        for (int i = 0; i < NC; ++i)
#pragma unroll
          for (int j = 0; j < VW; ++j) Ops::fma(CHAINS == 2 && (u & 1) ? odd[i][j] : acc[i][j], v, b[u][i].get(j));
      }
    }
    for (; p < e; ++p) {
      one(p, acc);
      if (CHAINS == 2 && ++p < e) one(p, odd);
    }
    if (CHAINS == 2) {
#pragma unroll
      for (int i = 0; i < NC; ++i)
#pragma unroll
        for (int j = 0; j < VW; ++j) acc[i][j] = Ops::add(acc[i][j], odd[i][j]);
    }
  };
  // the sum of segment g: to C, or to the arrays that the fix-up adds up
  auto finish = [&](int g, bool has_entries, const A (&acc)[NC][VW]) {
    const bool to_carry = g == nrf, to_head = g == 0 && s_head_partial;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int col = col0 + i * LR * VW;
      if (i > 0 && col >= n_dense) break;
      if (to_carry || to_head) {
        A* dst = (to_carry ? carry : head) + t * n_dense + col;
#pragma unroll
        for (int j = 0; j < VW; ++j) dst[j] = acc[i][j];
      } else {
        S* dst = C + ((int64_t)ra + g) * ldc + col;
        Pack<S, VW> out;
        if (!ACCUM) {
#pragma unroll
          for (int j = 0; j < VW; ++j) out.set(j, Ops::narrow(acc[i][j]));
          out.store_stream(dst);
        } else if (has_entries) {     // a row without entries leaves its row of C alone
          out.load_stream(dst);
#pragma unroll
          for (int j = 0; j < VW; ++j) out.set(j, Ops::narrow(Ops::add(acc[i][j], Ops::widen(out.get(j)))));
          out.store_stream(dst);
        }
      }
    }
  };

  for (int base = 0; base < nseg; base += RC) {
    const int m = (nseg - base) < RC ? (nseg - base) : RC;
    __syncthreads();
    for (int k = tid; k <= m; k += kMmThreads) {
      const int g = base + k;
      int32_t o = cnt;
      if (g <= nrf) {
        const int64_t row = (int64_t)ra + g;
        const int64_t d = (ptr64 ? static_cast<const int64_t*>(ptr)[row]
                                 : (int64_t) static_cast<const int32_t*>(ptr)[row]) - lo;
        o = d < 0 ? 0 : (d > cnt ? cnt : (int32_t)d);
        if (g == 0) s_head_partial = (d < 0 && nrf > 0) ? 1 : 0;
      }
      s_off[k] = o;
    }
    if (LONG && tid == 0) {
      s_n_long = 0;
      s_n_pieces = 0;
    }
    if (bulk && base == 0) {
      // every thread polls the barrier itself: completion makes the copied bytes visible to it
      if (!mbar_wait_bounded(&s_bar, 0)) s_failed = 1;
    }
    __syncthreads();
    if (bulk && s_failed) {
      // the copy did not land within the bound: report it and leave this tile unwritten
      if (tid == 0 && status != nullptr) *reinterpret_cast<volatile int32_t*>(status) = 1;  // may be host memory
      mbar_wait_bounded(&s_bar, 0);  // one more bounded wait so that no copy is in flight at exit
      return;
    }

    // (a group has one segment at most: nothing to choose from.  float64, 682 rows of 48, 16 columns: sorted 8.7 us, 8.4 us)
    const bool sorted = BY_LENGTH && m > ngrp;
    if (sorted) {
      auto bucket = [&](int k) {                 // the longest first
        const int len = s_off[k + 1] - s_off[k];
        return kMmBuckets - 1 - (len < 2 * kMmBuckets - 2 ? len : 2 * kMmBuckets - 2) / 2;
      };
      if (tid < kMmBuckets) s_bucket[tid] = 0;
      __syncthreads();
      for (int k = tid; k < m; k += kMmThreads) atomicAdd(&s_bucket[bucket(k)], 1);
      __syncthreads();
      if (tid < 32) {
        const int c0 = s_bucket[2 * tid], c1 = s_bucket[2 * tid + 1];
        int upto = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, upto, o);
          if (tid >= o) upto += v;
        }
        s_bucket[2 * tid] = upto - c0 - c1;
        s_bucket[2 * tid + 1] = upto - c1;
      }
      __syncthreads();
      for (int k = tid; k < m; k += kMmThreads) s_order[atomicAdd(&s_bucket[bucket(k)], 1)] = (uint16_t)k;
      __syncthreads();
    }
    for (int q = grp; q < m; q += ngrp) {
      const int k = sorted ? s_order[BY_LENGTH ? q : 0] : q;
      const int s = s_off[k], e = s_off[k + 1];
      if (LONG && e - s > 2 * piece) {
        if (lane == 0) {
          const int n = (e - s + piece - 1) / piece;
          const int first = atomicAdd(&s_n_pieces, n);
          s_long[atomicAdd(&s_n_long, 1)] = k | first << 16;
          for (int q = 0; q < n; ++q) {
            const int p = s + q * piece;
            s_piece_at[first + q] = p | (p + piece < e ? p + piece : e) << 16;
          }
        }
      } else if (col0 < n_dense) {
        A acc[NC][VW];
        clear(acc);
        walk(s, e, acc);
        finish(base + k, e > s, acc);
      }
    }
    if (!LONG) continue;
    __syncthreads();
    const int n_long = s_n_long;
    if (n_long > 0) {
      A* parts = reinterpret_cast<A*>(s_parts);
      const int n_pieces = s_n_pieces;
      for (int q = grp; q < n_pieces; q += ngrp) {
        if (col0 < n_dense) {
          A acc[NC][VW];
          clear(acc);
          walk(s_piece_at[q] & 0xFFFF, s_piece_at[q] >> 16, acc);
#pragma unroll
          for (int i = 0; i < NC; ++i)
#pragma unroll
            for (int j = 0; j < VW; ++j) parts[q * width + (i * LR + lane) * VW + j] = acc[i][j];
        }
      }
      __syncthreads();
      for (int q = grp; q < n_long; q += ngrp) {
        const int k = s_long[q] & 0xFFFF, first = s_long[q] >> 16;
        const int n = (s_off[k + 1] - s_off[k] + piece - 1) / piece;
        if (col0 < n_dense) {
          A acc[NC][VW];
          clear(acc);
          for (int p = first; p < first + n; ++p)
#pragma unroll
            for (int i = 0; i < NC; ++i)
#pragma unroll
              for (int j = 0; j < VW; ++j)
                acc[i][j] = Ops::add(acc[i][j], parts[p * width + (i * LR + lane) * VW + j]);
          finish(base + k, true, acc);
        }
      }
    }
  }
}

// one thread per (tile t >= 1, column): finish the row that started before tile t and ends in it.  Partial sums are added as doubles
// with what each addition loses, which takes a thread about 0.2 us each.  Floats whose exponents lie close enough together lose
// nothing, so they are added as they are, and again with the losses where they do not: the same bits (whole products, all with the
// losses / here: float32, 838860 Zipf rows of 5, 32 columns 171 / 139 us; bfloat16, 262144 such rows of 16, 128 columns 182 / 166).
// R: real type of the partial sums, D: real type of C (complex columns are taken as pairs of real ones)
template <typename R, typename D, typename P>
__global__ void __launch_bounds__(kMmThreads)
spmm_fixup_kernel(const P* __restrict__ ptr, const int32_t* __restrict__ tile_row,
                  const R* __restrict__ carry, const R* __restrict__ head, D* __restrict__ C, int64_t ldc,
                  int64_t n_tiles, int n_dense, int log2_tile, int accumulate) {
  const int64_t gid = (int64_t)blockIdx.x * kMmThreads + threadIdx.x;
  const int64_t t = gid / n_dense + 1;
  const int j = (int)(gid % n_dense);
  if (t >= n_tiles) return;
  const int32_t ra = tile_row[t];
  const int32_t rb = tile_row[t + 1];
  if (ra >= rb) return;
  const int64_t p = (int64_t)ptr[ra];
  if (p >= (t << log2_tile)) return;
  const R first = head[t * n_dense + j];
  const int n = (int)(t - (p >> log2_tile));          // partial sums in the tiles before
  const R* from = carry + (t - n) * n_dense + j;
  double sum = (double)first, comp = 0.0;
  if constexpr (sizeof(R) == 4) {
    // the largest magnitude, and the smallest that is not zero, less one
    uint32_t most = __float_as_uint(first) & 0x7FFFFFFFu, least = most - 1u;
    auto add = [&](float v) {
      const uint32_t bits = __float_as_uint(v) & 0x7FFFFFFFu;
      most = max(most, bits);
      least = min(least, bits - 1u);
      sum += (double)v;
    };
    int u = 0;
    for (; u + 8 <= n; u += 8) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __ldg(from + (int64_t)(u + k) * n_dense);
#pragma unroll
      for (int k = 0; k < 8; ++k) add(v[k]);
    }
    for (; u < n; ++u) add(__ldg(from + (int64_t)u * n_dense));
    // n + 1 numbers of 24 bits, exponents `range` apart: every sum of them has at most this many bits
    const int low = (int)((least + 1u) >> 23), range = (int)(most >> 23) - (low > 0 ? low : 1);
    if (24 + range + (32 - __clz(n)) > 53) {
      sum = (double)first;
#pragma unroll 1
      for (int u = 0; u < n; ++u) comp_add(sum, comp, (double)__ldg(from + (int64_t)u * n_dense));
    }
  } else {
    // (eight and more: four sums in turn, or each would wait for the one before it)
    double sums[4] = {(double)first, 0.0, 0.0, 0.0}, comps[4] = {0.0, 0.0, 0.0, 0.0};
    int u = 0;
    for (; u + 8 <= n; u += 8) {
      R v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __ldg(from + (int64_t)(u + k) * n_dense);
#pragma unroll
      for (int k = 0; k < 8; ++k) comp_add(sums[k & 3], comps[k & 3], (double)v[k]);
    }
    if (u > 0) {
#pragma unroll
      for (int k = 1; k < 4; ++k) {
        comp_add(sums[0], comps[0], sums[k]);
        comps[0] += comp_term(sums[k], comps[k]);
      }
    }
    for (; u < n; ++u) comp_add(sums[0], comps[0], (double)__ldg(from + (int64_t)u * n_dense));
    sum = sums[0];
    comp = comps[0];
  }
  D* dst = C + (int64_t)ra * ldc + j;
  comp = comp_term(sum, comp);
  // rounded to the accumulator type first, like every other row
  const R r = accumulate ? (R)(((double)MmOps<D>::widen(*dst) + sum) + comp) : (R)(sum + comp);
  *dst = MmOps<D>::narrow(r);
}

template <typename V>
__global__ void __launch_bounds__(kMmThreads) zero_rows_kernel(V* __restrict__ C, int64_t ldc, int64_t n_rows,
                                                              int64_t n_dense) {
  const int64_t gid = (int64_t)blockIdx.x * kMmThreads + threadIdx.x;
  const int64_t r = gid / n_dense;
  const int64_t j = gid % n_dense;
  if (r < n_rows) C[r * ldc + j] = (V)0;
}

struct SpmmArgs {
  const void *data, *idx, *ptr, *B;
  int64_t ldb;
  void* C;
  int64_t ldc, n_rows, n_dense, nnz;
  int algo, ptype;
  bool accumulate, long_rows, uneven_rows;
  const int32_t* tile_row;
  int32_t* own_plan;      // the plan has to be made first, here (tile_row is the same address)
  void* scratch;
  int32_t* status;
  cudaStream_t st;
};

static int pow2_at_least(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}

template <typename S, typename I, int VW, int NC>
static int launch_spmm(const SpmmArgs& a, int LR, int piece) {
  typedef typename MmOps<S>::Acc A;
  constexpr int T = kMmTile;
  constexpr bool REAL = sizeof(S) >= 4 && RealOf<S>::parts == 1;   // the types that are ever accumulated into C
  const int64_t n_tiles = (a.nnz + T - 1) / T;
  const int n_dense = (int)a.n_dense;
  const int width = LR * NC * VW;
  const int64_t col_tiles = (n_dense + width - 1) / width;
  const int cols = n_dense * RealOf<S>::parts;
  const int64_t fix_blocks = n_tiles > 1 ? ((n_tiles - 1) * cols + kMmThreads - 1) / kMmThreads : 0;
  if (col_tiles > 65535 || fix_blocks >= INT32_MAX) return FSB_ERANGE;
  if (a.own_plan != nullptr) {      // the first launch: whatever a call can be refused for has been looked at by now
    const int rc = fsb_csr_tile_plan(a.ptype, a.ptr, a.n_rows, a.nnz, T, a.own_plan, a.st);
    if (rc != FSB_OK) return rc;
  }
  A* carry = (A*)a.scratch;
  A* head = carry + n_tiles * n_dense;
  const int bulk = a.algo != FSB_SPMM_PLAIN && aligned_to(a.data, 16) && aligned_to(a.idx, 16);
  const dim3 grid((unsigned)n_tiles, (unsigned)col_tiles);
  constexpr bool SORTS_LONG = NC == 1 && !(RealOf<S>::parts == 2 && sizeof(S) == 8);
  const bool by_length = a.uneven_rows && !a.accumulate && (a.long_rows ? SORTS_LONG : NC == 1) && LR >= 8 && LR < 32;
#define FSB_SPMM_LAUNCH(LONG_, ACC_, LEN_, SMEM_)                                                                    \
  spmm_tile_kernel<S, I, VW, NC, LONG_, ACC_, LEN_><<<grid, kMmThreads, SMEM_, a.st>>>(                              \
      (const S*)a.data, (const I*)a.idx, a.ptr, a.ptype == FSB_I64, (const S*)a.B, a.ldb, (S*)a.C, a.ldc, a.tile_row, \
      carry, head, a.nnz, n_dense, LR, piece, bulk, a.status)
  // the long segments of a tile (more than 2 * piece entries each) have at most T / piece + T / (2 * piece) pieces
  const size_t parts = a.long_rows ? (size_t)(T / piece + T / (2 * piece)) * width * sizeof(A) : 0;
  if (a.accumulate && !REAL) return FSB_EINVAL;
  if (a.long_rows) {
    if constexpr (NC == 1 || VW * (int)sizeof(S) < 16) {       // spmm_shape gives long rows no other
      if constexpr (REAL) {
        if (a.accumulate) FSB_SPMM_LAUNCH(true, true, false, parts);
      }
      if constexpr (SORTS_LONG) {
        if (by_length) FSB_SPMM_LAUNCH(true, false, true, parts);
      }
      if (!a.accumulate && !by_length) FSB_SPMM_LAUNCH(true, false, false, parts);
    } else {
      return FSB_EINVAL;
    }
  } else {
    if constexpr (REAL) {
      if (a.accumulate) FSB_SPMM_LAUNCH(false, true, false, 0);
    }
    if constexpr (NC == 1) {
      if (by_length) FSB_SPMM_LAUNCH(false, false, true, 0);
    }
    if (!a.accumulate && !by_length) FSB_SPMM_LAUNCH(false, false, false, 0);
  }
#undef FSB_SPMM_LAUNCH
  FSB_RETURN_IF_LAUNCH_FAILED();
  if (fix_blocks > 0) {
    typedef RealOf<S> R;
    int log2_tile = 0;
    while ((1 << log2_tile) < T) ++log2_tile;
#define FSB_SPMM_FIXUP(P_)                                                                                          \
  spmm_fixup_kernel<typename R::Acc, typename R::Out, P_><<<(unsigned)fix_blocks, kMmThreads, 0, a.st>>>(          \
      (const P_*)a.ptr, a.tile_row, (const typename R::Acc*)carry, (const typename R::Acc*)head,                   \
      (typename R::Out*)a.C, a.ldc * R::parts, n_tiles, cols, log2_tile, a.accumulate)
    if (a.ptype == FSB_I64) FSB_SPMM_FIXUP(int64_t); else FSB_SPMM_FIXUP(int32_t);
#undef FSB_SPMM_FIXUP
    FSB_RETURN_IF_LAUNCH_FAILED();
  }
  return FSB_OK;
}

// Lanes per entry (LR, a power of two) and accesses per lane (NC).  Up to 32 accesses there is one per lane (5 columns as
// 2 lanes x 3: 66 us, as 8 lanes: 48 us, 200000 rows of 20 entries).  Beyond, the pair with the fewest idle lanes: 33
// single columns take 16 lanes x 3 instead of two passes over the matrix with 32 lanes.  NC is bounded by what a lane
// accumulates in registers (32 bytes); 8-byte values in 16-byte accesses take one, as two leave too few CTAs in flight
// (float64, 60000 rows of 31, 96 columns: 126 us and 113 us; 262144 rows of 16, 128 columns: 563 us and 455 us), and so do
// other 16-byte accesses where rows are long (float32, 160 columns, 262144 rows of 16 and one of 300: 427 us and 322 us).
template <typename S, typename I, int VW>
static int spmm_shape(const SpmmArgs& a) {
  typedef typename MmOps<S>::Acc A;
  constexpr int VMAX = 16 / (int)sizeof(S);
  constexpr int HELD = VW * (int)sizeof(A);      // accumulator bytes of one access
  // (16-byte values: one, or the pieces of long segments would not fit beside the staged tile)
  constexpr int NC_TYPE = sizeof(S) == 16 || HELD >= 32 || (sizeof(S) == 8 && VW == VMAX) ? 1 : (32 / HELD < 4 ? 32 / HELD : 4);
  const int nc_max = VW == VMAX && a.long_rows ? 1 : NC_TYPE;
  const int64_t need = (a.n_dense + VW - 1) / VW;
  const int64_t need_widest = (a.n_dense + VMAX - 1) / VMAX;
  const int LR_min = pow2_at_least((int)(need_widest < 32 ? need_widest : 32));   // what a 16-byte access would use
  // half a group's even share of a tile, at least kMmMinPiece: a segment is long from twice that on
  const int share = kMmTile / kMmThreads * LR_min;
  const int piece = share / 2 > kMmMinPiece ? share / 2 : kMmMinPiece;
  int LR = 32, NC = 1;
  if (need <= 32) {
    LR = pow2_at_least((int)need);
  } else {
    int64_t best = -1;
    for (int nc = 1; nc <= nc_max; ++nc)
      for (int lr = LR_min; lr <= 32; lr <<= 1) {
        const int64_t passes = (need + lr * nc - 1) / (lr * nc);
        const int64_t cost = passes * lr * nc * 64 + passes;   // idle lanes first, then passes over the matrix
        if (best < 0 || cost < best) {
          best = cost;
          LR = lr;
          NC = nc;
        }
      }
  }
  if constexpr (NC_TYPE >= 2) {
    if (NC == 2) return launch_spmm<S, I, VW, 2>(a, LR, piece);
  }
  if constexpr (NC_TYPE >= 4) {
    if (NC == 3) return launch_spmm<S, I, VW, 3>(a, LR, piece);
    if (NC == 4) return launch_spmm<S, I, VW, 4>(a, LR, piece);
  }
  return launch_spmm<S, I, VW, 1>(a, LR, piece);
}

template <typename S, typename I>
static int spmm_typed(const SpmmArgs& a) {
  // widest access that divides the row length and keeps every row of B and C aligned
  constexpr int VMAX = 16 / (int)sizeof(S);
  int vw = VMAX;
  while (vw > 1 && !(a.n_dense % vw == 0 && a.ldb % vw == 0 && a.ldc % vw == 0 &&
                     aligned_to(a.B, vw * sizeof(S)) && aligned_to(a.C, vw * sizeof(S))))
    vw >>= 1;
  if constexpr (VMAX >= 8) {
    if (vw == 8) return spmm_shape<S, I, 8>(a);
  }
  if constexpr (VMAX >= 4) {
    if (vw == 4) return spmm_shape<S, I, 4>(a);
  }
  if constexpr (VMAX >= 2) {
    if (vw == 2) return spmm_shape<S, I, 2>(a);
  }
  return spmm_shape<S, I, 1>(a);
}

static size_t stored_size(int vtype) {
  return vtype == FSB_F16 || vtype == FSB_BF16 ? 2 : vtype == FSB_F32 ? 4 : vtype == FSB_C128 ? 16 : 8;
}
static size_t acc_size(int vtype) { return stored_size(vtype) < 4 ? 4 : stored_size(vtype); }

static size_t spmm_scratch_bytes(int vtype, int64_t nnz, int64_t n_dense) {
  const int64_t n_tiles = fsb_csr_num_tiles(nnz, kMmTile);
  const size_t b = (size_t)n_tiles * 2 * (size_t)(n_dense > 0 ? n_dense : 0) * acc_size(vtype);
  return (b + 255) & ~(size_t)255;
}

static size_t spmm_plan_bytes(int64_t nnz) {
  return (((size_t)fsb_csr_num_tiles(nnz, kMmTile) + 1) * sizeof(int32_t) + 255) & ~(size_t)255;
}

// plan_in_scratch: no tile_row; the plan is made behind the partial rows, in the last spmm_plan_bytes() of the scratch
static int spmm_run(int vtype, int itype, int ptype, const void* data, const void* indices, const void* indptr,
                    const void* B, int64_t ldb, void* C, int64_t ldc, int64_t n_rows, int64_t n_cols, int64_t n_dense,
                    int64_t nnz, int algo, const int32_t* tile_row, bool plan_in_scratch, void* scratch,
                    size_t scratch_bytes, int32_t* status, cudaStream_t st) {
  if ((itype != FSB_I32 && itype != FSB_I64) || (ptype != FSB_I32 && ptype != FSB_I64)) return FSB_EINVAL;
  const bool accumulate = (algo & FSB_SPMM_ACCUMULATE) != 0;
  const bool long_rows = (algo & FSB_SPMM_LONG_ROWS) != 0, uneven_rows = (algo & FSB_SPMM_UNEVEN_ROWS) != 0;
  algo &= ~(FSB_SPMM_ACCUMULATE | FSB_SPMM_LONG_ROWS | FSB_SPMM_UNEVEN_ROWS);
  if (algo != FSB_SPMM_AUTO && algo != FSB_SPMM_PLAIN && algo != FSB_SPMM_BULK) return FSB_EINVAL;
  if (n_rows < 0 || n_cols < 0 || n_dense < 0 || nnz < 0) return FSB_EINVAL;
  if (n_rows >= INT32_MAX || n_cols >= INT32_MAX || n_dense >= (1 << 24)) return FSB_ERANGE;
  if (ptype == FSB_I32 && nnz > INT32_MAX) return FSB_ERANGE;
  if (n_rows == 0 || n_dense == 0) return FSB_OK;
  if (C == nullptr || indptr == nullptr || ldc < n_dense) return FSB_EINVAL;
  const size_t sv = stored_size(vtype), si = itype == FSB_I32 ? 4 : 8, sp = ptype == FSB_I32 ? 4 : 8;
  if (!aligned_to(C, sv) || !aligned_to(indptr, sp)) return FSB_EALIGN;
  FSB_WALK_FIRST(check_csr(itype, ptype, indices, indptr, n_rows, n_cols, nnz, st));
  if (nnz == 0 && accumulate) return FSB_OK;   // nothing to add
  if (nnz == 0) {
    const int64_t words = sv < 4 ? 1 : (int64_t)(sv / 4);    // 2- or 4-byte words per element
    const int64_t g = (n_rows * n_dense * words + kMmThreads - 1) / kMmThreads;
    if (g >= INT32_MAX) return FSB_ERANGE;
    if (sv == 2)
      zero_rows_kernel<uint16_t><<<(unsigned)g, kMmThreads, 0, st>>>((uint16_t*)C, ldc, n_rows, n_dense);
    else
      zero_rows_kernel<uint32_t><<<(unsigned)g, kMmThreads, 0, st>>>((uint32_t*)C, ldc * words, n_rows, n_dense * words);
    FSB_RETURN_IF_LAUNCH_FAILED();
    return FSB_OK;
  }
  if (data == nullptr || indices == nullptr || B == nullptr || ldb < n_dense) return FSB_EINVAL;
  if (!aligned_to(data, sv) || !aligned_to(B, sv) || !aligned_to(indices, si)) return FSB_EALIGN;
  if ((tile_row == nullptr && !plan_in_scratch) || scratch == nullptr) return FSB_EINVAL;
  const size_t parts_bytes = spmm_scratch_bytes(vtype, nnz, n_dense);
  if (scratch_bytes < parts_bytes + (plan_in_scratch ? spmm_plan_bytes(nnz) : 0)) return FSB_ESCRATCH;
  if (!aligned_to(scratch, 16)) return FSB_EALIGN;
  if (fsb_csr_num_tiles(nnz, kMmTile) >= 65535LL * 32768LL) return FSB_ERANGE;

  int32_t* own_plan = plan_in_scratch ? (int32_t*)((char*)scratch + parts_bytes) : nullptr;
  SpmmArgs a{data, indices, indptr, B, ldb, C, ldc, n_rows, n_dense, nnz, algo, ptype, accumulate, long_rows, uneven_rows,
             plan_in_scratch ? own_plan : tile_row, own_plan, scratch, status, st};
  if (vtype == FSB_F32) return itype == FSB_I32 ? spmm_typed<float, int32_t>(a) : spmm_typed<float, int64_t>(a);
  if (vtype == FSB_F64) return itype == FSB_I32 ? spmm_typed<double, int32_t>(a) : spmm_typed<double, int64_t>(a);
  if (itype != FSB_I32) return FSB_EINVAL;
  if (vtype == FSB_F16) return spmm_typed<__half, int32_t>(a);
  if (vtype == FSB_BF16) return spmm_typed<__nv_bfloat16, int32_t>(a);
  if (vtype == FSB_C64) return spmm_typed<float2, int32_t>(a);
  return spmm_typed<double2, int32_t>(a);
}

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_spmm_tile_nnz(int vtype) {
  (void)vtype;
  return kMmTile;
}

extern "C" size_t fsb_spmm_csr_scratch_bytes(int vtype, int64_t nnz, int64_t n_dense) {
  return spmm_scratch_bytes(vtype, nnz, n_dense);
}

extern "C" int fsb_spmm_csr(int vtype, int itype, int ptype, const void* data, const void* indices,
                            const void* indptr, const void* B, int64_t ldb, void* C, int64_t ldc,
                            int64_t n_rows, int64_t n_cols, int64_t n_dense, int64_t nnz, int algo,
                            const int32_t* tile_row, void* scratch, size_t scratch_bytes, int32_t* status,
                            void* stream_) {
  if (vtype != FSB_F32 && vtype != FSB_F64) return FSB_EINVAL;
  return spmm_run(vtype, itype, ptype, data, indices, indptr, B, ldb, C, ldc, n_rows, n_cols, n_dense, nnz, algo,
                  tile_row, false, scratch, scratch_bytes, status, static_cast<cudaStream_t>(stream_));
}

extern "C" size_t fsb_spmm_stored_scratch_bytes(int vtype, int64_t nnz, int64_t n_dense) {
  return spmm_scratch_bytes(vtype, nnz, n_dense) + spmm_plan_bytes(nnz);
}

extern "C" int fsb_spmm_csr_stored(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr,
                                   const void* B, int64_t ldb, void* C, int64_t ldc, int64_t n_rows, int64_t n_cols,
                                   int64_t n_dense, int64_t nnz, int long_rows, void* scratch, size_t scratch_bytes,
                                   void* stream_) {
  return fsb_spmm_csr_stored_rows(vtype, ptype, data, indices, indptr, B, ldb, C, ldc, n_rows, n_cols, n_dense, nnz,
                                  long_rows ? FSB_SPMM_LONG_ROWS : 0, scratch, scratch_bytes, stream_);
}

extern "C" int fsb_spmm_csr_stored_rows(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr,
                                        const void* B, int64_t ldb, void* C, int64_t ldc, int64_t n_rows, int64_t n_cols,
                                        int64_t n_dense, int64_t nnz, int hints, void* scratch, size_t scratch_bytes,
                                        void* stream_) {
  if (vtype != FSB_F16 && vtype != FSB_BF16 && vtype != FSB_C64 && vtype != FSB_C128) return FSB_EINVAL;
  if (hints & ~(FSB_SPMM_LONG_ROWS | FSB_SPMM_UNEVEN_ROWS)) return FSB_EINVAL;
  // staged by ordinary loads: no copy whose end would have to be waited for and reported
  return spmm_run(vtype, FSB_I32, ptype, data, indices, indptr, B, ldb, C, ldc, n_rows, n_cols, n_dense, nnz,
                  FSB_SPMM_PLAIN | hints, nullptr, true, scratch, scratch_bytes, nullptr, static_cast<cudaStream_t>(stream_));
}

extern "C" int fsb_spmm_csr_once(int vtype, int itype, int ptype, const void* data, const void* indices, const void* indptr,
                                 const void* B, int64_t ldb, void* C, int64_t ldc, int64_t n_rows, int64_t n_cols, int64_t n_dense,
                                 int64_t nnz, int64_t long_row, void* scratch, size_t scratch_bytes, void* work, int64_t* host,
                                 void* stream_) {
  const cudaStream_t st = static_cast<cudaStream_t>(stream_);
  if (vtype < FSB_F32 || vtype > FSB_C128 || n_dense < 0 || nnz <= 0) return FSB_EINVAL;
  const size_t parts = spmm_scratch_bytes(vtype, nnz, n_dense);
  if (scratch == nullptr) return FSB_EINVAL;
  if (scratch_bytes < parts + spmm_plan_bytes(nnz)) return FSB_ESCRATCH;
  if (!aligned_to(scratch, 16)) return FSB_EALIGN;
  int rc = csr_check_launch(itype, ptype, indices, indptr, n_rows, nnz, work, host, st);
  if (rc != FSB_OK) return rc;
  // the plan needs no checked row pointer: it reads n_rows + 1 numbers and writes its own array, whatever they are
  int32_t* tile_row = (int32_t*)((char*)scratch + parts);
  rc = fsb_csr_tile_plan(ptype, indptr, n_rows, nnz, kMmTile, tile_row, stream_);
  const int waited = csr_check_wait(host, st);
  if (rc != FSB_OK || waited != FSB_OK) return rc != FSB_OK ? rc : waited;
  if (!csr_check_passed(host, n_cols, nnz)) return FSB_NOT_LAUNCHED;
  const int64_t longest = csr_check_longest(host);
  const int algo = FSB_SPMM_PLAIN | (longest > long_row ? FSB_SPMM_LONG_ROWS : 0) |
                   (4 * longest * n_rows > 5 * nnz ? FSB_SPMM_UNEVEN_ROWS : 0);
  return spmm_run(vtype, itype, ptype, data, indices, indptr, B, ldb, C, ldc, n_rows, n_cols, n_dense, nnz, algo, tile_row, false,
                  scratch, parts, nullptr, st);
}
