// COO triples -> rows: a stable least-significant-digit radix sort of the row ids (after the column ids, where a row's
// entries are wanted in column order, too), the checks of both id arrays, and the row pointer.
//
// A row id of a matrix with n_rows rows has bits(n_rows - 1) digits' worth of information, not 32: 150001 rows are two passes
// of nine bits.  One pass is three launches: counts of every digit per tile of 2048 or 4096 entries; a scan over the tiles for
// every digit; and the move, in which a tile ranks its entries (equal digits of a warp find each other by votes, a warp
// counts its own in shared memory), brings them into digit order in shared memory and writes each digit's run to its place.
// The first count also takes the minimum and maximum of both id arrays, the last move fetches values and columns in their
// new order, so that nothing but (id, position) pairs is moved before.  All of it is enqueued without a look at the checks:
// ids out of range lead nowhere but to a place inside the arrays, and the caller reads the statistics once, at the end.
// 2.1 M triples in no order, 150001 rows, 64-bit ids: 105 us of kernels -- first count with the checks 14 us, moves 23 and 41 us
// (the latency of one wave of tiles; the last one waits for values and columns from anywhere), row pointer 10 us -- where a
// library sort, gathers, passes for the checks and an analysis took 210 us and two read-backs.
#include "fsb_common.cuh"

namespace fsb {

constexpr int kCooThreads = 256;
constexpr int kCooWarps = kCooThreads / 32;
constexpr int kCooMost = 16;                        // entries of a thread, at most
// Entries of a thread: 16, but 8 up to 3 M triples, which are fewer tiles of 4096 than the SMs hold at a time (us of all kernels with 8
// against 16: 1.3 M triples, four passes, 20 less; 64000, 10 less; 5.2 M, two passes, 3 % more).
static int coo_items(int64_t nnz) { return nnz <= 3 << 20 ? 8 : kCooMost; }
constexpr int kCooMaxBits = 9;                      // of a digit: 8 warps x 512 counters in shared memory
enum { C_PTR_FIRST = 0, C_PTR_LAST, C_DECREASING, C_MIN_COL, C_MAX_COL, C_MAX_ROW_NNZ, C_EMPTY, C_LONG, C_MIN_ROW, C_MAX_ROW, C_STATS };

// where the ids of a pass come from
template <typename T>
struct FromIds {                                    // first pass: the caller's array, in the caller's order
  const T* ids;
  __device__ __forceinline__ uint32_t id(int64_t i) const { return (uint32_t)ids[i]; }
  __device__ __forceinline__ uint32_t at(int64_t i) const { return (uint32_t)i; }
};
struct FromPairs {                                  // later passes over the same ids
  const uint32_t *ids, *order;
  __device__ __forceinline__ uint32_t id(int64_t i) const { return ids[i]; }
  __device__ __forceinline__ uint32_t at(int64_t i) const { return order[i]; }
};
template <typename T>
struct FromOrder {                                  // first pass over the row ids after the column ids
  const T* ids;
  const uint32_t* order;
  __device__ __forceinline__ uint32_t id(int64_t i) const { return (uint32_t)ids[order[i]]; }
  __device__ __forceinline__ uint32_t at(int64_t i) const { return order[i]; }
};

__global__ void coo_stats_init_kernel(int64_t* s, int64_t nnz) {
  s[C_PTR_FIRST] = 0;
  s[C_PTR_LAST] = nnz;
  s[C_DECREASING] = s[C_MAX_ROW_NNZ] = s[C_EMPTY] = s[C_LONG] = 0;
  s[C_MIN_COL] = s[C_MIN_ROW] = INT64_MAX;
  s[C_MAX_COL] = s[C_MAX_ROW] = INT64_MIN;
}

template <bool MAX>
__device__ __forceinline__ long long block_extreme(long long v, long long* s_part) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long u = __shfl_xor_sync(0xffffffffu, v, o);
    v = (MAX ? u > v : u < v) ? u : v;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = s_part[0];
#pragma unroll
  for (int w = 1; w < kCooWarps; ++w) v = (MAX ? s_part[w] > v : s_part[w] < v) ? s_part[w] : v;
  return v;
}

// counts[digit * n_tiles + tile]; RANGE: also the extremes of both id arrays
template <typename Src, typename R, typename C, bool RANGE, int kCooItems>
__global__ void __launch_bounds__(kCooThreads)
coo_count_kernel(Src src, int64_t nnz, int shift, int bits, int32_t* __restrict__ counts, const R* __restrict__ row,
                 const C* __restrict__ col, int64_t* __restrict__ stats) {
  constexpr int kCooTile = kCooThreads * kCooItems;
  extern __shared__ int32_t s_count[];
  __shared__ long long s_part[kCooWarps];
  const int n_digits = 1 << bits;
  for (int d = threadIdx.x; d < n_digits; d += kCooThreads) s_count[d] = 0;
  __syncthreads();
  const int64_t lo = (int64_t)blockIdx.x * kCooTile;
  uint32_t id[kCooItems];
#pragma unroll
  for (int k = 0; k < kCooItems; ++k) {
    const int64_t i = lo + k * kCooThreads + threadIdx.x;
    id[k] = i < nnz ? src.id(i) : 0u;
  }
#pragma unroll
  for (int k = 0; k < kCooItems; ++k)
    if (lo + k * kCooThreads + threadIdx.x < nnz) atomicAdd(&s_count[(id[k] >> shift) & (n_digits - 1)], 1);
  __syncthreads();
  for (int d = threadIdx.x; d < n_digits; d += kCooThreads) counts[(int64_t)d * gridDim.x + blockIdx.x] = s_count[d];
  if (RANGE) {
    long long r0 = INT64_MAX, r1 = INT64_MIN, c0 = INT64_MAX, c1 = INT64_MIN;
#pragma unroll
    for (int k = 0; k < kCooItems; ++k) {
      const int64_t i = lo + k * kCooThreads + threadIdx.x;
      if (i < nnz) {
        const long long r = (long long)row[i], c = (long long)col[i];
        r0 = r < r0 ? r : r0;
        r1 = r > r1 ? r : r1;
        c0 = c < c0 ? c : c0;
        c1 = c > c1 ? c : c1;
      }
    }
    r0 = block_extreme<false>(r0, s_part);
    r1 = block_extreme<true>(r1, s_part);
    c0 = block_extreme<false>(c0, s_part);
    c1 = block_extreme<true>(c1, s_part);
    if (threadIdx.x == 0) {
      atomicMin(reinterpret_cast<long long*>(stats + C_MIN_ROW), r0);
      atomicMax(reinterpret_cast<long long*>(stats + C_MAX_ROW), r1);
      atomicMin(reinterpret_cast<long long*>(stats + C_MIN_COL), c0);
      atomicMax(reinterpret_cast<long long*>(stats + C_MAX_COL), c1);
    }
  }
}

// inclusive scan over the CTA's threads
__device__ __forceinline__ int block_scan(int v, int* s_part) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  __syncthreads();
  if (lane == 31) s_part[w] = v;
  __syncthreads();
  for (int q = 0; q < w; ++q) v += s_part[q];
  return v;
}

// one CTA per digit: counts -> entries with this digit in earlier tiles; totals[digit]
__global__ void __launch_bounds__(kCooThreads) coo_scan_kernel(int32_t* __restrict__ counts, int n_tiles,
                                                               int32_t* __restrict__ totals) {
  __shared__ int s_part[kCooWarps];
  __shared__ int s_sum;
  int32_t* c = counts + (int64_t)blockIdx.x * n_tiles;
  int before = 0;
  for (int t0 = 0; t0 < n_tiles; t0 += kCooThreads) {
    const int t = t0 + threadIdx.x;
    const int v = t < n_tiles ? c[t] : 0;
    const int inc = block_scan(v, s_part);
    if (t < n_tiles) c[t] = before + inc - v;
    if (threadIdx.x == kCooThreads - 1) s_sum = inc;
    __syncthreads();
    before += s_sum;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = before;
}

template <int BYTES> struct CooValue;
template <> struct CooValue<2> { typedef unsigned short type; };
template <> struct CooValue<4> { typedef unsigned int type; };
template <> struct CooValue<8> { typedef uint2 type; };
template <> struct CooValue<16> { typedef uint4 type; };

// The move of one pass.  LAST: values and columns go to their final places, with the sorted row ids; else the pairs do.
template <typename Src, typename C, typename S, bool LAST, int kCooItems>
__global__ void __launch_bounds__(kCooThreads)
coo_move_kernel(Src src, int64_t nnz, int shift, int bits, const int32_t* __restrict__ counts,
                const int32_t* __restrict__ totals, uint32_t* __restrict__ out_ids, uint32_t* __restrict__ out_order,
                const S* __restrict__ data, const C* __restrict__ col, S* __restrict__ out_data, int32_t* __restrict__ out_col) {
  constexpr int kCooTile = kCooThreads * kCooItems;
  extern __shared__ int32_t s_raw[];
  const int n_digits = 1 << bits;
  int32_t* s_warp = s_raw;                            // [warp][digit]: entries of the warp, then of the warps before
  int32_t* s_to = s_warp + kCooWarps * n_digits;      // where a digit's run goes, less where it begins in the tile
  uint32_t* s_id = reinterpret_cast<uint32_t*>(s_to + n_digits);
  uint32_t* s_at = s_id + kCooTile;
  __shared__ int s_part[kCooWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int k = tid; k < kCooWarps * n_digits; k += kCooThreads) s_warp[k] = 0;
  __syncthreads();
  const int64_t lo = (int64_t)blockIdx.x * kCooTile;
  const int cnt = (int)((nnz - lo) < (int64_t)kCooTile ? (nnz - lo) : (int64_t)kCooTile);
  // a warp takes a stretch of its own, 32 consecutive entries at a time: (warp, step, lane) is the order of the entries
  uint32_t id[kCooItems], at[kCooItems];
  int rank[kCooItems];
#pragma unroll
  for (int k = 0; k < kCooItems; ++k) {
    const int i = warp * (32 * kCooItems) + k * 32 + lane;
    id[k] = i < cnt ? src.id(lo + i) : 0u;
    at[k] = i < cnt ? src.at(lo + i) : 0u;
  }
  int32_t* mine = s_warp + warp * n_digits;
#pragma unroll
  for (int k = 0; k < kCooItems; ++k) {
    const bool live = warp * (32 * kCooItems) + k * 32 + lane < cnt;
    const uint32_t d = (id[k] >> shift) & (n_digits - 1);
    // lanes with the same digit, a vote per bit (with __match_any_sync the first move of the triples above takes 31 us, with
    // votes 26 us)
    uint32_t peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
    for (int q = 0; q < kCooMaxBits; ++q) {
      if (q < bits) {
        const uint32_t vote = __ballot_sync(0xffffffffu, (d >> q) & 1);
        peers &= (d >> q) & 1 ? vote : ~vote;
      }
    }
    int first = 0;
    if (live) first = mine[d];
    __syncwarp();
    if (live && lane == __ffs(peers) - 1) mine[d] = first + __popc(peers);
    __syncwarp();
    rank[k] = first + __popc(peers & ((1u << lane) - 1u));
  }
  __syncthreads();
  // per digit: entries in the warps before; then the digits' runs in the tile, and their places
  int total_before = 0;                               // of all digits before this thread's, in the tile / in the output
  int out_before = 0;
  for (int d0 = 0; d0 < n_digits; d0 += kCooThreads) {
    const int d = d0 + tid;
    int in_tile = 0, in_all = 0;
    if (d < n_digits) {
#pragma unroll
      for (int w = 0; w < kCooWarps; ++w) {
        const int v = s_warp[w * n_digits + d];
        s_warp[w * n_digits + d] = in_tile;
        in_tile += v;
      }
      in_all = totals[d];
    }
    const int tile_inc = block_scan(in_tile, s_part), all_inc = block_scan(in_all, s_part);
    if (d < n_digits) {
      const int run = total_before + tile_inc - in_tile;
      s_to[d] = out_before + all_inc - in_all + counts[(int64_t)d * gridDim.x + blockIdx.x] - run;
#pragma unroll
      for (int w = 0; w < kCooWarps; ++w) s_warp[w * n_digits + d] += run;
    }
    __shared__ int s_sum[2];
    if (tid == kCooThreads - 1) {
      s_sum[0] = tile_inc;
      s_sum[1] = all_inc;
    }
    __syncthreads();
    total_before += s_sum[0];
    out_before += s_sum[1];
  }
#pragma unroll
  for (int k = 0; k < kCooItems; ++k) {
    if (warp * (32 * kCooItems) + k * 32 + lane < cnt) {
      const int p = mine[(id[k] >> shift) & (n_digits - 1)] + rank[k];
      s_id[p] = id[k];
      s_at[p] = at[k];
    }
  }
  __syncthreads();
  for (int p = tid; p < cnt; p += kCooThreads) {
    const uint32_t v = s_id[p], from = s_at[p];
    const int64_t to = (int64_t)s_to[(v >> shift) & (n_digits - 1)] + p;
    out_ids[to] = v;
    if (LAST) {
      out_data[to] = data[from];
      out_col[to] = (int32_t)col[from];
    } else {
      out_order[to] = from;
    }
  }
}

// ptr[r] = entries with a row id below r, by binary search; row lengths into the statistics
__global__ void __launch_bounds__(kCooThreads)
coo_pointer_kernel(const uint32_t* __restrict__ ids, int64_t nnz, int64_t n_rows, int64_t long_len, int32_t* __restrict__ ptr,
                   int64_t* __restrict__ stats) {
  __shared__ int32_t s_ptr[kCooThreads + 1];
  __shared__ long long s_part[kCooWarps];
  const int64_t r0 = (int64_t)blockIdx.x * kCooThreads;
  for (int k = threadIdx.x; k <= kCooThreads; k += kCooThreads) {
    const int64_t r = r0 + k;
    if (r > n_rows) break;
    int64_t lo = 0, hi = nnz;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if ((int64_t)ids[mid] < r) lo = mid + 1; else hi = mid;
    }
    s_ptr[k] = (int32_t)lo;
    if (k < kCooThreads || r == n_rows) ptr[r] = (int32_t)lo;
  }
  __syncthreads();
  const bool live = r0 + threadIdx.x < n_rows;
  const int len = live ? s_ptr[threadIdx.x + 1] - s_ptr[threadIdx.x] : 0;
  const int empty = __syncthreads_count(live && len == 0), lng = __syncthreads_count(live && len > long_len);
  const long long longest = block_extreme<true>(len, s_part);
  if (threadIdx.x == 0) {
    if (longest > 0) atomicMax(reinterpret_cast<long long*>(stats + C_MAX_ROW_NNZ), longest);
    if (empty) atomicAdd(reinterpret_cast<unsigned long long*>(stats + C_EMPTY), (unsigned long long)empty);
    if (lng) atomicAdd(reinterpret_cast<unsigned long long*>(stats + C_LONG), (unsigned long long)lng);
  }
}

static int id_bits(int64_t n) {      // of the ids 0 .. n - 1, at least one
  int b = 1;
  while (b < 32 && ((int64_t)1 << b) < n) ++b;
  return b;
}

struct CooScratch {
  uint32_t *ids[2], *order[2];
  int32_t *counts, *totals;
  size_t bytes;
};
static CooScratch coo_scratch(void* base, int64_t nnz) {
  const int64_t tile = (int64_t)kCooThreads * coo_items(nnz), n_tiles = (nnz + tile - 1) / tile;
  const size_t col = (((size_t)nnz * 4) + 255) & ~(size_t)255;
  char* p = (char*)base;
  CooScratch s;
  for (int k = 0; k < 2; ++k) {
    s.ids[k] = (uint32_t*)(p + k * col);
    s.order[k] = (uint32_t*)(p + (2 + k) * col);
  }
  s.counts = (int32_t*)(p + 4 * col);
  const size_t cells = (((size_t)n_tiles << kCooMaxBits) * 4 + 255) & ~(size_t)255;
  s.totals = (int32_t*)(p + 4 * col + cells);
  s.bytes = 4 * col + cells + ((size_t)4 << kCooMaxBits);
  return s;
}

struct CooArgs {
  const void *data, *row, *col;
  int64_t nnz, n_rows, n_cols;
  bool by_column;
  void* out_data;
  int32_t *out_row, *out_col, *ptr;
  int64_t* stats;
  CooScratch s;
  cudaStream_t st;
};

struct Yes { static constexpr bool value = true; };
struct No { static constexpr bool value = false; };

template <typename R, typename C, typename S, int kCooItems>
static int coo_passes(const CooArgs& a) {
  constexpr int kCooTile = kCooThreads * kCooItems;
  const int64_t n_tiles = (a.nnz + kCooTile - 1) / kCooTile;
  const R* row = (const R*)a.row;
  const C* col = (const C*)a.col;
  const int bits[2] = {a.by_column ? id_bits(a.n_cols) : 0, id_bits(a.n_rows)};
  int side = 0;                       // where the pairs of the last pass are
  bool first = true;
  cudaError_t e;
  for (int key = a.by_column ? 0 : 1; key < 2; ++key) {
    const int passes = (bits[key] + kCooMaxBits - 1) / kCooMaxBits;
    const int width = (bits[key] + passes - 1) / passes;
    for (int p = 0; p < passes; ++p) {
      const int shift = p * width;
      const size_t count_smem = (size_t)4 << width;
      const size_t move_smem = ((size_t)4 << width) * (kCooWarps + 1) + (size_t)kCooTile * 8;
      const bool last = key == 1 && p == passes - 1;
      uint32_t* ids = last ? (uint32_t*)a.out_row : a.s.ids[side ^ 1];
      auto pass = [&](auto src, auto range) -> int {
        typedef decltype(src) Src;
        coo_count_kernel<Src, R, C, decltype(range)::value, kCooItems><<<(unsigned)n_tiles, kCooThreads, count_smem, a.st>>>(
            src, a.nnz, shift, width, a.s.counts, row, col, a.stats);
        FSB_RETURN_IF_LAUNCH_FAILED();
        coo_scan_kernel<<<1u << width, kCooThreads, 0, a.st>>>(a.s.counts, (int)n_tiles, a.s.totals);
        FSB_RETURN_IF_LAUNCH_FAILED();
#define FSB_COO_MOVE(LAST_)                                                                                             \
  e = cudaFuncSetAttribute(coo_move_kernel<Src, C, S, LAST_, kCooItems>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);  \
  if (e != cudaSuccess) return cuda_rc(e);                                                                              \
  coo_move_kernel<Src, C, S, LAST_, kCooItems><<<(unsigned)n_tiles, kCooThreads, move_smem, a.st>>>(                               \
      src, a.nnz, shift, width, a.s.counts, a.s.totals, ids, a.s.order[side ^ 1], (const S*)a.data, col, (S*)a.out_data, \
      a.out_col)
        if (last) {
          FSB_COO_MOVE(true);
        } else {
          FSB_COO_MOVE(false);
        }
#undef FSB_COO_MOVE
        FSB_RETURN_IF_LAUNCH_FAILED();
        return FSB_OK;
      };
      int rc;
      if (first && key == 0) rc = pass(FromIds<C>{col}, Yes());
      else if (first) rc = pass(FromIds<R>{row}, Yes());
      else if (p == 0) rc = pass(FromOrder<R>{row, a.s.order[side]}, No());
      else rc = pass(FromPairs{a.s.ids[side], a.s.order[side]}, No());
      if (rc != FSB_OK) return rc;
      first = false;
      side ^= 1;
    }
  }
  return FSB_OK;
}

template <typename R, typename C, typename S>
static int coo_run(const CooArgs& a) {
  return coo_items(a.nnz) == 8 ? coo_passes<R, C, S, 8>(a) : coo_passes<R, C, S, kCooMost>(a);
}

}  // namespace fsb

using namespace fsb;

extern "C" size_t fsb_coo_scratch_bytes(int64_t nnz) { return nnz > 0 ? coo_scratch(nullptr, nnz).bytes : 0; }

extern "C" int fsb_coo_group(int value_bytes, int rtype, int ctype, const void* data, const void* row, const void* col,
                             int64_t nnz, int64_t n_rows, int64_t n_cols, int by_column, void* out_data, int32_t* out_row,
                             int32_t* out_col, int32_t* indptr, int64_t* stats, void* scratch, size_t scratch_bytes,
                             void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  if ((rtype != FSB_I32 && rtype != FSB_I64) || (ctype != FSB_I32 && ctype != FSB_I64)) return FSB_EINVAL;
  if (value_bytes != 2 && value_bytes != 4 && value_bytes != 8 && value_bytes != 16) return FSB_EINVAL;
  if (nnz <= 0 || n_rows < 0 || n_cols < 0) return FSB_EINVAL;
  if (nnz > INT32_MAX - kCooThreads * kCooMost || n_rows >= INT32_MAX || n_cols >= INT32_MAX) return FSB_ERANGE;
  if (!data || !row || !col || !out_data || !out_row || !out_col || !indptr || !stats || !scratch) return FSB_EINVAL;
  if (!aligned_to(data, value_bytes) || !aligned_to(out_data, value_bytes) || !aligned_to(row, rtype == FSB_I32 ? 4 : 8) ||
      !aligned_to(col, ctype == FSB_I32 ? 4 : 8) || !aligned_to(stats, 8) || !aligned_to(scratch, 16))
    return FSB_EALIGN;
  CooArgs a{data, row, col, nnz, n_rows, n_cols, by_column != 0, out_data, out_row, out_col, indptr, stats,
            coo_scratch(scratch, nnz), st};
  if (scratch_bytes < a.s.bytes) return FSB_ESCRATCH;
  coo_stats_init_kernel<<<1, 1, 0, st>>>(stats, nnz);
  FSB_RETURN_IF_LAUNCH_FAILED();
#define FSB_COO_IDS(S_)                                                                                        \
  (rtype == FSB_I32 ? (ctype == FSB_I32 ? coo_run<int32_t, int32_t, S_>(a) : coo_run<int32_t, int64_t, S_>(a)) \
                    : (ctype == FSB_I32 ? coo_run<int64_t, int32_t, S_>(a) : coo_run<int64_t, int64_t, S_>(a)))
  int rc;
  switch (value_bytes) {
    case 2: rc = FSB_COO_IDS(CooValue<2>::type); break;
    case 4: rc = FSB_COO_IDS(CooValue<4>::type); break;
    case 8: rc = FSB_COO_IDS(CooValue<8>::type); break;
    default: rc = FSB_COO_IDS(CooValue<16>::type); break;
  }
#undef FSB_COO_IDS
  if (rc != FSB_OK) return rc;
  // "long" as in fsb_csr_analyze
  const int64_t mean_up = n_rows > 0 ? (nnz + n_rows - 1) / n_rows : 0;
  const int64_t long_len = mean_up * 32 < 64 ? 64 : mean_up * 32;
  const int64_t blocks = n_rows / kCooThreads + 1;
  coo_pointer_kernel<<<(unsigned)blocks, kCooThreads, 0, st>>>((const uint32_t*)out_row, nnz, n_rows, long_len, indptr, stats);
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}
