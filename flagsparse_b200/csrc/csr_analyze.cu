// CSR structure analysis (one pass over indptr, one over indices) and the nnz-tile plan.
#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include <atomic>

#include "fsb_common.cuh"

namespace fsb {

constexpr int kCheckTicket = 8;      // behind the eight statistics in host memory
enum { S_PTR_FIRST = 0, S_PTR_LAST, S_DECREASING, S_MIN_IDX, S_MAX_IDX, S_MAX_ROW, S_EMPTY, S_LONG };

__global__ void stats_init_kernel(int64_t* s) {
  s[S_PTR_FIRST] = 0;
  s[S_PTR_LAST] = 0;
  s[S_DECREASING] = 0;
  s[S_MIN_IDX] = INT64_MAX;
  s[S_MAX_IDX] = INT64_MIN;
  s[S_MAX_ROW] = 0;
  s[S_EMPTY] = 0;
  s[S_LONG] = 0;
}

// (one instruction where all lanes hold 32-bit numbers, which is nearly always)
__device__ __forceinline__ long long warp_max(long long v) {
  if (__all_sync(0xffffffffu, v == (int)v)) return __reduce_max_sync(0xffffffffu, (int)v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    long long u = __shfl_xor_sync(0xffffffffu, v, o);
    v = u > v ? u : v;
  }
  return v;
}
__device__ __forceinline__ long long warp_min(long long v) {
  if (__all_sync(0xffffffffu, v == (int)v)) return __reduce_min_sync(0xffffffffu, (int)v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    long long u = __shfl_xor_sync(0xffffffffu, v, o);
    v = u < v ? u : v;
  }
  return v;
}
// One pass over the row pointer and one over the indices, grid-stride, in one launch.  Aligned indices are read at 16 bytes
// per thread and request; the statistics meet in shared memory, so that a block sends one atomic per statistic: one per warp, on six
// words that every block of the device shares, used to take longer than the reading (3 M entries,
// 250007 rows, 64-bit: two launches, 33 us; 10 us in this one; 2.1 M entries, 150001 rows: 30 us and 7 us).
// Thread k < 6 of a block returns what the block found: longest row, decreasing and empty rows, long rows, smallest and largest index.
template <typename I, typename P>
__device__ __forceinline__ long long csr_stats_block(const P* __restrict__ ptr, int64_t n_rows, int64_t long_len,
                                                     const I* __restrict__ idx, int64_t nnz, int wide_loads) {
  constexpr int E = 16 / (int)sizeof(I);
  constexpr int U = 4;                       // requests in flight
  __shared__ long long s_part[8][6];
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // the rows first: their loads are on their way while the indices are looked at
  long long longest = 0;
  unsigned n_dec = 0, n_empty = 0, n_long = 0;         // (of one thread, fewer than 2^32 / 32)
  for (int64_t i = first; i < n_rows; i += stride) {
    const long long len = (long long)ptr[i + 1] - (long long)ptr[i];
    longest = len > longest ? len : longest;
    n_dec += len < 0;
    n_empty += len == 0;
    n_long += len > long_len;
  }
  I mn = sizeof(I) == 4 ? (I)INT32_MAX : (I)INT64_MAX, mx = sizeof(I) == 4 ? (I)INT32_MIN : (I)INT64_MIN;
  int64_t done = 0;
  if (wide_loads) {
    const int64_t groups = nnz / E;
    const int4* src = reinterpret_cast<const int4*>(idx);
    for (int64_t i = first; i < groups; i += U * stride) {
      int4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = __ldg(src + (i + u * stride < groups ? i + u * stride : i));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const I* c = reinterpret_cast<const I*>(&v[u]);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          mn = c[e] < mn ? c[e] : mn;
          mx = c[e] > mx ? c[e] : mx;
        }
      }
    }
    done = groups * E;
  }
  for (int64_t i = done + first; i < nnz; i += stride) {
    const I c = idx[i];
    mn = c < mn ? c : mn;
    mx = c > mx ? c : mx;
  }
  const bool any = nnz > 0;                  // a thread without an entry holds the neutral values of I, not of int64
  const long long wide_mn = (!any || mn > mx) ? (long long)INT64_MAX : (long long)mn;
  const long long wide_mx = (!any || mn > mx) ? (long long)INT64_MIN : (long long)mx;
  longest = warp_max(longest);
  const long long dec = __reduce_add_sync(0xffffffffu, n_dec), empty = __reduce_add_sync(0xffffffffu, n_empty),
                  lng = __reduce_add_sync(0xffffffffu, n_long);
  const long long low = warp_min(wide_mn), high = warp_max(wide_mx);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_part[w][0] = longest; s_part[w][1] = dec; s_part[w][2] = empty; s_part[w][3] = lng;
    s_part[w][4] = low; s_part[w][5] = high;
  }
  __syncthreads();
  long long v = 0;
  if (threadIdx.x < 6) {
    const int k = threadIdx.x;
    v = s_part[0][k];
#pragma unroll
    for (int j = 1; j < 8; ++j) {
      const long long u = s_part[j][k];
      if (k == 0 || k == 5) v = u > v ? u : v;
      else if (k == 4) v = u < v ? u : v;
      else v += u;
    }
  }
  return v;
}

template <typename I, typename P>
__global__ void __launch_bounds__(256)
csr_stats_kernel(const P* __restrict__ ptr, int64_t n_rows, int64_t long_len, const I* __restrict__ idx, int64_t nnz,
                 int wide_loads, int64_t* __restrict__ s) {
  const long long v = csr_stats_block<I, P>(ptr, n_rows, long_len, idx, nnz, wide_loads);
  const int k = threadIdx.x;
  if (k == 0 && v > 0) atomicMax(reinterpret_cast<long long*>(s + S_MAX_ROW), v);
  if (k >= 1 && k <= 3 && v != 0)
    atomicAdd(reinterpret_cast<unsigned long long*>(s + (k == 1 ? S_DECREASING : k == 2 ? S_EMPTY : S_LONG)),
              (unsigned long long)v);
  if (k == 4 && v != INT64_MAX) atomicMin(reinterpret_cast<long long*>(s + S_MIN_IDX), v);
  if (k == 5 && v != INT64_MIN) atomicMax(reinterpret_cast<long long*>(s + S_MAX_IDX), v);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s[S_PTR_FIRST] = (int64_t)ptr[0];
    s[S_PTR_LAST] = (int64_t)ptr[n_rows];
  }
}

// The same for a host that waits: the block that ends last writes the eight numbers to host memory (`out`, page-locked), then
// `ticket` behind them, and leaves `work` zero, as it was found.  No launch to set up, no copy, no wait for the whole stream
// (250007 rows, 3 M entries with 64-bit indices: 10.7 us; set-up, csr_stats_kernel and copy were 13.5 us on the GPU, but the host's
// part of them and of the wait made a whole product of these arrays 62 us, 33 us now; 4096 rows of 16, 32 columns of B: 75 and 34).
// work: 0 longest, 1 to 3 counts, 4 and 5 the extreme indices in an order that has zero for none, 6 blocks that are done.
constexpr unsigned long long kSignBit = 1ull << 63;
template <typename I, typename P>
__global__ void __launch_bounds__(256)
csr_check_kernel(const P* __restrict__ ptr, int64_t n_rows, int64_t long_len, const I* __restrict__ idx, int64_t nnz,
                 int wide_loads, unsigned long long* __restrict__ work, volatile int64_t* out, int64_t ticket) {
  int64_t ptr_first = 0, ptr_last = 0;      // (asked for early: whichever block is the last one has them by then)
  if (threadIdx.x == 0) {
    ptr_first = (int64_t)ptr[0];
    ptr_last = (int64_t)ptr[n_rows];
  }
  const long long v = csr_stats_block<I, P>(ptr, n_rows, long_len, idx, nnz, wide_loads);
  const int k = threadIdx.x;
  if (k < 6) {
    const unsigned long long bits = (unsigned long long)v;
    if (k >= 1 && k <= 3) {
      if (v != 0) atomicAdd(work + k, bits);
    } else {
      const unsigned long long w = k == 0 ? (v > 0 ? bits : 0) : k == 4 ? ~(bits ^ kSignBit) : bits ^ kSignBit;
      if (w != 0) atomicMax(work + k, w);
    }
    __threadfence();
  }
  __syncthreads();
  if (k != 0) return;
  if (atomicAdd(work + 6, 1ull) != gridDim.x - 1) return;
  __threadfence();
  unsigned long long w[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) w[j] = atomicExch(work + j, 0ull);
  atomicExch(work + 6, 0ull);
  out[S_PTR_FIRST] = ptr_first;
  out[S_PTR_LAST] = ptr_last;
  out[S_DECREASING] = (int64_t)w[1];
  out[S_MIN_IDX] = (int64_t)(~w[4] ^ kSignBit);
  out[S_MAX_IDX] = (int64_t)(w[5] ^ kSignBit);
  out[S_MAX_ROW] = (int64_t)w[0];
  out[S_EMPTY] = (int64_t)w[2];
  out[S_LONG] = (int64_t)w[3];
  __threadfence_system();
  out[kCheckTicket] = ticket;
}

// tile_row[t] = (first j with ptr[j] > t*T) - 1, i.e. the row that holds nnz number t*T
template <typename P>
__global__ void __launch_bounds__(256) tile_plan_kernel(const P* __restrict__ ptr, int64_t n_rows,
                                                       int64_t n_tiles, int64_t tile_nnz,
                                                       int32_t* __restrict__ tile_row) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t > n_tiles) return;
  if (t == 0) { tile_row[0] = 0; return; }
  if (t == n_tiles) { tile_row[t] = (int32_t)n_rows; return; }
  const long long v = (long long)t * tile_nnz;
  int64_t lo = 0, hi = n_rows + 1;  // search over ptr[0..n_rows]; ptr[0] = 0 <= v, ptr[n_rows] = nnz > v
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if ((long long)ptr[mid] > v) hi = mid; else lo = mid + 1;
  }
  tile_row[t] = (int32_t)(lo - 1);
}

static int grid_for(int64_t n, int threads, int cap) {
  int64_t g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

static int stats_check_args(int itype, int ptype, const void* indices, const void* indptr, int64_t n_rows, int64_t nnz) {
  if ((itype != FSB_I32 && itype != FSB_I64) || (ptype != FSB_I32 && ptype != FSB_I64)) return FSB_EINVAL;
  if (n_rows < 0 || nnz < 0 || indptr == nullptr) return FSB_EINVAL;
  if (nnz > 0 && indices == nullptr) return FSB_EINVAL;
  if (!aligned_to(indptr, ptype == FSB_I32 ? 4 : 8) || !aligned_to(indices, itype == FSB_I32 ? 4 : 8)) return FSB_EALIGN;
  if (n_rows >= INT32_MAX) return FSB_ERANGE;
  return FSB_OK;
}
// "long" = more than 32x the mean row length (at least 64)
static int64_t stats_long_len(int64_t n_rows, int64_t nnz) {
  const int64_t mean_up = n_rows > 0 ? (nnz + n_rows - 1) / n_rows : 0;
  return mean_up * 32 < 64 ? 64 : mean_up * 32;
}
static int stats_grid(int itype, int64_t n_rows, int64_t nnz) {
  const int64_t per_thread = itype == FSB_I32 ? 16 : 8;      // four requests
  const int64_t rows_blocks = (n_rows + 1023) / 1024, idx_blocks = (nnz + 256 * per_thread - 1) / (256 * per_thread);
  return grid_for((rows_blocks > idx_blocks ? rows_blocks : idx_blocks) * 256, 256, 148 * 4);   // (8 an SM: 13.3 us, 4: 10.7)
}

int csr_check_launch(int itype, int ptype, const void* indices, const void* indptr, int64_t n_rows, int64_t nnz, void* work,
                     int64_t* host, cudaStream_t stream) {
  const int rc = stats_check_args(itype, ptype, indices, indptr, n_rows, nnz);
  if (rc != FSB_OK) return rc;
  if (work == nullptr || host == nullptr) return FSB_EINVAL;
  if (!aligned_to(work, 8) || !aligned_to(host, 8)) return FSB_EALIGN;
  // counted here, not from what the GPU wrote last: no two calls wait for the same number, however the earlier one ended
  const int64_t ticket = ++host[kCheckTicket + 1];
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(stream, &capturing);
  if (e != cudaSuccess) return cuda_rc(e);
  if (capturing != cudaStreamCaptureStatusNone) return FSB_CAPTURING;        // nothing would run before the wait
  const int wide_loads = nnz > 0 && aligned_to(indices, 16);
#define FSB_CHECK_CSR(I_, P_)                                                                                        \
  csr_check_kernel<I_, P_><<<stats_grid(itype, n_rows, nnz), 256, 0, stream>>>(                                      \
      (const P_*)indptr, n_rows, stats_long_len(n_rows, nnz), (const I_*)indices, nnz, wide_loads,                   \
      (unsigned long long*)work, host, ticket)
  if (itype == FSB_I32) {
    if (ptype == FSB_I32) FSB_CHECK_CSR(int32_t, int32_t); else FSB_CHECK_CSR(int32_t, int64_t);
  } else {
    if (ptype == FSB_I32) FSB_CHECK_CSR(int64_t, int32_t); else FSB_CHECK_CSR(int64_t, int64_t);
  }
#undef FSB_CHECK_CSR
  e = cudaGetLastError();
  if (e == cudaSuccess) return FSB_OK;
  // an older error of this thread may be what is reported, with the kernel on its way: `work` and `host` are the caller's again
  // only when it has ended
  const int rc_launch = cuda_rc(e);
  (void)cuda_rc(cudaStreamSynchronize(stream));
  return rc_launch;
}

int csr_check_wait(const int64_t* host, cudaStream_t stream) {
  const volatile int64_t* seen = host + kCheckTicket;
  const int64_t ticket = host[kCheckTicket + 1];
  for (int i = 0; i < (1 << 18) && *seen != ticket; ++i) {     // about 10 ms
#if defined(__x86_64__)
    _mm_pause();
#endif
  }
  if (*seen != ticket) {               // a long queue in front of it, or a failure: the runtime tells
    const cudaError_t e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_rc(e);
    if (*seen != ticket) return FSB_CUDA_ERROR_BASE + (int)cudaErrorUnknown;
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return FSB_OK;
}

bool csr_check_passed(const int64_t* host, int64_t n_cols, int64_t nnz) {
  return host[S_PTR_FIRST] == 0 && host[S_PTR_LAST] == nnz && host[S_DECREASING] == 0 &&
         (nnz == 0 || (host[S_MIN_IDX] >= 0 && host[S_MAX_IDX] < n_cols));
}
int64_t csr_check_longest(const int64_t* host) { return host[S_MAX_ROW]; }

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_version(void) { return FSB_VERSION; }

extern "C" int fsb_csr_analyze(int itype, int ptype, const void* indices, const void* indptr,
                               int64_t n_rows, int64_t nnz, int64_t* stats, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int rc = stats_check_args(itype, ptype, indices, indptr, n_rows, nnz);
  if (rc != FSB_OK) return rc;
  if (stats == nullptr) return FSB_EINVAL;
  if (!aligned_to(stats, 8)) return FSB_EALIGN;
  stats_init_kernel<<<1, 1, 0, stream>>>(stats);
  FSB_RETURN_IF_LAUNCH_FAILED();
  const int64_t long_len = stats_long_len(n_rows, nnz);
  const int wide_loads = nnz > 0 && aligned_to(indices, 16);
  const int g = stats_grid(itype, n_rows, nnz);
#define FSB_STATS(I_, P_)                                                                                           \
  csr_stats_kernel<I_, P_><<<g, 256, 0, stream>>>((const P_*)indptr, n_rows, long_len, (const I_*)indices, nnz,     \
                                                  wide_loads, stats)
  if (itype == FSB_I32) {
    if (ptype == FSB_I32) FSB_STATS(int32_t, int32_t); else FSB_STATS(int32_t, int64_t);
  } else {
    if (ptype == FSB_I32) FSB_STATS(int64_t, int32_t); else FSB_STATS(int64_t, int64_t);
  }
#undef FSB_STATS
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

extern "C" int fsb_csr_check(int itype, int ptype, const void* indices, const void* indptr, int64_t n_rows, int64_t nnz, void* work,
                             int64_t* host, void* stream_) {
  const cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int rc = csr_check_launch(itype, ptype, indices, indptr, n_rows, nnz, work, host, stream);
  return rc != FSB_OK ? rc : csr_check_wait(host, stream);
}

extern "C" int64_t fsb_csr_num_tiles(int64_t nnz, int tile_nnz) {
  if (nnz <= 0 || tile_nnz <= 0) return 0;
  return (nnz + tile_nnz - 1) / tile_nnz;
}

extern "C" int fsb_csr_tile_plan(int ptype, const void* indptr, int64_t n_rows, int64_t nnz, int tile_nnz,
                                 int32_t* tile_row, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (ptype != FSB_I32 && ptype != FSB_I64) return FSB_EINVAL;
  if (n_rows < 0 || nnz < 0 || tile_nnz <= 0 || (tile_nnz & (tile_nnz - 1)) != 0) return FSB_EINVAL;
  if (indptr == nullptr || tile_row == nullptr) return FSB_EINVAL;
  if (!aligned_to(indptr, ptype == FSB_I32 ? 4 : 8) || !aligned_to(tile_row, 4)) return FSB_EALIGN;
  if (n_rows >= INT32_MAX) return FSB_ERANGE;
  const int64_t n_tiles = fsb_csr_num_tiles(nnz, tile_nnz);
  if (n_tiles >= INT32_MAX) return FSB_ERANGE;
  const int64_t n = n_tiles + 1;
  const int g = (int)((n + 255) / 256);
  if (ptype == FSB_I32)
    tile_plan_kernel<int32_t><<<g, 256, 0, stream>>>((const int32_t*)indptr, n_rows, n_tiles, tile_nnz, tile_row);
  else
    tile_plan_kernel<int64_t><<<g, 256, 0, stream>>>((const int64_t*)indptr, n_rows, n_tiles, tile_nnz, tile_row);
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}
