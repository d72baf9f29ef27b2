// CSR structure analysis (one pass over indptr, one over indices) and the nnz-tile plan.
#include "fsb_common.cuh"

namespace fsb {

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

__device__ __forceinline__ long long warp_max(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    long long u = __shfl_xor_sync(0xffffffffu, v, o);
    v = u > v ? u : v;
  }
  return v;
}
__device__ __forceinline__ long long warp_min(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    long long u = __shfl_xor_sync(0xffffffffu, v, o);
    v = u < v ? u : v;
  }
  return v;
}
__device__ __forceinline__ long long warp_sum(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One pass over the row pointer and one over the indices, grid-stride, in one launch.  Aligned indices are read at 16 bytes
// per thread and request; the statistics meet in shared memory, so that a block sends one atomic per statistic: one per warp, on six
// words that every block of the device shares, used to take longer than the reading (3 M entries,
// 250007 rows, 64-bit: two launches, 33 us; 10 us in this one; 2.1 M entries, 150001 rows: 30 us and 7 us).
template <typename I, typename P>
__global__ void __launch_bounds__(256)
csr_stats_kernel(const P* __restrict__ ptr, int64_t n_rows, int64_t long_len, const I* __restrict__ idx, int64_t nnz,
                 int wide_loads, int64_t* __restrict__ s) {
  constexpr int E = 16 / (int)sizeof(I);
  constexpr int U = 4;                       // requests in flight
  __shared__ long long s_part[8][6];
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
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
  long long longest = 0, dec = 0, empty = 0, lng = 0;
  for (int64_t i = first; i < n_rows; i += stride) {
    const long long len = (long long)ptr[i + 1] - (long long)ptr[i];
    longest = len > longest ? len : longest;
    dec += len < 0;
    empty += len == 0;
    lng += len > long_len;
  }
  const bool any = nnz > 0;                  // a thread without an entry holds the neutral values of I, not of int64
  long long wide_mn = (!any || mn > mx) ? (long long)INT64_MAX : (long long)mn;
  long long wide_mx = (!any || mn > mx) ? (long long)INT64_MIN : (long long)mx;
  longest = warp_max(longest);
  dec = warp_sum(dec);
  empty = warp_sum(empty);
  lng = warp_sum(lng);
  wide_mn = warp_min(wide_mn);
  wide_mx = warp_max(wide_mx);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_part[w][0] = longest; s_part[w][1] = dec; s_part[w][2] = empty; s_part[w][3] = lng;
    s_part[w][4] = wide_mn; s_part[w][5] = wide_mx;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    const int k = threadIdx.x;
    long long v = s_part[0][k];
#pragma unroll
    for (int j = 1; j < 8; ++j) {
      const long long u = s_part[j][k];
      if (k == 0 || k == 5) v = u > v ? u : v;
      else if (k == 4) v = u < v ? u : v;
      else v += u;
    }
    if (k == 0 && v > 0) atomicMax(reinterpret_cast<long long*>(s + S_MAX_ROW), v);
    if (k >= 1 && k <= 3 && v != 0)
      atomicAdd(reinterpret_cast<unsigned long long*>(s + (k == 1 ? S_DECREASING : k == 2 ? S_EMPTY : S_LONG)),
                (unsigned long long)v);
    if (k == 4 && v != INT64_MAX) atomicMin(reinterpret_cast<long long*>(s + S_MIN_IDX), v);
    if (k == 5 && v != INT64_MIN) atomicMax(reinterpret_cast<long long*>(s + S_MAX_IDX), v);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s[S_PTR_FIRST] = (int64_t)ptr[0];
    s[S_PTR_LAST] = (int64_t)ptr[n_rows];
  }
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

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_version(void) { return FSB_VERSION; }

extern "C" int fsb_csr_analyze(int itype, int ptype, const void* indices, const void* indptr,
                               int64_t n_rows, int64_t nnz, int64_t* stats, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if ((itype != FSB_I32 && itype != FSB_I64) || (ptype != FSB_I32 && ptype != FSB_I64)) return FSB_EINVAL;
  if (n_rows < 0 || nnz < 0 || stats == nullptr || indptr == nullptr) return FSB_EINVAL;
  if (nnz > 0 && indices == nullptr) return FSB_EINVAL;
  if (!aligned_to(indptr, ptype == FSB_I32 ? 4 : 8) || !aligned_to(indices, itype == FSB_I32 ? 4 : 8) ||
      !aligned_to(stats, 8))
    return FSB_EALIGN;
  if (n_rows >= INT32_MAX) return FSB_ERANGE;
  stats_init_kernel<<<1, 1, 0, stream>>>(stats);
  FSB_RETURN_IF_LAUNCH_FAILED();
  // "long" = more than 32x the mean row length (at least 64)
  int64_t mean_up = n_rows > 0 ? (nnz + n_rows - 1) / n_rows : 0;
  int64_t long_len = mean_up * 32 < 64 ? 64 : mean_up * 32;
  const int wide_loads = nnz > 0 && aligned_to(indices, 16);
  const int64_t per_thread = itype == FSB_I32 ? 16 : 8;      // four requests
  const int64_t rows_blocks = (n_rows + 1023) / 1024, idx_blocks = (nnz + 256 * per_thread - 1) / (256 * per_thread);
  const int g = grid_for((rows_blocks > idx_blocks ? rows_blocks : idx_blocks) * 256, 256, 148 * 8);
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
