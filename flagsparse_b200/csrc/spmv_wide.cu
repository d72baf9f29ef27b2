// CSR SpMV and SpMM for the value types the float32 / float64 kernels do not stream themselves: float16 and bfloat16
// values (2 bytes per entry in memory, products and sums in float32) and complex64 / complex128 values (interleaved real
// and imaginary parts, one pass over the matrix, complex multiply-add in the component precision).  The values are read
// as they are stored -- no widened or split copy of the matrix exists anywhere.  Rows are summed in a fixed order:
// bit-reproducible.
//
// fsb_spmv_csr_stored (second half of this file): x and y in the matrix's own type too; lanes per row for even rows, tiles
// for uneven ones.  SpMM with operands as stored runs through the tiled kernel of spmm_csr.cu.
//
// fsb_spmv_csr_wide / fsb_spmm_csr_wide: one launch without scratch, dense operand and result in float32 for the half
// precisions (the caller widens x / B once per call and rounds y / C once, as the reference's base path does).  SpMV: L
// lanes per row (L = 2 .. 32 from the mean row length), every lane walks the row with stride L, two partial sums, a
// shuffle tree, lane 0 stores.  SpMM: a group of LN lanes per row (LN = dense width rounded up to a power of two, at most
// 32; wider B in column tiles of 32 along gridDim.y), every lane owns one column of C, walks the row's entries (value and
// column index are the same address for the whole group: one broadcast load) and gathers its element of B's row, two
// entries in flight.
#include <string.h>

#include "fsb_common.cuh"
#include "spmv_rows.cuh"
#include "stored_ops.cuh"

namespace fsb {

constexpr int kWideThreads = 256;

// How one stored value type is computed with: accumulator type, element type of x and y, multiply-add, shuffle.
template <typename S>
struct WideOps;

template <>
struct WideOps<__half> {
  typedef float Acc;
  typedef float Dense;
  static __device__ __forceinline__ void fma(Acc& acc, __half a, Dense b) { acc = fmaf(__half2float(a), b, acc); }
};
template <>
struct WideOps<__nv_bfloat16> {
  typedef float Acc;
  typedef float Dense;
  static __device__ __forceinline__ void fma(Acc& acc, __nv_bfloat16 a, Dense b) {
    acc = fmaf(__bfloat162float(a), b, acc);
  }
};
template <>
struct WideOps<float2> {
  typedef float2 Acc;
  typedef float2 Dense;
  static __device__ __forceinline__ void fma(Acc& acc, float2 a, Dense b) {
    acc.x += a.x * b.x - a.y * b.y;
    acc.y += a.x * b.y + a.y * b.x;
  }
};
template <>
struct WideOps<double2> {
  typedef double2 Acc;
  typedef double2 Dense;
  static __device__ __forceinline__ void fma(Acc& acc, double2 a, Dense b) {
    acc.x += a.x * b.x - a.y * b.y;
    acc.y += a.x * b.y + a.y * b.x;
  }
};

template <typename S, typename P, int L>
__global__ void __launch_bounds__(kWideThreads)
spmv_wide_kernel(const S* __restrict__ data, const int32_t* __restrict__ idx, const P* __restrict__ ptr,
                 const typename WideOps<S>::Dense* __restrict__ x, typename WideOps<S>::Dense* __restrict__ y,
                 int64_t n_rows) {
  typedef typename WideOps<S>::Acc A;
  const int64_t gtid = (int64_t)blockIdx.x * kWideThreads + threadIdx.x;
  const int64_t row = gtid / L;
  const int lane = (int)(gtid % L);
  int64_t s = 0, e = 0;
  if (row < n_rows) {
    s = (int64_t)ptr[row];
    e = (int64_t)ptr[row + 1];
  }
  A acc0 = w_zero((A*)nullptr), acc1 = w_zero((A*)nullptr);
  int64_t p = s + lane;
  for (; p + L < e; p += 2 * L) {
    const S a0 = __ldcs(data + p), a1 = __ldcs(data + p + L);
    const int64_t c0 = (int64_t)__ldcs(idx + p), c1 = (int64_t)__ldcs(idx + p + L);
    WideOps<S>::fma(acc0, a0, __ldg(x + c0));
    WideOps<S>::fma(acc1, a1, __ldg(x + c1));
  }
  if (p < e) WideOps<S>::fma(acc0, __ldcs(data + p), __ldg(x + (int64_t)__ldcs(idx + p)));
  A acc = w_add(acc0, acc1);
#pragma unroll
  for (int o = L >> 1; o > 0; o >>= 1) acc = w_add(acc, w_down(acc, o));
  if (lane == 0 && row < n_rows) y[row] = acc;
}

template <typename S, typename P>
__global__ void __launch_bounds__(kWideThreads)
spmm_wide_kernel(const S* __restrict__ data, const int32_t* __restrict__ idx, const P* __restrict__ ptr,
                 const typename WideOps<S>::Dense* __restrict__ B, int64_t ldb,
                 typename WideOps<S>::Dense* __restrict__ C, int64_t ldc, int64_t n_rows, int n_dense, int LN) {
  typedef typename WideOps<S>::Acc A;
  const int lane = threadIdx.x % LN;
  const int64_t row = (int64_t)blockIdx.x * (kWideThreads / LN) + threadIdx.x / LN;
  const int col = (int)blockIdx.y * LN + lane;
  if (row >= n_rows || col >= n_dense) return;   // no shuffles below: threads may leave on their own
  const int64_t s = (int64_t)ptr[row], e = (int64_t)ptr[row + 1];
  A acc0 = w_zero((A*)nullptr), acc1 = w_zero((A*)nullptr);
  int64_t p = s;
  for (; p + 1 < e; p += 2) {
    const S a0 = __ldg(data + p), a1 = __ldg(data + p + 1);
    const int64_t c0 = (int64_t)__ldg(idx + p), c1 = (int64_t)__ldg(idx + p + 1);
    WideOps<S>::fma(acc0, a0, __ldg(B + c0 * ldb + col));
    WideOps<S>::fma(acc1, a1, __ldg(B + c1 * ldb + col));
  }
  if (p < e) WideOps<S>::fma(acc0, __ldg(data + p), __ldg(B + (int64_t)__ldg(idx + p) * ldb + col));
  C[row * ldc + col] = w_add(acc0, acc1);
}

template <typename S, typename P>
static int wide_launch(const void* data, const int32_t* idx, const void* ptr, const void* x, void* y, int64_t n_rows,
                       int64_t nnz, cudaStream_t st) {
  typedef typename WideOps<S>::Dense D;
  const int64_t mean = n_rows > 0 ? nnz / n_rows : 0;
  int L = 2;
  while (L < 32 && 8 * L < mean + 3) L <<= 1;
  const int64_t blocks = (n_rows * L + kWideThreads - 1) / kWideThreads;
  if (blocks >= INT32_MAX) return FSB_ERANGE;
#define FSB_WIDE_CASE(L_)                                                                                         \
  case L_:                                                                                                        \
    spmv_wide_kernel<S, P, L_><<<(unsigned)blocks, kWideThreads, 0, st>>>((const S*)data, idx, (const P*)ptr,     \
                                                                          (const D*)x, (D*)y, n_rows);           \
    break
  switch (L) {
    FSB_WIDE_CASE(2);
    FSB_WIDE_CASE(4);
    FSB_WIDE_CASE(8);
    FSB_WIDE_CASE(16);
    default:
      FSB_WIDE_CASE(32);
  }
#undef FSB_WIDE_CASE
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_spmv_csr_wide(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr,
                                 const void* x, void* y, int64_t n_rows, int64_t n_cols, int64_t nnz, void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  if (vtype != FSB_F16 && vtype != FSB_BF16 && vtype != FSB_C64 && vtype != FSB_C128) return FSB_EINVAL;
  if (ptype != FSB_I32 && ptype != FSB_I64) return FSB_EINVAL;
  if (n_rows < 0 || n_cols < 0 || nnz < 0) return FSB_EINVAL;
  if (n_rows >= INT32_MAX || n_cols >= INT32_MAX) return FSB_ERANGE;
  if (n_rows == 0) return FSB_OK;
  if (indptr == nullptr || y == nullptr || (nnz > 0 && (data == nullptr || indices == nullptr || x == nullptr)))
    return FSB_EINVAL;
  const size_t sv = vtype == FSB_C128 ? 16 : (vtype == FSB_C64 ? 8 : 2);    // stored value
  const size_t sd = vtype == FSB_C128 ? 16 : (vtype == FSB_C64 ? 8 : 4);    // element of x and y
  if (!aligned_to(data, sv) || !aligned_to(x, sd) || !aligned_to(y, sd) || !aligned_to(indices, 4) ||
      !aligned_to(indptr, ptype == FSB_I32 ? 4 : 8))
    return FSB_EALIGN;
  FSB_WALK_FIRST(check_csr(FSB_I32, ptype, indices, indptr, n_rows, n_cols, nnz, st));
#define FSB_WIDE_TYPE(S_)                                                                                     \
  return ptype == FSB_I32 ? wide_launch<S_, int32_t>(data, indices, indptr, x, y, n_rows, nnz, st)            \
                          : wide_launch<S_, int64_t>(data, indices, indptr, x, y, n_rows, nnz, st)
  switch (vtype) {
    case FSB_F16: FSB_WIDE_TYPE(__half);
    case FSB_BF16: FSB_WIDE_TYPE(__nv_bfloat16);
    case FSB_C64: FSB_WIDE_TYPE(float2);
    default: FSB_WIDE_TYPE(double2);
  }
#undef FSB_WIDE_TYPE
}

template <typename S, typename P>
static int wide_spmm_launch(const void* data, const int32_t* idx, const void* ptr, const void* B, int64_t ldb, void* C,
                            int64_t ldc, int64_t n_rows, int n_dense, cudaStream_t st) {
  typedef typename WideOps<S>::Dense D;
  int LN = 1;
  while (LN < 32 && LN < n_dense) LN <<= 1;
  const int64_t gx = (n_rows + kWideThreads / LN - 1) / (kWideThreads / LN);
  const int64_t gy = (n_dense + LN - 1) / LN;
  if (gx >= INT32_MAX || gy > 65535) return FSB_ERANGE;
  spmm_wide_kernel<S, P><<<dim3((unsigned)gx, (unsigned)gy), kWideThreads, 0, st>>>(
      (const S*)data, idx, (const P*)ptr, (const D*)B, ldb, (D*)C, ldc, n_rows, n_dense, LN);
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

extern "C" int fsb_spmm_csr_wide(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr,
                                 const void* B, int64_t ldb, void* C, int64_t ldc, int64_t n_rows, int64_t n_cols,
                                 int64_t n_dense, int64_t nnz, void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  if (vtype != FSB_F16 && vtype != FSB_BF16 && vtype != FSB_C64 && vtype != FSB_C128) return FSB_EINVAL;
  if (ptype != FSB_I32 && ptype != FSB_I64) return FSB_EINVAL;
  if (n_rows < 0 || n_cols < 0 || nnz < 0 || n_dense < 0 || ldb < n_dense || ldc < n_dense) return FSB_EINVAL;
  if (n_rows >= INT32_MAX || n_cols >= INT32_MAX || n_dense >= (1 << 21)) return FSB_ERANGE;
  if (n_rows == 0 || n_dense == 0) return FSB_OK;
  if (indptr == nullptr || C == nullptr || (nnz > 0 && (data == nullptr || indices == nullptr || B == nullptr)))
    return FSB_EINVAL;
  const size_t sv = vtype == FSB_C128 ? 16 : (vtype == FSB_C64 ? 8 : 2);
  const size_t sd = vtype == FSB_C128 ? 16 : (vtype == FSB_C64 ? 8 : 4);
  if (!aligned_to(data, sv) || !aligned_to(B, sd) || !aligned_to(C, sd) || !aligned_to(indices, 4) ||
      !aligned_to(indptr, ptype == FSB_I32 ? 4 : 8))
    return FSB_EALIGN;
  FSB_WALK_FIRST(check_csr(FSB_I32, ptype, indices, indptr, n_rows, n_cols, nnz, st));
#define FSB_WIDE_TYPE(S_)                                                                                         \
  return ptype == FSB_I32                                                                                         \
             ? wide_spmm_launch<S_, int32_t>(data, indices, indptr, B, ldb, C, ldc, n_rows, (int)n_dense, st)      \
             : wide_spmm_launch<S_, int64_t>(data, indices, indptr, B, ldb, C, ldc, n_rows, (int)n_dense, st)
  switch (vtype) {
    case FSB_F16: FSB_WIDE_TYPE(__half);
    case FSB_BF16: FSB_WIDE_TYPE(__nv_bfloat16);
    case FSB_C64: FSB_WIDE_TYPE(float2);
    default: FSB_WIDE_TYPE(double2);
  }
#undef FSB_WIDE_TYPE
}

namespace fsb {

// ---------------------------------------------------------------------------------------------------
// y = A x with x and y in the matrix's own type
// ---------------------------------------------------------------------------------------------------
// four consecutive stored values: 8, 32 or 64 bytes in accesses of at most 16
__device__ __forceinline__ void ld_four(const __half* p, __half (&v)[4]) {
  const uint2 t = __ldcs(reinterpret_cast<const uint2*>(p));
  memcpy(v, &t, sizeof(t));
}
__device__ __forceinline__ void ld_four(const __nv_bfloat16* p, __nv_bfloat16 (&v)[4]) {
  const uint2 t = __ldcs(reinterpret_cast<const uint2*>(p));
  memcpy(v, &t, sizeof(t));
}
__device__ __forceinline__ void ld_four(const float2* p, float2 (&v)[4]) {
  const float4 a = __ldcs(reinterpret_cast<const float4*>(p)), b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
  v[0] = make_float2(a.x, a.y); v[1] = make_float2(a.z, a.w);
  v[2] = make_float2(b.x, b.y); v[3] = make_float2(b.z, b.w);
}
__device__ __forceinline__ void ld_four(const double2* p, double2 (&v)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __ldcs(p + i);
}

// Even rows: L lanes per row.  GROUPS (half precisions on aligned arrays): a lane reads whole groups of four entries, one
// request for the columns and one for the values, from the group that holds the row's first entry on, and masks what
// belongs to the neighbours; a walk entry by entry asks for 2 bytes at a time.  x is read and y written as they are, in
// this one pass (float16, 2e6 rows of 20 entries in a band of 2^15: 138 us with the passes that widen x and round y, here
// 90 us; 2e6 rows of 5, columns anywhere: 58 us and 49 us).  Otherwise one entry at a time: the lanes of a row then read neighbouring 8- or 16-byte
// values, and groups of four would spread each request over four times the lines (complex64, 500009 rows of 24,
// columns anywhere: 80 us in groups, 70 us entry by entry with four gathers on their way, 74 us with two; in a band of 2^15:
// 72 us, 63 us, 68 us).
template <typename S, typename P, int L, bool GROUPS>
__global__ void __launch_bounds__(kWideThreads)
spmv_stored_vector_kernel(const S* __restrict__ data, const int32_t* __restrict__ idx, const P* __restrict__ ptr,
                          const S* __restrict__ x, S* __restrict__ y, int64_t n_rows, int64_t nnz) {
  typedef StoredOps<S> Ops;
  typedef typename Ops::A A;
  const int64_t gtid = (int64_t)blockIdx.x * kWideThreads + threadIdx.x;
  const int64_t row = gtid / L;
  const int lane = (int)(gtid % L);
  int64_t s = 0, e = 0;
  if (row < n_rows) {
    s = (int64_t)ptr[row];
    e = (int64_t)ptr[row + 1];
  }
  A acc0 = w_zero((A*)nullptr), acc1 = w_zero((A*)nullptr);
  if (GROUPS) {
    const int64_t full = nnz & ~(int64_t)3;   // groups below this index lie wholly inside the arrays
    for (int64_t q = (s & ~(int64_t)3) + 4 * lane; q < e; q += 4 * L) {
      if (q >= s && q + 4 <= e && q + 4 <= full) {
        S a[4];
        int32_t c[4];
        ld_stream4(idx + q, c);
        ld_four(data + q, a);
        const S x0 = __ldg(x + c[0]), x1 = __ldg(x + c[1]), x2 = __ldg(x + c[2]), x3 = __ldg(x + c[3]);
        Ops::fma(acc0, a[0], x0);
        Ops::fma(acc1, a[1], x1);
        Ops::fma(acc0, a[2], x2);
        Ops::fma(acc1, a[3], x3);
      } else if (q + 4 <= full) {
        S a[4];
        int32_t c[4];
        ld_stream4(idx + q, c);
        ld_four(data + q, a);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (q + j >= s && q + j < e) {
            if (j & 1) Ops::fma(acc1, a[j], __ldg(x + c[j]));
            else Ops::fma(acc0, a[j], __ldg(x + c[j]));
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (q + j >= s && q + j < e) {
            const S xv = __ldg(x + __ldcs(idx + q + j));
            if (j & 1) Ops::fma(acc1, __ldcs(data + q + j), xv);
            else Ops::fma(acc0, __ldcs(data + q + j), xv);
          }
        }
      }
    }
  } else {
    int64_t p = s + lane;
    // (complex128: 2000000 rows of 20, 298 us with two gathers on their way, 289 us with four; 100000 rows of 60: 43 us, 41 us)
    for (; p + 3 * L < e; p += 4 * L) {
      S a[4];
      int32_t c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        a[j] = __ldcs(data + p + j * L);
        c[j] = __ldcs(idx + p + j * L);
      }
      S xv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) xv[j] = __ldg(x + c[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) Ops::fma(j & 1 ? acc1 : acc0, a[j], xv[j]);
    }
    for (; p + L < e; p += 2 * L) {
      const S a0 = __ldcs(data + p), a1 = __ldcs(data + p + L);
      const int32_t c0 = __ldcs(idx + p), c1 = __ldcs(idx + p + L);
      Ops::fma(acc0, a0, __ldg(x + c0));
      Ops::fma(acc1, a1, __ldg(x + c1));
    }
    if (p < e) Ops::fma(acc0, __ldcs(data + p), __ldg(x + __ldcs(idx + p)));
  }
  A acc = w_add(acc0, acc1);
#pragma unroll
  for (int o = L >> 1; o > 0; o >>= 1) acc = w_add(acc, w_down(acc, o));
  if (lane == 0 && row < n_rows) y[row] = Ops::narrow(acc);
}

// Uneven rows: tiles of a fixed number of entries, as in spmv_stream_kernel (spmv_csr.cu): products to shared memory,
// L lanes per segment, segments much longer than the tile's mean by whole warps; the rows that cross tiles leave
// partial sums for spmv_stored_fixup_kernel.  The lanes-per-row kernel gives a row of 2^17 entries the 2 to 32 lanes that
// the mean row length asks for (complex64, 3e6 rows of Zipf lengths, 36 M entries: 15.9 ms, here 226 us; complex128,
// 252377 such rows: 7.3 ms and 37 us; bfloat16, 27496 rows: 223 us and 16 us).
template <typename S>
__host__ __device__ constexpr int stored_tile() { return sizeof(S) == 16 ? 1024 : 2048; }

template <typename S, typename P, bool ALIGNED>
__global__ void __launch_bounds__(kWideThreads)
spmv_stored_stream_kernel(const S* __restrict__ data, const int32_t* __restrict__ idx, const P* __restrict__ ptr,
                          const S* __restrict__ x, S* __restrict__ y, const int32_t* __restrict__ tile_row,
                          typename StoredOps<S>::A* __restrict__ carry, typename StoredOps<S>::A* __restrict__ head,
                          int64_t nnz) {
  typedef StoredOps<S> Ops;
  typedef typename Ops::A A;
  constexpr int T = stored_tile<S>();
  constexpr int RC = T;                       // segments whose offsets are kept at a time
  constexpr int IPT = T / kWideThreads;
  constexpr int NW = kWideThreads / 32;
  __shared__ __align__(16) A s_prod[T];
  __shared__ int32_t s_off[RC + 1];
  __shared__ int32_t s_long[T / 32 + 2];      // a long segment has more than 32 entries
  __shared__ int s_n_long, s_head_partial;
  const int tid = threadIdx.x;
  const int64_t t = blockIdx.x;
  const int64_t lo = t * (int64_t)T;
  const int cnt = (int)((nnz - lo) < (int64_t)T ? (nnz - lo) : (int64_t)T);
  const int32_t ra = tile_row[t], rb = tile_row[t + 1];
  const int nrf = rb - ra, nseg = nrf + 1;    // rows that end here, and the one that goes on

  if (ALIGNED && cnt == T) {
#pragma unroll
    for (int j = 0; j < IPT / 4; ++j) {
      const int e = (j * kWideThreads + tid) * 4;
      S a[4];
      int32_t c[4];
      ld_four(data + lo + e, a);
      ld_stream4(idx + lo + e, c);
      S xv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) xv[k] = __ldg(x + c[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k) s_prod[e + k] = Ops::prod(a[k], xv[k]);
    }
  } else {
    for (int e = tid; e < cnt; e += kWideThreads)
      s_prod[e] = Ops::prod(__ldcs(data + lo + e), __ldg(x + __ldcs(idx + lo + e)));
  }

  int L = pow2_floor((cnt / nseg) >> 3);
  L = L > 32 ? 32 : L;
  const int lane = tid & (L - 1), grp = tid / L, ngrp = kWideThreads / L;
  for (int base = 0; base < nseg; base += RC) {
    const int m = (nseg - base) < RC ? (nseg - base) : RC;
    if (base > 0) __syncthreads();            // the previous pass is done with the tables
    for (int k = tid; k <= m; k += kWideThreads) {
      const int g = base + k;
      int32_t o = cnt;
      if (g <= nrf) {
        const int64_t d = (int64_t)ptr[(int64_t)ra + g] - lo;
        o = d < 0 ? 0 : (d > cnt ? cnt : (int32_t)d);
        if (g == 0) s_head_partial = (d < 0 && nrf > 0) ? 1 : 0;
      }
      s_off[k] = o;
    }
    if (tid == 0) s_n_long = 0;
    __syncthreads();                          // products and offsets are there
    auto finish = [&](int k, A acc) {
      const int g = base + k;
      if (g == nrf) carry[t] = acc;
      else if (g == 0 && s_head_partial) head[t] = acc;
      else y[(int64_t)ra + g] = Ops::narrow(acc);
    };
    const int iters = (m + ngrp - 1) / ngrp;  // the same for all lanes: the shuffles below are the whole warp's
    for (int it = 0; it < iters; ++it) {
      const int k = it * ngrp + grp;
      const bool valid = k < m;
      const int s = valid ? s_off[k] : 0, e = valid ? s_off[k + 1] : 0;
      const bool is_long = L < 32 && e - s > 32 * L;
      A acc = w_zero((A*)nullptr);
      if (!is_long) {
        A a1 = w_zero((A*)nullptr);
        for (int p = s + lane; p < e; p += 2 * L) {
          acc = w_add(acc, s_prod[p]);
          if (p + L < e) a1 = w_add(a1, s_prod[p + L]);
        }
        acc = w_add(acc, a1);
      }
      for (int o = L >> 1; o > 0; o >>= 1) acc = w_add(acc, w_down(acc, o));
      if (valid && lane == 0) {
        if (is_long) s_long[atomicAdd(&s_n_long, 1)] = k;
        else finish(k, acc);
      }
    }
    __syncthreads();
    const int n_long = s_n_long;
    const int w = tid >> 5, l32 = tid & 31;
    for (int q = w; q < n_long; q += NW) {
      const int k = s_long[q];
      const int s = s_off[k], e = s_off[k + 1];
      A a0 = w_zero((A*)nullptr), a1 = w_zero((A*)nullptr);
      int p = s + l32;
      for (; p + 32 < e; p += 64) {
        a0 = w_add(a0, s_prod[p]);
        a1 = w_add(a1, s_prod[p + 32]);
      }
      if (p < e) a0 = w_add(a0, s_prod[p]);
      A acc = w_add(a0, a1);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc = w_add(acc, w_down(acc, o));
      if (l32 == 0) finish(k, acc);
    }
  }
}

__device__ __forceinline__ double2 to_wide(float v) { return make_double2((double)v, 0.0); }
__device__ __forceinline__ double2 to_wide(float2 v) { return make_double2((double)v.x, (double)v.y); }
__device__ __forceinline__ double2 to_wide(double2 v) { return v; }
__device__ __forceinline__ void from_wide(double2 v, float& r) { r = (float)v.x; }
__device__ __forceinline__ void from_wide(double2 v, float2& r) { r = make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ void from_wide(double2 v, double2& r) { r = v; }

// one warp per tile t >= 1: finish the row that began in an earlier tile and ends in t.  The carries of the tiles it
// crossed are summed lane-strided in double and combined in a fixed order.
template <typename S, typename P>
__global__ void __launch_bounds__(kWideThreads)
spmv_stored_fixup_kernel(const P* __restrict__ ptr, const int32_t* __restrict__ tile_row,
                         const typename StoredOps<S>::A* __restrict__ carry,
                         const typename StoredOps<S>::A* __restrict__ head, S* __restrict__ y, int64_t n_tiles) {
  typedef StoredOps<S> Ops;
  constexpr int T = stored_tile<S>();
  const int64_t t = ((int64_t)blockIdx.x * kWideThreads + threadIdx.x) / 32 + 1;
  const int lane = threadIdx.x & 31;
  if (t >= n_tiles) return;
  const int32_t ra = tile_row[t];
  if (ra >= tile_row[t + 1]) return;
  const int64_t p = (int64_t)ptr[ra];
  if (p >= t * T) return;
  double2 sum = make_double2(0.0, 0.0);
  for (int64_t u = p / T + lane; u < t; u += 32) sum = w_add(sum, to_wide(carry[u]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum = w_add(sum, w_down(sum, o));
  if (lane == 0) {
    typename Ops::A r;
    from_wide(w_add(sum, to_wide(head[t])), r);
    y[ra] = Ops::narrow(r);
  }
}

template <typename S, typename P>
static int stored_launch(const void* data_, const int32_t* idx, const void* ptr_, const void* x_, void* y_, int64_t n_rows,
                         int64_t nnz, bool even, const int32_t* tile_row, void* scratch, cudaStream_t st) {
  typedef typename StoredOps<S>::A A;
  const S* data = (const S*)data_;
  const P* ptr = (const P*)ptr_;
  const S* x = (const S*)x_;
  S* y = (S*)y_;
  const bool aligned = aligned_to(data, sizeof(S) < 4 ? 8 : 16) && aligned_to(idx, 16);
  const bool groups = sizeof(S) < 4 && aligned;    // see spmv_stored_vector_kernel
  if (tile_row != nullptr) {
    constexpr int T = stored_tile<S>();
    const int64_t n_tiles = (nnz + T - 1) / T;
    if (n_tiles >= INT32_MAX / 32) return FSB_ERANGE;
    A* carry = (A*)scratch;
    A* head = carry + n_tiles;
    if (aligned)
      spmv_stored_stream_kernel<S, P, true><<<(unsigned)n_tiles, kWideThreads, 0, st>>>(data, idx, ptr, x, y, tile_row,
                                                                                        carry, head, nnz);
    else
      spmv_stored_stream_kernel<S, P, false><<<(unsigned)n_tiles, kWideThreads, 0, st>>>(data, idx, ptr, x, y, tile_row,
                                                                                         carry, head, nnz);
    FSB_RETURN_IF_LAUNCH_FAILED();
    if (n_tiles > 1) {
      const int64_t g = ((n_tiles - 1) * 32 + kWideThreads - 1) / kWideThreads;
      spmv_stored_fixup_kernel<S, P><<<(unsigned)g, kWideThreads, 0, st>>>(ptr, tile_row, carry, head, y, n_tiles);
      FSB_RETURN_IF_LAUNCH_FAILED();
    }
    return FSB_OK;
  }
  if (even && rows_apply<S>(data, idx, n_rows, nnz))
    return rows_run<S, int32_t, P>(data, idx, ptr, x, RowsOut<S>{y}, n_rows, nnz, st);
  // two to four groups of four entries per lane, as in the float32 / float64 kernel; entry by entry, three to six
  // (columns anywhere, 4 / 8 / 16 lanes a row: complex64, 500009 rows of 24: 70 / 64 / - us, 300000 rows of 30: 55 / 47 / 51 us,
  // 2000000 rows of 20: 209 / 212 / - us, 100000 rows of 60: - / 35 / 31 us; complex128: 84 / 78 / - us, 66 / 58 / 64 us, 289 / 294
  // / - us, - / 41 / 37 us)
  const int64_t mean = n_rows > 0 ? nnz / n_rows : 0;
  int L = 2;
  while (L < 32 && (groups ? 16 : 6) * L < mean + 3) L <<= 1;
  const int64_t blocks = (n_rows * L + kWideThreads - 1) / kWideThreads;
  if (blocks >= INT32_MAX) return FSB_ERANGE;
#define FSB_STORED_CASE(L_)                                                                                           \
  case L_:                                                                                                            \
    if constexpr (sizeof(S) < 4) {                                                                                    \
      if (groups) {                                                                                                   \
        spmv_stored_vector_kernel<S, P, L_, true><<<(unsigned)blocks, kWideThreads, 0, st>>>(data, idx, ptr, x, y,    \
                                                                                            n_rows, nnz);            \
        break;                                                                                                        \
      }                                                                                                               \
    }                                                                                                                 \
    spmv_stored_vector_kernel<S, P, L_, false><<<(unsigned)blocks, kWideThreads, 0, st>>>(data, idx, ptr, x, y,       \
                                                                                         n_rows, nnz);               \
    break
  switch (L) {
    FSB_STORED_CASE(2);
    FSB_STORED_CASE(4);
    FSB_STORED_CASE(8);
    FSB_STORED_CASE(16);
    default:
      FSB_STORED_CASE(32);
  }
#undef FSB_STORED_CASE
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_spmv_stored_tile_nnz(int vtype) { return vtype == FSB_C128 ? stored_tile<double2>() : stored_tile<float2>(); }

extern "C" size_t fsb_spmv_stored_scratch_bytes(int vtype, int64_t nnz) {
  const size_t sa = vtype == FSB_C128 ? 16 : (vtype == FSB_C64 ? 8 : 4);
  return ((size_t)fsb_csr_num_tiles(nnz, fsb_spmv_stored_tile_nnz(vtype)) * 2 * sa + 255) & ~(size_t)255;
}

static int spmv_stored(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr, const void* x, void* y,
                       int64_t n_rows, int64_t n_cols, int64_t nnz, bool even, const int32_t* tile_row, void* scratch,
                       size_t scratch_bytes, cudaStream_t st) {
  if (vtype != FSB_F16 && vtype != FSB_BF16 && vtype != FSB_C64 && vtype != FSB_C128) return FSB_EINVAL;
  if (ptype != FSB_I32 && ptype != FSB_I64) return FSB_EINVAL;
  if (n_rows < 0 || n_cols < 0 || nnz < 0) return FSB_EINVAL;
  if (n_rows >= INT32_MAX || n_cols >= INT32_MAX) return FSB_ERANGE;
  if (n_rows == 0) return FSB_OK;
  if (indptr == nullptr || y == nullptr || (nnz > 0 && (data == nullptr || indices == nullptr || x == nullptr)))
    return FSB_EINVAL;
  const size_t sv = vtype == FSB_C128 ? 16 : (vtype == FSB_C64 ? 8 : 2);
  if (!aligned_to(data, sv) || !aligned_to(x, sv) || !aligned_to(y, sv) || !aligned_to(indices, 4) ||
      !aligned_to(indptr, ptype == FSB_I32 ? 4 : 8))
    return FSB_EALIGN;
  if (nnz == 0) tile_row = nullptr;    // no tiles: the vector kernel writes the zeros
  if (tile_row != nullptr) {
    if (scratch == nullptr) return FSB_EINVAL;
    if (scratch_bytes < fsb_spmv_stored_scratch_bytes(vtype, nnz)) return FSB_ESCRATCH;
    if (!aligned_to(scratch, 16)) return FSB_EALIGN;
  }
  FSB_WALK_FIRST(check_csr(FSB_I32, ptype, indices, indptr, n_rows, n_cols, nnz, st));
#define FSB_STORED_TYPE(S_)                                                                                           \
  return ptype == FSB_I32                                                                                             \
             ? stored_launch<S_, int32_t>(data, indices, indptr, x, y, n_rows, nnz, even, tile_row, scratch, st)      \
             : stored_launch<S_, int64_t>(data, indices, indptr, x, y, n_rows, nnz, even, tile_row, scratch, st)
  switch (vtype) {
    case FSB_F16: FSB_STORED_TYPE(__half);
    case FSB_BF16: FSB_STORED_TYPE(__nv_bfloat16);
    case FSB_C64: FSB_STORED_TYPE(float2);
    default: FSB_STORED_TYPE(double2);
  }
#undef FSB_STORED_TYPE
}

extern "C" int fsb_spmv_csr_stored(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr,
                                   const void* x, void* y, int64_t n_rows, int64_t n_cols, int64_t nnz,
                                   const int32_t* tile_row, void* scratch, size_t scratch_bytes, void* stream_) {
  return spmv_stored(vtype, ptype, data, indices, indptr, x, y, n_rows, n_cols, nnz, false, tile_row, scratch, scratch_bytes,
                     static_cast<cudaStream_t>(stream_));
}

extern "C" int fsb_spmv_csr_stored_even(int vtype, int ptype, const void* data, const int32_t* indices, const void* indptr,
                                        const void* x, void* y, int64_t n_rows, int64_t n_cols, int64_t nnz, void* stream_) {
  return spmv_stored(vtype, ptype, data, indices, indptr, x, y, n_rows, n_cols, nnz, true, nullptr, nullptr, 0,
                     static_cast<cudaStream_t>(stream_));
}

// Check and product of arrays that are used once, whatever the value type.
extern "C" int fsb_spmv_csr_once(int vtype, int itype, int ptype, const void* data, const void* indices, const void* indptr,
                                 const void* x, void* y, int64_t n_rows, int64_t n_cols, int64_t nnz, int64_t longest, int64_t even,
                                 void* work, int64_t* host, void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  const bool stored = vtype != FSB_F32 && vtype != FSB_F64;
  if (stored && itype != FSB_I32) return FSB_EINVAL;
  int rc = csr_check_launch(itype, ptype, indices, indptr, n_rows, nnz, work, host, st);
  if (rc == FSB_OK) rc = csr_check_wait(host, st);
  if (rc != FSB_OK) return rc;
  if (!csr_check_passed(host, n_cols, nnz) || csr_check_longest(host) > longest) return FSB_NOT_LAUNCHED;
  const bool is_even = csr_check_longest(host) <= even;
  if (stored)
    return spmv_stored(vtype, ptype, data, (const int32_t*)indices, indptr, x, y, n_rows, n_cols, nnz, is_even, nullptr, nullptr, 0,
                       st);
  return fsb_spmv_csr(vtype, itype, ptype, data, indices, indptr, x, y, n_rows, n_cols, nnz, FSB_SPMV_VECTOR,
                      is_even ? FSB_SPMV_EVEN_ROWS : 0, nullptr, nullptr, 0, stream_);
}
