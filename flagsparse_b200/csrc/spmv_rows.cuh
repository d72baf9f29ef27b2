// CSR SpMV for rows of about equal length: one CTA per SM, which walks rows that follow each other.
#pragma once
#include <string.h>

#include "fsb_common.cuh"
#include "stored_ops.cuh"

namespace fsb {

constexpr int kRowsThreads = 1024;

template <int BYTES> struct RowsRaw;
template <> struct RowsRaw<4> { typedef unsigned int type; };
template <> struct RowsRaw<8> { typedef uint2 type; };
template <> struct RowsRaw<16> { typedef uint4 type; };

// N consecutive elements in accesses of at most 16 bytes
template <typename T, int N>
__device__ __forceinline__ void rows_load(const T* p, T (&v)[N]) {
  constexpr int BYTES = N * (int)sizeof(T), ONE = BYTES < 16 ? BYTES : 16;
  typedef typename RowsRaw<ONE>::type Raw;
#pragma unroll
  for (int i = 0; i < BYTES / ONE; ++i) {
    const Raw t = __ldcs(reinterpret_cast<const Raw*>(p) + i);
    memcpy(reinterpret_cast<char*>(v) + i * ONE, &t, ONE);
  }
}
template <int N>
__device__ __forceinline__ void rows_columns(const int32_t* p, int32_t (&c)[N]) { rows_load(p, c); }
template <int N>
__device__ __forceinline__ void rows_columns(const int64_t* p, int32_t (&c)[N]) {
  int64_t t[N];
  rows_load(p, t);
#pragma unroll
  for (int j = 0; j < N; ++j) c[j] = (int32_t)t[j];
}

// Share i of n: rows first(i) .. first(i + 1) - 1
struct RowsShares {
  int rows, more, most;       // rows of a share, and how many shares have one more; entries of one at most for the shares to be even
  __host__ RowsShares(int64_t n_rows, int64_t nnz, int n) {
    rows = (int)(n_rows / n);
    more = (int)(n_rows % n);
    const int64_t e = nnz / n + nnz / n / 8 + 1024;
    most = (int)(e < INT32_MAX ? e : INT32_MAX);
  }
  __device__ __forceinline__ int first(int i) const { return rows * i + (i < more ? i : more); }
};

// Why: a gather costs an SM one look into its L1 per clock whether it hits or not, but what misses goes to L2 for hundreds of
// cycles, on a port that takes about one request per clock.  A grid of small CTAs in the order of the rows puts rows from all over
// the matrix on one SM at a time; here the rows of an SM are neighbours, and the part of x that they share stays in its L1.
// A warp has the entries of its next U * 32 / L rows on their way while it works on its rows, and the row pointers of the rows after
// those: they wait for memory at the same time instead of one after the other.  L lanes a row, E
// entries a lane at a time (E * sizeof(S) bytes in one access), from the multiple of E below the row's first entry on.
// What is left is that look per gather: 12 M complex64 gathers take 42 us at one per clock and SM.
// 500009 rows of 24 in a band of 2^14, us through lanes-per-row CTAs / here: complex64 58 / 46, float16 44 / 27, float32 46 / 29; columns
// anywhere: complex64 64 / 57, bfloat16 64 / 50; float64, 300007 rows of 27, band 2^13: 43 / 29; 2000000 rows of 5, band 2^14:
// bfloat16 56 / 31, complex128 90 / 75; 64-bit indices, float64, 300000 rows of 30, band 2^13: 54 / 39, 3232656 rows of 4, band 2^18:
// 106 / 90.  Two CTAs of 512 threads on an SM, each with rows of its own: 55 instead of 46; without the entries on their way 2 to
// 4 us more; a window of x in shared memory instead of L1: 39 to 66 (where a tenth of the entries lies outside, most warps wait for it).
// Out::store(row, value) puts a finished row away.
template <typename S, typename I, typename P, int L, int U, int E, typename Out>
__global__ void __launch_bounds__(kRowsThreads, 1)
spmv_rows_kernel(const S* __restrict__ data, const I* __restrict__ idx, const P* __restrict__ ptr, const S* __restrict__ x,
                 const Out out, int64_t n_rows, int64_t nnz, const RowsShares shares) {
  typedef StoredOps<S> Ops;
  typedef typename Ops::A A;
  constexpr int G = 32 / L, RW = U * G, STEP = kRowsThreads / 32 * RW;
  static_assert(RW <= 32 && L >= U, "one lane per row of a warp");
  struct Rows {            // what a warp has of RW rows: bounds of this lane's rows, and its entries of them
    int s[U], e[U];
    S v[U][E];
    int32_t c[U][E];
  };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % L, grp = lane / L;
  // whether some share has many more entries than the others; every CTA looks at all of them, so all come to the same answer
  bool uneven = false;
  if (threadIdx.x < gridDim.x) {
    const int i = (int)threadIdx.x;
    uneven = (int)((int64_t)ptr[shares.first(i + 1)] - (int64_t)ptr[shares.first(i)]) > shares.most;
  }
  int row = shares.first((int)blockIdx.x) + warp * RW, end = shares.first((int)blockIdx.x + 1), hop = STEP;
  int a, b;                // lane l: the bounds of row number l of the warp's next ones
  auto bounds = [&](int at) {
    a = b = 0;
    if (lane < RW && at < end - lane) {
      a = (int)ptr[at + lane];
      b = (int)ptr[at + lane + 1];
    }
  };
  const int count = (int)nnz;
  auto load = [&](int q, S (&v)[E], int32_t (&c)[E]) {
    if (q + E <= count) {
      rows_load(data + q, v);
      rows_columns(idx + q, c);
    } else {
#pragma unroll
      for (int j = 0; j < E; ++j)
        if (q + j < count) {
          v[j] = data[q + j];
          c[j] = (int32_t)idx[q + j];
        }
    }
  };
  auto fetch = [&](Rows& f) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      f.s[u] = __shfl_sync(0xffffffffu, a, u * G + grp);
      f.e[u] = __shfl_sync(0xffffffffu, b, u * G + grp);
      const int q = (f.s[u] & ~(E - 1)) + E * sub;
      if (q < f.e[u]) load(q, f.v[u], f.c[u]);
    }
  };
  auto finish = [&](Rows& f, int row) {
    A acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int q = (f.s[u] & ~(E - 1)) + E * sub;
      A even = w_zero((A*)nullptr), odd = w_zero((A*)nullptr);
#pragma unroll
      for (int j = 0; j < E; ++j)
        if (q + j >= f.s[u] && q + j < f.e[u]) Ops::fma(j & 1 ? odd : even, f.v[u][j], __ldg(x + f.c[u][j]));
      acc[u] = w_add(even, odd);
    }
    // entries beyond L * E of a row: two more partial sums
#pragma unroll
    for (int u = 0; u < U; ++u) {
      int q = (f.s[u] & ~(E - 1)) + E * (sub + L);
      if (q < f.e[u]) {
        A even = w_zero((A*)nullptr), odd = w_zero((A*)nullptr);
        for (; q < f.e[u]; q += L * E) {
          load(q, f.v[u], f.c[u]);
#pragma unroll
          for (int j = 0; j < E; ++j)
            if (q + j < f.e[u]) Ops::fma(j & 1 ? odd : even, f.v[u][j], __ldg(x + f.c[u][j]));
        }
        acc[u] = w_add(acc[u], w_add(even, odd));
      }
    }
    // U rows over L lanes: an exchange halves the rows that a lane answers for, until one is left
    int held = U;
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      if (held > 1) {
        held >>= 1;
        const bool upper = (sub & o) != 0;
#pragma unroll
        for (int i = 0; i < U / 2; ++i)
          if (i < held) {
            const A send = upper ? acc[i] : acc[i + held];
            const A keep = upper ? acc[i + held] : acc[i];
            acc[i] = w_add(keep, w_xor(send, o));
          }
      } else {
        acc[0] = w_add(acc[0], w_xor(acc[0], o));
      }
    }
    constexpr int D = L / U;             // lanes with the same sum
    const int r = row + sub / D * G + grp;
    if (sub % D == 0 && r < end) out.store(r, Ops::narrow(acc[0]));
  };
  Rows f0, f1;
  auto begin = [&]() {
    bounds(row);
    fetch(f0);
    bounds(row + hop);
  };
  begin();
  // (the first entries are on their way by now)  Uneven shares: stretches of STEP rows are dealt to the CTAs in turn
  if (__syncthreads_or(uneven)) {
    row = (int)blockIdx.x * STEP + warp * RW;
    end = (int)n_rows;
    hop = (int)gridDim.x * STEP;
    begin();
  }
  while (row < end) {
    fetch(f1);
    bounds(row + 2 * hop);
    finish(f0, row);
    row += hop;
    if (row >= end) break;
    fetch(f0);
    bounds(row + 2 * hop);
    finish(f1, row);
    row += hop;
  }
}

template <typename S>
struct RowsOut {
  S* y;
  __device__ __forceinline__ void store(int64_t i, S v) const { y[i] = v; }
};

// Entries that a lane reads at once and rows of a group of lanes together: four and two; 8-byte values leave registers for one
// row of four (columns anywhere, float64, 1000000 rows of 8: 45 us, two rows of two entries 53 us), complex128 for one of two.
template <typename S> __host__ __device__ constexpr int rows_each() { return sizeof(S) == 16 ? 2 : 4; }
template <typename S> __host__ __device__ constexpr int rows_together() { return sizeof(S) <= 4 ? 2 : 1; }

// Lanes of a row: the fewest that hold four fifths of a mean row at once (complex128 two fifths: 4 / 8 / 16 lanes, columns anywhere,
// 1000000 rows of 12 80 / 86 / - us, 500000 rows of 36 111 / 101 / 115, 300000 rows of 60 107 / 99 / 102); more leave lanes idle
// (float32, 1000000 rows of 4, 2 / 4 / 8 lanes: 17 / 21 / 33 us), fewer a second turn for most rows (float64, 100000 rows of 50,
// 16 / 8 / 4 / 2 lanes: 27 / 25 / 27 / 30 us).
template <typename S>
static int rows_lanes(int64_t mean) {
  int L = 2;
  while (L < 32 && 5 * L * rows_each<S>() < (sizeof(S) == 16 ? 2 : 4) * mean) L <<= 1;
  return L;
}

// Mean row from which fewer rows than warps are no hindrance: the lanes-per-row kernel then has its own trouble with them.
template <typename S> constexpr int64_t rows_long() { return sizeof(S) == 4 ? 24 : 10; }
template <> constexpr int64_t rows_long<float2>() { return 0; }
template <> constexpr int64_t rows_long<double2>() { return INT32_MAX; }

// Matrices that take the kernel: 8192 to 2^30 rows, up to 2^30 entries (row + 2 * hop fits 32 bits), and rows for four fifths of the
// warps (32 to 1024 rows an SM) or rows that are long: short rows leave most warps without any.  us through lanes per row / here:
// float32, 8192 rows of 4 2.2 / 2.6, 32768 Poisson rows of 8 3.6 / 4.5, 80000 rows of 4 3.3 / 3.6, 131072 such rows 4.6 / 4.3; 12000
// Poisson rows of 30 4.4 / 4.2; float64, 32768 rows of 4 2.6 / 2.8, 20000 Poisson rows of 20 5.7 / 4.5; bfloat16, 32768 rows of 4 2.6 /
// 3.0; complex128, 12000 rows of 8 2.6 / 3.1, Poisson rows of 30 4.3 / 4.7; complex64, 20000 rows of 8 2.9 / 3.0, Poisson 4.6 / 3.5.
constexpr int kRowsLeast = 8192;
template <typename S>
static bool rows_apply(const void* data, const void* idx, int64_t n_rows, int64_t nnz) {
  if (n_rows < kRowsLeast || n_rows > (1 << 30) || nnz > (1 << 30) || !aligned_to(data, 16) || !aligned_to(idx, 16)) return false;
  const int64_t mean = nnz / n_rows;
  int sms = 0;
  if (mean >= rows_long<S>()) return true;
  if (sm_count(&sms) != FSB_OK) return false;
  return 5 * n_rows >= 4 * (int64_t)sms * (kRowsThreads / 32) * rows_together<S>() * (32 / rows_lanes<S>(mean));
}

template <typename S, typename I, typename P, typename Out>
static int rows_run(const void* data_, const void* idx_, const void* ptr_, const void* x_, Out out, int64_t n_rows, int64_t nnz,
                    cudaStream_t st) {
  constexpr int E = rows_each<S>(), U = rows_together<S>();
  const S *data = (const S*)data_, *x = (const S*)x_;
  const I* idx = (const I*)idx_;
  const P* ptr = (const P*)ptr_;
  int sms = 0;
  const int rc = sm_count(&sms);
  if (rc != FSB_OK) return rc;
  if (sms > kRowsThreads) sms = kRowsThreads;          // a thread looks at a share
  const RowsShares shares(n_rows, nnz, sms);
  switch (rows_lanes<S>(nnz / n_rows)) {
    case 2: spmv_rows_kernel<S, I, P, 2, U, E><<<sms, kRowsThreads, 0, st>>>(data, idx, ptr, x, out, n_rows, nnz, shares); break;
    case 4: spmv_rows_kernel<S, I, P, 4, U, E><<<sms, kRowsThreads, 0, st>>>(data, idx, ptr, x, out, n_rows, nnz, shares); break;
    case 8: spmv_rows_kernel<S, I, P, 8, U, E><<<sms, kRowsThreads, 0, st>>>(data, idx, ptr, x, out, n_rows, nnz, shares); break;
    case 16: spmv_rows_kernel<S, I, P, 16, U, E><<<sms, kRowsThreads, 0, st>>>(data, idx, ptr, x, out, n_rows, nnz, shares); break;
    default: spmv_rows_kernel<S, I, P, 32, U, E><<<sms, kRowsThreads, 0, st>>>(data, idx, ptr, x, out, n_rows, nnz, shares); break;
  }
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

}  // namespace fsb
