// CSR SpMV in two streaming passes, for matrices whose columns lie all over a long x ("bins" form).
//
// Why: where neither L1 nor a chunk of x in shared memory serves the gathers (columns anywhere, rows too short to fill a unit
// of the panel kernel), a one-pass kernel sends one request per entry towards L2, and once x outgrows L2 close to half of
// them go on to memory for 32 bytes each.  Here no gather leaves the SM.  Prepare cuts the rows into blocks of at most 24 576
// (float64: 12 288) entries and the columns into chunks, and stores the columns of the entries a second time, chunk by chunk,
// inside a chunk block by block; what a block has in a chunk (a "unit") is filled up to whole packs (8 entries, float64: 4).
//   gather    a CTA holds one chunk of x in shared memory and walks its share of the entries in storage order: 16-bit column
//             inside the chunk in, element of x out, two streams;
//   sum       a CTA owns a row block: it fetches the block's run of packs from every chunk (one 32-bit pack number per pack),
//             puts each element of x at its entry's CSR position in shared memory (16 bits per entry), multiplies by the values,
//             which lie in CSR order where the caller has them, and adds up the rows.
// Per float32 entry 2 bytes in and 4 out, then 4 + 2 + 0.5 + 4 in (float64: 10 and 19): twice the bytes of one pass, all of
// them streamed.  Rows are summed in CSR order, in double (float64: compensated inside a slice), so results do not depend on
// the order of the entries inside a unit and are bit-reproducible.  107 M entries in 16.7 M rows of Zipf lengths, columns
// anywhere in 2^24, float32: 640 us through spmv_stream_kernel, 442 us here: gather 135 us (0.64 GB), sum 305 us (1.13 GB; a
// block's elements arrive, are multiplied and added up and leave in turn, and two blocks an SM cover each other's phases in
// part).  With a copy of the values in storage order, multiplied by the first pass: 216 and 225 us, but 4 more bytes an entry,
// and values that the caller writes later would not be seen.  (Values asked for ahead with prefetch.global.L2: 3 us less
// here, but 4 us more for 2^24 entries, which L2 holds.)  The part of a row in the slice where it ends stays in double until what
// the slices before have is there: rounded before, two parts that cancel lose what they differ by.
#include "fsb_common.cuh"

namespace fsb {

constexpr int kBinGatherThreads = 1024;
constexpr int kBinSumThreads = 768;
constexpr int kBinBuildThreads = 512;
constexpr int kBinQuad = 4;                  // entries that a thread moves together
constexpr int kBinMaxChunks = 8192;          // cells of a block's counts in shared memory while the layout is built

template <typename V> __host__ __device__ constexpr int bin_pack() { return 32 / (int)sizeof(V); }    // entries of a pack
// entries that one thread adds up, and where entry i of a block is kept: one place in 33 (17) is left out, so that the
// lanes of a warp, a slice apart, read different banks
template <typename V> __host__ __device__ constexpr int bin_slice() { return 128 / (int)sizeof(V); }
template <typename V> __host__ __device__ constexpr int bin_cap() { return kBinSumThreads * bin_slice<V>(); }
template <typename V> __host__ __device__ __forceinline__ int bin_slot(int i) { return i + i / bin_slice<V>(); }
// two more places: a zero for the rows without entries, and where what fills a unit up goes
template <typename V> __host__ __device__ constexpr int bin_empty() { return kBinSumThreads * (bin_slice<V>() + 1); }
template <typename V> __host__ __device__ constexpr int bin_fill() { return bin_empty<V>() + 1; }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void unpack16(uint2 w, uint32_t (&c)[4]) {
  c[0] = w.x & 0xFFFFu; c[1] = w.x >> 16; c[2] = w.y & 0xFFFFu; c[3] = w.y >> 16;
}
__device__ __forceinline__ void st_quad(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st_quad(double* p, const double (&v)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// xg[e] = x[first column of e's chunk + col[e]] for all stored entries e.  CTA i takes the i-th equal share of the packs; a
// share crosses few chunks, so the chunks of x cost little beside the entries.
template <typename V>
__global__ void __launch_bounds__(kBinGatherThreads, 1)
bins_gather_kernel(const uint16_t* __restrict__ col, const int32_t* __restrict__ chunk_pack, int n_chunks, int chunk_cols,
                   const V* __restrict__ x, int64_t n_cols, V* __restrict__ xg) {
  extern __shared__ __align__(16) unsigned char b_smem[];
  V* xs = reinterpret_cast<V*>(b_smem);
  constexpr int QP = bin_pack<V>() / kBinQuad;        // quads of a pack
  const int tid = threadIdx.x;
  const int64_t total = chunk_pack[n_chunks];
  const int p0 = (int)(total * blockIdx.x / gridDim.x), p1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
  if (p0 >= p1) return;
  int c = 0;                                  // last chunk that starts at or before p0
  for (int lo = 0, hi = n_chunks; lo < hi;) {
    const int mid = (lo + hi) >> 1;
    if (chunk_pack[mid + 1] > p0) hi = mid; else lo = mid + 1;
    c = lo;
  }
  constexpr int E = 16 / (int)sizeof(V);
  constexpr int U = 2;                        // quads of a thread on their way together
  for (int p = p0; p < p1; ++c) {
    const int p_end = chunk_pack[c + 1] < p1 ? chunk_pack[c + 1] : p1;
    if (p_end <= p) continue;
    const int64_t c0 = (int64_t)c * chunk_cols;
    const int n = (int)((n_cols - c0) < (int64_t)chunk_cols ? (n_cols - c0) : (int64_t)chunk_cols);
    __syncthreads();                          // the previous chunk is no longer read
    const V* src = x + c0;
    if (aligned_to_dev(src)) {
      for (int i = tid; i < n / E; i += kBinGatherThreads) cp_async16(xs + i * E, src + i * E);
      for (int i = n / E * E + tid; i < n; i += kBinGatherThreads) xs[i] = src[i];
      cp_async_wait();
    } else {
      for (int i = tid; i < n; i += kBinGatherThreads) xs[i] = __ldg(src + i);
    }
    __syncthreads();
    // the next U quads are requested before the current ones are looked up
    const int64_t end = (int64_t)p_end * QP;
    uint2 w[2][U];
    auto request = [&](int64_t k, int s) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t kk = k + u * kBinGatherThreads;
        if (kk < end) w[s][u] = __ldcs(reinterpret_cast<const uint2*>(col + kk * kBinQuad));
      }
    };
    auto look_up = [&](int64_t k, int s) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t kk = k + u * kBinGatherThreads;
        if (kk < end) {
          uint32_t cc[4];
          V v[4];
          unpack16(w[s][u], cc);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = xs[cc[j]];
          st_quad(xg + kk * kBinQuad, v);
        }
      }
    };
    constexpr int STEP = U * kBinGatherThreads;
    int64_t k = (int64_t)p * QP + tid;
    request(k, 0);
    for (; k < end; k += 2 * STEP) {
      request(k + STEP, 1);
      look_up(k, 0);
      request(k + 2 * STEP, 0);
      look_up(k + STEP, 1);
    }
    p = p_end;
  }
}

// y of row block b = blockIdx.x.  ends[b * kBinSumThreads + t]: bit j is set where entry j of thread t's slice is the last of
// its row; row_slot[r]: where row r's last product is kept.  A thread adds up its slice, slot by slot, and a finished row's
// sum takes the place of its last product: by rows, most lanes would wait for the longest row of their warp.  What the slices
// before have of the row that a slice begins in the middle of comes from a segmented scan over the threads, and is added to the
// unrounded sum.
template <typename V>
__global__ void __launch_bounds__(kBinSumThreads, 2)
bins_sum_kernel(const V* __restrict__ data, const V* __restrict__ xg, const int32_t* __restrict__ place,
                const uint16_t* __restrict__ dst, const int32_t* __restrict__ block_pack, const int64_t* __restrict__ block_start,
                const uint32_t* __restrict__ ends, const uint16_t* __restrict__ row_slot, V* __restrict__ y) {
  extern __shared__ __align__(16) unsigned char b_smem[];
  V* s_prod = reinterpret_cast<V*>(b_smem);
  constexpr int S = bin_slice<V>();
  constexpr int QP = bin_pack<V>() / kBinQuad;
  constexpr int NW = kBinSumThreads / 32;
  __shared__ double s_tail[NW];
  __shared__ int s_any[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x;
  const int64_t r0 = block_start[2 * b], r1 = block_start[2 * b + 2];
  const int n = (int)(block_start[2 * b + 3] - block_start[2 * b + 1]);
  const int64_t q0 = (int64_t)block_pack[b] * QP + tid;
  int left = (int)((int64_t)block_pack[b + 1] * QP - q0);             // quads from this thread's first one on
  const uint32_t mask = __ldcs(ends + (int64_t)b * kBinSumThreads + tid);
  if (tid == 0) s_prod[bin_empty<V>()] = (V)0;
  {
    // (two or three packs of a thread on their way together: 235 and 238 us where one takes 225 us)
    const int32_t* at = place + q0 / QP;
    const uint16_t* to = dst + q0 * kBinQuad;
    const int within = (int)(q0 % QP);
    int from = left > 0 ? __ldcs(at) : 0;
    for (; left > 0; left -= kBinSumThreads) {
      V v[4];
      uint32_t d[4];
      ld_stream4(xg + ((int64_t)from * QP + within) * kBinQuad, v);
      unpack16(__ldcs(reinterpret_cast<const uint2*>(to)), d);
      at += kBinSumThreads / QP;
      to += kBinSumThreads * kBinQuad;
      if (left > kBinSumThreads) from = __ldcs(at);     // the next pack's place is on its way while this one is fetched
#pragma unroll
      for (int j = 0; j < 4; ++j) s_prod[d[j]] = v[j];
    }
  }
  // times the values, which lie in CSR order: entry i of the block is kept at bin_slot(i)
  {
    constexpr int D = sizeof(V) == 4 ? 8 : 4;          // values of a thread on their way together
    constexpr int STEP = kBinSumThreads + kBinSumThreads / S;
    const V* at = data + block_start[2 * b + 1] + tid;
    V* keep = s_prod + bin_slot<V>(tid);
    V a[D];
#pragma unroll
    for (int u = 0; u < D; ++u) a[u] = tid + u * kBinSumThreads < n ? __ldcs(at + u * kBinSumThreads) : (V)0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < S; k += D) {
#pragma unroll
      for (int u = 0; u < D; ++u) {
        if (tid + (k + u) * kBinSumThreads < n) keep[(k + u) * STEP] *= a[u];
        if (k + D < S) {
          const int next = k + D + u;
          a[u] = tid + next * kBinSumThreads < n ? __ldcs(at + next * kBinSumThreads) : (V)0;
        }
      }
    }
  }
  __syncthreads();
  V* slice = s_prod + tid * (S + 1);
  // float64: what every addition rounds off is kept beside the sum, or slot after slot would lose more than the lanes' tree of
  // the one-pass kernel (rows of 4 entries: rms error 8.9e-17 without it, 7.7e-17 in one pass)
  constexpr bool COMP = sizeof(V) == 8;
  double tail = 0, off = 0, head = 0;      // head: the first row that ends here, without what the slices before have of it
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const double v = (double)slice[j];
    if (COMP) {
      const double t = tail + v, u = t - tail;
      off += (tail - (t - u)) + (v - u);
      tail = t;
    } else {
      tail += v;
    }
    if (mask & (1u << j)) {
      if (COMP) tail += comp_term(tail, off);
      if ((mask & ((1u << j) - 1u)) == 0) head = tail;
      slice[j] = (V)tail;
      tail = 0;
      off = 0;
    }
  }
  if (COMP) tail += comp_term(tail, off);
  // inclusive segmented scan over the lanes: what lane l and the lanes before have of the row that goes on behind lane l
  const uint32_t closed = __ballot_sync(0xffffffffu, mask != 0);     // lanes in which a row ends
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(0xffffffffu, tail, o);
    // no row ends in the o lanes that the sum so far covers
    if (lane >= o && (closed >> (lane - o + 1) & ((1u << o) - 1u)) == 0) tail += t;
  }
  if (lane == 31) {
    s_tail[warp] = tail;
    s_any[warp] = closed != 0;
  }
  double carry = __shfl_up_sync(0xffffffffu, tail, 1);
  if (lane == 0) carry = 0;
  __syncthreads();
  if (mask != 0) {
    if ((closed & ((1u << lane) - 1u)) == 0)  // the row that goes on into this slice began in an earlier warp, or with this one
      for (int v = warp - 1; v >= 0; --v) {
        carry += s_tail[v];
        if (s_any[v]) break;
      }
    slice[__ffs(mask) - 1] = (V)(carry + head);
  }
  __syncthreads();
  // four rows of a thread at a time, from a multiple of four on; what is left at both ends one by one
  const int64_t a0 = (r0 + 3) & ~(int64_t)3, a1 = r1 & ~(int64_t)3;
  if (a0 < a1 && aligned_to_dev(y)) {
    for (int64_t r = a0 + 4 * tid; r < a1; r += 4 * kBinSumThreads) {
      uint32_t d[4];
      unpack16(__ldcs(reinterpret_cast<const uint2*>(row_slot + r)), d);
      V v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = s_prod[d[j]];
      st_quad(y + r, v);
    }
    const int64_t r = tid < 4 ? r0 + tid : a1 + (tid - 4);
    if (tid < 8 && (tid < 4 ? r < a0 : r < r1)) y[r] = s_prod[row_slot[r]];
  } else {
    for (int64_t r = r0 + tid; r < r1; r += kBinSumThreads) y[r] = s_prod[row_slot[r]];
  }
}

// ---- building the layout ---------------------------------------------------------------------------------------------
// entries of block b in every chunk
template <typename P>
__global__ void __launch_bounds__(kBinBuildThreads)
bins_count_kernel(const int32_t* __restrict__ idx, const P* __restrict__ ptr, const int32_t* __restrict__ block_row,
                  int n_chunks, int chunk_cols, int32_t* __restrict__ counts) {
  extern __shared__ int32_t s_cells[];
  const int b = blockIdx.x;
  for (int c = threadIdx.x; c < n_chunks; c += kBinBuildThreads) s_cells[c] = 0;
  __syncthreads();
  const int64_t lo = (int64_t)ptr[block_row[b]], hi = (int64_t)ptr[block_row[b + 1]];
  for (int64_t i = lo + threadIdx.x; i < hi; i += kBinBuildThreads)
    atomicAdd(&s_cells[(uint32_t)idx[i] / (uint32_t)chunk_cols], 1);
  __syncthreads();
  for (int c = threadIdx.x; c < n_chunks; c += kBinBuildThreads) counts[(int64_t)b * n_chunks + c] = s_cells[c];
}

// Every entry of block b to its unit, in any order inside the unit (the sum puts the products back in CSR order); what is
// left of a unit's last pack is filled with first columns that no row reads.  unit_chunk[b * n_chunks + c], unit_block[...]: first
// pack of the unit in chunk order and in block order; the last of each array is the number of packs.
template <typename V, typename P>
__global__ void __launch_bounds__(kBinBuildThreads)
bins_place_kernel(const int32_t* __restrict__ idx, const P* __restrict__ ptr,
                  const int32_t* __restrict__ block_row, int n_chunks, int chunk_cols, const int32_t* __restrict__ unit_chunk,
                  const int32_t* __restrict__ unit_block, uint16_t* __restrict__ col,
                  int32_t* __restrict__ place, uint16_t* __restrict__ dst, uint32_t* __restrict__ ends,
                  uint16_t* __restrict__ row_slot) {
  constexpr int PACK = bin_pack<V>(), S = bin_slice<V>();
  extern __shared__ int32_t s_cells[];
  __shared__ uint32_t s_ends[kBinSumThreads];
  const int b = blockIdx.x;
  const int32_t* cm = unit_chunk + (int64_t)b * n_chunks;
  const int32_t* bm = unit_block + (int64_t)b * n_chunks;
  for (int c = threadIdx.x; c < n_chunks; c += kBinBuildThreads) s_cells[c] = 0;
  for (int t = threadIdx.x; t < kBinSumThreads; t += kBinBuildThreads) s_ends[t] = 0;
  __syncthreads();
  const int r0 = block_row[b], r1 = block_row[b + 1];
  const int64_t lo = (int64_t)ptr[r0], hi = (int64_t)ptr[r1];
  for (int r = r0 + (int)threadIdx.x; r < r1; r += kBinBuildThreads) {
    const int64_t e = (int64_t)ptr[r + 1];
    int slot = bin_empty<V>();
    if (e > (int64_t)ptr[r]) {
      const int last = (int)(e - 1 - lo);
      atomicOr(&s_ends[last / S], 1u << (last % S));
      slot = bin_slot<V>(last);
    }
    row_slot[r] = (uint16_t)slot;
  }
  for (int64_t i = lo + threadIdx.x; i < hi; i += kBinBuildThreads) {
    const uint32_t j = (uint32_t)idx[i], c = j / (uint32_t)chunk_cols;
    const int rank = atomicAdd(&s_cells[c], 1);
    col[(int64_t)cm[c] * PACK + rank] = (uint16_t)(j - c * (uint32_t)chunk_cols);
    dst[(int64_t)bm[c] * PACK + rank] = (uint16_t)bin_slot<V>((int)(i - lo));
  }
  __syncthreads();
  for (int c = threadIdx.x; c < n_chunks; c += kBinBuildThreads) {
    const int n = s_cells[c], packs = (n + PACK - 1) / PACK;
    for (int k = 0; k < packs; ++k) place[bm[c] + k] = cm[c] + k;
    for (int k = n; k < packs * PACK; ++k) {
      col[(int64_t)cm[c] * PACK + k] = 0;
      dst[(int64_t)bm[c] * PACK + k] = (uint16_t)bin_fill<V>();
    }
  }
  for (int t = threadIdx.x; t < kBinSumThreads; t += kBinBuildThreads) ends[(int64_t)b * kBinSumThreads + t] = s_ends[t];
}

static int bins_check_shape(int vtype, int ptype, int32_t n_blocks, int32_t n_chunks, int32_t chunk_cols, int64_t n_cols) {
  if ((vtype != FSB_F32 && vtype != FSB_F64) || (ptype != FSB_I32 && ptype != FSB_I64)) return FSB_EINVAL;
  if (n_blocks < 0 || n_chunks <= 0 || chunk_cols <= 0 || n_cols < 0) return FSB_EINVAL;
  if (chunk_cols % 4 != 0 || chunk_cols > 65536 || n_chunks > kBinMaxChunks || n_cols >= INT32_MAX) return FSB_ERANGE;
  if ((int64_t)n_chunks * chunk_cols < n_cols || (int64_t)(n_chunks - 1) * chunk_cols >= n_cols) return FSB_EINVAL;
  return FSB_OK;
}

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_spmv_bins_max_chunks(void) { return kBinMaxChunks; }
extern "C" int fsb_spmv_bins_chunk_cols(int vtype) { return vtype == FSB_F32 ? 49152 : vtype == FSB_F64 ? 24576 : 0; }
extern "C" int fsb_spmv_bins_cap(int vtype) { return vtype == FSB_F32 ? bin_cap<float>() : vtype == FSB_F64 ? bin_cap<double>() : 0; }
extern "C" int fsb_spmv_bins_pack(int vtype) { return vtype == FSB_F32 ? bin_pack<float>() : vtype == FSB_F64 ? bin_pack<double>() : 0; }
extern "C" int fsb_spmv_bins_ends(void) { return kBinSumThreads; }

extern "C" int fsb_spmv_bins_count(int ptype, const int32_t* indices, const void* indptr, const int32_t* block_row,
                                   int32_t n_blocks, int32_t n_chunks, int32_t chunk_cols, int64_t n_cols, int32_t* counts,
                                   void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  const int rc = bins_check_shape(FSB_F32, ptype, n_blocks, n_chunks, chunk_cols, n_cols);
  if (rc != FSB_OK) return rc;
  if (n_blocks == 0) return FSB_OK;
  if (!indices || !indptr || !block_row || !counts) return FSB_EINVAL;
  const size_t smem = (size_t)n_chunks * sizeof(int32_t);
  if (ptype == FSB_I32)
    bins_count_kernel<int32_t><<<(unsigned)n_blocks, kBinBuildThreads, smem, st>>>(indices, (const int32_t*)indptr, block_row,
                                                                                   n_chunks, chunk_cols, counts);
  else
    bins_count_kernel<int64_t><<<(unsigned)n_blocks, kBinBuildThreads, smem, st>>>(indices, (const int64_t*)indptr, block_row,
                                                                                   n_chunks, chunk_cols, counts);
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

extern "C" int fsb_spmv_bins_place(int vtype, int ptype, const int32_t* indices, const void* indptr,
                                   const int32_t* block_row, int32_t n_blocks, int32_t n_chunks, int32_t chunk_cols,
                                   int64_t n_cols, const int32_t* unit_chunk, const int32_t* unit_block,
                                   uint16_t* col, int32_t* place, uint16_t* dst, uint32_t* ends, uint16_t* row_slot,
                                   void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  const int rc = bins_check_shape(vtype, ptype, n_blocks, n_chunks, chunk_cols, n_cols);
  if (rc != FSB_OK) return rc;
  if (n_blocks == 0) return FSB_OK;
  if (!indices || !indptr || !block_row || !unit_chunk || !unit_block || !col || !place || !dst || !ends ||
      !row_slot)
    return FSB_EINVAL;
  const size_t smem = (size_t)n_chunks * sizeof(int32_t);
#define FSB_BINS_PLACE(V_, P_)                                                                                         \
  bins_place_kernel<V_, P_><<<(unsigned)n_blocks, kBinBuildThreads, smem, st>>>(                                       \
      indices, (const P_*)indptr, block_row, n_chunks, chunk_cols, unit_chunk, unit_block, col, \
      place, dst, ends, row_slot)
  if (vtype == FSB_F32) {
    if (ptype == FSB_I32) FSB_BINS_PLACE(float, int32_t); else FSB_BINS_PLACE(float, int64_t);
  } else {
    if (ptype == FSB_I32) FSB_BINS_PLACE(double, int32_t); else FSB_BINS_PLACE(double, int64_t);
  }
#undef FSB_BINS_PLACE
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

extern "C" int fsb_spmv_csr_bins(int vtype, const uint16_t* col, const int32_t* place, const uint16_t* dst, const uint32_t* ends,
                                 const uint16_t* row_slot, const int32_t* chunk_pack, const int32_t* block_pack,
                                 const int64_t* block_start, const void* data, int32_t n_blocks, int32_t n_chunks,
                                 int32_t chunk_cols, int64_t n_packs, void* xg, size_t xg_bytes, const void* x, void* y,
                                 int64_t n_rows, int64_t n_cols, void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  int rc = bins_check_shape(vtype, FSB_I32, n_blocks, n_chunks, chunk_cols, n_cols);
  if (rc != FSB_OK) return rc;
  if (n_rows < 0 || n_packs < 0) return FSB_EINVAL;
  if (n_rows >= INT32_MAX || n_packs >= INT32_MAX) return FSB_ERANGE;
  if (n_rows == 0) return FSB_OK;
  if (n_blocks == 0 || !col || !place || !dst || !ends || !row_slot || !chunk_pack || !block_pack || !block_start || !data ||
      !xg || !x || !y)
    return FSB_EINVAL;
  const size_t sv = vtype == FSB_F32 ? 4 : 8;
  if (xg_bytes < (size_t)n_packs * 32) return FSB_ESCRATCH;
  if (!aligned_to(col, 16) || !aligned_to(dst, 16) || !aligned_to(row_slot, 16) || !aligned_to(xg, 32) ||
      !aligned_to(data, sv) || !aligned_to(x, sv) || !aligned_to(y, sv))
    return FSB_EALIGN;
  const size_t gather_smem = (size_t)chunk_cols * sv;
  const size_t sum_smem = (size_t)(vtype == FSB_F32 ? bin_fill<float>() + 1 : bin_fill<double>() + 1) * sv;
  if (gather_smem > 226 * 1024) return FSB_ERANGE;
  FSB_WALK_FIRST(check_bins(vtype, col, place, dst, ends, row_slot, chunk_pack, block_pack, block_start, n_blocks, n_chunks,
                            chunk_cols, n_packs, n_rows, n_cols, st));
  int sms = 0;
  rc = sm_count(&sms);
  if (rc != FSB_OK) return rc;
  cudaError_t e;
#define FSB_BINS_RUN(V_)                                                                                                    \
  do {                                                                                                                      \
    e = cudaFuncSetAttribute(bins_gather_kernel<V_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gather_smem);        \
    if (e != cudaSuccess) return cuda_rc(e);                                                                                \
    e = cudaFuncSetAttribute(bins_sum_kernel<V_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem);              \
    if (e != cudaSuccess) return cuda_rc(e);                                                                                \
    bins_gather_kernel<V_><<<(unsigned)sms, kBinGatherThreads, gather_smem, st>>>(col, chunk_pack, n_chunks, chunk_cols,    \
                                                                                  (const V_*)x, n_cols, (V_*)xg);           \
    FSB_RETURN_IF_LAUNCH_FAILED();                                                                                          \
    bins_sum_kernel<V_><<<(unsigned)n_blocks, kBinSumThreads, sum_smem, st>>>(                                              \
        (const V_*)data, (const V_*)xg, place, dst, block_pack, block_start, ends, row_slot, (V_*)y);                       \
  } while (0)
  if (vtype == FSB_F32) FSB_BINS_RUN(float); else FSB_BINS_RUN(double);
#undef FSB_BINS_RUN
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}
