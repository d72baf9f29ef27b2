// CSR SDDMM for sm_100a: out[p] = alpha * dot(X[row(p), :], Y[col(p), :]) + beta * data[p] for every entry p of a
// CSR pattern (X is n_rows x K, Y is n_cols x K, both row-major with a row stride).
//
// A group of LG lanes (LG = K / VW rounded up to a power of two, at most 32; VW = elements per 128-bit access)
// owns batches of 8 consecutive entries.  A CTA first copies the column and row ids of its tile (about 1024
// entries; the row of an entry comes from the row-id array built at prepare time, 4 bytes per entry) into shared
// memory, so that the only trip to global memory inside the loop over batches is the gather; every lane then
// requests its slice of all eight rows of Y through the read-only path before it uses any of them, so a group has
// eight gathers in flight; a batch that lies inside one row needs one slice of X's row, one that meets two rows a slice of
// each, a batch that crosses more loads a slice of X per entry.  Each lane ends with eight partial sums (one per entry);
// they are reduced across the group by a transposed exchange (halve the entries a lane is responsible for at every
// step: 7 shuffles for 8 entries x 8 lanes instead of 24), and put into shared memory, from where the tile's results leave
// in order.  Rows of X longer than LG * VW elements are walked in several steps.  The summation order is fixed, so results are bit-reproducible.
// CUDA-core work on purpose: one dot product per entry over gathered rows is about 0.5 flop per byte.
#include "fsb_common.cuh"

namespace fsb {

constexpr int kSdThreads = 256;
constexpr int kSdBatch = 8;   // consecutive entries one group handles

// Resident CTAs the register budget is set for: 64 registers, but 80 for 16-byte accesses (float64, 131072 rows of 16, K 200: 476 us,
// with 64 registers 603 us; float32, 69905 rows of 30, K 60: 46 and 67 us, 87381 rows of 48, K 16 37 and 46 us), except for groups of
// one lane or two, whose CTAs handle one batch a group (262144 rows of 16, K 8: 47 and 40 us), and for rows that take several steps:
// with 64 the gathers of a step wait for one another (float32, 2048 rows of 16, K 160: 15.4 us, 8.9 us; 209715 rows of 5, K 129: 161 us, 140 us).
__host__ __device__ constexpr int sddmm_ctas(int vw, size_t size, int LG, bool multi) {
  return (vw * (int)size == 16 && !(size == 4 && LG <= 2)) || multi ? 3 : 4;
}

// entries one CTA handles: J passes of (threads / LG) groups x 8 entries, about 1024 (262144 rows of 6, K 8: 17.3 us, with 2048
// 20.3 us, a last wave that is a quarter full; 2^19 rows of 16, K 64: 251 us, with 512 265 us)
__host__ __device__ constexpr int sddmm_passes(int LG) {
  const int per_pass = (kSdThreads / LG) * kSdBatch;
  return per_pass >= 1024 ? 1 : (1024 / per_pass < 8 ? 1024 / per_pass : 8);
}
__host__ __device__ constexpr int sddmm_tile(int LG) { return (kSdThreads / LG) * kSdBatch * sddmm_passes(LG); }

// row `id` of a matrix whose rows are `stride` bytes apart, from `base` on: one wide multiply-add and one for the high word
template <typename V>
__device__ __forceinline__ const V* row_at(const char* base, int32_t id, uint64_t stride) {
  return reinterpret_cast<const V*>(base + (uint64_t)(uint32_t)id * stride);
}

// dot product of what one lane holds of two rows (one product after the other: pairs of floats in packed multiply-adds end with one more
// addition of two sums, 2 % more rms error at K 8, 16, 100 and 128)
template <typename V, int VW>
__device__ __forceinline__ V lane_dot(const V (&a)[VW], const V (&b)[VW]) {
  V s = a[0] * b[0];
#pragma unroll
  for (int i = 1; i < VW; ++i) s = fma(a[i], b[i], s);
  return s;
}
// The form of a batch of eight entries: bit e is set where entry e lies in the row of the first one; kSdOne: all of them do;
// kSdTwo: the others lie in the row of the last one.
//
// Row ids never decrease along a CSR pattern.  Most batches meet one row of X or two: a slice of each then serves all eight
// gathers, which leave together.  Where a batch meets more rows every entry gets its own slice of X, four entries at a time
// (reloading X only where the row changes would make each gather wait for the previous entry's arithmetic).
// vote (two to four groups in a warp, 16-byte gathers): the groups agree on the form that all of their batches fit, as a
// warp whose groups differ runs one form after the other (2^19 rows of 16, K 64, Zipf lengths: 392 us without it, 292 us with
// it; float64, 2^18 such rows, K 32: 204 us, 146 us).  With eight groups and more, or smaller gathers, agreeing costs more than
// it saves (K 16: 98 us, with it 109 us; K 33: 558 us, 614 us), and a batch of one row takes the form of two.
//
// What bounded the kernel before its present shape was its own arithmetic: 340 warp instructions for 16 entries (2^19 rows of
// 16, K 64, float32), of which the gathers, the products and their sums need about a third; 4.8 of the 10.2 cycles that a
// warp took per instruction were spent waiting for memory.  So the forms are worked out once per batch while the ids are staged
// (not by every lane of the group), rows are found by one wide multiply-add from a stride in bytes, and the results leave
// through shared memory with alpha, beta and `data` at the end.
// That case 254 us before, 234 us now, Poisson rows 290 and 249; 131072 rows of 32: 108 us, 95 us; K 33: 554 us, 362 us; float64,
// 2^18 rows of 16, K 32: 131 us, 120 us.  A group that walks whole rows instead, as the SpMM kernel
// does, with the next row's slice of X on its way: 309 us (groups of a warp wait for the longest row among theirs).
constexpr uint32_t kSdOne = 1u << 8, kSdTwo = 1u << 9;
template <typename V>
__host__ __device__ constexpr bool sddmm_vote(int VW, int LG) { return VW * (int)sizeof(V) == 16 && (LG == 8 || LG == 16); }

// MULTI: rows of X longer than one access per lane of a warp, walked in several steps.  With 16-byte accesses (WIDE) products are then
// added to the sums one by one, as the pairs of lane_dot want registers of their own; and float32 has no form for batches of two
// rows, whose second slice of X finds no room beside eight gathers: the row ids themselves tell the two forms that are left apart.
// us, as for one step / here: float32, 65536 rows of 16, K 160 98 / 72; 2048 rows of 16, K 200 15.5 / 9.0; float64, 65536 rows of
// 16, K 72 97 / 74, Poisson rows 90 / 74.
template <typename V, int VW, int LG, bool MULTI>
__global__ void __launch_bounds__(kSdThreads, sddmm_ctas(VW, sizeof(V), LG, MULTI))
sddmm_kernel(const int32_t* __restrict__ indices, const int32_t* __restrict__ row_ids, const V* __restrict__ X,
             int64_t ldx, const V* __restrict__ Y, int64_t ldy, const V* data, V* out,
             int64_t nnz, int k_dim, V alpha, V beta, int ids_aligned) {
  constexpr int E = kSdBatch;
  constexpr int step = LG * VW;
  constexpr int kGroups = kSdThreads / LG;
  constexpr int J = sddmm_passes(LG);
  constexpr int T = sddmm_tile(LG);
  constexpr int kHeld = (LG >= E) ? 1 : E / LG;   // results a lane ends up with
  constexpr int kDup = (LG > E) ? LG / E : 1;     // lanes that end up with the same result
  constexpr bool VOTE = sddmm_vote<V>(VW, LG);
  constexpr bool ONE = VOTE || LG == 32;          // batches of one row have a form of their own
  constexpr bool WIDE = MULTI && VW * (int)sizeof(V) == 16;
  constexpr bool TWO = !WIDE || sizeof(V) == 8;   // ... and batches of two
  __shared__ __align__(16) int32_t s_cols[T];
  __shared__ __align__(16) int32_t s_rows[T];
  __shared__ __align__(16) V s_out[T];
  __shared__ uint32_t s_form[!TWO ? 1 : T / E];

  // the tile's column and row ids go to shared memory once (entries past the end repeat the last one; they are
  // never stored), so that the loop below has one trip to global memory per batch: the gathers
  const int64_t tile0 = (int64_t)blockIdx.x * T;
  const int64_t left = nnz - tile0;
  if (left >= T && ids_aligned) {
    for (int i = threadIdx.x; i < T / 4; i += kSdThreads) {
      reinterpret_cast<int4*>(s_cols)[i] = __ldcs(reinterpret_cast<const int4*>(indices + tile0) + i);
      reinterpret_cast<int4*>(s_rows)[i] = __ldcs(reinterpret_cast<const int4*>(row_ids + tile0) + i);
    }
  } else {
    for (int i = threadIdx.x; i < T; i += kSdThreads) {
      const int64_t p = tile0 + (i < left ? i : left - 1);
      s_cols[i] = __ldg(indices + p);
      s_rows[i] = __ldg(row_ids + p);
    }
  }
  __syncthreads();
  if constexpr (TWO) {
    for (int b = threadIdx.x; b < T / E; b += kSdThreads) {
      const int32_t* r = s_rows + b * E;
      const int32_t row_a = r[0], row_b = r[E - 1];
      uint32_t form = row_a == row_b ? kSdOne : 0;
      bool two = true;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        two = two && (r[e] == row_a || r[e] == row_b);
        form |= (r[e] == row_a ? 1u : 0u) << e;
      }
      s_form[b] = form | (two ? kSdTwo : 0);
    }
    __syncthreads();
  }

  const int lane = threadIdx.x & (LG - 1);
  const int group = threadIdx.x / LG;
  const int k0 = lane * VW;
  const char* Xk = reinterpret_cast<const char*>(X + k0);
  const char* Yk = reinterpret_cast<const char*>(Y + k0);
  const uint64_t xs = (uint64_t)ldx * sizeof(V), ys = (uint64_t)ldy * sizeof(V);
  const unsigned gmask = LG == 32 ? 0xffffffffu : (((1u << LG) - 1u) << ((threadIdx.x & 31) & ~(LG - 1)));
  unsigned active = 0xffffffffu;   // lanes of the warp that have a batch
#pragma unroll 1
  for (int j = 0; j < J; ++j) {
    const int local = (j * kGroups + group) * E;
    if constexpr (VOTE) active = __ballot_sync(active, local < left);
    if (local >= left) break;   // whole groups leave together: the shuffles below stay inside a group
    V acc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = (V)0;
    uint32_t form;
    if constexpr (!TWO) form = s_rows[local] == s_rows[local + E - 1] ? kSdOne : 0;
    else form = s_form[local / E];
    bool one = (form & kSdOne) != 0, two = (form & kSdTwo) != 0;
    if constexpr (VOTE) {
      one = __all_sync(active, one);
      two = __all_sync(active, two);
    }
    const int32_t* cols = s_cols + local;
    const int32_t* rows = s_rows + local;
    if (WIDE && one) {
      const V *xp = X + k0 + (int64_t)rows[0] * ldx, *yp = Y + k0;
      for (int k = k0; k < k_dim; k += step, xp += step, yp += step) {
        V xa[VW], yv[E][VW];
        ld_dense<V, VW>(xp, xa);
#pragma unroll
        for (int e = 0; e < E; ++e) ld_dense<V, VW>(yp + (int64_t)cols[e] * ldy, yv[e]);
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
          for (int i = 0; i < VW; ++i) acc[e] += xa[i] * yv[e][i];
      }
    } else if (ONE && one) {
      const char *xp = reinterpret_cast<const char*>(row_at<V>(Xk, rows[0], xs)), *yp = Yk;
      for (int k = k0; k < k_dim; k += step, xp += step * sizeof(V), yp += step * sizeof(V)) {
        V xa[VW], yv[E][VW];
        ld_dense<V, VW>(reinterpret_cast<const V*>(xp), xa);
#pragma unroll
        for (int e = 0; e < E; ++e) ld_dense<V, VW>(row_at<V>(yp, cols[e], ys), yv[e]);
        // (four floats onto the sum itself: 2^19 rows of 16, K 64 234 us, as a product of its own 235; 32768 rows of 16, K 64 1 % less)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if constexpr (sizeof(V) == 4 && VW == 4) {
#pragma unroll
            for (int i = 0; i < VW; ++i) acc[e] = fma(xa[i], yv[e][i], acc[e]);
          } else {
            acc[e] += lane_dot(xa, yv[e]);
          }
        }
      }
    } else if (TWO && two) {
      const char *xp = reinterpret_cast<const char*>(row_at<V>(Xk, rows[0], xs)), *yp = Yk;
      const char *xq = reinterpret_cast<const char*>(row_at<V>(Xk, rows[E - 1], xs));
      for (int k = k0; k < k_dim; k += step, xp += step * sizeof(V), xq += step * sizeof(V), yp += step * sizeof(V)) {
        V xa[VW], xb[VW], yv[E][VW];
        ld_dense<V, VW>(reinterpret_cast<const V*>(xp), xa);
        ld_dense<V, VW>(reinterpret_cast<const V*>(xq), xb);
#pragma unroll
        for (int e = 0; e < E; ++e) ld_dense<V, VW>(row_at<V>(yp, cols[e], ys), yv[e]);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if constexpr (WIDE) {
            if (form >> e & 1) {
#pragma unroll
              for (int i = 0; i < VW; ++i) acc[e] += xa[i] * yv[e][i];
            } else {
#pragma unroll
              for (int i = 0; i < VW; ++i) acc[e] += xb[i] * yv[e][i];
            }
          } else {
            V t;                     // (a branch of the group; choosing the slice first takes an instruction per element)
            if (form >> e & 1) t = lane_dot(xa, yv[e]);
            else t = lane_dot(xb, yv[e]);
            acc[e] += t;
          }
        }
      }
    } else {
      const char *xp = Xk, *yp = Yk;
      for (int k = k0; k < k_dim; k += step, xp += step * sizeof(V), yp += step * sizeof(V)) {
#pragma unroll
        for (int h = 0; h < E; h += E / 2) {
          V xv[E / 2][VW], yv[E / 2][VW];
#pragma unroll
          for (int e = 0; e < E / 2; ++e) {
            ld_dense<V, VW>(row_at<V>(xp, rows[h + e], xs), xv[e]);
            ld_dense<V, VW>(row_at<V>(yp, cols[h + e], ys), yv[e]);
          }
#pragma unroll
          for (int e = 0; e < E / 2; ++e) acc[h + e] += lane_dot(xv[e], yv[e]);
        }
      }
    }

    // transposed reduction: at each step a lane hands half of its entries to its partner and takes the partner's
    // partial sums of the half it keeps; once one entry is left the remaining steps are plain butterfly adds
    int held = E;
#pragma unroll
    for (int off = LG >> 1; off >= 1; off >>= 1) {
      if (held > 1) {
        held >>= 1;
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < E / 2; ++i) {
          if (i < held) {
            const V send = upper ? acc[i] : acc[i + held];
            const V keep = upper ? acc[i + held] : acc[i];
            acc[i] = keep + __shfl_xor_sync(gmask, send, off, LG);
          }
        }
      } else {
        acc[0] += __shfl_xor_sync(gmask, acc[0], off, LG);
      }
    }
    // a lane now holds kHeld consecutive entries; where LG > E, kDup lanes hold the same sum
    if (lane % kDup == 0) {
#pragma unroll
      for (int i = 0; i < kHeld; ++i) s_out[local + (lane / kDup) * kHeld + i] = acc[i];
    }
  }
  __syncthreads();
  // results leave in order, with `data`, which may be the same array
  for (int i = threadIdx.x; i < T && i < left; i += kSdThreads) {
    V v = s_out[i] * alpha;
    if (data != nullptr) v += __ldcs(data + tile0 + i) * beta;
    __stcs(out + tile0 + i, v);
  }
}

// Which rows of several steps take the instance for them: not those of float32 in accesses of 8 bytes (65536 rows of 16, K 130: 65 us
// with 80 registers, 59 with 64); of single elements not where four CTAs an SM hold all tiles and three do not (float32, 16384 rows of
// 16, K 65: 15 % less with 64), nor where there are more tiles than that and most batches
// lie in one row or two (float32, 65536 rows of 16, K 129: 71 us, 66; but 209715 rows of 5 140, 161; float64 from more tiles on:
// 262144 rows of 16, K 33 275, 241, and 25000 such rows 26.5, 27.2).
template <typename V, int VW>
static bool sddmm_multi(int k_dim, int64_t n_rows, int64_t nnz) {
  constexpr bool SINGLE = sizeof(V) == 4;
  if (k_dim <= 32 * VW || (SINGLE && VW == 2)) return false;
  if (sddmm_ctas(VW, sizeof(V), 32, false) == sddmm_ctas(VW, sizeof(V), 32, true)) return true;
  int sms = 0;
  if (sm_count(&sms) != FSB_OK) return true;
  const int64_t tiles = (nnz + sddmm_tile(32) - 1) / sddmm_tile(32);
  if (tiles > 3 * sms && tiles <= 4 * sms) return false;
  return !(VW == 1 && tiles > (SINGLE ? 4 : 14) * sms && nnz >= 12 * n_rows);
}

template <typename V, int VW>
static int sddmm_launch(int LG, int64_t n_rows, unsigned blocks, cudaStream_t st, const int32_t* indices, const int32_t* row_ids,
                        const V* X, int64_t ldx, const V* Y, int64_t ldy, const V* data, V* out, int64_t nnz,
                        int k_dim, V alpha, V beta, int ids_aligned) {
#define FSB_SDDMM_LAUNCH(LG_, MULTI_)                                                                            \
  sddmm_kernel<V, VW, LG_, MULTI_><<<blocks, kSdThreads, 0, st>>>(indices, row_ids, X, ldx, Y, ldy, data, out,   \
                                                                  nnz, k_dim, alpha, beta, ids_aligned)
#define FSB_SDDMM_CASE(LG_)                                                                                      \
  case LG_:                                                                                                      \
    FSB_SDDMM_LAUNCH(LG_, false);                                                                                \
    break
  switch (LG) {
    FSB_SDDMM_CASE(1);
    FSB_SDDMM_CASE(2);
    FSB_SDDMM_CASE(4);
    FSB_SDDMM_CASE(8);
    FSB_SDDMM_CASE(16);
    case 32:
      if (sddmm_multi<V, VW>(k_dim, n_rows, nnz)) FSB_SDDMM_LAUNCH(32, true);
      else FSB_SDDMM_LAUNCH(32, false);
      break;
    default: return FSB_EINVAL;
  }
#undef FSB_SDDMM_CASE
#undef FSB_SDDMM_LAUNCH
  FSB_RETURN_IF_LAUNCH_FAILED();
  return FSB_OK;
}

template <typename V>
static int sddmm_typed(const int32_t* indices, const int32_t* row_ids, const void* X, int64_t ldx, const void* Y,
                       int64_t ldy, const void* data, void* out, int64_t n_rows, int64_t nnz, int k_dim, double alpha, double beta,
                       cudaStream_t st) {
  constexpr int VMAX = 16 / sizeof(V);
  int vw = VMAX;
  while (vw > 1 && !(k_dim % vw == 0 && ldx % vw == 0 && ldy % vw == 0 && aligned_to(X, vw * sizeof(V)) &&
                     aligned_to(Y, vw * sizeof(V))))
    vw >>= 1;
  const int need = (k_dim + vw - 1) / vw;
  int LG = 1;
  while (LG < 32 && LG < need) LG <<= 1;
  const int tile = LG == 1 ? sddmm_tile(1) : LG == 2 ? sddmm_tile(2) : LG == 4 ? sddmm_tile(4) : LG == 8 ? sddmm_tile(8)
                   : LG == 16 ? sddmm_tile(16) : sddmm_tile(32);
  const int64_t blocks = (nnz + tile - 1) / tile;
  if (blocks >= INT32_MAX) return FSB_ERANGE;
  const int ids_aligned = aligned_to(indices, 16) && aligned_to(row_ids, 16);
  const V* Xv = (const V*)X;
  const V* Yv = (const V*)Y;
  const V* dv = (const V*)data;
  V* ov = (V*)out;
  if constexpr (VMAX == 4) {
    if (vw == 4)
      return sddmm_launch<V, 4>(LG, n_rows, (unsigned)blocks, st, indices, row_ids, Xv, ldx, Yv, ldy, dv, ov, nnz, k_dim,
                                (V)alpha, (V)beta, ids_aligned);
  }
  if (vw == 2)
    return sddmm_launch<V, 2>(LG, n_rows, (unsigned)blocks, st, indices, row_ids, Xv, ldx, Yv, ldy, dv, ov, nnz, k_dim,
                              (V)alpha, (V)beta, ids_aligned);
  return sddmm_launch<V, 1>(LG, n_rows, (unsigned)blocks, st, indices, row_ids, Xv, ldx, Yv, ldy, dv, ov, nnz, k_dim,
                            (V)alpha, (V)beta, ids_aligned);
}

}  // namespace fsb

using namespace fsb;

extern "C" int fsb_sddmm_csr(int vtype, const int32_t* indices, const int32_t* row_ids, const void* X, int64_t ldx,
                             const void* Y, int64_t ldy, const void* data, void* out, int64_t n_rows, int64_t n_cols,
                             int64_t nnz, int64_t k_dim, double alpha, double beta, void* stream_) {
  cudaStream_t st = static_cast<cudaStream_t>(stream_);
  if (vtype != FSB_F32 && vtype != FSB_F64) return FSB_EINVAL;
  if (n_rows < 0 || n_cols < 0 || nnz < 0 || k_dim < 0) return FSB_EINVAL;
  if (n_rows >= INT32_MAX || n_cols >= INT32_MAX || k_dim >= (1 << 24)) return FSB_ERANGE;
  if (nnz == 0) return FSB_OK;
  if (indices == nullptr || row_ids == nullptr || out == nullptr) return FSB_EINVAL;
  if (k_dim > 0 && (X == nullptr || Y == nullptr || ldx < k_dim || ldy < k_dim)) return FSB_EINVAL;
  const size_t sv = vtype == FSB_F32 ? 4 : 8;
  if (!aligned_to(X, sv) || !aligned_to(Y, sv) || !aligned_to(out, sv) || !aligned_to(data, sv) ||
      !aligned_to(indices, 4) || !aligned_to(row_ids, 4))
    return FSB_EALIGN;
  FSB_WALK_FIRST(check_entry_ids(indices, row_ids, n_rows, n_cols, nnz, st));
  if (vtype == FSB_F32)
    return sddmm_typed<float>(indices, row_ids, X, ldx, Y, ldy, data, out, n_rows, nnz, (int)k_dim, alpha, beta, st);
  return sddmm_typed<double>(indices, row_ids, X, ldx, Y, ldy, data, out, n_rows, nnz, (int)k_dim, alpha, beta, st);
}
