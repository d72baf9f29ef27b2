// How the kernels that read matrix and vector as they are stored compute with a value type: accumulator, product, sum, exchange
// between lanes.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace fsb {

__device__ __forceinline__ float w_zero(float*) { return 0.f; }
__device__ __forceinline__ double w_zero(double*) { return 0.0; }
__device__ __forceinline__ float2 w_zero(float2*) { return make_float2(0.f, 0.f); }
__device__ __forceinline__ double2 w_zero(double2*) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ float w_add(float a, float b) { return a + b; }
__device__ __forceinline__ double w_add(double a, double b) { return a + b; }
__device__ __forceinline__ float2 w_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 w_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float w_down(float v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }
__device__ __forceinline__ float2 w_down(float2 v, int o) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ double2 w_down(double2 v, int o) {
  return make_double2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o));
}
template <typename T>
__device__ __forceinline__ T w_xor(T v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ float2 w_xor(float2 v, int o) { return make_float2(w_xor(v.x, o), w_xor(v.y, o)); }
__device__ __forceinline__ double2 w_xor(double2 v, int o) { return make_double2(w_xor(v.x, o), w_xor(v.y, o)); }

// Products and sums in the accumulator type, every element of y rounded once.  `prod` is the product in the accumulator
// type: exact for the half precisions, a multiplication and a fused multiply-add per component for complex values.
template <typename S> struct StoredOps;
template <>
struct StoredOps<__half> {
  typedef float A;
  typedef float R;
  static __device__ __forceinline__ A prod(__half a, __half b) { return __half2float(a) * __half2float(b); }
  static __device__ __forceinline__ void fma(A& acc, __half a, __half b) {
    acc = fmaf(__half2float(a), __half2float(b), acc);
  }
  static __device__ __forceinline__ __half narrow(A v) { return __float2half_rn(v); }
};
template <>
struct StoredOps<__nv_bfloat16> {
  typedef float A;
  typedef float R;
  static __device__ __forceinline__ A prod(__nv_bfloat16 a, __nv_bfloat16 b) {
    return __bfloat162float(a) * __bfloat162float(b);
  }
  static __device__ __forceinline__ void fma(A& acc, __nv_bfloat16 a, __nv_bfloat16 b) {
    acc = fmaf(__bfloat162float(a), __bfloat162float(b), acc);
  }
  static __device__ __forceinline__ __nv_bfloat16 narrow(A v) { return __float2bfloat16_rn(v); }
};
template <typename C2, typename Real>
struct StoredComplex {
  typedef C2 A;
  typedef Real R;
  static __device__ __forceinline__ A prod(C2 a, C2 b) {
    C2 r;
    r.x = ::fma(a.x, b.x, -(a.y * b.y));
    r.y = ::fma(a.x, b.y, a.y * b.x);
    return r;
  }
  // one rounding at the size of the sum: rows of 700 entries, rms error 1.11 times as large with both products fused into it
  static __device__ __forceinline__ void fma(A& acc, C2 a, C2 b) {
    const C2 p = prod(a, b);
    acc.x += p.x;
    acc.y += p.y;
  }
  static __device__ __forceinline__ C2 narrow(A v) { return v; }
};
template <typename V>
struct StoredReal {
  typedef V A;
  typedef V R;
  static __device__ __forceinline__ A prod(V a, V b) { return a * b; }
  static __device__ __forceinline__ void fma(A& acc, V a, V b) { acc = ::fma(a, b, acc); }
  static __device__ __forceinline__ V narrow(A v) { return v; }
};
template <> struct StoredOps<float> : StoredReal<float> {};
template <> struct StoredOps<double> : StoredReal<double> {};
template <> struct StoredOps<float2> : StoredComplex<float2, float> {};
template <> struct StoredOps<double2> : StoredComplex<double2, double> {};

}  // namespace fsb
