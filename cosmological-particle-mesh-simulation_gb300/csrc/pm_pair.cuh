// Float32 pairs hi + lo, |lo| <= ulp(hi) / 2: 48 bits and more, on the FP32 pipe (Dekker's and
// Knuth's error-free transformations).  Functions of the host too, for the tests: there a plain
// operation is rounded to nearest (compile without contraction).
#pragma once
#include <cuda_runtime.h>

#include <cmath>

namespace pm {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
#else
inline float add_rn(float a, float b) { return a + b; }
inline float mul_rn(float a, float b) { return a * b; }
#endif

__host__ __device__ __forceinline__ float2 split(double v) {
  const float h = (float)v;
  return make_float2(h, (float)(v - (double)h));
}
__host__ __device__ __forceinline__ float2 two_sum(float a, float b) {
  const float s = add_rn(a, b), t = add_rn(s, -a);
  return make_float2(s, add_rn(add_rn(a, -add_rn(s, -t)), add_rn(b, -t)));
}
// (c.x + c.y) * v
__host__ __device__ __forceinline__ float2 pair_mul(float2 c, float v) {
  const float p = mul_rn(c.x, v);
  return make_float2(p, fmaf(c.x, v, -p) + c.y * v);
}

// numpy float remainder: fmod, moved into the divisor's sign
__host__ __device__ __forceinline__ double py_mod(double a, double b) {
  double m = fmod(a, b);
  if (m != 0.0) {
    if ((b < 0.0) != (m < 0.0)) m += b;
  } else {
    m = copysign(0.0, b);
  }
  return m;
}

// (v.x + v.y) mod n, rounded to float32
__host__ __device__ __forceinline__ float pair_mod(float2 v, float n) {
  const float hi = v.x, lo = v.y;
  if (!(hi > -n && hi < 2.f * n)) return (float)py_mod((double)hi + (double)lo, (double)n);  // (and NaN)
  if (hi > n || (hi == n && lo >= 0.f)) return add_rn(add_rn(hi, -n), lo);  // hi - n is exact
  if (hi < 0.f || (hi == 0.f && lo < 0.f)) {
    const float2 t = two_sum(hi, n);
    return add_rn(t.x, add_rn(t.y, lo));
  }
  return add_rn(hi, lo);
}

}  // namespace pm
