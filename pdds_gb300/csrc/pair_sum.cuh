// Two running sums of FP32 values, each in three floats, without FP64.
//
// FP64 issues at 1/64 of the FP32 rate here.  TwoSum (Knuth, TAOCP vol. 2,
// 4.2.2) gives the exact rounding error of an FP32 addition, so s + e + f
// follows the exact sum to about 2^-72 of the largest partial sum: further
// than an FP64 sum of the same values (2^-53 per addition), which two floats
// (2^-48) would not reach.
#pragma once
#include <cuda_runtime.h>

namespace pdds {

struct PairSum {
  float2 s, e, f;  // of both sums: the sum, what s leaves out, what e leaves out
};

// a + b rounded; err = what that leaves out, exactly
__device__ __forceinline__ float2 two_sum(float2 a, float2 b, float2& err) {
  auto sub = [](float2 x, float2 y) { return __fadd2_rn(x, make_float2(-y.x, -y.y)); };
  const float2 t = __fadd2_rn(a, b), c = sub(t, a);
  err = __fadd2_rn(sub(a, sub(t, c)), sub(b, c));
  return t;
}
__device__ __forceinline__ void pair_add(PairSum& p, float2 v) {
  float2 e1, e2;
  p.s = two_sum(p.s, v, e1);
  p.e = two_sum(p.e, e1, e2);
  p.f = __fadd2_rn(p.f, e2);
}
// one of the two; a sum that is not finite has no error terms
__device__ __forceinline__ double pair_total(const PairSum& p, int second) {
  const float s = second ? p.s.y : p.s.x, e = second ? p.e.y : p.e.x, f = second ? p.f.y : p.f.x;
  return isfinite(s) ? (double)s + ((double)e + (double)f) : (double)s;
}

}  // namespace pdds
