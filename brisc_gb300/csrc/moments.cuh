// Sum and sum of squares of floats as unevaluated pairs of floats (error-free
// transformations: Knuth's TwoSum, a product and its remainder by FMA), for
// the per-gene moments.
//
// GB300's FP64 pipe does one addition or multiply-add per 64 FP32 lanes; the
// moments need two of them and a conversion per stored entry, 300 us of
// k_xt_sell at 300k x 2000 (28.5M entries) against 35 us for the FP32 product
// over the same entries. As pairs the sums take FP32 additions only and carry
// 2^-46 of their value over a few hundred terms; each short sum is converted to
// FP64 once and the FP64 totals are as before. The standard deviation is
// stored as a float, so its error against FP64 sums stays that rounding.
#pragma once

namespace bgpu {

struct PairMoments {
  float sh = 0.f, sl = 0.f, qh = 0.f, ql = 0.f;

  static __device__ __forceinline__ void two_sum(float& h, float& l, float v) {
    const float t = __fadd_rn(h, v), z = __fsub_rn(t, h);
    const float e = __fadd_rn(__fsub_rn(h, __fsub_rn(t, z)), __fsub_rn(v, z));
    h = t;
    l = __fadd_rn(l, e);
  }
  __device__ __forceinline__ void add(float v) {
    two_sum(sh, sl, v);
    const float p = __fmul_rn(v, v);
    ql = __fadd_rn(ql, __fmaf_rn(v, v, -p));
    two_sum(qh, ql, p);
  }
  // Whether the pairs hold the sums: squares within the range where a
  // product's remainder is exact. Otherwise (tiny, huge or non-finite values,
  // or nothing but zeros) the caller sums in FP64.
  __device__ __forceinline__ bool good() const { return qh > 1e-25f && qh < 1e30f; }
  __device__ __forceinline__ double sum() const { return (double)sh + (double)sl; }
  __device__ __forceinline__ double squares() const { return (double)qh + (double)ql; }
};

}  // namespace bgpu
