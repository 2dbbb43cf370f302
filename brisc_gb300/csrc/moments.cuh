// Sum and sum of squares of floats as unevaluated sums of floats (error-free
// transformations: Knuth's TwoSum, a product and its remainder by FMA), for the
// per-gene moments.
//
// GB300's FP64 pipe does one addition or multiply-add per 64 FP32 lanes; the
// moments need two of them and a conversion per stored entry, 300 us of
// k_xt_sell at 300k x 2000 (28.5M entries) against 35 us for the FP32 product
// over the same entries. So a short run of entries is summed in FP32 additions
// (18 per entry) and converted to FP64 once.
// The variance is n s2 - s1^2: a gene whose mean is r times its spread loses
// r^2 of the sums' precision, so these have to be as good as FP64 sums of the
// run. The values, the squares and the squares' remainders each have a float
// for the sum and one for what its rounding lost (the remainders of four squares
// are added first: rounding those costs 2^-48 of a square). Over runs of
// kMomentTerms or fewer values within a factor of four of one another (squares:
// of 16) the lost parts add up without another rounding (they are multiples of
// the smallest term's ulp, below 2^24 of it), so a run's sums are exact but for
// the remainders' last bits: that is nearly every value of a gene with r >> 1.
// Values further apart leave 2^-42, in genes whose spread is of their mean's size.
// Measured over 1024 runs of 256 values with mean 10 and sd 0.001: error of the
// sd 6e-8, with FP64 sums 9e-8; with the remainders added to the squares' lost
// part 1.2e-6.
#pragma once

namespace bgpu {

constexpr int kMomentTerms = 1024;

struct FloatMoments {
  // of the values, their squares and the squares' remainders: sum, what it lost
  float s[2] = {0.f, 0.f}, q[2] = {0.f, 0.f}, r[2] = {0.f, 0.f};

  static __device__ __forceinline__ void two_sum(float (&a)[2], float v) {
    const float t = __fadd_rn(a[0], v), z = __fsub_rn(t, a[0]);
    const float e = __fadd_rn(__fsub_rn(a[0], __fsub_rn(t, z)), __fsub_rn(v, z));
    a[0] = t;
    a[1] = __fadd_rn(a[1], e);
  }
  __device__ __forceinline__ void add(float v0, float v1, float v2, float v3) {
    const float v[4] = {v0, v1, v2, v3};
    float e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      two_sum(s, v[i]);
      const float p = __fmul_rn(v[i], v[i]);
      two_sum(q, p);
      e[i] = __fmaf_rn(v[i], v[i], -p);
    }
    two_sum(r, __fadd_rn(__fadd_rn(e[0], e[1]), __fadd_rn(e[2], e[3])));
  }
  // The totals of the G lanes of `mask` (aligned, a power of two): a[0] the same in
  // each of them, so that good() is.
  template <int G>
  __device__ __forceinline__ void merge(unsigned mask) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      auto join = [&](float (&a)[2]) {
        const float hi = __shfl_xor_sync(mask, a[0], o), lo = __shfl_xor_sync(mask, a[1], o);
        two_sum(a, hi);
        a[1] = __fadd_rn(a[1], lo);
      };
      join(s);
      join(q);
      join(r);
    }
  }
  // Whether the floats hold the sums: squares within the range where a
  // product's remainder is exact. Otherwise (tiny, huge or non-finite values,
  // or nothing but zeros) the caller sums in FP64.
  __device__ __forceinline__ bool good() const { return q[0] > 1e-25f && q[0] < 1e30f; }
  __device__ __forceinline__ double sum() const { return (double)s[0] + (double)s[1]; }
  __device__ __forceinline__ double squares() const {
    float t[2] = {q[1], r[1]};
    two_sum(t, r[0]);
    return (double)q[0] + ((double)t[0] + (double)t[1]);
  }
};

}  // namespace bgpu
