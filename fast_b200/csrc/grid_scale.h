// grid_scale.h - the fixed-point form in which the persistent PCG kernel's
// grid sums travel (grid_sum in solve_kernels.cu), apart from the exchange
// itself: a value's limbs and the choice of the scale.  Host and device.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FG_HD __host__ __device__ __forceinline__
#else
#define FG_HD inline
#endif

namespace fastgpu {

FG_HD uint64_t double_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
FG_HD double bits_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
FG_HD int double_exponent(double x) { return (int)((double_bits(x) >> 52) & 2047) - 1023; }

FG_HD double pow2(int e) { return bits_double((uint64_t)(e + 1023) << 52); }  // |e| <= 1022
FG_HD double scale2(double x, int e) {  // x 2^e for |e| <= 2044 in two steps
  const int h = e / 2;
  return x * pow2(h) * pow2(e - h);
}

// Limb 0 holds 38 bits below 2^e, limbs 1 and 2 46 bits each below that.  Up to
// 148 limbs 0 add up to less than 2^46 in size; one mark in them makes the sum
// larger.
constexpr int64_t kSumMark = (int64_t)1 << 47, kSumMarked = (int64_t)1 << 46;
FG_HD int limb_exponent(int e, int limb) { return e - 38 - 46 * limb; }  // of its lowest bit

// the limb of x: its mantissa shifted to the limb's lowest bit (what lies below
// 2^(e - 130) is dropped), with the sign of x; a mark in limb 0 where |x| is not
// below 2^e (or not finite)
FG_HD int64_t sum_limb(double x, int e, int limb) {
  const uint64_t xb = double_bits(x);
  const int xe = (int)((xb >> 52) & 2047);
  const int sft = (xe ? xe : 1) - 1075 - limb_exponent(e, limb);
  uint64_t m = (xb & (((uint64_t)1 << 52) - 1)) | ((uint64_t)(xe != 0) << 52);
  m = sft >= 0 ? (sft < 46 ? m << sft : 0) : (sft > -53 ? m >> -sft : 0);
  if (limb > 0) m &= ((uint64_t)1 << 46) - 1;
  if (xe - 1023 >= e) return limb == 0 ? kSumMark : 0;
  return (int64_t)xb < 0 ? -(int64_t)m : (int64_t)m;
}

// The scale 2^e of a sum, and what its repeats have shown so far
struct SumScale {
  int e;
  int fit;  // smallest scale without a mark
  bool up;  // a mark was seen
};
// (at the lowest scale the last limb ends with the smallest FP64 number)
constexpr int kScaleMin = -944, kScaleMax = 1024;

// 40 bits above the last value of the same sum
FG_HD SumScale sum_scale(double ref) {
  const double r = ref < 0.0 ? -ref : ref;
  int e = r > 0.0 && r < 1e300 ? double_exponent(r) + 40 : 40;
  e = e < kScaleMin ? kScaleMin : (e > kScaleMax ? kScaleMax : e);
  return {e, kScaleMax, false};
}

// Whether the sum res, formed at s (over: with a mark), has to be formed again,
// and then the scale for it.  A sum that leaves fewer than 64 bits goes down
// (46 bits at least); a partial that does not fit goes up by 64, and the first
// sum that fits then is taken: 2^-58 of the largest partial is the most that is
// dropped, less than its own rounding.  So where partials cancel the scale never
// turns down again, and a sum is formed at most 43 + 31 times more, mostly none.
FG_HD bool sum_again(SumScale &s, bool over, double &res) {
  if (over) {
    if (s.e >= kScaleMax) {  // not finite
      res = bits_double(0x7FF8000000000000ull);
      return false;
    }
    s.up = true;
    s.e = s.e + 64 < s.fit ? s.e + 64 : s.fit;
    return true;
  }
  const int re = double_exponent(res);
  if (re >= s.e - 66 || s.up || s.e <= kScaleMin) return false;
  s.fit = s.e;
  const int e = res != 0.0 ? re + 20 : s.e - 60;
  s.e = e > kScaleMin ? e : kScaleMin;
  return true;
}

}  // namespace fastgpu
