// wg_compare.cuh -- comparisons of doubles from integer instructions.
#pragma once
#include <stdint.h>

namespace wg {

// Comparisons of the day step's hot loops.  On GB300 a double compare issues on
// the FP64 pipe (2 lanes per SM per clock) like an FMA; these give the same
// answers for every non-NaN operand from integer instructions on the bit
// patterns: x >= 0 orders like its bits as a signed integer, x < 0 like the
// negated magnitude (key below, which maps -0 and +0 to the same key), and a
// compare with a positive constant needs no key at all.  FP32 compares are
// cheap and stay as they are.
template <class R> struct C;
template <> struct C<double> {
  static __device__ __forceinline__ long long key(double x) {
    const long long b = __double_as_longlong(x);
    return b >= 0 ? b : (long long)(0x8000000000000000ull - (unsigned long long)b);
  }
  static __device__ __forceinline__ bool gt(double a, double b) { return key(a) > key(b); }
  static __device__ __forceinline__ bool le(double a, double b) { return key(a) <= key(b); }
  static __device__ __forceinline__ bool lt(double a, double b) { return key(a) < key(b); }
  static __device__ __forceinline__ bool lt0(double a) { return key(a) < 0; }
  static __device__ __forceinline__ bool gt0(double a) { return __double_as_longlong(a) > 0; }
  static __device__ __forceinline__ bool le0(double a) { return __double_as_longlong(a) <= 0; }
  // a < c and a <= c for a constant c > 0
  static __device__ __forceinline__ bool lt_c(double a, double c) { return __double_as_longlong(a) < __double_as_longlong(c); }
  // a > c and |a| <= c for a constant c > 0
  static __device__ __forceinline__ bool gt_c(double a, double c) { return __double_as_longlong(a) > __double_as_longlong(c); }
  static __device__ __forceinline__ bool abs_le_c(double a, double c) {
    return (__double_as_longlong(a) & 0x7FFFFFFFFFFFFFFFll) <= __double_as_longlong(c);
  }
  static __device__ __forceinline__ bool is_zero(double a) { return (__double_as_longlong(a) << 1) == 0; }
  static __device__ __forceinline__ bool is_one(double a) { return __double_as_longlong(a) == 0x3FF0000000000000ll; }
  static __device__ __forceinline__ bool equal(double a, double b) { return key(a) == key(b); }
};
// The same for the water bodies, whose storages keep a NaN where the inputs bring one:
// false with a NaN on either side, as the FP64 compares are (a NaN that arithmetic
// left has its quiet bit, the top one of the fraction, set).
template <class R> struct Cn;
template <> struct Cn<double> {
  typedef C<double> c;
  static __device__ __forceinline__ bool nan(double a) { return ((uint32_t)__double2hiint(a) << 1) > 0xffe00000u; }
  static __device__ __forceinline__ bool gt(double a, double b) { return c::gt(a, b) && !nan(a) && !nan(b); }
  static __device__ __forceinline__ bool ge(double a, double b) { return c::le(b, a) && !nan(a) && !nan(b); }
  static __device__ __forceinline__ bool lt0(double a) { return c::lt0(a) && !nan(a); }
  static __device__ __forceinline__ bool gt0(double a) { return c::gt0(a) && !nan(a); }
  static __device__ __forceinline__ bool le0(double a) { return c::le0(a) && !nan(a); }
  static __device__ __forceinline__ bool gt_c(double a, double k) { return c::gt_c(a, k) && !nan(a); }
  static __device__ __forceinline__ bool abs_le_c(double a, double k) { return c::abs_le_c(a, k); }
};
template <> struct C<float> {
  static __device__ __forceinline__ bool gt(float a, float b) { return a > b; }
  static __device__ __forceinline__ bool le(float a, float b) { return a <= b; }
  static __device__ __forceinline__ bool lt(float a, float b) { return a < b; }
  static __device__ __forceinline__ bool ge(float a, float b) { return a >= b; }
  static __device__ __forceinline__ bool lt0(float a) { return a < 0.f; }
  static __device__ __forceinline__ bool gt0(float a) { return a > 0.f; }
  static __device__ __forceinline__ bool le0(float a) { return a <= 0.f; }
  static __device__ __forceinline__ bool lt_c(float a, float c) { return a < c; }
  static __device__ __forceinline__ bool gt_c(float a, float c) { return a > c; }
  static __device__ __forceinline__ bool abs_le_c(float a, float c) { return fabsf(a) <= c; }
  static __device__ __forceinline__ bool is_zero(float a) { return a == 0.f; }
  static __device__ __forceinline__ bool is_one(float a) { return a == 1.f; }
  static __device__ __forceinline__ bool equal(float a, float b) { return a == b; }
};
template <> struct Cn<float> : C<float> {};

}  // namespace wg
