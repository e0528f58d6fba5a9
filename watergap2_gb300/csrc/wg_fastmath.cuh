// wg_fastmath.cuh -- FP64 exp / log / pow / reciprocal for the day step on GB300,
// computed on the integer pipe.
//
// GB300 has two FP64 lanes per SM: one FP64 instruction of a warp holds its
// sub-partition's share of the pipe for about 77 cycles, while 32-bit integer
// instructions issue every one or two.  A 64 x 64-bit high product from three
// 32-bit multiplies costs 17 cycles, so these functions carry their arguments as
// 64-bit fixed-point numbers and round once, at the end, to the 53 bits of a
// double: fewer cycles and more bits than a chain of FP64 FMAs.  Measured per warp
// instruction and sub-partition (all warps busy), before = table-driven FP64:
//   exp 898 -> 138 cycles, pow 1866 -> 235, reciprocal 291 -> 73
//   largest error in ulp: exp (|x| < 12) 1.25 -> 0.53, pow(x, 2/3) for x in
//   1e-8 .. 1e4 19 -> 0.64, pow(x, 2.5) 73 -> 0.77, reciprocal 0.505 -> 0.501
// and on the global grid (67,420 cells, one year, five days per step) 47.2 ->
// 33.5 ms; k_vertical_ahead 0.66 -> 0.45 ms per 20 days, k_pipeline 1.07 -> 0.76.
// Methods: table-driven exp and log after P. T. P. Tang (ACM TOMS 15(2), 1989;
// 16(4), 1990) with 256 intervals,
//   2^f     = 2^(j/256) 2^r,  r < 1/256, polynomial of degree 5,
//   log2(y) = log2(1/c_j) + log2(1 + z), c_j ~ 1/(1 + j/256) in 32 bits and
//             z = y c_j - 1 < 1/256, polynomial of degree 5 without constant term,
// the polynomials interpolated at Chebyshev nodes (errors 2^-70 and 2^-59); the
// reciprocal from the single-precision hardware approximation by one third-order
// Newton step (P. Markstein, "IA-64 and Elementary Functions", 2000, ch. 8) in
// fixed point.  The tables are filled on the host (FastmathTables, wg_capi.cpp).
//
// pow takes x >= 0 (x <= 0 gives 0, as the hot path's pow(0, y > 0) does).
#pragma once
#include <stdint.h>

namespace wg {
namespace fm {

typedef unsigned long long u64;
typedef long long i64;

// tables, filled from the host (the one translation unit that includes this file)
__device__ u64 g_exp2_tab[256];       // 2^(j/256) in units of 2^-63
__device__ ulonglong2 g_log2_tab[256];   // x: log2(1/c_j) in units of 2^-63, y: c_j in units of 2^-31

__device__ __forceinline__ u64 bits_of(double x) { return (u64)__double_as_longlong(x); }
__device__ __forceinline__ double double_of(u64 b) { return __longlong_as_double((i64)b); }
__device__ __forceinline__ uint32_t hi32(u64 a) { return (uint32_t)(a >> 32); }
__device__ __forceinline__ uint32_t lo32(u64 a) { return (uint32_t)a; }
__device__ __forceinline__ u64 mul_wide(uint32_t a, uint32_t b) { return (u64)a * b; }

// the high 64 bits of a * b from three of its four partial products: up to three
// units low
__device__ __forceinline__ u64 mul_hi(u64 a, u64 b) {
  return mul_wide(hi32(a), hi32(b)) + __umulhi(hi32(a), lo32(b)) + __umulhi(lo32(a), hi32(b));
}

// 2^f, f in units of 2^-64, in units of 2^-63 (at least 2^63).  The polynomial is
// exact at both ends of its interval.
__device__ __forceinline__ u64 exp2_mant(u64 f) {
  const u64 t = g_exp2_tab[hi32(f) >> 24];
  const u64 r = f << 8;                                      // 256 (f - j/256)
  const uint32_t rh = hi32(r);
  const uint32_t a4 = 0x276555u + __umulhi(rh, 0x578u);        // units of 2^-60
  const uint32_t a3 = 0xe35846b9u + __umulhi(rh, a4);
  const u64 a2 = 0x3d7f7bff0589ull + ((u64)__umulhi(rh, a3) << 4);   // units of 2^-64
  const u64 a1 = 0xb17217f7d1cf7aull + mul_hi(r, a2);
  return t + mul_hi(t, mul_hi(r, a1));
}

// 2^(n + f), f in units of 2^-64, rounded to a double; n within the exponents of
// normal doubles
__device__ __forceinline__ double exp2_normal(int n, u64 f) {
  const u64 u = exp2_mant(f);
  return double_of((u >> 11) + (((u64)((uint32_t)(n + 1022) << 20) << 32) | ((lo32(u) >> 10) & 1u)));
}

// the same for any n
__device__ __forceinline__ double exp2_fixed(int n, u64 f) {
  const u64 u = exp2_mant(f);
  if ((unsigned)(n + 1021) >= 2045u) {                       // subnormal, zero or infinite
    if (n > 1023) return double_of(0x7ff0000000000000ull);
    if (n < -1022) {
      const int down = -1011 - n;
      return down > 63 ? 0. : double_of((u >> down) + ((u >> (down - 1)) & 1));
    }
  }
  return double_of((u >> 11) + (((u64)((uint32_t)(n + 1022) << 20) << 32) | ((lo32(u) >> 10) & 1u)));
}

// exp of an argument of 32 or more, or not a number: out of line, since the hot path
// never has one and a branch that holds no code of its own costs least
__device__ __noinline__ double exp_any(double x) {
  const u64 b = bits_of(x), log2e = 0xb8aa3b295c17f0bcull;   // units of 2^-63
  const int e = (int)((hi32(b) >> 20) & 0x7ff) - 1023;
  if (e >= 10) {                                             // beyond the range of a double
    if ((b << 1) > 0xffe0000000000000ull) return x;          // NaN
    return (i64)b < 0 ? 0. : double_of(0x7ff0000000000000ull);
  }
  const u64 m = (b << 11) | 0x8000000000000000ull;           // |x| = m 2^(e - 63)
  const u64 p = __umul64hi(m, log2e);
  const uint32_t s = (uint32_t)((int)hi32(b) >> 31);         // -(n + f) = ~n + ~f
  return exp2_fixed((int)((uint32_t)(p >> (62 - e)) ^ s),
                    ((p << (e + 2)) | ((m * log2e) >> (62 - e))) ^ (u64)(i64)(int)s);
}

__device__ __forceinline__ double exp(double x) {
  const u64 b = bits_of(x);
  const int e = (int)((hi32(b) >> 20) & 0x7ff) - 1023;
  if (e >= 5) return exp_any(x);
  const u64 m = (b << 11) | 0x8000000000000000ull;           // |x| = m 2^(e - 63), below 32
  u64 p = mul_hi(m, 0xb8aa3b295c17f0bcull);                  // |x| log2 e = p 2^(e - 62)
  p >>= min(max(-2 - e, 0), 63);
  const int k = max(e + 2, 0);
  const uint32_t s = (uint32_t)((int)hi32(b) >> 31);         // -(n + f) = ~n + ~f
  const uint32_t n = __funnelshift_l(hi32(p), 0u, k) ^ s;
  const u64 f = (((u64)__funnelshift_l(lo32(p), hi32(p), k) << 32) | (lo32(p) << k)) ^ (u64)(i64)(int)s;
  return exp2_normal((int)n, f);
}

// exp(-x) for x >= 0 where the caller goes on with 1 - exp(-x), as the river's
// linear reservoir does: below 2^-8 the distance from 1 is computed to 2^-60 of
// itself and subtracted exactly, so that the result is rounded once, as the
// correctly rounded function is but for one case in 2^50 (a last bit of exp(-x)
// is 2^-53 / x of 1 - exp(-x): 2e-10 for a river at its least velocity).
__device__ __forceinline__ double exp_neg(double x) {
  const u64 b = bits_of(x);
  const int e = (int)((hi32(b) >> 20) & 0x7ff) - 1023;
  if (e >= -8 || (i64)b < 0) return fm::exp(-x);
  const u64 m = (b << 11) | 0x8000000000000000ull;           // x = m 2^(e - 63)
  const u64 h = m >> min(-1 - e, 63);                        // units of 2^-64
  const uint32_t hh = hi32(h);
  // (x - 1 + exp(-x)) / x = x/2 - x^2/6 + x^3/24 - x^4/120 + x^5/720 (next term below 2^-58)
  const uint32_t c4 = 0x02222222u - __umulhi(hh, 0x005b05b0u);             // units of 2^-32
  const u64 c3 = 0x0aaaaaaaaaaaaaaaull - ((u64)__umulhi(hh, c4) << 32 | hh * c4);
  const u64 c2 = 0x2aaaaaaaaaaaaaabull - mul_hi(h, c3);
  const u64 c1 = 0x8000000000000000ull - mul_hi(h, c2);
  const u64 z = m - mul_hi(m, mul_hi(h, c1));                // 1 - exp(-x) = z 2^(e - 63)
  const int down = -1 - e;                                   // at least 8
  const u64 q = down > 63 ? 0 : z >> down;
  const u64 u = ~q + (down <= 63 && (q << down) == z);       // floor of 1 - z, units of 2^-64
  // rounded to 53 bits; from 1 - 2^-54 on it is 1
  return double_of((u >> 11) + (((u64)(1021u << 20) << 32) | ((lo32(u) >> 10) & 1u)));
}

// log2 of a positive normal number with bits b: m + (result in units of 2^-63)
__device__ __forceinline__ u64 log2_frac(u64 b, int &m) {
  const uint32_t h = hi32(b);
  m = (int)(h >> 20) - 1023;
  const ulonglong2 t = g_log2_tab[(h >> 12) & 0xff];
  const u64 y = (b << 11) | 0x8000000000000000ull;
  const uint32_t c = lo32(t.y);
  const u64 p = mul_wide(hi32(y), c) + __umulhi(lo32(y), c);               // y c, units of 2^-62
  const u64 z = (p - (1ull << 62)) << 10;                                  // 256 (y c - 1)
  const uint32_t zh = hi32(z);
  const uint32_t u4 = 0x5c5497e4u - __umulhi(zh, 0x4944a3u);               // units of 2^-64 from here
  const u64 u3 = 0x7b1c274132ull - __umulhi(zh, u4);
  const u64 u2 = 0xb8aa3b295622ull - mul_hi(z, u3);
  const u64 u1 = 0x171547652b82fc3ull - mul_hi(z, u2);
  return t.x + (mul_hi(z, u1) >> 1);
}

// log2 with its sign, in units of 2^-(64 - sh): sh - 1 bits hold its integer part
__device__ __forceinline__ i64 log2_fixed(u64 b, int &sh) {
  int m;
  const u64 f = log2_frac(b, m);
  const uint32_t a = (uint32_t)(m ^ (m >> 31));
  sh = max(33 - __clz(a), 5);
  const u64 fs = ((u64)(hi32(f) >> (sh - 1)) << 32) | __funnelshift_r(lo32(f), hi32(f), sh - 1);
  return (i64)(((u64)((uint32_t)m << (32 - sh)) << 32) + fs);
}

// natural log of a positive normal number
__device__ __forceinline__ double log(double x) {
  int sh;
  const i64 l = log2_fixed(bits_of(x), sh);
  return (double)l * double_of((u64)(959 + sh) << 52) * 0.6931471805599453;   // 2^(sh - 64)
}

// x^y for any x and y
__device__ __noinline__ double pow_any(double x, double y) {
  const u64 b = bits_of(x), yb = bits_of(y);
  if ((i64)b <= 0) return 0.0;                               // x <= 0 (and -0)
  if (b == 0x3ff0000000000000ull) return 1.0;                // x == 1
  if (b >= 0x7ff0000000000000ull) return x;
  int sh;
  const i64 l = log2_fixed(b, sh);
  const int ls = (int)(hi32((u64)l)) >> 31;
  const u64 la = ((u64)l ^ (u64)(i64)ls) - (u64)(i64)ls;
  const int ey = (int)((hi32(yb) >> 20) & 0x7ff) - 1023;
  const u64 ym = (yb << 11) | 0x8000000000000000ull;
  u64 p = mul_hi(la, ym);                                    // |y log2 x| = p 2^(k - 64)
  int k = sh + ey + 1;
  if ((unsigned)(k - 1) >= 31u) {                            // y below 2^-5 or beyond 2^18
    if (k < 1) {
      p >>= min(1 - k, 63);
      k = 1;
    } else if (ey == 1024 || k > 63 || (p >> (64 - k)) > 1100) {   // beyond the range of a double
      if ((yb << 1) > 0xffe0000000000000ull) return y;       // NaN
      return (ls ^ ((int)hi32(yb) >> 31)) ? 0. : double_of(0x7ff0000000000000ull);
    } else {                                                 // few enough integer bits after all
      p <<= k - 31;
      k = 31;
    }
  }
  const uint32_t n = hi32(p) >> (32 - k);
  const u64 f = ((u64)__funnelshift_l(lo32(p), hi32(p), k) << 32) | (lo32(p) << k);
  const uint32_t s = (uint32_t)(ls ^ ((int)hi32(yb) >> 31));
  return exp2_fixed((int)(n ^ s), f ^ (u64)(i64)(int)s);
}

// x^y: the integer part of y log2 x in k bits of the product, 1 <= k <= 31, and the
// result a normal double, else pow_any; x <= 0 gives 0
__device__ __forceinline__ double pow(double x, double y) {
  const u64 b = bits_of(x), yb = bits_of(y);
  int sh;
  const i64 l = log2_fixed(b, sh);
  const uint32_t ls = (uint32_t)((int)hi32((u64)l) >> 31);
  const u64 la = ((u64)l ^ (u64)(i64)(int)ls) - (u64)(i64)(int)ls;
  const int k = sh + (int)((hi32(yb) >> 20) & 0x7ff) - 1022;
  const u64 p = mul_hi(la, (yb << 11) | 0x8000000000000000ull);
  const uint32_t s = ls ^ (uint32_t)((int)hi32(yb) >> 31);
  const uint32_t n = (hi32(p) >> ((32 - k) & 31)) ^ s;
  const u64 f = (((u64)__funnelshift_l(lo32(p), hi32(p), k) << 32) | (lo32(p) << (k & 31))) ^ (u64)(i64)(int)s;
  // x positive and not a normal number, or a format or result outside the above
  if ((i64)b > 0 && (hi32(b) - 0x00100000u >= 0x7fe00000u || (unsigned)(k - 1) >= 31u || n + 1000u > 2000u))
    return pow_any(x, y);
  return (i64)b <= 0 ? 0. : exp2_normal((int)n, f);
}

// 1/(m 2^-63) for m in [2^63, 2^64), in units of 2^-64: the single-precision
// hardware reciprocal r of the leading 24 bits, lowered so that e = 1 - m r is
// positive (below 2^-20), then r (1 + e + e^2)
__device__ __forceinline__ u64 rcp_mant(u64 m) {
  float r0;                                                  // in (0.5, 1]
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(__uint_as_float(0x3f800000u | ((hi32(m) << 1) >> 9))));
  const uint32_t rb = __float_as_uint(r0);
  const uint32_t r = (rb >= 0x3f800000u ? 0xffffffffu : ((rb << 8) | 0x80000000u)) - 0x400u;   // units of 2^-32
  const u64 e = (1ull << 63) - (mul_wide(hi32(m), r) + __umulhi(lo32(m), r));               // units of 2^-63
  const uint32_t eh = (uint32_t)(e >> 20);
  const u64 g = e + (mul_wide(eh, eh) >> 23);
  return ((u64)r << 32) + ((mul_wide(r, hi32(g)) + __umulhi(r, lo32(g))) << 1);
}

// 1/x for finite normal x of either sign, to half an ulp and 2^-8 more.  The hot
// path calls it only with divisors bounded away from zero.
__device__ __forceinline__ double rcp_pos(double x) {
  const u64 b = bits_of(x);
  const uint32_t ex = (hi32(b) >> 20) & 0x7ff;
  const u64 u = rcp_mant((b << 11) | 0x8000000000000000ull);
  const double v = double_of((u >> 11) + (((u64)((2044u - ex) << 20) << 32) | ((lo32(u) >> 10) & 1u)) |
                             (b & 0x8000000000000000ull));
  // zero, subnormal, infinite and NaN arguments give NaN, those from 2^1022 on 0
  if (ex - 1u >= 2044u) return double_of(ex - 1u >= 2046u ? 0x7ff8000000000000ull : 0ull);
  return v;
}

__device__ __noinline__ double div_any(double a, double b) { return a / b; }

// a / b, correctly rounded (the midpoint next to the approximate quotient, times b,
// compared with a): normal a and b with a normal quotient, and a = 0; anything else
// through the general division. 130 cycles per warp (the
// root 127), 108 without the last comparison
__device__ __forceinline__ double div(double a, double b) {
  const u64 ab = bits_of(a), bb = bits_of(b);
  const int ea = (int)((hi32(ab) >> 20) & 0x7ff), eb = (int)((hi32(bb) >> 20) & 0x7ff);
  const u64 sign = (ab ^ bb) & 0x8000000000000000ull;
  const u64 am = (ab << 11) | 0x8000000000000000ull, bm = (bb << 11) | 0x8000000000000000ull;
  u64 q = mul_hi(am, rcp_mant(bm));
  const uint32_t low = (hi32(q) >> 31) ^ 1u;                 // the quotient of the mantissas is below 1
  q <<= low;
  const int e = ea - eb + 1022 - (int)low;                   // biased exponent less one
  const uint32_t up = __umul64hi((q & ~0x7ffull) | 0x400u, bm) < am >> (low ^ 1u);
  const double r = double_of(((q >> 11) + (((u64)((uint32_t)e << 20) << 32) | up)) | sign);
  if ((unsigned)(eb - 1) >= 2046u || ((unsigned)(ea - 1) >= 2046u && (ab << 1) != 0) || (ea && (unsigned)(e - 1) >= 2043u))
    return div_any(a, b);
  return ea ? r : double_of(sign);
}

__device__ __noinline__ double sqrt_any(double x) { return ::sqrt(x); }

// square root of a positive normal number, correctly rounded: m in [1/4, 1),
// the single-precision reciprocal root y of its leading bits, e = 1 - m y^2, then
// m y (1 + e/2 + 3 e^2/8) (Markstein 2000, ch. 9, the third-order step), and the square
// of the midpoint next to it compared with m
__device__ __forceinline__ double sqrt(double x) {
  const u64 b = bits_of(x);
  const uint32_t ex = (hi32(b) >> 20) & 0x7ff;
  const uint32_t odd = (ex & 1u) ^ 1u;                       // ex even: the unbiased exponent is odd
  const u64 m = ((b << 11) | 0x8000000000000000ull) >> (1u - odd);   // units of 2^-64: [1/4, 1/2) or [1/2, 1)
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(__uint2float_rz(hi32(m)) * 0x1p-32f));   // in [1, 2]
  const uint32_t y = min((uint32_t)(y0 * 0x1p31f), 0xffffff00u) - 0x400u;   // units of 2^-31, a little low
  const u64 my = mul_wide(hi32(m), y) + __umulhi(lo32(m), y);        // m y, units of 2^-63, below 1
  const u64 e = (1ull << 62) - (mul_wide(hi32(my), y) + __umulhi(lo32(my), y));   // 1 - m y^2, units of 2^-62, below 2^-19
  const uint32_t eh = (uint32_t)(e >> 20);                   // units of 2^-42
  const u64 g = (e >> 1) + ((mul_wide(eh, eh) * 3) >> 25);    // e/2 + 3 e^2/8, units of 2^-62
  const u64 u = (my << 1) + (mul_hi(my, g) << 3);            // units of 2^-64: the root, in [1/2, 1)
  const u64 mid = (u & ~0x7ffull) | 0x400u;
  const uint32_t up = __umul64hi(mid, mid) < m;
  const double r = double_of((u >> 11) + (((u64)((((ex + 1u) >> 1) + 510u) << 20) << 32) | up));
  if (hi32(b) - 0x00100000u >= 0x7fe00000u) return sqrt_any(x);   // zero, subnormal, negative, infinite, NaN
  return r;
}

}  // namespace fm

}  // namespace wg
