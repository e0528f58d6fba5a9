// wg_radiation.cuh -- the terms of the day's radiation balance and
// Priestley-Taylor evaporation that depend on the air temperature alone
// (daily.cpp:382-532), in fixed point:
//   rlh  1 / latent heat                     latent heat 2.501 - 0.002361 T, 2.835 below 0 C
//   apt  s / (s + gamma)                     s the slope of the saturation vapour pressure,
//                                            gamma the psychrometric constant
//   lwt  eps sigma (T + 273.2)^4 / latent heat   net longwave radiation = -cloud factor x lwt
//
// In FP64 they were 27 multiplications and additions, two exponentials and three
// reciprocals of every cell-day, a fifth of the vertical balance's FP64-pipe
// time.  T is a float, so here it is one 64-bit integer; products are 64 x 64-bit
// high parts at constant scales, and only the three results are rounded to double:
// rlh and apt to a relative error below 2^-52, where the FP64 chain rounded some twenty
// times; lwt to 2^-51 of 0.281 sigma (T + 273.2)^4 / latent heat, an absolute error, since
// its emissivity 0.261 exp(-0.000777 T^2) - 0.02 changes sign near |T| = 57.5 C (in FP64
// the same subtraction cancels there).
#pragma once
#include <stdint.h>

#include "wg_fastmath.cuh"

namespace wg {
namespace fm {

struct TempTerms { double rlh, apt, lwt; };

// m 2^e (m > 0) rounded to a double; results below the normal range are 0
__device__ __forceinline__ double round_to_double(u64 m, int e) {
  const int lz = __clzll((i64)m);
  m <<= lz;
  e += 63 - lz;                               // m 2^(e - 63)
  return e < -1022 ? 0. : double_of((m >> 11) + (((u64)((uint32_t)(e + 1022) << 20) << 32) | ((lo32(m) >> 10) & 1u)));
}

// the same terms by the reference's expressions, for temperatures no climate has
// (128 C and more, NaN)
__device__ __noinline__ TempTerms temp_terms_any(float Tf) {
  const double T = (double)Tf, inv_t2 = rcp_pos(T + 237.3);
  const double e_s = 0.6108 * fm::exp(17.27 * T * inv_t2);
  const double rlh = rcp_pos((Tf > 0.f) ? 2.501 - 0.002361 * T : 2.835);
  const double inc_svp = 4098. * e_s * (inv_t2 * inv_t2), gamma = 0.0016286 * 101.3 * rlh;
  const double tK = T + 273.2, tK2 = tK * tK;
  TempTerms o;
  o.rlh = rlh;
  o.apt = inc_svp * rcp_pos(inc_svp + gamma);
  o.lwt = (-0.02 + 0.261 * fm::exp(-0.000777 * T * T)) * 0.000000004903 * (tK2 * tK2) * rlh;
  return o;
}

__device__ __forceinline__ TempTerms temp_terms(float Tf) {
  if (!(fabsf(Tf) < 128.f)) return temp_terms_any(Tf);
  TempTerms o;
  const i64 t = __float2ll_rn(Tf * 0x1p55f);                 // T in units of 2^-55
  const u64 ta = (u64)(t < 0 ? -t : t);
  const uint32_t below = (uint32_t)((int)hi32((u64)t) >> 31);
  // latent heat in units of 2^-62 (2.2 to 2.84), its reciprocal in units of 2^-65
  const u64 lh = (Tf > 0.f) ? 0xa010624dd2f1a800ull - mul_hi(ta, 0x4d5d80e496edec00ull) : 0xb570a3d70a3d7000ull;
  const u64 rl = rcp_mant(lh);
  o.rlh = round_to_double(rl, -65);
  // 1 / (T + 237.3) = r 2^(lz - 72); 17.27 log2(e) |T| / (T + 237.3) in units of 2^-58
  const u64 t2 = (u64)t + 0x76a6666666666800ull;
  const int lz = __clzll((i64)t2);
  const u64 r = rcp_mant(t2 << lz);
  const u64 y = mul_hi(mul_hi(ta, r) << lz, 0xc7529f899a488e23ull);
  const int n = (int)((hi32(y) >> 26) ^ below);
  const u64 es = exp2_mant((y << 6) ^ (u64)(i64)(int)below);             // exp(.) = es 2^(n - 63)
  // s = v 2^(d - 66) and gamma = g 2^-66; their quotient keeps v's own scale
  const u64 v = mul_hi(mul_hi(es, mul_hi(r, r)), 0x4e38779a6b50b14bull);
  const u64 g = mul_hi(rl, 0x5477e3915f636800ull);
  const int d = n + 2 * lz;
  const u64 sum = (v >> min(max(-d, 0), 63)) + (g >> min(max(d, 0), 63));
  const int ls = __clzll((i64)sum);
  o.apt = round_to_double(mul_hi(v, rcp_mant(sum << ls)), ls - 63 + min(d, 0));
  // net emissivity in units of 2^-64, of either sign
  const u64 sq = mul_hi(ta << 1, ta << 1);                               // T^2 in units of 2^-48
  const u64 y2 = mul_hi(sq, 0x92eda5bdb8143b71ull);                      // 0.000777 log2(e) T^2, units of 2^-57
  const u64 ex = mul_hi(exp2_mant(~(y2 << 7)), 0x85a1cac083127000ull);
  const i64 em = (i64)(ex >> ((hi32(y2) >> 25) + 1)) - 0x51eb851eb851ec0ll;
  const u64 ea = (u64)(em < 0 ? -em : em) << 2;
  const u64 tk = (u64)t + 0x8899999999999800ull;
  const u64 tk2 = mul_hi(tk, tk);                                        // units of 2^-46
  const u64 b = mul_hi(mul_hi(mul_hi(ea, mul_hi(tk2, tk2)), rl), 0xa8773e7c8b2ef800ull);   // units of 2^-58
  o.lwt = b == 0 ? 0. : double_of(bits_of(round_to_double(b, -58)) | ((u64)em & 0x8000000000000000ull));
  return o;
}

}  // namespace fm
}  // namespace wg
