// gfx_fixed_kp.cuh -- the Kennedy-Pendleton SU(2) heatbath draw in 64-bit fixed point
// (gfx_fixed.cuh), for the FP64-accurate thermalization.
//
// With the staple products in fixed point, the draw's FP64 logarithm, square roots, divisions
// and sine would be two thirds of a link update (about 450 FP64 operations of the three
// subgroups, at 2 per SM and clock).  Here the logarithm is the series of 2 artanh, sine and
// cosine are their Taylor series on an eighth of a turn, and square roots are x / sqrt(x).
// The random numbers are FP32 values, exact on the grid.  Errors are a few 2^-60 of the
// quantities that FP64 rounds at 2^-54 (tests/fixed_check.cpp).
#pragma once

#include "gfx_fixed.cuh"

namespace gfx {

// a non-negative float below 4, exact where it is a multiple of 2^-61 (the uniform numbers
// are multiples of 2^-32), times 2^-shift
GFX_FX fx64 fx_from_float(float f, int shift) {
#ifdef __CUDA_ARCH__
  const uint32_t b = __float_as_uint(f);
#else
  uint32_t b;
  std::memcpy(&b, &f, 4);
#endif
  // f = m 2^(e - 150); on the grid m 2^(e - 89) = (m 2^39) >> (128 - e)
  const uint64_t m = (uint64_t)((b & 0x7fffffu) | 0x800000u) << 39;
  const uint32_t sh = 128u + (uint32_t)shift - (b >> 23);
  return (fx64)(m >> (sh < 63u ? sh : 63u));
}

// sqrt(z) for 0 <= z <= 1: z / sqrt(4 z) doubled
GFX_FX fx64 fx_sqrt(fx64 z) {
  fx64 n = (z + 1) >> 1;  // 4 z on the grid of 2^-58
  n = n < 1 ? 1 : n;
  int s;
  const Fx y = fx_split(fx_rsqrt(n, s));
  return 2 * fx_mul(fx_prescale(z, s), y);
}

// -log(a) / 16 for a = a61 2^-61, 0 < a <= 1.  a = m 2^-e with m in [3/4, 3/2), and
// log m = 2 artanh(t), t = (m - 1) / (m + 1), |t| <= 1/5: artanh t = t (1 + t^2/3 + t^4/5 + ..),
// 13 terms (t^26 / 27 < 2^-65).
GFX_FX fx64 fx_neg_log_16th(fx64 a61) {
  int e = fx_clz(a61) - 2;  // a 2^e in [1, 2)
  fx64 m = a61 << e;
  if (m >= kFxOne + kFxOne / 2) {
    m >>= 1;
    e--;
  }
  // r = 1 / ((m + 1) / 2) in [4/5, 8/7]: an FP32 estimate and r0 (1 + d + d^2), d = 1 - r0 (m + 1)/2
  const fx64 half = (m + kFxOne) >> 1;
  const Fx h = fx_split(half);
#ifdef __CUDA_ARCH__
  const float rf = __fdividef(1.0f, (float)(int)(half >> 32) * (1.0f / 536870912.0f));
#else
  const float rf = 1.0f / ((float)(int)(half >> 32) * (1.0f / 536870912.0f));
#endif
  Fx r0;
  r0.h = (int)(rf * 536870912.0f);
  r0.l = 0;
  const fx64 d = kFxOne - fx_mul(h, r0);  // |d| < 2^-20
  const Fx ds = fx_split(d);
  const fx64 r = fx_join(r0) + fx_mul(fx_split(d + fx_mul(ds, ds)), r0);
  const fx64 t = fx_mul(fx_split((m - kFxOne) / 2), fx_split(r));
  const Fx ts = fx_split(t);
  const Fx t2 = fx_split(fx_mul(ts, ts));
  // 1 / (2 k + 1) on the grid
  fx64 p = 92233720368547758ll;  // 1/25
  p = fx_mul(t2, fx_split(p)) + 100254043878856259ll;  // 1/23
  p = fx_mul(t2, fx_split(p)) + 109802048057794950ll;
  p = fx_mul(t2, fx_split(p)) + 121360158379668103ll;
  p = fx_mul(t2, fx_split(p)) + 135637824071393762ll;
  p = fx_mul(t2, fx_split(p)) + 153722867280912930ll;
  p = fx_mul(t2, fx_split(p)) + 177372539170284150ll;
  p = fx_mul(t2, fx_split(p)) + 209622091746699450ll;
  p = fx_mul(t2, fx_split(p)) + 256204778801521550ll;
  p = fx_mul(t2, fx_split(p)) + 329406144173384850ll;
  p = fx_mul(t2, fx_split(p)) + 461168601842738790ll;
  p = fx_mul(t2, fx_split(p)) + 768614336404564651ll;
  p = fx_mul(t2, fx_split(p)) + kFxOne;
  // e log 2 / 16 - 2 artanh(t) / 16
  return e * 99893036290645747ll - ((fx_mul(ts, fx_split(p)) + 4) >> 3);
}

// sine and cosine of a turn times u61 2^-61, 0 <= u <= 1: a quarter of a turn taken off, x in
// [-pi/4, pi/4], Taylor series to x^17 and x^18
GFX_FX void fx_sincos_turns(fx64 u61, fx64& sn, fx64& cs) {
  const int q = (int)((u61 + (1ll << 58)) >> 59);  // nearest quarter
  const fx64 r = u61 - ((fx64)q << 59);
  const Fx x = fx_split(2 * fx_mul(fx_split(r), fx_split(7244019458077122842ll)));  // 2 pi r
  const Fx z = fx_split(fx_mul(x, x));
  fx64 p = 6483;  // 1/17!, .. with alternating signs
  p = fx_mul(z, fx_split(p)) - 1763316;
  p = fx_mul(z, fx_split(p)) + 370296340;
  p = fx_mul(z, fx_split(p)) - 57766228987ll;
  p = fx_mul(z, fx_split(p)) + 6354285188530ll;
  p = fx_mul(z, fx_split(p)) - 457508533574146ll;
  p = fx_mul(z, fx_split(p)) + 19215358410114116ll;
  p = fx_mul(z, fx_split(p)) - 384307168202282325ll;
  p = fx_mul(z, fx_split(p)) + kFxOne;
  const fx64 s = fx_mul(x, fx_split(p));
  p = -360;  // 1/18!
  p = fx_mul(z, fx_split(p)) + 110207;
  p = fx_mul(z, fx_split(p)) - 26449739;
  p = fx_mul(z, fx_split(p)) + 4813852416ll;
  p = fx_mul(z, fx_split(p)) - 635428518853ll;
  p = fx_mul(z, fx_split(p)) + 57188566696768ll;
  p = fx_mul(z, fx_split(p)) - 3202559735019019ll;
  p = fx_mul(z, fx_split(p)) + 96076792050570581ll;
  p = fx_mul(z, fx_split(p)) - 1152921504606846976ll;
  const fx64 c = fx_mul(z, fx_split(p)) + kFxOne;
  sn = (q & 1) ? c : s;
  cs = (q & 1) ? s : c;
  if (q & 2) sn = -sn;
  if ((q + 1) & 2) cs = -cs;
}

// The update of heatbath_su2_kp: the SU(2) element (p, q) that replaces the subgroup's, from
// v = w / 8 (the projection of link times staple), the standard normal g and the uniform
// numbers u; inv_beta = 1 / beta3 on the grid (beta3 = beta / 3 >= 5/4).  A rejected trial
// and a vanishing projection leave the subgroup unchanged.
GFX_FX void fx_kp(fx64 v0, fx64 v1, fx64 v2, fx64 v3, fx64 inv_beta, float g, float u0, float u1,
                  float u2, float u3, CFx& p, CFx& q) {
  p.re = fx_split(kFxOne);
  p.im = q.re = q.im = fx_split(0ll);
  // a small projection at a scale where its square keeps its accuracy
  const int c = fx_clz((v0 ^ (v0 >> 63)) | (v1 ^ (v1 >> 63)) | (v2 ^ (v2 >> 63)) |
                       (v3 ^ (v3 >> 63))) - 3;
  const int up = c < 0 ? 0 : c > 60 ? 60 : c;
  const fx64 v[4] = {v0 << up, v1 << up, v2 << up, v3 << up};
  FxAcc t = fx_acc();
#pragma unroll
  for (int k = 0; k < 4; k++) fx_sqr(t, fx_split(v[k]));
  const fx64 n = fx_sqr_val(t);
  const fx64 a = kFxOne - fx_from_float(u0, 0);
  if (n <= 0 || a <= 0) return;
  int s;
  const Fx y = fx_split(fx_rsqrt(n, s));
  // 1 - a0 = (E + g^2 / 2) / (beta3 8 |v|), as qv 2^(s/2 - 1 + up); above 2 it is rejected
  const Fx g4 = fx_split(fx_from_float(fabsf(g), 2));
  const fx64 T = fx_neg_log_16th(a) + ((fx_mul(g4, g4) + 1) >> 1);
  const fx64 qv = fx_mul(fx_split(fx_mul(fx_split(T), fx_split(inv_beta))), y);
  const int sh = (s >> 1) - 1 + up;
  if (qv > (sh > 0 ? (2 * kFxOne) >> (sh < 63 ? sh : 63) : 2 * kFxOne)) return;
  const fx64 yk = sh >= 0 ? qv << sh : (qv + 1) >> 1;
  const Fx us = fx_split(fx_from_float(u1, 0));
  if (fx_mul(us, us) > kFxOne - ((yk + 1) >> 1)) return;
  const fx64 a0 = kFxOne - yk;
  const fx64 norm = fx_sqrt(fx_mul(fx_split(yk), fx_split(2 * kFxOne - yk)));
  const fx64 uz = fx_from_float(u2, 0);
  const fx64 sin_theta = fx_sqrt(4 * fx_mul(fx_split(uz), fx_split(kFxOne - uz)));
  fx64 sphi, cphi;
  fx_sincos_turns(fx_from_float(u3, 0), sphi, cphi);
  const Fx ns = fx_split(fx_mul(fx_split(norm), fx_split(sin_theta)));
  const Fx A0 = fx_split(a0), A1 = fx_split(fx_mul(ns, fx_split(cphi))),
           A2 = fx_split(fx_mul(ns, fx_split(sphi))),
           A3 = fx_split(fx_mul(fx_split(norm), fx_split(2 * uz - kFxOne)));
  const Fx b0 = fx_split(fx_mul(fx_prescale(v[0], s), y)),
           b1 = fx_split(fx_mul(fx_prescale(v[1], s), y)),
           b2 = fx_split(fx_mul(fx_prescale(v[2], s), y)),
           b3 = fx_split(fx_mul(fx_prescale(v[3], s), y));
  const Fx n1 = fx_neg(A1), n2 = fx_neg(A2), n3 = fx_neg(A3);
  FxAcc c0 = fx_acc(), c1 = fx_acc(), c2 = fx_acc(), c3 = fx_acc();
  fx_mac(c0, A0, b0);
  fx_mac(c1, A0, b1);
  fx_mac(c2, A0, b2);
  fx_mac(c3, A0, b3);
  fx_mac(c0, n1, b1);
  fx_mac(c1, A1, b0);
  fx_mac(c2, A1, b3);
  fx_mac(c3, n1, b2);
  fx_mac(c0, n2, b2);
  fx_mac(c1, n2, b3);
  fx_mac(c2, A2, b0);
  fx_mac(c3, A2, b1);
  fx_mac(c0, n3, b3);
  fx_mac(c1, A3, b2);
  fx_mac(c2, n3, b1);
  fx_mac(c3, A3, b0);
  p.re = fx_split(fx_val(c0));
  p.im = fx_split(fx_val(c3));
  q.re = fx_split(fx_val(c2));
  q.im = fx_split(fx_val(c1));
}

}  // namespace gfx
