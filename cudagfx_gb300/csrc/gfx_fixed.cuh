// gfx_fixed.cuh -- SU(3) arithmetic in 64-bit fixed point on the integer units, for the
// FP64-accurate kernels.
//
// GB300 issues 2 FP64 FMAs per SM and clock, against 32 32 x 32 -> 64 bit integer
// multiply-adds (mad.wide, on one half of the FMA units), and everything the gauge-fixing update
// forms from unitary matrices is bounded: entries of links and g by 1, the star by 8.
// So a number |x| < 4 is held on a grid of 2^-61 (fx64) and, as a factor, in two words (Fx)
//     x = h 2^-29 + l 2^-61,
// one instruction apart.  A sum of products is kept in two 64-bit sums,
//     a += hx hy   (2^-58, exact),     c += hx ly + lx hy   (2^-90, exact),
// three mad.wide per real multiply-add; lx ly < 2^-60 is dropped and c is rounded into a
// once per sum.  Grid and dropped terms lie below the rounding of the FP64 kernels (2^-54
// for entries near 1/2, 2^-51 in the star): one update errs less than in FP64 on random
// SU(3) fields (tests/fixed_check.cpp), and with small stars, projections and rows
// (tests/fixed_small_check.cpp).  These are absolute bounds on matrices of norm 1: an entry
// below 2^-8 is read at 2^-61, where FP64 holds it to 53 bits, the star's cross terms are
// summed in FP32 (2^-54 of a product of 1), and a site's trace goes into the functional at 2^-49.
// So what is left of nearly cancelling stars errs up to twice as much as in FP64, and the small
// entries of links and g near the identity are right to 2^-61, not to their own 53 bits.
//
// Bounds (matrices unitary to 1e-3): a holds sums below 32, the star stays below 8.1; an
// entry's cross terms are below sum |hx ly| + |lx hy| <= 2^60 (|x|_1 + |y|_1) < 2^63, with
// the 1-norms of its factors' six reals noted where they exceed sqrt(6).  Inputs outside
// those bounds (matrices far from unitary, NaN) never reach this code: the conversions from
// FP64 check every matrix and the callers keep to FP64 arithmetic when one fails.
#pragma once

#include <cstdint>

#ifndef __CUDA_ARCH__
#include <cmath>
#include <cstring>
#endif

namespace gfx {

#ifdef __CUDACC__
#define GFX_FX __host__ __device__ __forceinline__
#else
#define GFX_FX inline
#endif

struct Fx {
  int h, l;
};
struct CFx {
  Fx re, im;
};
struct MFx {
  CFx e[3][3];
};
typedef long long fx64;  // a value on the 2^-61 grid
struct CV {
  fx64 re, im;
};
constexpr fx64 kFxOne = 1ll << 61;

// s + x y.  In PTX so that the negations of factors stay 32-bit operations (the compiler
// otherwise moves them behind the product, at three more instructions each), and as a
// product and a sum, which become one IMAD.WIDE; mad.wide.s32 became a product and two
// adds in two of five places (a sweep executed 10,090 instructions a site instead of 6,420).
GFX_FX fx64 fx_wide(int x, int y, fx64 s) {
#ifdef __CUDA_ARCH__
  fx64 r;
  asm("{ .reg .s64 t; mul.wide.s32 t, %1, %2; add.s64 %0, t, %3; }"
      : "=l"(r)
      : "r"(x), "r"(y), "l"(s));
  return r;
#else
  return s + (fx64)x * y;
#endif
}

// a sum of products
struct FxAcc {
  fx64 a, c;
};
GFX_FX FxAcc fx_acc() {
  FxAcc s;
  s.a = 0;
  s.c = 1ll << 28;  // rounds c >> 29: no step of the update may be biased, as the same error
                    // at every site of every sweep adds up to a rotation of the whole field
  return s;
}
GFX_FX void fx_mac(FxAcc& s, Fx x, Fx y) {
  s.a = fx_wide(x.h, y.h, s.a);
  s.c = fx_wide(x.h, y.l, s.c);
  s.c = fx_wide(x.l, y.h, s.c);
}
GFX_FX fx64 fx_val(const FxAcc& s) { return (s.a << 3) + (s.c >> 29); }

// the words of a value, l = its low word, and back
GFX_FX Fx fx_split(fx64 v) {
  Fx x;
  x.l = (int)(uint32_t)v;
  x.h = (int)(v >> 32) + (int)((uint32_t)v >> 31);
  return x;
}
GFX_FX fx64 fx_join(Fx x) { return (fx64)(((uint64_t)(uint32_t)x.h << 32) + (uint64_t)(fx64)x.l); }
// -x (l = -2^31, which has no negative, counts as 1 - 2^31)
GFX_FX Fx fx_neg(Fx x) {
  Fx y;
  y.h = -x.h;
  y.l = x.l > -0x7fffffff ? -x.l : 0x7fffffff;
  return y;
}
GFX_FX CFx fx_conj(CFx x) {
  x.im = fx_neg(x.im);
  return x;
}
GFX_FX CFx fx_neg(CFx x) {
  x.re = fx_neg(x.re);
  x.im = fx_neg(x.im);
  return x;
}
GFX_FX CFx fx_split(CV v) {
  CFx x;
  x.re = fx_split(v.re);
  x.im = fx_split(v.im);
  return x;
}
GFX_FX CV fx_join(CFx x) {
  CV v;
  v.re = fx_join(x.re);
  v.im = fx_join(x.im);
  return v;
}

struct CAcc {
  FxAcc re, im;
};
GFX_FX CAcc fx_cacc() {
  CAcc s;
  s.re = fx_acc();
  s.im = fx_acc();
  return s;
}
// re += x y, im += u v, interleaved
GFX_FX void fx_mac2(CAcc& s, Fx x, Fx y, Fx u, Fx v) {
  s.re.a = fx_wide(x.h, y.h, s.re.a);
  s.im.a = fx_wide(u.h, v.h, s.im.a);
  s.re.c = fx_wide(x.h, y.l, s.re.c);
  s.im.c = fx_wide(u.h, v.l, s.im.c);
  s.re.c = fx_wide(x.l, y.h, s.re.c);
  s.im.c = fx_wide(u.l, v.h, s.im.c);
}
// s += x y
GFX_FX void fx_cmac(CAcc& s, CFx x, CFx y) {
  fx_mac2(s, x.re, y.re, x.re, y.im);
  fx_mac2(s, fx_neg(x.im), y.im, x.im, y.re);
}
// s += x conj(y)
GFX_FX void fx_cmacc(CAcc& s, CFx x, CFx y) {
  fx_mac2(s, x.re, y.re, x.im, y.re);
  fx_mac2(s, x.im, y.im, fx_neg(x.re), y.im);
}
GFX_FX CV fx_cval(const CAcc& s) {
  CV v;
  v.re = fx_val(s.re);
  v.im = fx_val(s.im);
  return v;
}
GFX_FX CV fx_cmul(CFx x, CFx y) {
  CAcc s = fx_cacc();
  fx_cmac(s, x, y);
  return fx_cval(s);
}
GFX_FX fx64 fx_mul(Fx x, Fx y) {
  FxAcc t = fx_acc();
  fx_mac(t, x, y);
  return fx_val(t);
}

// conj(p q - r s)
GFX_FX CV fx_cross_conj(CFx p, CFx q, CFx r, CFx s) {
  CAcc t = fx_cacc();
  fx_cmac(t, p, q);
  fx_cmac(t, fx_neg(r), s);
  CV v = fx_cval(t);
  v.im = -v.im;
  return v;
}
// row 2 = conj(row 0 x row 1)
GFX_FX void fx_row2(MFx& m) {
  m.e[2][0] = fx_split(fx_cross_conj(m.e[0][1], m.e[1][2], m.e[0][2], m.e[1][1]));
  m.e[2][1] = fx_split(fx_cross_conj(m.e[0][2], m.e[1][0], m.e[0][0], m.e[1][2]));
  m.e[2][2] = fx_split(fx_cross_conj(m.e[0][0], m.e[1][1], m.e[0][1], m.e[1][0]));
}

// ---------------------------------------------------------------------------
// conversions
// ---------------------------------------------------------------------------
GFX_FX uint64_t fx_bits(double d) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(d);
#else
  uint64_t b;
  std::memcpy(&b, &d, 8);
  return b;
#endif
}
// d to the grid, on the integer units and without branches: exact for 2^-8 <= |d| < 2,
// truncated towards zero below.  The high words are collected in `most`: fx_in_range(most)
// says whether every |d| was below 2 (else, infinities and NaN included, the value is 0).
GFX_FX fx64 fx_from_double(double d, uint32_t& most) {
  const uint64_t b = fx_bits(d);
  const uint32_t hi = (uint32_t)(b >> 32);
  most |= hi;
  // d = m 2^(e - 1075); on the grid m 2^(e - 1014) = (m 2^9) >> (1023 - e)
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32 | (uint32_t)b) << 9;
  const uint32_t sh = 1023u - ((hi >> 20) & 0x7ffu);
  const fx64 r = (fx64)(m >> (sh < 63u ? sh : 63u));
  const fx64 s = (int32_t)hi >> 31;
  return (r ^ s) - s;
}
GFX_FX bool fx_in_range(uint32_t most) { return !(most & 0x40000000u); }
GFX_FX double fx_to_double(fx64 v) { return (double)v * (1.0 / (double)kFxOne); }

GFX_FX int fx_clz(fx64 v) {
#ifdef __CUDA_ARCH__
  return __clzll(v);
#else
  return v ? __builtin_clzll((unsigned long long)v) : 64;
#endif
}
// v rounded to 53 bits, ties to even, as (double)v is
GFX_FX fx64 fx_round53(fx64 v) {
  const int h = (int)(v >> 32) ^ (int)(v >> 63);
#ifdef __CUDA_ARCH__
  const int top = 31 - __clz(h);
#else
  const int top = h ? 31 - __builtin_clz((unsigned)h) : -1;
#endif
  const int s = top > 20 ? top - 20 : 0;  // bits to drop
  // half a unit less one, and one more where the bit above is set (s = 0: none)
  const uint32_t below = (1u << s) - 1u, lo = (uint32_t)v;
  v += (below >> 1) + ((lo >> s) & (below & 1u));
  return (fx64)((uint64_t)v & (0xffffffff00000000ull | ~below));
}

// ---------------------------------------------------------------------------
// 1 / sqrt
// ---------------------------------------------------------------------------
// a sum of squares, s += x^2, and its value on a grid of 2^-58 (below 16)
GFX_FX void fx_sqr(FxAcc& s, Fx x) {
  s.a = fx_wide(x.h, x.h, s.a);
  s.c = fx_wide(x.h, x.l, s.c);
}
GFX_FX fx64 fx_sqr_val(const FxAcc& s) { return s.a + ((s.c + (3ll << 28)) >> 31); }

// For 0 < n < 2^62 on the grid of 2^-58: y (in [1, 2]) and s even with
// 1/sqrt(n) = y 2^(s/2 - 2).  An FP32 estimate, refined by one third-order step
// y0 (1 + h/2 + 3 h^2/8), h = 1 - m y0^2 (|h| < 2^-20): relative error below 2^-57.
GFX_FX fx64 fx_rsqrt(fx64 n, int& s) {
  s = (fx_clz(n) - 2) & ~1;
  const fx64 m62 = n << s;  // m = m62 2^-62 in [1/4, 1)
  const float mf = (float)(int)(m62 >> 32) * (1.0f / 1073741824.0f);
#ifdef __CUDA_ARCH__
  const int y0 = __float2int_rn(rsqrtf(mf) * 268435456.0f);
#else
  const int y0 = (int)std::lrintf((1.0f / std::sqrt(mf)) * 268435456.0f);
#endif
  // (2 m) (y0^2 / 2)
  const fx64 h = kFxOne - fx_mul(fx_split(m62), fx_split(fx_wide(y0, y0, 0) << 4));
  const int hh = (int)(h >> 11);
  const fx64 corr = ((h + 1) >> 1) + ((3 * (fx_wide(hh, hh, 0) >> 39) + 4) >> 3);
  const fx64 step = fx_wide(y0, (int)(corr >> 11), fx_wide(y0, (int)(corr & 2047), 0) >> 11);
  return ((fx64)y0 << 33) + ((step + (1 << 16)) >> 17);
}
// v 2^(s/2 - 2): times y, v / sqrt(n).  |v| <= sqrt(n) up to rounding.
GFX_FX Fx fx_prescale(fx64 v, int s) { return fx_split(((v + 2) >> 2) << (s >> 1)); }

// ---------------------------------------------------------------------------
// the overrelaxation update
// ---------------------------------------------------------------------------
// The star w is on a grid of 2^-58 (its entries reach 8), which is w / 8 on the grid of 2^-61.
// A mad.wide holds its half of the FMA units twice as long as an FP32 FMA holds either half,
// so the star, two thirds of the products, leaves the cross terms h l to FP32, which fits in
// beside it: they are below 2^-28 and rounded at 2^-24 of that, once per product of two
// matrices.  In the star's error that is what FP64 makes of it or less (tests/fixed_check.cpp).
struct FFx {
  int h;
  float hf, lf;  // the words as floats
};
struct CFFx {
  FFx re, im;
};
GFX_FX FFx fx_float(Fx x) {
  FFx y;
  y.h = x.h;
  y.hf = (float)x.h;
  y.lf = (float)x.l;
  return y;
}
GFX_FX CFFx fx_float(CFx x) {
  CFFx y;
  y.re = fx_float(x.re);
  y.im = fx_float(x.im);
  return y;
}
GFX_FX float fx_fma(float x, float y, float s) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(x, y, s);
#else
  return std::fma(x, y, s);
#endif
}
// a sum of products on the grid of 2^-58, the cross terms (2^-90) apart
struct FAcc {
  fx64 a;
  float c;
};
GFX_FX void fx_fmac(FAcc& s, FFx x, FFx y) {
  s.a = fx_wide(x.h, y.h, s.a);
  s.c = fx_fma(x.hf, y.lf, s.c);
  s.c = fx_fma(x.lf, y.hf, s.c);
}
GFX_FX fx64 fx_fval(const FAcc& s) {
  const float c = s.c * (1.0f / 4294967296.0f);
#ifdef __CUDA_ARCH__
  return s.a + __float2int_rn(c);
#else
  return s.a + (int)std::lrintf(c);
#endif
}
GFX_FX FFx fx_neg(FFx x) {
  x.h = -x.h;
  x.hf = -x.hf;
  x.lf = -x.lf;
  return x;
}
// w_ij += sum_k a_ik conj(b_jk): row b = b_j of g, the forward term a b^+
GFX_FX void fx_star_fwd(CV (&w)[3][3], int j, const CFFx (&a)[3][3], const CFFx (&b)[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    FAcc re = {w[i][j].re, 0.0f}, im = {w[i][j].im, 0.0f};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      fx_fmac(re, a[i][k].re, b[k].re);
      fx_fmac(im, a[i][k].im, b[k].re);
      fx_fmac(re, a[i][k].im, b[k].im);
      fx_fmac(im, a[i][k].re, fx_neg(b[k].im));
    }
    w[i][j].re = fx_fval(re);
    w[i][j].im = fx_fval(im);
  }
}
// w_ij += conj(sum_k b_jk a_ki), the backward term (b a)^+
GFX_FX void fx_star_bwd(CV (&w)[3][3], int j, const CFFx (&a)[3][3], const CFFx (&b)[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    FAcc re = {w[i][j].re, 0.0f}, im = {w[i][j].im, 0.0f};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      fx_fmac(re, a[k][i].re, b[k].re);
      fx_fmac(im, a[k][i].im, fx_neg(b[k].re));
      fx_fmac(re, a[k][i].im, fx_neg(b[k].im));
      fx_fmac(im, a[k][i].re, fx_neg(b[k].im));
    }
    w[i][j].re = fx_fval(re);
    w[i][j].im = fx_fval(im);
  }
}

// The bits of |v| (of -v - 1 for a negative v); or-ed for the size of the largest of several.
GFX_FX fx64 fx_bits_of(fx64 v) { return v ^ (v >> 63); }
// Squares are summed on a grid of 2^-58, so 1/sqrt has a relative error of 2^-60 divided by the
// sum: 2^-56 for a sum of 2^-4, where FP64's is 2^-53 whatever the sum is.  Where a projection's
// or a row's sum is smaller the values are scaled up first, and so is a star below 1/32 (of 8),
// for its product with g, which is rounded at 2^-61; the update does not depend on the scale of
// any of them.  The shift brings the largest of values with these bits to [1/4, 1/2).  (Six reals
// of a row or a column then have a norm of 1.23 and a 1-norm of 3, within the bounds above.)
constexpr fx64 kFxSmall = 1ll << 54;
GFX_FX int fx_room(fx64 bits) {
  const int n = fx_clz(bits);
  return n <= 4 ? 0 : n > 63 ? 60 : n - 4;
}

// a small star scaled up; false for another
GFX_FX bool fx_scale_up(CV (&w)[3][3]) {
  fx64 b = 0;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) b |= fx_bits_of(w[i][j].re) | fx_bits_of(w[i][j].im);
  if (b >> 56 || b == 0) return false;
  const int up = fx_room(b);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      w[i][j].re <<= up;
      w[i][j].im <<= up;
    }
  return true;
}

// X / 8 = g (w / 8)
GFX_FX void fx_x8(CV (&X)[3][3], const MFx& g, const CV (&w)[3][3]) {
#pragma unroll
  for (int j = 0; j < 3; j++) {
    CFx c[3];
    Fx nim[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      c[k] = fx_split(w[k][j]);
      nim[k] = fx_neg(c[k].im);
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      CAcc s = fx_cacc();
#pragma unroll
      for (int k = 0; k < 3; k++) {
        fx_mac(s.re, g.e[i][k].re, c[k].re);
        fx_mac(s.re, g.e[i][k].im, nim[k]);
        fx_mac(s.im, g.e[i][k].re, c[k].im);
        fx_mac(s.im, g.e[i][k].im, c[k].re);
      }
      X[i][j] = fx_cval(s);
    }
  }
}

// su2_pq: the projection of subgroup (a, b) from four entries of X, its squared norm on a grid
// of 2^-58, and the unit SU(2) element (p, q).  A vanishing projection (FP64: NaN) leaves the
// subgroup unchanged.
struct FxProj {
  fx64 v0, v1, v2, v3;
};
GFX_FX FxProj fx_proj(CV xaa, CV xbb, CV xab, CV xba) {
  FxProj v;
  v.v0 = xaa.re + xbb.re;
  v.v3 = xbb.im - xaa.im;
  v.v1 = -xab.im - xba.im;
  v.v2 = xba.re - xab.re;
  return v;
}
GFX_FX fx64 fx_norm2(const FxProj& v) {
  FxAcc t = fx_acc();
  fx_sqr(t, fx_split(v.v0));
  fx_sqr(t, fx_split(v.v1));
  fx_sqr(t, fx_split(v.v2));
  fx_sqr(t, fx_split(v.v3));
  return fx_sqr_val(t);
}
GFX_FX void fx_su2(FxProj v, fx64 n, CFx& p, CFx& q) {
  if (n < kFxSmall) {
    const int up =
        fx_room(fx_bits_of(v.v0) | fx_bits_of(v.v1) | fx_bits_of(v.v2) | fx_bits_of(v.v3));
    v.v0 <<= up;
    v.v1 <<= up;
    v.v2 <<= up;
    v.v3 <<= up;
    n = fx_norm2(v);
    n = n < 1 ? 1 : n;  // 0: p = q = 0 below, then
  }
  int s;
  const Fx y = fx_split(fx_rsqrt(n, s));
  p.re = fx_split(fx_mul(fx_prescale(v.v0, s), y));
  p.im = fx_split(fx_mul(fx_prescale(v.v3, s), y));
  q.re = fx_split(fx_mul(fx_prescale(v.v2, s), y));
  q.im = fx_split(fx_mul(fx_prescale(v.v1, s), y));
  if ((v.v0 | v.v1 | v.v2 | v.v3) == 0) p.re = fx_split(kFxOne);
}
GFX_FX void fx_su2(CV xaa, CV xbb, CV xab, CV xba, CFx& p, CFx& q) {
  const FxProj v = fx_proj(xaa, xbb, xab, xba);
  fx_su2(v, fx_norm2(v), p, q);
}
// p x + q y and -conj(q) x + conj(p) y
GFX_FX CV fx_high(CFx p, CFx q, CFx x, CFx y) {
  CAcc s = fx_cacc();
  fx_cmac(s, p, x);
  fx_cmac(s, q, y);
  return fx_cval(s);
}
GFX_FX CV fx_low(CFx p, CFx q, CFx x, CFx y) {
  CAcc s = fx_cacc();
  fx_cmac(s, fx_neg(fx_conj(q)), x);
  fx_cmac(s, fx_conj(p), y);
  return fx_cval(s);
}

GFX_FX void fx_scale_up(CV (&v)[3]) {
  fx64 b = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) b |= fx_bits_of(v[k].re) | fx_bits_of(v[k].im);
  const int up = fx_room(b);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    v[k].re <<= up;
    v[k].im <<= up;
  }
}
GFX_FX fx64 fx_norm2(const CV (&v)[3]) {
  FxAcc t = fx_acc();
#pragma unroll
  for (int k = 0; k < 3; k++) {
    fx_sqr(t, fx_split(v[k].re));
    fx_sqr(t, fx_split(v[k].im));
  }
  return fx_sqr_val(t);
}
// v / sqrt(n), n = fx_norm2(v)
GFX_FX CV fx_unit(CV v, Fx y, int s) {
  CV z;
  z.re = fx_mul(fx_prescale(v.re, s), y);
  z.im = fx_mul(fx_prescale(v.im, s), y);
  return z;
}
GFX_FX void fx_unit(CV (&z)[3], const CV (&v)[3], fx64 n) {
  int s;
  const Fx y = fx_split(fx_rsqrt(n < 1 ? 1 : n, s));
#pragma unroll
  for (int k = 0; k < 3; k++) z[k] = fx_unit(v[k], y, s);
}
// r = v - (v . z) z
GFX_FX void fx_beside(CV (&r)[3], const CV (&v)[3], const CFx (&z)[3]) {
  CAcc pr = fx_cacc();
#pragma unroll
  for (int k = 0; k < 3; k++) fx_cmacc(pr, fx_split(v[k]), z[k]);
  const CFx np = fx_neg(fx_split(fx_cval(pr)));
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const CV o = fx_cmul(np, z[k]);
    r[k].re = v[k].re + o.re;
    r[k].im = v[k].im + o.im;
  }
}

// the words of v rounded to FP64
GFX_FX CFx fx_split53(CV v) {
  v.re = fx_round53(v.re);
  v.im = fx_round53(v.im);
  return fx_split(v);
}

// rows 0, 1 of v (below 2 in norm, changed here) orthonormalized into g, row 2 rebuilt.  The rows
// are FP64 numbers, so that a field that is written out as FP64 and read again is the same one:
// what a program reads, saves or sets between two calls does not change what comes after.  False
// where a row, or what its part along row 0 leaves of row 1, vanishes (FP64: NaN): the caller
// then keeps the matrix that it has
GFX_FX bool fx_normalize(MFx& g, CV (&v)[2][3]) {
  fx64 n = fx_norm2(v[0]);
  if (n < kFxSmall) {
    fx_scale_up(v[0]);
    n = fx_norm2(v[0]);
  }
  bool ok = n >= 1;
  CV u[3], r[3];
  CFx z[3];
  fx_unit(u, v[0], n);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    z[k] = fx_split(u[k]);
    g.e[0][k] = fx_split53(u[k]);
  }
  fx_beside(r, v[1], z);
  n = fx_norm2(r);
  if (n < kFxSmall) {
    fx_scale_up(v[1]);
    fx_beside(r, v[1], z);
    fx_scale_up(r);
    n = fx_norm2(r);
  }
  ok = ok && n >= 1;
  fx_unit(u, r, n);
#pragma unroll
  for (int k = 0; k < 3; k++) g.e[1][k] = fx_split53(u[k]);
  fx_row2(g);
  return ok;
}

// omega / 4 and omega (omega - 1) / 8, for 0 <= omega <= 2, on the grid
struct FxOmega {
  fx64 w4, c4;
};

// The step of or_update_composed: g <- normalize((1 + omega R + c2 R^2) g), R = S - 1, with
// R^2 from the Cayley-Hamilton relation of S in SU(3), S^2 = t S - conj(t) + S^+ (t = tr S):
//   R^2 = tau R + R + R^+ + 2 i Im tau,   tau = tr R,
// so  omega R + c2 R^2 = (omega + c2 (1 + tau)) R + c2 R^+ + 2 i c2 Im tau = M.
// Sizes: |omega + c2 (1 + tau)| <= 7 is held as a quarter, |M| <= 2.5 as a half.
// False: the new rows vanish (fx_normalize), and the site keeps its g, which g no longer holds.
GFX_FX bool fx_or_update(MFx& g, CV (&w)[3][3], FxOmega om) {
  CV X[3][3];
  FxProj v1;
  fx64 n1;
#pragma unroll 1
  do {
    fx_x8(X, g, w);
    v1 = fx_proj(X[0][0], X[1][1], X[0][1], X[1][0]);
    n1 = fx_norm2(v1);
  } while (n1 < kFxSmall && fx_scale_up(w));
  CFx p1, q1, p2, q2, p3, q3;
  fx_su2(v1, n1, p1, q1);  // subgroup (0,1)
  CV x00, x02, x11, x12, x01;
  {
    const CFx a0 = fx_split(X[0][0]), a1 = fx_split(X[0][1]), a2 = fx_split(X[0][2]),
              b0 = fx_split(X[1][0]), b1 = fx_split(X[1][1]), b2 = fx_split(X[1][2]);
    x00 = fx_high(p1, q1, a0, b0);
    x01 = fx_high(p1, q1, a1, b1);
    x02 = fx_high(p1, q1, a2, b2);
    x11 = fx_low(p1, q1, a1, b1);
    x12 = fx_low(p1, q1, a2, b2);
  }
  fx_su2(x00, X[2][2], x02, X[2][0], p2, q2);  // subgroup (0,2)
  const CV y21 = fx_low(p2, q2, fx_split(x01), fx_split(X[2][1]));
  const CV y22 = fx_low(p2, q2, fx_split(x02), fx_split(X[2][2]));
  fx_su2(x11, y22, x12, y21, p3, q3);  // subgroup (1,2)
  // R = S3 S2 S1 - 1
  CV R[3][3];
  {
    const CFx nq2c = fx_neg(fx_conj(q2)), r0 = fx_neg(fx_conj(q1)), r1 = fx_conj(p1);
    const CFx t0 = fx_split(fx_cmul(nq2c, p1)), t1 = fx_split(fx_cmul(nq2c, q1)),
              t2 = fx_conj(p2);
    R[0][0] = fx_cmul(p2, p1);
    R[0][1] = fx_cmul(p2, q1);
    R[0][2] = fx_join(q2);
    R[1][0] = fx_high(p3, q3, r0, t0);
    R[1][1] = fx_high(p3, q3, r1, t1);
    R[1][2] = fx_cmul(q3, t2);
    R[2][0] = fx_low(p3, q3, r0, t0);
    R[2][1] = fx_low(p3, q3, r1, t1);
    R[2][2] = fx_cmul(fx_conj(p3), t2);
    R[0][0].re -= kFxOne;
    R[1][1].re -= kFxOne;
    R[2][2].re -= kFxOne;
  }
  // tau / 2 and the quarter of omega + c2 (1 + tau)
  const fx64 tre = ((R[0][0].re + 1) >> 1) + ((R[1][1].re + 1) >> 1) + ((R[2][2].re + 1) >> 1);
  const fx64 tim = ((R[0][0].im + 1) >> 1) + ((R[1][1].im + 1) >> 1) + ((R[2][2].im + 1) >> 1);
  const Fx c4 = fx_split(om.c4), c2h = fx_split(2 * om.c4);
  CV al;
  al.im = fx_mul(c2h, fx_split(tim));
  al.re = om.w4 + fx_mul(c2h, fx_split(tre + kFxOne / 2));
  const CFx alpha = fx_split(al);
  CV v[2][3];  // rows of (1 + M) g, halved
#pragma unroll
  for (int r = 0; r < 2; r++) {
    CFx M[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      CAcc s = fx_cacc();
      fx_cmac(s, alpha, fx_split(R[r][j]));
      const CFx rt = fx_split(R[j][r]);
      fx_mac(s.re, c4, rt.re);
      fx_mac(s.im, c4, fx_neg(rt.im));
      CV m = fx_cval(s);
      if (j == r) m.im += 2 * al.im;
      m.re *= 2;
      m.im *= 2;
      M[j] = fx_split(m);
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const CV g0 = fx_join(g.e[r][j]);
      CAcc o = fx_cacc();
#pragma unroll
      for (int k = 0; k < 3; k++) fx_cmac(o, M[k], g.e[k][j]);
      v[r][j] = fx_cval(o);
      v[r][j].re += (g0.re + 1) >> 1;
      v[r][j].im += (g0.im + 1) >> 1;
    }
  }
  return fx_normalize(g, v);
}

}  // namespace gfx
