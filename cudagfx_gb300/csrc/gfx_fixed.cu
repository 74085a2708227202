// gfx_fixed.cu -- the FP64-accurate overrelaxation sweep and functional in 64-bit fixed
// point (gfx_fixed.cuh), with the conversions of links and g from and to FP64.
//
// Fields: one complex entry per 16-byte vector {re.h, re.l, im.h, im.l}, nine planes per
// matrix (all three rows, so nothing is rebuilt in the sweep), blocks as in the FP64
// 18-real layout: links (p*4 + mu)*9*vh, g p*9*vh.
#include <algorithm>
#include <cmath>

#include "gfx_common.cuh"
#include "gfx_fixed_site.cuh"
#include "gfx_internal.h"
#include "gfx_launch.cuh"

namespace gfx {

// ---------------------------------------------------------------------------
// conversions (once per set of links, once per g handed over)
// ---------------------------------------------------------------------------
// FP64 links of NR reals to fixed point; flags[0] is set when a matrix is further from
// unitary than 1e-3 (entries of 2 and more, infinities and NaN included): the bounds of
// gfx_fixed.cuh then do not hold.  HBM-bound apart from row 2 of the 12-real layout, which
// is rebuilt as the FP64 kernels rebuild it.
template <int NR>
__global__ void __launch_bounds__(128) links_to_fx_kernel(Lattice L, const double2* __restrict__ U,
                                                          int4* __restrict__ Ufx, int* flags) {
  const int blk = blockIdx.y;  // parity*4 + mu
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.vh) return;
  const size_t vh = (size_t)L.vh;
  Mat3<double> d;
  Field<double, NR>::load(U + (size_t)blk * Field<double, NR>::NCHUNK * vh, vh, i, d);
  MFx m;
  uint32_t most = 0;
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      m.e[r][c].re = fx_split(fx_from_double(d.e[r][c].re, most));
      m.e[r][c].im = fx_split(fx_from_double(d.e[r][c].im, most));
    }
  float worst = 0.0f;
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int s = r; s < 3; s++) worst = fmaxf(worst, fx_overlap(m.e[r], m.e[s], r == s));
  if (!fx_in_range(most) || worst > kFxUnitary) flags[0] = 1;  // the same value from every thread
  store_fx(Ufx + (size_t)blk * 9 * vh, vh, i, m);
}

// FP64 g (rows 0, 1) to fixed point, row 2 rebuilt; flags[1] is set when a site's rows are
// further from orthonormal than 1e-13: the update's algebra takes g as unitary, where the
// FP64 one forms g_relax g_old^+ with g as it is
__global__ void __launch_bounds__(128) g_to_fx_kernel(Lattice L, const double2* __restrict__ G,
                                                      int4* __restrict__ Gfx, int* flags) {
  const int parity = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.vh) return;
  const size_t vh = (size_t)L.vh;
  const double2* base = G + (size_t)parity * 6 * vh;
  MFx m;
  uint32_t most = 0;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const double2 v = ld_field(base + k * vh + i);
    m.e[k / 3][k % 3].re = fx_split(fx_from_double(v.x, most));
    m.e[k / 3][k % 3].im = fx_split(fx_from_double(v.y, most));
  }
  bool ok = fx_in_range(most);
  if (ok) {
    FxAcc n0 = fx_acc(), n1 = fx_acc();
    CAcc p = fx_cacc();
#pragma unroll
    for (int k = 0; k < 3; k++) {
      fx_sqr(n0, m.e[0][k].re);
      fx_sqr(n0, m.e[0][k].im);
      fx_sqr(n1, m.e[1][k].re);
      fx_sqr(n1, m.e[1][k].im);
      fx_cmacc(p, m.e[1][k], m.e[0][k]);
    }
    const CV q = fx_cval(p);
    const fx64 one = 1ll << 58, tol = 28823;  // 1 and 1e-13 on a grid of 2^-58
    ok = llabs(fx_sqr_val(n0) - one) <= tol && llabs(fx_sqr_val(n1) - one) <= tol &&
         llabs(q.re >> 3) <= tol && llabs(q.im >> 3) <= tol;
  }
  if (!ok) flags[1] = 1;
  fx_row2(m);
  store_fx(Gfx + (size_t)parity * 9 * vh, vh, i, m);
}

__global__ void __launch_bounds__(128) fx_to_g_kernel(Lattice L, const int4* __restrict__ Gfx,
                                                      double2* __restrict__ G, int parity0) {
  const int parity = parity0 + blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.vh) return;
  const size_t vh = (size_t)L.vh;
  const int4* base = Gfx + (size_t)parity * 9 * vh;
  double2* out = G + (size_t)parity * 6 * vh;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int4 v = ld_field(base + k * vh + i);
    Fx re, im;
    re.h = v.x;
    re.l = v.y;
    im.h = v.z;
    im.l = v.w;
    out[k * vh + i] = make_double2(fx_to_double(fx_join(re)), fx_to_double(fx_join(im)));
  }
}

void launch_links_to_fx(int link_nr, const Lattice& L, const void* U64, void* Ufx, int* flags,
                        cudaStream_t s) {
  const dim3 grid((L.vh + 127) / 128, 8);
  if (link_nr == 18)
    links_to_fx_kernel<18><<<grid, 128, 0, s>>>(L, (const double2*)U64, (int4*)Ufx, flags);
  else
    links_to_fx_kernel<12><<<grid, 128, 0, s>>>(L, (const double2*)U64, (int4*)Ufx, flags);
}
void launch_g_to_fx(const Lattice& L, const void* G64, void* Gfx, int* flags, cudaStream_t s) {
  const dim3 grid((L.vh + 127) / 128, 2);
  g_to_fx_kernel<<<grid, 128, 0, s>>>(L, (const double2*)G64, (int4*)Gfx, flags);
}
void launch_fx_to_g(const Lattice& L, const void* Gfx, void* G64, int parities, cudaStream_t s) {
  if (!parities) return;
  const dim3 grid((L.vh + 127) / 128, parities == 3 ? 2 : 1);
  fx_to_g_kernel<<<grid, 128, 0, s>>>(L, (const int4*)Gfx, (double2*)G64, parities == 2);
}

// ---------------------------------------------------------------------------
// the sweep and the functional
// ---------------------------------------------------------------------------
// One overrelaxation half-sweep.  The FP64 kernel (or_halfsweep_kernel<double>) was bound by
// the FP64 pipe: 1664 FP64 operations a site at 2 per SM and clock, 1.5 ms per half-sweep of
// 32^4.  Here a site takes 2300 mad.wide (32 lanes per SM and clock on one half of the FMA
// units), 1730 FP32 FMAs beside them and 4300 other instructions: 0.224 ms, with that half
// of the units 60% busy and 3.7 TB/s of fields.  Rows rounded to FP64 and norms kept from getting
// small take 0.009 of it.  Measured on 32^4 without them (0.215 ms a half-sweep): cross
// terms in mad.wide as well 0.265 ms; loads straight into registers 0.236 ms; four blocks an
// SM (128 registers, 60 bytes spilled) 0.243 ms; two blocks 0.227 ms.
template <int NDIR>
__global__ void __launch_bounds__(kFxBlock, 3) or_fx_kernel(Lattice L, const int4* U,
                                                       int4* G, int parity, FxOmega om, int rev) {
  start_after();
  const int blk = rev ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
  const int i = blk * blockDim.x + threadIdx.x;
  if (i >= L.vh) return;
  extern __shared__ int4 fx_smem[];
  or_site_fx<NDIR>(L, site_of(L, i, parity), parity, U, G, om, fx_smem);
}

// ---------------------------------------------------------------------------
// The same half-sweep with four neighbouring threads on a site, for lattices that leave an
// SM's schedulers less than a warp each: a half-sweep then lasts as long as one thread's
// instructions (12.9 us on 8^4, with four 7.4).  Thread l forms the products
// of direction l and thread j = min(l, 2) holds column j in the update; sums over the threads
// are exact and every other step is that of fx_or_update, so the result has the bits of
// or_fx_kernel.
// ---------------------------------------------------------------------------
__device__ __forceinline__ CV quad_get(CV v, int src) {
  CV r;
  r.re = __shfl_sync(0xffffffffu, v.re, src, 4);
  r.im = __shfl_sync(0xffffffffu, v.im, src, 4);
  return r;
}
__device__ __forceinline__ Fx quad_get(Fx v, int src) {
  Fx r;
  r.h = __shfl_sync(0xffffffffu, v.h, src, 4);
  r.l = __shfl_sync(0xffffffffu, v.l, src, 4);
  return r;
}
__device__ __forceinline__ CFx quad_get(CFx v, int src) {
  CFx r;
  r.re = quad_get(v.re, src);
  r.im = quad_get(v.im, src);
  return r;
}
__device__ __forceinline__ fx64 quad_sum(fx64 v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ CV pick(int j, CV a, CV b, CV c) {
  CV r;
  r.re = j == 0 ? a.re : j == 1 ? b.re : c.re;
  r.im = j == 0 ? a.im : j == 1 ? b.im : c.im;
  return r;
}
__device__ __forceinline__ Fx pick(int j, Fx a, Fx b, Fx c) {
  Fx r;
  r.h = j == 0 ? a.h : j == 1 ? b.h : c.h;
  r.l = j == 0 ? a.l : j == 1 ? b.l : c.l;
  return r;
}
__device__ __forceinline__ CFx pick(int j, CFx a, CFx b, CFx c) {
  CFx r;
  r.re = pick(j, a.re, b.re, c.re);
  r.im = pick(j, a.im, b.im, c.im);
  return r;
}
// the threads' shares of a sum, with the rounding that fx_acc starts a sum with
__device__ __forceinline__ FxAcc quad_acc(FxAcc s, bool mine) {
  FxAcc r;
  r.a = quad_sum(mine ? s.a : 0);
  r.c = quad_sum(mine ? s.c : 0) + (1ll << 28);
  return r;
}
__device__ __forceinline__ FxAcc share() {
  FxAcc s;
  s.a = s.c = 0;
  return s;
}

// fx_scale_up, fx_norm2, fx_unit and fx_beside of a row whose entries the threads hold
__device__ __forceinline__ void quad_scale_up(CV& v, bool small) {
  fx64 b = fx_bits_of(v.re) | fx_bits_of(v.im);
  b |= __shfl_xor_sync(0xffffffffu, b, 1);
  b |= __shfl_xor_sync(0xffffffffu, b, 2);
  const int up = small ? fx_room(b) : 0;
  v.re <<= up;
  v.im <<= up;
}
__device__ __forceinline__ fx64 quad_norm2(CV v, bool mine) {
  FxAcc t = share();
  fx_sqr(t, fx_split(v.re));
  fx_sqr(t, fx_split(v.im));
  return fx_sqr_val(quad_acc(t, mine));
}
__device__ __forceinline__ CV quad_unit(CV v, fx64 n) {
  int s;
  const Fx y = fx_split(fx_rsqrt(n < 1 ? 1 : n, s));
  return fx_unit(v, y, s);
}
__device__ __forceinline__ CV quad_beside(CV v, CFx z, bool mine) {
  CAcc pr;
  pr.re = share();
  pr.im = share();
  fx_cmacc(pr, fx_split(v), z);
  pr.re = quad_acc(pr.re, mine);
  pr.im = quad_acc(pr.im, mine);
  const CV o = fx_cmul(fx_neg(fx_split(fx_cval(pr))), z);
  v.re += o.re;
  v.im += o.im;
  return v;
}

template <int NDIR>
__global__ void __launch_bounds__(32) or_fx_quad_kernel(Lattice L, const int4* U,
                                                        int4* G, int parity, FxOmega om) {
  start_after();
  const int thread = blockIdx.x * blockDim.x + threadIdx.x;
  const int l = thread & 3, j = l < 2 ? l : 2;
  const bool in = thread / 4 < L.vh;
  const int i = in ? thread / 4 : L.vh - 1;  // whole warps take part in the exchanges
  const size_t vh = (size_t)L.vh;
  const int q = 1 - parity;
  const Site c = site_of(L, i, parity);
  const int4* Gq = G + (size_t)q * 9 * vh;
  int4* Gp = G + (size_t)parity * 9 * vh + i;
  MFx g;
#pragma unroll
  for (int k = 0; k < 9; k++) g.e[k / 3][k % 3] = cfx_of(ld_field(Gp + k * vh));
  CV w[3][3];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int k = 0; k < 3; k++) w[r][k].re = w[r][k].im = 0;
  if (l < NDIR) {
    CFFx a[3][3], b[3][3];
    const int4* Uf = U + (size_t)(parity * 4 + l) * 9 * vh + i;
    const int4* Gf = Gq + nb_fwd(L, c, l);
    const int jb = nb_bwd(L, c, l);
    const int4* Ub = U + (size_t)(q * 4 + l) * 9 * vh + jb;
    const int4* Gb = Gq + jb;
    int4 ub[9], gb[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
      a[k / 3][k % 3] = fx_float(cfx_of(ld_field(Uf + k * vh)));
      b[k / 3][k % 3] = fx_float(cfx_of(ld_field(Gf + k * vh)));
      ub[k] = ld_field(Ub + k * vh);
      gb[k] = ld_field(Gb + k * vh);
    }
#pragma unroll
    for (int r = 0; r < 3; r++) fx_star_fwd(w, r, a, b[r]);
#pragma unroll
    for (int k = 0; k < 9; k++) {
      a[k / 3][k % 3] = fx_float(cfx_of(ub[k]));
      b[k / 3][k % 3] = fx_float(cfx_of(gb[k]));
    }
#pragma unroll
    for (int r = 0; r < 3; r++) fx_star_bwd(w, r, a, b[r]);
  }
  // column j of w, and of X / 8 = g (w / 8)
  CFx wc[3];
#pragma unroll
  for (int r = 0; r < 3; r++) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      w[r][k].re = quad_sum(w[r][k].re);
      w[r][k].im = quad_sum(w[r][k].im);
    }
  }
  CV X[3];
  FxProj v1;
  fx64 m1;
#pragma unroll 1
  for (;;) {
#pragma unroll
    for (int r = 0; r < 3; r++) wc[r] = fx_split(pick(j, w[r][0], w[r][1], w[r][2]));
#pragma unroll
    for (int r = 0; r < 3; r++) {
      CAcc t = fx_cacc();
#pragma unroll
      for (int k = 0; k < 3; k++) fx_cmac(t, g.e[r][k], wc[k]);
      X[r] = fx_cval(t);
    }
    v1 = fx_proj(quad_get(X[0], 0), quad_get(X[1], 1), quad_get(X[0], 1), quad_get(X[1], 0));
    m1 = fx_norm2(v1);
    const bool again = m1 < kFxSmall && fx_scale_up(w);
    if (!__any_sync(0xffffffffu, again)) break;
  }
  // the three subgroups (fx_or_update), each thread rotating its column
  CFx p1, q1, p2, q2, p3, q3;
  fx_su2(v1, m1, p1, q1);
  const CFx x0 = fx_split(X[0]), x1 = fx_split(X[1]);
  const CV y0 = fx_high(p1, q1, x0, x1), y1 = fx_low(p1, q1, x0, x1);
  fx_su2(quad_get(y0, 0), quad_get(X[2], 2), quad_get(y0, 2), quad_get(X[2], 0), p2, q2);
  const CV y2 = fx_low(p2, q2, fx_split(y0), fx_split(X[2]));
  fx_su2(quad_get(y1, 1), quad_get(y2, 2), quad_get(y1, 2), quad_get(y2, 1), p3, q3);
  // column j of R = S3 S2 S1 - 1
  Fx zero;
  zero.h = zero.l = 0;
  CFx none;
  none.re = none.im = zero;
  const CFx al1 = j == 0 ? p1 : q1;
  const CFx tj = pick(j == 2, fx_split(fx_cmul(fx_neg(fx_conj(q2)), al1)), fx_conj(p2), none);
  const CFx rj = pick(j, fx_neg(fx_conj(q1)), fx_conj(p1), none);
  CV R[3];
  R[0] = pick(j == 2, fx_cmul(p2, al1), fx_join(q2), fx_join(none));
  R[1] = fx_high(p3, q3, rj, tj);
  R[2] = fx_low(p3, q3, rj, tj);
#pragma unroll
  for (int r = 0; r < 3; r++)
    if (r == j) R[r].re -= kFxOne;
  // row j of R's columns 0 and 1
  CV T[2];
  CV d0, d1;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const CV a = quad_get(R[0], k), b = quad_get(R[1], k), e = quad_get(R[2], k);
    T[k] = pick(j, a, b, e);
    if (k == 0) d0 = a;
    else d1 = b;
  }
  const CV d2 = quad_get(R[2], 2);
  const fx64 tre = ((d0.re + 1) >> 1) + ((d1.re + 1) >> 1) + ((d2.re + 1) >> 1);
  const fx64 tim = ((d0.im + 1) >> 1) + ((d1.im + 1) >> 1) + ((d2.im + 1) >> 1);
  const Fx c4 = fx_split(om.c4), c2h = fx_split(2 * om.c4);
  CV al;
  al.im = fx_mul(c2h, fx_split(tim));
  al.re = om.w4 + fx_mul(c2h, fx_split(tre + kFxOne / 2));
  const CFx alpha = fx_split(al);
  // column j of M / 2, rows 0, 1, then both rows of all threads
  CFx M[2][3];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    CAcc t = fx_cacc();
    fx_cmac(t, alpha, fx_split(R[r]));
    const CFx rt = fx_split(T[r]);
    fx_mac(t.re, c4, rt.re);
    fx_mac(t.im, c4, fx_neg(rt.im));
    CV m = fx_cval(t);
    if (j == r) m.im += 2 * al.im;
    m.re *= 2;
    m.im *= 2;
    const CFx mine = fx_split(m);
#pragma unroll
    for (int k = 0; k < 3; k++) M[r][k] = quad_get(mine, k);
  }
  // column j of the rows of (1 + M) g, halved
  CFx gc[3];
#pragma unroll
  for (int k = 0; k < 3; k++) gc[k] = pick(j, g.e[k][0], g.e[k][1], g.e[k][2]);
  CV v[2];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    CAcc o = fx_cacc();
#pragma unroll
    for (int k = 0; k < 3; k++) fx_cmac(o, M[r][k], gc[k]);
    const CV g0 = fx_join(gc[r]);
    v[r] = fx_cval(o);
    v[r].re += (g0.re + 1) >> 1;
    v[r].im += (g0.im + 1) >> 1;
  }
  // fx_normalize
  const bool mine = l < 3;
  fx64 n = quad_norm2(v[0], mine);
  bool small = n < kFxSmall;
  if (__any_sync(0xffffffffu, small)) {  // whole warps take part in the exchanges
    quad_scale_up(v[0], small);
    n = quad_norm2(v[0], mine);
  }
  bool ok = n >= 1;
  const CV u0 = quad_unit(v[0], n);
  const CFx z0 = fx_split(u0), n0 = fx_split53(u0);
  CV r1 = quad_beside(v[1], z0, mine);
  n = quad_norm2(r1, mine);
  small = n < kFxSmall;
  if (__any_sync(0xffffffffu, small)) {
    quad_scale_up(v[1], small);
    r1 = quad_beside(v[1], z0, mine);
    quad_scale_up(r1, small);
    n = quad_norm2(r1, mine);
  }
  ok = ok && n >= 1;
  const CFx n1 = fx_split53(quad_unit(r1, n));
  const int jp = j == 2 ? 0 : j + 1, jq = j == 0 ? 2 : j - 1;
  const CFx n2 = fx_split(fx_cross_conj(quad_get(n0, jp), quad_get(n1, jq), quad_get(n0, jq),
                                        quad_get(n1, jp)));
  if (in && mine && ok) {
    Gp[(size_t)j * vh] = make_int4(n0.re.h, n0.re.l, n0.im.h, n0.im.l);
    Gp[(size_t)(3 + j) * vh] = make_int4(n1.re.h, n1.re.l, n1.im.h, n1.im.l);
    Gp[(size_t)(6 + j) * vh] = make_int4(n2.re.h, n2.re.l, n2.im.h, n2.im.l);
  }
}

// the partials of measure_kernel, in its order
template <int NDIR>
__global__ void __launch_bounds__(kMeasBlock, 4) measure_fx_kernel(Lattice L,
                                                                   const int4* U,
                                                                   const int4* G,
                                                                   double* partials) {
  start_after();
  const int parity = blockIdx.y, t = blockIdx.z;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  extern __shared__ int4 fx_smem[];
  fx64 f = 0;
  double d = 0.0;
  if (k < L.st)
    measure_site_fx<NDIR>(L, site_of(L, t * L.st + k, parity), parity, U, G, fx_smem, f, d);
  block_reduce_fx(f, d,
                  partials + 3 * ((size_t)(parity * L.lt + t) * gridDim.x + blockIdx.x));
}

// The partials of measure_kernel from the FP64 fields, converted site by site (no copies to
// keep, so also for the checks of a mixed solve, which measures FP64 fields once)
template <int NRU, int NDIR>
__global__ void __launch_bounds__(kMeasBlock, 3) measure_fp64_kernel(
    Lattice L, const double2* __restrict__ U, const double2* __restrict__ G, double* partials) {
  const int parity = blockIdx.y, t = blockIdx.z;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  extern __shared__ int4 fx_smem[];
  SiteSums v;
  if (k < L.st) {
    const int i = t * L.st + k;
    measure_site<NRU, NDIR>(L, site_of(L, i, parity), parity, U, G, fx_smem, v);
  }
  block_reduce_sites(v, partials + 3 * ((size_t)(parity * L.lt + t) * gridDim.x + blockIdx.x));
}

void launch_measure_fp64(int link_nr, int ndir, const Lattice& L, const void* U64, const void* G64,
                         double* partials, cudaStream_t s) {
  const dim3 grid(measure_blocks_x(L, kMeasBlock), 2, L.lt);
  const double2 *u = (const double2*)U64, *g = (const double2*)G64;
  const size_t sm = link_nr == 18 ? measure_site_bytes<18>(kMeasBlock)
                                  : measure_site_bytes<12>(kMeasBlock);
  if (link_nr == 18) {
    if (ndir == 4) measure_fp64_kernel<18, 4><<<grid, kMeasBlock, sm, s>>>(L, u, g, partials);
    else measure_fp64_kernel<18, 3><<<grid, kMeasBlock, sm, s>>>(L, u, g, partials);
  } else {
    if (ndir == 4) measure_fp64_kernel<12, 4><<<grid, kMeasBlock, sm, s>>>(L, u, g, partials);
    else measure_fp64_kernel<12, 3><<<grid, kMeasBlock, sm, s>>>(L, u, g, partials);
  }
}

bool fx_omega_ok(double omega) { return omega >= 0.0 && omega <= 2.0; }

static int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    cudaGetLastError();
  return n;
}

// up to two warps of quads (16 sites) for each of an SM's four schedulers, 9,728 sites on 152 SMs;
// per half-sweep, a thread a site against four: 2048 sites 12.9 and 7.4 us, 8192 13.3 and 9.1,
// 9600 13.5 and 9.5, with a third warp on some schedulers 10,368 13.6 and 11.8, 12,288 13.5 and
// 12.1, with a fourth 15,120 13.7 and 16.3
bool or_fx_quads(const Lattice& L) { return L.vh <= 4 * 16 * sm_count(); }

void launch_or_fx(int ndir, const Lattice& L, const void* Ufx, void* Gfx, int parity, double omega,
                  int block, int mode, cudaStream_t s) {
  block = std::min(block, kFxBlock);
  // small lattices: blocks down to one warp, until there are two for each SM
  const int two = 2 * sm_count();
  while (block >= 64 && block % 64 == 0 && (L.vh + block - 1) / block < two) block /= 2;
  const int grid = (L.vh + block - 1) / block;
  const FxOmega om = fx_omega(omega);
  if (or_fx_quads(L)) {
    const int n = (4 * L.vh + 31) / 32;
    if (ndir == 4)
      launch_next(or_fx_quad_kernel<4>, n, 32, 0, s, L, (const int4*)Ufx, (int4*)Gfx, parity, om);
    else
      launch_next(or_fx_quad_kernel<3>, n, 32, 0, s, L, (const int4*)Ufx, (int4*)Gfx, parity, om);
    return;
  }
  const int rev = mode >= 2 ? parity : 0;
  const size_t sm = fx_stage_bytes(block);
  if (ndir == 4)
    launch_next(or_fx_kernel<4>, grid, block, sm, s, L, (const int4*)Ufx, (int4*)Gfx, parity, om,
                rev);
  else
    launch_next(or_fx_kernel<3>, grid, block, sm, s, L, (const int4*)Ufx, (int4*)Gfx, parity, om,
                rev);
}

void launch_measure_fx(int ndir, const Lattice& L, const void* Ufx, const void* Gfx,
                       double* partials, cudaStream_t s) {
  const dim3 grid(measure_blocks_x(L, kMeasBlock), 2, L.lt);
  const size_t sm = fx_stage_bytes(kMeasBlock);
  if (ndir == 4)
    launch_next(measure_fx_kernel<4>, grid, kMeasBlock, sm, s, L, (const int4*)Ufx,
                (const int4*)Gfx, partials);
  else
    launch_next(measure_fx_kernel<3>, grid, kMeasBlock, sm, s, L, (const int4*)Ufx,
                (const int4*)Gfx, partials);
}

// ---------------------------------------------------------------------------
// plaquette
// ---------------------------------------------------------------------------
// (a b)_ij
__device__ __forceinline__ CV mul_entry_ffx(const CFFx (&a)[3][3], const CFFx (&b)[3][3], int i,
                                            int j) {
  FAcc re = {0, 0.0f}, im = {0, 0.0f};
#pragma unroll
  for (int k = 0; k < 3; k++) {
    fx_fmac(re, a[i][k].re, b[k][j].re);
    fx_fmac(im, a[i][k].re, b[k][j].im);
    fx_fmac(re, a[i][k].im, fx_neg(b[k][j].im));
    fx_fmac(im, a[i][k].im, b[k][j].re);
  }
  CV v;
  v.re = fx_fval(re) << 3;
  v.im = fx_fval(im) << 3;
  return v;
}

template <int NR>
__device__ __noinline__ double plaquette_site_fp64(const Lattice& L, const double2* __restrict__ U,
                                                   const Site& c, int parity) {
  constexpr int NC = NR / 2;
  const size_t vh = (size_t)L.vh;
  const int q = 1 - parity;
  double acc = 0.0;
#pragma unroll 1
  for (int nu = 0; nu < 3; nu++)
#pragma unroll 1
    for (int mu = nu + 1; mu < 4; mu++) {
      Mat3<double> m1, m2, a, b;
      Field<double, NR>::load(U + (size_t)(parity * 4 + mu) * NC * vh, vh, c.i, m1);
      Field<double, NR>::load(U + (size_t)(q * 4 + nu) * NC * vh, vh, nb_fwd(L, c, mu), m2);
      mul(a, m1, m2);  // U_mu(x) U_nu(x+mu)
      Field<double, NR>::load(U + (size_t)(parity * 4 + nu) * NC * vh, vh, c.i, m1);
      Field<double, NR>::load(U + (size_t)(q * 4 + mu) * NC * vh, vh, nb_fwd(L, c, nu), m2);
      mul(b, m1, m2);  // U_nu(x) U_mu(x+nu)
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
          acc += a.e[i][j].re * b.e[i][j].re + a.e[i][j].im * b.e[i][j].im;
    }
  return acc;
}

// Sums of Re tr of the six plaquettes at a site (overrelax.cu:34-138), one block sum a triple.
// The FP64 pipe took 2.6 ms on 32^4 (1400 operations a site).  Here 24 links are converted and
// twelve products formed a site in 0.75 ms.  The links of the next product are copied to shared
// memory meanwhile.
template <int NR>
__global__ void __launch_bounds__(kFxBlock, 3) plaquette_fx_kernel(Lattice L,
                                                                   const double2* __restrict__ U,
                                                                   double* partials) {
  extern __shared__ int4 fx_smem[];
  constexpr int NC = NR / 2;
  const int parity = blockIdx.y, q = 1 - parity;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  SiteSums v;
  if (i < L.vh) {
    const size_t vh = (size_t)L.vh;
    const Site c = site_of(L, i, parity);
    const double2* Up = U + (size_t)parity * 4 * NC * vh + i;
    const double2* Uq = U + (size_t)q * 4 * NC * vh;
    int4* sa = fx_smem + threadIdx.x;
    int4* sb = sa + 2 * NC * blockDim.x;
    // U_a(x) and U_b(x+a)
    auto stage = [&](int4* place, int a, int b) {
      const double2* first = Up + (size_t)a * NC * vh;
#pragma unroll
      for (int k = 0; k < NC; k++) cp_async16(place + k * blockDim.x, first + k * vh);
      stage_planes<NC>(place + NC * blockDim.x, Uq + (size_t)b * NC * vh + nb_fwd(L, c, a), vh);
    };
    FxGuard guard;
    fx64 sum = 0;  // a grid of 2^-58
    int nu = 0, mu = 1;
    stage(sa, mu, nu);
#pragma unroll 1
    for (int p = 0; p < 6; p++) {
      CFFx a[3][3], b[3][3];
      CFx m[3][3];
      stage(sb, nu, mu);
      if (mu == 3) {
        nu++;
        mu = nu;
      }
      mu++;  // the next plane
      stage_wait<1>();
      load_fp64_fx<NR>(sa, a, guard);
      load_fp64_fx<NR>(sa + NC * blockDim.x, b, guard);
      if (p < 5) stage(sa, mu, nu);
      else stage_commit();
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int k = 0; k < 3; k++) m[r][k] = fx_split(mul_entry_ffx(a, b, r, k));
      stage_wait<1>();
      load_fp64_fx<NR>(sb, a, guard);
      load_fp64_fx<NR>(sb + NC * blockDim.x, b, guard);
#pragma unroll
      for (int r = 0; r < 3; r++) {
        FxAcc t = fx_acc();  // a row at a time: the bound on the cross terms is for six reals
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const CFx z = fx_split(mul_entry_ffx(a, b, r, k));
          fx_mac(t, m[r][k].re, z.re);
          fx_mac(t, m[r][k].im, z.im);
        }
        sum += t.a + ((t.c + (1ll << 31)) >> 32);
      }
    }
    if (guard.ok()) {
      v.f = (sum + 256) >> 9;
    } else {
      v.f64 = plaquette_site_fp64<NR>(L, U, c, parity);
      v.fp64 = true;
    }
  }
  block_reduce_sites(v, partials + 3 * ((size_t)parity * gridDim.x + blockIdx.x));
}

template <int NR>
static constexpr size_t plaquette_bytes() {
  return (size_t)2 * 2 * (NR / 2) * sizeof(int4) * kFxBlock;
}

void launch_plaquette_fx(int link_nr, const Lattice& L, const void* U64, double* partials,
                         cudaStream_t s) {
  const dim3 grid((L.vh + kFxBlock - 1) / kFxBlock, 2);
  if (link_nr == 18)
    plaquette_fx_kernel<18><<<grid, kFxBlock, plaquette_bytes<18>(), s>>>(
        L, (const double2*)U64, partials);
  else
    plaquette_fx_kernel<12><<<grid, kFxBlock, plaquette_bytes<12>(), s>>>(
        L, (const double2*)U64, partials);
}

// the kernels whose places in shared memory need more than a launch may ask for by default;
// called for every context (the attribute belongs to the device's context)
bool fx_setup() {
  auto most = [](const void* f, size_t bytes) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) ==
           cudaSuccess;
  };
  const size_t b = fx_stage_bytes(kFxBlock), m12 = measure_site_bytes<12>(kMeasBlock),
               m18 = measure_site_bytes<18>(kMeasBlock);
  return most((const void*)or_fx_kernel<4>, b) && most((const void*)or_fx_kernel<3>, b) &&
         most((const void*)measure_fx_kernel<4>, b) && most((const void*)measure_fx_kernel<3>, b) &&
         most((const void*)plaquette_fx_kernel<12>, plaquette_bytes<12>()) &&
         most((const void*)plaquette_fx_kernel<18>, plaquette_bytes<18>()) &&
         most((const void*)measure_fp64_kernel<12, 4>, m12) &&
         most((const void*)measure_fp64_kernel<12, 3>, m12) &&
         most((const void*)measure_fp64_kernel<18, 4>, m18) &&
         most((const void*)measure_fp64_kernel<18, 3>, m18);
}

}  // namespace gfx
