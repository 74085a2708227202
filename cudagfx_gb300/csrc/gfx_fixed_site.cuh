// gfx_fixed_site.cuh -- the functional and theta of a site in fixed point (gfx_fixed.cuh), from
// fixed-point or FP64 fields, and the block sums of the checks; shared by the single-lattice
// and the batched kernels, so that a batched copy has the bits of its single measurement.
#pragma once

#include <cmath>

#include "gfx_common.cuh"
#include "gfx_fixed.cuh"

namespace gfx {

__device__ __forceinline__ CFx cfx_of(int4 v) {
  CFx z;
  z.re.h = v.x;
  z.re.l = v.y;
  z.im.h = v.z;
  z.im.l = v.w;
  return z;
}

// |a b^+ - delta|, the larger of its parts, in FP32: rows that pass kFxUnitary keep the
// bounds of gfx_fixed.cuh
constexpr float kFxUnitary = 1e-3f;
__device__ __forceinline__ float fx_overlap(const CFx (&a)[3], const CFx (&b)[3], bool same) {
  const float s = 1.0f / 536870912.0f;
  float re = same ? -1.0f : 0.0f, im = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float ar = s * (float)a[k].re.h, ai = s * (float)a[k].im.h;
    const float br = s * (float)b[k].re.h, bi = s * (float)b[k].im.h;
    re = fmaf(ar, br, fmaf(ai, bi, re));
    im = fmaf(ai, br, fmaf(-ar, bi, im));
  }
  return fmaxf(fabsf(re), fabsf(im));
}

// Re tr X and tr[Delta Delta^+] of a site from X / 8 (site_functional): f on a grid of
// 2^-49 (exact sums of integers follow), d in FP64 from squares formed at the scale of the
// largest entry
__device__ __forceinline__ void site_functional_fx(const MFx& g, const CV (&w)[3][3], fx64& f,
                                                   double& d) {
  CV X[3][3];
  fx_x8(X, g, w);
  f = (X[0][0].re + X[1][1].re + X[2][2].re + 256) >> 9;
  // with u_a = 3 Im X_aa - Im tr X and r, m the off-diagonal Re X_ab - Re X_ba,
  // Im X_ab + Im X_ba:  d = sum u^2 / 9 + sum (r^2 + m^2) / 2 = (2 sum u^2 + 9 sum (..)) / 18
  fx64 im[3], u[3], o[6];
#pragma unroll
  for (int a = 0; a < 3; a++) im[a] = X[a][a].im >> 2;  // a grid of 2^-59: |u| <= 6
  const fx64 tim = im[0] + im[1] + im[2];
  fx64 most = 1;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    u[a] = 3 * im[a] - tim;
    most |= u[a] < 0 ? -u[a] : u[a];
    const int p = a == 2 ? 1 : 0, q = a == 0 ? 1 : 2;
    o[2 * a] = (X[p][q].re - X[q][p].re) >> 2;
    o[2 * a + 1] = (X[p][q].im + X[q][p].im) >> 2;
#pragma unroll
    for (int k = 0; k < 2; k++) most |= o[2 * a + k] < 0 ? -o[2 * a + k] : o[2 * a + k];
  }
  // scaled by 2^sh to below 2^59 (1/4 on the grid of 2^-61) and as close to it as possible
  const int sh = fx_clz(most) - 5;
  FxAcc su = fx_acc(), so = fx_acc();
#pragma unroll
  for (int a = 0; a < 3; a++) {
    fx_sqr(su, fx_split(sh >= 0 ? u[a] << sh : u[a] >> -sh));
    fx_sqr(so, fx_split(sh >= 0 ? o[2 * a] << sh : o[2 * a] >> -sh));
    fx_sqr(so, fx_split(sh >= 0 ? o[2 * a + 1] << sh : o[2 * a + 1] >> -sh));
  }
  // X / 8 was scaled by 2^(sh - 2): the sum is d 18 / 64 2^(2 sh - 4), on a grid of 2^-58
  const fx64 t = 2 * fx_sqr_val(su) + 9 * fx_sqr_val(so);
  d = (double)t * (64.0 / 18.0) *
      __longlong_as_double((long long)(1023 - 58 + 4 - 2 * sh) << 52);
}

// block sums of f (exact) and d (FP64, fixed order) and the largest d; block_reduce3's place
__device__ __forceinline__ void block_reduce_fx(fx64 f, double d, double* out) {
  __shared__ fx64 shf[32];
  __shared__ double shd[2][32];
  long long m = __double_as_longlong(d);  // d >= 0: ordered as integers
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    f += __shfl_xor_sync(0xffffffffu, f, o);
    d += __shfl_xor_sync(0xffffffffu, d, o);
    const long long b = __shfl_xor_sync(0xffffffffu, m, o);
    m = b > m ? b : m;
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    shf[w] = f;
    shd[0][w] = d;
    shd[1][w] = __longlong_as_double(m);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    double ds = shd[0][0], ms = shd[1][0];
    fx64 fs = shf[0];
    for (int k = 1; k < nw; k++) {
      fs += shf[k];
      ds += shd[0][k];
      ms = fmax(ms, shd[1][k]);
    }
    out[0] = (double)fs * (1.0 / (double)(1ll << 49));
    out[1] = ds;
    out[2] = ms;
  }
}


// ---------------------------------------------------------------------------
// the same from FP64 links and g
// ---------------------------------------------------------------------------
// Whether the matrices of a site keep the bounds of gfx_fixed.cuh: entries below 2 and rows
// of norm 1 to kFxUnitary (and rows 0, 1 of an 18-real link orthogonal to it).  Then columns
// are below sqrt(2) (12 reals: row 2 is orthogonal to rows 0, 1) or 1.42 and the star below
// 9.7, its columns' 1-norm / 8 below 5.2.
struct FxGuard {
  uint32_t most = 0;
  float worst = 0.0f;
  __device__ __forceinline__ void row(const CFFx (&r)[3]) {
    const float s = 1.0f / 536870912.0f;
    float n = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; k++)
      n = fmaf(r[k].re.hf, r[k].re.hf, fmaf(r[k].im.hf, r[k].im.hf, n));
    worst = fmaxf(worst, fabsf(fmaf(n * s, s, -1.0f)));
  }
  __device__ __forceinline__ void orthogonal(const CFFx (&a)[3], const CFFx (&b)[3]) {
    const float s = 1.0f / 536870912.0f;
    float re = 0.0f, im = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      re = fmaf(a[k].re.hf, b[k].re.hf, fmaf(a[k].im.hf, b[k].im.hf, re));
      im = fmaf(a[k].im.hf, b[k].re.hf, fmaf(-a[k].re.hf, b[k].im.hf, im));
    }
    worst = fmaxf(worst, fmaxf(fabsf(re * s), fabsf(im * s)) * s);
  }
  __device__ __forceinline__ bool ok() const { return fx_in_range(most) && worst <= kFxUnitary; }
};

// row 2 = conj(row 0 x row 1), its cross terms in FP32 as in the star
__device__ __forceinline__ void row2_ffx(CFFx (&m)[3][3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int p = k == 2 ? 0 : k + 1, q = k == 0 ? 2 : k - 1;
    FAcc re = {0, 0.0f}, im = {0, 0.0f};  // conj(m0p m1q - m0q m1p)
    fx_fmac(re, m[0][p].re, m[1][q].re);
    fx_fmac(im, m[0][p].re, fx_neg(m[1][q].im));
    fx_fmac(re, m[0][p].im, fx_neg(m[1][q].im));
    fx_fmac(im, m[0][p].im, fx_neg(m[1][q].re));
    fx_fmac(re, m[0][q].re, fx_neg(m[1][p].re));
    fx_fmac(im, m[0][q].re, m[1][p].im);
    fx_fmac(re, m[0][q].im, m[1][p].im);
    fx_fmac(im, m[0][q].im, m[1][p].re);
    CV v;
    v.re = fx_fval(re) << 3;
    v.im = fx_fval(im) << 3;
    m[2][k] = fx_float(fx_split(v));
  }
}

// An FP64 matrix of NR reals from its place in shared memory (stage_planes); row 2 of 12 reals
// is left to the caller
template <int NR>
__device__ __forceinline__ void load_rows_fx(const int4* place, MFx& m, CFFx (&f)[3][3],
                                             FxGuard& guard) {
#pragma unroll
  for (int k = 0; k < NR / 2; k++) {
    const int4 v = place[k * blockDim.x];
    CV z;
    z.re = fx_from_double(__hiloint2double(v.y, v.x), guard.most);
    z.im = fx_from_double(__hiloint2double(v.w, v.z), guard.most);
    m.e[k / 3][k % 3] = fx_split(z);
    f[k / 3][k % 3] = fx_float(m.e[k / 3][k % 3]);
  }
  guard.row(f[0]);
  guard.row(f[1]);
  if (NR == 18) {
    guard.row(f[2]);
    guard.orthogonal(f[0], f[1]);
  }
}
template <int NR>
__device__ __forceinline__ void load_fp64_fx(const int4* place, CFFx (&m)[3][3], FxGuard& guard) {
  MFx x;
  load_rows_fx<NR>(place, x, m, guard);
  if (NR == 12) row2_ffx(m);
}
// a link and a g with the row 2 that they have as fixed-point fields: a link's from FP64
// (links_to_fx_kernel), a g's in fixed point (g_to_fx_kernel)
template <int NR>
__device__ __forceinline__ void load_link_fx(const int4* place, CFFx (&f)[3][3], FxGuard& guard) {
  MFx x;
  load_rows_fx<NR>(place, x, f, guard);
  if (NR == 12) {
    Mat3<double> d;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const int4 v = place[k * blockDim.x];
      d.e[k / 3][k % 3] = cmk(__hiloint2double(v.y, v.x), __hiloint2double(v.w, v.z));
    }
    row2_from_01(d);
    uint32_t most = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      CV z;
      z.re = fx_from_double(d.e[2][k].re, most);
      z.im = fx_from_double(d.e[2][k].im, most);
      f[2][k] = fx_float(fx_split(z));
    }
  }
}
__device__ __forceinline__ void load_g_fx(const int4* place, CFFx (&f)[3][3], FxGuard& guard) {
  MFx x;
  load_rows_fx<12>(place, x, f, guard);
  fx_row2(x);
#pragma unroll
  for (int k = 0; k < 3; k++) f[2][k] = fx_float(x.e[2][k]);
}

// N planes of 16 bytes copied to shared memory, vector k of thread t at [k * blockDim.x + t];
// a thread reads only what it copied itself, so no barrier is needed
__device__ __forceinline__ void cp_async16(int4* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void stage_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
template <int N, typename V>
__device__ __forceinline__ void stage_planes(int4* place, const V* __restrict__ src, size_t vh) {
#pragma unroll
  for (int k = 0; k < N; k++) cp_async16(place + k * blockDim.x, src + k * vh);
  stage_commit();
}

// ---------------------------------------------------------------------------
// a site of the fixed-point fields
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load_fx(const int4* __restrict__ base, size_t stride, int i,
                                        MFx& m) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const int4 v = ld_field(base + k * stride + i);
    CFx& z = m.e[k / 3][k % 3];
    z.re.h = v.x;
    z.re.l = v.y;
    z.im.h = v.z;
    z.im.l = v.w;
  }
}
__device__ __forceinline__ void store_fx(int4* __restrict__ base, size_t stride, int i,
                                         const MFx& m) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const CFx& z = m.e[k / 3][k % 3];
    base[k * stride + i] = make_int4(z.re.h, z.re.l, z.im.h, z.im.l);
  }
}

// The fields of one product (a link and a g, nine vectors each) are copied to shared memory
// while the product before it is formed: the link into the place that the last one left for
// registers, g into the other of two places (stage_planes).
constexpr int kFxPlaces = 3;
constexpr int kFxBlock = 128;  // most threads of a block
inline size_t fx_stage_bytes(int block) { return (size_t)kFxPlaces * 9 * sizeof(int4) * block; }
__device__ __forceinline__ void row_fx(const int4* place, int r, CFFx (&z)[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) z[k] = fx_float(cfx_of(place[(3 * r + k) * blockDim.x]));
}

// One direction at a time: the loop is kept rolled, so that it stays in the instruction
// cache.  Of a product, the link is held whole and g comes row by row.  At most three copies
// are under way: g and the link of the next product, in this order.
template <int NDIR>
__device__ __forceinline__ void star_fx(const Lattice& L, const Site& c, int parity,
                                        const int4* __restrict__ U, const int4* __restrict__ G,
                                        int4* smem, CV (&w)[3][3]) {
  const size_t vh = (size_t)L.vh;
  const int q = 1 - parity;
  const int4* Gq = G + (size_t)q * 9 * vh;
  const int4* Up = U + (size_t)parity * 36 * vh + c.i;
  const int4* Uq = U + (size_t)q * 36 * vh;
  int4* su = smem + threadIdx.x;
  int4* sf = su + 9 * blockDim.x;
  int4* sb = sf + 9 * blockDim.x;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) w[i][j].re = w[i][j].im = 0;
  stage_planes<9>(sf, Gq + nb_fwd(L, c, 0), vh);
  stage_planes<9>(su, Up, vh);
#pragma unroll 1
  for (int mu = 0; mu < NDIR; mu++) {
    CFFx a[3][3], b[3];
    const int jb = nb_bwd(L, c, mu);
    stage_planes<9>(sb, Gq + jb, vh);
    stage_wait<1>();
#pragma unroll
    for (int r = 0; r < 3; r++) row_fx(su, r, a[r]);
    stage_planes<9>(su, Uq + (size_t)mu * 9 * vh + jb, vh);
#pragma unroll
    for (int r = 0; r < 3; r++) {
      row_fx(sf, r, b);
      fx_star_fwd(w, r, a, b);
    }
    const bool more = mu + 1 < NDIR;
    if (more) stage_planes<9>(sf, Gq + nb_fwd(L, c, mu + 1), vh);
    else stage_commit();
    stage_wait<1>();
#pragma unroll
    for (int r = 0; r < 3; r++) row_fx(su, r, a[r]);
    if (more) stage_planes<9>(su, Up + (size_t)(mu + 1) * 9 * vh, vh);
    else stage_commit();
#pragma unroll
    for (int r = 0; r < 3; r++) {
      row_fx(sb, r, b);
      fx_star_bwd(w, r, a, b);
    }
  }
}

inline FxOmega fx_omega(double omega) {
  FxOmega om;
  om.w4 = (fx64)std::llrint(std::ldexp(omega, 59));
  om.c4 = (fx64)std::llrint(std::ldexp(omega * (omega - 1.0), 58));
  return om;
}

// the overrelaxation update of a site, in place
template <int NDIR>
__device__ __forceinline__ void or_site_fx(const Lattice& L, const Site& c, int parity,
                                           const int4* U, int4* G, FxOmega om, int4* smem) {
  const size_t vh = (size_t)L.vh;
  CV w[3][3];
  star_fx<NDIR>(L, c, parity, U, G, smem, w);
  int4* Gp = G + (size_t)parity * 9 * vh;
  MFx g;
  load_fx(Gp, vh, c.i, g);
  if (fx_or_update(g, w, om)) store_fx(Gp, vh, c.i, g);
}
// its contribution to a check
template <int NDIR>
__device__ __forceinline__ void measure_site_fx(const Lattice& L, const Site& c, int parity,
                                                const int4* U, const int4* G, int4* smem, fx64& f,
                                                double& d) {
  CV w[3][3];
  star_fx<NDIR>(L, c, parity, U, G, smem, w);
  MFx g;
  load_fx(G + (size_t)parity * 9 * L.vh, (size_t)L.vh, c.i, g);
  site_functional_fx(g, w, f, d);
}

// a site's contribution to a check: in fixed point, or (fp64) in FP64 for fields outside
// the bounds of the fixed-point arithmetic
struct SiteSums {
  fx64 f = 0;  // a grid of 2^-49
  double f64 = 0.0, d = 0.0;
  bool fp64 = false;
};

template <int NRU, int NDIR>
__device__ __noinline__ void measure_site_fp64(const Lattice& L, const Site& c, int parity,
                                               const double2* __restrict__ U,
                                               const double2* __restrict__ G, double& f,
                                               double& d) {
  Mat3<double> star, g;
  compute_star<double, double, NRU, double, 12, NDIR>(L, c, parity, U, G, star);
  Field<double, 12>::load(G + (size_t)parity * 6 * L.vh, (size_t)L.vh, c.i, g);
  site_functional(g, star, f, d);
}

// The FP64 pipe made the FP64 measurement as long as two thirds of an FP64 sweep (2.4 ms on
// 32^4, 12 reals; 1250 FP64 operations a site); here it takes 0.67 ms.  A site converts 204
// reals on the ALU (about 15 operations each), the largest part.  Row 2 of links (12 reals, in
// FP64: that pipe is 51% busy) and of g (in fixed point) is that of the fixed-point fields, so that
// both functionals have the same bits; with all of it from FP32 cross terms it took 0.57 ms.  The links and g of the next product are copied to shared memory meanwhile
// (two places each).
template <int NRU, int NDIR>
__device__ __forceinline__ void measure_site(const Lattice& L, const Site& c, int parity,
                                             const double2* __restrict__ U,
                                             const double2* __restrict__ G, int4* smem,
                                             SiteSums& v) {
  constexpr int NCU = NRU / 2;
  const size_t vh = (size_t)L.vh;
  const int q = 1 - parity;
  const double2* Gq = G + (size_t)q * 6 * vh;
  const double2* Up = U + (size_t)parity * 4 * NCU * vh + c.i;
  const double2* Uq = U + (size_t)q * 4 * NCU * vh;
  int4* sf = smem + threadIdx.x;
  int4* sb = sf + (NCU + 6) * blockDim.x;
  FxGuard guard;
  CV w[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) w[i][j].re = w[i][j].im = 0;
  auto stage = [&](int4* place, const double2* u, const double2* g) {
#pragma unroll
    for (int k = 0; k < NCU; k++) cp_async16(place + k * blockDim.x, u + k * vh);
    stage_planes<6>(place + NCU * blockDim.x, g, vh);
  };
  stage(sf, Up, Gq + nb_fwd(L, c, 0));
#pragma unroll 1
  for (int mu = 0; mu < NDIR; mu++) {
    CFFx a[3][3], b[3][3];
    const int jb = nb_bwd(L, c, mu);
    stage(sb, Uq + (size_t)mu * NCU * vh + jb, Gq + jb);
    stage_wait<1>();
    load_link_fx<NRU>(sf, a, guard);
    load_g_fx(sf + NCU * blockDim.x, b, guard);
    if (mu + 1 < NDIR)
      stage(sf, Up + (size_t)(mu + 1) * NCU * vh, Gq + nb_fwd(L, c, mu + 1));
    else
      stage_planes<6>(sf, G + (size_t)parity * 6 * vh + c.i, vh);  // the site's own g
#pragma unroll
    for (int r = 0; r < 3; r++) fx_star_fwd(w, r, a, b[r]);
    stage_wait<1>();
    load_link_fx<NRU>(sb, a, guard);
    load_g_fx(sb + NCU * blockDim.x, b, guard);
#pragma unroll
    for (int r = 0; r < 3; r++) fx_star_bwd(w, r, a, b[r]);
  }
  stage_wait<0>();
  MFx g;
  CFFx rows[2][3];
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int4 x = sf[k * blockDim.x];
    CV z;
    z.re = fx_from_double(__hiloint2double(x.y, x.x), guard.most);
    z.im = fx_from_double(__hiloint2double(x.w, x.z), guard.most);
    g.e[k / 3][k % 3] = fx_split(z);
    rows[k / 3][k % 3] = fx_float(g.e[k / 3][k % 3]);
  }
  guard.row(rows[0]);
  guard.row(rows[1]);
  if (guard.ok()) {
    fx_row2(g);
    site_functional_fx(g, w, v.f, v.d);
  } else {
    measure_site_fp64<NRU, NDIR>(L, c, parity, U, G, v.f64, v.d);
    v.fp64 = true;
  }
}
template <int NRU>
constexpr size_t measure_site_bytes(int block) {
  return (size_t)2 * (NRU / 2 + 6) * sizeof(int4) * block;
}

// the sums of a block: exact in f where every site is in fixed point, else in FP64
__device__ __forceinline__ void block_reduce_sites(const SiteSums& v, double* out) {
  if (!__syncthreads_or(v.fp64)) {
    block_reduce_fx(v.f, v.d, out);
    return;
  }
  const double f = v.fp64 ? v.f64 : (double)v.f * (1.0 / (double)(1ll << 49));
  block_reduce3(f, v.d, v.d, out);
}

}  // namespace gfx
