// gfx_fixed_hb.cu -- the FP64-accurate Kennedy-Pendleton link heatbath in 64-bit fixed point
// (gfx_fixed.cuh, gfx_fixed_kp.cuh), on the fixed-point links that gfx_fixed.cu converts.
#include <cmath>

#include "gfx_fixed_kp.cuh"
#include "gfx_fixed_site.cuh"
#include "gfx_internal.h"

namespace gfx {

namespace {
constexpr int kHbBlock = 128;
constexpr int kHbPlaces = 4;  // the three links of a term and the product of two

struct Pos {
  int x[4];
};
__device__ __forceinline__ Pos step(const Lattice& L, Pos c, int mu, int d) {
  const int n[4] = {L.lx, L.ly, L.lz, L.lt};
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k == mu) {
      const int v = c.x[k] + d;
      c.x[k] = v < 0 ? v + n[k] : v >= n[k] ? v - n[k] : v;
    }
  return c;
}
// the planes of link (c, mu) at c's index
__device__ __forceinline__ const int4* link_at(const Lattice& L, const int4* __restrict__ U, Pos c,
                                               int mu) {
  const int p = (c.x[0] + c.x[1] + c.x[2] + c.x[3]) & 1;
  const int i = (c.x[0] >> 1) + L.lxh * (c.x[1] + L.ly * (c.x[2] + L.lz * c.x[3]));
  return U + (size_t)(p * 4 + mu) * 9 * L.vh + i;
}
__device__ __forceinline__ CFFx vec_ffx(const int4* place, int k) {
  return fx_float(cfx_of(place[k * blockDim.x]));
}
__device__ __forceinline__ void row_ffx(const int4* place, int r, CFFx (&z)[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) z[k] = vec_ffx(place, 3 * r + k);
}
__device__ __forceinline__ void mat_ffx(const int4* place, CFFx (&m)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; r++) row_ffx(place, r, m[r]);
}
__device__ __forceinline__ cplx<double> fp64_of(CFx z) {
  const CV v = fx_join(z);
  return cmk<double>(fx_to_double(v.re), fx_to_double(v.im));
}
// x or -x without a branch
__device__ __forceinline__ FFx fx_neg_if(bool neg, FFx x) {
  const float s = neg ? -1.0f : 1.0f;
  x.h = neg ? -x.h : x.h;
  x.hf *= s;
  x.lf *= s;
  return x;
}
__device__ __noinline__ void draw(CV xaa, CV xbb, CV xab, CV xba, fx64 inv_beta, float g, float4 u,
                                  CFx& p, CFx& q) {
  fx_kp(xaa.re + xbb.re, -xab.im - xba.im, xba.re - xab.re, xbb.im - xaa.im, inv_beta, g, u.x,
        u.y, u.z, u.w, p, q);
}
}  // namespace

// link_heatbath_kernel<NR, 1> (heatbath_thermalization.cu:235-308, 493-550, with the
// Kennedy-Pendleton draw).  In FP64 an update took about 2650 operations of the FP64 pipe: 2.2 ms
// for the 524,288 links of a launch on 32^4; here 0.37 ms (14,480 instructions a link, 3,170 of
// them mad.wide; FMA-heavy half 59% busy, 12 warps an SM).  The six staple terms are two products
// each: forward P = A B^+ and P C^+ with the links A = U_mu(x+nu), B = U_nu(x+mu), C = U_mu(x);
// backward (B A)^+ C with A = U_mu(x+nu-mu), B = U_nu(x-mu), C = U_mu(x-mu), which is
// conj(P C'^+) with P = A^T B^T and C' = C^T.  So one loop body does both, on transposed indexes
// and a sum that is kept conjugated between; written out for both, and for each row of P, the
// kernel was bound by the fetch of its instructions (1.7 of 6.7 cycles an instruction; 0.40 ms).
// A term's first product goes through shared memory, where its rows become those of the second,
// and the links of the next term are copied while this one's are in use.
__global__ void __launch_bounds__(kHbBlock, 3) link_heatbath_fx_kernel(
    Lattice L, int4* U, int parity, int nu, fx64 inv_beta, const float* __restrict__ gauss,
    const float4* __restrict__ unif4) {
  extern __shared__ int4 fx_smem[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.vh) return;
  const size_t vh = (size_t)L.vh;
  const Site c = site_of(L, i, parity);
  const Pos x = {{2 * c.xh + c.s, c.y, c.z, c.t}};
  const Pos xpn = step(L, x, nu, 1);
  int4* sa = fx_smem + threadIdx.x;
  int4* sb = sa + 9 * blockDim.x;
  int4* sc = sb + 9 * blockDim.x;
  int4* sp = sc + 9 * blockDim.x;
  // links A, B, C (k = 0, 1, 2) of term t: mu the t/2-th direction but nu, t odd: backward
  auto source = [&](int t, int k) {
    const int m = t >> 1, mu = m + (m >= nu ? 1 : 0);
    if (t & 1) {
      if (k == 0) return link_at(L, U, step(L, xpn, mu, -1), mu);
      return link_at(L, U, step(L, x, mu, -1), k == 1 ? nu : mu);
    }
    if (k == 1) return link_at(L, U, step(L, x, mu, 1), nu);
    return link_at(L, U, k == 0 ? xpn : x, mu);
  };
  auto stage = [&](int4* place, int t, int k) {
    if (t < 6) stage_planes<9>(place, source(t, k), vh);
    else stage_commit();
  };
  CV S[3][3];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int k = 0; k < 3; k++) S[r][k].re = S[r][k].im = 0;
  stage(sa, 0, 0);
  stage(sb, 0, 1);
  stage(sc, 0, 2);
#pragma unroll 1
  for (int t = 0; t < 6; t++) {
    const bool back = t & 1;
    const int dr = back ? 1 : 3, dk = back ? 3 : 1;
    CFFx a[3][3], b[3];
    stage_wait<1>();
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int k = 0; k < 3; k++) a[r][k] = vec_ffx(sa, dr * r + dk * k);
    stage(sa, t + 1, 0);
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
      row_ffx(sb, r, b);
#pragma unroll
      for (int k = 0; k < 3; k++) b[k].im = fx_neg_if(back, b[k].im);
      CV P[3][3];
#pragma unroll
      for (int k = 0; k < 3; k++) P[k][0].re = P[k][0].im = 0;
      fx_star_fwd(P, 0, a, b);
      // on a grid of 2^-58, as words
#pragma unroll
      for (int k = 0; k < 3; k++) {
        CV v;
        v.re = P[k][0].re << 3;
        v.im = P[k][0].im << 3;
        const CFx z = fx_split(v);
        sp[(3 * k + r) * blockDim.x] = make_int4(z.re.h, z.re.l, z.im.h, z.im.l);
      }
    }
    stage(sb, t + 1, 1);
    stage_wait<2>();
    mat_ffx(sp, a);
#pragma unroll
    for (int r = 0; r < 3; r++) {
#pragma unroll
      for (int k = 0; k < 3; k++) b[k] = vec_ffx(sc, dr * r + dk * k);
      fx_star_fwd(S, r, a, b);
    }
    stage(sc, t + 1, 2);
    // conjugated for a backward term, back again after it
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int k = 0; k < 3; k++) S[r][k].im = -S[r][k].im;
  }
  int4* blk = U + (size_t)(parity * 4 + nu) * 9 * vh;
  MFx g;
#pragma unroll
  for (int k = 0; k < 9; k++) g.e[k / 3][k % 3] = cfx_of(blk[k * vh + i]);
  CV X[3][3];
  fx_x8(X, g, S);
  // the three subgroups, as in fx_or_update; subgroup s draws slot 4 i + ((nu + s) & 3)
  auto slot = [&](int s) { return 4 * i + ((nu + s) & 3); };
  CFx p1, q1, p2, q2, p3, q3;
  draw(X[0][0], X[1][1], X[0][1], X[1][0], inv_beta, __ldg(gauss + slot(0)), __ldg(unif4 + slot(0)),
       p1, q1);
  CV x00, x01, x02, x11, x12;
  {
    const CFx a0 = fx_split(X[0][0]), a1 = fx_split(X[0][1]), a2 = fx_split(X[0][2]),
              b0 = fx_split(X[1][0]), b1 = fx_split(X[1][1]), b2 = fx_split(X[1][2]);
    x00 = fx_high(p1, q1, a0, b0);
    x01 = fx_high(p1, q1, a1, b1);
    x02 = fx_high(p1, q1, a2, b2);
    x11 = fx_low(p1, q1, a1, b1);
    x12 = fx_low(p1, q1, a2, b2);
  }
  draw(x00, X[2][2], x02, X[2][0], inv_beta, __ldg(gauss + slot(1)), __ldg(unif4 + slot(1)), p2, q2);
  const CV y21 = fx_low(p2, q2, fx_split(x01), fx_split(X[2][1]));
  const CV y22 = fx_low(p2, q2, fx_split(x02), fx_split(X[2][2]));
  draw(x11, y22, x12, y21, inv_beta, __ldg(gauss + slot(2)), __ldg(unif4 + slot(2)), p3, q3);
  // rows 0, 1 of S3 S2 S1, and of its product with the link
  CFx s[2][3];
  {
    const CFx nq2c = fx_neg(fx_conj(q2));
    const CFx t0 = fx_split(fx_cmul(nq2c, p1)), t1 = fx_split(fx_cmul(nq2c, q1));
    s[0][0] = fx_split(fx_cmul(p2, p1));
    s[0][1] = fx_split(fx_cmul(p2, q1));
    s[0][2] = q2;
    s[1][0] = fx_split(fx_high(p3, q3, fx_neg(fx_conj(q1)), t0));
    s[1][1] = fx_split(fx_high(p3, q3, fx_conj(p1), t1));
    s[1][2] = fx_split(fx_cmul(q3, fx_conj(p2)));
  }
  CV v[2][3];
#pragma unroll
  for (int r = 0; r < 2; r++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      CAcc o = fx_cacc();
#pragma unroll
      for (int k = 0; k < 3; k++) fx_cmac(o, s[r][k], g.e[k][j]);
      v[r][j] = fx_cval(o);
    }
  if (!fx_normalize(g, v)) return;
  // row 2 as links_to_fx_kernel has it from the FP64 links
  Mat3<double> d;
#pragma unroll
  for (int k = 0; k < 6; k++) d.e[k / 3][k % 3] = fp64_of(g.e[k / 3][k % 3]);
  row2_from_01(d);
  uint32_t most = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    g.e[2][k].re = fx_split(fx_from_double(d.e[2][k].re, most));
    g.e[2][k].im = fx_split(fx_from_double(d.e[2][k].im, most));
  }
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const CFx& z = g.e[k / 3][k % 3];
    blk[k * vh + i] = make_int4(z.re.h, z.re.l, z.im.h, z.im.l);
  }
}

// the FP64 links of NR reals from the fixed-point ones, whose rows 0, 1 are FP64 numbers
template <int NR>
__global__ void __launch_bounds__(128) fx_to_links_kernel(Lattice L, const int4* __restrict__ Ufx,
                                                          double2* __restrict__ U, int blk0) {
  const int blk = blk0 + blockIdx.y;  // parity*4 + mu
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.vh) return;
  const size_t vh = (size_t)L.vh;
  Mat3<double> d;
#pragma unroll
  for (int k = 0; k < 6; k++)
    d.e[k / 3][k % 3] = fp64_of(cfx_of(__ldg(Ufx + ((size_t)blk * 9 + k) * vh + i)));
  if (NR == 18) row2_from_01(d);
#pragma unroll
  for (int k = 0; k < NR / 2; k++)
    U[((size_t)blk * (NR / 2) + k) * vh + i] =
        make_double2(d.e[k / 3][k % 3].re, d.e[k / 3][k % 3].im);
}

void launch_fx_to_links(int link_nr, const Lattice& L, const void* Ufx, void* U64, int blk,
                        cudaStream_t s) {
  const dim3 grid((L.vh + 127) / 128, blk < 0 ? 8 : 1);
  const int first = blk < 0 ? 0 : blk;
  if (link_nr == 18)
    fx_to_links_kernel<18><<<grid, 128, 0, s>>>(L, (const int4*)Ufx, (double2*)U64, first);
  else
    fx_to_links_kernel<12><<<grid, 128, 0, s>>>(L, (const int4*)Ufx, (double2*)U64, first);
}

// 1 / beta3 has to stay below 4/5: (E + g^2 / 2) / 16 < 2.5 times it, times 1 / sqrt in [1, 2]
bool fx_beta_ok(double beta3) { return beta3 >= 1.25 && beta3 <= 1e6; }

static size_t heatbath_fx_bytes(int block) {
  return (size_t)kHbPlaces * 9 * sizeof(int4) * block;
}

bool fx_heatbath_setup() {
  return cudaFuncSetAttribute((const void*)link_heatbath_fx_kernel,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)heatbath_fx_bytes(kHbBlock)) == cudaSuccess;
}

void launch_link_heatbath_fx(const Lattice& L, void* Ufx, int parity, int nu, double beta3,
                             const float* gauss, const float* unif, cudaStream_t s) {
  constexpr int block = kHbBlock;
  link_heatbath_fx_kernel<<<(L.vh + block - 1) / block, block, heatbath_fx_bytes(block), s>>>(
      L, (int4*)Ufx, parity, nu, (fx64)std::llrint(std::ldexp(1.0 / beta3, 61)), gauss,
      (const float4*)unif);
}

}  // namespace gfx
