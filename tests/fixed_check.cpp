// The fixed-point update of gfx_fixed.cuh on the CPU against the reference's update
// (overrelax.cu:149-269, 411-417) in long double, with the same update in FP64 beside it.
//   fixed_check <cases>  prints, per spread of the random SU(3) matrices, the errors of the
// star and of rows 0, 1 of the new g, and exits non-zero when
//   * the star is off by more than 3e-14: eight products, each with the FP32 sum of its cross
//     terms off by at most 14 roundings of 2^-24 of 2 sqrt(6) 2^-30;
//   * the star's or the update's error (root mean square) is above that of FP64;
//   * a conversion from FP64 is off by the grid, or 1/sqrt by 2^-56.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "gfx_fixed.cuh"

using namespace gfx;
typedef long double L;
template <class R>
struct M {
  std::complex<R> e[3][3];
};

template <class R>
void normalize(M<R>& m) {
  auto unit = [&](int r) {
    R s = 0;
    for (int k = 0; k < 3; k++) s += std::norm(m.e[r][k]);
    for (int k = 0; k < 3; k++) m.e[r][k] /= std::sqrt(s);
  };
  unit(0);
  std::complex<R> p = 0;
  for (int k = 0; k < 3; k++) p += m.e[1][k] * std::conj(m.e[0][k]);
  for (int k = 0; k < 3; k++) m.e[1][k] -= p * m.e[0][k];
  unit(1);
  for (int k = 0; k < 3; k++) {
    const int a = (k + 1) % 3, b = (k + 2) % 3;
    m.e[2][k] = std::conj(m.e[0][a] * m.e[1][b] - m.e[0][b] * m.e[1][a]);
  }
}
template <class R>
M<R> mul(const M<R>& a, const M<R>& b) {
  M<R> r;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      r.e[i][j] = 0;
      for (int k = 0; k < 3; k++) r.e[i][j] += a.e[i][k] * b.e[k][j];
    }
  return r;
}
template <class R>
M<R> dag(const M<R>& a) {
  M<R> r;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) r.e[i][j] = std::conj(a.e[j][i]);
  return r;
}
// u[2d], g[2d] forward, u[2d+1], g[2d+1] backward
template <class R>
M<R> star(const M<R>* u, const M<R>* g) {
  M<R> w{};
  for (int d = 0; d < 4; d++) {
    const M<R> f = mul(u[2 * d], dag(g[2 * d])), b = dag(mul(g[2 * d + 1], u[2 * d + 1]));
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) w.e[i][j] += f.e[i][j] + b.e[i][j];
  }
  return w;
}
// the FP64 kernels' star: one chain of FMAs over all products
static M<double> star_fma(const M<double>* u, const M<double>* g) {
  M<double> w{};
  auto mac = [](std::complex<double>& s, std::complex<double> x, std::complex<double> y) {
    s = {std::fma(-x.imag(), y.imag(), std::fma(x.real(), y.real(), s.real())),
         std::fma(x.imag(), y.real(), std::fma(x.real(), y.imag(), s.imag()))};
  };
  for (int d = 0; d < 8; d++)
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++)
        for (int k = 0; k < 3; k++) {
          if (d % 2 == 0) mac(w.e[i][j], u[d].e[i][k], std::conj(g[d].e[j][k]));
          else mac(w.e[i][j], std::conj(u[d].e[k][i]), std::conj(g[d].e[j][k]));
        }
  return w;
}
template <class R>
void update(M<R>& g, const M<R>& w, R omega) {
  const M<R> old = g;
  for (int s = 0; s < 3; s++) {
    const int a = s == 2 ? 1 : 0, b = s == 0 ? 1 : 2;
    const M<R> x = mul(g, w);
    const R v0 = x.e[a][a].real() + x.e[b][b].real(), v3 = x.e[b][b].imag() - x.e[a][a].imag(),
            v1 = -x.e[a][b].imag() - x.e[b][a].imag(), v2 = x.e[b][a].real() - x.e[a][b].real();
    const R n = std::sqrt(v0 * v0 + v1 * v1 + v2 * v2 + v3 * v3);
    const std::complex<R> p(v0 / n, v3 / n), q(v2 / n, v1 / n);
    for (int k = 0; k < 3; k++) {
      const std::complex<R> ra = g.e[a][k], rb = g.e[b][k];
      g.e[a][k] = p * ra + q * rb;
      g.e[b][k] = std::conj(p) * rb - std::conj(q) * ra;
    }
  }
  normalize(g);
  M<R> r = mul(g, dag(old));
  for (int k = 0; k < 3; k++) r.e[k][k] -= R(1);
  M<R> n = mul(r, r);
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      n.e[i][j] = R(i == j) + omega * r.e[i][j] + omega * (omega - 1) / 2 * n.e[i][j];
  g = mul(n, old);
  normalize(g);
}
template <class R, class S>
M<R> cast(const M<S>& a) {
  M<R> r;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      r.e[i][j] = std::complex<R>((R)a.e[i][j].real(), (R)a.e[i][j].imag());
  return r;
}

static int bad = 0;
static MFx fixed_of(const M<double>& a) {
  MFx m;
  uint32_t most = 0;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      CV v;
      v.re = fx_from_double(a.e[i][j].real(), most);
      v.im = fx_from_double(a.e[i][j].imag(), most);
      m.e[i][j] = fx_split(v);
      if (std::fabs((L)v.re / kFxOne - (L)a.e[i][j].real()) >= std::ldexp((L)1, -61)) bad++;
      if (fx_join(m.e[i][j]).re != v.re || fx_join(m.e[i][j]).im != v.im) bad++;  // exact
    }
  if (!fx_in_range(most)) bad++;
  return m;
}
static void floats(const MFx& m, CFFx (&f)[3][3]) {
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) f[i][j] = fx_float(m.e[i][j]);
}

struct Err {
  double sum = 0, most = 0;
  long n = 0;
  void add(L d) {
    sum += (double)(d * d);
    most = std::max(most, (double)std::fabs(d));
    n++;
  }
  double rms() const { return std::sqrt(sum / (double)n); }
};

int main(int argc, char** argv) {
  const long cases = argc > 1 ? std::atol(argv[1]) : 20000;
  std::mt19937_64 rng(7);
  std::normal_distribution<double> gauss;
  const double omegas[] = {1.7, 1.0, 0.0, 2.0, 1.68};
  int trial = 0;
  for (double eps : {1.0, 0.25, 1e-3, 1e-6}) {
    auto random = [&]() {
      M<L> m{};
      for (int r = 0; r < 2; r++)
        for (int k = 0; k < 3; k++)
          m.e[r][k] = std::complex<L>(eps * gauss(rng), eps * gauss(rng)) +
                      (L)(eps < 1 && r == k ? 1 : 0);
      normalize(m);
      return cast<double>(m);
    };
    Err sd, sf, ud, uf;
    for (long t = 0; t < cases; t++) {
      const double omega = omegas[trial++ % 5];
      M<double> u[8], g[8], g0 = random();
      M<L> ul[8], gl[8], gref = cast<L>(g0);
      CV w[3][3] = {};
      for (int k = 0; k < 8; k++) {
        u[k] = random();
        g[k] = random();
        ul[k] = cast<L>(u[k]);
        gl[k] = cast<L>(g[k]);
        CFFx a[3][3], b[3][3];
        floats(fixed_of(u[k]), a);
        floats(fixed_of(g[k]), b);
        for (int j = 0; j < 3; j++) {
          if (k % 2 == 0) fx_star_fwd(w, j, a, b[j]);
          else fx_star_bwd(w, j, a, b[j]);
        }
      }
      const M<L> wl = star(ul, gl);
      const M<double> wd = star_fma(u, g);
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
          sd.add(wd.e[i][j].real() - wl.e[i][j].real());
          sd.add(wd.e[i][j].imag() - wl.e[i][j].imag());
          sf.add((L)w[i][j].re / (kFxOne / 8) - wl.e[i][j].real());
          sf.add((L)w[i][j].im / (kFxOne / 8) - wl.e[i][j].imag());
        }
      update<L>(gref, wl, (L)omega);
      M<double> gd = g0;
      update<double>(gd, wd, omega);
      MFx gf = fixed_of(g0);
      FxOmega om;
      om.w4 = (fx64)std::llrint(std::ldexp(omega, 59));
      om.c4 = (fx64)std::llrint(std::ldexp(omega * (omega - 1), 58));
      fx_or_update(gf, w, om);
      for (int i = 0; i < 2; i++)
        for (int j = 0; j < 3; j++) {
          ud.add(gd.e[i][j].real() - gref.e[i][j].real());
          ud.add(gd.e[i][j].imag() - gref.e[i][j].imag());
          uf.add((L)fx_join(gf.e[i][j]).re / kFxOne - gref.e[i][j].real());
          uf.add((L)fx_join(gf.e[i][j]).im / kFxOne - gref.e[i][j].imag());
        }
    }
    std::printf("eps %-6g star: FP64 %.3g (max %.3g), fixed %.3g (max %.3g)   update: FP64 %.3g "
                "(max %.3g), fixed %.3g (max %.3g)\n",
                eps, sd.rms(), sd.most, sf.rms(), sf.most, ud.rms(), ud.most, uf.rms(), uf.most);
    if (sf.most > 3e-14 || sf.rms() > sd.rms() || uf.rms() > ud.rms()) bad++;
  }
  // 1 / sqrt over the whole range, and around powers of four
  for (long t = 0; t < 20 * cases; t++) {
    fx64 n = (fx64)(rng() >> 2) >> (rng() % 60);
    if (t % 4 == 0) n = (1ll << (rng() % 62)) + (fx64)(rng() % 5) - 2;
    if (n < 1 || n >= 1ll << 62) continue;
    int s;
    const fx64 y = fx_rsqrt(n, s);
    const L got = (L)y / kFxOne * std::ldexp((L)1, s / 2 - 2);
    if (std::fabs(got * std::sqrt((L)n / (1ll << 58)) - 1) > std::ldexp((L)1, -56)) bad++;
  }
  // what the conversion turns away
  for (double d : {2.0, -2.0, 1e300, (double)INFINITY, -(double)INFINITY, (double)NAN}) {
    uint32_t most = 0;
    fx_from_double(d, most);
    if (fx_in_range(most)) bad++;
  }
  for (double d : {0.0, -0.0, 1.0, -1.0, 1.9999999999999998, 1e-300, 5e-324, 0x1p-62, -0x1.8p-61}) {
    uint32_t most = 0;
    const L v = (L)fx_from_double(d, most) / kFxOne;
    if (!fx_in_range(most) || std::fabs(v - d) >= std::ldexp((L)1, -61)) bad++;
    if (std::fabs(d) >= 0x1p-8 && v != d) bad++;
  }
  std::printf("bad %d\n", bad);
  return bad ? 1 : 0;
}
