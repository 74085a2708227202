// The fixed-point update of gfx_fixed.cuh on the CPU where norms are small, against long double
// and FP64 as in fixed_check.cpp: exits non-zero where the new g's error (root mean square over
// a family) or its distance from unitary (largest) is above FP64's, or an SU(2) element's
// |p|^2 + |q|^2 is off 1 by more than 2^-52.
//   stars of a small size, given exactly
//   stars of eight products that nearly cancel: twice FP64's error, whose roundings shrink with
//     the partial sums, where those of the FP32 cross terms stay at 2^-54 of a product of 1
//   a first projection that nearly vanishes, g star = diag(a, -a, b) + noise
//   S = diag(-1, -1, 1), where 1 + M = diag(r, r, 1) with r = 1 - 4 omega + 2 omega^2
#define main generic_main
#include "fixed_check.cpp"
#undef main

static M<double> fp64_of(const MFx& m) {
  M<double> r;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      r.e[i][j] = {fx_to_double(fx_join(m.e[i][j]).re), fx_to_double(fx_join(m.e[i][j]).im)};
  return r;
}
// |g g^+ - 1| of rows 0, 1
template <class R>
static double off_unitary(const M<R>& g) {
  L most = 0;
  for (int i = 0; i < 2; i++)
    for (int j = 0; j < 2; j++) {
      std::complex<L> s = i == j ? -1 : 0;
      for (int k = 0; k < 3; k++)
        s += std::complex<L>(g.e[i][k]) * std::conj(std::complex<L>(g.e[j][k]));
      most = std::max(most, std::abs(s));
    }
  return (double)most;
}

struct Family {
  Err fp64, fixed;
  double un64 = 0, unfx = 0;
  // one update of g0 with the star w / 8 on the grid
  void add(const M<double>& g0, const CV (&w8)[3][3], double omega) {
    M<L> wl;
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++)
        wl.e[i][j] = {(L)w8[i][j].re / (kFxOne / 8), (L)w8[i][j].im / (kFxOne / 8)};
    add(g0, wl, cast<double>(wl), w8, omega);
  }
  void add(const M<double>& g0, const M<L>& wl, const M<double>& wd, const CV (&w8)[3][3],
           double omega) {
    M<L> ref = cast<L>(g0);
    update<L>(ref, wl, (L)omega);
    M<double> gd = g0;
    update<double>(gd, wd, omega);
    FxOmega om;
    om.w4 = (fx64)std::llrint(std::ldexp(omega, 59));
    om.c4 = (fx64)std::llrint(std::ldexp(omega * (omega - 1), 58));
    CV w[3][3];
    std::copy(&w8[0][0], &w8[0][0] + 9, &w[0][0]);
    MFx gf = fixed_of(g0);
    fx_or_update(gf, w, om);
    const M<double> gx = fp64_of(gf);
    for (int i = 0; i < 2; i++)
      for (int j = 0; j < 3; j++) {
        fp64.add(gd.e[i][j].real() - ref.e[i][j].real());
        fp64.add(gd.e[i][j].imag() - ref.e[i][j].imag());
        fixed.add(gx.e[i][j].real() - ref.e[i][j].real());
        fixed.add(gx.e[i][j].imag() - ref.e[i][j].imag());
      }
    un64 = std::max(un64, off_unitary(gd));
    unfx = std::max(unfx, off_unitary(gx));
  }
  void report(const char* name, double at, double times = 1.0) {
    std::printf("%s %-8g rms: FP64 %.3g, fixed %.3g   unitary: FP64 %.3g, fixed %.3g\n", name, at,
                fp64.rms(), fixed.rms(), un64, unfx);
    if (!(fixed.rms() <= times * fp64.rms()) || !(unfx <= un64)) bad++;
  }
};

int main(int argc, char** argv) {
  const long cases = argc > 1 ? std::atol(argv[1]) : 2000;
  std::mt19937_64 rng(11);
  std::normal_distribution<double> gauss;
  auto random = [&](double eps) {
    M<L> m{};
    for (int r = 0; r < 2; r++)
      for (int k = 0; k < 3; k++)
        m.e[r][k] = std::complex<L>(eps * gauss(rng), eps * gauss(rng)) + (L)(eps < 1 && r == k);
    normalize(m);
    return cast<double>(m);
  };
  auto grid = [](double x) { return (fx64)std::llrint(std::ldexp(x, 58)); };
  // the star g^+ X on the grid, from a long double X
  auto star_of = [&](const M<double>& g, const M<L>& X, CV (&w)[3][3]) {
    const M<L> s = mul(dag(cast<L>(g)), X);
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) {
        w[i][j].re = (fx64)std::llrint(std::ldexp(s.e[i][j].real(), 58));
        w[i][j].im = (fx64)std::llrint(std::ldexp(s.e[i][j].imag(), 58));
      }
  };
  for (double size : {1.0, 1e-1, 1e-2, 1e-3, 1e-6}) {
    Family f;
    for (long t = 0; t < cases; t++) {
      CV w[3][3];
      for (auto& row : w)
        for (CV& z : row) {
          z.re = grid(size * std::tanh(gauss(rng)));
          z.im = grid(size * std::tanh(gauss(rng)));
        }
      f.add(random(1.0), w, 1.7);
    }
    f.report("exact star of size", size);
  }
  for (double size : {1e-1, 1e-2, 1e-3, 1e-6}) {
    Family f;
    for (long t = 0; t < cases; t++) {
      // terms z_k A n_k with phases z_k that sum to zero and n_k close to 1
      M<double> u[8], g[8];
      M<L> ul[8], gl[8];
      const M<L> a = cast<L>(random(1.0));
      CV w[3][3] = {};
      for (int k = 0; k < 8; k++) {
        const M<L> v = cast<L>(random(1.0)), n = cast<L>(random(size));
        const L x = 2 * std::acos((L)-1) * (k < 6 ? (L)(k % 3) / 3 : (L)(k - 6) / 2);
        M<L> b = mul(mul(a, n), v);  // u g^+ = z A n forward, (g u)^+ = z A n backward
        for (auto& row : b.e)
          for (auto& e : row) e *= std::complex<L>(std::cos(x), std::sin(x));
        u[k] = cast<double>(k % 2 ? dag(b) : b);
        g[k] = cast<double>(v);
        ul[k] = cast<L>(u[k]);
        gl[k] = cast<L>(g[k]);
        CFFx fa[3][3], fb[3][3];
        floats(fixed_of(u[k]), fa);
        floats(fixed_of(g[k]), fb);
        for (int j = 0; j < 3; j++) {
          if (k % 2 == 0) fx_star_fwd(w, j, fa, fb[j]);
          else fx_star_bwd(w, j, fa, fb[j]);
        }
      }
      f.add(random(1.0), star(ul, gl), star_fma(u, g), w, 1.7);
    }
    f.report("cancelling star of size", size, 2.0);
  }
  for (int e = 0; e <= 40; e += 4) {
    Family f;
    for (long t = 0; t < cases; t++) {
      const M<double> g = random(1.0);
      M<L> X{};
      for (auto& row : X.e)
        for (auto& z : row) z = std::ldexp((L)1, -e) * std::complex<L>(gauss(rng), gauss(rng)) / (L)4;
      X.e[0][0] += 3;
      X.e[1][1] -= 3;
      X.e[2][2] += 2;
      CV w[3][3];
      star_of(g, X, w);
      f.add(g, w, 1.7);
    }
    f.report("vanishing projection, 2^-", e);
  }
  for (double omega : {1.7, 1.707, 1.7071}) {
    Family f;
    for (long t = 0; t < cases; t++) {
      const M<double> g = random(1.0);
      M<L> X{};
      X.e[0][0] = X.e[1][1] = -5 - (L)std::tanh(gauss(rng));
      X.e[2][2] = 6;
      CV w[3][3];
      star_of(g, X, w);
      f.add(g, w, omega);
    }
    f.report("S = diag(-1, -1, 1) at omega", omega);
  }
  // the SU(2) element of a projection of any size
  for (long t = 0; t < 100 * cases; t++) {
    const int down = (int)(rng() % 62);
    CV x[4];
    for (CV& z : x) {
      z.re = (fx64)((int64_t)rng() >> 2) >> down;
      z.im = (fx64)((int64_t)rng() >> 2) >> down;
    }
    CFx p, q;
    fx_su2(x[0], x[1], x[2], x[3], p, q);
    L n = 0;
    for (fx64 v : {fx_join(p).re, fx_join(p).im, fx_join(q).re, fx_join(q).im})
      n += (L)v / kFxOne * ((L)v / kFxOne);
    if (std::fabs(n - 1) > std::ldexp((L)1, -52)) bad++;
  }
  // rows that vanish are reported
  CV v[2][3] = {};
  v[1][2].re = kFxOne / 2;
  MFx g;
  if (fx_normalize(g, v)) bad++;
  std::printf("bad %d\n", bad);
  return bad ? 1 : 0;
}
