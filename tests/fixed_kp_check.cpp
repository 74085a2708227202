// The Kennedy-Pendleton draw of gfx_fixed_kp.cuh on the CPU against long double, with the FP64
// form (heatbath_su2_kp) beside it.  Exits non-zero when
//   * log, sine and cosine, or square root are off by more than 2^-55, 2^-58, 2^-57 / sqrt(x);
//   * a trial is accepted where long double rejects it, or the other way round;
//   * the drawn element's error (root mean square) is above FP64's for |w| of 0.2 and more, the
//     sizes that the projections of a staple have (smaller ones lose digits in the sum that
//     both are given).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "gfx_fixed_kp.cuh"

using namespace gfx;
typedef long double L;

template <class R>
bool draw(const R* w, R beta, R g, const float* u, R* al) {
  const R k = std::sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2] + w[3] * w[3]);
  al[0] = 1;
  al[1] = al[2] = al[3] = 0;
  if (!(k > 0)) return false;
  const R rk = 1 / k;
  const R y = (-std::log(R(1) - (R)u[0]) + R(0.5) * g * g) / (beta * k);
  if (!((R)u[1] * (R)u[1] <= 1 - R(0.5) * y)) return false;
  const R a0 = 1 - y, c = 2 * (R)u[2] - 1;
  const R norm = std::sqrt(std::max(R(0), 1 - a0 * a0)), st = std::sqrt(std::max(R(0), 1 - c * c));
  const R phi = 2 * std::acos(R(-1)) * (R)u[3];
  const R a1 = norm * st * std::cos(phi), a2 = norm * st * std::sin(phi), a3 = norm * c;
  R v[4];
  for (int i = 0; i < 4; i++) v[i] = w[i] * rk;
  al[0] = a0 * v[0] - a1 * v[1] - a2 * v[2] - a3 * v[3];
  al[1] = a0 * v[1] + a1 * v[0] - a2 * v[3] + a3 * v[2];
  al[2] = a0 * v[2] + a2 * v[0] - a3 * v[1] + a1 * v[3];
  al[3] = a0 * v[3] + a3 * v[0] - a1 * v[2] + a2 * v[1];
  return true;
}

int main(int argc, char** argv) {
  const long cases = argc > 1 ? std::atol(argv[1]) : 100000;
  std::mt19937_64 rng(5);
  std::normal_distribution<double> normal;
  auto uniform = [&]() { return ((float)(uint32_t)rng() + 1.0f) * 2.3283064365386963e-10f; };
  int bad = 0;
  double wl = 0, ws = 0, wq = 0;
  for (long t = 0; t < cases; t++) {
    const fx64 a = (fx64)((rng() >> 3) >> (rng() % 60)), u = (fx64)(rng() >> 3);
    const L av = (L)a / kFxOne, x = 2 * std::acos((L)-1) * ((L)u / kFxOne);
    if (a > 0) {
      wl = std::max(wl, (double)std::fabs((L)fx_neg_log_16th(a) / kFxOne + std::log(av) / 16));
      wq = std::max(wq, (double)(std::fabs((L)fx_sqrt(a) / kFxOne - std::sqrt(av)) * std::sqrt(av)));
    }
    fx64 s, c;
    fx_sincos_turns(u, s, c);
    ws = std::max({ws, (double)std::fabs((L)s / kFxOne - std::sin(x)),
                   (double)std::fabs((L)c / kFxOne - std::cos(x))});
  }
  std::printf("log/16 %.3g  sincos %.3g  sqrt(x) sqrt %.3g\n", wl, ws, wq);
  if (wl > 0x1p-55 || ws > 0x1p-58 || wq > 0x1p-57) bad++;
  // the ends of the uniform numbers' range
  fx64 s, c;
  for (float f : {1.0f, 0.5f, 0.25f, 2.3283064365386963e-10f, 0.99999994f})
    if ((L)fx_from_float(f, 0) / kFxOne != (L)f) bad++;
  fx_sincos_turns(kFxOne, s, c);
  if (s != 0 || c != kFxOne) bad++;
  for (double size : {4.0, 1.0, 0.1, 0.01}) {
    double ed = 0, ef = 0;
    long n = 0, flips = 0, taken = 0;
    for (long t = 0; t < cases; t++) {
      float u[4] = {uniform(), uniform(), uniform(), uniform()};
      if (t % 1000 < 4) u[t % 1000] = 1.0f;
      const float g = (float)normal(rng);
      const double beta = 1.25 + 0.25 * (t % 5);
      fx64 v[4];
      double wd[4];
      L w[4];
      for (int i = 0; i < 4; i++) {
        v[i] = std::llrint(std::ldexp(std::max(-15.0, std::min(15.0, size * normal(rng))), 58));
        wd[i] = (double)((L)v[i] / (kFxOne / 8));
        w[i] = wd[i];
        v[i] = std::llrint(std::ldexp(wd[i], 58));
      }
      if (t % 1000 == 9) v[0] = v[1] = v[2] = v[3] = 0, w[0] = w[1] = w[2] = w[3] = 0,
                         wd[0] = wd[1] = wd[2] = wd[3] = 0;
      L al[4];
      double ad[4];
      const bool in_l = draw<L>(w, beta, g, u, al), in_d = draw<double>(wd, beta, g, u, ad);
      CFx p, q;
      fx_kp(v[0], v[1], v[2], v[3], (fx64)std::llrint(std::ldexp(1.0 / beta, 61)), g, u[0], u[1],
            u[2], u[3], p, q);
      const L f[4] = {(L)fx_join(p.re) / kFxOne, (L)fx_join(q.im) / kFxOne,
                      (L)fx_join(q.re) / kFxOne, (L)fx_join(p.im) / kFxOne};
      const bool in_f = !(f[0] == 1 && f[1] == 0 && f[2] == 0 && f[3] == 0);
      if (in_f != in_l) flips++;
      if (in_f != in_l || in_d != in_l) continue;
      taken += in_l;
      for (int i = 0; i < 4; i++) {
        ed += (double)((ad[i] - al[i]) * (ad[i] - al[i]));
        ef += (double)((f[i] - al[i]) * (f[i] - al[i]));
        n++;
      }
    }
    ed = std::sqrt(ed / (double)n);
    ef = std::sqrt(ef / (double)n);
    std::printf("|w| ~ %-5g taken %ld of %ld, flips %ld, error FP64 %.3g fixed %.3g\n", 2 * size,
                taken, cases, flips, ed, ef);
    if (flips || (size >= 0.1 && ef > ed)) bad++;
  }
  std::printf("bad %d\n", bad);
  return bad ? 1 : 0;
}
