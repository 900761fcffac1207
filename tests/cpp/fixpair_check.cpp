// Fixed-point pair terms (csrc/fixpair.cuh) on the host, against the same terms in long double:
// prints the largest error of a term in units of 2^-53 of its size over seeded pairs of every
// separation inside the window, then checks the conversions from and to double.
#include <cmath>
#include <cstdio>
#include <random>

#include "fixpair.cuh"

using namespace gb;
typedef long double Q;

static double worst_term(int ex, int lg, double offset, bool soft) {
  std::mt19937_64 g(17 * lg + ex + 1000);
  std::uniform_real_distribution<double> U(-1, 1);
  const double M = std::ldexp(1.0, ex) * 0.999;
  double worst = 0.0;
  for (int t = 0; t < 500; ++t) {
    double u[3], xi[3], xj[3], nn = 0.0;
    for (double& v : u) nn += (v = U(g)) * v;
    const double sep = std::ldexp(M, lg) * (0.7 + 0.3 * U(g)) / std::sqrt(nn);
    bool fits = true;
    for (int c = 0; c < 3; ++c) {
      xi[c] = offset + 0.4 * M * U(g);
      xj[c] = xi[c] + sep * u[c];
      fits = fits && std::fabs(xj[c] - xi[c]) < M;
    }
    if (!fits) continue;
    const double eps = soft ? std::ldexp(M, lg - 2) : 0.0, eps2 = eps * eps;
    FxRow tab[kFxRows];
    for (int k = 0; k < kFxRows; ++k) tab[k] = fx_row(k, eps2, ex);
    FxBody j{};
    j.x = fx_from_double(xj[0], ex);
    j.y = fx_from_double(xj[1], ex);
    j.z = fx_from_double(xj[2], ex);
    FxAcc a[3] = {};
    const int k = fx_term<false>(j, fx_from_double(xi[0], ex), fx_from_double(xi[1], ex),
                                fx_from_double(xi[2], ex), fx_eps2f(eps2, ex), tab, a);
    if (k > kFxMaxK) {
      for (auto& s : a)
        if (s.h | (long long)s.l | s.m) return 1e9;  // outside the window: nothing is added
      continue;
    }
    Q d[3], r2 = eps2, err = 0, size = 0;
    for (int c = 0; c < 3; ++c) r2 += (d[c] = (Q)xj[c] - (Q)xi[c]) * d[c];
    const Q s = 1 / (r2 * sqrtl(r2));
    for (int c = 0; c < 3; ++c) {
      __int128 tot = 0;
      fx_fold(tot, a[c]);
      const Q got = ldexpl((Q)tot, fx_out_exp(ex));
      err += (got - s * d[c]) * (got - s * d[c]);
      size += s * d[c] * s * d[c];
    }
    worst = std::fmax(worst, (double)sqrtl(err / size) * 0x1p53);
  }
  return worst;
}

int main() {
  double worst = 0.0;
  for (int ex : {0, 7, -30, 200})
    for (int lg = 0; lg >= -13; --lg)
      for (double off : {0.0, 1.0e6})
        for (bool soft : {false, true}) {
          const double o = std::ldexp(off, ex);
          worst = std::fmax(worst, worst_term(ex, lg, o, soft));
        }
  std::printf("worst %.4f\n", worst);
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> U(-0.5, 0.5);
  for (int t = 0; t < 100000; ++t) {
    __int128 v = (((__int128)(long long)g() << 62) ^ (__int128)(unsigned long long)g()) >> (g() % 120);
    const int sc = (int)(g() % 400) - 200;
    if (fx_to_double(v, sc) != std::ldexp((double)v, sc)) return 1;
  }
  for (int t = 0; t < 100000; ++t) {
    const double v = U(g) * std::ldexp(1.0, -(int)(g() % 80));
    const Fx96 f = fx_from_double(v, 0);
    const __int128 x = ((__int128)(int32_t)f.w2 << 64) | fx_pair(f.w0, f.w1);
    const long double back = ldexpl((long double)(long long)(x >> 32), -62) +
                             ldexpl((long double)(uint32_t)x, -94);
    if (fabsl(back - v) > ldexpl(1.0L, -62 - 11)) return 2;
    if (std::fabs(v) > 0x1p-41 && back != v) return 3;
  }
  std::printf("ok\n");
  return 0;
}
