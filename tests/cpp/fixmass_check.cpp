// Fixed-point terms with per-body masses (csrc/fixpair.cuh) on the host, against long double: for
// partners lighter than the heaviest body by every power of two down to 2^-84, prints the largest
// error of an acceleration term and of a potential term in units of 2^-53 of its own size.
#include <cmath>
#include <cstdio>
#include <random>

#include "fixpair.cuh"

using namespace gb;
typedef long double Q;

int main() {
  std::mt19937_64 g(11);
  std::uniform_real_distribution<double> U(-1, 1);
  double worst_acc = 0.0, worst_pot = 0.0;
  for (int em : {0, 3, -299, 300})
    for (int down = 0; down <= 84; ++down)
      for (int lg = 0; lg >= -13; --lg)
        for (int t = 0; t < 200; ++t) {
          const double mass = std::ldexp(1.0 + 0.5 * (1.0 + U(g)), em - down);
          double xi[3], xj[3], u[3], nn = 0.0;
          for (double& v : u) nn += (v = U(g)) * v;
          const double sep = std::ldexp(0.9, lg) * (0.8 + 0.2 * U(g)) / std::sqrt(nn);
          for (int c = 0; c < 3; ++c) {
            xi[c] = 0.05 * U(g);
            xj[c] = xi[c] + sep * u[c];
          }
          const double eps = std::ldexp(1.0, lg - 3), eps2 = eps * eps;
          FxRow tab[kFxRows];
          for (int k = 0; k < kFxRows; ++k) tab[k] = fx_row(k, eps2, 0);
          FxBody j{};
          j.x = fx_from_double(xj[0], 0);
          j.y = fx_from_double(xj[1], 0);
          j.z = fx_from_double(xj[2], 0);
          fx_mass(j, mass, em);
          const int cls = fx_tag_class(j.tag);
          if (em - down < -300) {  // below the range: the caller's FP64 terms
            if (cls != kFxClassFp64) return 1;
            continue;
          }
          const Fx96 x = fx_from_double(xi[0], 0), y = fx_from_double(xi[1], 0),
                     z = fx_from_double(xi[2], 0);
          const float e2 = fx_eps2f(eps2, 0);
          Q d[3], r2 = eps2;
          for (int c = 0; c < 3; ++c) r2 += (d[c] = (Q)xj[c] - (Q)xi[c]) * d[c];
          FxAcc a[3] = {}, p = {};
          if (fx_term<true>(j, x, y, z, e2, tab, a) <= kFxMaxKMass) {
            Q err = 0, size = 0;
            for (int c = 0; c < 3; ++c) {
              __int128 tot = 0;
              fx_fold(tot, a[c]);
              const Q got = ldexpl((Q)tot, fx_out_exp(0) + fx_class_exp(em, cls) + 1);
              const Q ref = mass / (r2 * sqrtl(r2)) * d[c];
              err += (got - ref) * (got - ref) / mass / mass;
              size += ref * ref / mass / mass;
            }
            worst_acc = std::fmax(worst_acc, (double)sqrtl(err / size) * 0x1p53);
          }
          if (fx_term_pot<true>(j, x, y, z, e2, tab, true, p) <= kFxMaxK) {
            __int128 tot = 0;
            fx_fold(tot, p);
            const Q got = ldexpl((Q)tot, fx_out_exp_pot(0) + fx_class_exp(em, cls) + 2);
            const Q ref = mass / sqrtl(r2);
            worst_pot = std::fmax(worst_pot, (double)fabsl(got / ref - 1) * 0x1p53);
          }
        }
  FxBody zero{};
  fx_mass(zero, 0.0, 0);
  if (zero.mu_hi | zero.mu_lo | zero.tag) return 2;
  FxBody tiny{};
  fx_mass(tiny, 0x1p-1074, 0);
  if (fx_tag_class(tiny.tag) != kFxClassFp64) return 3;
  std::printf("%.4f %.4f ok\n", worst_acc, worst_pot);
  return 0;
}
