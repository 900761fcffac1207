// Small components of the fixed-point acceleration terms (csrc/fixpair.cuh) on the host, against long
// double: separations with one component smaller than the distance by every power of two down to
// 2^-40, near the origin (coordinates off the grid) and away from it. Prints the largest error of a
// component above 2^-kFxThin of the bound of the term's size, in units of 2^-53 of itself, and how
// many were above and below; a term above its bound, or a bound more than twice it without
// softening, fails; the same with two words for components above 2^kFxEnough weights. Then the 160-bit total.
#include <cmath>
#include <cstdio>
#include <random>

#include "fixpair.cuh"

using namespace gb;
typedef long double Q;

int main() {
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> U(-1, 1);
  double worst = 0.0, narrow = 0.0;
  int above = 0, below = 0;
  for (int ratio = 0; ratio <= 40; ++ratio)
    for (int lg = 0; lg >= -12; --lg)
      for (double off : {0.0, 0.25, 1.0e6})
        for (int axis = 0; axis < 3; ++axis)
          for (int soft = 0; soft < 2; ++soft)
            for (int t = 0; t < 12; ++t) {
              const double sep = std::ldexp(0.4, lg);
              double xi[3], xj[3];
              for (int c = 0; c < 3; ++c) {
                const double d = sep * (0.5 + 0.2 * U(g)) * (g() & 1 ? 1 : -1);
                xi[c] = c == axis ? off + std::ldexp(sep, -ratio) * U(g) : off + 0.1 * U(g);
                xj[c] = xi[c] + (c == axis ? std::ldexp(d, -ratio) : d);
              }
              const double eps = soft ? sep : 0.0, eps2 = eps * eps;
              FxRow tab[kFxRows];
              for (int k = 0; k < kFxRows; ++k) tab[k] = fx_row(k, eps2, 0);
              FxBody j{};
              j.x = fx_from_double(xj[0], 0);
              j.y = fx_from_double(xj[1], 0);
              j.z = fx_from_double(xj[2], 0);
              const Fx96 x = fx_from_double(xi[0], 0), y = fx_from_double(xi[1], 0),
                         z = fx_from_double(xi[2], 0);
              const float e2 = fx_eps2f(eps2, 0);
              Q d[3], r2 = eps2;
              for (int c = 0; c < 3; ++c) r2 += (d[c] = (Q)xj[c] - (Q)xi[c]) * d[c];
              FxAcc a[3] = {};
              FxSize zw = {}, zn = {};
              if (fx_term<false, true>(j, x, y, z, e2, tab, a, zw) > kFxMaxK) continue;
              FxAcc an[3] = {};
              fx_term<false, false>(j, x, y, z, e2, tab, an, zn);
              const Q size = ldexpl((Q)zw.m, fx_out_exp(0) + 30);
              const Q s = 1 / (r2 * sqrtl(r2));
              const Q dist = sqrtl(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
              if (s * dist > size * 1.0001L) return 1;
              if (!soft && size > 2 * s * dist) return 2;
              for (int c = 0; c < 3; ++c) {
                __int128 tot = 0;
                fx_fold(tot, a[c]);
                if (d[c] == 0) {
                  if (tot != 0) return 3;
                  continue;
                }
                if (zn.c[c] >= ldexpf((float)zn.p, kFxEnough - 31)) {
                  if (fabsl(ldexpl((Q)zn.c[c], fx_out_exp(0) + 31) / (s * fabsl(d[c])) - 1) > 0.01) return 6;
                  __int128 t2 = 0;
                  fx_fold(t2, an[c]);
                  const Q got = ldexpl((Q)t2, fx_out_exp(0));
                  narrow = std::fmax(narrow, (double)fabsl(got / (s * d[c]) - 1) * 0x1p53);
                }
                if (s * fabsl(d[c]) < ldexpl(size, -kFxThin)) {
                  ++below;
                  continue;
                }
                ++above;
                const Q got = ldexpl((Q)tot, fx_out_exp(0));
                worst = std::fmax(worst, (double)fabsl(got / (s * d[c]) - 1) * 0x1p53);
              }
            }
  std::printf("%.4f %d %d %.4f", worst, above, below, narrow);
  // the 160-bit total: sums and differences beyond 128 bits
  for (int t = 0; t < 100000; ++t) {
    FxTot tot{};
    long double ref = 0;
    const int n = 1 << (g() % 10);
    for (int v = 0; v < n; ++v) {
      FxAcc a{(long long)g() >> 4, g() >> 2, g() >> 2};
      if (t & 1) a.h = a.h < 0 ? -a.h : a.h;
      ref += ldexpl((long double)a.h, 64) + ldexpl((long double)a.m, 32) + (long double)a.l;
      fx_fold(tot, a);
    }
    const double got = fx_to_double(tot, -100);
    if (std::fabs(got - (double)ldexpl(ref, -100)) > 0x1p-52 * std::fabs(got) + n * 0x1p-40) return 4;
  }
  std::printf(" ok\n");
  return 0;
}
