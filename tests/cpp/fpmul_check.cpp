// Products by a constant on integers (csrc/fpmul.cuh) against the host's multiplication, bit for
// bit: random significands and exponents over the whole range, significands that make ties and
// carries, and zeros.  Prints how many products were exact and how many were left to FP64.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "fpmul.cuh"

static double from_bits(uint64_t b) {
  double d;
  std::memcpy(&d, &b, 8);
  return d;
}
static uint64_t to_bits(double d) {
  uint64_t b;
  std::memcpy(&b, &d, 8);
  return b;
}

int main() {
  std::mt19937_64 g(11);
  long exact = 0, left = 0;
  auto sig = [&]() -> uint64_t {
    switch (g() % 5) {
      case 0: return 0;
      case 1: return (1ull << 52) - 1 - g() % 4;
      case 2: return (g() % (1ull << 26)) << 26;  // products of 27-bit significands: ties
      case 3: return 1ull << (g() % 52);
      default: return g() >> 12;
    }
  };
  for (long t = 0; t < 4000000; ++t) {
    const uint64_t ec = g() % 3 ? 1023 - 40 + g() % 80 : g() % 2048;
    const uint64_t ek = g() % 3 ? 1023 - 200 + g() % 400 : g() % 2048;
    const double c = from_bits((g() << 63) | (ec << 52) | sig());
    double k = from_bits((g() << 63) | (ek << 52) | sig());
    if (t % 1000 == 0) k = t % 2000 ? 0.0 : -0.0;
    const gb::MulConst m = gb::make_mul_const(c);
    bool bad = false;
    const double got = gb::mul_const(k, m, bad);
    const double want = k * c;
    const int cl = std::fpclassify(want);
    if (bad) {
      // left out only where it has to be, or where the exponents are one short of the limit
      const bool c_normal = std::fpclassify(c) == FP_NORMAL, k_normal = std::fpclassify(k) == FP_NORMAL;
      if (c_normal && k_normal && cl == FP_NORMAL && std::ilogb(want) > -1021 &&
          std::ilogb(want) < 1022)
        return 1;
      if (k == 0.0 && c_normal) return 2;
      ++left;
    } else {
      // a constant that is not normal leaves every product but those of a zero
      if (std::fpclassify(c) != FP_NORMAL && !(k == 0.0)) return 3;
      if (std::fpclassify(c) == FP_NORMAL && to_bits(got) != to_bits(want)) {
        std::printf("%a * %a: %a, want %a\n", k, c, got, want);
        return 4;
      }
      ++exact;
    }
  }
  std::printf("exact %ld left %ld\nok\n", exact, left);
  return 0;
}
