// fpmul.cuh -- IEEE double products by a constant on the integer pipes.
//
// The element-wise Runge-Kutta sums need an IEEE product and a separate IEEE
// addition per coefficient (the reference's operation order, bit for bit), and
// GB300's FP64 pipe takes 76 cycles of a sub-partition for either.  A product by
// a constant is four 32 x 32 -> 64 bit multiplications, a normalisation by 0 or
// 1 bit and a rounding, about 35 cycles of the integer pipes, which run beside
// the FP64 additions.
//
// k c for a normal constant c: the significand of c is kept shifted to 64 bits,
// so that the product's top word pair holds 52 or 53 significand bits.  Exact
// for every k whose product is normal, and for k = +-0; other k (subnormal,
// infinite, NaN, or a product beyond the normal range) are reported and left to
// the FP64 unit.
#pragma once

#include "fixpair.cuh"

namespace gb {

struct MulConst {
  uint32_t ch, cl;  // significand 2^11, bit 63 set
  uint32_t ec;      // (biased exponent of c - 1023 - 1) << 20
  uint32_t sign;
  uint32_t lo;      // least high word (no sign) of an exact k
  uint32_t span;    // above it: number of such words - 1; 0 with lo = ~0: none
};

inline MulConst make_mul_const(double c) {
  uint64_t bits;
  std::memcpy(&bits, &c, 8);
  const int e = (int)((bits >> 52) & 0x7ff);
  MulConst m{};
  m.lo = 0xffffffffu;
  if (e == 0 || e == 0x7ff) return m;
  const uint64_t sig = ((bits & 0xfffffffffffffull) | (1ull << 52)) << 11;
  m.ch = (uint32_t)(sig >> 32);
  m.cl = (uint32_t)sig;
  m.ec = (uint32_t)(e - 1024) << 20;
  m.sign = (uint32_t)(bits >> 32) & 0x80000000u;
  // 1 <= ek + e - 1023 <= 2045: the product's exponent is that or one more
  const int lo = e >= 1023 ? 1 : 1024 - e, hi = e <= 1022 ? 2046 : 3068 - e;
  if (lo > hi) return m;
  m.lo = (uint32_t)lo << 20;
  m.span = ((uint32_t)(hi + 1) << 20) - 1 - m.lo;
  return m;
}

// k c; sets `bad` where the result is not exact.
GB_HD double mul_const(double k, const MulConst& c, bool& bad) {
#ifdef __CUDA_ARCH__
  const uint32_t kh = (uint32_t)__double2hiint(k), kl = (uint32_t)__double2loint(k);
#else
  uint64_t kb;
  std::memcpy(&kb, &k, 8);
  const uint32_t kh = (uint32_t)(kb >> 32), kl = (uint32_t)kb;
#endif
  const uint32_t ka = kh & 0x7fffffffu;
  const bool zero = (ka | kl) == 0;
  bad |= ka - c.lo > c.span && !zero;
  const uint32_t mh = (kh & 0xfffffu) | 0x100000u;
  // 117-bit product in words p3 .. p0
  const uint64_t t0 = fx_mul(kl, c.cl);
  const uint64_t t1 = fx_mad(kl, c.ch, fx_pair(fx_hi(t0), 0));
  const uint64_t t2 = fx_mad(mh, c.cl, fx_pair(fx_lo(t1), 0));
  const uint64_t t3 = fx_mad(mh, c.ch, fx_pair(fx_hi(t1), 0)) + fx_hi(t2);
  const uint32_t p0 = fx_lo(t0), p1 = fx_lo(t2), p2 = fx_lo(t3), p3 = fx_hi(t3);
  // 53 significand bits in (sh, sl), the rest below bit 63 of (r1, r0)
  const int up = (int)(~p3 >> 20) & 1;  // bit 52 of the top pair is clear
  const uint32_t sh = fx_shl(p2, p3, up), sl = fx_shl(p1, p2, up), r1 = fx_shl(p0, p1, up);
  const uint32_t rest = r1 | ((p0 << up) != 0 ? 1u : 0u);
  // nearest even: carry of rest + 2^31 - 1 + (last bit)
  const uint32_t half = 0x7fffffffu + (sl & 1u);
  uint32_t hw = (ka & 0x7ff00000u) + c.ec + (p3 & 0x100000u) + sh, lw;
#ifdef __CUDA_ARCH__
  asm("{.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, 0;}"
      : "=r"(lw), "=r"(hw)
      : "r"(rest), "r"(half), "r"(sl), "r"(hw));
#else
  const uint64_t carry = ((uint64_t)rest + half) >> 32;
  const uint64_t w = fx_pair(sl, hw) + carry;
  lw = (uint32_t)w;
  hw = (uint32_t)(w >> 32);
#endif
  const uint32_t sign = (kh & 0x80000000u) ^ c.sign;
  hw = zero ? sign : hw | sign;
  lw = zero ? 0u : lw;
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hw, (int)lw);
#else
  const uint64_t rb = fx_pair(lw, hw);
  double r;
  std::memcpy(&r, &rb, 8);
  return r;
#endif
}

}  // namespace gb
