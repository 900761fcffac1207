// fixpair.cuh -- softened pair terms of FP64 accuracy on the integer pipes.
//
// GB300 retires two FP64 operations per SM and clock, 16 times fewer than
// 32 x 32 -> 64 bit integer multiply-adds (IMAD.WIDE: measured 4 cycles per
// warp and sub-partition against 64 for a DFMA), and a pair term in FP64 takes
// 18 of them even with a refined reciprocal square root.  Here the whole term
// is fixed point: positions are 96-bit integers on a grid common to the bodies
// a CTA reads, so the difference of two is exact; r^2, its reciprocal square
// root and r^-3 keep 57 bits or more; and the sums are integers, exact and
// independent of the order.  33 IMAD.WIDE per term.
//
// Scales.  The grid is U = 2^(Ex - 94) with |x_j - x_i| < 2^Ex in every
// component and eps < 2^(Ex - 1); coordinates are taken modulo 2^96 U, so only
// the differences have to fit and a system far from the origin loses nothing.
// A pair is normalised by 2^k, k >= 0 such that R = (|d|^2 + eps^2) 4^k in
// units of (2^64 U)^2 lies in [2^60, 2^62); its contribution carries the
// weight 4^k.  Pairs closer than about 2^-12 2^Ex (k > kFxMaxK) do not fit the
// sums' window: they get weight 0 here and are added by the caller in FP64.
//
// Error: d is exact where a coordinate's last bit is a multiple of U (every
// coordinate above 2^-41 2^Ex); R and the Newton residual hold 2^-58.  A term is
// within 2^-55 of its size (0.04 2^-53 rms; a term in FP64: 1.3 2^-53 rms, up to
// 5 2^-53).  Its components are products of two words' precision, 2^-57 of the
// term and not of the component; the sizes of a sum's terms and of their
// components say where that is not enough (kFxEnough, kFxThin), and those sums
// are taken with three words or in FP64, so that every component is as good as
// its FP64 sum.
//
// Measured at N = 16384 (right-hand side): 1.65 ms against 22.3 ms for the FP64
// loop in the reference's operation order and 12 ms with the refined
// reciprocal square root (1.60 ms with two words and no look at the components,
// 1.92 ms with three words everywhere).
#pragma once

#include <cstdint>
#include <cstring>

namespace gb {

#ifdef __CUDACC__
#define GB_HD __host__ __device__ __forceinline__
#else
#define GB_HD inline
#endif

constexpr int kFxMaxK = 13;       // largest normalisation inside the window
constexpr int kFxRows = kFxMaxK + 2;  // table rows (the last: weight 0)
// with per-body masses, whose weight is 4^k times up to 8
constexpr int kFxMaxKMass = 11;
template <bool MASS>
constexpr int fx_max_k() {
  return MASS ? kFxMaxKMass : kFxMaxK;
}

struct Fx96 {  // two's complement, w0 least significant
  uint32_t w0, w1, w2;
};

// row k of the softening table: eps^2 at normalisation k, the weight 4^k, 8^k 2^-62
struct alignas(16) FxRow {
  uint32_t e_lo, e_hi;
  uint32_t p;
  float pf;
};

struct FxAcc {  // sum of the terms, weight 2^64, 1 and 2^32
  long long h;
  unsigned long long l;
  unsigned long long m;
};

struct FxTot {  // sum of FxAcc, 160 bits two's complement
  unsigned __int128 l;
  int32_t h;
};

// 32 x 32 -> 64 bit products and words, each one instruction.  In PTX: from C
// the compiler turns products of a 64-bit value's high word into full 64-bit
// multiplications (a term took 168 instructions so, against 109).
GB_HD uint32_t fx_lo(uint64_t v) { return (uint32_t)v; }
GB_HD uint32_t fx_hi(uint64_t v) {
#ifdef __CUDA_ARCH__
  uint32_t hi;
  asm("{.reg .b32 lo; mov.b64 {lo, %0}, %1;}" : "=r"(hi) : "l"(v));
  return hi;
#else
  return (uint32_t)(v >> 32);
#endif
}
GB_HD uint64_t fx_pair(uint32_t lo, uint32_t hi) {
#ifdef __CUDA_ARCH__
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  return v;
#else
  return ((uint64_t)hi << 32) | lo;
#endif
}
GB_HD uint64_t fx_mul(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  uint64_t v;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(v) : "r"(a), "r"(b));
  return v;
#else
  return (uint64_t)a * b;
#endif
}
GB_HD uint64_t fx_mad(uint32_t a, uint32_t b, uint64_t c) {
#ifdef __CUDA_ARCH__
  uint64_t v;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(v) : "r"(a), "r"(b), "l"(c));
  return v;
#else
  return (uint64_t)a * b + c;
#endif
}
GB_HD int64_t fx_muls(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  int64_t v;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(v) : "r"(a), "r"(b));
  return v;
#else
  return (int64_t)a * b;
#endif
}
GB_HD int64_t fx_mads(int32_t a, int32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  int64_t v;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(v) : "r"(a), "r"(b), "l"(c));
  return v;
#else
  return (int64_t)a * b + c;
#endif
}

GB_HD uint32_t fx_shl(uint32_t lo, uint32_t hi, int k) {  // high word of (hi:lo) << k, k < 32
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, k);
#else
  return k ? (hi << k) | (lo >> (32 - k)) : hi;
#endif
}

GB_HD uint32_t fx_float_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
#endif
}

GB_HD float fx_abs(float v) {
#ifdef __CUDA_ARCH__
  return fabsf(v);
#else
  return __builtin_fabsf(v);
#endif
}

GB_HD float fx_float_of(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}

// v in units of U = 2^(ex - 94) modulo 2^96, truncated (exact when v is a
// multiple of U).
GB_HD Fx96 fx_from_double(double v, int ex) {
#ifdef __CUDA_ARCH__
  const uint64_t bits = (uint64_t)__double_as_longlong(v);
#else
  uint64_t bits;
  memcpy(&bits, &v, 8);
#endif
  const int e = (int)((bits >> 52) & 0x7ff);
  uint64_t m = bits & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  const int sh = (e ? e : 1) - 1075 - ex + 94;
  uint64_t lo = 0, hi = 0;
  if (sh >= 64) {
    hi = sh < 96 ? m << (sh - 64) : 0;
  } else if (sh > 0) {
    lo = m << sh;
    hi = m >> (64 - sh);
  } else if (sh > -64) {
    lo = m >> -sh;
  }
  if (bits >> 63) {
    lo = ~lo + 1;
    hi = ~hi + (lo == 0);
  }
  return Fx96{(uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi};
}

GB_HD Fx96 fx_sub(const Fx96& a, const Fx96& b) {
  Fx96 r;
#ifdef __CUDA_ARCH__
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=r"(r.w0), "=r"(r.w1), "=r"(r.w2)
      : "r"(a.w0), "r"(a.w1), "r"(a.w2), "r"(b.w0), "r"(b.w1), "r"(b.w2));
#else
  const uint64_t al = fx_pair(a.w0, a.w1), bl = fx_pair(b.w0, b.w1), d = al - bl;
  r.w0 = fx_lo(d);
  r.w1 = fx_hi(d);
  r.w2 = a.w2 - b.w2 - (al < bl);
#endif
  return r;
}

// Normalisation of a difference from the high words, clamped to max_k + 1:
// R 4^k in [2^60 (1 - 2^-8), 2^62 (1 - 2^-9)], so that every component's high
// word stays below 2^31 (the high words, truncated, know r to 2^-13 at k = 13).
GB_HD int fx_norm(const Fx96& dx, const Fx96& dy, const Fx96& dz, float eps2f, int max_k) {
  const float fx = (float)(int32_t)dx.w2, fy = (float)(int32_t)dy.w2, fz = (float)(int32_t)dz.w2;
#ifdef __CUDA_ARCH__
  const float f = __fmaf_rn(fx, fx, __fmaf_rn(fy, fy, __fmaf_rn(fz, fz, eps2f)));
#else
  const float f = fx * fx + fy * fy + fz * fz + eps2f;
#endif
  const int k = (int)((0x5e7fffffu - 0x8000u - fx_float_bits(f)) >> 24);
  return k < max_k + 1 ? k : max_k + 1;
}

// A normalised component, h 2^32 + l + ll 2^-32.  The middle word is signed, so
// that its products with a signed word are single instructions.
struct FxDiff {
  int32_t h, l;
  uint32_t ll;
};

GB_HD FxDiff fx_scale(const Fx96& d, int k) {
  const uint32_t w1 = fx_shl(d.w0, d.w1, k);
  return FxDiff{(int32_t)(fx_shl(d.w1, d.w2, k) + (w1 >> 31)), (int32_t)w1, d.w0 << k};
}

// R = (|d|^2 + eps^2) 4^k; the table's eps^2 carries the mean of what is dropped.
GB_HD uint64_t fx_r2(const FxDiff& x, const FxDiff& y, const FxDiff& z, uint64_t eps2) {
  int64_t a = fx_mads(z.h, z.h, fx_mads(y.h, y.h, fx_mads(x.h, x.h, (int64_t)eps2)));
  const int64_t b = fx_mads(z.h, z.l, fx_mads(y.h, y.l, fx_muls(x.h, x.l)));
  return (uint64_t)fx_mads((int32_t)fx_hi((uint64_t)b), 2, a);
}

// Y <= 2^61 / sqrt(R), within 2^-19.9 of it from below: 24 bits from the SFU's
// reciprocal square root (relative error <= 2^-22.9), scaled down by 5 2^-24
// so that the residual 1 - R Y^2 / 2^122 is positive.
GB_HD float fx_rsqrt_seed_float(uint64_t r) {
  const float rh = (float)fx_hi(r);
  constexpr float kScale = 35184372088832.0f * (1.0f - 5.0f / 16777216.0f);
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(rh));
  return __fmul_rn(y, kScale);
#else
  return (float)(1.0 / __builtin_sqrt((double)rh)) * kScale;
#endif
}
GB_HD uint32_t fx_rsqrt_seed(float y) {
#ifdef __CUDA_ARCH__
  return __float2uint_rz(y);
#else
  return (uint32_t)y;
#endif
}

// Residual e = 1 - R Q / 2^122 of Q = Y^2, in units of 2^-58.
GB_HD uint64_t fx_residual(uint64_t r, uint64_t q) {
  const uint64_t m = fx_mad(fx_lo(r), fx_hi(q), fx_mul(fx_hi(r), fx_lo(q)));
  const uint64_t rq = fx_mad(fx_hi(r), fx_hi(q), fx_pair(fx_hi(m), 0));
  return (1ull << 58) - 1 - rq;
}

// y (1 - e)^(-c) in units of 2^-32 for Y = y, to the second order in e (the
// third is below 2^-58): e1 = 2^6 c, e2 = 2^4 c (c + 1) / 2.
GB_HD uint64_t fx_refine(uint32_t y, uint64_t e, uint32_t e1, uint32_t e2) {
  const uint32_t eh = (uint32_t)(e >> 12);
  // the correction in units of 2^-64
  const uint64_t g0 = fx_mad(fx_lo(e), e1, fx_pair(fx_hi(fx_mul(eh * e2, eh)), 0));
  const uint32_t gl = fx_lo(g0), gh = fx_hi(g0) + fx_hi(e) * e1;
  return fx_mad(y, gh, fx_pair(fx_hi(fx_mul(y, gl)), y));
}

// The high 64 bits of a product (without the low words' part: 1 unit).
GB_HD uint64_t fx_mul_hi(uint64_t a, uint64_t b) {
  const uint64_t m = fx_mad(fx_lo(a), fx_hi(b), fx_mul(fx_hi(a), fx_lo(b)));
  return fx_mad(fx_hi(a), fx_hi(b), fx_pair(fx_hi(m), 0));
}

// S = 2^151 R^(-3/2) = Y^3 (1 - e)^(-3/2) (in [2^58, 2^61]); yf = Y.
GB_HD uint64_t fx_rinv3(uint64_t r, float& yf) {
  yf = fx_rsqrt_seed_float(r);
  const uint32_t y = fx_rsqrt_seed(yf);
  const uint64_t q = fx_mul(y, y);
  return fx_mul_hi(fx_refine(y, fx_residual(r, q), 96u, 30u), q);
}

// 2^93 R^(-1/2) = Y (1 - e)^(-1/2) 2^32 (in [2^62, 2^63]).
GB_HD uint64_t fx_rinv1(uint64_t r) {
  const uint32_t y = fx_rsqrt_seed(fx_rsqrt_seed_float(r));
  return fx_refine(y, fx_residual(r, fx_mul(y, y)), 32u, 6u);
}

// Adds weight p times the component V = 2 S (h 2^32 + l + ll 2^-32) / 2^32, of
// which a term has 2^90 to 2^92; s = 2 S.  With S split like the component, the words' carries go
// through the multiply-adds' addends.  Two words, within 0.8 2^32 (2^-58 of the
// term, 2^-60 in the mean), or, WIDE, three, within 2: the parts that two drop are all that a
// component far smaller than the distance has.
template <bool WIDE>
GB_HD void fx_add(FxAcc& a, uint64_t s, const FxDiff& d, uint32_t p) {
  const int32_t sl = (int32_t)fx_lo(s), sh = (int32_t)(fx_hi(s) + (fx_lo(s) >> 31));
  int64_t low = 1ll << 31;
  if (WIDE) low = (int32_t)fx_hi((uint64_t)fx_mads(sl, d.l, (int64_t)fx_mul((uint32_t)sh, d.ll)));
  const int64_t m = fx_mads(sl, d.h, fx_mads(sh, d.l, low));
  const uint64_t h = (uint64_t)fx_mads(sh, d.h, (int32_t)fx_hi((uint64_t)m));
  a.h = fx_mads((int32_t)fx_hi(h), (int32_t)p, a.h);
  a.m = fx_mad(fx_lo(h), p, a.m);
  if (WIDE) a.l = fx_mad(fx_lo((uint64_t)m), p, a.l);
}

// Terms added between two folds: a.l and a.m stay below 2^63 (2^32 2^26 a term).
constexpr int kFxChunk = 32;

GB_HD void fx_fold(__int128& tot, FxAcc& a) {
  tot += ((__int128)a.h << 64) + ((__int128)a.m << 32) + (__int128)a.l;
  a.h = 0;
  a.l = 0;
  a.m = 0;
}

// A term is below 2^118 in size, a fold of 32 below 2^123: 2^36 folds in 160 bits.
GB_HD void fx_tot_add(FxTot& t, unsigned __int128 l, int32_t h) {
  t.l += l;
  t.h += h + (t.l < l ? 1 : 0);
}
GB_HD void fx_fold(FxTot& tot, FxAcc& a) {
  __int128 v = 0;
  fx_fold(v, a);
  fx_tot_add(tot, (unsigned __int128)v, v < 0 ? -1 : 0);
}

// v 2^sc to the nearest double (|v| < 2^126, the result's exponent in range).
GB_HD double fx_to_double(__int128 v, int sc) {
  const bool neg = v < 0;
  unsigned __int128 u = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
  uint64_t hi = (uint64_t)(u >> 64), lo = (uint64_t)u;
  if ((hi | lo) == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int z = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
#else
  const int z = hi ? __builtin_clzll(hi) : 64 + __builtin_clzll(lo);
#endif
  u <<= z;
  hi = (uint64_t)(u >> 64);
  lo = (uint64_t)u;
  // 53 bits, nearest even
  uint64_t m = hi >> 11;
  const uint64_t rest = hi & 0x7ff;
  if (rest > 0x400 || (rest == 0x400 && (lo != 0 || (m & 1)))) ++m;
  // value = m 2^(127 - z - 52 + sc); m may have become 2^53
  const uint64_t bits = ((uint64_t)(127 - z + sc + 1022) << 52) + m + (neg ? 1ull << 63 : 0);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)bits);
#else
  double d;
  memcpy(&d, &bits, 8);
  return d;
#endif
}

GB_HD double fx_to_double(const FxTot& t, int sc) {
  if (t.h == ((__int128)t.l < 0 ? -1 : 0)) return fx_to_double((__int128)t.l, sc);
  const __int128 v = (__int128)((unsigned __int128)(uint32_t)t.h << 96 | t.l >> 32);
  return fx_to_double(v | ((uint32_t)t.l != 0 ? 1 : 0), sc + 32);
}

// Row k of the softening table on the grid of ex: eps^2 in units of (2^64 U)^2
// times 4^k, truncated (the 2 is the mean of what fx_r2 drops), 4^k as the
// weight.  A row whose eps^2 does not fit is never read: R would exceed 2^62.
GB_HD FxRow fx_row(int k, double eps2, int ex) {
#ifdef __CUDA_ARCH__
  const uint64_t bits = (uint64_t)__double_as_longlong(eps2);
#else
  uint64_t bits;
  memcpy(&bits, &eps2, 8);
#endif
  const int ee = (int)(bits >> 52);  // eps^2 >= 0; subnormals count as zero
  const uint64_t m = ee ? (bits & 0xfffffffffffffull) | (1ull << 52) : 0;
  const int sh = ee - 1075 + 2 * (30 - ex + k);
  const uint64_t e = (sh > 9 ? 1ull << 62 : sh >= 0 ? m << sh : sh > -64 ? m >> -sh : 0) + 2;
  return FxRow{(uint32_t)e, (uint32_t)(e >> 32), k <= kFxMaxK ? 1u << (2 * k) : 0u,
               k <= kFxMaxK ? fx_float_of((uint32_t)(127 - 62 + 3 * k) << 23) : 0.0f};
}

// A partner's record.  Per-body masses come in classes of four binary orders,
// class c the exponents em - 4 c - 3 ... em - 4 c with em the largest mass's:
// mass = mu 2^(eb + q - 62), mu in [2^62, 2^63), eb the class's lowest exponent
// and 0 <= q <= 3, mu = 0 for a mass of 0.  Every class has sums of its own
// (fx_class_exp), so a term keeps its bits however light its partner is: the
// heaviest body feels only the others.
struct alignas(16) FxBody {
  Fx96 x, y, z;
  uint32_t mu_lo, mu_hi;
  uint32_t tag;  // q, class, index in the tile, end of the class's run of records
};

constexpr int kFxClassFp64 = 255;  // masses below 2^-300: terms in FP64
GB_HD uint32_t fx_tag(int q, int cls, int index, int end) {
  return (uint32_t)(q | cls << 2 | index << 10 | end << 18);
}
GB_HD int fx_tag_q(uint32_t t) { return (int)(t & 3); }
GB_HD int fx_tag_class(uint32_t t) { return (int)(t >> 2 & 255); }
GB_HD int fx_tag_index(uint32_t t) { return (int)(t >> 10 & 255); }
GB_HD int fx_tag_end(uint32_t t) { return (int)(t >> 18); }
GB_HD int fx_class_exp(int em, int cls) { return em - 4 * cls - 3; }

// Mantissa and tag (class and q) of a mass; em - 300 exponents at most.
GB_HD void fx_mass(FxBody& b, double mass, int em) {
#ifdef __CUDA_ARCH__
  const uint64_t bits = (uint64_t)__double_as_longlong(mass);
#else
  uint64_t bits;
  memcpy(&bits, &mass, 8);
#endif
  const int e = (int)((bits >> 52) & 0x7ff) - 1023;
  const bool normal = e >= -300;
  const uint64_t mu = normal ? ((bits & 0xfffffffffffffull) | (1ull << 52)) << 10 : 0;
  b.mu_lo = fx_lo(mu);
  b.mu_hi = fx_hi(mu);
  const int down = normal ? em - e : 0;
  b.tag = fx_tag(normal ? 3 - (down & 3) : 0,
                 normal ? down >> 2 : bits << 1 ? kFxClassFp64 : 0, 0, 0);
}

// Sizes of the terms added.  Two words: the sum p of the weights (V is within
// 0.8 2^32 p), and in FP32 the sums c[3] of the components' sizes, in units of
// 2^31 of V's, with masses without their mantissas (at least half of it).  Three
// words: m, at least the sum of the terms' sizes (as S |d| <= 2^151 / R), in units
// of 2^30.
struct FxSize {
  uint32_t p;  // of kFxChunk terms
  float c[3], m;
};

// One term of the accelerations into the three sums and its sizes into z.
// Returns its normalisation (above fx_max_k: not added).  With masses the weight
// is 4^k 2^q.
template <bool MASS, bool WIDE>
GB_HD int fx_term(const FxBody& j, const Fx96& xi, const Fx96& yi, const Fx96& zi, float eps2f,
                  const FxRow* tab, FxAcc (&a)[3], FxSize& z) {
  const Fx96 ux = fx_sub(j.x, xi), uy = fx_sub(j.y, yi), uz = fx_sub(j.z, zi);
  const int k = fx_norm(ux, uy, uz, eps2f, fx_max_k<MASS>());
  const FxRow row = tab[k];
  const FxDiff dx = fx_scale(ux, k), dy = fx_scale(uy, k), dz = fx_scale(uz, k);
  float yf;
  uint64_t s = fx_rinv3(fx_r2(dx, dy, dz, fx_pair(row.e_lo, row.e_hi)), yf) << 1;
  uint32_t p = row.p;
  float pf = row.pf;
  if (MASS) {
    s = fx_mul_hi(s << 1, fx_pair(j.mu_lo, j.mu_hi));  // 2 S mass 2^(-eb - q - 1)
    const bool on = k <= kFxMaxKMass && j.mu_hi != 0;
    p = on ? p << fx_tag_q(j.tag) : 0u;
    if (!WIDE)
      pf = on ? fx_float_of(fx_float_bits(pf) + ((uint32_t)fx_tag_q(j.tag) << 23)) : 0.0f;
  }
  if (WIDE) {
    z.m += (float)p * (yf * yf);
  } else {
    z.p += p;
    // |h| = |high word| 2^k, and S = Y^3 2^-32
    const float w = pf * yf * (yf * yf);
    z.c[0] += w * fx_abs((float)(int32_t)ux.w2);
    z.c[1] += w * fx_abs((float)(int32_t)uy.w2);
    z.c[2] += w * fx_abs((float)(int32_t)uz.w2);
  }
  fx_add<WIDE>(a[0], s, dx, p);
  fx_add<WIDE>(a[1], s, dy, p);
  fx_add<WIDE>(a[2], s, dz, p);
  return k;
}

// What a body's term with itself adds to z.p (its components are zero).
template <bool MASS>
GB_HD uint32_t fx_self_weight(float eps2f, const FxRow* tab, const FxBody& j) {
  const int k = fx_norm(Fx96{}, Fx96{}, Fx96{}, eps2f, fx_max_k<MASS>());
  if (k > fx_max_k<MASS>()) return 0u;
  return !MASS ? tab[k].p : j.mu_hi ? tab[k].p << fx_tag_q(j.tag) : 0u;
}
template <bool MASS>
GB_HD int fx_term(const FxBody& j, const Fx96& xi, const Fx96& yi, const Fx96& zi, float eps2f,
                  const FxRow* tab, FxAcc (&a)[3]) {
  FxSize z = {};
  return fx_term<MASS, false>(j, xi, yi, zi, eps2f, tab, a, z);
}

// One term of the potential, [mass] / sqrt(|d|^2 + eps^2), into a.m and a.l;
// with weight 0 where `on` is false.
template <bool MASS>
GB_HD int fx_term_pot(const FxBody& j, const Fx96& xi, const Fx96& yi, const Fx96& zi, float eps2f,
                      const FxRow* tab, bool on, FxAcc& a) {
  const Fx96 ux = fx_sub(j.x, xi), uy = fx_sub(j.y, yi), uz = fx_sub(j.z, zi);
  const int k = fx_norm(ux, uy, uz, eps2f, kFxMaxK);
  const FxRow row = tab[k];
  const FxDiff dx = fx_scale(ux, k), dy = fx_scale(uy, k), dz = fx_scale(uz, k);
  uint64_t y = fx_rinv1(fx_r2(dx, dy, dz, fx_pair(row.e_lo, row.e_hi)));
  int t = k;
  if (MASS) {
    y = fx_mul_hi(y, fx_pair(j.mu_lo, j.mu_hi));  // y mass 2^(-eb - q - 2)
    t += fx_tag_q(j.tag);
  }
  const uint32_t p = on && k <= kFxMaxK ? 1u << t : 0u;
  a.m = fx_mad(fx_hi(y), p, a.m);
  a.l = fx_mad(fx_lo(y), p, a.l);
  return k;
}

// Two words serve a component whose terms' sizes come to 2^kFxEnough times the
// weights or more, 2^-8 to 2^-10 of the terms: V's error, 0.8 2^32 of a weight at
// most and 0.3 2^32 in the mean, is then 6 2^-53 and 2 2^-53 of it, as that of a
// term in FP64 (5 and 1.3 2^-53).  Three words serve one whose sum is above
// 2^-kFxThin of the terms' sizes: V's 2 units and the coordinates' last bits,
// 2^-80 of a term at most, are then within 2^-54 of it.  A sum below that (of a
// body in a plane, nearly) is taken in FP64.
constexpr int kFxEnough = 82;
constexpr int kFxThin = 26;
constexpr int kFxShort = 8;  // an axis 2^-kFxShort of the longest: three words

// exponent of a term's unit: sum 2^(fx_out_exp(ex)) is the sum of d / r^3, and
// sum 2^(fx_out_exp(ex) + eb + 1) that of mass d / r^3; of the potential:
// 1 / r, and with eb + 2 mass / r
GB_HD int fx_out_exp(int ex) { return -92 - 2 * ex; }
GB_HD int fx_out_exp_pot(int ex) { return -63 - ex; }

// eps^2 in units of (2^64 U)^2
GB_HD float fx_eps2f(double eps2, int ex) {
  const FxRow r = fx_row(0, eps2, ex);  // at most 2^58 and its first row
  return (float)fx_pair(r.e_lo, r.e_hi);
}

}  // namespace gb
