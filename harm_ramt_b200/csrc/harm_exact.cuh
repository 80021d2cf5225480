// Correctly rounded FP64 quotients and square roots without branches.
//
// The step's FP64 results are the reference's bit for bit, so every `/` and
// sqrt() has to round as IEEE does.  Compiled from `a / b` and `sqrt(x)`,
// each is a sequence of its own with a branch for the operands it cannot
// take; a zone of the step has about 130 of them, and between two branches
// the scheduler has one short dependency chain to work with.  Here a group
// of them is straight-line code, quotients by one divisor share its
// reciprocal, and the operands are only watched: after the group, ok() tells
// whether every one was in the range where the results are exact.  Where it
// does not, the caller evaluates the group again with the operators (rare:
// numbers below 2^-950 that are not zero, wild values, branches that only
// the general code follows).
//
// Method: Newton's iteration for the reciprocal (and, in the cubic form, for
// the reciprocal root) from the hardware's documented approximation, then one
// residual correction of the result, the residual formed exactly by a fused
// multiply-add (Markstein, IBM J. Res. Dev. 34 (1990); Muller et al.,
// Handbook of Floating-Point Arithmetic, 4.7).  Why they round correctly:
//  * reciprocal: y1 is 1/b within e1 = 1 - b y1, |e1| < 2^-52.8, e1 exact;
//    y = fl(y1 (1 + e1 + 2^-95)) is 1/b rounded, but for an error between 0
//    and 2^-95 / b before the rounding;
//  * quotient: q0 = fl(a y) is off by less than 1.5 ulp, and by half of one
//    where a / b lies next to a tie, so r = a - b q0 is exact there and
//    q0 + r y differs from a / b by half an ulp times |1 - b y|.  With B in
//    [2^52, 2^53) the integer significand of b a quotient is at least 1 / B
//    half ulps from every tie (|2^k A - B M| >= 1 for an odd M of 54 bits).
//    |1 - b y| < 1 / B: for y the nearest number to 1/b, and, below B =
//    2^53 - 2^11, also for the other neighbour of a tie within 2^-95 / b.
//    Above it 1/b is never within 2^-95 / b below a tie (for b = 2 (1 - x) it
//    is 1/2 (1 + x + x^2 + ...), with x an odd or even multiple of 2^-53), so
//    there y is the nearest (without the 2^-95, B = 2^53 - 1 rounds down);
//  * root: g + d h with d = x - g g differs from sqrt(x) by less than 60 *
//    2^-107 / sqrt(x) (x in [1, 4)); x is nearer than that to the square of a
//    tie only for the few x with (2^53 tie)^2 - 2^106 x = N, |N| < 64, which
//    the tests evaluate one by one.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "harm_device.cuh"

namespace harm {

HD_INLINE uint64_t bits_of(double x)
{
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
HD_INLINE uint32_t hi_word(double x) { return (uint32_t)(bits_of(x) >> 32); }
HD_INLINE uint32_t lo_word(double x) { return (uint32_t)bits_of(x); }

// Approximations of 1/b and 1/sqrt(x) to about 20 bits: the hardware's on
// the device; on the host (tests) the quotient cut to its upper word, with
// `nudge` units of that word added to try other seeds.
HD_INLINE double seed_cut(double v, int nudge)
{
  uint64_t u = bits_of(v);
  u = ((u >> 32) + (uint64_t)(int64_t)nudge) << 32;
  double r;
  memcpy(&r, &u, 8);
  return r;
}
HD_INLINE double rcp_seed(double b, int nudge = 0)
{
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#else
  return seed_cut(1.0 / b, nudge);
#endif
}
HD_INLINE double rsqrt_seed(double x, int nudge = 0)
{
#ifdef __CUDA_ARCH__
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
#else
  return seed_cut(1.0 / sqrt(x), nudge);
#endif
}

// a divisor and its reciprocal
struct Recip {
  double b, y;
};

struct Exact {
  // operand ranges, as binary exponents: a quotient of operands inside is
  // normal and its residual is a multiple of 2^-1074.  Divisors and radicands
  // are positive.
  static constexpr int NUM_LO = -950, NUM_HI = 600, POS_LO = -200, POS_HI = 60;
  static HD_INLINE constexpr uint32_t word(int e) { return (uint32_t)(1023 + e) << 20; }
  // the largest distance of an operand's upper word above its range's lower
  // end (an operand below it wraps past the upper end, as do a negative
  // divisor, an infinity and a NaN)
  uint32_t num = 0, pos = 0;

  HD_INLINE bool ok() const { return num <= word(NUM_HI) - word(NUM_LO) && pos <= word(POS_HI) - word(POS_LO); }
  static HD_INLINE uint32_t above(uint32_t m, uint32_t h, uint32_t lo)
  {
#ifdef __CUDA_ARCH__
    return __viaddmax_u32(h, 0u - lo, m);
#else
    return (h - lo > m) ? h - lo : m;
#endif
  }
  // a factor of sums and products that are to stay finite: |a| below 2^528
  HD_INLINE void bounded(double a) { num = above(num, hi_word(a) & 0x7fffffffu, 0); }
  // a value that only the general code handles
  HD_INLINE void need(bool c) { pos = c ? pos : 0xffffffffu; }
  // a numerator: zero (a quotient of zero is exact), or in the range (its
  // lower end raised where only a factor of the numerator is watched)
  template <int LO = NUM_LO>
  HD_INLINE void numerator(double a)
  {
    const uint32_t t = hi_word(a) & 0x7fffffffu;
    if (((hi_word(a) & 0x7fffffffu) | lo_word(a)) != 0) num = above(num, t, word(LO));
  }
  HD_INLINE Recip rcp(double b, int nudge = 0)
  {
    pos = above(pos, hi_word(b), word(POS_LO));
    const double y0 = rcp_seed(b, nudge);
    const double e0 = fma(-b, y0, 1.0);
    const double y1 = fma(y0, fma(e0, e0, e0), y0);
    const double e1 = fma(-b, y1, 1.0);
    return Recip{b, fma(y1, e1 + 0x1p-95, y1)};
  }
  // the reciprocal of b from a value y1 within 2^-51 of it
  HD_INLINE Recip rcp_from(double b, double y1)
  {
    pos = above(pos, hi_word(b), word(POS_LO));
    return Recip{b, fma(y1, fma(-b, y1, 1.0) + 0x1p-95, y1)};
  }
  // a / d.b for a numerator known to be in range, or zero (the quotient of a
  // negative zero is a positive one: no nonzero value depends on it, see
  // ExactTiny::quot)
  static HD_INLINE double quot(double a, const Recip& d)
  {
    const double q = a * d.y;
    return fma(fma(-d.b, q, a), d.y, q);
  }
  HD_INLINE double div(double a, const Recip& d)
  {
    numerator(a);
    return quot(a, d);
  }
  // sqrt(x), x > 0
  HD_INLINE double sqrt_of(double x, int nudge = 0)
  {
    pos = above(pos, hi_word(x), word(POS_LO));
    const double y0 = rsqrt_seed(x, nudge);
    const double e = fma(-(x * y0), y0, 1.0);
    const double y1 = fma(y0 * e, fma(0.375, e, 0.5), y0);
    const double g = x * y1;
    return fma(fma(-g, g, x), 0.5 * y1, g);
  }
};

// The same with numerators down to the smallest subnormal number, for groups
// that carry such numbers (the field ahead of the front it spreads with): the
// quotient is formed 2^400 times as large and scaled down.  Scaling rounds a
// second time where the quotient is subnormal (one just below 2^-1022 may
// become that number): there the residual of the rounded value, exact at the
// larger scale, tells whether it is off by more than half the spacing 2^-1074,
// and moves it by one.
// Its quotients also keep the sign of a zero (the residual is formed with the
// other sign), which the primitives show; the faces' fluxes may be zeros of
// either sign (with this form k_flux of the 1024^2 torus took 267 us instead
// of 265), which the update's sums leave out.
struct ExactTiny : Exact {
  static HD_INLINE double quot(double a, const Recip& d)
  {
    const double q = a * d.y;
    return fma(-fma(d.b, q, -a), d.y, q);
  }
  // a numerator of Exact's range
  HD_INLINE double div_normal(double a, const Recip& d)
  {
    numerator(a);
    return quot(a, d);
  }
  HD_INLINE double div(double a, const Recip& d)
  {
    const double as = a * 0x1p400;
    numerator(as);
    const double q = quot(as, d) * 0x1p-400;
    const double r = fma(-d.b, q * 0x1p400, as);
    const bool off = fabs(q) <= 0x1p-1022 && fabs(r) > fabs(d.b) * 0x1p-675;
    const bool up = (r > 0.) == (as > 0.);
    const uint64_t u = bits_of(q) + (off ? (up ? 1 : ~0ull) : 0);
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v;
    memcpy(&v, &u, 8);
    return v;
#endif
  }
};

}  // namespace harm
