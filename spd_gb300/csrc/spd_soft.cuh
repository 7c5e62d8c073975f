// Correctly rounded FP64 products on the integer pipes.
//
// Why: GB300 issues about 1.7 FP64 lane-operations per clock and SM (DADD and
// DMUL chains: 76 issue cycles of an SM sub-partition per warp instruction),
// against 64 integer lanes.  The step's contractions are a rounded product and
// a rounded sum per term, so half of the FP64 instructions that bound them are
// products with a constant operator entry.  The product of two 53-bit
// significands is four 32x32 -> 64-bit multiplies and a carry chain; rounded
// to nearest-even in integer registers, its operand's preparation included, it
// takes 49 issue cycles and runs beside the FP64 additions (product + DADD: 76
// cycles, DMUL + DADD: 152).  Measured by profiles/integer_pipe_rates.cu.
//
// The result is the IEEE 754 product bit for bit: the operands are finite,
// nonzero and far from underflow and overflow (tested per line of values,
// see Line), every other operand is multiplied by the FP64 unit.
//
// The build with fused multiply-adds keeps a*b + c as one FP64 instruction;
// it takes quotients, roots and the first product of each sum from here (that
// one has nothing to fuse with).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

// device code; also host-callable so the scalar maps can be checked on a CPU
#ifndef SPD_FN
#define SPD_FN __host__ __device__ __forceinline__
#endif

namespace spd {

#ifdef __CUDA_ARCH__
__device__ __noinline__ double div_ieee_slow(double a, double b) { return a / b; }
#else
inline double div_ieee_slow(double a, double b) { return a / b; }
#endif
// Predicates on a double's bit pattern evaluated on its two 32-bit words
// (integer pipes).  The same tests written on the 64-bit pattern (for
// instance (bits & ~sign) > bits(inf) for NaN) were compiled to FP64-pipe
// instructions, measured with ncu (one per test), on the pipe that bounds
// the step's kernels.
SPD_FN unsigned hi_word(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(x);
#else
  unsigned long long b;
  memcpy(&b, &x, sizeof(b));
  return (unsigned)(b >> 32);
#endif
}
SPD_FN unsigned lo_word(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(x);
#else
  unsigned long long b;
  memcpy(&b, &x, sizeof(b));
  return (unsigned)b;
#endif
}
// x is a NaN
SPD_FN bool nan_w(double x) {
  const unsigned h = hi_word(x) & 0x7fffffffu;
  return h > 0x7ff00000u || (h == 0x7ff00000u && lo_word(x) != 0u);
}
// x != 0 (true for NaN, false for both zeros)
SPD_FN bool nonzero_w(double x) { return ((hi_word(x) & 0x7fffffffu) | lo_word(x)) != 0u; }
// x > 0 (false for zeros, negatives and NaN)
SPD_FN bool gt0_w(double x) {
  const unsigned h = hi_word(x), l = lo_word(x);
  return (h >> 31) == 0u && (h | l) != 0u && (h < 0x7ff00000u || (h == 0x7ff00000u && l == 0u));
}

// An operator entry (made on the host, coef_of).  For soft_prod: the
// significand scaled to [2^62, 2^63), and sign and exponent less the bias in
// the upper 12 bits; the double's own high word gives the value back.
struct alignas(16) Coef {
  uint32_t ml, mh, e, hi;
};
inline Coef coef_of(double a) {
  unsigned long long b;
  memcpy(&b, &a, sizeof(b));
  const unsigned long long m = ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 10;
  const uint32_t hi = (uint32_t)(b >> 32);
  return Coef{(uint32_t)m, (uint32_t)(m >> 32), (hi & 0xfff00000u) - (1023u << 20), hi};
}
// Magnitudes for which an operator takes part, all of its entries within
// [2^-256, 2^256] (so none zero): with the other operand's exponent window
// (Line) no product can then leave the normal range.
inline bool coef_in_range(double a) {
  const double m = fabs(a);
  return m >= 0x1p-256 && m <= 0x1p256;
}

// The other operand: significand scaled to [2^53, 2^54), sign and exponent.
// A zero has significand 0, a stand-in exponent that keeps the sign bit of
// the exponent sum right, and a mask that leaves nothing but the sign of its
// products (fluids at rest are full of exact zeros next to values of the
// size of a rounding error).
struct Opnd {
  uint32_t ml, mh, e, keep;
};
SPD_FN double from_words(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const unsigned long long b = ((unsigned long long)hi << 32) | lo;
  double x;
  memcpy(&x, &b, sizeof(x));
  return x;
#endif
}
SPD_FN uint32_t funnel_l1(uint32_t lo, uint32_t hi) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, 1);
#else
  return (hi << 1) | (lo >> 31);
#endif
}
// ``ok`` keeps bit 30 when x is a zero or its biased exponent lies in
// [512, 1535] (the two upper exponent bits differ: |x| in [2^-511, 2^513)).
SPD_FN Opnd opnd_of(double x, uint32_t& ok) {
  const uint32_t h = hi_word(x), l = lo_word(x), h2 = h << 1;
  const bool zero = (h2 | l) == 0u;
  const uint32_t m = zero ? 0u : (h & 0xfffffu) | 0x100000u;
  ok &= zero ? 0x40000000u : h ^ h2;
  return Opnd{l << 1, funnel_l1(l, m), zero ? h | (1023u << 20) : h & 0xfff00000u, zero ? 0x80000000u : 0xffffffffu};
}
// The same of a product, whose mask ``keep`` says whether a factor is a zero:
// the fields by the mask's bits instead of a choice each.
SPD_FN Opnd opnd_of_product(double x, uint32_t keep, uint32_t& ok) {
  const uint32_t h = hi_word(x), l = lo_word(x);
  ok &= (h ^ (h << 1)) | ~keep;
  return Opnd{l << 1, funnel_l1(l, ((h & 0xfffffu) | 0x100000u) & keep), (h & 0xfff00000u) | (~keep & (1023u << 20)), keep};
}

// the entry, times 2^k with ``eoff`` = k << 20
SPD_FN double coef_value(const Coef& c, uint32_t eoff) {
  return from_words(c.hi + eoff, (c.ml >> 10) | (c.mh << 22));
}
// The product of the scaled significands of a coefficient-like operand
// (mh:ml in [2^62, 2^63)) and an Opnd, in [2^115, 2^117): words 3:2 hold the
// 53-bit result when bit 116 is set and one bit less otherwise; then the
// words are shifted up by one and the exponent is one less.  mh < 2^31 and
// the operand's mh < 2^22 keep the middle sum below 2^64.  Word 0 is not
// shifted with the rest: only whether it is zero matters, and only where
// word 1 is a tie, which the bit shifted into word 1 excludes.
struct Prod {
  uint32_t p0, w1, w2, w3, e;
  bool up;  // shifted
};
SPD_FN Prod soft_words(uint32_t cl, uint32_t ch, uint32_t e, const Opnd& x) {
  const unsigned long long p = (unsigned long long)cl * x.ml;
  const unsigned long long q = (unsigned long long)ch * x.ml + (unsigned long long)cl * x.mh;
  const unsigned long long r = (unsigned long long)ch * x.mh;
  Prod o;
  o.p0 = (uint32_t)p;
  o.w1 = (uint32_t)(p >> 32);
  o.w2 = (uint32_t)r;
  o.w3 = (uint32_t)(r >> 32);
  o.e = e;
#ifdef __CUDA_ARCH__
  asm("add.cc.u32 %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32 %2, %2, 0;"
      : "+r"(o.w1), "+r"(o.w2), "+r"(o.w3)
      : "r"((uint32_t)q), "r"((uint32_t)(q >> 32)));
#else
  {
    const unsigned long long s = (unsigned long long)o.w1 + (uint32_t)q;
    const unsigned long long t = (unsigned long long)o.w2 + (uint32_t)(q >> 32) + (s >> 32);
    o.w1 = (uint32_t)s;
    o.w2 = (uint32_t)t;
    o.w3 += (uint32_t)(t >> 32);
  }
#endif
  o.up = o.w3 < 0x100000u;
  if (o.up) {
    o.w3 = funnel_l1(o.w2, o.w3);
    o.w2 = funnel_l1(o.w1, o.w2);
    o.w1 = funnel_l1(o.p0, o.w1);
    o.e -= 0x100000u;
  }
  return o;
}

// The product rounded: adds 2^63 - 1 (2^63 when the result is odd) to words
// 1:0; the carry into the exponent field is the rounding up to the next power
// of two.
SPD_FN double soft_round(Prod o, uint32_t keep) {
  const uint32_t t = o.p0 | (o.w2 & 1u);
#ifdef __CUDA_ARCH__
  asm("{\n\t"
      ".reg .u32 drop;\n\t"
      "add.cc.u32 drop, %2, 0xffffffff;\n\t"
      "addc.cc.u32 drop, %3, 0x7fffffff;\n\t"
      "addc.cc.u32 %0, %0, 0;\n\t"
      "addc.u32 %1, %1, %4;\n\t"
      "}"
      : "+r"(o.w2), "+r"(o.w3)
      : "r"(t), "r"(o.w1), "r"(o.e));
#else
  {
    const unsigned long long s = (unsigned long long)o.w1 + 0x7fffffffu + (t != 0u);
    const unsigned long long u = (unsigned long long)o.w2 + (s >> 32);
    o.w2 = (uint32_t)u;
    o.w3 += o.e + (uint32_t)(u >> 32);
  }
#endif
  return from_words(o.w3 & keep, o.w2);
}
SPD_FN double soft_prod(const Coef& c, const Opnd& x) {
  return soft_round(soft_words(c.ml, c.mh, c.e + x.e, x), x.keep);
}

// A divisor b prepared for several quotients: 2^63 over its significand,
// rounded down to within 4 units (so in [2^62, 2^63)), the quotient's
// exponent offset, and whether b lies in [2^-256, 2^256).
struct alignas(16) Recip {
  uint32_t ml, mh, e, ok;
};

// Reciprocal of a significand by two Newton steps y += y (1 - b y) in fixed
// point from the FP32 approximation (the integer form of the iteration in
// Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed., 4.7):
// relative error 2^-22, then 2^-43.9, then the rounding of the last step.
// Each step rounds down, and one unit is taken off at the end, so the result
// is below the exact value.  62 issue cycles, 344 for the FP64 1 / x (a whole
// quotient 135 against 572; profiles/integer_pipe_rates.cu).
SPD_FN Recip recip_soft(double b) {
  const uint32_t h = hi_word(b), l = lo_word(b);
  const uint32_t bh = (((h & 0xfffffu) | 0x100000u) << 11) | (l >> 21), bl = l << 11;  // [2^63, 2^64)
  const uint32_t fb = (bh >> 8) + 0x3f000000u;  // the significand in [1, 2), truncated to FP32
#ifdef __CUDA_ARCH__
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(__uint_as_float(fb)));
  const uint32_t y0 = (__float_as_uint(r0) << 6) + 0x60000000u;  // scale 2^30, [2^29, 2^30]
  const uint32_t t0 = __umulhi(bl, y0);
#else
  float f, r0;
  memcpy(&f, &fb, sizeof(f));
  r0 = 1.0f / f;
  uint32_t rb;
  memcpy(&rb, &r0, sizeof(rb));
  const uint32_t y0 = (rb << 6) + 0x60000000u;
  const uint32_t t0 = (uint32_t)(((unsigned long long)bl * y0) >> 32);
#endif
  // 1 - b y0 in scale 2^61, then 2^52 in 32 bits; y1 in scale 2^63
  const long long e0 = (long long)(0x2000000000000000ULL - ((unsigned long long)bh * y0 + t0));
  const long long d0 = (long long)(int)(uint32_t)(e0 >> 9) * (int)y0;
  const unsigned long long y1 = ((unsigned long long)y0 << 33) + (unsigned long long)(d0 >> 19);
  const uint32_t yh = (uint32_t)(y1 >> 32), yl = (uint32_t)y1;
  // 1 - b y1 (below 2^-43): words 2:1 of the product, scale 2^94
#ifdef __CUDA_ARCH__
  const uint32_t p1 = __umulhi(bl, yl);
#else
  const uint32_t p1 = (uint32_t)(((unsigned long long)bl * yl) >> 32);
#endif
  const unsigned long long m = (unsigned long long)bh * yl + (unsigned long long)bl * yh + p1 +
                               ((unsigned long long)(bh * yh) << 32);
  const int e1 = (int)(uint32_t)((long long)(0ULL - m) >> 20);  // scale 2^74
#ifdef __CUDA_ARCH__
  const int dy = __mulhi((int)(yh >> 1), e1);
#else
  const int dy = (int)(((long long)(int)(yh >> 1) * e1) >> 32);
#endif
  const unsigned long long y = y1 + (unsigned long long)(long long)((dy >> 9) - 1);
  Recip r;
  r.ml = (uint32_t)y;
  r.mh = (uint32_t)(y >> 32);
  r.e = (1022u << 20) - (h & 0xfff00000u);
  r.ok = ((h & 0x7fffffffu) - (767u << 20)) < (512u << 20) ? 0x40000000u : 0u;
  return r;
}

// a / b rounded to nearest, b's reciprocal prepared.  The truncated product
// of a with the reciprocal is the quotient's 53-bit floor or, rarely, one
// less; the exact remainder a - b q (its low 64 bits hold it) against half of
// b decides the last place.  A quotient of two 53-bit numbers is never a tie.
// a: a zero or within opnd_of's window; any other pair is divided by the
// FP64 unit.
SPD_FN double div_words(const Opnd& x, double b, const Recip& rb) {
  const Prod o = soft_words(rb.ml, rb.mh, rb.e + x.e, x);
  const uint32_t bl = lo_word(b), bh = (hi_word(b) & 0xfffffu) | 0x100000u;
  // b + 2 (b q - a 2^s), negative where the remainder exceeds b/2; a 2^s has
  // only bits above 52 (s = 52, or 53 when the product was shifted)
  const unsigned long long pl = (unsigned long long)bl * o.w2;
  const unsigned long long p = pl + ((unsigned long long)(bl * o.w3 + bh * o.w2) << 32);
  const uint32_t a2 = x.ml << (o.up ? 21 : 20);
  const unsigned long long t = (((unsigned long long)bh << 32) | bl) + (p << 1) - ((unsigned long long)a2 << 32);
  const unsigned long long q = (((unsigned long long)(o.w3 + o.e) << 32) | o.w2) + (t >> 63);
  return from_words((uint32_t)(q >> 32) & x.keep, (uint32_t)q);
}

SPD_FN double div_soft(double a, double b, const Recip& rb) {
  uint32_t ok = rb.ok;
  const Opnd x = opnd_of(a, ok);
  return ok != 0u ? div_words(x, b, rb) : div_ieee_slow(a, b);
}

// sqrt(x) rounded to nearest.  With x = m 4^k, m in [1, 4): the FP32
// reciprocal root y (relative error below 2^-22), s = m y (1 + (1 - m y^2)/2)
// to 2^-43, then s += (m - s^2) y / 2 to the last place of scale 2^60, taken
// down by 4 units so that its 53-bit floor q is at most one below the
// root's; the exact m - q^2 against q decides the last place (a root of a
// 53-bit number is never a tie).  125 issue cycles, 574 for the FP64 root
// (profiles/integer_pipe_rates.cu).
SPD_FN double sqrt_soft(double x) {
  const uint32_t h = hi_word(x), l = lo_word(x);
  if (((h ^ (h << 1)) & 0x40000000u) == 0u || (h >> 31) != 0u) return sqrt(x);
  const uint32_t odd = ~(h >> 20) & 1u;  // the unbiased exponent is odd
  const unsigned long long mant = ((unsigned long long)((h & 0xfffffu) | 0x100000u) << 32) | l;
  const unsigned long long m = mant << (10 + odd);  // scale 2^62
  const uint32_t fb = 0x3f800000u + (odd << 23) + ((h & 0xfffffu) << 3) + (l >> 29);
#ifdef __CUDA_ARCH__
  float r0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(__uint_as_float(fb)));
  const uint32_t y = (__float_as_uint(r0) << 6) + 0x60000000u;  // scale 2^30
  const unsigned long long a = (unsigned long long)(uint32_t)(m >> 32) * y + __umulhi((uint32_t)m, y);  // m y, 2^60
  const unsigned long long u = (unsigned long long)(uint32_t)(a >> 32) * y + __umulhi((uint32_t)a, y);  // m y^2, 2^58
#else
  float f, r0;
  memcpy(&f, &fb, sizeof(f));
  r0 = (float)(1.0 / sqrt((double)f));
  uint32_t rb;
  memcpy(&rb, &r0, sizeof(rb));
  const uint32_t y = (rb << 6) + 0x60000000u;
  const unsigned long long a =
      (unsigned long long)(uint32_t)(m >> 32) * y + (((unsigned long long)(uint32_t)m * y) >> 32);
  const unsigned long long u =
      (unsigned long long)(uint32_t)(a >> 32) * y + (((unsigned long long)(uint32_t)a * y) >> 32);
#endif
  const int e = (int)(uint32_t)((long long)(0x400000000000000ULL - u) >> 6);  // 1 - m y^2, 2^52
  const unsigned long long s = a + (unsigned long long)(((long long)(int)(uint32_t)(a >> 32) * e) >> 21);
  const uint32_t sh = (uint32_t)(s >> 32), sl = (uint32_t)s;
  // m - s^2 in scale 2^88 (words 2:1 of the square)
#ifdef __CUDA_ARCH__
  const uint32_t p1 = __umulhi(sl, sl);
#else
  const uint32_t p1 = (uint32_t)(((unsigned long long)sl * sl) >> 32);
#endif
  const unsigned long long w = 2ULL * ((unsigned long long)sl * sh) + p1 + ((unsigned long long)(sh * sh) << 32);
  const int d = (int)(uint32_t)((long long)((m << 26) - w) >> 16);  // 2^72
#ifdef __CUDA_ARCH__
  const int c = __mulhi(d, (int)y);
#else
  const int c = (int)(((long long)d * (int)y) >> 32);
#endif
  const unsigned long long q = (s + (unsigned long long)(long long)((c >> 11) - 4)) >> 8;
  const uint32_t qh = (uint32_t)(q >> 32), ql = (uint32_t)q;
  const unsigned long long q2 = (unsigned long long)ql * ql + ((unsigned long long)(2u * ql * qh) << 32);
  const unsigned long long rem = ((unsigned long long)(l << (20 + odd)) << 32) - q2;
  // exponent: (E - odd)/2 of the unbiased E, re-biased, less the leading bit
  const uint32_t eo = ((((h >> 20) - odd - 1023u) >> 1) << 20) + (1022u << 20);
  const unsigned long long out = (((unsigned long long)(qh + eo) << 32) | ql) + ((q - rem) >> 63);
  return from_words((uint32_t)(out >> 32), (uint32_t)out);
}

// A double with its prepared operand, for expressions whose products all run
// on the integer pipes (sums stay on the FP64 pipe).  ``ok`` (bit 30): the
// value and every value it came from are zeros or within opnd_of's window.
// A product of two such values is at least 2^-1022; one above the largest
// double leaves the exponent field 2047, or 0 with a carry into the sign bit,
// and fails the window itself.  Its words can be those of a zero (a product
// that rounds to 2^1025), so whether a product is a zero is taken from its
// factors.  A result without ``ok`` is computed again in plain FP64
// arithmetic.  Unused preparations are dead code.
struct Num {
  double v;
  Opnd o;
  uint32_t ok;
  SPD_FN Num() {}
  SPD_FN Num(double x, uint32_t from = 0x40000000u) : v(x) {
    ok = from;
    o = opnd_of(x, ok);
  }
};
SPD_FN Num operator+(const Num& a, const Num& b) { return Num(a.v + b.v, a.ok & b.ok); }
SPD_FN Num operator-(const Num& a, const Num& b) { return Num(a.v - b.v, a.ok & b.ok); }
SPD_FN Num operator-(const Num& a) { return Num(from_words(hi_word(a.v) ^ 0x80000000u, lo_word(a.v)), a.ok); }
SPD_FN Num operator*(const Num& a, const Num& b) {
  const uint32_t ch = (a.o.mh << 9) | (a.o.ml >> 23);
  const uint32_t keep = a.o.keep & b.o.keep;
  Num r;
  r.v = soft_round(soft_words(a.o.ml << 9, ch, a.o.e + b.o.e - (1023u << 20), b.o), keep);
  r.ok = a.ok & b.ok;
  r.o = opnd_of_product(r.v, keep, r.ok);
  return r;
}
SPD_FN Num operator+(const Num& a, double b) { return a + Num(b); }
SPD_FN Num operator-(const Num& a, double b) { return a - Num(b); }
SPD_FN Num operator-(double a, const Num& b) { return Num(a) - b; }
SPD_FN Num operator*(const Num& a, double b) { return a * Num(b); }
SPD_FN Num operator*(double a, const Num& b) { return Num(a) * b; }
SPD_FN Num div_by(const Num& a, const Num& b, const Recip& rb) { return Num(div_words(a.o, b.v, rb), a.ok & b.ok & rb.ok); }
SPD_FN Num div_by(const Num& a, double b, const Recip& rb) { return Num(div_words(a.o, b, rb), a.ok & rb.ok); }
SPD_FN Recip recip_of(const Num& b) { return recip_soft(b.v); }
SPD_FN Num operator/(const Num& a, const Num& b) { return div_by(a, b, recip_of(b)); }
// x / 2: one less in the exponent
SPD_FN Num half(const Num& a) {
  const uint32_t h = hi_word(a.v);
  return Num(from_words(a.o.keep == 0x80000000u ? h : h - 0x100000u, lo_word(a.v)), a.ok);
}
SPD_FN Num ad_sqrt(const Num& a) { return Num(sqrt_soft(a.v), a.ok); }
SPD_FN Num ad_abs(const Num& a) { return Num(from_words(hi_word(a.v) & 0x7fffffffu, lo_word(a.v)), a.ok); }
SPD_FN double sval(const Num& a) { return a.v; }

}  // namespace spd
