// fp64emu.cuh -- IEEE-754 binary64 operations computed on the integer and
// FP32 pipes, bit-identical to the hardware's round-to-nearest-even results.
//
// GB300 executes FP64 at about 1/57 of its FP32 rate (measured: DFMA 0.6 Top/s,
// DDIV 59 Gop/s vs IMAD 19 Top/s), so a plan that divides or compares doubles
// per row is bound by the FP64 pipe long before HBM.  These routines give the
// exact same bits as the native instructions using 32/64-bit integer
// arithmetic: division by a float-seeded fixed-point Newton reciprocal with an
// exact integer remainder correction (Muller et al., "Handbook of
// Floating-Point Arithmetic", ch. 9: reciprocal iteration + remainder-based
// correction), conversions and comparisons by bit manipulation.
//
// The header compiles for the host too (g++), where the tests check it against
// the CPU's IEEE arithmetic.
#pragma once

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
#define GXE_FN __device__ __forceinline__
#define GXE_ON_DEVICE 1
#else
#include <cstdint>
#include <cstring>
#define GXE_FN static inline
#define GXE_ON_DEVICE 0
#endif

typedef unsigned long long gxe_u64;
typedef long long gxe_i64;

#define GXE_SIGN 0x8000000000000000ull
#define GXE_FRAC 0x000FFFFFFFFFFFFFull
#define GXE_HIDDEN 0x0010000000000000ull
#define GXE_INF 0x7FF0000000000000ull
#define GXE_QNAN 0x7FF8000000000000ull

GXE_FN gxe_u64 gxe_umulhi(gxe_u64 a, gxe_u64 b) {
#if GXE_ON_DEVICE
  return __umul64hi(a, b);
#else
  return (gxe_u64)(((unsigned __int128)a * b) >> 64);
#endif
}

GXE_FN int gxe_clz(gxe_u64 x) {
#if GXE_ON_DEVICE
  return __clzll((gxe_i64)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

GXE_FN float gxe_rcp_approx(float x) {
#if GXE_ON_DEVICE
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#elif defined(GXE_TEST_PERTURB_RCP)
  // host test mode: a seed up to +-2 ulp off (worse than rcp.approx's 1 ulp)
  float r = 1.0f / x;
  unsigned u;
  std::memcpy(&u, &r, 4);
  unsigned xb;
  std::memcpy(&xb, &x, 4);
  u += (unsigned)((xb * 2654435761u) >> 29) % 5u - 2u;
  std::memcpy(&r, &u, 4);
  return r;
#else
  return 1.0f / x;
#endif
}

GXE_FN unsigned gxe_f2u(float f) {
#if GXE_ON_DEVICE
  return __float_as_uint(f);
#else
  unsigned u;
  std::memcpy(&u, &f, 4);
  return u;
#endif
}

GXE_FN float gxe_u2f(unsigned u) {
#if GXE_ON_DEVICE
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, 4);
  return f;
#endif
}

GXE_FN bool gxe_isnan_(gxe_u64 a) { return (a & ~GXE_SIGN) > GXE_INF; }

// Rounds Q * 2^(e - 54) (Q in [2^54, 2^55), `rem` nonzero if inexact beyond Q)
// to binary64 with round-to-nearest-even; handles overflow and subnormals.
GXE_FN gxe_u64 gxe_round_pack(gxe_u64 sign, int e, gxe_u64 q, bool rem) {
  int eb = e + 1023;
  if (eb >= 1) {
    gxe_u64 m = q >> 2;
    const bool round = (q >> 1) & 1u;
    const bool sticky = (q & 1u) || rem;
    m += (round && (sticky || (m & 1u))) ? 1u : 0u;
    if (m == (1ull << 53)) {
      m >>= 1;
      eb++;
    }
    if (eb >= 2047) return sign | GXE_INF;
    return sign | ((gxe_u64)eb << 52) | (m & GXE_FRAC);
  }
  const int sh = 3 - eb;  // >= 3
  if (sh > 55) return sign;
  gxe_u64 m = q >> sh;
  const bool round = (q >> (sh - 1)) & 1u;
  const bool sticky = (q & ((1ull << (sh - 1)) - 1u)) != 0 || rem;
  m += (round && (sticky || (m & 1u))) ? 1u : 0u;
  return sign | m;  // m == 2^52 encodes the smallest normal
}

// r ~ 2^116 / mb for a significand mb in [2^52, 2^53): an FP32 reciprocal of
// mb's top 24 bits refined by two Newton steps in 64-bit fixed point
// (r += r * (2^116 - mb*r) / 2^116).  Any r within a few units of the exact
// value serves gxe_div_finish, whose remainder correction absorbs the error.
GXE_FN gxe_u64 gxe_recip_fixed(gxe_u64 mb) {
  const unsigned d24 = (unsigned)(mb >> 29);                      // [2^23, 2^24)
  const float df = gxe_u2f((150u << 23) | (d24 & 0x7FFFFFu));    // == (float)d24
  const unsigned rb = gxe_f2u(gxe_rcp_approx(df));                // ~1/d24 in (2^-24, 2^-23]
  const int rexp = (int)((rb >> 23) & 0xFF) - 127;                // -24 or -23
  gxe_u64 r = (gxe_u64)((rb & 0x7FFFFFu) | 0x800000u) << (40 + (rexp + 24));  // * 2^(87+rexp-23)
  if (rexp >= -23) r = ~0ull;                                     // 1/d24 == 2^-23 -> clamp 2^64
#if GXE_ON_DEVICE
#pragma unroll
#endif
  for (int it = 0; it < 2; it++) {
    const gxe_u64 ph = gxe_umulhi(mb, r), pl = mb * r;
    const gxe_u64 t = (ph << 12) | (pl >> 52);   // (mb*r) >> 52, modulo 2^64
    const gxe_i64 err = -(gxe_i64)t;             // (2^116 - mb*r) / 2^52
    const gxe_u64 corr = gxe_umulhi(r, (gxe_u64)(err < 0 ? -err : err));
    r = err < 0 ? r - corr : r + corr;
  }
  return r;
}

// Quotient of significands ma, mb in [2^52, 2^53) with r = gxe_recip_fixed(mb):
// Q0 ~ floor(ma * 2^54 / mb) = (ma * r) >> 62, exact remainder correction, then
// rounding of the result with exponent e (before the ma < mb adjustment).
GXE_FN gxe_u64 gxe_div_finish(gxe_u64 sign, int e, gxe_u64 ma, gxe_u64 mb, gxe_u64 r) {
  if (ma < mb) {
    ma <<= 1;
    e -= 1;
  }
  gxe_u64 q = (gxe_umulhi(ma, r) << 2) | ((ma * r) >> 62);
  gxe_i64 rem = (gxe_i64)((ma << 54) - q * mb);  // exact: |rem| < 2^55
  if (rem < 0) { q--; rem += (gxe_i64)mb; }
  if (rem < 0) { q--; rem += (gxe_i64)mb; }
  if (rem >= (gxe_i64)mb) { q++; rem -= (gxe_i64)mb; }
  if (rem >= (gxe_i64)mb) { q++; rem -= (gxe_i64)mb; }
  return gxe_round_pack(sign, e, q, rem != 0);
}

// x / y, correctly rounded (round to nearest even), as bits.
GXE_FN gxe_u64 gxe_div(gxe_u64 a, gxe_u64 b) {
  const gxe_u64 sign = (a ^ b) & GXE_SIGN;
  int ea = (int)((a >> 52) & 0x7FF), eb = (int)((b >> 52) & 0x7FF);
  gxe_u64 fa = a & GXE_FRAC, fb = b & GXE_FRAC;
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u) {
    const bool nan_a = ea == 0x7FF && fa != 0, nan_b = eb == 0x7FF && fb != 0;
    if (nan_a || nan_b) return GXE_QNAN | (nan_a ? fa : fb) | (nan_a ? (a & GXE_SIGN) : (b & GXE_SIGN));
    const bool inf_a = ea == 0x7FF, inf_b = eb == 0x7FF;
    const bool zero_a = ea == 0 && fa == 0, zero_b = eb == 0 && fb == 0;
    if ((inf_a && inf_b) || (zero_a && zero_b)) return GXE_QNAN | GXE_SIGN;
    if (inf_a || zero_b) return sign | GXE_INF;
    if (inf_b || zero_a) return sign;
    if (ea == 0) {
      const int lz = gxe_clz(fa) - 11;
      fa <<= lz;
      ea = 1 - lz;
    }
    if (eb == 0) {
      const int lz = gxe_clz(fb) - 11;
      fb <<= lz;
      eb = 1 - lz;
    }
  }
  const gxe_u64 mb = fb | GXE_HIDDEN;
  return gxe_div_finish(sign, ea - eb, fa | GXE_HIDDEN, mb, gxe_recip_fixed(mb));
}

// x / y for a constant y that is normal and finite, with r =
// gxe_recip_fixed(y's significand) computed ahead: same bits as gxe_div(x, y).
GXE_FN gxe_u64 gxe_div_r(gxe_u64 a, gxe_u64 b, gxe_u64 r) {
  const gxe_u64 sign = (a ^ b) & GXE_SIGN;
  int ea = (int)((a >> 52) & 0x7FF);
  const int eb = (int)((b >> 52) & 0x7FF);
  gxe_u64 fa = a & GXE_FRAC;
  if ((unsigned)(ea - 1) >= 2046u) {
    if (ea == 0x7FF) return fa != 0 ? (GXE_QNAN | fa | (a & GXE_SIGN)) : (sign | GXE_INF);
    if (fa == 0) return sign;
    const int lz = gxe_clz(fa) - 11;
    fa <<= lz;
    ea = 1 - lz;
  }
  return gxe_div_finish(sign, ea - eb, fa | GXE_HIDDEN, (b & GXE_FRAC) | GXE_HIDDEN, r);
}

// x / b for a constant b (normal, finite) on the FMA unit, with y = RN(1/b)
// and bd = b: Markstein's correction step (Muller et al., "Handbook of
// Floating-Point Arithmetic", the theorem on the final correction of a
// quotient): q = RN(x * y) is within an ulp of x / b, so r = x - q * b is
// exact (one FMA), and RN(q + r * y) (one FMA) is the correctly rounded
// quotient, provided nothing underflows or overflows.  So the step is taken
// for x whose exponent field lies in [lo, hi] (chosen with b's exponent so
// that x, the quotient and r stay normal); a zero gives the signed zero;
// every other x (tiny, huge, subnormal, infinite, NaN) goes to gxe_div_r
// with rr = gxe_recip_fixed(b's significand).  Same bits as gxe_div(x, b).
GXE_FN double gxe_fma_(double a, double b, double c) {
#if GXE_ON_DEVICE
  return __fma_rn(a, b, c);
#else
  return __builtin_fma(a, b, c);
#endif
}
GXE_FN double gxe_mul_rn_(double a, double b) {
#if GXE_ON_DEVICE
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
GXE_FN gxe_u64 gxe_div_c(gxe_u64 a, gxe_u64 b, gxe_u64 rr, gxe_u64 ybits, int lo, int hi) {
  if ((a & ~GXE_SIGN) == 0) return (a ^ b) & GXE_SIGN;
  const int ea = (int)((a >> 52) & 0x7FF);
  if (ea < lo || ea > hi) return gxe_div_r(a, b, rr);
  double x, bd, y;
#if GXE_ON_DEVICE
  x = __longlong_as_double((long long)a);
  bd = __longlong_as_double((long long)b);
  y = __longlong_as_double((long long)ybits);
#else
  std::memcpy(&x, &a, 8);
  std::memcpy(&bd, &b, 8);
  std::memcpy(&y, &ybits, 8);
#endif
  const double q = gxe_mul_rn_(x, y);
  const double r = gxe_fma_(-q, bd, x);
  const double z = gxe_fma_(r, y, q);
  gxe_u64 zb;
#if GXE_ON_DEVICE
  zb = (gxe_u64)__double_as_longlong(z);
#else
  std::memcpy(&zb, &z, 8);
#endif
  return zb;
}
// the exponent-field window of gxe_div_c for a divisor whose exponent field is eb
GXE_FN void gxe_div_c_window(int eb, int* lo, int* hi) {
  // x, x / b and the remainder (about 2^-106 |x|) all normal and far from overflow
  *lo = 300 + (eb > 1023 ? eb - 1023 : 0);
  *hi = 1700 + (eb < 1023 ? eb - 1023 : 0);
}

// x + y, correctly rounded, as bits (guard / round / sticky alignment).
GXE_FN gxe_u64 gxe_add(gxe_u64 a, gxe_u64 b) {
  int ea = (int)((a >> 52) & 0x7FF), eb = (int)((b >> 52) & 0x7FF);
  if (ea == 0x7FF || eb == 0x7FF) {
    if (gxe_isnan_(a)) return a | (1ull << 51);
    if (gxe_isnan_(b)) return b | (1ull << 51);
    if (ea == 0x7FF && eb == 0x7FF) return ((a ^ b) & GXE_SIGN) ? (GXE_QNAN | GXE_SIGN) : a;  // inf - inf
    return ea == 0x7FF ? a : b;
  }
  gxe_u64 aa = a & ~GXE_SIGN, bb = b & ~GXE_SIGN;
  if (aa < bb) {  // |a| >= |b|
    gxe_u64 t = a; a = b; b = t;
    t = aa; aa = bb; bb = t;
    int te = ea; ea = eb; eb = te;
  }
  if (bb == 0) return aa == 0 ? (a & b & GXE_SIGN) : a;
  const int xa = ea ? ea : 1, xb = eb ? eb : 1;
  gxe_u64 ma = ((a & GXE_FRAC) | (ea ? GXE_HIDDEN : 0)) << 3;
  gxe_u64 mb = ((b & GXE_FRAC) | (eb ? GXE_HIDDEN : 0)) << 3;
  const int d = xa - xb;
  if (d >= 58) {
    mb = 1;
  } else if (d > 0) {
    const gxe_u64 lost = mb & ((1ull << d) - 1u);
    mb = (mb >> d) | (lost != 0 ? 1u : 0u);
  }
  const gxe_u64 sign = a & GXE_SIGN;
  gxe_u64 s;
  int e = xa;
  if (((a ^ b) & GXE_SIGN) == 0) {
    s = ma + mb;
    if (s >> 56) {
      s = (s >> 1) | (s & 1u);
      e++;
    }
  } else {
    s = ma - mb;
    if (s == 0) return 0;
    int lz = gxe_clz(s) - 8;
    if (lz > 0) {
      if (e - lz < 1) lz = e - 1;
      s <<= lz;
      e -= lz;
    }
  }
  gxe_u64 m = s >> 3;
  const unsigned low = (unsigned)(s & 7u);
  if (low > 4u || (low == 4u && (m & 1u))) m++;
  if (m >> 53) {
    m >>= 1;
    e++;
  }
  if (e >= 2047) return sign | GXE_INF;
  if (!(m & GXE_HIDDEN)) return sign | m;  // subnormal
  return sign | ((gxe_u64)e << 52) | (m & GXE_FRAC);
}

GXE_FN gxe_u64 gxe_sub(gxe_u64 a, gxe_u64 b) { return gxe_add(a, b ^ GXE_SIGN); }

// x * y, correctly rounded, as bits (106-bit product).
GXE_FN gxe_u64 gxe_mul(gxe_u64 a, gxe_u64 b) {
  const gxe_u64 sign = (a ^ b) & GXE_SIGN;
  int ea = (int)((a >> 52) & 0x7FF), eb = (int)((b >> 52) & 0x7FF);
  gxe_u64 fa = a & GXE_FRAC, fb = b & GXE_FRAC;
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u) {
    const bool nan_a = ea == 0x7FF && fa != 0, nan_b = eb == 0x7FF && fb != 0;
    if (nan_a) return a | (1ull << 51);
    if (nan_b) return b | (1ull << 51);
    const bool inf_a = ea == 0x7FF, inf_b = eb == 0x7FF;
    const bool zero_a = ea == 0 && fa == 0, zero_b = eb == 0 && fb == 0;
    if ((inf_a && zero_b) || (inf_b && zero_a)) return GXE_QNAN | GXE_SIGN;
    if (inf_a || inf_b) return sign | GXE_INF;
    if (zero_a || zero_b) return sign;
    if (ea == 0) {
      const int lz = gxe_clz(fa) - 11;
      fa <<= lz;
      ea = 1 - lz;
    }
    if (eb == 0) {
      const int lz = gxe_clz(fb) - 11;
      fb <<= lz;
      eb = 1 - lz;
    }
  }
  const gxe_u64 ma = fa | GXE_HIDDEN, mb = fb | GXE_HIDDEN;
  const gxe_u64 hi = gxe_umulhi(ma, mb), lo = ma * mb;  // product in [2^104, 2^106)
  if (hi >> 41) {  // >= 2^105
    return gxe_round_pack(sign, ea + eb - 2045, (hi << 13) | (lo >> 51), (lo & ((1ull << 51) - 1u)) != 0);
  }
  return gxe_round_pack(sign, ea + eb - 2046, (hi << 14) | (lo >> 50), (lo & ((1ull << 50) - 1u)) != 0);
}

// (double)(int64) with round-to-nearest-even, as bits.
GXE_FN gxe_u64 gxe_i2d(gxe_i64 v) {
  if (v == 0) return 0;
  const gxe_u64 sign = v < 0 ? GXE_SIGN : 0;
  gxe_u64 u = v < 0 ? 0ull - (gxe_u64)v : (gxe_u64)v;
  const int lz = gxe_clz(u);
  const int msb = 63 - lz;                     // exponent
  if (msb <= 52) return sign | ((gxe_u64)(msb + 1023) << 52) | ((u << (52 - msb)) & GXE_FRAC);
  const int sh = msb - 52;                     // 1..11
  gxe_u64 m = u >> sh;
  const bool round = (u >> (sh - 1)) & 1u;
  const bool sticky = (u & ((1ull << (sh - 1)) - 1u)) != 0;
  m += (round && (sticky || (m & 1u))) ? 1u : 0u;
  int eb = msb + 1023;
  if (m == (1ull << 53)) {
    m >>= 1;
    eb++;
  }
  return sign | ((gxe_u64)eb << 52) | (m & GXE_FRAC);
}

// (double)(float) (exact), as bits.
GXE_FN gxe_u64 gxe_f2d(unsigned f) {
  const gxe_u64 sign = (gxe_u64)(f >> 31) << 63;
  const unsigned ef = (f >> 23) & 0xFF, mf = f & 0x7FFFFFu;
  if (ef == 0xFF) return sign | GXE_INF | ((gxe_u64)mf << 29) | (mf ? (1ull << 51) : 0);
  if (ef == 0) {
    if (mf == 0) return sign;
    const int lz = gxe_clz((gxe_u64)mf) - 40;     // bring the leading 1 to bit 23
    return sign | ((gxe_u64)(1 - lz - 127 + 1023) << 52) | (((gxe_u64)(mf << lz) & 0x7FFFFFu) << 29);
  }
  return sign | ((gxe_u64)(ef - 127 + 1023) << 52) | ((gxe_u64)mf << 29);
}

// x / k for an integer divisor k: when 1 <= |k| <= n, Markstein's
// correction step (as gxe_div_c) on the FMA unit with y = RN(1/|k|) read from
// the table rcp (rcp[i] = RN(1 / (i + 1)) as bits) and the quotient's sign
// flipped for a negative k (x / -k = -(x / k) exactly); a zero x gives the
// signed zero.  Other k, and x outside the exponent window, take gxe_div.
// Same bits as gxe_div(x, (double)k).
GXE_FN gxe_u64 gxe_div_small(gxe_u64 a, gxe_i64 k, const gxe_u64* rcp, int n) {
  const gxe_u64 ak = k < 0 ? 0ull - (gxe_u64)k : (gxe_u64)k;
  const int ea = (int)((a >> 52) & 0x7FF);
  const bool zero = (a & ~GXE_SIGN) == 0;
  if (ak - 1ull >= (gxe_u64)n || (!zero && (ea < 310 || ea > 1700))) return gxe_div(a, gxe_i2d(k));
  gxe_u64 q;
  if (zero) {
    q = a & GXE_SIGN;
  } else {
#if GXE_ON_DEVICE
    const double y = __longlong_as_double((long long)__ldg(rcp + (ak - 1ull)));
    const double x = __longlong_as_double((long long)a);
    const double b = (double)(long long)ak;  // exact: |k| <= n
#else
    double y, x;
    std::memcpy(&y, rcp + (ak - 1ull), 8);
    std::memcpy(&x, &a, 8);
    const double b = (double)(long long)ak;
#endif
    const double q0 = gxe_mul_rn_(x, y);
    const double r = gxe_fma_(-q0, b, x);
    const double z = gxe_fma_(r, y, q0);
#if GXE_ON_DEVICE
    q = (gxe_u64)__double_as_longlong(z);
#else
    std::memcpy(&q, &z, 8);
#endif
  }
  return k < 0 ? q ^ GXE_SIGN : q;
}

// ---- division by a divisor whose reciprocal is known ahead ------------------
// Quotients by a literal or by a small integer need no FP64-pipe instruction
// at all.  That pipe issues one warp instruction every 16 clocks per SM, so the
// FMA-unit form above (a multiply and two FMAs, plus the conversions of integer
// operands) holds it for 48 to 80 clocks per 32 rows, where the form below
// takes about 30 integer instructions (64 lanes a clock on each of the ALU and
// IMAD pipes).  gxe_quot is that form: with the divisor's reciprocal rounded
// down to 64 bits (gxe_recip_floor), one 64 x 64 multiply-high gives the
// quotient's leading 64 bits, at most 4 units too low; the 11 bits below the
// significand decide the rounding except within 4 units of the midpoint, where
// the exact remainder's sign does.  (A quotient of two 53-bit significands is
// never itself a midpoint.)

// floor(2^116 / mb) for a significand mb in [2^52, 2^53); 2^64 - 1 for 2^52
GXE_FN gxe_u64 gxe_recip_floor(gxe_u64 mb) {
  // restoring long division: 2^63 / (mb / 2^53) bit by bit
  gxe_u64 rem = GXE_HIDDEN, q = 0;  // rem < mb unless mb == 2^52
  if (mb == GXE_HIDDEN) return ~0ull;
  for (int i = 0; i < 64; i++) {
    rem <<= 1;
    q <<= 1;
    if (rem >= mb) {
      rem -= mb;
      q |= 1ull;
    }
  }
  return q;
}

// A / (mb 2^11) for a normalised numerator A (top bit set, at most 53 leading
// bits used), r = gxe_recip_floor(mb); e is the quotient's biased exponent when
// A >= mb 2^11, and [e - 1, e] lies within the normal range (a carry out of
// the top exponent gives the infinity).
GXE_FN gxe_u64 gxe_quot(gxe_u64 sign, int e, gxe_u64 A, gxe_u64 mb, gxe_u64 r) {
  gxe_u64 h = gxe_umulhi(A, r);
  const int s = (gxe_i64)h < 0 ? 0 : 1;
  h <<= s;
  const gxe_u64 m = h >> 11;
  const unsigned low = (unsigned)h & 0x7FFu;
  unsigned up = low >> 10;
  if (low - 0x3FCu < 4u) up = (gxe_i64)((A << (42 + s)) - (2ull * m + 1ull) * mb) > 0 ? 1u : 0u;
  return sign | (((gxe_u64)(unsigned)(e - 1 - s) << 52) + m + up);
}

// x / y for the operands no fast path takes: subnormals, infinities, NaNs, zero
// divisors, quotients outside the normal range.  Same bits as gxe_div, whose
// reciprocal and products inlined here cost the whole kernel 8 to 17 registers; one
// quotient bit a step keeps the remainder, the divisor and the quotient alive and
// little code at every division (eleven bits a step: the deep plan 1404 us a call,
// 2^26 rows, 1373 with one).
GXE_FN gxe_u64 gxe_div_rare(gxe_u64 a, gxe_u64 b) {
  const gxe_u64 sign = (a ^ b) & GXE_SIGN;
  if (gxe_isnan_(a)) return GXE_QNAN | (a & (GXE_FRAC | GXE_SIGN));
  if (gxe_isnan_(b)) return GXE_QNAN | (b & (GXE_FRAC | GXE_SIGN));
  a &= ~GXE_SIGN;
  b &= ~GXE_SIGN;
  if (a == b && (a == 0 || a == GXE_INF)) return GXE_QNAN | GXE_SIGN;
  if (a == GXE_INF || b == 0) return sign | GXE_INF;
  if (a == 0 || b == GXE_INF) return sign;
  int e = (int)(a >> 52) - (int)(b >> 52);
  gxe_u64 m = a & GXE_FRAC, d = b & GXE_FRAC;
  if (a >> 52) m |= GXE_HIDDEN;
  else e++;
  if (b >> 52) d |= GXE_HIDDEN;
  else e--;
  while (!(m >> 52)) { m <<= 1; e--; }
  while (!(d >> 52)) { d <<= 1; e++; }
  if (m < d) { m <<= 1; e--; }
  gxe_u64 q = 0;  // 55 bits, the first one set
#if GXE_ON_DEVICE
#pragma unroll 1
#endif
  for (int i = 0; i < 55; i++) {
    q <<= 1;
    if (m >= d) { m -= d; q |= 1ull; }
    m <<= 1;
  }
  return gxe_round_pack(sign, e, q, m != 0);
}

// x / b for a literal b (normal, finite), r = gxe_recip_floor(b's significand)
GXE_FN gxe_u64 gxe_div_lit(gxe_u64 a, gxe_u64 b, gxe_u64 r) {
  const int ea = (int)((a >> 52) & 0x7FF), eb = (int)((b >> 52) & 0x7FF);
  // x normal and the quotient's exponent (or one less) normal too
  const int lo = eb > 1022 ? eb - 1021 : 1, hi = eb < 1023 ? eb + 1023 : 2046;
  if ((unsigned)(ea - lo) > (unsigned)(hi - lo)) return (a << 1) == 0 ? (a ^ b) & GXE_SIGN : gxe_div_rare(a, b);
  const gxe_u64 A = ((a & GXE_FRAC) | GXE_HIDDEN) << 11;
  return gxe_quot((a ^ b) & GXE_SIGN, ea - eb + 1023, A, (b & GXE_FRAC) | GXE_HIDDEN, r);
}

// A 64-bit integer with its top bit set, rounded to its leading 53 bits as the
// conversion to binary64 rounds it (nearest, ties to even); true on a carry,
// which leaves 2^63 and one more in the exponent.
GXE_FN bool gxe_round53(gxe_u64* A) {
  if ((*A & 0x7FFull) == 0) return false;
  const gxe_u64 t = *A + 0x3FFull + ((*A >> 11) & 1ull);
  const bool carry = t < *A;
  *A = carry ? 1ull << 63 : t & ~0x7FFull;
  return carry;
}

// (double)x / b for a literal b and an integer x: as gxe_div_lit, without the
// conversion
GXE_FN gxe_u64 gxe_divi_lit(gxe_i64 x, gxe_u64 b, gxe_u64 r) {
  const int eb = (int)((b >> 52) & 0x7FF);
  const gxe_u64 u = x < 0 ? 0ull - (gxe_u64)x : (gxe_u64)x;
  const gxe_u64 sign = ((gxe_u64)x ^ b) & GXE_SIGN;
  const int lz = gxe_clz(u);
  gxe_u64 A = u << (lz & 63);
  int e = 1023 + 63 - lz - eb + 1023;
  if (u == 0) return sign;
  if (gxe_round53(&A)) e++;
  if ((unsigned)(e - 2) > 2044u) return gxe_div_rare(gxe_i2d(x), b);
  return gxe_quot(sign, e, A, (b & GXE_FRAC) | GXE_HIDDEN, r);
}

// A / (mb 2^11) as gxe_quot, without a reciprocal: a first quotient bit, then
// three digits of 20 bits, each estimated in binary32 from the leading 24 bits of
// the remainder and the divisor, off by at most one, and corrected by the exact
// remainder.  It keeps few values alive: gxe_recip_fixed in its place costs the
// order-line plan 10 registers of 68.
GXE_FN gxe_u64 gxe_quot_steps(gxe_u64 sign, int e, gxe_u64 A, gxe_u64 mb) {
  gxe_u64 m = A >> 11;
  if (m < mb) { m <<= 1; e--; }
  m -= mb;
  gxe_u64 q = 1;
  const float inv = 1048576.0f * gxe_rcp_approx((float)(unsigned)(mb >> 29));
#if GXE_ON_DEVICE
#pragma unroll 1
#endif
  for (int i = 0; i < 3; i++) {  // m < mb < 2^53
    unsigned digit = (unsigned)((float)(unsigned)(m >> 29) * inv);
    m = (m << 20) - (gxe_u64)digit * mb;  // in [-mb, 2 mb)
    if ((gxe_i64)m < 0) { digit--; m += mb; }
    else if (m >= mb) { digit++; m -= mb; }
    q = (q << 20) + digit;
  }
  return sign | (((gxe_u64)(unsigned)(e - 1) << 52) + (q >> 8) + ((q >> 7) & 1ull));
}

// A / (the double of |k| = uk, times 2^11) for an integer divisor, e the biased
// exponent of the quotient by one: the table's reciprocal for uk <= n, else by
// steps.  Call us, 2^25 rows, doubles by integers up to 10^6 / integers by them /
// 62-bit integers by 7.0: 433 / 437 / 287 with gxe_div for what no table serves and
// the FMA unit for the rest, 516 / 492 / 381 with gxe_div_rare, 320 / 340 / 164 now.
GXE_FN gxe_u64 gxe_quot_k(gxe_u64 sign, int e, gxe_u64 A, gxe_u64 uk, const gxe_u64* rcp, int n) {
  const int lz = gxe_clz(uk);
  gxe_u64 m = uk << (lz & 63);
  e += lz - 63;
  if (uk - 1ull < (gxe_u64)n) {
#if GXE_ON_DEVICE
    const gxe_u64 r = __ldg(rcp + (uk - 1ull));
#else
    const gxe_u64 r = rcp[uk - 1ull];
#endif
    return gxe_quot(sign, e, A, m >> 11, r);
  }
  if (gxe_round53(&m)) e--;
  return gxe_quot_steps(sign, e, A, m >> 11);
}

// x / k for an integer k: rcp[i] = gxe_recip_floor(significand of i + 1), for
// 1 <= |k| <= n.  Zeros of either side are answered here: a filter's idle lanes
// divide 0 by 0, and must not draw their warp into the rare path.
GXE_FN gxe_u64 gxe_div_k(gxe_u64 a, gxe_i64 k, const gxe_u64* rcp, int n) {
  const gxe_u64 uk = k < 0 ? 0ull - (gxe_u64)k : (gxe_u64)k;
  const int ea = (int)((a >> 52) & 0x7FF);
  // |k| <= 2^63: the quotient's exponent stays normal for ea in [66, 2046]
  if (k == 0 || (unsigned)(ea - 66) > 1980u) {
    const bool zero = (a << 1) == 0;
    if (k == 0 && !gxe_isnan_(a)) return zero ? GXE_QNAN | GXE_SIGN : (a & GXE_SIGN) | GXE_INF;
    if (zero) return a ^ ((gxe_u64)k & GXE_SIGN);
    return gxe_div_rare(a, gxe_i2d(k));
  }
  return gxe_quot_k((a ^ (gxe_u64)k) & GXE_SIGN, ea, ((a & GXE_FRAC) | GXE_HIDDEN) << 11, uk, rcp, n);
}

// (double)x / (double)k for integers: as gxe_div_k, without the conversions
GXE_FN gxe_u64 gxe_divi_k(gxe_i64 x, gxe_i64 k, const gxe_u64* rcp, int n) {
  const gxe_u64 uk = k < 0 ? 0ull - (gxe_u64)k : (gxe_u64)k;
  const gxe_u64 u = x < 0 ? 0ull - (gxe_u64)x : (gxe_u64)x;
  if (k == 0) return u == 0 ? GXE_QNAN | GXE_SIGN : ((gxe_u64)x & GXE_SIGN) | GXE_INF;
  if (u == 0) return (gxe_u64)k & GXE_SIGN;
  int lx = gxe_clz(u);
  gxe_u64 A = u << lx;
  if (gxe_round53(&A)) lx--;
  return gxe_quot_k(((gxe_u64)x ^ (gxe_u64)k) & GXE_SIGN, 1023 + 63 - lx, A, uk, rcp, n);
}

// (double)v of an integer known to fit 32 bits: one shift instead of the
// 64-bit normalisation and rounding of gxe_i2d
GXE_FN gxe_u64 gxe_i2d32(int v) {
  const unsigned u = v < 0 ? 0u - (unsigned)v : (unsigned)v;
#if GXE_ON_DEVICE
  const int lz = __clz((int)u);
#else
  const int lz = u ? __builtin_clz(u) : 32;
#endif
  const unsigned m = u << (lz & 31);
  const unsigned hi = ((unsigned)(1023 + 30 - lz) << 20) + (m >> 11) + ((unsigned)v & 0x80000000u);
  return u == 0 ? 0ull : ((gxe_u64)hi << 32) | (gxe_u64)(m << 21);
}

// round half away from zero (exact), as bits
GXE_FN gxe_u64 gxe_round(gxe_u64 a) {
  const int e = (int)((a >> 52) & 0x7FF) - 1023;
  if (e >= 52) return (a & ~GXE_SIGN) > GXE_INF ? (a | (1ull << 51)) : a;  // integral, inf, nan
  if (e < 0) return (a & GXE_SIGN) | (e == -1 ? 0x3FF0000000000000ull : 0ull);
  a += (GXE_HIDDEN >> 1) >> e;  // half a unit, in magnitude
  return a & ~(GXE_FRAC >> e);
}

// comparisons with a literal c (not NaN): ranges of the other operand's bits,
// two 64-bit integer compares each
GXE_FN bool gxe_ltc(gxe_u64 x, gxe_u64 c) {  // x < c
  if ((c << 1) == 0) return x > GXE_SIGN && x <= (GXE_SIGN | GXE_INF);
  if (c & GXE_SIGN) return x > c && x <= (GXE_SIGN | GXE_INF);
  return (gxe_i64)x < (gxe_i64)c && x <= (GXE_SIGN | GXE_INF);
}
GXE_FN bool gxe_gtc(gxe_u64 x, gxe_u64 c) {  // x > c
  if ((c << 1) == 0) return x - 1ull < GXE_INF;
  if (c & GXE_SIGN) return x < c && (x <= GXE_INF || x >= GXE_SIGN);
  return (gxe_i64)x > (gxe_i64)c && (gxe_i64)x <= (gxe_i64)GXE_INF;
}
GXE_FN bool gxe_eqc(gxe_u64 x, gxe_u64 c) { return (c << 1) == 0 ? (x << 1) == 0 : x == c; }
GXE_FN bool gxe_lec(gxe_u64 x, gxe_u64 c) {  // x <= c
  if ((c << 1) == 0) return x == 0 || (x >= GXE_SIGN && x <= (GXE_SIGN | GXE_INF));
  if (c & GXE_SIGN) return x >= c && x <= (GXE_SIGN | GXE_INF);
  return (gxe_i64)x <= (gxe_i64)c && x <= (GXE_SIGN | GXE_INF);
}
GXE_FN bool gxe_gec(gxe_u64 x, gxe_u64 c) {  // x >= c
  if ((c << 1) == 0) return x <= GXE_INF || x == GXE_SIGN;
  if (c & GXE_SIGN) return x <= c && (x <= GXE_INF || x >= GXE_SIGN);
  return (gxe_i64)x >= (gxe_i64)c && (gxe_i64)x <= (gxe_i64)GXE_INF;
}

GXE_FN bool gxe_isnan(gxe_u64 a) { return (a & ~GXE_SIGN) > GXE_INF; }

// total order key for non-NaN values with -0 == +0
GXE_FN gxe_u64 gxe_key(gxe_u64 a) {
  if ((a << 1) == 0) a = 0;
  return (a & GXE_SIGN) ? ~a : (a | GXE_SIGN);
}
GXE_FN bool gxe_lt(gxe_u64 a, gxe_u64 b) { return !gxe_isnan(a) && !gxe_isnan(b) && gxe_key(a) < gxe_key(b); }
GXE_FN bool gxe_le(gxe_u64 a, gxe_u64 b) { return !gxe_isnan(a) && !gxe_isnan(b) && gxe_key(a) <= gxe_key(b); }
GXE_FN bool gxe_eq(gxe_u64 a, gxe_u64 b) { return !gxe_isnan(a) && !gxe_isnan(b) && gxe_key(a) == gxe_key(b); }
GXE_FN bool gxe_nz(gxe_u64 a) { return (a << 1) != 0; }  // != 0.0 (NaN counts as nonzero)

// floor / ceil (exact), as bits
GXE_FN gxe_u64 gxe_floor(gxe_u64 a) {
  const int e = (int)((a >> 52) & 0x7FF) - 1023;
  if (e >= 52) return gxe_isnan(a) ? (a | (1ull << 51)) : a;  // integral, inf, nan
  if (e < 0) {
    if ((a << 1) == 0) return a;                                 // +-0
    return (a & GXE_SIGN) ? 0xBFF0000000000000ull : 0;           // -1 or +0
  }
  const gxe_u64 fmask = GXE_FRAC >> e;
  if ((a & fmask) == 0) return a;
  if (a & GXE_SIGN) a += (GXE_HIDDEN >> e);  // round toward -inf in magnitude
  return a & ~fmask;
}
GXE_FN gxe_u64 gxe_ceil(gxe_u64 a) {
  const int e = (int)((a >> 52) & 0x7FF) - 1023;
  if (e >= 52) return gxe_isnan(a) ? (a | (1ull << 51)) : a;
  if (e < 0) {
    if ((a << 1) == 0) return a;
    return (a & GXE_SIGN) ? GXE_SIGN : 0x3FF0000000000000ull;    // -0 or +1
  }
  const gxe_u64 fmask = GXE_FRAC >> e;
  if ((a & fmask) == 0) return a;
  if (!(a & GXE_SIGN)) a += (GXE_HIDDEN >> e);
  return a & ~fmask;
}

// static_cast<int64_t>(double) as the GPU does it: truncate, saturate, NaN -> 0
GXE_FN gxe_i64 gxe_d2ll(gxe_u64 a) {
  if (gxe_isnan(a)) return 0;
  const int e = (int)((a >> 52) & 0x7FF) - 1023;
  const bool neg = (a & GXE_SIGN) != 0;
  if (e < 0) return 0;
  if (e >= 63) return neg ? (gxe_i64)GXE_SIGN : 0x7FFFFFFFFFFFFFFFll;
  const gxe_u64 m = (a & GXE_FRAC) | GXE_HIDDEN;
  const gxe_u64 mag = e >= 52 ? (m << (e - 52)) : (m >> (52 - e));
  return neg ? -(gxe_i64)mag : (gxe_i64)mag;
}
