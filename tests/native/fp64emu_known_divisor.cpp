// Checks the known-divisor and literal-operand routines of fp64emu.cuh against
// the host CPU's IEEE-754 arithmetic, bit for bit (any NaN matches any NaN).
// Usage: fp64emu_known_divisor <cases> <seed>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "fp64emu.cuh"

static uint64_t bits(double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; }
static double dbl(uint64_t u) { double d; std::memcpy(&d, &u, 8); return d; }
static long long bad = 0;
static void check(uint64_t got, double want, const char* what) {
  if (std::isnan(want) ? gxe_isnan(got) : got == bits(want)) return;
  if (bad++ < 10) printf("%s: got %016llx want %016llx\n", what, (unsigned long long)got, (unsigned long long)bits(want));
}

static std::mt19937_64 rng;
static double any() {  // uniform bits, subnormals, tiny, huge, specials, integers, moderate, near one
  static const double S[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 10.0, 1000.0, 0.5, -0.5,
                             0.49999999999999994, 1.7976931348623157e308, 2.2250738585072014e-308, 4.9e-324};
  const uint64_t r = rng(), f = r & 0x800FFFFFFFFFFFFFull;
  switch (rng() % 8) {
    case 0: return dbl(r);
    case 1: return dbl(f);
    case 2: return dbl(f | ((uint64_t)(1 + rng() % 60) << 52));
    case 3: return dbl(f | ((uint64_t)(2046 - rng() % 60) << 52));
    case 4: return S[r % (sizeof S / sizeof S[0])];
    case 5: return (double)(int64_t)(r >> (rng() % 64));
    case 6: return dbl(f | ((uint64_t)(991 + rng() % 64) << 52));
    default: return dbl(0x3FF0000000000000ull | (r & 0xFFFFF));
  }
}
static uint64_t sig53(double d) { return (bits(d) & GXE_FRAC) | GXE_HIDDEN; }

int main(int argc, char** argv) {
  const long long cases = argc > 1 ? atoll(argv[1]) : 1000000;
  rng.seed(argc > 2 ? strtoull(argv[2], nullptr, 10) : 1);
  const int n = 1024;
  static gxe_u64 table[1024];
  for (int i = 0; i < n; i++) table[i] = gxe_recip_floor(sig53((double)(i + 1)));
  for (long long i = 0; i < cases; i++) {
    const double a = any(), b = any();
    const int eb = (int)((bits(b) >> 52) & 0x7FF);
    const int64_t x = (int64_t)rng() >> (rng() % 64);
    const int64_t k = rng() % 8 ? (int64_t)(rng() % 2300) - 1150 : (int64_t)rng() >> (rng() % 64);
    if (eb >= 1 && eb <= 2046) {
      const uint64_t r = gxe_recip_floor(sig53(b));
      check(gxe_div_lit(bits(a), bits(b), r), a / b, "double / literal");
      check(gxe_divi_lit(x, bits(b), r), (double)x / b, "integer / literal");
    }
    check(gxe_div_rare(bits(a), bits(b)), a / b, "rare");
    check(gxe_div_k(bits(a), k, table, n), a / (double)k, "double / integer");
    check(gxe_divi_k(x, k, table, n), (double)x / (double)k, "integer / integer");
    // dividends whose quotient lies next to a midpoint of two doubles
    const uint64_t m = sig53(dbl(rng()));
    const double by[2] = {(double)(1 + rng() % n), dbl((rng() & GXE_FRAC) | 0x3FF0000000000000ull)};
    for (int w = 0; w < 2; w++) {
      const uint64_t r = gxe_recip_floor(sig53(by[w]));
      uint64_t near = (uint64_t)(((unsigned __int128)(2 * m + 1) * sig53(by[w])) >> 53);
      while (near >> 53) near >>= 1;
      for (int d = -1; d <= 1; d++) {
        const double y = (double)(near + d);
        check(gxe_div_lit(bits(y), bits(by[w]), r), y / by[w], "near a midpoint, literal");
        if (w == 0) {
          check(gxe_div_k(bits(y), (int64_t)by[0], table, n), y / by[0], "near a midpoint, integer");
          check(gxe_divi_k((int64_t)y, (int64_t)by[0], table, n), y / by[0], "near a midpoint, integers");
        }
      }
    }
    const int32_t v = i ? (int32_t)rng() >> (rng() % 32) : INT32_MIN;
    check(gxe_i2d32(v), (double)v, "32-bit conversion");
    check(gxe_round(bits(a)), std::round(a), "round");
    const double h = std::floor(a) + 0.5;
    check(gxe_round(bits(h)), std::round(h), "round of a half");
    if (std::isnan(b)) continue;
    for (double c : {a, b, -b}) {
      const uint64_t p = bits(c), q = bits(b);
      if (gxe_ltc(p, q) != (c < b) || gxe_gtc(p, q) != (c > b) || gxe_lec(p, q) != (c <= b) ||
          gxe_gec(p, q) != (c >= b) || gxe_eqc(p, q) != (c == b))
        if (bad++ < 10) printf("compare %.17g %.17g\n", c, b);
    }
  }
  printf("cases=%lld mismatches=%lld\n", cases, bad);
  return bad ? 1 : 0;
}
