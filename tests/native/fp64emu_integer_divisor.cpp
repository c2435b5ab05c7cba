// Checks quotients by integers of any size, those next to midpoints of two
// doubles included, and by significands of every kind (gxe_quot_steps) against
// gxe_div bit for bit.
// Usage: fp64emu_integer_divisor <cases> <seed>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "fp64emu.cuh"

static std::mt19937_64 rng;
static long long bad = 0;
static void check(gxe_u64 got, gxe_u64 want, const char* what, gxe_u64 a, gxe_u64 b) {
  if (got == want || bad++ >= 10) return;
  printf("%s %016llx %016llx: got %016llx want %016llx\n", what, a, b, got, want);
}

int main(int argc, char** argv) {
  const long long cases = argc > 1 ? atoll(argv[1]) : 1000000;
  rng.seed(argc > 2 ? strtoull(argv[2], nullptr, 10) : 1);
  const int n = 1024;
  static gxe_u64 table[1024];
  for (int i = 0; i < n; i++) table[i] = gxe_recip_floor((gxe_i2d(i + 1) & GXE_FRAC) | GXE_HIDDEN);
  for (long long i = 0; i < cases; i++) {
    // significands: any, close to either end, few bits set
    gxe_u64 mb = rng() & GXE_FRAC;
    switch (rng() % 4) {
      case 0: mb >>= rng() % 53; break;
      case 1: mb = GXE_FRAC - (mb >> (rng() % 53)); break;
      case 2: mb = (mb << (rng() % 53)) & GXE_FRAC; break;
      default: break;
    }
    mb |= GXE_HIDDEN;
    gxe_u64 num = rng() % 3 ? rng() : mb + rng() % 5 - 2;  // any, or next to the divisor's
    num = (num & GXE_FRAC) | GXE_HIDDEN;
    const gxe_u64 one = 1023ull << 52;
    check(gxe_quot_steps(0, 1023, num << 11, mb), gxe_div((num & GXE_FRAC) | one, (mb & GXE_FRAC) | one), "steps", num, mb);

    gxe_i64 k = (gxe_i64)(rng() >> (1 + rng() % 63));
    if (rng() % 4 == 0) k = (gxe_i64)(mb << (rng() % 11) | (rng() & ((1u << (rng() % 11)) - 1u)));
    if (rng() % 16 == 0) k = (gxe_i64)(~0ull << 63) + (gxe_i64)(rng() % 3);
    if (rng() % 2) k = (gxe_i64)(0ull - (gxe_u64)k);
    const gxe_u64 kb = gxe_i2d(k);
    // a dividend next to (m + 1/2) |k|
    const gxe_u64 sk = (kb & GXE_FRAC) | GXE_HIDDEN, m = (rng() & GXE_FRAC) | GXE_HIDDEN;
    const unsigned __int128 p = (unsigned __int128)(2 * m + 1) * sk;  // 106 or 107 bits
    const int sh = (p >> 106) ? 54 : 53;
    const gxe_u64 a = (((gxe_u64)(p >> sh) + rng() % 3 - 1) & GXE_FRAC) | ((gxe_u64)(60 + rng() % 1987) << 52) | (rng() & GXE_SIGN);
    check(gxe_div_k(a, k, table, n), gxe_div(a, kb), "double / integer", a, k);
    const gxe_i64 x = rng() % 2 ? (gxe_i64)(rng() >> (rng() % 64)) : (gxe_i64)(~0ull >> (rng() % 12)) - (gxe_i64)(rng() % 2000);
    check(gxe_divi_k(x, k, table, n), gxe_div(gxe_i2d(x), kb), "integer / integer", x, k);
    const gxe_u64 lit = ((rng() & GXE_FRAC) | ((gxe_u64)(1 + rng() % 2046) << 52)) ^ (rng() & GXE_SIGN);
    check(gxe_divi_lit(x, lit, gxe_recip_floor((lit & GXE_FRAC) | GXE_HIDDEN)), gxe_div(gxe_i2d(x), lit), "integer / literal", x, lit);
  }
  printf("cases=%lld mismatches=%lld\n", cases, bad);
  return bad ? 1 : 0;
}
