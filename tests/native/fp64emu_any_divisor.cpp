// Checks the known-divisor divisions of fp64emu.cuh against gxe_div bit for bit,
// NaNs' signs and payloads included, over the operands that no reciprocal table
// and no 53-bit numerator serves.
// Usage: fp64emu_any_divisor <cases> <seed>
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
static gxe_u64 any() {
  const gxe_u64 r = rng(), f = r & (GXE_SIGN | GXE_FRAC);
  switch (rng() % 6) {
    case 0: return f | GXE_INF;                                      // NaNs (rarely an infinity)
    case 1: return f >> (rng() % 50);                                // subnormals, tiny, zeros
    case 2: return (r & GXE_SIGN) | (rng() % 2 ? GXE_INF : 0);
    case 3: return gxe_i2d((gxe_i64)(r >> (rng() % 64)));
    default: return r;
  }
}

int main(int argc, char** argv) {
  const long long cases = argc > 1 ? atoll(argv[1]) : 1000000;
  rng.seed(argc > 2 ? strtoull(argv[2], nullptr, 10) : 1);
  const int n = 1024;
  static gxe_u64 table[1024];
  for (int i = 0; i < n; i++) table[i] = gxe_recip_floor((gxe_i2d(i + 1) & GXE_FRAC) | GXE_HIDDEN);
  for (long long i = 0; i < cases; i++) {
    const gxe_u64 a = any(), b = any();
    const gxe_i64 k = (gxe_i64)rng() >> (rng() % 64), x = (gxe_i64)rng() >> (rng() % 64);
    const gxe_u64 kb = gxe_i2d(k), xb = gxe_i2d(x);
    check(gxe_div_rare(a, b), gxe_div(a, b), "any", a, b);
    check(gxe_div_rare(xb, kb), gxe_div(xb, kb), "any, integers", xb, kb);
    check(gxe_div_k(a, k, table, n), gxe_div(a, kb), "double / integer", a, kb);
    check(gxe_divi_k(x, k, table, n), gxe_div(xb, kb), "integer / integer", xb, kb);
    const int eb = (int)((b >> 52) & 0x7FF);
    if (eb < 1 || eb > 2046) continue;
    const gxe_u64 r = gxe_recip_floor((b & GXE_FRAC) | GXE_HIDDEN);
    check(gxe_div_lit(a, b, r), gxe_div(a, b), "double / literal", a, b);
    check(gxe_divi_lit(x, b, r), gxe_div(xb, b), "integer / literal", xb, b);
  }
  printf("cases=%lld mismatches=%lld\n", cases, bad);
  return bad ? 1 : 0;
}
