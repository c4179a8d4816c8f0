// gr_fp64i.h against the IEEE operations: square root, quotient, uniforms,
// scaled uniforms and sine / cosine, over random operands, operands next to the
// places where a rounding or a comparison turns, and operands outside the fast
// forms' range.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "gr_fp64i.h"

using namespace gr;

static uint64_t st = 0x9e3779b97f4a7c15ull;
static uint64_t rnd() {  // splitmix64
  uint64_t z = (st += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
static long bad = 0, total = 0;
static void same(const char* what, double got, double want, double a, double b) {
  ++total;
  if (grd_bits(got) != grd_bits(want) && !(got != got && want != want) && ++bad < 20)
    printf("%s(%a, %a): %a, not %a\n", what, a, b, got, want);
}
static double sparse(uint64_t r) {  // a significand of few ones or few zeros
  const uint64_t m = (1ull << (r % 53)) ^ (1ull << (r / 53 % 53)) ^ ((r >> 40) & 1 ? 0xfffffffffffffull : 0);
  return grd_double((m & 0xfffffffffffffull) | ((1023ull + r / 2809 % 3) << 52));
}
static void trig(double x) {
  double s, c, ls, lc;
  sincos_long(x, &ls, &lc);
  sincos_d<4>(x, s, c);
  same("sin4", s, ls, x, 0);
  same("cos4", c, lc, x, 0);
  sincos_d<2>(x, s, c);
  same("sin2", s, ls, x, 0);
  same("cos2", c, lc, x, 0);
  sincos_d<1>(x, s, c);
  same("sin1", s, ls, x, 0);
  same("cos1", c, lc, x, 0);
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 3000000;
  const double pi = 3.1415926535897932, two_pi = 2 * 3.1415926535897932;
  for (long i = 0; i < n; ++i) {
    const uint64_t r = rnd(), q = rnd();
    const double a = i & 1 ? sparse(r) : grd_double((r & 0xfffffffffffffull) | ((r >> 52) % 1200 + 423) << 52);
    const double b = i & 2 ? sparse(q) : grd_double((q & 0xfffffffffffffull) | ((q >> 52) % 1200 + 423) << 52);
    same("sqrt", sqrt_d(a), sqrt(a), a, 0);
    const double sq = b * b;  // next to a perfect square
    same("sqrt", sqrt_d(sq), sqrt(sq), sq, 0);
    same("sqrt", sqrt_d(nextafter(sq, 0)), sqrt(nextafter(sq, 0)), sq, 0);
    same("sqrt", sqrt_d(nextafter(sq, 1e308)), sqrt(nextafter(sq, 1e308)), sq, 0);
    same("div", div_d(a, b), a / b, a, b);
    same("div", div_d(-a, b), -a / b, -a, b);
    const double ab = a * b;  // next to an exact quotient
    same("div", div_d(ab, b), ab / b, ab, b);
    const uint64_t x = i % 3 == 0 ? r : r & ((1ull << (r >> 58)) - 1);
    const double u = grd_double((x & 0xfffffffffffffull) | 0x3ff0000000000000ull) - 1.0;
    same("ur_nz", ur_nz_int(x), u + 2.220446049250313e-16 / 8, u, 0);
    const uint64_t F = x & 0xfffffffffffffull;
    same("2 pi u", scaled52(F, sc53(0x401921fb54442d18ull), 1025), two_pi * u, u, 0);
    same("pi u", scaled52(F, sc53(0x400921fb54442d18ull), 1024), pi * u, u, 0);
    trig(two_pi * u);
    trig(pi * u);
    trig(pi * (u - 0.5));
  }
  const uint64_t turn[5] = {0x3fe921fb54442d27ull, 0x4002d97c7f3321ddull, 0x400f6a7a29553870ull, 0x4015fdbbe9bba782ull,
                            0x401c463abeccb2cbull};
  for (uint64_t t : turn)
    for (int j = -2000; j <= 2000; ++j) trig(grd_double(t + (int64_t)j)), trig(-grd_double(t + (int64_t)j));
  for (double t : {pi / 2, pi, 3 * pi / 2, two_pi})
    for (int j = -2000; j <= 2000; ++j) trig(grd_double(grd_bits(t) + (int64_t)j));
  const double odd[] = {0.0, -0.0, 5e-324, 2.2250738585072014e-308, 1e-300, 1e300, 1.7976931348623157e308, INFINITY, -INFINITY,
                        NAN, 1.0, -1.0, 2.0, 4.0, 0.25, 1e-160, 1e160};
  for (double a : odd) {
    same("sqrt", sqrt_d(a), sqrt(a), a, 0);
    if (!(fabs(a) > 1e6)) trig(a);
    for (double b : odd) same("div", div_d(a, b), a / b, a, b);
  }
  printf("mismatches %ld of %ld\n", bad, total);
  return bad != 0;
}
