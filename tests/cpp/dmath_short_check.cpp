// The short forms of the integer double log / exp (gr_dmath.h) against the
// long ones, bit for bit, over the ranges the samplers use and random bits.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "gr_dmath.h"

using namespace gr;

static long bad = 0, total = 0;
static void check_log(double x) {
  ++total;
  bad += grd_bits(grd_log(x)) != grd_bits(grd_log_long(x));
}
static void check_exp(double x) {
  ++total;
  bad += grd_bits(grd_exp(x)) != grd_bits(grd_exp_long(x));
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 400000;
  std::mt19937_64 g(17);
  for (long i = 0; i < n; ++i) {
    const uint64_t r = g();
    const double u = (double)(r >> 11) * 0x1p-53, v = (double)(g() >> 11) * 0x1p-53;
    check_log(1.0 - (double)(r >> 12) * 0x1p-52);
    check_log((double)(r >> 12) * 0x1p-52 + 0x1p-55);
    check_log(u * v);
    check_log(grd_double(r & 0x7fffffffffffffffull));
    check_log(1.0 + std::ldexp(u - 0.5, -(int)(g() % 50)));
    check_log(-std::log(u + 1e-300));
    check_exp((v - 0.5) * 1400);
    check_exp(-std::ldexp(v, (int)(g() % 45) - 35));
    check_exp(std::ldexp(v, (int)(g() % 45) - 35));
    check_exp(2 * std::log(u + 1e-17));
    // near multiples of ln2 / 64, where the reduction changes its step
    check_exp((double)((int)(g() % 130000) - 65000) * 0.01083042469624914 / 2 + (v - 0.5) * 1e-9);
    check_exp(grd_double(g()));
  }
  std::printf("mismatches %ld of %ld\n", bad, total);
  return bad != 0;
}
