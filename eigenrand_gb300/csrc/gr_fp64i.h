// IEEE double operations in integer arithmetic, bit for bit.
//
// An SM issues two FP64 thread-operations per clock and 64 to 128 integer
// ones, and the double samplers are chains of 20 to 50 FP64 operations: those
// chains bound them, with the integer pipes idle.  The operations here round
// as the IEEE ones do (to nearest, ties to even) from exact integer products
// and remainders, for the operands the samplers have (positive normal numbers,
// known ranges); any other operand goes to the FP64 instruction.  Which steps
// of a chain are done here and which stay on the FP64 pipe is a matter of
// keeping both busy (noted at the functions).
//
// Square root and quotient: a single-precision estimate of the reciprocal
// (root), one Newton step in 32-bit integers, one step with the exact residual,
// and the last unit from the sign of the exact remainder.
//
// Compiles for the host as well; a CPU test compares every function with the
// IEEE operation it stands for.
#pragma once
#include <math.h>

#include "gr_dmath.h"
#include "gr_exact.h"

namespace gr {

GRD_HD uint32_t grf_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
GRD_HD float grf_float(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}
// 1 / x and 1 / sqrt(x) to within 2 units of 2^-24, 1 <= x < 4 (the host adds
// GRF_HOST_ULPS units, for the test)
#ifndef GRF_HOST_ULPS
#define GRF_HOST_ULPS 0
#endif
GRD_HD float grf_rcp(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return grf_float(grf_bits(1.0f / x) + (uint32_t)(GRF_HOST_ULPS));
#endif
}
GRD_HD float grf_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return grf_float(grf_bits(1.0f / sqrtf(x)) + (uint32_t)(GRF_HOST_ULPS));
#endif
}
// such an estimate, held to [1/2, 1 - 2^-24], as a 32-bit fraction
GRD_HD uint32_t grf_fraction(float y) {
  uint32_t b = grf_bits(y);
  b = b < 0x3f000000u ? 0x3f000000u : (b > 0x3f7fffffu ? 0x3f7fffffu : b);
  return (b << 8) | 0x80000000u;
}

// the 53-bit significand of a constant
constexpr uint64_t kSigOnes = 0xfffffffffffffull, kSigLead = 0x10000000000000ull;
#define sc53(bits) (((bits) & kSigOnes) | kSigLead)

// The product of two 53-bit significands rounded to 53 bits: m 2^(52 + k).
// m may be 2^53, which carries into the exponent when the caller adds it there.
GRD_HD uint64_t mul53(uint64_t a, uint64_t b, int& k) {
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  const uint64_t p0 = grd_wide(a0, b0);
  const uint64_t p1 = grd_wide(a1, b0) + (p0 >> 32);  // the high halves have 21 bits: no carry out
  const uint64_t p2 = grd_wide(a0, b1) + p1;
  const uint64_t p3 = grd_wide(a1, b1) + (p2 >> 32);  // the product from bit 64: bit 41 or 40 leads
  const uint32_t c = (uint32_t)p2;
  k = (int)(p3 >> 41);
  const int s = 22 - k;                               // bits 42 + k up, the leading one at bit 62
  const uint64_t t = (p3 << s) | (c >> (32 - s));
  const uint32_t rest = (c << s) | (uint32_t)p0;
  const uint64_t t1 = t | (rest != 0 ? 1 : 0);
  return (t1 + 0x1ff + ((uint32_t)(t >> 10) & 1)) >> 10;
}

// c - p for c = C 2^(ec - 52) (53-bit C) and p = m 2^(e - 52) below c / 8, the
// difference known to stay in c's binade: its significand, rounded.
GRD_HD uint64_t sub53(uint64_t C, int ec, uint64_t m, int e) {
  int d = ec - e;  // >= 3
  d = d > 60 ? 60 : d;
  const uint64_t q = m >> d, rem = m << (64 - d);
  const uint64_t w = C - q;
  const uint64_t half = 0x8000000000000000ull;
  return w - ((rem > half || (rem == half && (w & 1))) ? 1 : 0);
}

// sqrt of a positive normal v
GRD_HD double sqrt_pos(uint64_t uv) {
  const uint32_t h = (uint32_t)(uv >> 32);
  const uint32_t odd = ((h >> 20) & 1) ^ 1;  // of the unbiased exponent
  const uint64_t M = (uv & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint32_t Xh = (uint32_t)(M >> 21);   // X = m 2^odd in [1, 4), Q(31 - odd)
  const uint32_t Y0 = grf_fraction(grf_rsqrt(grf_float(((Xh >> 8) & 0x7fffffu) | ((127u + odd) << 23))));
  const int64_t d0 = (int64_t)((1ull << (63 - odd)) - grd_wide(Xh, grd_umulhi32(Y0, Y0)));
  const uint32_t Y = Y0 + (uint32_t)(int32_t)(((int64_t)(int32_t)(d0 >> 20) * (int32_t)(Y0 >> 1)) >> (43 - odd));
  const uint32_t S = grd_umulhi32(Xh, Y);    // sqrt X, Q(31 - odd), within 3 units
  const int64_t R = (int64_t)((M << (10 - odd)) - grd_wide(S, S));
  const int sh = 38 - 2 * (int)odd;
  const int64_t corr = ((int64_t)(int32_t)(R >> 4) * (int32_t)(Y >> 1) + (1ll << (sh - 1))) >> sh;
  const uint64_t c = ((uint64_t)S << (21 + odd)) + (uint64_t)corr;  // sqrt of M 2^(52 + odd), within 0.7
  // c 1/2 above or below the root: M 2^(52 + odd) against c^2 +- c
  const int64_t rem = (int64_t)((M << (52 + odd)) - c * c);
  const int adj = rem > (int64_t)c ? 1 : (rem <= -(int64_t)c ? -1 : 0);
  const uint64_t e = ((h >> 20) + 1023 - odd) >> 1;
  return grd_double(((e - 1) << 52) + c + (int64_t)adj);
}
GRD_HD double sqrt_d(double v) {
  const uint64_t uv = grd_bits(v);
  if ((uint32_t)(uv >> 32) - 0x00100000u < 0x7fe00000u) return sqrt_pos(uv);
#ifdef __CUDA_ARCH__
  return __dsqrt_rn(v);
#else
  return sqrt(v);
#endif
}

// a / b
GRD_HD double div_d(double a, double b) {
  const uint64_t ua = grd_bits(a), ub = grd_bits(b);
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ff, eb = (uint32_t)(ub >> 52) & 0x7ff;
  if (ea - 523u > 1000u || eb - 523u > 1000u) {  // beyond 2^-500 .. 2^500, zero, not finite
#ifdef __CUDA_ARCH__
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
  }
  uint64_t A = (ua & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t B = (ub & 0xfffffffffffffull) | 0x10000000000000ull;
  const int lt = A < B ? 1 : 0;
  A <<= lt;  // A / B in [1, 2)
  const uint32_t Bh = (uint32_t)(B >> 21);  // Q31
  const uint32_t Y0 = grf_fraction(grf_rcp(grf_float(((Bh >> 8) & 0x7fffffu) | 0x3f800000u)));
  const int64_t d0 = (int64_t)((1ull << 63) - grd_wide(Bh, Y0));
  const uint32_t Y = Y0 + (uint32_t)(int32_t)(((int64_t)(int32_t)(d0 >> 20) * (int32_t)(Y0 >> 1)) >> 42);  // 2^84 / B
  const uint32_t Q1 = grd_umulhi32((uint32_t)(A >> 22), Y);                       // Q30, within 4 units
  const int64_t R = (int64_t)((A << 30) - Q1 * B);
  const int64_t q2 = (int64_t)(int32_t)(R >> 24) * (int32_t)(Y >> 1);             // R / B, Q59
  const uint64_t c = ((uint64_t)Q1 << 22) + (uint64_t)((q2 + (1ll << 36)) >> 37);  // Q52, within 0.6
  const int64_t rem = (int64_t)((A << 52) - c * B);
  const int adj = 2 * rem > (int64_t)B ? 1 : (2 * rem < -(int64_t)B ? -1 : 0);
  const uint64_t bits = ((uint64_t)(ea - eb + 1022 - lt) << 52) + c + (int64_t)adj;
  return grd_double(((ua ^ ub) & 0x8000000000000000ull) | bits);
}

// D 2^-52 as a significand and the exponent field of its leading bit, for
// D >= 2^32
GRD_HD uint64_t norm52(uint64_t D, int& field) {
  const uint32_t h = (uint32_t)(D >> 32);
#ifdef __CUDA_ARCH__
  const int lz = __clz((int)h);
#else
  const int lz = __builtin_clz(h);
#endif
  field = 1023 + 11 - lz;  // D = 2^52 (lz 11): 1
  return lz >= 11 ? D << (lz - 11) : D;
}

// u + 2^-55 for u = F 2^-52, F the fraction of x: exact below 1/4 (8 F + 1 < 2^53); above, 2^-55 is at most half a
// unit of u, and the tie at 1/4 <= u < 1/2 goes to the even 8 F
GRD_HD double ur_nz_int(uint64_t x) {
  const uint64_t F = x & 0xfffffffffffffull;
  if ((F >> 32) == 0) return (grd_double(F | 0x3ff0000000000000ull) - 1.0) + 2.220446049250313e-16 / 8;
  int f;
  uint64_t m = norm52(F, f);
  if (F < (1ull << 50)) m |= 1ull << (1020 - f);
  return grd_double(((uint64_t)(f - 1) << 52) + m);
}
// RN(D 2^-52 c) for 0 <= D <= 2^52 and a constant c with 53-bit significand cm
// and exponent field cf
GRD_HD double scaled52(uint64_t D, uint64_t cm, int cf) {
  if ((D >> 32) == 0) return ((double)(uint32_t)D * 2.220446049250313e-16) * grd_double(((uint64_t)(cf - 1) << 52) + cm);
  int f, k;
  const uint64_t m = mul53(norm52(D, f), cm, k);
  return grd_double(((uint64_t)(f + cf - 1023 + k - 1) << 52) + m);
}

// EigenRand psincos, double lanes (MorePacketMath.h:395-491): the float-grade
// Cephes polynomials in double arithmetic, operation by operation.
//   n = number of octant pairs: (floor(|x| 4/pi) + 1) / 2, found by comparing
//       |x| with the least doubles whose product with 4/pi rounds to 1, 3, 5, 7;
//   |x| - 2 n DP1 - 2 n DP2 is exact (|x| is a multiple of 2^-53 there, both
//       products of 2^-23, and the differences do not grow), so one
//       subtraction of 2 n (DP1 + DP2) gives it;
//   z / 2 is exact, so (p - z / 2) is one fused operation;
//   the masked sums at the end are selections (no addend is -0).
// The first five steps of both polynomials run on the integer pipes, the other
// ten operations (with the two products of a Box-Muller pair) on the FP64 pipe.
// 4096 x 4096 on 608 engines, us, normal / Cauchy: 707 / 1 383 with the
// reference's operations and the library's square root and quotient; 405 / 768
// with those two, the angle and the reduction as here; 333 / 511 with four of
// the five steps, 321 / 521 with five (328 / 575 with four in the kernel as it
// is now, two words per thread).
// TOP: |x| is below the threshold 2 TOP + 1, and not tiny, in all but unusual
// calls, which go to sincos_long.
GRD_SLOW void sincos_long(double x, double* s, double* c) {
  uint64_t sign_bit_sin = grd_bits(x) & 0x8000000000000000ull;
  x = fabs(x);
  double y = x * 1.27323954473516;
  int64_t emm2 = (int64_t)floor(y);
  emm2 = emm2 + 1;
  emm2 = emm2 & ~(int64_t)1;
  y = (double)emm2;
  int64_t emm4 = emm2;
  const uint64_t swap_sign_bit_sin = ((uint64_t)(emm2 & 4)) << 61;
  emm2 = emm2 & 2;
  const uint64_t poly_mask = (emm2 == 0) ? ~0ull : 0ull;
  x = x + y * -0.78515625;
  x = x + y * -2.4187564849853515625e-4;
  x = x + y * -3.77489497744594108e-8;
  emm4 = emm4 - 2;
  emm4 = 4 & ~emm4;
  const uint64_t sign_bit_cos = ((uint64_t)emm4) << 61;
  sign_bit_sin ^= swap_sign_bit_sin;
  const double z = x * x;
  double yy = 2.443315711809948E-005;
  yy = yy * z;
  yy = yy + -1.388731625493765E-003;
  yy = yy * z;
  yy = yy + 4.166664568298827E-002;
  yy = yy * z;
  yy = yy * z;
  yy = yy - z * 0.5;
  yy = yy + 1.0;
  double y2 = -1.9515295891E-4;
  y2 = y2 * z;
  y2 = y2 + 8.3321608736E-3;
  y2 = y2 * z;
  y2 = y2 + -1.6666654611E-1;
  y2 = y2 * z;
  y2 = y2 * x;
  y2 = y2 + x;
  const double ysin2 = grd_double(poly_mask & grd_bits(y2));
  const double ysin1 = grd_double(grd_bits(yy) & ~poly_mask);
  y2 = y2 - ysin2;
  yy = yy - ysin1;
  *s = grd_double(grd_bits(ysin1 + ysin2) ^ sign_bit_sin);
  *c = grd_double(grd_bits(yy + y2) ^ sign_bit_cos);
}

template <int TOP>
GRD_HD void sincos_d(double x, double& s, double& c) {
  const uint64_t ux = grd_bits(x), ax = ux & 0x7fffffffffffffffull;
  // 2^-63, and just below the least |x| with product 3, 5, 9 (high words)
  constexpr uint32_t kLow = 0x3c000000u, kEnd = TOP == 1 ? 0x4002d97cu : TOP == 2 ? 0x400f6a7au : 0x401c463au;
  if ((uint32_t)(ax >> 32) - kLow >= kEnd - kLow) {
    sincos_long(x, &s, &c);
    return;
  }
  int n = ax >= 0x3fe921fb54442d27ull ? 1 : 0;
  if (TOP > 1) n += ax >= 0x4002d97c7f3321ddull ? 1 : 0;
  if (TOP > 2) n += (ax >= 0x400f6a7a29553870ull ? 1 : 0) + (ax >= 0x4015fdbbe9bba782ull ? 1 : 0);
  double a = grd_double(ax);
  const uint32_t dp12 = n == 0 ? 0u : n == 1 ? 0x3ff921fbu : n == 2 ? 0x400921fbu : n == 3 ? 0x4012d97cu : 0x401921fbu;
  const uint32_t dp12l = (n & 3) == 3 ? 0x70000000u : n == 0 ? 0u : 0x40000000u;
  const uint32_t dp3 = n == 0 ? 0u : n == 1 ? 0x3e74442du : n == 2 ? 0x3e84442du : n == 3 ? 0x3e8e6643u : 0x3e94442du;
  const uint32_t dp3l = n == 3 ? 0xa469e4e6u : n == 0 ? 0u : 0x18469899u;
  a = a - grd_double(((uint64_t)dp12 << 32) | dp12l);
  a = a - grd_double(((uint64_t)dp3 << 32) | dp3l);
  const double z = a * a;
  const uint64_t uz = grd_bits(z);
  const uint64_t Z = (uz & 0xfffffffffffffull) | 0x10000000000000ull;
  const int ez = (int)(uz >> 52) - 1023;
  int k;
  uint64_t m = mul53(sc53(0x3ef99eb9c5ac8ebfull), Z, k);                          // 2.443315711809948E-005
  const uint64_t p1 = sub53(sc53(0x3f56c0c33a85cd5full), -10, m, ez + k - 16);     // 1.388731625493765E-003
  m = mul53(sc53(0x3f29943f27086a6cull), Z, k);                                    // 1.9515295891E-4
  const uint64_t q1 = sub53(sc53(0x3f811073b3a82ffeull), -7, m, ez + k - 13);  // 8.3321608736E-3
  m = mul53(p1, Z, k);
  const uint64_t p2 = sub53(sc53(0x3fa55554a115bc8full), -5, m, ez + k - 10);  // 4.166664568298827E-002
  m = mul53(q1, Z, k);
  const uint64_t q2 = sub53(sc53(0x3fc5555452709addull), -3, m, ez + k - 7);       // 1.6666654611E-1
  m = mul53(p2, Z, k);
  const double pz = grd_double(((uint64_t)(1022 - 5 + ez + k) << 52) + m);
  m = mul53(q2, Z, k);
  const double qz = grd_double(((uint64_t)(1022 - 3 + ez + k) << 52) + m);
  const double yc = fma(-0.5, z, pz * z) + 1.0;
  const double ys = a - qz * a;
  const uint64_t bs = grd_bits((n & 1) ? yc : ys), bc = grd_bits((n & 1) ? ys : yc);
  s = grd_double(bs ^ ((ux & 0x8000000000000000ull) ^ ((uint64_t)(n & 2) << 62)));
  c = grd_double(bc ^ ((uint64_t)((n + 1) & 2) << 62));
}

// sin and cos of 2 pi u, pi u and pi (u - 1/2), u = F 2^-52 for the fraction F
// of x
GRD_HD void sincos_2pi_u(uint64_t x, double& s, double& c) {
  sincos_d<4>(scaled52(x & kSigOnes, sc53(0x401921fb54442d18ull), 1025), s, c);
}
GRD_HD void sincos_pi_u(uint64_t x, double& s, double& c) {
  sincos_d<2>(scaled52(x & kSigOnes, sc53(0x400921fb54442d18ull), 1024), s, c);
}
GRD_HD void sincos_pi_centred(uint64_t x, double& s, double& c) {
  const int64_t D = (int64_t)(x & kSigOnes) - (1ll << 51);
  const double t = scaled52((uint64_t)(D < 0 ? -D : D), sc53(0x400921fb54442d18ull), 1024);
  sincos_d<1>(D < 0 ? -t : t, s, c);
}
// sqrt(-2 l) for l = log of a number in (0, 1]: -2 l is exact (-0 for l = 0)
GRD_HD double sqrt_neg2(double l) {
  const uint64_t b = grd_bits(l);
  return sqrt_d(grd_double(b == 0 ? 0x8000000000000000ull : (b + (1ull << 52)) ^ 0x8000000000000000ull));
}

}  // namespace gr
