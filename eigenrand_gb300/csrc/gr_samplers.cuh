// Rejection trials and gamma components shared by the sampling kernels.
#pragma once
#include <cmath>
#include <cstdint>

#include "gr_exact.h"
#include "gr_internal.h"
#include "gr_kernels.cuh"
#include "gr_math.cuh"
#include "gr_mt.cuh"

namespace gr {

enum StagedDT { SD_F32 = 0, SD_F64 = 1, SD_I32H = 2 };
enum RejKind { RK_GAMMA_GS = 0, RK_GAMMA_TAN = 1, RK_BETA_SMALL = 2, RK_POISSON = 3, RK_BINOMIAL = 4 };

// Accept test of a GS trial (GammaGen, alpha < 1, NormalExp.h:535-556) decided
// by the special-function unit where its result lies clearly on one side of
// the comparison: 1 accept, 0 reject, -1 undecided (the caller evaluates the
// reference's expressions).  lg2.approx is within 2^-22 absolutely on (1/2, 2)
// and relatively elsewhere, ex2.approx within 2^-22 relatively (PTX ISA), so
// with vx and ux2 exact the bound qx is within 2e-6 (1 + 1/alpha) of the exact
// one, relatively (x1 |log x1| <= 1/e keeps the first branch's error from
// growing with 1/alpha); the reference's own float evaluation is within
// 1.5e-6.  The band is 2^-18 (1 + 40/alpha), over 19 times both for alpha < 1.
// ux < px is the caller's to trust.  Four special-function operations and a
// dozen others where the reference's expressions take about 110 instructions:
// the masks of 8.1 M positions of beta(0.5, 2) float, 395 us with those.
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ int gs_filter(float ux, float vx, float ux2, float px, float inv_a, float am1, float band) {
  const float l2 = lg2_approx(vx);
  const bool c = ux < px;
  const float e1 = ex2_approx(c ? inv_a * l2 : lg2_approx(fmaf(-0.693147182f, l2, 1.0f)) * am1);
  const float qx = c ? ex2_approx(-1.44269502f * e1) : e1;
  if (ux2 < qx * (1.0f - band)) return 1;
  if (ux2 > qx * (1.0f + band)) return 0;
  return -1;
}

// The same for a double trial, from the top bits of its uniforms: vx converts
// with relative error < 2^-19 (vx >= 2^-12 here), which adds 2.8e-6 / alpha to
// the error of qx, ux2 with absolute error < 2^-24 (qx >= 0.027); the branch
// test ux < px is trusted outside |ux - px| <= 2^-21 (float ux is within 2^-24
// of ux).
__device__ __forceinline__ int gs_filter_f64(uint64_t bux, uint64_t bvx, uint64_t bux2, float pxf, float inv_a,
                                             float am1, float band) {
  constexpr uint64_t M = 0xfffffffffffffull;
  // top 32 of the 52 fraction bits (absolute error < 2^-32)
  const float ux = __uint2float_rn((uint32_t)((bux & M) >> 20)) * 0x1p-32f;
  const uint64_t mv = bvx & M;
  const float vx = __uint2float_rn((uint32_t)(mv >> 20)) * 0x1p-32f;
  const float ux2 = __uint2float_rn((uint32_t)((bux2 & M) >> 20)) * 0x1p-32f;
  if (fabsf(ux - pxf) <= 0x1p-21f || (mv >> 40) == 0) return -1;
  return gs_filter(ux, vx, ux2, pxf, inv_a, am1, band);
}

// Accept test of a tan-proposal trial (GammaGen, alpha > 1, NormalExp.h:588-604)
// decided by the special-function unit, as gs_filter: with y = tan(pi u),
// x = sq y + a1 (a1 = alpha - 1, sq = sqrt(2 alpha - 1)), accept when x > 0
// and ux <= (1 + y^2) exp(a1 log(x / a1) - sq y).
// delta bounds the absolute errors of sin and cos, here and in the reference's
// polynomials (sin.approx / cos.approx: 2^-20.5 on [-2 pi, 2 pi]; PTX ISA), so
// y is off by at most dy = delta (1 + |y|)^2 (|y| <= 64), the exponent with the
// logarithm of 1 + y^2 by dy (1 + sq |a1 / x - 1|) from y and by
// 2^-20 (1 + a1 + sq |y| + |a1 log|) from roundings on both sides.  Twice that
// is the band; where it is wide, or the sign of x open, the caller evaluates
// the reference's expressions.  Five special-function operations and some
// twenty others where those take about 150 instructions (double: about 100 of
// them on the FP64 pipe), and rejected lanes need nothing more.
// eps: absolute error of ux.
__device__ __forceinline__ int tan_filter(float u, float ux, float a1, float sq, float delta, float eps = 0.0f) {
  const float t = 3.14159274f * u;
  float s, c, rc, ra, rx;
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(t));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(t));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(c));
  const float y = s * rc, ay = fabsf(y), dy = delta * (1.0f + ay) * (1.0f + ay);
  if (!(ay <= 64.0f)) return -1;
  const float x = fmaf(sq, y, a1), gap = 2.0f * sq * dy + 1e-6f * a1;
  if (x < -gap) return 0;
  if (!(x > gap)) return -1;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ra) : "f"(a1));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"(x));
  const float al = a1 * lg2_approx(x * ra) * 0.693147182f, sy = sq * y;
  const float tol = 2.0f * (dy * (1.0f + sq * fabsf(sy) * rx) + 0x1p-20f * (1.0f + a1 + fabsf(sy) + fabsf(al)));
  const float ub = fmaf(y, y, 1.0f) * ex2_approx(1.44269502f * (al - sy));
  if (!(tol < 0.25f)) return -1;
  if (ux + eps < ub * (1.0f - tol)) return 1;
  if (ux - eps > ub * (1.0f + tol)) return 0;
  return -1;
}
constexpr float kTanDeltaF = 0x1p-20f;   // float trials
constexpr float kTanDeltaD = 0x1p-19f;   // double trials: pi u rounds to float besides

__device__ __forceinline__ int tan_filter_f64(uint64_t bu, uint64_t bux, float a1, float sq) {
  constexpr uint64_t M = 0xfffffffffffffull;
  const float u = __uint2float_rn((uint32_t)((bu & M) >> 20)) * 0x1p-32f;
  const float ux = __uint2float_rn((uint32_t)((bux & M) >> 20)) * 0x1p-32f;
  // ux is within 2^-24
  return tan_filter(u, ux, a1, sq, kTanDeltaD, 0x1p-23f);
}

// Candidate of a double GS trial already known to be accepted: xx only
// (no acceptance bound); ux < px is decided on the integer fraction against
// tpx = ceil(px * 2^52).
__device__ __forceinline__ double gs_value_f64(uint64_t bux, uint64_t bvx, uint64_t tpx, double inv_a) {
  const double vx = ur_d(bvx) + 2.220446049250313e-16 / 8;
  const double lv = log_(vx);
  return ((bux & 0xfffffffffffffull) < tpx) ? exp_(inv_a * lv) : 1.0 - lv;
}

// One rejection trial, lane j: candidate bits and accept flag.  Trial t
// reads words [t * Wt, (t + 1) * Wt) of the cache-inclusive word stream
// (word(w)); full-packet double kinds read u64 lane values (rval(r)).
// CAND false: the accept flag alone is wanted.
template <int RK, int DT, bool CAND = true, class WF, class RF>
__device__ __forceinline__ bool rej_trial(const DistParams& d, int64_t t, int j, WF&& word, RF&& rval,
                                          uint64_t& cbits) {
  constexpr int Wt = (RK == RK_GAMMA_GS) ? 3 * 8 : (RK == RK_POISSON || RK == RK_BINOMIAL) ? 8 : 2 * 8;
  bool acc = false;
  cbits = 0;

  const int64_t w0 = t * Wt;
  if (DT == SD_F32) {
    if (RK == RK_GAMMA_GS) {
      const float ux = ur_f(word(w0 + j));
      const float vx = ur_f(word(w0 + 8 + j)) + 1.1920928955078125e-07f / 8;
      const float ux2 = ur_f(word(w0 + 16 + j));
      // the reference evaluates both branches and blends (NormalExp.h:543-553);
      // evaluating only the selected one gives the same bits
      // branch c: xx = exp(lv / alpha), bound exp(-xx); else xx = 1 - lv,
      // bound exp(log(xx) (alpha - 1))
      const bool c = ux < d.fe;  // px
      const int f = gs_filter(ux, vx, ux2, d.fe, d.fc, d.fd, d.fh);
      acc = f == 1;
      if ((CAND && f != 0) || f < 0) {
        const float lv = logf_(vx);
        float xx = 1.0f - lv;
        if (f < 0) {  // the reference's comparison; 1/alpha, alpha - 1
          const float e1 = expf_(c ? d.fc * lv : logf_(xx) * d.fd);
          if (c) xx = e1;
          acc = ux2 < (c ? expf_(-e1) : e1);
        } else if (c) {
          xx = expf_(d.fc * lv);
        }
        cbits = f2u(d.fb * xx);
      }
    } else if (RK == RK_GAMMA_TAN) {
      const float u = ur_f(word(w0 + j));
      const float ux = ur_f(word(w0 + 8 + j));
      const int f = tan_filter(u, ux, d.fd, d.ff, kTanDeltaF);
      acc = f == 1;
      if ((CAND && f != 0) || f < 0) {
        float ys, yc;
        sincosf_((float)3.1415926535897932 * u, ys, yc);
        const float yx = ys / yc;
        const float xx = d.ff * yx + d.fd;  // sqrt * yx + (alpha - 1)
        if (f < 0) {
          const bool c = 0.0f < xx;
          const float ub = (yx * yx + 1.0f) * expf_(d.fd * logf_(xx / d.fd) - yx * d.ff);
          acc = c && (ux <= ub);
        }
        cbits = f2u(d.fb * xx);
      }
    } else if (RK == RK_BETA_SMALL) {
      const float u1 = ur_f(word(w0 + j));
      const float u2 = ur_f(word(w0 + 8 + j));
      const float p1 = expf_(logf_(u1) * d.fc);  // 1/a
      const float p2 = expf_(logf_(u2) * d.fd);  // 1/b
      const float x = p1 + p2;
      cbits = f2u(p1 / x);
      acc = x <= 1.0f;
    }
  } else if (DT == SD_F64) {
    const int64_t r0 = (t * Wt / 8) * 4 + j;  // u64 lane index of the trial's first packet
    if (RK == RK_GAMMA_GS) {
      // float filter first: rejected lanes need nothing more, accepted ones
      // only the candidate (the exact branch is known)
      const int f = gs_filter_f64(rval(r0), rval(r0 + 4), rval(r0 + 8), d.fe, d.fc, d.fd, d.fh);
      if (f == 0) {
        acc = false;
      } else if (f == 1) {
        if (CAND) cbits = d2u(d.db * gs_value_f64(rval(r0), rval(r0 + 4), d2u(d.dg), d.dc));  // dg holds tpx as bits
        acc = true;
      } else {
        const double ux = ur_d(rval(r0));
        const double vx = ur_nz_int(rval(r0 + 4));
        const double ux2 = ur_d(rval(r0 + 8));
        const double lv = log_(vx);
        const bool c = ux < d.de;
        double xx, qx;
        if (c) {
          xx = exp_(d.dc * lv);
          qx = exp_(-xx);
        } else {
          xx = 1.0 - lv;
          qx = exp_(log_(xx) * d.dd);
        }
        cbits = d2u(d.db * xx);
        acc = ux2 < qx;
      }
    } else if (RK == RK_GAMMA_TAN) {
      const int f = tan_filter_f64(rval(r0), rval(r0 + 4), d.fd, d.ff);
      acc = f == 1;
      if ((CAND && f != 0) || f < 0) {
        double ys, yc;
        sincos_pi_u(rval(r0), ys, yc);
        const double yx = div_d(ys, yc);
        const double xx = d.df * yx + d.dd;
        if (f < 0) {
          const double ux = ur_d(rval(r0 + 4));
          const bool c = 0.0 < xx;
          const double ub = (yx * yx + 1.0) * exp_(d.dd * log_(xx / d.dd) - yx * d.df);
          acc = c && (ux <= ub);
        }
        cbits = d2u(d.db * xx);
      }
    } else if (RK == RK_BETA_SMALL) {
      const double u1 = ur_d(rval(r0));
      const double u2 = ur_d(rval(r0 + 4));
      const double p1 = exp_(log_(u1) * d.dc);
      const double p2 = exp_(log_(u2) * d.dd);
      const double x = p1 + p2;
      cbits = d2u(div_d(p1, x));
      acc = x <= 1.0;
    }
  } else {  // int32 kinds with Packet4f internals over half packets
    const float u = ur_f(word(w0 + j));
    const float u2 = ur_f(word(w0 + 4 + j));
    float s, c;
    sincosf_((float)3.1415926535897932 * u, s, c);
    const float yx = s / c;
    if (RK == RK_POISSON) {
      const float fres = truncf(d.fa * yx + d.fb);  // sqrt(2 mean) * yx + mean
      const float p1 = (yx * yx + 1.0f) * 0.9f;
      const float p2 = expf_((fres * d.fc - lgamma_approxf_(fres + 1.0f)) - d.fd);
      acc = (0.0f <= fres) && (u2 <= p1 * p2);
      cbits = f2u(fres);
    } else {  // binomial, BinomialGen::packetOp tan branch (Discrete.h:1014-1046)
      const float fres = truncf(d.fa * yx + d.fb);  // sqrt_v * ys + mean
      const float p1 = ((float)1.2 * d.fa) * (1.0f + yx * yx);
      float tt = (d.fg - lgamma_approxf_(fres + 1.0f)) - lgamma_approxf_((d.fh + 1.0f) - fres);
      tt = tt + fres * d.fc;
      tt = tt + (d.fh - fres) * d.fd;
      const float p2 = expf_(tt);
      acc = (0.0f <= fres) && (fres <= d.fh) && (u2 <= p1 * p2);
      cbits = f2u(fres);
    }
  }
  return acc;
}

// The candidate of a trial's lane that is known to be accepted: rej_trial's
// expressions for it alone.
template <int RK, int DT, class WF, class RF>
__device__ __forceinline__ uint64_t rej_value(const DistParams& d, int64_t t, int j, WF&& word, RF&& rval) {
  constexpr int Wt = (RK == RK_GAMMA_GS) ? 3 * 8 : (RK == RK_POISSON || RK == RK_BINOMIAL) ? 8 : 2 * 8;
  const int64_t w0 = t * Wt;
  if (DT == SD_F32) {
    if (RK == RK_GAMMA_GS) {
      const float lv = logf_(ur_f(word(w0 + 8 + j)) + 1.1920928955078125e-07f / 8);
      return f2u(d.fb * (ur_f(word(w0 + j)) < d.fe ? expf_(d.fc * lv) : 1.0f - lv));
    }
    if (RK == RK_GAMMA_TAN) {
      float ys, yc;
      sincosf_((float)3.1415926535897932 * ur_f(word(w0 + j)), ys, yc);
      return f2u(d.fb * (d.ff * (ys / yc) + d.fd));
    }
    const float p1 = expf_(logf_(ur_f(word(w0 + j))) * d.fc);
    const float p2 = expf_(logf_(ur_f(word(w0 + 8 + j))) * d.fd);
    return f2u(p1 / (p1 + p2));
  }
  if (DT == SD_F64) {
    const int64_t r0 = (t * Wt / 8) * 4 + j;
    if (RK == RK_GAMMA_GS) return d2u(d.db * gs_value_f64(rval(r0), rval(r0 + 4), d2u(d.dg), d.dc));
    if (RK == RK_GAMMA_TAN) {
      double ys, yc;
      sincos_pi_u(rval(r0), ys, yc);
      return d2u(d.db * (d.df * div_d(ys, yc) + d.dd));
    }
    const double p1 = exp_(log_(ur_d(rval(r0))) * d.dc);
    const double p2 = exp_(log_(ur_d(rval(r0 + 4))) * d.dd);
    return d2u(div_d(p1, p1 + p2));
  }
  float ys, yc;
  sincosf_((float)3.1415926535897932 * ur_f(word(w0 + j)), ys, yc);
  return f2u(truncf(d.fa * (ys / yc) + d.fb));
}

template <int DT>
__host__ __device__ constexpr int beta_lanes() {
  return DT == SD_F64 ? 4 : 8;
}

// Constants of one GammaGen component of a BetaGen, computed on the host
// with the same IEEE expressions the generator uses (so with the same bits),
// and passed as a kernel parameter: in the sampling loops they cost a
// constant-bank load, never a division.
struct BetaComp {
  int type, U;                      // gamma_branch: type << 8 | packets
  float af, f_px, f_inv, f_am1, f_sq;
  float f_band;                     // band of the float pre-test of a double GS trial
  double ad, d_px, d_inv, d_am1, d_sq;
  uint64_t tpx;                     // ceil(px * 2^52): double GS branch on the integer fraction
};
struct BetaConsts {
  BetaComp c[2];
  int post;              // FisherFGen: write (b/a) x / (1 - x)
  float fpost;           // b/a in the scalar type
  double dpost;
};

inline BetaComp beta_component(int branch, float af, double ad) {
  BetaComp b;
  b.type = branch >> 8;
  b.U = branch & 0xff;
  b.af = af;
  b.f_px = (float)(2.7182818284590452 / ((double)af + 2.7182818284590452));
  b.f_inv = 1 / af;
  b.f_am1 = af - 1;
  b.f_sq = std::sqrt(2 * af - 1);
  b.f_band = (float)(0x1p-18 * (1.0 + 40.0 / ad));
  b.ad = ad;
  b.d_px = 2.7182818284590452 / (ad + 2.7182818284590452);
  b.d_inv = 1 / ad;
  b.d_am1 = ad - 1;
  b.d_sq = std::sqrt(2 * ad - 1);
  b.tpx = (uint64_t)std::ceil(b.d_px * 0x1p52);
  return b;
}

// Value (closed form) or candidate (rejection trial) of one GammaGen
// component of sampler type `type` at one lane: Uf(q) gives the
// lane's uniform in the q-th packet of the draw, Ud(q) its word.  ACC: also decide
// acceptance (the rejection types); without it only the candidate is
// computed, for lanes already known to be accepted (the same expressions,
// so the same bits).
template <int DT, bool ACC, class UFF, class UDF>
__device__ __forceinline__ uint64_t beta_comp_u(const BetaComp g, const int type, UFF&& Uf, UDF&& Ud, bool& acc) {
  acc = true;
  const int U = g.U;
  if (DT == SD_F32) {
    if (type == 0) return f2u(1.0f * (-(logf_(1.0f - Uf(0)) / 1.0f)));
    if (type == 1) {
      float y = Uf(0) + 1.1920928955078125e-07f / 8;
      for (int t = 1; t < U; ++t) y = y * (Uf(t) + 1.1920928955078125e-07f / 8);
      return f2u(-(1.0f * logf_(y)));
    }
    if (type == 2) {
      const float ux = Uf(0), vx = Uf(1) + 1.1920928955078125e-07f / 8;
      const float lv = logf_(vx);
      const bool c = ux < g.f_px;
      if (!ACC) return f2u(1.0f * (c ? expf_(g.f_inv * lv) : 1.0f - lv));
      const float e1 = expf_(c ? g.f_inv * lv : logf_(1.0f - lv) * g.f_am1);  // one exp for both branches
      acc = Uf(2) < (c ? expf_(-e1) : e1);
      return f2u(1.0f * (c ? e1 : 1.0f - lv));
    }
    const float a1 = g.f_am1, sq = g.f_sq;
    float ys, yc;
    sincosf_((float)3.1415926535897932 * Uf(0), ys, yc);
    const float yx = ys / yc;
    const float xx = sq * yx + a1;
    if (ACC) {
      const float ub = (yx * yx + 1.0f) * expf_(a1 * logf_(xx / a1) - yx * sq);
      acc = (0.0f < xx) && (Uf(1) <= ub);
    }
    return f2u(1.0f * xx);
  } else {
    if (type == 0) return d2u(1.0 * (-(log_(one_minus_ur_d(Ud(0))) / 1.0)));
    if (type == 1) {
      double y = ur_nz_int(Ud(0));
      for (int t = 1; t < U; ++t) y = y * ur_nz_int(Ud(t));
      return d2u(-(1.0 * log_(y)));
    }
    if (type == 2) {
      const double ux = ur_d(Ud(0)), vx = ur_nz_int(Ud(1));
      const double lv = log_(vx);
      double xx;
      if (ux < g.d_px) {
        xx = exp_(g.d_inv * lv);
        if (ACC) acc = ur_d(Ud(2)) < exp_(-xx);
      } else {
        xx = 1.0 - lv;
        if (ACC) acc = ur_d(Ud(2)) < exp_(log_(xx) * g.d_am1);
      }
      return d2u(1.0 * xx);
    }
    const double a1 = g.d_am1, sq = g.d_sq;
    double ys, yc;
    sincos_pi_u(Ud(0), ys, yc);
    const double yx = div_d(ys, yc);
    const double xx = sq * yx + a1;
    if (ACC) {
      const double ub = (yx * yx + 1.0) * exp_(a1 * log_(xx / a1) - yx * sq);
      acc = (0.0 < xx) && (ur_d(Ud(1)) <= ub);
    }
    return d2u(1.0 * xx);
  }
}

// Lane j of unit u (the call's words: word / rword) to output element o.
template <int KIND, int DT, class WF, class RF>
__device__ __forceinline__ void staged_value(const Plan& p, const DistParams& d, int U, int64_t u, int j, int64_t o,
                                             WF&& word, RF&& rword) {
  const int64_t wpu = (DT == SD_I32H) ? 4 * (int64_t)U : 8 * (int64_t)U;  // u32 words per unit
  if (DT == SD_F32) {
    const int64_t w0 = u * wpu + j;  // full kinds: c0w == 0
    if (KIND == GR_GAMMA || KIND == GR_CHI_SQUARED) {
      float y = ur_f(word(w0)) + 1.1920928955078125e-07f / 8;
      for (int t = 1; t < U; ++t) y = y * (ur_f(word(w0 + 8 * t)) + 1.1920928955078125e-07f / 8);
      reinterpret_cast<float*>(p.out)[o] = -(d.fb * logf_(y));
    } else if (KIND == GR_STUDENT_T) {
      const float u1 = 1.0f - ur_f(word(w0));
      const float u2 = ur_f(word(w0 + 8));
      // StudentTVGen (NormalExp.h:327-342): n of the element, -2 / n per lane
      const float nn = (d.flags & kParamVecA) ? __ldg(static_cast<const float*>(d.vparam) + o) : d.fa;
      const float ex = (d.flags & kParamVecA) ? -2.0f / nn : d.fc;
      const float radius = sqrtf(nn * (expf_(logf_(u1) * ex) - 1.0f));
      float sn, cs;
      sincosf_((float)(2 * 3.1415926535897932) * u2, sn, cs);
      reinterpret_cast<float*>(p.out)[o] = radius * sn;
    }
  } else if (DT == SD_F64) {
    const int64_t r0 = u * (int64_t)U * 4 + j;
    if (KIND == GR_GAMMA || KIND == GR_CHI_SQUARED) {
      double y = ur_nz_int(rword(r0));
      for (int t = 1; t < U; ++t) y = y * ur_nz_int(rword(r0 + 4 * t));
      const double l = log_(y);
      reinterpret_cast<double*>(p.out)[o] = (d.flags & kParamUnitScale) ? -l : -(d.db * l);
    } else if (KIND == GR_STUDENT_T) {
      const double u1 = one_minus_ur_d(rword(r0));
      const double nn = (d.flags & kParamVecA) ? __ldg(static_cast<const double*>(d.vparam) + o) : d.da;
      const double ex = (d.flags & kParamVecA) ? -2.0 / nn : d.dc;
      const double radius = sqrt_d(nn * (exp_(log_(u1) * ex) - 1.0));
      double sn, cs;
      sincos_2pi_u(rword(r0 + 4), sn, cs);
      reinterpret_cast<double*>(p.out)[o] = radius * sn;
    }
  } else {  // int32 over half packets
    const int64_t w0 = u * wpu + j;
    if (KIND == GR_BINOMIAL) {
      int32_t res = d.ia;  // trials
      // p <= F 2^-23 with the fraction's integer F (p 2^23 is exact)
      const int least = d.fa <= 1.0f ? (int)ceilf(d.fa * 8388608.0f) : 1 << 23;
      for (int t = 0; t < U; ++t) res += (int)(word(w0 + 4 * t) & 0x7fffffu) >= least ? -1 : 0;
      reinterpret_cast<int32_t*>(p.out)[o] = res;
    }
  }
}

}  // namespace gr
