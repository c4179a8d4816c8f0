// Samplers whose draws per output span several packets, over words in memory
// (k_staged_words; on many engines k_units of gr_trials.cu) or drawn with a
// scalar engine (k_sx_*), and the samplers that walk their stream: Poisson,
// Beta, UniformInt, NegativeBinomial.
//
// A unit of P outputs of the fixed-unit kinds consumes a run of U packets (or U
// half packets for the int32 kinds): GammaGen with integer alpha < 20 multiplies
// alpha uniforms per output (EigenRand/Dists/NormalExp.h:577-587), BinomialGen
// with trials < 25 compares `trials` uniforms (Discrete.h:1000-1009).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "../../include/gpurand.h"
#include "gr_exact.h"
#include "gr_internal.h"
#include "gr_kernels.cuh"
#include "gr_math.cuh"
#include "gr_mt.cuh"
#include "gr_samplers.cuh"

namespace gr {

// Units [u0, u0 + cnt) of every engine over words in memory, one thread per
// output lane; block 0 of an engine leaves its state.
template <int KIND, int DT>
__global__ void __launch_bounds__(256) k_staged_words(Plan p, DistParams d, const CallSnap* snap, int U, int64_t u0,
                                                      int64_t cnt) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  const int k = blockIdx.y, tid = threadIdx.x;
  int64_t off, n;
  slice_left(p, k, off, n);
  const int64_t m = min(cnt, n / P - u0);  // this engine's units
  if (m <= 0) return;
  const int c0w = (DT == SD_I32H && snap[k].half_valid) ? 4 : 0;
  const uint64_t* w = p.words + (size_t)k * kLanes * p.wstride;
  auto lane64 = [&](int64_t packet, int l) { return mt_temper(__ldg(w + (size_t)l * p.wstride + kN + packet)); };
  auto word = [&](int64_t q) -> uint32_t {
    if (q < c0w) return snap[k].half_cache[q];
    q -= c0w;
    const uint64_t v = lane64(q >> 3, (int)((q & 7) >> 1));
    return (q & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
  };
  auto rword = [&](int64_t r) { return lane64(r >> 2, (int)(r & 3)); };
  const int64_t e = (int64_t)blockIdx.x * 256 + tid;
  if (e < m * P) staged_value<KIND, DT>(p, d, U, e / P, (int)(e % P), off + u0 * P + e, word, rword);
  if (blockIdx.x != 0) return;
  const int64_t wpu = (DT == SD_I32H) ? 4 * (int64_t)U : 8 * (int64_t)U;
  const int64_t w_last = m * wpu - 1 - c0w;
  const int64_t np = w_last < 0 ? 0 : w_last / 8 + 1;
  EngState* st = p.eng + k;
  if (np > 0)
    for (int t = tid; t < kLanes * kN; t += 256) st->win[t / kN][t % kN] = w[(size_t)(t / kN) * p.wstride + np + t % kN];
  if (tid == 0) {
    if (DT == SD_I32H) {
      // the last unit may end mid-packet: the packet's upper half stays cached
      const bool half_left = w_last >= 0 && (w_last & 7) == 3;
      if (half_left) {
        const uint64_t lo = lane64(np - 1, 2), hi = lane64(np - 1, 3);
        st->half_cache[0] = (uint32_t)lo;
        st->half_cache[1] = (uint32_t)(lo >> 32);
        st->half_cache[2] = (uint32_t)hi;
        st->half_cache[3] = (uint32_t)(hi >> 32);
      }
      st->half_valid = half_left ? 1 : 0;
    }
    st->consumed += (uint64_t)np;
  }
}

// The staged kinds drawn with a scalar engine as the Urng: output packet k
// reads U uniform packets from pre-drawn 64-bit words, float packets as
// rawbits_34 of three draws (c.lo, c.hi, b.lo, top bytes, b.hi, a.lo, a.hi,
// top bytes; a the first draw), double packets as four draws in order; the
// same per-lane arithmetic as staged_value.  One thread per output lane.
template <int KIND, int DT>
__global__ void __launch_bounds__(256) k_sx_staged(const uint64_t* w, void* out, int64_t npk, DistParams d, int U) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  const int64_t g = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (g >= npk * P) return;
  const int64_t k = g / P;
  const int j = (int)(g % P);
  if (DT == SD_F32) {
    // lane j of uniform packet t of output packet k
    auto word = [&](int t) -> uint32_t {
      const uint64_t* q = w + 3 * (k * U + t);
      const uint32_t v[6] = {(uint32_t)q[2], (uint32_t)(q[2] >> 32), (uint32_t)q[1], (uint32_t)(q[1] >> 32),
                             (uint32_t)q[0], (uint32_t)(q[0] >> 32)};
      switch (j) {
        case 0: return v[0];
        case 1: return v[1];
        case 2: return v[2];
        case 3: return (v[0] >> 24) | ((v[1] >> 24) << 8) | ((v[2] >> 24) << 16) | ((v[2] >> 24) << 24);
        case 4: return v[3];
        case 5: return v[4];
        case 6: return v[5];
        default: return (v[3] >> 24) | ((v[4] >> 24) << 8) | ((v[5] >> 24) << 16) | ((v[5] >> 24) << 24);
      }
    };
    if (KIND == GR_GAMMA) {
      float y = ur_f(word(0)) + 1.1920928955078125e-07f / 8;
      for (int t = 1; t < U; ++t) y = y * (ur_f(word(t)) + 1.1920928955078125e-07f / 8);
      static_cast<float*>(out)[g] = -(d.fb * logf_(y));
    } else {  // GR_STUDENT_T
      const float u1 = 1.0f - ur_f(word(0));
      const float u2 = ur_f(word(1));
      const float radius = sqrtf(d.fa * (expf_(logf_(u1) * d.fc) - 1.0f));
      float sn, cs;
      sincosf_((float)(2 * 3.1415926535897932) * u2, sn, cs);
      static_cast<float*>(out)[g] = radius * sn;
    }
  } else {
    const uint64_t* q = w + 4 * k * U + j;
    if (KIND == GR_GAMMA) {
      double y = ur_nz_int(q[0]);
      for (int t = 1; t < U; ++t) y = y * ur_nz_int(q[4 * t]);
      const double l = log_(y);
      static_cast<double*>(out)[g] = (d.flags & kParamUnitScale) ? -l : -(d.db * l);
    } else {  // GR_STUDENT_T
      const double u1 = one_minus_ur_d(q[0]);
      const double radius = sqrt_d(d.da * (exp_(log_(u1) * d.dc) - 1.0));
      double sn, cs;
      sincos_2pi_u(q[4], sn, cs);
      static_cast<double*>(out)[g] = radius * sn;
    }
  }
}

cudaError_t launch_sx_staged(const uint64_t* w, void* out, int64_t npk, const DistParams& d, int U,
                             cudaStream_t s) {
  const int P = d.dtype == GR_F32 ? 8 : 4;
  const unsigned blocks = (unsigned)((npk * P + 255) / 256);
  const bool gam = d.kind == GR_GAMMA;
  if (d.dtype == GR_F32) {
    if (gam) k_sx_staged<GR_GAMMA, SD_F32><<<blocks, 256, 0, s>>>(w, out, npk, d, U);
    else k_sx_staged<GR_STUDENT_T, SD_F32><<<blocks, 256, 0, s>>>(w, out, npk, d, U);
  } else {
    if (gam) k_sx_staged<GR_GAMMA, SD_F64><<<blocks, 256, 0, s>>>(w, out, npk, d, U);
    else k_sx_staged<GR_STUDENT_T, SD_F64><<<blocks, 256, 0, s>>>(w, out, npk, d, U);
  }
  return cudaGetLastError();
}

template <int KIND, int DT>
static cudaError_t run_staged(const Plan& p, const DistParams& d, const CallSnap* snap, int U, int64_t u0, int64_t cnt,
                              cudaStream_t s) {
  if (p.words) {
    constexpr int P = DT == SD_F32 ? 8 : 4;
    k_staged_words<KIND, DT>
        <<<dim3((unsigned)((cnt * P + 255) / 256), (unsigned)p.K), 256, 0, s>>>(p, d, snap, U, u0, cnt);
  } else {
    return launch_units(p, d, U, s);
  }
  return cudaGetLastError();
}

cudaError_t launch_staged(const Plan& p, const DistParams& d, const CallSnap* snap, int U, int64_t u0, int64_t cnt,
                          cudaStream_t s) {
  if (d.kind == GR_GAMMA || d.kind == GR_CHI_SQUARED) {
    if (d.dtype == GR_F32) return run_staged<GR_GAMMA, SD_F32>(p, d, snap, U, u0, cnt, s);
    if (d.dtype == GR_F64) return run_staged<GR_GAMMA, SD_F64>(p, d, snap, U, u0, cnt, s);
  }
  if (d.kind == GR_STUDENT_T) {
    if (d.dtype == GR_F32) return run_staged<GR_STUDENT_T, SD_F32>(p, d, snap, U, u0, cnt, s);
    if (d.dtype == GR_F64) return run_staged<GR_STUDENT_T, SD_F64>(p, d, snap, U, u0, cnt, s);
  }
  if (d.kind == GR_BINOMIAL && d.dtype == GR_I32) return run_staged<GR_BINOMIAL, SD_I32H>(p, d, snap, U, u0, cnt, s);
  return cudaErrorNotSupported;
}

}  // namespace gr

namespace gr {

// GammaGen's rejection trials drawn with a scalar engine (std::mt19937_64,
// P8_mt19937_64) as the Urng: trial t's candidate lanes from pre-drawn 64-bit
// words, a rejected lane written as NaN (accepted gamma candidates are never
// NaN), for TruncGen's CompressMask filter with an unbounded support.  A float
// uniform packet is RawbitsMaker<Packet8i, Rng, uint64_t, scalar_fullbit>::
// rawbits_34 of three draws (arch/AVX/RandUtils.h:59-144: lanes c.lo, c.hi,
// b.lo, top bytes, b.hi, a.lo, a.hi, top bytes, a the first draw); a double
// packet is rawbits, four draws in order.
template <int RK, int DT>
__global__ void __launch_bounds__(256) k_sx_cand(const uint64_t* w, int64_t M, DistParams d, void* cand) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  const int64_t g = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (g >= M * P) return;
  const int64_t t = g / P;
  const int j = (int)(g % P);
  auto word = [&](int64_t wi) -> uint32_t {
    const uint64_t* q = w + 3 * (wi >> 3);
    const uint32_t v[6] = {(uint32_t)q[2], (uint32_t)(q[2] >> 32), (uint32_t)q[1], (uint32_t)(q[1] >> 32),
                           (uint32_t)q[0], (uint32_t)(q[0] >> 32)};
    switch (wi & 7) {
      case 0: return v[0];
      case 1: return v[1];
      case 2: return v[2];
      case 3: return (v[0] >> 24) | ((v[1] >> 24) << 8) | ((v[2] >> 24) << 16) | ((v[2] >> 24) << 24);
      case 4: return v[3];
      case 5: return v[4];
      case 6: return v[5];
      default: return (v[3] >> 24) | ((v[4] >> 24) << 8) | ((v[5] >> 24) << 16) | ((v[5] >> 24) << 24);
    }
  };
  auto rval = [&](int64_t r) -> uint64_t { return w[r]; };
  uint64_t cb;
  const bool acc = rej_trial<RK, DT>(d, t, j, word, rval, cb);
  if (DT == SD_F32)
    static_cast<uint32_t*>(cand)[g] = acc ? (uint32_t)cb : 0x7fc00000u;
  else
    static_cast<uint64_t*>(cand)[g] = acc ? cb : 0x7ff8000000000000ull;
}

cudaError_t launch_sx_cand(int rk, int dtype, const uint64_t* w, int64_t M, const DistParams& d, void* cand,
                           cudaStream_t s) {
  const int P = dtype == GR_F32 ? 8 : 4;
  const unsigned blocks = (unsigned)((M * P + 255) / 256);
  if (dtype == GR_F32 && rk == RK_GAMMA_GS) k_sx_cand<RK_GAMMA_GS, SD_F32><<<blocks, 256, 0, s>>>(w, M, d, cand);
  else if (dtype == GR_F32 && rk == RK_GAMMA_TAN) k_sx_cand<RK_GAMMA_TAN, SD_F32><<<blocks, 256, 0, s>>>(w, M, d, cand);
  else if (dtype == GR_F64 && rk == RK_GAMMA_GS) k_sx_cand<RK_GAMMA_GS, SD_F64><<<blocks, 256, 0, s>>>(w, M, d, cand);
  else if (dtype == GR_F64 && rk == RK_GAMMA_TAN) k_sx_cand<RK_GAMMA_TAN, SD_F64><<<blocks, 256, 0, s>>>(w, M, d, cand);
  else return cudaErrorNotSupported;
  return cudaGetLastError();
}

// BetaGen / FisherFGen drawn with a scalar engine (std::mt19937_64,
// P8_mt19937_64) as the Urng, a fresh generator (the free functions;
// NormalExp.h:949-976, 1016-1021).  The draws are a chain: in the general
// branch every output packet is GammaGen(a)'s packetOp then GammaGen(b)'s,
// each a CompressMask loop with its own carried lanes when it rejects, so
// one warp walks it over a chunk of pre-drawn 64-bit words, lane j computing
// packet lane j with the same per-lane expressions as the packet engine's
// kernels (rej_trial; the exponential for alpha = 1; the product of alpha
// uniforms for an integral alpha < 20).  The a, b < 1 branch is the beta's
// own CompressMask loop over pairs of uniform packets; its mask is carried
// explicitly (an accepted lane may be 0/0).  A float uniform packet is three
// draws (rawbits_34), a double packet four.  The carried lanes are
// snapshotted at every completed output packet: the launch reports the
// packets it completed and the draws they used, and leaves the carried
// lanes as of that point, so the next chunk continues exactly there.
template <int DT>
__global__ void __launch_bounds__(32) k_sx_beta(const uint64_t* w, int64_t W, SxBetaArgs a) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  constexpr int64_t DPK = DT == SD_F32 ? 3 : 4;  // draws per uniform packet
  constexpr unsigned kFull = (1u << P) - 1u;
  const int lane = threadIdx.x;
  __shared__ uint64_t cache[3][2 * P], snap[3][2 * P];
  __shared__ int s_cnt[3], s_snap[3];
  for (int c = 0; c < 3; ++c) {
    if (lane < 2 * P) cache[c][lane] = snap[c][lane] = a.carry[c * 2 * P + lane];
    if (lane == 0) s_cnt[c] = s_snap[c] = a.cnt[c];
  }
  __syncwarp();
  int64_t pos = 0, used = 0, done = 0;  // draws consumed; by completed packets; packets completed

  // lane wi & 7 of float uniform packet wi >> 3 at draw offset pos (rawbits_34
  // of three draws a, b, c: c.lo, c.hi, b.lo, top bytes, b.hi, a.lo, a.hi, top bytes)
  auto word = [&](int64_t wi) -> uint32_t {
    const uint64_t* q = w + pos + 3 * (wi >> 3);
    const uint32_t v[6] = {(uint32_t)q[2], (uint32_t)(q[2] >> 32), (uint32_t)q[1], (uint32_t)(q[1] >> 32),
                           (uint32_t)q[0], (uint32_t)(q[0] >> 32)};
    switch (wi & 7) {
      case 0: return v[0];
      case 1: return v[1];
      case 2: return v[2];
      case 3: return (v[0] >> 24) | ((v[1] >> 24) << 8) | ((v[2] >> 24) << 16) | ((v[2] >> 24) << 24);
      case 4: return v[3];
      case 5: return v[4];
      case 6: return v[5];
      default: return (v[3] >> 24) | ((v[4] >> 24) << 8) | ((v[5] >> 24) << 16) | ((v[5] >> 24) << 24);
    }
  };
  // lane r & 3 of double uniform packet r >> 2 at draw offset pos (rawbits: four draws in order)
  auto rval = [&](int64_t r) -> uint64_t { return w[pos + r]; };

  // CompressMask::compress_append over lanes 0 .. P-1 into carried set c
  // (arch/AVX/PacketFilter.h:147-184): a full packet is returned as it is;
  // otherwise the accepted lanes join the carried ones and the first P leave
  auto compress = [&](int c, uint64_t bits, bool acc, uint64_t& res) -> bool {
    const unsigned m = __ballot_sync(0xffffffffu, acc && lane < P) & kFull;
    if (m == kFull) {
      res = bits;
      return true;
    }
    int fc = s_cnt[c];
    if (lane < P && ((m >> lane) & 1u)) cache[c][fc + __popc(m & ((1u << lane) - 1u))] = bits;
    fc += __popc(m);
    __syncwarp();
    if (fc < P) {
      if (lane == 0) s_cnt[c] = fc;
      __syncwarp();
      return false;
    }
    res = lane < P ? cache[c][lane] : 0;
    const uint64_t mv = lane < fc - P ? cache[c][P + lane] : 0;
    __syncwarp();
    if (lane < fc - P) cache[c][lane] = mv;
    if (lane == 0) s_cnt[c] = fc - P;
    __syncwarp();
    return true;
  };

  // GammaGen(alpha)'s packetOp for component c (0: a, 1: b); false when the
  // chunk runs out first
  auto gamma_packet = [&](int c, uint64_t& v) -> bool {
    const DistParams& g = a.g[c];
    if (g.ic) {  // alpha < 1: GS rejection, three uniform packets per trial
      for (;;) {
        if (pos + 3 * DPK > W) return false;
        uint64_t cb = 0;
        const bool acc = lane < P && rej_trial<RK_GAMMA_GS, DT>(g, 0, lane, word, rval, cb);
        pos += 3 * DPK;
        if (compress(c, cb, acc, v)) return true;
      }
    }
    if (g.ia) {  // alpha == 1: beta * ExponentialGen
      if (pos + DPK > W) return false;
      if (lane < P) {
        if (DT == SD_F32) {
          v = f2u(g.fb * (-(logf_(1.0f - ur_f(word(lane))) / 1.0f)));
        } else {
          const double l = -(log_(one_minus_ur_d(rval(lane))) / 1.0);
          v = d2u((g.flags & kParamUnitScale) ? l : g.db * l);
        }
      }
      pos += DPK;
      return true;
    }
    if (g.ib >= 2) {  // integral alpha < 20: product of alpha nonzero uniforms
      if (pos + g.ib * DPK > W) return false;
      if (lane < P) {
        if (DT == SD_F32) {
          float y = ur_f(word(lane)) + 1.1920928955078125e-07f / 8;
          for (int t = 1; t < g.ib; ++t) y = y * (ur_f(word(8 * t + lane)) + 1.1920928955078125e-07f / 8);
          v = f2u(-(g.fb * logf_(y)));
        } else {
          double y = ur_nz_int(rval(lane));
          for (int t = 1; t < g.ib; ++t) y = y * ur_nz_int(rval(4 * t + lane));
          const double l = log_(y);
          v = d2u((g.flags & kParamUnitScale) ? -l : -(g.db * l));
        }
      }
      pos += g.ib * DPK;
      return true;
    }
    for (;;) {  // the tan proposal, two uniform packets per trial
      if (pos + 2 * DPK > W) return false;
      uint64_t cb = 0;
      const bool acc = lane < P && rej_trial<RK_GAMMA_TAN, DT>(g, 0, lane, word, rval, cb);
      pos += 2 * DPK;
      if (compress(c, cb, acc, v)) return true;
    }
  };

  while (done < a.npk) {
    uint64_t v = 0;
    bool ok = true;
    if (a.beta.ic) {  // a < 1 and b < 1: the beta's own rejection loop
      for (;;) {
        if (pos + 2 * DPK > W) {
          ok = false;
          break;
        }
        uint64_t cb = 0;
        const bool acc = lane < P && rej_trial<RK_BETA_SMALL, DT>(a.beta, 0, lane, word, rval, cb);
        pos += 2 * DPK;
        if (compress(2, cb, acc, v)) break;
      }
    } else {
      uint64_t p1 = 0, p2 = 0;
      ok = gamma_packet(0, p1) && gamma_packet(1, p2);
      if (ok) {
        if (DT == SD_F32) v = f2u(u2f((uint32_t)p1) / (u2f((uint32_t)p1) + u2f((uint32_t)p2)));
        else v = d2u(u2d(p1) / (u2d(p1) + u2d(p2)));
      }
    }
    if (!ok) break;
    v = beta_post<DT == SD_F64>(v, a.beta);
    if (lane < P) {
      if (DT == SD_F32) static_cast<uint32_t*>(a.out)[done * P + lane] = (uint32_t)v;
      else static_cast<uint64_t*>(a.out)[done * P + lane] = v;
    }
    ++done;
    used = pos;
    for (int c = 0; c < 3; ++c) {
      if (lane < 2 * P) snap[c][lane] = cache[c][lane];
      if (lane == 0) s_snap[c] = s_cnt[c];
    }
    __syncwarp();
  }
  // the carried lanes as of the last completed packet
  for (int c = 0; c < 3; ++c) {
    if (lane < 2 * P) a.carry[c * 2 * P + lane] = snap[c][lane];
    if (lane == 0) a.cnt[c] = s_snap[c];
  }
  if (lane == 0) {
    a.res[0] = done;
    a.res[1] = used;
  }
}

cudaError_t launch_sx_beta(const uint64_t* w, int64_t W, const SxBetaArgs& a, int dtype, cudaStream_t s) {
  if (dtype == GR_F32) k_sx_beta<SD_F32><<<1, 32, 0, s>>>(w, W, a);
  else k_sx_beta<SD_F64><<<1, 32, 0, s>>>(w, W, a);
  return cudaGetLastError();
}


}  // namespace gr

namespace gr {

// ===========================================================================
// k_poisson: PoissonGen with mean < 12 (Discrete.h:870-882), also BinomialGen
// with trials * min(p, 1-p) < 1 (its PoissonGen member).  One packetOp
// multiplies half packets of uniforms until every lane's product is
// <= exp(-mean) and returns, per lane, how many products stayed above it; the
// step from half packet s consumes L(s) half packets and the next starts at
// s + L(s).  Per block of 312 packets: the uniforms go to a float ring as the
// packets are made; every new start position gets its step (L and the four
// counts, packed in one word) in parallel; thread 0 follows s += L(s); all
// threads write the visited steps' counts.
// ===========================================================================
namespace {
constexpr int kPoisThreads = 160;
constexpr int kPoisLook = 64;    // half packets one step may read; a longer step is reported
constexpr int kPoisRing = 1024;  // start positions kept (>= 2 * 312 + kPoisLook)
constexpr int kPoisRec = 704;    // steps recorded per block (<= 624 + kPoisLook)
constexpr size_t kPoisSmem = (size_t)3 * kLanes * kN * 8 +  // raw x3
                             (size_t)2 * kN * 8 * 4 +       // uniforms of the two newest blocks
                             (size_t)kPoisRing * 4 +        // per position: L << 24 | counts (6 bits each)
                             (size_t)kPoisRec * 2;          // visited positions (ring index)
}  // namespace

__global__ void __launch_bounds__(kPoisThreads) k_poisson(Plan p, DistParams d, int64_t max_blocks) {
  extern __shared__ __align__(16) uint64_t pois_dyn[];
  // raw: three block buffers so the window before the end of the call is
  // still in shared memory when the call ends in the previous block
  uint64_t(*raw)[kLanes][kN] = reinterpret_cast<uint64_t(*)[kLanes][kN]>(pois_dyn);
  float(*uf)[kN][8] = reinterpret_cast<float(*)[kN][8]>(pois_dyn + 3 * kLanes * kN);
  uint32_t* pos = reinterpret_cast<uint32_t*>(pois_dyn + 3 * kLanes * kN + kN * 8);
  uint16_t* rec = reinterpret_cast<uint16_t*>(pos + kPoisRing);
  __shared__ int s_nrec, s_stop, s_err;
  __shared__ int64_t s_ebase, s_end;
  __shared__ float4 s_cache;  // uniforms of the engine's cached half packet
  const int k = blockIdx.x;
  const int tid = threadIdx.x;
  EngState* st = p.eng + k;
  int64_t off, n;
  slice_left(p, k, off, n);
  if (n == 0) return;
  const int64_t Npk = n / 4;
  const int c0w = st->half_valid ? 4 : 0;  // the first half packet comes from the engine's cache
  load_window(raw[0], &st->win[0][0], kN);
  if (tid == 0) {
    s_err = 0;
    s_stop = 0;
    s_cache = make_float4(ur_f(st->half_cache[0]), ur_f(st->half_cache[1]), ur_f(st->half_cache[2]),
                          ur_f(st->half_cache[3]));
  }
  __syncthreads();
  int64_t s = 0, E = 0, done_pos = 0;  // walk (thread 0); positions evaluated up to done_pos
  int cur = 0;
  int64_t nb = 0;
  for (; nb < max_blocks; ++nb) {
    const int slot = (int)(nb & 1);
    const int nxt = cur == 2 ? 0 : cur + 1;
    mt_block(raw[cur], raw[nxt], [&](int i, const uint64_t* pk) {
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        uf[slot][i][2 * l] = ur_f((uint32_t)pk[l]);
        uf[slot][i][2 * l + 1] = ur_f((uint32_t)(pk[l] >> 32));
      }
    });
    cur = nxt;
    // positions whose whole step (<= kPoisLook half packets) exists
    const int64_t lim = c0w / 4 + 2 * (nb + 1) * kN - kPoisLook;
    if (tid == 0 && lim - s > kPoisRing) s_err = 1;
    // ---- steps of the new start positions
    for (int64_t x = done_pos + tid; x < lim; x += kPoisThreads) {
      // half packet x starts at packet-stream word 4x - c0w (negative: the
      // engine's cached half packet); w = offset from the newest block's first word
      const bool cached = 4 * x < c0w;
      int w = (int)(4 * x - c0w - 8 * nb * (int64_t)kN);
      float val[4] = {1.0f, 1.0f, 1.0f, 1.0f};
      int kk[4] = {0, 0, 0, 0};
      int L = 0;
      bool any = true;
      for (int it = 0; it < kPoisLook && any; ++it, w += 4) {
        float4 u;
        if (it == 0 && cached) {
          u = s_cache;
        } else {
          int pk = w >> 3, sl = slot;
          if (pk < 0) {
            pk += kN;
            sl ^= 1;
          }
          u = *reinterpret_cast<const float4*>(&uf[sl][pk][w & 7]);
        }
        const float uu[4] = {u.x, u.y, u.z, u.w};
        any = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          val[j] = val[j] * uu[j];
          const bool c = d.fe < val[j];  // exp(-mean) < val
          kk[j] += c ? 1 : 0;
          any |= c;
        }
        L = it + 1;
      }
      if (any) atomicOr(&s_err, 1);
      pos[(int)(x & (kPoisRing - 1))] =
          ((uint32_t)L << 24) | (uint32_t)kk[0] | ((uint32_t)kk[1] << 6) | ((uint32_t)kk[2] << 12) | ((uint32_t)kk[3] << 18);
    }
    done_pos = max(done_pos, lim);
    __syncthreads();
    // ---- walk (thread 0)
    if (tid == 0) {
      s_ebase = E;
      int nrec = 0;
      while (s < done_pos && E < Npk && nrec < kPoisRec) {
        const int ri = (int)(s & (kPoisRing - 1));
        rec[nrec++] = (uint16_t)ri;
        s += pos[ri] >> 24;
        ++E;
      }
      s_nrec = nrec;
      if (E >= Npk) {
        s_stop = 1;
        s_end = s;
      }
    }
    __syncthreads();
    // ---- write the visited steps
    const int nrec = s_nrec;
    const int64_t e_first = s_ebase;
    for (int e = tid; e < nrec * 4; e += kPoisThreads) {
      const int i = e >> 2, j = e & 3;
      int32_t v = (int32_t)((pos[rec[i]] >> (6 * j)) & 63);
      if (d.ic) v = d.ia - v;  // BinomialGen: trials - res when p > 1/2
      reinterpret_cast<int32_t*>(p.out)[off + (e_first + i) * 4 + j] = v;
    }
    __syncthreads();
    if (s_stop || s_err) break;
  }
  // ---- state after the call
  if (tid == 0 && (!s_stop || s_err)) {
    if (!s_stop) s_end = s;
    atomicOr(&st->status, (int)GR_DEV_REJECT_LIMIT);
  }
  __syncthreads();
  const int64_t fresh = s_end - c0w / 4;  // half packets drawn fresh
  const int64_t np = (fresh + 1) / 2;     // packets consumed
  const int prv = cur == 0 ? 2 : cur - 1, prv2 = prv == 0 ? 2 : prv - 1;
  const int64_t nblk = min(nb + 1, max_blocks);  // blocks generated
  if (np > 0) {
    const int64_t lastb = (np - 1) / kN;
    const int64_t rr = np - lastb * kN;  // in [1, 312]
    if (lastb == nblk - 1) store_window(st, raw[cur], raw[prv], (int)rr);
    else if (lastb == nblk - 2) store_window(st, raw[prv], raw[prv2], (int)rr);
    else if (tid == 0) atomicOr(&st->status, (int)GR_DEV_BAD_INPUT);
  }
  if (tid == 0) {
    if (fresh & 1) {  // the last packet's upper half stays in the engine's half cache
      const int64_t pl = np - 1;
      const int buf = (pl / kN == nblk - 1) ? cur : prv;
      const uint64_t a = mt_temper(raw[buf][2][pl % kN]), b = mt_temper(raw[buf][3][pl % kN]);
      st->half_cache[0] = (uint32_t)a;
      st->half_cache[1] = (uint32_t)(a >> 32);
      st->half_cache[2] = (uint32_t)b;
      st->half_cache[3] = (uint32_t)(b >> 32);
      st->half_valid = 1;
    } else {
      st->half_valid = 0;
    }
    st->consumed += (uint64_t)max(np, (int64_t)0);
  }
}

static cudaError_t run_poisson(const Plan& p, const DistParams& d, int64_t max_blocks, cudaStream_t s) {
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr[dev]) {
    cudaError_t e = cudaFuncSetAttribute(k_poisson, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPoisSmem);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  k_poisson<<<p.K, kPoisThreads, kPoisSmem, s>>>(p, d, max_blocks);
  return cudaGetLastError();
}

// ===========================================================================
// k_beta: BetaGen with a >= 1 or b >= 1 (NormalExp.h:970-975).  Each output
// packet draws one packet from GammaGen(a), then one from GammaGen(b); a
// component is closed form (alpha == 1: 1 packet; integer alpha < 20: alpha
// packets) or a rejection sampler (GS trials of 3 packets, tan trials of 2)
// with its own CompressMask carry.
// The ring of packets is the newest three raw engine blocks in shared
// memory, tempered where read (no tempered copy), so four CTAs fit on an SM
// and all engines run in one wave.  Every start position of a rejection
// component gets its P-lane accept mask ahead of the walk; the walk over
// the masks and the value work run on separate warps (the kernel below).
// ===========================================================================
namespace {

constexpr int kBetaRing = 1024;  // positions whose accept masks are kept (a power of two)

}  // namespace

// ===========================================================================
// k_beta: the walk with the reference automaton on a warp of its own, one
// step ahead of the workers.
//   chase  (warp 0) follows the automaton over the accept masks: per trial
//          of a rejection component one mask read, its popcount and two
//          compares.  Per step it records the source of every output packet
//          (closed-form position, full-trial value slot or FIFO offset) and,
//          for every accepted lane of a consumed partial trial, its FIFO slot
//          (position and lane, written by the warp's first P lanes at once),
//          into one of two buffers.
//   work   (warps 1-5) take the previous step's buffer: the full-trial values
//          of the rejection component, the accepted partial lanes and the
//          positional values of the other component as one task list;
//          p1 / (p1 + p2) per output lane; the carried lanes to the front of
//          the lane buffer; then they twist the next engine block and
//          evaluate its accept masks.
// The chase of step t reads only masks; the workers of step t - 1 read the
// raw ring (blocks t - 2 .. t) before they overwrite block t - 2 with block
// t + 1, so the step's packets must start at block t - 2 or later (checked;
// a record longer than two blocks ends the call with the iteration-cap
// status).  Buffers hold more than one block's worth of records, partial
// lanes and FIFO lanes, so a chase that fell behind catches up.
// TY0 / TY1: the components' sampler types when known at compile time (the
// kernel then carries only their code), else -1.
// ONE: exactly one component is a rejection sampler.  The trial-by-trial chase
// (125 ns a trial, one warp) then bounds the kernel, so the workers also resolve,
// for every position and number of carried lanes, the visit that would start
// there (how many trials, full or carried lanes after it): the chase is one
// look-up per output, and the workers list the accepted lanes of the visits it
// took.  GS masks: one thread per 64-bit word, its uniforms converted once for
// the three trials they are in.  What bounds it now is instruction issue.
// Beta(0.5, 2), 4096 x 4096 on 608 engines, us, float / double: 1 176 / 2 200 with
// the trial-by-trial chase, 980 / 2 014 with look-ups, 806 / 1 873 with the masks
// by word.
// ===========================================================================
namespace {

constexpr int kBcThreads = 192;       // four CTAs per SM
constexpr int kBcRec = 160;         // output packets per step (a block holds at most 156)
constexpr int kBcFifo = 112;        // FIFO outputs per component per step (at most 104 per block)
constexpr int kBcFull = 112;        // full-trial outputs of the buffered component per step
constexpr int kBcFullTag = 16384;   // record source >= this: full-trial value slot

template <int DT>
__host__ __device__ constexpr int bc_lb() {  // lane buffer per component: carried + one step's FIFO lanes
  return 16 + kBcFifo * beta_lanes<DT>();
}

struct BcStep {
  int64_t base, e0;  // first packet of the step (sources are relative to it), first output packet
  int nrec, nf, fs[2], A[2], f[2];
};

template <int DT, bool ONE>
__host__ __device__ constexpr size_t bc_smem_bytes() {
  if (ONE)
    return (size_t)3 * kLanes * kN * 8 +                                                 // raw windows
           (size_t)2 * kBcRec * 8 +                                                      // outputs of a step
           ((size_t)bc_lb<DT>() + (size_t)(kBcFull + kBcRec) * beta_lanes<DT>()) *       // lane buffer, full-
               (DT == SD_F64 ? 8 : 4) +                                                  //   trial and positional values
           (size_t)kBetaRing * beta_lanes<DT>() +                                        // visits per position
           (size_t)kBcRec * 2 + (size_t)kBcFull * 2 + (size_t)bc_lb<DT>() * 2 +          // sources, full trials, tasks
           (size_t)kBetaRing;                                                            // masks per position
  return (size_t)3 * kLanes * kN * 8 +                                                   // raw windows
         ((size_t)2 * bc_lb<DT>() + (size_t)(kBcFull + kBcRec) * beta_lanes<DT>()) *     // lane buffers, full-
             (DT == SD_F64 ? 8 : 4) +                                                    //   trial and positional values
         (size_t)2 * kBcRec * 2 * 2 +                                                    // records
         (size_t)2 * kBcFull * 2 +                                                       // full-trial positions
         (size_t)2 * 2 * bc_lb<DT>() * 2 +                                               // partial-lane tasks
         (size_t)2 * kBetaRing;                                                          // masks per position
}

}  // namespace

// DT: SD_F32 or SD_F64
template <int DT, int TY0, int TY1, bool ONE>
__global__ void __maxnreg__(80) k_beta(Plan p, BetaConsts bk, int64_t max_blocks) {
  constexpr int NT = kBcThreads;
  constexpr int kBcWork = NT - 32;
  constexpr int P = beta_lanes<DT>();
  constexpr int LB = bc_lb<DT>();
  constexpr unsigned FULL = 0xffffffffu;
  using V = typename std::conditional<DT == SD_F64, uint64_t, uint32_t>::type;
  extern __shared__ __align__(16) uint64_t bc_dyn[];
  uint64_t(*raw)[kLanes][kN] = reinterpret_cast<uint64_t(*)[kLanes][kN]>(bc_dyn);
  // ONE: [1][LB] lanes, single-buffered sources and tasks, xrec and visits
  uint64_t* xrec = bc_dyn + 3 * kLanes * kN;                             // [2][kBcRec]
  V* lanebuf = reinterpret_cast<V*>(xrec + (ONE ? 2 * kBcRec : 0));      // [2][LB]
  V* fullval = lanebuf + (ONE ? 1 : 2) * LB;                             // [kBcFull][P]
  V* posval = fullval + kBcFull * P;                                     // [kBcRec][P]
  uint8_t* visits = reinterpret_cast<uint8_t*>(posval + kBcRec * P);     // [kBetaRing][P]
  int16_t* rec = reinterpret_cast<int16_t*>(visits + (ONE ? kBetaRing * P : 0));  // [2][kBcRec][2]
  int16_t* fpos = rec + (ONE ? kBcRec : 2 * kBcRec * 2);                 // [2][kBcFull]
  uint16_t* ptask = reinterpret_cast<uint16_t*>(fpos + (ONE ? 1 : 2) * kBcFull);  // [2][2][LB]
  uint8_t* pmask = reinterpret_cast<uint8_t*>(ptask + (ONE ? 1 : 2 * 2) * LB);    // [2][kBetaRing]
  __shared__ BcStep s_step[2];
  __shared__ int s_done, s_err, s_fc[2];
  __shared__ int64_t s_end;

  const int k = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  EngState* st = p.eng + k;
  GenState* gs = p.gen + k;
  int64_t off, n;
  slice_left(p, k, off, n);
  if (n == 0) return;
  const int64_t Npk = n / P;

  const int type0 = TY0 >= 0 ? TY0 : bk.c[0].type, type1 = TY1 >= 0 ? TY1 : bk.c[1].type;
  const int U0 = bk.c[0].U, U1 = bk.c[1].U;
  const bool post = bk.post == 1;
  const int umax = max(max(U0, U1), 3);
  // bc: the rejection component whose full-trial values get a slot; ob: the
  // component whose positional values are computed with them
  const int bc = type0 >= 2 ? 0 : (type1 >= 2 ? 1 : -1);
  const int ob = bc == 0 ? 1 : (bc == 1 ? 0 : 1);
  const int rc = ONE ? bc : 0;  // ONE: the rejection component; its buffers are the only ones
  const int Ur = rc == 0 ? U0 : U1, Uc = rc == 0 ? U1 : U0;
  load_window(raw[2], &st->win[0][0], kN);  // block -1; block b lives in window b mod 3
  // carried lanes of the two GammaGens (generator slots 1 and 2)
  if (tid < 2 * 8) {
    const int c = tid / 8, j = tid % 8;
    const GenSlot& g = gs->s[1 + c];
    if (j < g.rest_cnt && (!ONE || c == rc))
      lanebuf[(ONE ? 0 : c) * LB + j] = (V)(DT == SD_F64 ? ((uint64_t)g.rest[2 * j] | ((uint64_t)g.rest[2 * j + 1] << 32))
                                             : (uint64_t)g.rest[j]);
  }
  if (tid == 0) {
    s_err = 0;
    s_done = 0;
  }
  __syncthreads();
  // The newest three raw blocks are the ring of packets; words are tempered
  // where they are read.  Each thread keeps its own view of the newest block.
  int64_t ring_new = 0;
  int wb0 = 0, wb1 = 2, wb2 = 1;
  auto set_ring = [&](int64_t B) {
    ring_new = B * kN;
    wb0 = (int)(B % 3);
    wb1 = (int)((B + 2) % 3);
    wb2 = (int)((B + 1) % 3);
  };
  // word l of the packet at dd, relative to the newest block's first
  auto tword = [&](int dd, int l) -> uint64_t {
    int w = wb0;
    if (dd < 0) {
      dd += kN;
      w = wb1;
      if (dd < 0) {
        dd += kN;
        w = wb2;
      }
    }
    if ((unsigned)dd >= (unsigned)kN) dd = 0;  // outside the ring: never read past the buffers
    return mt_temper(raw[w][l][dd]);
  };
  auto word = [&](int dd, int j) -> uint32_t {
    const uint64_t v = tword(dd, j >> 1);
    return (j & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
  };
  // value of an accepted trial lane or a closed-form draw; double GS lanes
  // use the branch threshold in integer form
  auto value = [&](int c, int x, int j) -> uint64_t {
    bool acc;
    auto uf = [&](int q) { return ur_f(word(x + q, j)); };
    auto ud = [&](int q) { return tword(x + q, j); };
    if (c == 0) {
      if (DT == SD_F64 && type0 == 2)
        return d2u(1.0 * gs_value_f64(tword(x, j), tword(x + 1, j), bk.c[0].tpx, bk.c[0].d_inv));
      return beta_comp_u<DT, false>(bk.c[0], type0, uf, ud, acc);
    }
    if (DT == SD_F64 && type1 == 2)
      return d2u(1.0 * gs_value_f64(tword(x, j), tword(x + 1, j), bk.c[1].tpx, bk.c[1].d_inv));
    return beta_comp_u<DT, false>(bk.c[1], type1, uf, ud, acc);
  };
  // The GS + integral-alpha pairs: the value of either component is one log
  // (of the GS trial's vx, or of the product of the integral draw's
  // uniforms), then an exp for GS lanes below the branch threshold; every
  // lane of a warp shares the log whichever component it computes.
  constexpr bool kFused = (TY0 == 2 && TY1 == 1) || (TY0 == 1 && TY1 == 2);
  constexpr int gc = TY0 == 2 ? 0 : 1;  // the GS component of a fused pair
  auto value_task = [&](int c, int x, int j) -> uint64_t {
    if (!kFused) return value(c, x, j);
    const BetaComp& g = c == 0 ? bk.c[0] : bk.c[1];
    const bool gsv = c == gc;
    if (DT == SD_F64) {
      const uint64_t b0 = tword(x, j), b1 = tword(x + 1, j);
      double arg = ur_nz_int(b1);
      if (!gsv) {
        double y = ur_nz_int(b0);
        y = y * arg;
        for (int q = 2; q < g.U; ++q) y = y * ur_nz_int(tword(x + q, j));
        arg = y;
      }
      const double l = log_(arg);
      if (!gsv) return d2u(-(1.0 * l));
      return d2u(1.0 * (((b0 & 0xfffffffffffffull) < g.tpx) ? exp_(g.d_inv * l) : 1.0 - l));
    } else {
      constexpr float e = 1.1920928955078125e-07f / 8;
      const float u0 = ur_f(word(x, j)), u1 = ur_f(word(x + 1, j));
      float arg = u1 + e;
      if (!gsv) {
        float y = u0 + e;
        y = y * arg;
        for (int q = 2; q < g.U; ++q) y = y * (ur_f(word(x + q, j)) + e);
        arg = y;
      }
      const float l = logf_(arg);
      if (!gsv) return f2u(-(1.0f * l));
      return f2u(1.0f * ((u0 < g.f_px) ? expf_(g.f_inv * l) : 1.0f - l));
    }
  };
  const int nrej = (type0 >= 2 ? 1 : 0) + (type1 >= 2 ? 1 : 0);
  const int rej0 = type0 >= 2 ? 0 : 1;
  // accept masks of the rejection components at positions [from, to), by
  // threads t = 0 .. T-1 of whole warps.  Each group of P threads (one per
  // lane) walks a run of consecutive positions and slides a window of the
  // lane's three tempered words along it (one word fetched per position);
  // a ballot per step gives the masks of the warp's 32 / P runs.
  auto masks = [&](int64_t first, int64_t last, int t, int T) {
    if (nrej == 0 || last <= first) return;
    const int from = (int)(first - ring_new), to = (int)(last - ring_new), rm = (int)(ring_new & (kBetaRing - 1));
    if (ONE && (TY0 == 2 || TY1 == 2 || (rc == 0 ? type0 : type1) == 2)) {
      // GS trials: a thread per 64-bit word (two float lanes), whose uniforms
      // it converts once for the three trials they are in
      const BetaComp& g = bk.c[TY0 == 2 ? 0 : TY1 == 2 ? 1 : rc];
      const int runs = (T >> 5) * 8;
      const int L = (to - from + runs - 1) / runs;
      const int wl = t & 3, x0 = from + ((t >> 5) * 8 + (t & 31) / 4) * L;
      const uint64_t* next = x0 < 0 ? &raw[wb1][wl][x0 + kN] : &raw[wb0][wl][min(x0, kN - 1)];
      int turn = x0 < 0 ? -x0 : kN;  // packets until the newest block begins
      uint64_t w0 = 0, w1 = 0, w2 = 0;
      float a0 = 0, a1 = 0, a2 = 0, b0 = 0, b1 = 0, b2 = 0;
      for (int i = -2; i < L; ++i) {
        const int x = x0 + i;
        w0 = w1;
        w1 = w2;
        a0 = a1;
        a1 = a2;
        b0 = b1;
        b1 = b2;
        if (x < to) {
          w2 = mt_temper(*next);
          ++next;
          if (--turn == 0) next = raw[wb0][wl];
          if (DT == SD_F32) {
            a2 = ur_f((uint32_t)w2);
            b2 = ur_f((uint32_t)(w2 >> 32));
          } else {
            a2 = __uint2float_rn((uint32_t)((w2 & 0xfffffffffffffull) >> 20)) * 0x1p-32f;
          }
        }
        if (i < 0) continue;
        int fa = 0, fb = 0;
        if (x < to) {
          if (DT == SD_F32) {
            constexpr float e = 1.1920928955078125e-07f / 8;
            fa = gs_filter(a0, a1 + e, a2, g.f_px, g.f_inv, g.f_am1, g.f_band);
            fb = gs_filter(b0, b1 + e, b2, g.f_px, g.f_inv, g.f_am1, g.f_band);
          } else {
            // gs_filter_f64's range tests
            fa = fabsf(a0 - g.f_px) <= 0x1p-21f || a1 < 0x1.001p-12f
                     ? -1 : gs_filter(a0, a1, a2, g.f_px, g.f_inv, g.f_am1, g.f_band);
          }
          auto exact = [&](int hi) -> int {
            auto uf = [&](int q) { return hi ? (q == 0 ? b0 : (q == 1 ? b1 : b2)) : (q == 0 ? a0 : (q == 1 ? a1 : a2)); };
            auto ud = [&](int q) { return q == 0 ? w0 : (q == 1 ? w1 : w2); };
            bool acc;
            beta_comp_u<DT, true>(g, 2, uf, ud, acc);
            return acc ? 1 : 0;
          };
          if (fa < 0) fa = exact(0);
          if (fb < 0) fb = exact(1);
        }
        __syncwarp();
        const uint32_t ba = __ballot_sync(FULL, fa == 1) >> (t & 28) & 15u;
        uint32_t m = ba;
        if (DT == SD_F32) {
          const uint32_t bb = __ballot_sync(FULL, fb == 1) >> (t & 28) & 15u;
          const uint32_t ea = (ba | ba << 2) & 0x33u, eb = (bb | bb << 2) & 0x33u;
          m = ((ea | ea << 1) & 0x55u) | ((eb | eb << 1) & 0x55u) << 1;
        }
        if (x < to && wl == 0) pmask[(rm + x) & (kBetaRing - 1)] = (uint8_t)m;
      }
      return;
    }
    constexpr int G = 32 / P;
    const int runs = (T >> 5) * G;
    const int L = (to - from + runs - 1) / runs;
    const int r = (t >> 5) * G + (t & 31) / P, j = t & (P - 1);
    const int lw = DT == SD_F64 ? j : (j >> 1);  // the lane's 64-bit word
    const int x0 = from + r * L;
    // the filters decide most positions; a thread then evaluates those they leave
    // open one after the other (L is 16 at most), or every position in which one of
    // the warp's lanes is open would cost all of them the reference's expressions
    for (int ci = 0; ci < nrej; ++ci) {
      const int c = nrej == 2 ? ci : rej0;
      const int ty = c == 0 ? type0 : type1;
      const BetaComp& g = c == 0 ? bk.c[0] : bk.c[1];
      const int sh = (j & 1) * 32;
      uint32_t accepted = 0, open = 0;
      uint64_t w0 = 0, w1 = tword(x0, lw), w2 = tword(x0 + 1, lw);
      for (int i = 0; i < L; ++i) {
        w0 = w1;
        w1 = w2;
        w2 = tword(x0 + i + 2, lw);
        if (x0 + i >= to) continue;
        int f;
        if (DT == SD_F64)
          f = ty == 2 ? gs_filter_f64(w0, w1, w2, g.f_px, g.f_inv, g.f_am1, g.f_band)
                      : tan_filter_f64(w0, w1, g.f_am1, g.f_sq);
        else
          f = ty == 2 ? gs_filter(ur_f((uint32_t)(w0 >> sh)), ur_f((uint32_t)(w1 >> sh)) + 1.1920928955078125e-07f / 8,
                                  ur_f((uint32_t)(w2 >> sh)), g.f_px, g.f_inv, g.f_am1, g.f_band)
                      : tan_filter(ur_f((uint32_t)(w0 >> sh)), ur_f((uint32_t)(w1 >> sh)), g.f_am1, g.f_sq, kTanDeltaF);
        accepted |= (f == 1 ? 1u : 0u) << i;
        open |= (f < 0 ? 1u : 0u) << i;
      }
      while (__any_sync(FULL, open != 0)) {
        if (open) {
          const int i = __ffs(open) - 1;
          open &= open - 1;
          const uint64_t v0 = tword(x0 + i, lw), v1 = tword(x0 + i + 1, lw), v2 = tword(x0 + i + 2, lw);
          auto uf = [&](int q) { return ur_f((uint32_t)((q == 0 ? v0 : (q == 1 ? v1 : v2)) >> sh)); };
          auto ud = [&](int q) { return q == 0 ? v0 : (q == 1 ? v1 : v2); };
          bool acc = false;
          if (c == 0) beta_comp_u<DT, true>(bk.c[0], type0, uf, ud, acc);
          else beta_comp_u<DT, true>(bk.c[1], type1, uf, ud, acc);
          accepted |= (acc ? 1u : 0u) << i;
        }
        __syncwarp();
      }
      for (int i = 0; i < L; ++i) {
        const int x = x0 + i;
        const uint32_t bal = __ballot_sync(FULL, (accepted >> i) & 1u);
        if (x < to && j == 0)
          pmask[(ONE ? 0 : c) * kBetaRing + ((rm + x) & (kBetaRing - 1))] =
              (uint8_t)((bal >> (threadIdx.x & 31 & ~(P - 1))) & ((1u << P) - 1));
      }
    }
  };
  // ONE: the visits that start at positions [from, to): byte f of a position's
  // entry is the visit with f carried lanes, 16 trials + 8 (ends with a full
  // trial) + lanes carried after it; 0: more than 15 trials.  After n trials
  // with S accepted lanes the visits with f >= P - S are over.
  using E = typename std::conditional<P == 8, uint64_t, uint32_t>::type;
  auto build = [&](int64_t from, int64_t to, int t, int T) {
    constexpr E kOnes = (E)0x0101010101010101ull, kPat = (E)0x0706050403020100ull;
    for (int64_t x = from + t; x < to; x += T) {
      E w = 0, over = 0;
      int S = 0;
      for (int n = 1; n < 16; ++n) {
        const int m = __popc(pmask[(int)((x + (int64_t)(n - 1) * Ur) & (kBetaRing - 1))]);
        if (m == P) {
          w |= ((kPat + (E)S * kOnes) | (E)(16 * n + 8) * kOnes) & ~over;
          over = ~(E)0;
        } else {
          S += m;
          const E now = (S >= P ? ~(E)0 : S > 0 ? ~(E)0 << (8 * (P - S)) : (E)0) & ~over;
          const E after = S >= P ? kPat + (E)(S - P) * kOnes : S > 0 ? kPat << (8 * (P - S)) : (E)0;
          w |= (after | (E)(16 * n) * kOnes) & now;
          over |= now;
        }
        if (over == ~(E)0) break;
      }
      reinterpret_cast<E*>(visits)[(int)(x & (kBetaRing - 1))] = w;
    }
  };
  // block 0 and its masks (all threads)
  mt_block(raw[2], raw[0], [&](int, const uint64_t*) {});
  set_ring(0);
  // (ONE: a short call's, no more than it should need; up to 16 outputs go without
  // look-ups)
  const bool looks = ONE && Npk > 16;
  int64_t M = kN - umax + 1;  // positions with masks
  if (ONE) M = min(M, (looks ? 16 * Ur : 0) + 32 + (Uc + 3 * Ur) * min(Npk, (int64_t)kN));
  masks(0, M, tid, NT);
  __syncthreads();
  if (looks) {
    build(0, M - 16 * Ur, tid, NT);
    __syncthreads();
  }

  // chase state (warp 0, the same in every lane)
  int64_t cx = 0, cE = 0;
  int cf[2] = {0, 0};
  if (warp == 0) {
    cf[0] = gs->s[1].rest_cnt;
    cf[1] = gs->s[2].rest_cnt;
  }
  int64_t B = 0;  // newest block generated
  bool done = false;
  for (int64_t t = 0;; ++t) {
    const bool gen = !done && t + 1 < max_blocks;
    if (warp == 0) {
      if (!done) {
        // ---- chase step t into buffer t mod 2
        const int q = (int)(t & 1);
        const int64_t pk_lim = (t + 1) * kN;  // packets generated
        int16_t* rq = rec + q * kBcRec * 2;
        int16_t* fq = fpos + q * kBcFull;
        uint16_t* tq = ptask + q * 2 * LB;
        const int64_t base = cx, e0 = cE;
        const int fs0 = cf[0], fs1 = cf[1];
        int nrec = 0, nf = 0, A[2] = {cf[0], cf[1]};
        const bool lag = cx < (t - 1) * kN;
        const int Mr = (int)(M - base), bm = (int)(base & (kBetaRing - 1));
        if (ONE && !lag) {
          // one look-up per output; every trial of a visit that starts below
          // Mr - 16 Ur has its mask
          const int64_t rest = Npk - cE;
          const int pkr = (int)(pk_lim - base), left = (int)min(rest, (int64_t)kBcRec);
          int xr = 0, f = cf[rc], At = f;
          while (looks && nrec < left) {
            const int xt = rc == 0 ? xr : xr + Uc;
            if (xt >= Mr - 16 * Ur || At + 2 * P > LB || nf >= kBcFull) break;
            const uint32_t v = visits[((bm + xt) & (kBetaRing - 1)) * P + f];
            int nt = v >> 4, full = (v >> 3) & 1, f2 = v & 7;
            if (nt == 0) {  // a long visit: trial by trial
              int acc = 0, cn = 0, y = xt;
              bool end = false;
              for (; y < Mr && nt < 127 && !end; y += Ur) {
                cn = __popc(pmask[(bm + y) & (kBetaRing - 1)]);
                ++nt;
                if (cn == P) full = 1;
                else acc += cn;
                end = full || f + acc >= P;
              }
              if (!end) break;
              f2 = full ? f + acc : f + acc - P;
            }
            const int xe = xr + Uc + nt * Ur;
            if (xe > pkr) break;
            if (lane == 0)
              xrec[q * kBcRec + nrec] = (uint64_t)(uint32_t)(xt | At << 16) |
                                        (uint64_t)(uint32_t)(nf | (nt | full << 7) << 8 | f << 16) << 32;
            At += full ? f2 - f : f2 + P - f;
            nf += full;
            f = f2;
            xr = xe;
            ++nrec;
          }
          // the call's last outputs go trial by trial to the end of the masks: left for
          // the next step they cost a block, and the way back from it (96 packets of
          // beta(0.5, 2) on 64 engines, us, float / double: 42 / 49, 29 / 34 so)
          if (rest - nrec <= 16) {
#pragma unroll 1
            while (nrec < left && At + 2 * P <= LB && nf < kBcFull) {
              const int xt = rc == 0 ? xr : xr + Uc;
              int nt = 0, acc = 0, full = 0;
              bool end = false;
#pragma unroll 1
              for (int y = xt; y < Mr && nt < 127 && !end; y += Ur) {
                const int cn = __popc(pmask[(bm + y) & (kBetaRing - 1)]);
                ++nt;
                if (cn == P) full = 1;
                else acc += cn;
                end = full || f + acc >= P;
              }
              const int xe = xr + Uc + nt * Ur;
              if (!end || xe > pkr) break;
              if (lane == 0)
                xrec[q * kBcRec + nrec] = (uint64_t)(uint32_t)(xt | At << 16) |
                                          (uint64_t)(uint32_t)(nf | (nt | full << 7) << 8 | f << 16) << 32;
              At += acc;
              nf += full;
              f += full ? acc : acc - P;
              xr = xe;
              ++nrec;
            }
          }
          A[rc] = At;
          cf[rc] = f;
          cx = base + xr;
          cE += nrec;
        }
        if (!ONE && !lag) {
          while (cE < Npk && nrec < kBcRec) {
            const int64_t xs = cx;
            const int cf0 = cf[0], cf1 = cf[1], A0 = A[0], A1 = A[1], nfs = nf;
            // one component of record nrec: 0 done, 1 a buffer is full,
            // 2 positions not evaluated or packets not generated yet
            auto visit = [&](auto cc) -> int {
              constexpr int c = decltype(cc)::value;
              const int ty = c == 0 ? type0 : type1, U = c == 0 ? U0 : U1;
              if (ty <= 1) {
                if (cx + U > pk_lim) return 2;
                if (lane == 0) rq[nrec * 2 + c] = (int16_t)(cx - base);
                cx += U;
                return 0;
              }
              const int fsc = c == 0 ? fs0 : fs1;
              int acc = 0;
              int xr = (int)(cx - base);  // trial position relative to the step
              for (;;) {
                if (xr >= Mr) return 2;
                const uint32_t m = pmask[c * kBetaRing + ((bm + xr) & (kBetaRing - 1))];
                const int cn = __popc(m);
                if (cn == P) {  // a full trial ends the visit; the partial lanes stay carried
                  if (c == bc) {
                    if (nf >= kBcFull) return 1;
                    if (lane == 0) {
                      fq[nf] = (int16_t)xr;
                      rq[nrec * 2 + c] = (int16_t)(kBcFullTag + nf);
                    }
                    ++nf;
                  } else if (lane == 0) {
                    rq[nrec * 2 + c] = (int16_t)xr;
                  }
                  cf[c] += acc;
                  break;
                }
                if (A[c] + acc + cn > LB) return 1;
                // FIFO slots of the trial's accepted lanes
                if (lane < P && ((m >> lane) & 1u))
                  tq[c * LB + A[c] + acc - fsc + __popc(m & ((1u << lane) - 1u))] = (uint16_t)((xr << 3) | lane);
                acc += cn;
                if (cf[c] + acc >= P) {  // the carry fills: its oldest P lanes are the output
                  if (lane == 0) rq[nrec * 2 + c] = (int16_t)(-(1 + (A[c] - cf[c])));
                  cf[c] += acc - P;
                  break;
                }
                xr += U;
              }
              A[c] += acc;
              cx = base + xr + U;
              return 0;
            };
            int r = visit(std::integral_constant<int, 0>{});
            if (!r) r = visit(std::integral_constant<int, 1>{});
            if (r) {
              cx = xs;
              cf[0] = cf0;
              cf[1] = cf1;
              A[0] = A0;
              A[1] = A1;
              nf = nfs;
              break;
            }
            ++nrec;
            ++cE;
          }
        }
        if (lane == 0) {
          BcStep& S = s_step[q];
          S.base = base;
          S.e0 = e0;
          S.nrec = nrec;
          S.nf = nf;
          S.fs[0] = fs0;
          S.fs[1] = fs1;
          S.A[0] = A[0];
          S.A[1] = A[1];
          S.f[0] = cf[0];
          S.f[1] = cf[1];
          if (lag) s_err = 1;
          if (cE >= Npk) {
            s_done = 1;
            s_end = cx;
          }
        }
      }
    } else {
      const int tt = tid - 32;
      if (t >= 1 && s_step[(t - 1) & 1].nrec > 0) {
        // ---- step t - 1: values and outputs
        const int q = (int)((t - 1) & 1);
        const BcStep& S = s_step[q];
        const int nrec = S.nrec, nf = S.nf;
        const int fs0 = S.fs[0], fs1 = S.fs[1];
        const int64_t base = S.base;
        const int16_t* rq = rec + q * kBcRec * 2;
        uint16_t* tq = ptask + q * 2 * LB;
        set_ring(t);
        const int rbase = (int)(base - ring_new);
        if (ONE) {
          // the outputs' sources and the accepted partial lanes, in order
          const int bm = (int)(base & (kBetaRing - 1)), fs = rc == 0 ? fs0 : fs1;
          for (int i = tt; i < nrec; i += kBcWork) {
            const uint64_t v = xrec[q * kBcRec + i];
            const int x = (int)(v & 0xffff), Ai = (int)(v >> 16) & 0xffff, hi = (int)(v >> 32);
            const int nt = (hi >> 8) & 0x7f, full = (hi >> 15) & 1;
            int at = Ai - fs;
            for (int y = x; y < x + (nt - full) * Ur; y += Ur)
              for (uint32_t m = pmask[(bm + y) & (kBetaRing - 1)]; m; m &= m - 1) ptask[at++] = (uint16_t)((y << 3) | (__ffs(m) - 1));
            if (full) fpos[hi & 0xff] = (int16_t)(x + (nt - 1) * Ur);
            rec[i] = (int16_t)(full ? kBcFullTag + (hi & 0xff) : -(1 + Ai - (hi >> 16)));
          }
          asm volatile("bar.sync 1, %0;" ::"r"(kBcWork) : "memory");
        }
        // one task list, one lane per thread: full trials of the buffered
        // component, the accepted partial-trial lanes, positional values of
        // the other component
        const int t0 = nf * P, tp0 = S.A[0] - fs0, tp1 = S.A[1] - fs1;
        const int t1 = t0 + tp0 + tp1;
        for (int u = tt; u < t1 + nrec * P; u += kBcWork) {
          int c, j, rel;
          V* dst;
          if (u < t0) {
            const int i = u / P;
            j = u % P;
            c = bc;
            rel = fpos[(ONE ? 0 : q * kBcFull) + i];
            dst = fullval + i * P + j;
          } else if (u < t1) {
            c = u < t0 + tp0 ? 0 : 1;
            const int qq = c == 0 ? u - t0 : u - t0 - tp0;
            const int tk = ONE ? ptask[qq] : tq[c * LB + qq];
            j = tk & 7;
            rel = tk >> 3;
            dst = lanebuf + (ONE ? 0 : c * LB) + (c == 0 ? fs0 : fs1) + qq;
          } else {
            const int i = (u - t1) / P;
            j = (u - t1) % P;
            c = ob;
            if (ONE) {
              const uint64_t v = xrec[q * kBcRec + i];
              rel = (int)(v & 0xffff) + (rc == 0 ? ((int)(v >> 40) & 0x7f) * Ur : -Uc);
            } else {
              rel = rq[i * 2 + ob];
            }
            dst = (rel >= 0 && rel < kBcFullTag) ? posval + i * P + j : nullptr;
          }
          if (dst) *dst = (V)value_task(c, rbase + rel, j);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(kBcWork) : "memory");
        // output packets
        const int64_t e0 = S.e0;
        for (int u = tt; u < nrec * P; u += kBcWork) {
          const int i = u / P, j = u % P;
          uint64_t v[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (ONE && c == ob) {
              v[c] = (uint64_t)posval[i * P + j];
              continue;
            }
            const int src = ONE ? rec[i] : rq[i * 2 + c];
            if (src < 0) v[c] = (uint64_t)lanebuf[(ONE ? 0 : c * LB) + (-src - 1) + j];
            else if (src >= kBcFullTag) v[c] = (uint64_t)fullval[(src - kBcFullTag) * P + j];
            else if (c == ob) v[c] = (uint64_t)posval[i * P + j];
            else v[c] = value(c, rbase + src, j);  // both components closed form
          }
          if (DT == SD_F32) {
            const float p1 = u2f((uint32_t)v[0]), p2 = u2f((uint32_t)v[1]);
            const float x = p1 / (p1 + p2);
            reinterpret_cast<float*>(p.out)[off + (e0 + i) * P + j] = post ? (bk.fpost * x) / (1.0f - x) : x;
          } else {
            const double p1 = u2d(v[0]), p2 = u2d(v[1]);
            const double x = div_d(p1, p1 + p2);
            reinterpret_cast<double*>(p.out)[off + (e0 + i) * P + j] = post ? div_d(bk.dpost * x, 1.0 - x) : x;
          }
        }
        // lanes still carried move to the front of each lane buffer
        V carry = 0;
        const int cc = tt / 8, cj = tt % 8;
        const bool mover = tt < 16 && cj < S.f[cc];
        V* lb = lanebuf + (ONE ? 0 : cc * LB);
        if (mover) carry = lb[S.A[cc] - S.f[cc] + cj];
        asm volatile("bar.sync 1, %0;" ::"r"(kBcWork) : "memory");
        if (mover) lb[cj] = carry;
      }
      if (gen) {
        // ---- block t + 1 and its masks.  Word i < 156 of the new block needs
        // only the old block; word 156 + i needs new word i, which the same
        // thread made (word 311 needs new word 0: recomputed), so the twist
        // needs no barrier of its own
        uint64_t(*old)[kN] = raw[t % 3];
        uint64_t(*nw)[kN] = raw[(t + 1) % 3];
        for (int i = tt; i < kM; i += kBcWork) {
#pragma unroll
          for (int l = 0; l < kLanes; ++l) {
            const uint64_t lo = mt_twist(old[l][i], old[l][i + 1], old[l][i + kM]);
            const uint64_t n0 = i == kM - 1 ? mt_twist(old[l][0], old[l][1], old[l][kM]) : 0;
            const uint64_t hi = mt_twist(old[l][i + kM], i == kM - 1 ? n0 : old[l][i + kM + 1], lo);
            nw[l][i] = lo;
            nw[l][i + kM] = hi;
          }
        }
        asm volatile("bar.sync 1, %0;" ::"r"(kBcWork) : "memory");
        set_ring(t + 1);
        const int64_t M1 = (t + 2) * kN - umax + 1;
        masks(M, M1, tt, kBcWork);
        if (looks) {
          asm volatile("bar.sync 1, %0;" ::"r"(kBcWork) : "memory");
          build(M - 16 * Ur, M1 - 16 * Ur, tt, kBcWork);
        }
      }
    }
    __syncthreads();
    if (gen) M = (t + 2) * kN - umax + 1;
    if (done || s_err) break;
    done = s_done != 0;
    if (gen) B = t + 1;
    if (!done && !gen) break;  // no block left for the chase: the iteration cap
  }

  // ---- state after the call
  if (tid == 0) {
    if (!s_done) s_end = cx;
    if (!s_done || s_err) atomicOr(&st->status, (int)GR_DEV_REJECT_LIMIT);
    s_fc[0] = cf[0];
    s_fc[1] = cf[1];
  }
  __syncthreads();
  const int64_t np = s_end;  // packets consumed
  if (np > 0) {
    const int64_t lastb = (np - 1) / kN;
    const int rr = (int)(np - lastb * kN);  // in [1, 312]
    if (lastb == B) {
      store_window(st, raw[B % 3], raw[(B + 2) % 3], rr);
    } else if (lastb == B - 1) {
      store_window(st, raw[(B + 2) % 3], raw[(B + 1) % 3], rr);
    } else if (lastb == B - 2 && B >= 2) {
      // block B - 3 was overwritten by block B: recover it from block B - 2
      // into block B's window (MT19937-64's twist inverts)
      if (tid < kLanes) {
        uint64_t* nwl = raw[(B + 1) % 3][tid];
        uint64_t* odl = raw[B % 3][tid];
        mt_untwist_block([&](int i) -> uint64_t& { return nwl[i]; }, [&](int i) -> uint64_t& { return odl[i]; });
      }
      __syncthreads();
      store_window(st, raw[(B + 1) % 3], raw[B % 3], rr);
    } else if (tid == 0) {
      atomicOr(&st->status, (int)GR_DEV_BAD_INPUT);
    }
  }
  if (tid < 2 * 8) {
    const int c = tid / 8, j = tid % 8;
    GenSlot& g = gs->s[1 + c];
    const uint64_t v = j < s_fc[c] && (!ONE || c == rc) ? (uint64_t)lanebuf[(ONE ? 0 : c) * LB + j] : 0;
    if (DT == SD_F64) {
      g.rest[2 * j] = (uint32_t)v;
      g.rest[2 * j + 1] = (uint32_t)(v >> 32);
    } else {
      g.rest[j] = (uint32_t)v;
    }
  }
  __syncthreads();
  if (tid == 0) {
    gs->s[1].rest_cnt = s_fc[0];
    gs->s[2].rest_cnt = s_fc[1];
    st->consumed += (uint64_t)max(np, (int64_t)0);
  }
}

template <int DT>
static cudaError_t run_beta(const Plan& p, const DistParams& d, int64_t max_blocks, cudaStream_t s) {
  BetaConsts bk;
  bk.c[0] = beta_component(d.ia, d.fa, d.da);
  bk.c[1] = beta_component(d.ib, d.fb, d.db);
  bk.post = d.post;
  bk.fpost = d.fh;
  bk.dpost = d.dh;
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  constexpr size_t smem = bc_smem_bytes<DT, false>(), smem1 = bc_smem_bytes<DT, true>();
  if (!attr[dev]) {
    constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_beta<DT, -1, -1, false>, kAttr, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_beta<DT, -1, -1, true>, kAttr, (int)smem1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_beta<DT, 2, 1, true>, kAttr, (int)smem1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_beta<DT, 1, 2, true>, kAttr, (int)smem1);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  // the GS + integral-alpha pairs (beta(a < 1, integer b) and the mirror)
  // have kernels of their own
  const int t0 = bk.c[0].type, t1 = bk.c[1].type;
  if (t0 == 2 && t1 == 1) k_beta<DT, 2, 1, true><<<p.K, kBcThreads, smem1, s>>>(p, bk, max_blocks);
  else if (t0 == 1 && t1 == 2) k_beta<DT, 1, 2, true><<<p.K, kBcThreads, smem1, s>>>(p, bk, max_blocks);
  else if ((t0 >= 2) != (t1 >= 2)) k_beta<DT, -1, -1, true><<<p.K, kBcThreads, smem1, s>>>(p, bk, max_blocks);
  else k_beta<DT, -1, -1, false><<<p.K, kBcThreads, smem, s>>>(p, bk, max_blocks);
  return cudaGetLastError();
}


// ===========================================================================
// k_uniform_int: UniformIntGen<int32_t>(min, max) whose range is not a power
// of two (Discrete.h:296-331).  Each output packet starts a fresh
// rx = rng.half(), tries its bit slices (the low `bits` bits, then rx >> bits
// while bitcnt + bits < 32) through CompressMask, and draws again until a
// packet is full; a packet with all four lanes accepted is returned as is and
// leaves the carried lanes alone.  One CTA per engine: all threads twist and
// temper a block into its 624 half-packet draws, then thread 0 runs the
// automaton over them (a few integer operations per slice).  A range of one
// value draws nothing and writes the constant.
// ===========================================================================
namespace {
constexpr int kUiThreads = 160;
}

__global__ void __launch_bounds__(kUiThreads) k_uniform_int(Plan p, DistParams d, int64_t max_blocks) {
  __shared__ uint64_t raw[2][kLanes][kN];
  __shared__ uint32_t hw[2 * kN][4];  // draw 2i: low half of packet i, 2i + 1: high half
  __shared__ int s_done;
  __shared__ int s_last;              // last draw consumed in the newest block, or -1
  const int k = blockIdx.x;
  const int tid = threadIdx.x;
  EngState* st = p.eng + k;
  GenSlot* gsl = &p.gen[k].s[0];
  const int64_t g0 = (int64_t)k * p.gran_per_k + min((int64_t)k, p.gran_rem);
  const int64_t ng = p.gran_per_k + ((int64_t)k < p.gran_rem ? 1 : 0);
  const int64_t off = g0 * p.gran, n = ng * p.gran;
  if (n == 0) return;
  int32_t* out = reinterpret_cast<int32_t*>(p.out) + off;
  const int32_t pmin = d.ia;
  if (d.ib == 0) {  // pdiff == 0: pset1(pmin), no draws
    for (int64_t i = tid; i < n; i += kUiThreads) out[i] = pmin;
    return;
  }
  const uint32_t mask = d.bitmask;
  const int32_t plen = d.ic;
  const int bits = d.ncdf;
  const int64_t Npk = n / 4;

  // thread-0 automaton state: carried lanes and packets written
  uint32_t cache[8];
  int fc = 0;
  int64_t e = 0;
  auto put = [&](int64_t pk, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3) {
    int32_t* o = out + pk * 4;
    o[0] = (int32_t)(a0 + (uint32_t)pmin);
    o[1] = (int32_t)(a1 + (uint32_t)pmin);
    o[2] = (int32_t)(a2 + (uint32_t)pmin);
    o[3] = (int32_t)(a3 + (uint32_t)pmin);
  };
  // one rng.half() draw; true when it completed an output packet
  auto draw = [&](const uint32_t* w) -> bool {
    uint32_t rx[4] = {w[0], w[1], w[2], w[3]};
    int bitcnt = bits;
    for (;;) {
      uint32_t c[4];
      unsigned m = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        c[j] = rx[j] & mask;
        if ((int32_t)c[j] < plen) m |= 1u << j;
      }
      if (m == 15u) {
        put(e++, c[0], c[1], c[2], c[3]);
        return true;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((m >> j) & 1u) cache[fc++] = c[j];
      if (fc >= 4) {
        put(e++, cache[0], cache[1], cache[2], cache[3]);
#pragma unroll
        for (int j = 0; j < 3; ++j) cache[j] = cache[j + 4];
        fc -= 4;
        return true;
      }
      if (bitcnt + bits < 32) {
#pragma unroll
        for (int j = 0; j < 4; ++j) rx[j] >>= bits;
        bitcnt += bits;
      } else {
        return false;
      }
    }
  };

  load_window(raw[0], &st->win[0][0], kN);
  const int hv = st->half_valid;
  if (tid == 0) {
    fc = min(max(gsl->rest_cnt, 0), 3);  // at most P - 1 lanes are ever carried
    for (int j = 0; j < fc; ++j) cache[j] = gsl->rest[j];
    s_done = 0;
    s_last = -1;
    if (hv) {  // the engine's cached half is the first draw
      uint32_t w[4];
      for (int j = 0; j < 4; ++j) w[j] = st->half_cache[j];
      draw(w);
      if (e >= Npk) s_done = 1;
    }
  }
  __syncthreads();
  int cur = 0;
  int64_t nb = 0;
  for (; nb < max_blocks && !s_done; ++nb) {
    mt_block(raw[cur], raw[cur ^ 1], [&](int i, const uint64_t* pk) {
      hw[2 * i][0] = (uint32_t)pk[0];
      hw[2 * i][1] = (uint32_t)(pk[0] >> 32);
      hw[2 * i][2] = (uint32_t)pk[1];
      hw[2 * i][3] = (uint32_t)(pk[1] >> 32);
      hw[2 * i + 1][0] = (uint32_t)pk[2];
      hw[2 * i + 1][1] = (uint32_t)(pk[2] >> 32);
      hw[2 * i + 1][2] = (uint32_t)pk[3];
      hw[2 * i + 1][3] = (uint32_t)(pk[3] >> 32);
    });
    cur ^= 1;
    if (tid == 0) {
      for (int h = 0; h < 2 * kN; ++h) {
        draw(hw[h]);
        if (e >= Npk) {
          s_last = h;
          s_done = 1;
          break;
        }
      }
    }
    __syncthreads();
  }

  // ---- state after the call
  const int last = s_last;
  if (last >= 0) {  // draws of the newest block were consumed: packets up to last / 2
    const int rr = last / 2 + 1;
    store_window(st, raw[cur], raw[cur ^ 1], rr);
  }
  if (tid == 0) {
    if (!s_done) atomicOr(&st->status, (int)GR_DEV_REJECT_LIMIT);
    if (last >= 0) {
      const int64_t np = (nb - 1) * kN + last / 2 + 1;
      st->consumed += (uint64_t)np;
      if ((last & 1) == 0) {  // the high half of the last packet stays in the half() cache
        for (int j = 0; j < 4; ++j) st->half_cache[j] = hw[last + 1][j];
        st->half_valid = 1;
      } else {
        st->half_valid = 0;
      }
    } else if (hv) {
      st->half_valid = 0;  // only the cached half was drawn
    }
    gsl->rest_cnt = fc;
    for (int j = 0; j < fc; ++j) gsl->rest[j] = cache[j];
  }
}

static cudaError_t run_uniform_int(const Plan& p, const DistParams& d, int64_t max_blocks, cudaStream_t s) {
  k_uniform_int<<<p.K, kUiThreads, 0, s>>>(p, d, max_blocks);
  return cudaGetLastError();
}

// ===========================================================================
// k_negbin: NegativeBinomialGen<int32_t>(trials, p) (GammaPoisson.h:42-98).
// Per output packet: a Packet4f GammaGen((float)trials, (float)((1-p)/p))
// draw over rng.half() words (NormalExp.h:568-604), then a Poisson draw with
// those per-lane means: the multiplicative loop while no lane's mean exceeds
// 12, else tan rejection whose CompressMask carry is the GammaGen's.  One
// warp per engine: the warp twists its own engine blocks into 624
// half-packet draws, and lanes 0-3 run the packet code in lock step (one
// lane per packet lane, decisions by ballot).
// ===========================================================================
namespace {
constexpr int kNbWarps = 1;  // engines per CTA (30 KB of shared memory each: 7 CTAs per SM)
constexpr size_t kNbWarpBytes = (size_t)2 * kLanes * kN * 8 + (size_t)2 * kN * 16 + 64;  // windows, draws, carry
}

__global__ void __launch_bounds__(32 * kNbWarps) k_negbin(Plan p, DistParams d, int64_t max_blocks) {
  extern __shared__ __align__(16) uint64_t nb_dyn[];
  const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x * kNbWarps + wi;
  if (k >= p.K) return;  // the whole warp
  uint8_t* base = reinterpret_cast<uint8_t*>(nb_dyn) + (size_t)wi * kNbWarpBytes;
  uint64_t(*raw)[kLanes][kN] = reinterpret_cast<uint64_t(*)[kLanes][kN]>(base);
  uint32_t(*hw)[4] = reinterpret_cast<uint32_t(*)[4]>(base + (size_t)2 * kLanes * kN * 8);
  uint32_t* carry = reinterpret_cast<uint32_t*>(base + (size_t)2 * kLanes * kN * 8 + (size_t)2 * kN * 16);
  EngState* st = p.eng + k;
  GenSlot* gsl = &p.gen[k].s[0];
  const int64_t g0 = (int64_t)k * p.gran_per_k + min((int64_t)k, p.gran_rem);
  const int64_t ng = p.gran_per_k + ((int64_t)k < p.gran_rem ? 1 : 0);
  const int64_t off = g0 * p.gran, n = ng * p.gran;
  if (n == 0) return;
  int32_t* out = reinterpret_cast<int32_t*>(p.out) + off;
  const int64_t Npk = n / 4;
  const float alpha = d.fa, beta = d.fb, gsq = d.fc, a1 = d.fd;
  const int count = d.ia, mode = d.ic;  // mode 0: alpha == 1, 1: product of count uniforms, 2: tan rejection
  const float eps8 = 1.1920928955078125e-07f / 8;
  const float fpi = (float)3.1415926535897932;
  (void)alpha;

  for (int i = lane; i < kLanes * kN; i += 32) raw[0][i / kN][i % kN] = st->win[i / kN][i % kN];
  int fc = min(max(gsl->rest_cnt, 0), 3);
  if (lane < fc) carry[lane] = gsl->rest[lane];
  __syncwarp();

  // draws: the engine's cached half first, then the halves of new blocks
  bool pending = st->half_valid != 0, abort = false;
  int h = 2 * kN, cur = 0;
  int64_t nb = 0;
  auto next = [&]() -> uint32_t {
    if (pending) {
      pending = false;
      return lane < 4 ? st->half_cache[lane] : 0u;
    }
    if (h == 2 * kN) {
      if (nb >= max_blocks) {
        abort = true;
        return 0u;
      }
      __syncwarp();
      uint64_t(*old)[kN] = raw[cur];
      uint64_t(*nw)[kN] = raw[cur ^ 1];
#pragma unroll 1
      for (int ph = 0; ph < 2; ++ph) {
        for (int ii = lane; ii < kM; ii += 32) {
          const int i = ph * kM + ii;
          uint64_t pk[kLanes];
#pragma unroll
          for (int l = 0; l < kLanes; ++l) {
            const uint64_t b = (i + 1 < kN) ? old[l][i + 1] : nw[l][0];
            const uint64_t c = (ph == 0) ? old[l][i + kM] : nw[l][i - kM];
            const uint64_t v = mt_twist(old[l][i], b, c);
            nw[l][i] = v;
            pk[l] = mt_temper(v);
          }
          hw[2 * i][0] = (uint32_t)pk[0];
          hw[2 * i][1] = (uint32_t)(pk[0] >> 32);
          hw[2 * i][2] = (uint32_t)pk[1];
          hw[2 * i][3] = (uint32_t)(pk[1] >> 32);
          hw[2 * i + 1][0] = (uint32_t)pk[2];
          hw[2 * i + 1][1] = (uint32_t)(pk[2] >> 32);
          hw[2 * i + 1][2] = (uint32_t)pk[3];
          hw[2 * i + 1][3] = (uint32_t)(pk[3] >> 32);
        }
        __syncwarp();
      }
      cur ^= 1;
      ++nb;
      h = 0;
    }
    const uint32_t v = lane < 4 ? hw[h][lane] : 0u;
    ++h;
    return v;
  };
  auto mask4 = [&](bool pr) -> unsigned { return __ballot_sync(0xffffffffu, pr && lane < 4) & 0xfu; };
  // CompressMask::compress_append over lanes 0-3 (arch/AVX/PacketFilter.h:147-184)
  auto compress = [&](uint32_t bits, bool acc, uint32_t& res) -> bool {
    const unsigned m = mask4(acc);
    if (m == 0xfu) {
      res = bits;
      return true;
    }
    if (lane < 4 && ((m >> lane) & 1u)) carry[fc + __popc(m & ((1u << lane) - 1))] = bits;
    fc += __popc(m);
    __syncwarp();
    if (fc < 4) return false;
    res = lane < 4 ? carry[lane] : 0u;
    const uint32_t mv = lane < fc - 4 ? carry[4 + lane] : 0u;
    __syncwarp();
    if (lane < fc - 4) carry[lane] = mv;
    fc -= 4;
    __syncwarp();
    return true;
  };

  int64_t e = 0;
  for (; e < Npk && !abort; ++e) {
    float mean = 0.0f;
    if (mode == 0) {
      mean = beta * (-(logf_(1.0f - ur_f(next())) / 1.0f));
    } else if (mode == 1) {
      float y = ur_f(next()) + eps8;
      for (int c = 1; c < count; ++c) y = y * (ur_f(next()) + eps8);
      mean = -(beta * logf_(y));
    } else {
      for (;;) {
        float ys, yc;
        sincosf_(fpi * ur_f(next()), ys, yc);
        const float ux = ur_f(next());
        if (abort) break;
        const float yx = ys / yc;
        const float xx = gsq * yx + a1;
        const float ub = (yx * yx + 1.0f) * expf_<true>(a1 * logf_(xx / a1) - yx * gsq);
        uint32_t r;
        if (compress(f2u(beta * xx), (0.0f < xx) && (ux <= ub), r)) {
          mean = u2f(r);
          break;
        }
      }
    }
    if (abort) break;
    const float pne = expf_<true>(-mean);
    if (mask4(12.0f < mean) == 0) {
      float val = 1.0f;
      int32_t res = 0;
      for (;;) {
        val = val * ur_f(next());
        if (abort) break;
        const bool c = pne < val;
        if (mask4(c) == 0) break;
        res += c ? 1 : 0;
      }
      if (abort) break;
      if (lane < 4) out[e * 4 + lane] = res;
    } else {
      const float sq = sqrtf(2.0f * mean), lm = logf_(mean), g1 = mean * lm - lgamma_approxf_(mean + 1.0f);
      for (;;) {
        float s, c;
        sincosf_(fpi * ur_f(next()), s, c);
        const float yx = s / c;
        const float fres = truncf(sq * yx + mean);
        const float p1 = (yx * yx + 1.0f) * 0.9f;
        const float u2 = ur_f(next());
        if (abort) break;
        const float p2 = expf_<true>((fres * lm - lgamma_approxf_(fres + 1.0f)) - g1);
        uint32_t r;
        if (compress(f2u(fres), (0.0f <= fres) && (u2 <= p1 * p2), r)) {
          if (lane < 4) out[e * 4 + lane] = cvtt_f32(u2f(r));
          break;
        }
      }
    }
  }

  // ---- state after the call
  if (abort) {
    if (lane == 0) atomicOr(&st->status, (int)GR_DEV_REJECT_LIMIT);
    return;
  }
  const bool used_block = nb > 0;  // the last draw came from the newest block (h >= 1)
  if (used_block) {
    const int last = h - 1;          // last draw consumed in the newest block
    const int rr = last / 2 + 1;     // packets used of it
    uint64_t(*lastb)[kN] = raw[cur];
    uint64_t(*prevb)[kN] = raw[cur ^ 1];
    for (int t = lane; t < kLanes * kN; t += 32) {
      const int l = t / kN, i = t % kN;
      st->win[l][i] = (i < kN - rr) ? prevb[l][rr + i] : lastb[l][i - (kN - rr)];
    }
    if (lane < 4) st->half_cache[lane] = (last & 1) == 0 ? hw[last + 1][lane] : 0u;
    if (lane == 0) {
      st->half_valid = (last & 1) == 0 ? 1 : 0;
      st->consumed += (uint64_t)((nb - 1) * kN + rr);
    }
  } else if (lane == 0 && st->half_valid && Npk > 0) {
    st->half_valid = 0;  // only the cached half was drawn
  }
  if (lane < fc) gsl->rest[lane] = carry[lane];
  if (lane == 0) gsl->rest_cnt = fc;
}

static cudaError_t run_negbin(const Plan& p, const DistParams& d, int64_t max_blocks, cudaStream_t s) {
  constexpr size_t smem = kNbWarpBytes * kNbWarps;
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr[dev]) {
    cudaError_t e = cudaFuncSetAttribute(k_negbin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  k_negbin<<<(p.K + kNbWarps - 1) / kNbWarps, 32 * kNbWarps, smem, s>>>(p, d, max_blocks);
  return cudaGetLastError();
}

cudaError_t launch_walk(const Plan& p, const DistParams& d, int64_t max_blocks, cudaStream_t s) {
  if (d.kind == GR_NEGATIVE_BINOMIAL) return run_negbin(p, d, max_blocks, s);
  if (d.kind == GR_UNIFORM_INT) return run_uniform_int(p, d, max_blocks, s);
  if (d.dtype == GR_I32) return run_poisson(p, d, max_blocks, s);
  if (d.dtype == GR_F32) return run_beta<SD_F32>(p, d, max_blocks, s);
  if (d.dtype == GR_F64) return run_beta<SD_F64>(p, d, max_blocks, s);
  return cudaErrorNotSupported;
}

}  // namespace gr
