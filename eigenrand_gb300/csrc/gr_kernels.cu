// MT19937-64 packet engine and fused engine+transform kernels for sm_103a.
//
// Engine: each Vmt19937_64 has 4 MT19937-64 lanes (lane l = std::mt19937_64
// seeded seed+l), EigenRand/PacketRandomEngine.h:196-426.  One CTA owns one
// engine (or one jump-ahead segment of it): the 4 x 312-word lane states sit
// in shared memory, the twist runs in two phases of 156 independent words,
// and each thread tempers the 4 lane words of one packet index and turns them
// into output samples in registers, so raw bits never reach HBM.
//
// Jump-ahead: a segment starting e packets into the call gets its lane state
// from  window(a+e) = sum_i c_i * window(a+i),  c = x^e mod P(x)  (P the
// characteristic polynomial of MT19937-64), i.e. a GF(2) correlation of the
// polynomial's coefficients with the lane's next 20k raw words (the "prefix").
#include <cuda_runtime.h>

#include <cstdint>

#include "gr_exact.h"
#include "gr_internal.h"
#include "gr_kernels.cuh"
#include "gr_math.cuh"
#include "../../include/gpurand.h"

namespace gr {

// The twist and the tempering in 32-bit halves: 6 + 12 instructions of the logic
// pipe and 2 products.  Uniform floats, 8192 x 8192 on 608 engines: 66 us, 73
// with the 64-bit expressions that the other kernels use (gr_mt.cuh), where
// these cost 1 to 2 % instead (integral gamma, binomial; the products wait for
// the pipe that the addressing uses).
__device__ __forceinline__ uint64_t twist1(uint64_t a, uint64_t b, uint64_t c) {
  const uint32_t ah = (uint32_t)(a >> 32), bl = (uint32_t)b, odd = bl & 1u;
  const uint32_t tl = ((uint32_t)a & 0x80000000u) | (bl & 0x7fffffffu);
  const uint32_t lo = __funnelshift_r(tl, ah, 1) ^ (odd * (uint32_t)kMatA) ^ (uint32_t)c;
  const uint32_t hi = (ah >> 1) ^ (odd * (uint32_t)(kMatA >> 32)) ^ (uint32_t)(c >> 32);
  return (uint64_t)lo | (uint64_t)hi << 32;
}
static_assert(kUpper == ~0ull << 31, "the halves above");

__device__ __forceinline__ uint64_t temper(uint64_t r) {
  uint32_t lo = (uint32_t)r, hi = (uint32_t)(r >> 32);
  lo ^= __funnelshift_r(lo, hi, 29) & 0x55555555u;
  hi ^= (hi >> 29) & 0x55555555u;
  const uint32_t l0 = lo;
  lo ^= (lo << 17) & 0xeda60000u;
  hi ^= __funnelshift_l(l0, hi, 17) & 0x71d67fffu;
  hi ^= (lo << 5) & 0xfff7eee0u;
  lo ^= hi >> 11;
  return (uint64_t)lo | (uint64_t)hi << 32;
}

// ---------------------------------------------------------------- seeding
// MersenneTwister::seed, PacketRandomEngine.h:256-265; engine k lane l is
// seeded seed + 4k + l.
__global__ void k_seed(EngState* st, int K, uint64_t seed) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= K * kLanes) return;
  int k = t / kLanes, l = t % kLanes;
  uint64_t prev = seed + (uint64_t)kLanes * (uint64_t)k + (uint64_t)l;
  uint64_t* w = st[k].win[l];
  w[0] = prev;
  for (int i = 1; i < kN; ++i) {
    prev = (prev ^ (prev >> 62)) * kSeedF + (uint64_t)i;
    w[i] = prev;
  }
  if (l == 0) {
    st[k].half_valid = 0;
    st[k].status = 0;
    st[k].consumed = 0;
    for (int q = 0; q < kLanes; ++q) st[k].half_cache[q] = 0;
  }
}

cudaError_t launch_seed(EngState* st, int K, uint64_t seed, cudaStream_t s) {
  int n = K * kLanes;
  k_seed<<<(n + 127) / 128, 128, 0, s>>>(st, K, seed);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- word streams
// The recurrence x[i+312] = twist(x[i], x[i+1], x[i+156]) gives 156 words at a
// time (a phase).  A word's own two predecessors x[i], x[i+156] are the words
// the same thread made two phases and one phase before, so they stay in
// registers and only x[i+1], two phases old, comes from the next lane by a
// shuffle: no shared memory and no barrier between phases.
__device__ __forceinline__ uint64_t xor64(uint64_t v, int m) {
  return ((uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)(v >> 32), m) << 32) |
         (uint64_t)__shfl_xor_sync(0xffffffffu, (uint32_t)v, m);
}
__device__ __forceinline__ uint64_t shfl64(uint64_t v, int src) {
  return ((uint64_t)__shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src) << 32) |
         (uint64_t)__shfl_sync(0xffffffffu, (uint32_t)v, src);
}

// One MT19937-64 lane on four warps of a CTA, for calls with too few lanes to
// fill the GPU: warp w holds the phase's words [40 w, 40 w + 64), two per
// thread, of which the first 40 (36) are its own and the rest a halo that
// repeats the next warp's work.  The halo loses one word every two phases (its
// last word misses its neighbour), so the warps exchange words only every 48
// phases.  Bound by the logic pipe, at one warp per scheduler two cycles an
// instruction: some 24 of them per warp and phase.  Measured
// against the one-barrier-per-phase form (156 threads, three shared-memory
// reads per word): 20 280 words in 4.5 us against 17 us.
// win: the CTA's 312-word window in shared memory (loaded, all threads past
// a barrier); put(i, v0, v1) stores words i, i + 1 (i even) after the window.
constexpr int kWideThreads = 128;
template <class Put>
__device__ __forceinline__ void lane_words_wide(uint64_t* win, int64_t n, Put&& put) {
  const int w = threadIdx.x >> 5, q = threadIdx.x & 31;
  const int i0 = 40 * w + 2 * q;
  const bool own = q < 20 && i0 < kM;
  const int src = q < 31 ? q + 1 : 31;
  for (int64_t base = 0; base < n;) {
    uint64_t a[2], c[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int i = i0 + j;
      a[j] = win[i];
      // words past the window (the last warp's halo) are made here
      c[j] = i < kM ? win[kM + i] : twist1(win[i - kM], win[i - kM + 1], win[i]);
    }
    int ph = 0;
    if (n - base >= 48 * kM) {
      // the words' roles alternate: two phases per trip, without moves (131 072
      // words 31 us with them, 21 without; the shuffles a trip ahead: no change)
      for (; ph < 48; ph += 2) {
        const uint64_t n0 = shfl64(a[0], src);
        const uint64_t n1 = shfl64(c[0], src);
        a[0] = twist1(a[0], a[1], c[0]);
        a[1] = twist1(a[1], n0, c[1]);
        if (own) put(base + i0, a[0], a[1]);
        c[0] = twist1(c[0], c[1], a[0]);
        c[1] = twist1(c[1], n1, a[1]);
        if (own) put(base + kM + i0, c[0], c[1]);
        base += 2 * kM;
      }
    }
    const int phases = ph ? 48 : (int)min((int64_t)48, (n - base + kM - 1) / kM);
    for (; ph < phases; ++ph) {
      const uint64_t nb = shfl64(a[0], src);
      const uint64_t v0 = twist1(a[0], a[1], c[0]), v1 = twist1(a[1], nb, c[1]);
      const int64_t i = base + i0;
      if (own && i < n) put(i, v0, v1);
      a[0] = c[0];
      a[1] = c[1];
      c[0] = v0;
      c[1] = v1;
      base += kM;
    }
    if (base >= n) break;
    __syncthreads();
    if (own) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        win[i0 + j] = a[j];
        win[kM + i0 + j] = c[j];
      }
    }
    __syncthreads();
  }
}

// prefix[k][l][0..312) = current window, then the lane's next 20 280 raw words.
// Also snapshots the caches the call starts from (lane 0's CTA).
__device__ __forceinline__ void snap_caches(const EngState& st, const GenState* gen, CallSnap& snap) {
  snap.half_valid = st.half_valid;
  for (int q = 0; q < kLanes; ++q) snap.half_cache[q] = st.half_cache[q];
  snap.gen_valid = gen ? gen->s[0].valid : 0;
  for (int q = 0; q < 16; ++q) snap.gen_cache[q] = gen ? gen->s[0].cache[q] : 0u;
}

__global__ void __launch_bounds__(kWideThreads) k_prefix(const EngState* st, uint64_t* prefix, CallSnap* snap,
                                                         const GenState* gen) {
  __shared__ uint64_t win[kN];
  const int k = blockIdx.x / kLanes, l = blockIdx.x % kLanes;
  uint64_t* out = prefix + ((size_t)k * kLanes + l) * kPrefixLen;
  for (int i = threadIdx.x; i < kN; i += kWideThreads) out[i] = win[i] = st[k].win[l][i];
  if (snap && l == 0 && threadIdx.x == 0) snap_caches(st[k], gen ? gen + k : nullptr, snap[k]);
  __syncthreads();
  lane_words_wide(win, kPrefixLen - kN, [&](int64_t i, uint64_t v0, uint64_t v1) {
    *reinterpret_cast<ulonglong2*>(out + kN + i) = make_ulonglong2(v0, v1);
  });
}

// Raw words of a call into memory: words[(k * 4 + l) * stride + 312 + i] =
// raw word i of lane l of engine k (the window before them at [0, 312)), i <
// n, segment s of an engine making words [s J, (s + 1) J) from its jump
// window.  The transforms then run over the whole GPU whatever the number of
// engines (k_xform below, gr_chain.cu).  k_words_wide: one CTA per lane and
// segment; k_words_warp: one warp per lane and segment (26 threads of 6
// consecutive words per phase), 28% fewer instructions per word, where there
// are enough lanes to fill the GPU.
__global__ void __launch_bounds__(kWideThreads) k_words_wide(const EngState* st, const GenState* gen, WordsArgs a) {
  __shared__ uint64_t win[kN];
  const int l = blockIdx.x % kLanes, s = (blockIdx.x / kLanes) % a.S, k = blockIdx.x / (kLanes * a.S);
  uint64_t* out = a.words + ((size_t)k * kLanes + l) * a.stride;
  const uint64_t* src = s == 0 ? st[k].win[l] : a.segwin + (((size_t)k * (a.S - 1) + (s - 1)) * kLanes + l) * kN;
  for (int i = threadIdx.x; i < kN; i += kWideThreads) {
    win[i] = src[i];
    if (s == 0) out[i] = src[i];
  }
  if (a.snap && s == 0 && l == 0 && threadIdx.x == 0) snap_caches(st[k], gen ? gen + k : nullptr, a.snap[k]);
  __syncthreads();
  const int64_t i0 = (int64_t)s * a.J;
  uint64_t* o = out + kN + i0;
  lane_words_wide(win, min(a.J, a.n - i0), [&](int64_t i, uint64_t v0, uint64_t v1) {
    *reinterpret_cast<ulonglong2*>(o + i) = make_ulonglong2(v0, v1);
  });
}

__global__ void __launch_bounds__(32 * kLanes) k_words_warp(const EngState* st, const GenState* gen, WordsArgs a) {
  const int l = threadIdx.x >> 5, q = threadIdx.x & 31;
  const int s = blockIdx.x % a.S, k = blockIdx.x / a.S;
  uint64_t* out = a.words + ((size_t)k * kLanes + l) * a.stride;
  const uint64_t* src = s == 0 ? st[k].win[l] : a.segwin + (((size_t)k * (a.S - 1) + (s - 1)) * kLanes + l) * kN;
  if (s == 0)
    for (int i = q; i < kN; i += 32) out[i] = src[i];
  if (a.snap && s == 0 && threadIdx.x == 0) snap_caches(st[k], gen ? gen + k : nullptr, a.snap[k]);
  const int qq = min(q, 25);
  uint64_t x[6], c[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    x[j] = src[6 * qq + j];
    c[j] = src[kM + 6 * qq + j];
  }
  const int64_t i0 = (int64_t)s * a.J, n = min(a.J, a.n - i0);
  uint64_t* o = out + kN + i0;
  const int nsrc = q == 25 ? 0 : min(q + 1, 31);
  for (int64_t base = 0; base < n; base += kM) {
    // the last thread's neighbour is the first word of the next phase, one phase old
    const uint64_t nb = shfl64(q == 0 ? c[0] : x[0], nsrc);
    uint64_t v[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) v[j] = twist1(x[j], j < 5 ? x[j + 1] : nb, c[j]);
    const int64_t i = base + 6 * q;
    if (q < 26) {
#pragma unroll
      for (int j = 0; j < 6; j += 2)
        if (i + j < n) *reinterpret_cast<ulonglong2*>(o + i + j) = make_ulonglong2(v[j], v[j + 1]);
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      x[j] = c[j];
      c[j] = v[j];
    }
  }
}

cudaError_t launch_words(const EngState* st, const GenState* gen, int K, const WordsArgs& a, cudaStream_t s) {
  // four lanes of one warp each per CTA: the narrow form fills the SMs'
  // schedulers from about one CTA per SM on
  if ((int64_t)K * a.S >= 256) k_words_warp<<<K * a.S, 32 * kLanes, 0, s>>>(st, gen, a);
  else k_words_wide<<<K * a.S * kLanes, kWideThreads, 0, s>>>(st, gen, a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- jump
// segwin[k][s1][l][j] = XOR over the polynomial's set coefficients i of
// prefix word i + j.  One CTA per (engine, segment s >= 1, lane, part of the
// terms); its warps split the part, lane q of a warp covers output words
// [11 q, 11 q + 11) (an odd stride: the 8-byte shared-memory reads are free of
// bank conflicts).  A thread slides a register window over the prefix words;
// two coefficients at a time, the same for the whole warp, pick one of four
// unrolled cases: none, either word, or both in three-input XORs, 0.75 operations
// per 32-bit word for the two terms on average.  Parts meet by atomic XOR (segwin
// zeroed beforehand).  Bound by issue.
constexpr int kJumpThreads = 256;
constexpr int kJumpOut = 11;
// PARTS CTAs per segment and lane
template <int PARTS>
struct JumpDims {
  static constexpr int kPer = 19968 / (PARTS * (kJumpThreads / 32));  // terms per warp
  static constexpr int kSpan = kPer * (kJumpThreads / 32);            // terms per CTA
  static constexpr int kLoad = kSpan + 32 * kJumpOut + 8;             // prefix words a CTA reads
  static constexpr int kRed = (kJumpThreads / 32) * 32 * kJumpOut;    // the warps' sums, in the same memory
  static_assert(PARTS * kSpan == 19968 && kSpan % 64 == 0 && kPer % 8 == 0, "coefficient bytes stay within one word");
};

// acc[j] ^= the words of terms 0 / 1 (at w[j], w[j + 1]) whose coefficient
// bits are set; c is the same in every thread of the warp
__device__ __forceinline__ void xor_terms2(uint64_t (&acc)[kJumpOut], const uint64_t* w, uint32_t c) {
  if (c == 3) {
#pragma unroll
    for (int j = 0; j < kJumpOut; ++j) acc[j] ^= w[j] ^ w[j + 1];
  } else if (c == 1) {
#pragma unroll
    for (int j = 0; j < kJumpOut; ++j) acc[j] ^= w[j];
  } else if (c == 2) {
#pragma unroll
    for (int j = 0; j < kJumpOut; ++j) acc[j] ^= w[j + 1];
  }
}

template <int PARTS>
__global__ void __launch_bounds__(kJumpThreads, 4)
    k_jump(const uint64_t* prefix, const uint64_t* polys, int S, unsigned long long* segwin) {
  using D = JumpDims<PARTS>;
  constexpr int kJumpParts = PARTS, kJumpPer = D::kPer, kJumpSpan = D::kSpan, kJumpLoad = D::kLoad;
  __shared__ uint64_t px[kJumpLoad > D::kRed ? kJumpLoad : D::kRed];
  __shared__ uint64_t cf[kJumpSpan / 64];
  const int nseg = S - 1;
  const int part = blockIdx.x % kJumpParts;
  const int l = (blockIdx.x / kJumpParts) % kLanes;
  const int s1 = (blockIdx.x / (kJumpParts * kLanes)) % nseg;  // segment - 1
  const int k = blockIdx.x / (kJumpParts * kLanes * nseg);
  const int tid = threadIdx.x;
  const int t0 = part * kJumpSpan;
  const uint64_t* src = prefix + ((size_t)k * kLanes + l) * kPrefixLen + t0;
  for (int i = tid; i < kJumpLoad; i += kJumpThreads) px[i] = t0 + i < kPrefixLen ? src[i] : 0;
  for (int i = tid; i < kJumpSpan / 64; i += kJumpThreads) cf[i] = polys[(size_t)s1 * kN + t0 / 64 + i];
  __syncthreads();

  const int g = tid >> 5, q = tid & 31;
  const int ibeg = g * kJumpPer;
  const uint64_t* p = px + ibeg + kJumpOut * q;
  uint64_t acc[kJumpOut];
#pragma unroll
  for (int j = 0; j < kJumpOut; ++j) acc[j] = 0;
  uint64_t w[kJumpOut + 7];
#pragma unroll
  for (int m = 0; m < kJumpOut - 1; ++m) w[m] = p[m];
#pragma unroll 1
  for (int i0 = 0; i0 < kJumpPer; i0 += 8) {
#pragma unroll
    for (int m = 0; m < 8; ++m) w[kJumpOut - 1 + m] = p[i0 + kJumpOut - 1 + m];
    const uint32_t cb = (uint32_t)(cf[(ibeg + i0) >> 6] >> ((ibeg + i0) & 63)) & 0xffu;
#pragma unroll
    for (int t = 0; t < 4; ++t) xor_terms2(acc, w + 2 * t, (cb >> (2 * t)) & 3u);
#pragma unroll
    for (int m = 0; m < kJumpOut - 1; ++m) w[m] = w[m + 8];
  }
  __syncthreads();
  uint64_t* red = px;  // reuse: [8][352]
#pragma unroll
  for (int j = 0; j < kJumpOut; ++j) red[g * (32 * kJumpOut) + kJumpOut * q + j] = acc[j];
  __syncthreads();
  unsigned long long* dst = segwin + (((size_t)k * nseg + s1) * kLanes + l) * kN;
  for (int j = tid; j < kN; j += kJumpThreads) {
    uint64_t v = 0;
#pragma unroll
    for (int gg = 0; gg < kJumpThreads / 32; ++gg) v ^= red[gg * (32 * kJumpOut) + j];
    atomicXor(dst + j, (unsigned long long)v);
  }
}
constexpr int kJumpFew = 39, kJumpMany = 8, kJumpFewMax = 160;

// ---------------------------------------------------------------- transforms
// Truncated.h inverse-CDF forms, one lane: u is UniformRealGen(phi(lower),
// phi(upper))'s value.  TruncNormalGen::packetOp (:322-331), lognormal
// (:593-598), exponential (:477-484), Cauchy (:534-543), extreme value
// (:649-656), Weibull (:709-718).
template <int KIND>
__device__ __forceinline__ float trunc32(float u, const DistParams& d) {
  if (KIND == kTruncNormalKind || KIND == kTruncLognormalKind) {
    const float x = ((float)-1.4142135623730951 * erfinvf_(1.0f - 2.0f * u)) * d.fc + d.fd;
    return KIND == kTruncLognormalKind ? expf_(x) : x;
  }
  if (KIND == kTruncExponentialKind) return -logf_(1.0f - u) * d.fc;
  if (KIND == kTruncCauchyKind) {
    float s, c;
    sincosf_((float)3.1415926535897932 * (u - 0.5f), s, c);
    return d.fc + d.fd * (s / c);
  }
  if (KIND == kTruncExtremeKind) return d.fc - d.fd * logf_(-logf_(u));
  return d.fd * expf_(logf_(-logf_(1.0f - u)) * d.fc);  // Weibull
}

template <int KIND>
__device__ __forceinline__ double trunc64(double u, const DistParams& d) {
  if (KIND == kTruncNormalKind || KIND == kTruncLognormalKind) {
    const double x = (-1.4142135623730951 * erfinv_(1.0 - 2.0 * u)) * d.dc + d.dd;
    return KIND == kTruncLognormalKind ? exp_(x) : x;
  }
  if (KIND == kTruncExponentialKind) return -log_(1.0 - u) * d.dc;
  if (KIND == kTruncCauchyKind) {
    double s, c;
    sincos_d<1>(3.1415926535897932 * (u - 0.5), s, c);
    return d.dc + d.dd * div_d(s, c);
  }
  if (KIND == kTruncExtremeKind) return d.dc - d.dd * log_(-log_(u));
  return d.dd * exp_(log_(-log_(1.0 - u)) * d.dc);
}

// float samples from one u32 word (one lane of a Packet8f), per kind.
template <int KIND>
__device__ __forceinline__ float tf32(uint32_t w, const DistParams& d) {
  if (KIND == GR_UNIFORM_REAL) return ur_f(w);
  if (KIND == GR_UNIFORM_REAL2) return ur_f(w) * d.fa + d.fb;
  if (KIND == GR_BALANCED || KIND == GR_BALANCED2) {
    float z = (float)(int32_t)(w & 0x7fffffffu) / (float)0x7FFFFFFF;
    return KIND == GR_BALANCED ? z * 2.0f - 1.0f : z * d.fa + d.fb;
  }
  if (KIND == GR_EXPONENTIAL) return -(logf_<true>(1.0f - ur_f(w)) / d.fa);
  if (KIND == GR_GAMMA) return d.fb * (-(logf_<true>(1.0f - ur_f(w)) / 1.0f));
  if (KIND == GR_CAUCHY) {
    float s, c;
    sincosf_((float)3.1415926535897932 * (ur_f(w) - 0.5f), s, c);
    return d.fa + d.fb * (s / c);
  }
  if (KIND == GR_WEIBULL) return expf_(logf_(-logf_<true>(1.0f - ur_f(w))) * d.fa) * d.fb;
  if (KIND == GR_EXTREME_VALUE) return d.fa - logf_(-logf_(ur_f(w) + 1.1920928955078125e-07f / 8)) * d.fb;
  // BernoulliGen<float>: the word of the lane, masked, compared signed
  if (KIND == GR_BERNOULLI) return ((int32_t)(w & 0x7fffffffu) < d.ia) ? 1.0f : 0.0f;
  if (KIND >= kTruncNormalKind && KIND <= kTruncWeibullKind) return trunc32<KIND>(ur_f(w) * d.fa + d.fb, d);
  return 0.0f;
}

template <int KIND>
__device__ __forceinline__ double tf64(uint64_t r, const DistParams& d) {
  if (KIND == GR_UNIFORM_REAL) return ur_d(r);
  if (KIND == GR_UNIFORM_REAL2) return ur_d(r) * d.da + d.db;
  if (KIND == GR_EXPONENTIAL) {
    const double l = log_(one_minus_ur_d(r));
    return (d.flags & kParamUnitDiv) ? -l : -div_d(l, d.da);
  }
  if (KIND == GR_GAMMA) {
    const double l = -(log_(one_minus_ur_d(r)) / 1.0);
    return (d.flags & kParamUnitScale) ? l : d.db * l;
  }
  if (KIND == GR_CAUCHY) {
    double s, c;
    sincos_pi_centred(r, s, c);
    return d.da + d.db * div_d(s, c);
  }
  if (KIND == GR_WEIBULL) {
    const double w = exp_(log_(-log_(one_minus_ur_d(r))) * d.da);
    return (d.flags & kParamUnitScale) ? w : w * d.db;
  }
  if (KIND == GR_EXTREME_VALUE) return d.da - log_(-log_(ur_nz_int(r))) * d.db;
  // BernoulliGen<double>: the compare runs on the eight 32-bit words and the
  // blend reads each 64-bit element's sign, the compare of its high word
  if (KIND == GR_BERNOULLI) return ((int32_t)((uint32_t)(r >> 32) & 0x7fffffffu) < d.ia) ? 1.0 : 0.0;
  if (KIND >= kTruncNormalKind && KIND <= kTruncWeibullKind) return trunc64<KIND>(ur_d(r) * d.da + d.db, d);
  return 0.0;
}

// double balanced from one u32 word (rng.half() path); the quotient by
// 2^31 - 1 in integer form (gr_exact.h), bit-identical to the division
template <int KIND>
__device__ __forceinline__ double tw64(uint32_t w, const DistParams& d) {
  double z = div_2p31m1(w & 0x7fffffffu);
  return KIND == GR_BALANCED ? z * 2.0 - 1.0 : z * d.da + d.db;
}

template <int KIND>
__device__ __forceinline__ int32_t tw32(uint32_t w, const DistParams& d) {
  if (KIND == GR_RANDBITS) return (int32_t)w;
  if (KIND == GR_BERNOULLI) return ((int32_t)(w & 0x7fffffffu) < d.ia) ? 1 : 0;
  // UniformIntGen<int32_t> over a power-of-two range: (rx & bitmask) + pmin (Discrete.h:302-305)
  if (KIND == GR_UNIFORM_INT) return (int32_t)((w & d.bitmask) + (uint32_t)d.ia);
  // GeometricGen<int32_t>: pcast(ptruncate(plog(1 - u) * rlog_q)), Discrete.h:1368-1374
  if (KIND == GR_GEOMETRIC) return cvtt_f32(truncf(logf_<true>(1.0f - ur_f(w)) * d.fa));
  // DiscreteGen<int32_t,int32_t>, Discrete.h:455-470
  if (d.ncdf > 0) {
    int32_t r = d.ncdf - 1;
    int32_t x = (int32_t)(w & 0x7fffffffu);
    for (int i = 0; i < d.ncdf - 1; ++i) r += (x < __ldg(d.prob + i)) ? -1 : 0;
    return r;
  }
  int32_t albit = (int32_t)(w & d.bitmask);
  return ((int32_t)(w >> 1) < __ldg(d.prob + albit)) ? albit : __ldg(d.alias + albit);
}

template <int KIND>
__device__ __forceinline__ float nscale32(float x, const DistParams& d) {
  if (KIND == GR_NORMAL_STD) return x;
  if (KIND == GR_NORMAL) return x * d.fb + d.fa;
  return expf_(x * d.fb + d.fa);  // lognormal
}
template <int KIND>
__device__ __forceinline__ double nscale64(double x, const DistParams& d) {
  if (KIND == GR_NORMAL_STD) return x;
  if (KIND == GR_NORMAL) return x * d.db + d.da;
  return exp_(x * d.db + d.da);
}

// ---------------------------------------------------------------- per-element forms
// The *VGen packetOp arguments of output element idx, mapped onto the
// constants the scalar-parameter transform reads: UniformRealVGen and
// BalancedVGen slope b - a, bias a (Basic.h:486-491, :660-665); NormalVGen and
// LognormalVGen mean a, stdev b (NormalExp.h:155-162, :230-235);
// ExponentialVGen lambda a (:420-426); WeibullVGen 1 / a and b (:679-685);
// ExtremeValueVGen and CauchyVGen a, b (:757-764, :879-888).  Each is the
// same packet arithmetic as the scalar generator with the lane's own values.
template <int BK>
__device__ __forceinline__ DistParams vparams32(const DistParams& d, int64_t idx) {
  const float a = (d.flags & kParamVecA) ? __ldg(static_cast<const float*>(d.vparam) + idx) : d.fe;
  const float b = (d.flags & kParamVecB) ? __ldg(static_cast<const float*>(d.vparam2) + idx) : d.ff;
  DistParams e = d;
  e.flags = 0;
  if (BK == GR_UNIFORM_REAL2 || BK == GR_BALANCED2) {
    e.fa = b - a;
    e.fb = a;
  } else if (BK == GR_WEIBULL) {
    e.fa = 1.0f / a;
    e.fb = b;
  } else {
    e.fa = a;
    e.fb = b;
  }
  return e;
}
template <int BK>
__device__ __forceinline__ DistParams vparams64(const DistParams& d, int64_t idx) {
  const double a = (d.flags & kParamVecA) ? __ldg(static_cast<const double*>(d.vparam) + idx) : d.de;
  const double b = (d.flags & kParamVecB) ? __ldg(static_cast<const double*>(d.vparam2) + idx) : d.df;
  DistParams e = d;
  e.flags = 0;
  if (BK == GR_UNIFORM_REAL2 || BK == GR_BALANCED2) {
    e.da = b - a;
    e.db = a;
  } else if (BK == GR_WEIBULL) {
    e.da = 1.0 / a;
    e.db = b;
  } else {
    e.da = a;
    e.db = b;
  }
  return e;
}

// Transforms with the output element index: a per-element kind reads its
// parameters there, the others ignore it.
template <int KIND>
__device__ __forceinline__ float tf32i(uint32_t w, const DistParams& d, int64_t idx) {
  if constexpr (KIND >= kVecBase) return tf32<KIND - kVecBase>(w, vparams32<KIND - kVecBase>(d, idx));
  else return tf32<KIND>(w, d);
}
template <int KIND>
__device__ __forceinline__ double tf64i(uint64_t r, const DistParams& d, int64_t idx) {
  if constexpr (KIND >= kVecBase) return tf64<KIND - kVecBase>(r, vparams64<KIND - kVecBase>(d, idx));
  else return tf64<KIND>(r, d);
}
template <int KIND>
__device__ __forceinline__ double tw64i(uint32_t w, const DistParams& d, int64_t idx) {
  if constexpr (KIND >= kVecBase) return tw64<KIND - kVecBase>(w, vparams64<KIND - kVecBase>(d, idx));
  else return tw64<KIND>(w, d);
}
template <int KIND>
__device__ __forceinline__ float nscale32i(float x, const DistParams& d, int64_t idx) {
  if constexpr (KIND >= kVecBase) return nscale32<KIND - kVecBase>(x, vparams32<KIND - kVecBase>(d, idx));
  else return nscale32<KIND>(x, d);
}
template <int KIND>
__device__ __forceinline__ double nscale64i(double x, const DistParams& d, int64_t idx) {
  if constexpr (KIND >= kVecBase) return nscale64<KIND - kVecBase>(x, vparams64<KIND - kVecBase>(d, idx));
  else return nscale64<KIND>(x, d);
}

// ---------------------------------------------------------------- direct kernel
// M_RAW2 / M_F32H / M_F64H: the 2-lane Vmt19937_64 (SSE / NEON profile,
// Pmt19937_64<Packet4i>): its packets are the first two lanes of the 4-lane
// engine with the same seed, a Packet4f (4 floats) or Packet2d (2 doubles)
// per packet; the other two lanes are made and left unused.
enum Mode { M_RAW, M_F32, M_F64, M_W32, M_W64, M_N32, M_N64, M_RAW0, M_RAW2, M_F32H, M_F64H };

template <int MODE>
struct ModeInfo {
  static constexpr int OPP = (MODE == M_RAW || MODE == M_RAW0) ? 4 : MODE == M_F32 ? 8 : MODE == M_F64 ? 4 : MODE == M_N32 ? 8 : MODE == M_N64 ? 4
                           : MODE == M_RAW2 ? 2 : MODE == M_F32H ? 4 : MODE == M_F64H ? 2 : 8;
  static constexpr int kCacheOut = MODE == M_N32 ? 8 : MODE == M_N64 ? 4 : (MODE == M_W32 || MODE == M_W64) ? 4 : 0;
};

__device__ __forceinline__ void st16(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  *reinterpret_cast<uint4*>(p) = make_uint4(a, b, c, d);
}

// 32 bytes of one thread, a sector: two 16-byte stores would reach L2 as two
// partial writes of it.  An output that is only 16-byte aligned (or starts after
// an odd cached packet) takes the two.
__device__ __forceinline__ void st32(void* p, const uint64_t a, const uint64_t b, const uint64_t c, const uint64_t d) {
  if (((uintptr_t)p & 31) == 0) {
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
  } else {
    reinterpret_cast<ulonglong2*>(p)[0] = make_ulonglong2(a, b);
    reinterpret_cast<ulonglong2*>(p)[1] = make_ulonglong2(c, d);
  }
}

// int32 kinds whose packets are rng.half() words leave raw words in the
// engine's half cache; DiscreteGen caches its own computed results
template <int MODE, int KIND>
struct CacheUse {
  static constexpr bool half_kind =
      KIND == GR_RANDBITS || KIND == GR_BERNOULLI || KIND == GR_GEOMETRIC || KIND == GR_UNIFORM_INT;
  static constexpr bool half = (MODE == M_W64) || (MODE == M_W32 && half_kind);
  static constexpr bool gen = (MODE == M_N32) || (MODE == M_N64) || (MODE == M_W32 && KIND == GR_DISCRETE);
};

// The samples of half h of packet pidx of a call (pk: the half's two tempered
// words), output element obase + pidx * OPP on; oend: end of the engine's slice
// (the half of a packet or unit past it goes to the cache).  Called by whole
// warps whose lanes hold consecutive halves from an even packet on: the
// Box-Muller kinds exchange words within packet pairs.  FULL: the call's last
// packet is none of these.
template <int MODE, int KIND, bool FULL = false>
__device__ __forceinline__ void emit_half(const uint64_t (&pk)[2], const int h, const int64_t pidx, const bool valid,
                                          const Plan& p, const DistParams& d, const int64_t obase, const int64_t oend,
                                          EngState* st, GenState* gs) {
  constexpr bool kHalfKind = CacheUse<MODE, KIND>::half_kind;
  const uint32_t wd[4] = {(uint32_t)pk[0], (uint32_t)(pk[0] >> 32), (uint32_t)pk[1], (uint32_t)(pk[1] >> 32)};
  if (MODE == M_RAW) {
    if (valid && p.out)  // p.out == nullptr: discard
      *reinterpret_cast<ulonglong2*>(reinterpret_cast<uint64_t*>(p.out) + obase + pidx * 4 + 2 * h) =
          make_ulonglong2(pk[0], pk[1]);
  } else if (MODE == M_RAW2) {
    if (valid && h == 0 && p.out)
      *reinterpret_cast<ulonglong2*>(reinterpret_cast<uint64_t*>(p.out) + obase + pidx * 2) = make_ulonglong2(pk[0], pk[1]);
  } else if (MODE == M_RAW0) {
    // a scalar draw takes the engine's whole packet and keeps its first
    // element (StdUniformRealGen::operator(), Dists/Basic.h:533-540)
    if (valid && h == 0) reinterpret_cast<uint64_t*>(p.out)[obase / 4 + pidx] = pk[0];
  } else if (MODE == M_F32H || MODE == M_F32) {
    if (valid && (MODE == M_F32 || h == 0)) {
      const int64_t ib = obase + (MODE == M_F32 ? pidx * 8 + 4 * h : pidx * 4);
      float v[4];
      if (KIND == kBernoulliVKind) {
        // BernoulliVGen<float>: p = cvttps(a * 2^31), compared signed with
        // the masked word (Basic.h:735-745)
        const float4 a = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(d.vparam) + ib);
        const float pa[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
          v[q] = ((int32_t)(wd[q] & 0x7fffffffu) < cvtt_f32(pa[q] * 2147483648.0f)) ? 1.0f : 0.0f;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = tf32i<KIND>(wd[q], d, ib + q);
      }
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + ib) = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else if (MODE == M_F64H || MODE == M_F64) {
    if (valid && (MODE == M_F64 || h == 0)) {
      const int64_t ib = obase + (MODE == M_F64 ? pidx * 4 + 2 * h : pidx * 2);
      *reinterpret_cast<double2*>(reinterpret_cast<double*>(p.out) + ib) =
          make_double2(tf64i<KIND>(pk[0], d, ib), tf64i<KIND>(pk[1], d, ib + 1));
    }
  } else if (MODE == M_W32 || MODE == M_W64) {
    if (valid) {
      const int64_t ob = obase + pidx * 8 + 4 * h;
      const bool in = FULL || ob + 4 <= oend;
      if (MODE == M_W32) {
        int32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = tw32<KIND>(wd[q], d);
        if (in) {
          st16(reinterpret_cast<int32_t*>(p.out) + ob, v[0], v[1], v[2], v[3]);
        } else if (gs || kHalfKind) {
          // leftover half: rng.half() kinds leave raw words in the engine's
          // half() cache; DiscreteGen caches its computed upper 4 results
          uint32_t* cdst = kHalfKind ? st->half_cache : gs->s[0].cache;
#pragma unroll
          for (int q = 0; q < 4; ++q) cdst[q] = kHalfKind ? wd[q] : (uint32_t)v[q];
        }
      } else if (in) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = tw64i<KIND>(wd[q], d, ob + q);
        st32(reinterpret_cast<double*>(p.out) + ob, d2u(v[0]), d2u(v[1]), d2u(v[2]), d2u(v[3]));
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) st->half_cache[q] = wd[q];
      }
    }
  } else {
    // unit = packets (2j, 2j+1): u1 words in the even packet, u2 in the odd.
    // The even packet's thread makes the pairs of its half's first word, the
    // odd one's those of the second: they exchange one word.
    const bool odd = (pidx & 1);
    const uint64_t other = xor64(odd ? pk[0] : pk[1], 2);
    if (valid) {
      const int64_t unit = pidx >> 1;
      const uint64_t w1 = odd ? other : pk[0], w2 = odd ? pk[1] : other;
      if (MODE == M_N32) {
        const int i0 = 4 * h + (odd ? 2 : 0);
        float sv[2], cv[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float u1 = ur_f((uint32_t)(w1 >> (32 * q))), u2 = ur_f((uint32_t)(w2 >> (32 * q)));
          const float radius = sqrtf((float)-2 * logf_<true>(1.0f - u1));
          const float theta = (float)(2 * 3.1415926535897932) * u2;
          float sn, cs;
          sincosf_(theta, sn, cs);
          sv[q] = radius * sn;
          cv[q] = radius * cs;
        }
        const int64_t ob = obase + unit * 16 + i0;
        float* o = reinterpret_cast<float*>(p.out) + ob;
        *reinterpret_cast<float2*>(o) = make_float2(nscale32i<KIND>(sv[0], d, ob), nscale32i<KIND>(sv[1], d, ob + 1));
        if (ob - i0 + 16 <= oend) {
          *reinterpret_cast<float2*>(o + 8) =
              make_float2(nscale32i<KIND>(cv[0], d, ob + 8), nscale32i<KIND>(cv[1], d, ob + 9));
        } else if (gs) {
          gs->s[0].cache[i0] = f2u(cv[0]);
          gs->s[0].cache[i0 + 1] = f2u(cv[1]);
        }
      } else {
        const int i0 = 2 * h + (odd ? 1 : 0);
        const double radius = sqrt_neg2(log_(one_minus_ur_d(w1)));
        double sn, cs;
        sincos_2pi_u(w2, sn, cs);
        const int64_t ob = obase + unit * 8 + i0;
        double* o = reinterpret_cast<double*>(p.out) + ob;
        o[0] = nscale64i<KIND>(radius * sn, d, ob);
        const double cv = radius * cs;
        if (ob - i0 + 8 <= oend) {
          o[4] = nscale64i<KIND>(cv, d, ob + 4);
        } else if (gs) {
          const uint64_t b = d2u(cv);
          gs->s[0].cache[2 * i0] = (uint32_t)b;
          gs->s[0].cache[2 * i0 + 1] = (uint32_t)(b >> 32);
        }
      }
    }
  }
}

// One CTA per stream or jump segment, two threads per packet of a phase.  The
// cheap kinds are bound by the logic pipe (uniform floats: 12 of its
// instructions per sample, 43 of 60 us), float transforms by instruction issue,
// double ones by the FP64 and logic pipes together (gr_fp64i.h).  608 engines
// give an SM four CTAs whatever their size: with a thread per packet (160
// threads) it held 20 warps, here 40, which also store 512 consecutive bytes at
// a time.  8192 x 8192 on 608 engines, us, a thread per packet / two, with the other
// code as it was then: uniform f32 74.9 / 59.5, discrete 143 / 122, weibull f32 309 /
// 284, exponential f64 746 / 711, lognormal f64 2 168 / 1 876, weibull f64 2 093 /
// 1 832 (now 57.4, 124, 236, 700, 1 902, 1 809).
constexpr int kDirThreads = 320;

// Kinds whose transform takes a few operations per word: their loop is unrolled
// over two blocks with shared-memory offsets and the registers' roles fixed
// (0.60 instead of 0.83 warp-instructions per uniform float).
template <int MODE, int KIND>
constexpr bool kLightKind = MODE == M_RAW || MODE == M_RAW0 || MODE == M_RAW2 || KIND == GR_UNIFORM_REAL ||
                            KIND == GR_UNIFORM_REAL2 || (KIND == GR_BALANCED && MODE != M_W64) || KIND == GR_BERNOULLI ||
                            KIND == GR_RANDBITS || KIND == GR_UNIFORM_INT;

// Kinds that need more than the 48 registers of four CTAs per SM.
template <int MODE, int KIND>
constexpr bool kWideKind = MODE == M_F64 && (KIND == kTruncNormalKind || KIND == kTruncLognormalKind);

template <int MODE, int KIND>
__global__ void __launch_bounds__(kDirThreads, kWideKind<MODE, KIND> ? 2 : 4)
    k_direct(Plan p, DistParams d, const CallSnap* snap) {
  const int k = blockIdx.x / p.S, s = blockIdx.x % p.S;
  const int tid = threadIdx.x;
  EngState* st = p.eng + k;
  GenState* gs = p.gen ? p.gen + k : nullptr;

  const int64_t g0 = (int64_t)k * p.gran_per_k + min((int64_t)k, p.gran_rem);
  const int64_t ng = p.gran_per_k + ((int64_t)k < p.gran_rem ? 1 : 0);
  const int64_t off = g0 * p.gran, n = ng * p.gran;
  if (n == 0) return;

  // --- caches the call starts from
  constexpr bool kHalfKind = CacheUse<MODE, KIND>::half_kind;
  constexpr bool kUsesHalf = CacheUse<MODE, KIND>::half;
  constexpr bool kUsesGen = CacheUse<MODE, KIND>::gen;
  int cvalid = 0;
  const uint32_t* cwords = nullptr;
  if (kUsesHalf) {
    cvalid = p.S > 1 ? snap[k].half_valid : st->half_valid;
    cwords = p.S > 1 ? snap[k].half_cache : st->half_cache;
  } else if (kUsesGen) {
    cvalid = p.S > 1 ? snap[k].gen_valid : (gs ? gs->s[0].valid : 0);
    cwords = p.S > 1 ? snap[k].gen_cache : (gs ? gs->s[0].cache : nullptr);
  }
  constexpr int CO = ModeInfo<MODE>::kCacheOut;
  const int64_t Q0 = (cvalid && CO) ? min((int64_t)CO, n) : 0;
  const int64_t r = n - Q0;
  constexpr int OPP = ModeInfo<MODE>::OPP;  // outputs per packet (N modes: per packet of a 2-packet unit)
  const int64_t Np = (MODE == M_N32 || MODE == M_N64) ? 2 * ((r + 2 * OPP - 1) / (2 * OPP)) : (r + OPP - 1) / OPP;
  const int64_t pbeg = (int64_t)s * p.J;
  const int64_t pend = min(pbeg + p.J, Np);
  const bool last = (pbeg < Np && Np <= pbeg + p.J) || (Np == 0 && s == 0);
  if (pbeg >= Np && !(Np == 0 && s == 0)) return;

  // --- prefix outputs served from the cache (segment 0 only)
  if (s == 0 && tid < Q0) {
    const int i = tid;
    if (MODE == M_W64) reinterpret_cast<double*>(p.out)[off + i] = tw64i<KIND>(cwords[i], d, off + i);
    if (MODE == M_W32)
      reinterpret_cast<int32_t*>(p.out)[off + i] = kHalfKind ? tw32<KIND>(cwords[i], d) : (int32_t)cwords[i];
    if (MODE == M_N32) reinterpret_cast<float*>(p.out)[off + i] = nscale32i<KIND>(u2f(cwords[i]), d, off + i);
    if (MODE == M_N64) {
      uint64_t b = (uint64_t)cwords[2 * i] | ((uint64_t)cwords[2 * i + 1] << 32);
      reinterpret_cast<double*>(p.out)[off + i] = nscale64i<KIND>(u2d(b), d, off + i);
    }
  }

  // --- lane windows.  With several segments the last one rewrites st->win,
  // so segment 0 reads the copy the prefix kernel made at call start.
  const uint64_t* w0;
  size_t wl = kN;  // stride of the window's lanes
  if (s == 0 && p.S > 1) {
    w0 = p.prefix + (size_t)k * kLanes * kPrefixLen;
    wl = kPrefixLen;
  } else {
    w0 = s == 0 ? &st->win[0][0] : p.segwin + ((size_t)k * (p.S - 1) + (s - 1)) * kLanes * kN;
  }
  // Threads 2 t and 2 t + 1 (t < 156) hold word t of the last two phases (156
  // words) of two lanes each, half a packet: x[i] and x[i + 156] of the
  // recurrence are a thread's own registers, and x[i + 1], two phases old, is
  // read from the words every thread puts into `nbr` as it makes them.  The
  // last pair's x[i + 1] is the first pair's word of the phase just made: there
  // in every first phase of a pair, made again from the first two pairs' words
  // in the second, so one barrier serves two phases.
  __shared__ ulonglong2 nbr[4][kDirThreads];  // [phase mod 4][thread]
  const int h = tid & 1, ti = min(tid >> 1, kM - 1), right = min(tid + 2, kDirThreads - 1);
  uint64_t x[2], c[2];  // words of phases g - 2 and g - 1
#pragma unroll
  for (int l = 0; l < 2; ++l) {
    x[l] = w0[(2 * h + l) * wl + ti];
    c[l] = w0[(2 * h + l) * wl + kM + ti];
  }
  nbr[2][tid] = make_ulonglong2(x[0], x[1]);
  nbr[3][tid] = make_ulonglong2(c[0], c[1]);
  const int64_t obase = off + Q0;
  const int64_t oend = off + n;
  // one phase: slot g (mod 4) of nbr, the second of a pair or the first
  auto phase = [&](const int g, const bool second, uint64_t (&pk)[2]) {
    ulonglong2 nb = nbr[g ^ 2][right];
    if (tid >> 1 == kM - 1) {
      if (!second) {
        nb = nbr[(g + 3) & 3][h];
      } else {
        const ulonglong2 a0 = nbr[(g + 1) & 3][h], a1 = nbr[(g + 1) & 3][2 + h], a2 = nbr[g ^ 2][h];
        nb = make_ulonglong2(twist1(a0.x, a1.x, a2.x), twist1(a0.y, a1.y, a2.y));
      }
    }
    const uint64_t v0 = twist1(x[0], nb.x, c[0]), v1 = twist1(x[1], nb.y, c[1]);
    nbr[g][tid] = make_ulonglong2(v0, v1);
    pk[0] = temper(v0);
    pk[1] = temper(v1);
    x[0] = c[0];
    x[1] = c[1];
    c[0] = v0;
    c[1] = v1;
  };
  int64_t base = pbeg;
  if constexpr (kLightKind<MODE, KIND>) {
    // the cheap transforms: two blocks at a time with every shared-memory
    // offset and register's role fixed, short of the call's last packet
    for (; base + 2 * kN < pend; base += 2 * kN) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if ((g & 1) == 0) __syncthreads();
        uint64_t pk[2];
        phase(g, g & 1, pk);
        emit_half<MODE, KIND, true>(pk, h, base + (tid >> 1) + g * kM, tid < 2 * kM, p, d, obase, oend, st, gs);
      }
    }
  }
  int slot = 0;  // the phase to make, mod 4
  for (; base < pend; base += kN, slot ^= 2) {
    __syncthreads();
    const int here = (int)min(pend - base, (int64_t)kN);
#pragma unroll 1
    for (int ph = 0; ph < 2; ++ph) {
      if (ph * kM >= here) break;
      uint64_t pk[2];
      phase(slot + ph, ph, pk);
      const int i = ph * kM + (tid >> 1);
      emit_half<MODE, KIND>(pk, h, base + i, tid < 2 * kM && i < here, p, d, obase, oend, st, gs);
    }
  }

  // --- end-of-call state: new lane windows and cache flags.  A call that the
  // cache serves whole has met no barrier yet: every thread has read the flag
  // before it changes.
  if (CO > 0 && Np == 0) __syncthreads();
  if (last) {
    if (Np > 0 && tid < 2 * kM) {
      // the 312 words before packet pend: the end of phase g - 3, phase g - 2
      // and the first rr of phase g - 1, each thread's own
      const int rr = (int)((pend - pbeg - 1) % kM) + 1;
      const int g1 = (int)((pend - pbeg - 1) / kM) & 3;  // phase g - 1
      const ulonglong2 o3 = nbr[(g1 + 2) & 3][tid];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        uint64_t* win = st->win[2 * h + l];
        if (ti >= rr) win[ti - rr] = l ? o3.y : o3.x;
        win[kM - rr + ti] = x[l];
        if (ti < rr) win[kN - rr + ti] = c[l];
      }
    }
    if (tid == 0) {
      int64_t left = 0;  // leftover outputs cached for the next call
      if (MODE == M_W32 || MODE == M_W64) left = (r % 8) ? 4 : 0;
      if (MODE == M_N32) left = (r % 16) ? 8 : 0;
      if (MODE == M_N64) left = (r % 8) ? 4 : 0;
      if (kUsesHalf) st->half_valid = left ? 1 : (Q0 ? 0 : st->half_valid);
      if (kUsesGen && gs) gs->s[0].valid = left ? 1 : 0;
      st->consumed += (uint64_t)Np;
    }
  }
}

// The same transforms over words that k_words_* left in memory: one thread per
// half packet, grid (packets, engines).  Packets [wbase, wbase + wcount) of every
// engine's call are in memory; block 0 of an engine leaves the engine state.
constexpr int kXfThreads = 256;
template <int MODE, int KIND>
__global__ void __launch_bounds__(kXfThreads) k_xform(Plan p, DistParams d, const CallSnap* snap) {
  const int k = blockIdx.y, tid = threadIdx.x;
  EngState* st = p.eng + k;
  GenState* gs = p.gen ? p.gen + k : nullptr;
  const int64_t g0 = (int64_t)k * p.gran_per_k + min((int64_t)k, p.gran_rem);
  const int64_t ng = p.gran_per_k + ((int64_t)k < p.gran_rem ? 1 : 0);
  const int64_t off = g0 * p.gran, n = ng * p.gran;
  if (n == 0) return;
  constexpr bool kHalfKind = CacheUse<MODE, KIND>::half_kind;
  constexpr bool kUsesHalf = CacheUse<MODE, KIND>::half;
  constexpr bool kUsesGen = CacheUse<MODE, KIND>::gen;
  const int cvalid = kUsesHalf ? snap[k].half_valid : (kUsesGen ? snap[k].gen_valid : 0);
  const uint32_t* cwords = kUsesHalf ? snap[k].half_cache : snap[k].gen_cache;
  constexpr int CO = ModeInfo<MODE>::kCacheOut;
  constexpr int OPP = ModeInfo<MODE>::OPP;
  const int64_t Q0 = (cvalid && CO) ? min((int64_t)CO, n) : 0;
  const int64_t r = n - Q0;
  const int64_t Np = (MODE == M_N32 || MODE == M_N64) ? 2 * ((r + 2 * OPP - 1) / (2 * OPP)) : (r + OPP - 1) / OPP;
  const int64_t obase = off + Q0, oend = off + n;
  const int64_t pend = min(p.wbase + p.wcount, Np);
  const int64_t pidx = p.wbase + (int64_t)blockIdx.x * (kXfThreads / 2) + (tid >> 1);
  const int h = tid & 1;
  const uint64_t* w = p.words + (size_t)k * kLanes * p.wstride;
  const bool valid = pidx < pend;
  uint64_t pk[2];
#pragma unroll
  for (int l = 0; l < 2; ++l)
    pk[l] = valid ? temper(w[(size_t)(2 * h + l) * p.wstride + kN + (pidx - p.wbase)]) : 0;
  emit_half<MODE, KIND>(pk, h, pidx, valid, p, d, obase, oend, st, gs);
  if (blockIdx.x != 0) return;
  if (p.wbase == 0 && tid < Q0) {  // outputs served from the cache
    const int i = tid;
    if (MODE == M_W64) reinterpret_cast<double*>(p.out)[off + i] = tw64i<KIND>(cwords[i], d, off + i);
    if (MODE == M_W32)
      reinterpret_cast<int32_t*>(p.out)[off + i] = kHalfKind ? tw32<KIND>(cwords[i], d) : (int32_t)cwords[i];
    if (MODE == M_N32) reinterpret_cast<float*>(p.out)[off + i] = nscale32i<KIND>(u2f(cwords[i]), d, off + i);
    if (MODE == M_N64) {
      const uint64_t b = (uint64_t)cwords[2 * i] | ((uint64_t)cwords[2 * i + 1] << 32);
      reinterpret_cast<double*>(p.out)[off + i] = nscale64i<KIND>(u2d(b), d, off + i);
    }
  }
  const int64_t used = max(pend - p.wbase, (int64_t)0);  // packets of this run
  if (used > 0)
    for (int t = tid; t < kLanes * kN; t += kXfThreads)
      st->win[t / kN][t % kN] = w[(size_t)(t / kN) * p.wstride + used + t % kN];
  if (tid == 0) {
    if (Np <= p.wbase + p.wcount && (p.wbase < Np || p.wbase == 0)) {  // the call ends here
      int64_t left = 0;  // leftover outputs cached for the next call
      if (MODE == M_W32 || MODE == M_W64) left = (r % 8) ? 4 : 0;
      if (MODE == M_N32) left = (r % 16) ? 8 : 0;
      if (MODE == M_N64) left = (r % 8) ? 4 : 0;
      if (kUsesHalf) st->half_valid = left ? 1 : (Q0 ? 0 : cvalid);
      if (kUsesGen && gs) gs->s[0].valid = left ? 1 : 0;
    }
    st->consumed += (uint64_t)used;
  }
}

template <int MODE, int KIND>
static cudaError_t run_direct(const Plan& p, const DistParams& d, const CallSnap* snap, cudaStream_t s) {
  if (p.words) {
    const dim3 grid((unsigned)((p.wcount + kXfThreads / 2 - 1) / (kXfThreads / 2)), (unsigned)p.K);
    k_xform<MODE, KIND><<<grid, kXfThreads, 0, s>>>(p, d, snap);
  } else {
    k_direct<MODE, KIND><<<p.K * p.S, kDirThreads, 0, s>>>(p, d, snap);
  }
  return cudaGetLastError();
}

cudaError_t launch_prefix(const EngState* st, const GenState* gen, int K, uint64_t* prefix, CallSnap* snap,
                          cudaStream_t s) {
  k_prefix<<<K * kLanes, kWideThreads, 0, s>>>(st, prefix, snap, gen);
  return cudaGetLastError();
}

cudaError_t launch_jump(const uint64_t* prefix, const uint64_t* polys, int K, int S, uint64_t* segwin,
                        cudaStream_t s) {
  if (S <= 1) return cudaSuccess;
  const int ctas = K * (S - 1) * kLanes;
  cudaError_t e = cudaMemsetAsync(segwin, 0, (size_t)ctas * kN * sizeof(uint64_t), s);
  if (e != cudaSuccess) return e;
  // One engine, us: 4 segments 22.2 with 8 parts each, 14.3 with 39; 8: 26.4 and
  // 21.6; 13: 34.6 and 29.5.  The gap closes (a part reads 350 words beside its
  // own), and 1 300 CTAs of eight parts fill the GPU anyway.
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(segwin);
  if (ctas <= kJumpFewMax) k_jump<kJumpFew><<<ctas * kJumpFew, kJumpThreads, 0, s>>>(prefix, polys, S, dst);
  else k_jump<kJumpMany><<<ctas * kJumpMany, kJumpThreads, 0, s>>>(prefix, polys, S, dst);
  return cudaGetLastError();
}

cudaError_t preload_raw_stream_kernels() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_prefix);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_jump<kJumpFew>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_jump<kJumpMany>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_direct<M_RAW, kRawKind>);
  return e;
}

// ---------------------------------------------------------------- scalar tails
// A size that is not a whole number of packets ends with n % P elements made
// by the generator's scalar operator() (Eigen's linear vectorised assignment
// loop: packets up to the last whole one, then scalars).  Each takes one draw:
// the first 64-bit lane of an engine packet (pfirst of the packet), or one
// draw of a scalar engine.  Exact bit arithmetic for these kinds:
// randBits (Basic.h:386-391), balanced (:416-420), balanced(a, b)
// (:456-460), uniformReal (:533-540, ExtractFirstUint :345-371),
// uniformReal(min, max) (:620-624), bernoulli (:689-693).
bool kind_has_exact_tail(int kind, int dtype) {
  switch (kind) {
    case GR_UNIFORM_REAL:
    case GR_UNIFORM_REAL2:
    case GR_BALANCED:
    case GR_BALANCED2:
      return dtype == GR_F32 || dtype == GR_F64;
    case GR_BERNOULLI:
      return true;
    case GR_RANDBITS:
      return dtype == GR_I32;
    default:
      return false;
  }
}

__global__ void k_tail(const uint64_t* w, void* out, int n, DistParams d, int packet_engine) {
  const int i = threadIdx.x;
  if (i >= n) return;
  const uint64_t r = w[i];
  const uint32_t lo = (uint32_t)r;
  // pfirst of an engine packet is its first 32-bit word; of a scalar engine's
  // draw, the whole 64-bit value
  const uint64_t first = packet_engine ? (uint64_t)(int64_t)(int32_t)lo : r;
  const bool f64 = d.dtype == GR_F64;
  switch (d.kind) {
    case GR_UNIFORM_REAL:
      // ExtractFirstUint: the first 32-bit word (float), the first 64-bit lane (double)
      if (f64) reinterpret_cast<double*>(out)[i] = ur_d(r);
      else reinterpret_cast<float*>(out)[i] = ur_f(lo);
      break;
    case GR_UNIFORM_REAL2:  // bias + to_ur(pfirst(rng())) * slope
      if (f64) reinterpret_cast<double*>(out)[i] = d.db + ur_d(first) * d.da;
      else reinterpret_cast<float*>(out)[i] = d.fb + ur_f(lo) * d.fa;
      break;
    case GR_BALANCED:
    case GR_BALANCED2: {
      const uint32_t k = lo & 0x7fffffffu;
      if (f64) {
        const double z = div_2p31m1(k);
        reinterpret_cast<double*>(out)[i] = d.kind == GR_BALANCED ? z * 2.0 - 1.0 : z * d.da + d.db;
      } else {
        const float z = (float)(int32_t)k / (float)0x7FFFFFFF;
        reinterpret_cast<float*>(out)[i] = d.kind == GR_BALANCED ? z * 2.0f - 1.0f : z * d.fa + d.fb;
      }
      break;
    }
    case GR_BERNOULLI: {
      const int v = ((int32_t)(lo & 0x7fffffffu) < d.ia) ? 1 : 0;
      if (d.dtype == GR_I32) reinterpret_cast<int32_t*>(out)[i] = v;
      else if (f64) reinterpret_cast<double*>(out)[i] = v;
      else reinterpret_cast<float*>(out)[i] = (float)v;
      break;
    }
    case GR_RANDBITS:
      reinterpret_cast<int32_t*>(out)[i] = (int32_t)lo;
      break;
    default:
      break;
  }
}

cudaError_t launch_tail(const uint64_t* w, void* out, int n, const DistParams& d, bool packet_engine, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_tail<<<1, 32, 0, s>>>(w, out, n, d, packet_engine ? 1 : 0);
  return cudaGetLastError();
}

int kind_granule(int kind, int dtype) {
  if (kind == kRawKind || kind == kRawLane0Kind) return 4;
  if (dtype == GR_F32) return 8;
  return 4;  // double packets and int32 packets hold 4 lanes
}

int kind_packets_per_unit(int kind, int dtype) {
  (void)dtype;
  if (kind >= kVecBase) kind -= kVecBase;
  if (kind == GR_NORMAL_STD || kind == GR_NORMAL || kind == GR_LOGNORMAL) return 2;
  return 1;
}

bool kind_is_direct(int kind, int dtype, const DistParams& d) {
  switch (kind) {
    case kRawKind:
    case kRawLane0Kind:
    case GR_UNIFORM_REAL:
    case GR_UNIFORM_REAL2:
    case GR_BALANCED:
    case GR_BALANCED2:
    case GR_NORMAL_STD:
    case GR_NORMAL:
    case GR_LOGNORMAL:
    case GR_EXPONENTIAL:
    case GR_CAUCHY:
    case GR_WEIBULL:
    case GR_EXTREME_VALUE:
      return true;
    case GR_GAMMA:
      return d.ia == 1;  // alpha == 1: beta * exponential
    case GR_BERNOULLI:
      return true;
    case kTruncNormalKind:
    case kTruncLognormalKind:
    case kTruncExponentialKind:
    case kTruncCauchyKind:
    case kTruncExtremeKind:
    case kTruncWeibullKind:
      return dtype == GR_F32 || dtype == GR_F64;
    case kBernoulliVKind:
      return dtype == GR_F32;
    case kVecBase + GR_UNIFORM_REAL2:
    case kVecBase + GR_BALANCED2:
    case kVecBase + GR_NORMAL:
    case kVecBase + GR_LOGNORMAL:
    case kVecBase + GR_EXPONENTIAL:
    case kVecBase + GR_WEIBULL:
    case kVecBase + GR_EXTREME_VALUE:
    case kVecBase + GR_CAUCHY:
      return dtype == GR_F32 || dtype == GR_F64;
    case GR_RANDBITS:
    case GR_DISCRETE:
    case GR_GEOMETRIC:
      return dtype == GR_I32;
    case GR_UNIFORM_INT:
      return dtype == GR_I32 && d.ib == 1;
    default:
      return false;
  }
}

#define GR_F32_CASE(K) \
  case K:              \
    return run_direct<M_F32, K>(p, d, snap, s);
#define GR_F64_CASE(K) \
  case K:              \
    return run_direct<M_F64, K>(p, d, snap, s);

bool kind_two_lane(int kind, int dtype) {
  if (kind == kRawKind) return true;
  switch (kind) {
    case GR_UNIFORM_REAL:
    case GR_UNIFORM_REAL2:
    case GR_EXPONENTIAL:
    case GR_CAUCHY:
    case GR_WEIBULL:
    case GR_EXTREME_VALUE:
    case GR_GAMMA:  // alpha == 1 (the caller checks)
      return dtype == GR_F32 || dtype == GR_F64;
    case GR_BALANCED:
    case GR_BALANCED2:
    case GR_BERNOULLI:
      return dtype == GR_F32;
    default:
      return false;
  }
}

#define GR_F32H_CASE(K) \
  case K:               \
    return run_direct<M_F32H, K>(p, d, snap, s);
#define GR_F64H_CASE(K) \
  case K:               \
    return run_direct<M_F64H, K>(p, d, snap, s);

cudaError_t launch_direct(const Plan& p, const DistParams& d, const CallSnap* snap, cudaStream_t s) {
  if (d.flags & kParamTwoLane) {
    if (d.kind == kRawKind) return run_direct<M_RAW2, kRawKind>(p, d, snap, s);
    if (d.dtype == GR_F32) {
      switch (d.kind) {
        GR_F32H_CASE(GR_UNIFORM_REAL)
        GR_F32H_CASE(GR_UNIFORM_REAL2)
        GR_F32H_CASE(GR_BALANCED)
        GR_F32H_CASE(GR_BALANCED2)
        GR_F32H_CASE(GR_EXPONENTIAL)
        GR_F32H_CASE(GR_CAUCHY)
        GR_F32H_CASE(GR_WEIBULL)
        GR_F32H_CASE(GR_EXTREME_VALUE)
        GR_F32H_CASE(GR_GAMMA)
        GR_F32H_CASE(GR_BERNOULLI)
        default:
          return cudaErrorNotSupported;
      }
    }
    if (d.dtype == GR_F64) {
      switch (d.kind) {
        GR_F64H_CASE(GR_UNIFORM_REAL)
        GR_F64H_CASE(GR_UNIFORM_REAL2)
        GR_F64H_CASE(GR_EXPONENTIAL)
        GR_F64H_CASE(GR_CAUCHY)
        GR_F64H_CASE(GR_WEIBULL)
        GR_F64H_CASE(GR_EXTREME_VALUE)
        GR_F64H_CASE(GR_GAMMA)
        default:
          return cudaErrorNotSupported;
      }
    }
    return cudaErrorNotSupported;
  }
  if (d.kind == kRawKind) return run_direct<M_RAW, kRawKind>(p, d, snap, s);
  if (d.kind == kRawLane0Kind) return run_direct<M_RAW0, kRawLane0Kind>(p, d, snap, s);
  if (d.dtype == GR_F32) {
    switch (d.kind) {
      GR_F32_CASE(GR_UNIFORM_REAL)
      GR_F32_CASE(GR_UNIFORM_REAL2)
      GR_F32_CASE(GR_BALANCED)
      GR_F32_CASE(GR_BALANCED2)
      GR_F32_CASE(GR_EXPONENTIAL)
      GR_F32_CASE(GR_CAUCHY)
      GR_F32_CASE(GR_WEIBULL)
      GR_F32_CASE(GR_EXTREME_VALUE)
      GR_F32_CASE(GR_GAMMA)
      GR_F32_CASE(GR_BERNOULLI)
      GR_F32_CASE(kBernoulliVKind)
      GR_F32_CASE(kTruncNormalKind)
      GR_F32_CASE(kTruncLognormalKind)
      GR_F32_CASE(kTruncExponentialKind)
      GR_F32_CASE(kTruncCauchyKind)
      GR_F32_CASE(kTruncExtremeKind)
      GR_F32_CASE(kTruncWeibullKind)
      GR_F32_CASE(kVecBase + GR_UNIFORM_REAL2)
      GR_F32_CASE(kVecBase + GR_BALANCED2)
      GR_F32_CASE(kVecBase + GR_EXPONENTIAL)
      GR_F32_CASE(kVecBase + GR_WEIBULL)
      GR_F32_CASE(kVecBase + GR_EXTREME_VALUE)
      GR_F32_CASE(kVecBase + GR_CAUCHY)
      case kVecBase + GR_NORMAL:
        return run_direct<M_N32, kVecBase + GR_NORMAL>(p, d, snap, s);
      case kVecBase + GR_LOGNORMAL:
        return run_direct<M_N32, kVecBase + GR_LOGNORMAL>(p, d, snap, s);
      case GR_NORMAL_STD:
        return run_direct<M_N32, GR_NORMAL_STD>(p, d, snap, s);
      case GR_NORMAL:
        return run_direct<M_N32, GR_NORMAL>(p, d, snap, s);
      case GR_LOGNORMAL:
        return run_direct<M_N32, GR_LOGNORMAL>(p, d, snap, s);
      default:
        return cudaErrorNotSupported;
    }
  }
  if (d.dtype == GR_F64) {
    switch (d.kind) {
      GR_F64_CASE(GR_UNIFORM_REAL)
      GR_F64_CASE(GR_UNIFORM_REAL2)
      GR_F64_CASE(GR_EXPONENTIAL)
      GR_F64_CASE(GR_CAUCHY)
      GR_F64_CASE(GR_WEIBULL)
      GR_F64_CASE(GR_EXTREME_VALUE)
      GR_F64_CASE(GR_GAMMA)
      GR_F64_CASE(GR_BERNOULLI)
      GR_F64_CASE(kTruncNormalKind)
      GR_F64_CASE(kTruncLognormalKind)
      GR_F64_CASE(kTruncExponentialKind)
      GR_F64_CASE(kTruncCauchyKind)
      GR_F64_CASE(kTruncExtremeKind)
      GR_F64_CASE(kTruncWeibullKind)
      GR_F64_CASE(kVecBase + GR_UNIFORM_REAL2)
      GR_F64_CASE(kVecBase + GR_EXPONENTIAL)
      GR_F64_CASE(kVecBase + GR_WEIBULL)
      GR_F64_CASE(kVecBase + GR_EXTREME_VALUE)
      GR_F64_CASE(kVecBase + GR_CAUCHY)
      case kVecBase + GR_BALANCED2:
        return run_direct<M_W64, kVecBase + GR_BALANCED2>(p, d, snap, s);
      case kVecBase + GR_NORMAL:
        return run_direct<M_N64, kVecBase + GR_NORMAL>(p, d, snap, s);
      case kVecBase + GR_LOGNORMAL:
        return run_direct<M_N64, kVecBase + GR_LOGNORMAL>(p, d, snap, s);
      case GR_BALANCED:
        return run_direct<M_W64, GR_BALANCED>(p, d, snap, s);
      case GR_BALANCED2:
        return run_direct<M_W64, GR_BALANCED2>(p, d, snap, s);
      case GR_NORMAL_STD:
        return run_direct<M_N64, GR_NORMAL_STD>(p, d, snap, s);
      case GR_NORMAL:
        return run_direct<M_N64, GR_NORMAL>(p, d, snap, s);
      case GR_LOGNORMAL:
        return run_direct<M_N64, GR_LOGNORMAL>(p, d, snap, s);
      default:
        return cudaErrorNotSupported;
    }
  }
  if (d.dtype == GR_I32) {
    if (d.kind == GR_RANDBITS) return run_direct<M_W32, GR_RANDBITS>(p, d, snap, s);
    if (d.kind == GR_DISCRETE) return run_direct<M_W32, GR_DISCRETE>(p, d, snap, s);
    if (d.kind == GR_BERNOULLI) return run_direct<M_W32, GR_BERNOULLI>(p, d, snap, s);
    if (d.kind == GR_GEOMETRIC) return run_direct<M_W32, GR_GEOMETRIC>(p, d, snap, s);
    if (d.kind == GR_UNIFORM_INT) return run_direct<M_W32, GR_UNIFORM_INT>(p, d, snap, s);
  }
  return cudaErrorNotSupported;
}

// ---------------------------------------------------------------- scalar engines
// Samples drawn with a scalar engine as the Urng (std::mt19937_64,
// P8_mt19937_64): the packets come from RawbitsMaker<Packet8i, Rng, uint64_t,
// scalar_fullbit> (arch/AVX/RandUtils.h:59-144) and RawbitsMaker<Packet4i,
// ...> (arch/SSE/RandUtils.h:22-65) over the engine's 64-bit words, with GCC's
// right-to-left argument evaluation:
//   S_F32U  uniform_real<Packet8f> = rawbits_34: 3 words (a, b, c) ->
//           (c.lo, c.hi, b.lo, t0, b.hi, a.lo, a.hi, t1), t0 / t1 the top
//           bytes of their half's three words (the third twice)
//   S_F32R  rawbits (zero_to_one, BernoulliGen): 4 words in order, lo / hi
//   S_F64   rawbits as 4 double lanes
//   S_F64H  rawbits_half (zero_to_one<Packet4d>): 2 words -> 4 int32 words
//   S_N32 / S_N64  StdNormalGen units of two uniform packets
//   S_I32   Packet4i rawbits: 2 words -> 4 int32
// Packet k of the call reads its words at w[k * wpp]; one thread per packet
// (per unit for the normal kinds).
enum SMode { S_F32U, S_F32R, S_F64, S_F64H, S_N32, S_N64, S_I32 };

__device__ __forceinline__ void words34(const uint64_t* w, uint32_t* v8) {
  const uint64_t a = w[0], b = w[1], c = w[2];
  const uint32_t v[6] = {(uint32_t)c, (uint32_t)(c >> 32), (uint32_t)b, (uint32_t)(b >> 32), (uint32_t)a,
                         (uint32_t)(a >> 32)};
  v8[0] = v[0];
  v8[1] = v[1];
  v8[2] = v[2];
  v8[3] = (v[0] >> 24) | ((v[1] >> 24) << 8) | ((v[2] >> 24) << 16) | ((v[2] >> 24) << 24);
  v8[4] = v[3];
  v8[5] = v[4];
  v8[6] = v[5];
  v8[7] = (v[3] >> 24) | ((v[4] >> 24) << 8) | ((v[5] >> 24) << 16) | ((v[5] >> 24) << 24);
}

template <int SM, int KIND>
__global__ void __launch_bounds__(256) k_sxform(const uint64_t* w, void* out, int64_t npk, DistParams d) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (SM == S_N32 || SM == S_N64) {
    constexpr int WPP = SM == S_N32 ? 3 : 4;
    const int64_t u = t;
    if (2 * u >= npk) return;
    const uint64_t* w1 = w + 2 * u * WPP;
    if (SM == S_N32) {
      uint32_t a[8], b[8];
      words34(w1, a);
      words34(w1 + WPP, b);
      float* o = reinterpret_cast<float*>(out) + 2 * u * 8;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float radius = sqrtf((float)-2 * logf_(1.0f - ur_f(a[q])));
        float sn, cs;
        sincosf_((float)(2 * 3.1415926535897932) * ur_f(b[q]), sn, cs);
        o[q] = nscale32<KIND>(radius * sn, d);
        if (2 * u + 1 < npk) o[8 + q] = nscale32<KIND>(radius * cs, d);
      }
    } else {
      double* o = reinterpret_cast<double*>(out) + 2 * u * 4;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double radius = sqrt_neg2(log_(one_minus_ur_d(w1[q])));
        double sn, cs;
        sincos_2pi_u(w1[WPP + q], sn, cs);
        o[q] = nscale64<KIND>(radius * sn, d);
        if (2 * u + 1 < npk) o[4 + q] = nscale64<KIND>(radius * cs, d);
      }
    }
    return;
  }
  if (t >= npk) return;
  if (SM == S_F32U || SM == S_F32R) {
    uint32_t v[8];
    if (SM == S_F32U) {
      words34(w + 3 * t, v);
    } else {
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        v[2 * l] = (uint32_t)w[4 * t + l];
        v[2 * l + 1] = (uint32_t)(w[4 * t + l] >> 32);
      }
    }
    float r[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) r[q] = tf32<KIND>(v[q], d);
    float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + 8 * t);
    o[0] = make_float4(r[0], r[1], r[2], r[3]);
    o[1] = make_float4(r[4], r[5], r[6], r[7]);
  } else if (SM == S_F64) {
    double r[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) r[l] = tf64<KIND>(w[4 * t + l], d);
    double2* o = reinterpret_cast<double2*>(reinterpret_cast<double*>(out) + 4 * t);
    o[0] = make_double2(r[0], r[1]);
    o[1] = make_double2(r[2], r[3]);
  } else if (SM == S_F64H) {
    const uint64_t a = w[2 * t], b = w[2 * t + 1];
    const uint32_t v[4] = {(uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32)};
    double2* o = reinterpret_cast<double2*>(reinterpret_cast<double*>(out) + 4 * t);
    o[0] = make_double2(tw64<KIND>(v[0], d), tw64<KIND>(v[1], d));
    o[1] = make_double2(tw64<KIND>(v[2], d), tw64<KIND>(v[3], d));
  } else {  // S_I32
    const uint64_t a = w[2 * t], b = w[2 * t + 1];
    int4* o = reinterpret_cast<int4*>(reinterpret_cast<int32_t*>(out) + 4 * t);
    o[0] = make_int4(tw32<KIND>((uint32_t)a, d), tw32<KIND>((uint32_t)(a >> 32), d), tw32<KIND>((uint32_t)b, d),
                     tw32<KIND>((uint32_t)(b >> 32), d));
  }
}

template <int SM, int KIND>
static cudaError_t run_sx(const uint64_t* w, void* out, int64_t npk, const DistParams& d, cudaStream_t s) {
  const int64_t threads = (SM == S_N32 || SM == S_N64) ? (npk + 1) / 2 : npk;
  k_sxform<SM, KIND><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(w, out, npk, d);
  return cudaGetLastError();
}

int scalar_words_per_packet(int kind, int dtype) {
  // int32 kinds on one SSE packet of two draws (rawbits / rawbits_34)
  if (dtype == GR_I32) return (kind == GR_RANDBITS || kind == GR_BERNOULLI || kind == GR_GEOMETRIC) ? 2 : 0;
  const bool bal = kind == GR_BALANCED || kind == GR_BALANCED2;
  switch (kind) {
    case GR_UNIFORM_REAL:
    case GR_UNIFORM_REAL2:
    case GR_BALANCED:
    case GR_BALANCED2:
    case GR_NORMAL_STD:
    case GR_NORMAL:
    case GR_LOGNORMAL:
    case GR_EXPONENTIAL:
    case GR_CAUCHY:
    case GR_WEIBULL:
    case GR_EXTREME_VALUE:
    case GR_GAMMA:
    case GR_BERNOULLI:
      if (dtype == GR_F32) return (bal || kind == GR_BERNOULLI) ? 4 : 3;
      return bal ? 2 : 4;
    default:
      return 0;
  }
}

#define GR_SX(SMODE, K) \
  case K:               \
    return run_sx<SMODE, K>(w, out, npk, d, s);

cudaError_t launch_scalar_xform(const uint64_t* w, void* out, int64_t npk, const DistParams& d, cudaStream_t s) {
  if (d.dtype == GR_I32) {
    if (d.kind == GR_RANDBITS) return run_sx<S_I32, GR_RANDBITS>(w, out, npk, d, s);
    if (d.kind == GR_BERNOULLI) return run_sx<S_I32, GR_BERNOULLI>(w, out, npk, d, s);
    if (d.kind == GR_GEOMETRIC) return run_sx<S_I32, GR_GEOMETRIC>(w, out, npk, d, s);
    // DiscreteGen: a Packet8i of four draws per two output packets, so packet
    // t still reads draws 2t and 2t + 1
    if (d.kind == GR_DISCRETE) return run_sx<S_I32, GR_DISCRETE>(w, out, npk, d, s);
    return cudaErrorNotSupported;
  }
  if (d.dtype == GR_F32) {
    switch (d.kind) {
      GR_SX(S_F32U, GR_UNIFORM_REAL)
      GR_SX(S_F32U, GR_UNIFORM_REAL2)
      GR_SX(S_F32U, GR_EXPONENTIAL)
      GR_SX(S_F32U, GR_CAUCHY)
      GR_SX(S_F32U, GR_WEIBULL)
      GR_SX(S_F32U, GR_EXTREME_VALUE)
      GR_SX(S_F32U, GR_GAMMA)
      GR_SX(S_F32R, GR_BALANCED)
      GR_SX(S_F32R, GR_BALANCED2)
      GR_SX(S_F32R, GR_BERNOULLI)
      GR_SX(S_N32, GR_NORMAL_STD)
      GR_SX(S_N32, GR_NORMAL)
      GR_SX(S_N32, GR_LOGNORMAL)
      default:
        return cudaErrorNotSupported;
    }
  }
  switch (d.kind) {
    GR_SX(S_F64, GR_UNIFORM_REAL)
    GR_SX(S_F64, GR_UNIFORM_REAL2)
    GR_SX(S_F64, GR_EXPONENTIAL)
    GR_SX(S_F64, GR_CAUCHY)
    GR_SX(S_F64, GR_WEIBULL)
    GR_SX(S_F64, GR_EXTREME_VALUE)
    GR_SX(S_F64, GR_GAMMA)
    GR_SX(S_F64, GR_BERNOULLI)
    GR_SX(S_F64H, GR_BALANCED)
    GR_SX(S_F64H, GR_BALANCED2)
    GR_SX(S_N64, GR_NORMAL_STD)
    GR_SX(S_N64, GR_NORMAL)
    GR_SX(S_N64, GR_LOGNORMAL)
    default:
      return cudaErrorNotSupported;
  }
}

}  // namespace gr
