// Samplers driven by CompressMask::compress_append (EigenRand/arch/AVX/
// PacketFilter.h:147-184), one CTA per stream.
//
// Each trial consumes a fixed run of words and yields P candidates with an
// accept mask.  The reference's packetOp loop is an automaton over trials: a
// fully accepted trial is returned as is; otherwise its accepted lanes are
// appended, in lane order, to a FIFO carried in the generator, and a packet is
// returned once the FIFO holds P lanes.  With  NF_t = fully accepted trials
// before t  and  A_t = carried lanes + lanes appended before t,  trial t's
// emission (if any) is packet  E + NF_t + floor(A_t / P),  so a batch of
// trials is resolved with one block-wide prefix sum.  The call stops at the
// trial that completes its last output packet; later trials are not consumed.
//
// k_trials draws one row (one generator call) or several rows one after the
// other from the same stream (Dirichlet's GammaGen rows, Wishart's chi-squared
// rows), which stay in one launch with the stream's window and its unused
// words in shared memory.  Rows may be fixed runs of packets (integral alpha,
// alpha = 1): trials that are always fully accepted.
//
// Bound by instruction issue.  The tempered words of the two newest engine
// blocks are a ring of 4 992 32-bit words, a trial's words follow each other
// in it, and all indices are 32-bit: gamma(0.5) float at 4096 x 4096 on 608
// engines took 20 warp-instructions per sample (348 us) with 64-bit stream
// positions mapped to the ring per word.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/gpurand.h"
#include "gr_samplers.cuh"

namespace gr {

namespace {

constexpr int kTrThreads = 320;     // ten warps; 312 of the threads make a block's words
constexpr int kTrRing = 16 * kN;    // ring words: two blocks of 312 packets of 8

// RAW blocks kept untempered: two, each made from the other, or one, made over
// itself behind one more barrier, where the CTA needs the room.  BATCH: most
// trials of a batch (a block holds 104 trials of three packets, 156 of two, and
// at most 313 of one).
template <int RAW, int BATCH>
struct TrialSmem {
  static constexpr int kRaw = RAW, kBatch = BATCH;
  uint64_t raw[RAW][kLanes][kN];
  alignas(16) uint32_t w[kTrRing];
  alignas(16) uint32_t cand[BATCH * 8];  // accepted candidates (double: four per trial)
  uint32_t scan[BATCH];                  // exclusive: (fulls << 16) | lanes appended
  uint32_t emit[BATCH + 1];              // output packet (from the batch's first) of each FIFO packet
  uint64_t fifo[2][16];                  // carried lanes (ping-pong)
  uint32_t warp_tot[kTrThreads / 32];
  int tstar;
  uint8_t mask[BATCH];
  TrialRow row;
};
using EngSmem = TrialSmem<2, kTrThreads>;  // an engine's call
using SetSmem = TrialSmem<1, 160>;         // a parameter set: beside it lies the next set's window

// Where a stream stands in the ring.
struct TrialPos {
  int sp;      // ring index of the next trial's first word
  int av;      // words made and not used
  int64_t nb;  // blocks made
};

// The ten warps that draw; a set's CTA has an eleventh.
template <class SM>
__device__ __forceinline__ void tr_sync() {
  if (SM::kRaw == 2) __syncthreads();
  else asm volatile("bar.sync 1, %0;" ::"n"(kTrThreads) : "memory");
}

// The next engine block: two lanes per thread (words 2 h and 2 h + 1 of a packet
// are neighbours in the ring), word i + 156 from word i made by the same thread,
// word 311 with the block's word 0 made again.
template <class SM>
__device__ __forceinline__ void next_block(SM& sm, TrialPos& ps) {
  const int from = SM::kRaw == 2 ? (int)(ps.nb & 1) : 0, to = SM::kRaw == 2 ? from ^ 1 : 0;
  const int tid = threadIdx.x;
  uint32_t* ring = sm.w + (ps.nb & 1) * (kTrRing / 2);
  const int h = tid >= kM ? 1 : 0, i = tid - h * kM;
  uint64_t lo[2], hi[2];
  if (tid < 2 * kM) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint64_t* old = sm.raw[from][2 * h + q];
      const uint64_t c = old[i + kM];
      lo[q] = mt_twist(old[i], old[i + 1], c);
      const uint64_t b = i == kM - 1 ? mt_twist(old[0], old[1], old[kM]) : old[i + kM + 1];
      hi[q] = mt_twist(c, b, lo[q]);
    }
  }
  if (SM::kRaw == 1) tr_sync<SM>();
  if (tid < 2 * kM) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      sm.raw[to][2 * h + q][i] = lo[q];
      sm.raw[to][2 * h + q][i + kM] = hi[q];
    }
    *reinterpret_cast<ulonglong2*>(ring + 8 * i + 4 * h) = make_ulonglong2(mt_temper(lo[0]), mt_temper(lo[1]));
    *reinterpret_cast<ulonglong2*>(ring + 8 * (i + kM) + 4 * h) = make_ulonglong2(mt_temper(hi[0]), mt_temper(hi[1]));
  }
  ++ps.nb;
  ps.av += 8 * kN;
  tr_sync<SM>();
}

// A row's candidate at the ring index a of its trial, lane j.
template <int DT, int RK, class SM>
__device__ __forceinline__ bool trial_eval(const SM& sm, const DistParams& d, const int rk, const int U, const int a,
                                           const int j, uint64_t& c) {
  auto word = [&](int q) -> uint32_t {
    int i = a + q;
    i -= i >= kTrRing ? kTrRing : 0;
    return sm.w[i];
  };
  auto rval = [&](int r) -> uint64_t {
    int i = a + 2 * r;
    i -= i >= kTrRing ? kTrRing : 0;
    return *reinterpret_cast<const uint64_t*>(&sm.w[i]);
  };
  auto rej = [&](auto k) { return rej_trial<decltype(k)::value, DT>(d, 0, j, word, rval, c); };
  if (RK >= 0) return rej(std::integral_constant<int, RK < 0 ? 0 : RK>{});
  // NormalExp.h:527-534 (alpha = 1), :577-587 (integral alpha)
  if (DT == SD_F32) {
    if (rk == kRowExp) {
      c = f2u(d.fb * (-(logf_(1.0f - ur_f(word(j))) / 1.0f)));
    } else {
      constexpr float e = 1.1920928955078125e-07f / 8;
      float y = ur_f(word(j)) + e;
      for (int t = 1; t < U; ++t) y = y * (ur_f(word(8 * t + j)) + e);
      c = f2u(-(d.fb * logf_(y)));
    }
  } else {
    if (rk == kRowExp) {
      const double l = -(log_(one_minus_ur_d(rval(j))) / 1.0);
      c = d2u((d.flags & kParamUnitScale) ? l : d.db * l);
    } else {
      double y = ur_nz_int(rval(j));
      for (int t = 1; t < U; ++t) y = y * ur_nz_int(rval(4 * t + j));
      const double l = log_(y);
      c = d2u((d.flags & kParamUnitScale) ? -l : -(d.db * l));
    }
  }
  return true;
}

// Npk output packets of one row to out (CUT: its first `count` values only),
// from the stream at ps; rcnt lanes carried in sm.fifo[fsl].  False: the block
// cap came first.
template <int DT, int RK, bool CUT, class SM, class V>
__device__ __forceinline__ bool draw_row(SM& sm, const DistParams& d, const int rk, const int U, const float per_packet,
                                         V* out, const int64_t Npk, int64_t count, TrialPos& ps, int& rcnt, int& fsl,
                                         const int64_t max_blocks) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  constexpr uint32_t kFull = (1u << P) - 1u;
  constexpr int kBatch = SM::kBatch;
  V* cand = reinterpret_cast<V*>(sm.cand);
  const int tid = threadIdx.x;
  const int Wt = 8 * U;
  int64_t left = Npk;
  while (left > 0) {
    if (ps.av < Wt) {
      if (ps.nb >= max_blocks) return false;
      next_block(sm, ps);
    }
    // a batch: the trials whose words exist, and near the end of the row no
    // more than it should still need
    const int need = (int)min(left, (int64_t)1 << 20);
    const float want = (float)need * per_packet;
    const int B = min(ps.av / Wt, min(kBatch, (int)(CUT ? fminf(want, 1e6f) : want) + 4));
    // ---- candidates and accept masks
    for (int e0 = 0; e0 < B * P; e0 += kTrThreads) {
      const int e = e0 + tid, t = e / P, j = e % P;
      bool acc = false;
      uint64_t c = 0;
      if (e < B * P) {
        int a = ps.sp + t * Wt;
        a -= a >= kTrRing ? kTrRing : 0;
        acc = trial_eval<DT, RK>(sm, d, rk, U, a, j, c);
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, acc);
      if (acc) cand[e] = (V)c;
      if (j == 0 && e < B * P) sm.mask[t] = (uint8_t)((bal >> (tid & 31)) & kFull);
    }
    tr_sync<SM>();
    // ---- prefix sums over trials: (fulls << 16) |
    // appended lanes
    const uint32_t m0 = tid < B ? sm.mask[tid] : 0;
    const uint32_t v0 = m0 == kFull ? 1u << 16 : (uint32_t)__popc(m0);
    uint32_t v = v0;
    if (tid < kBatch) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, v, o);
        if ((tid & 31) >= o) v += x;
      }
      if ((tid & 31) == 31) sm.warp_tot[tid >> 5] = v;
    }
    if (tid == kTrThreads - 1) sm.tstar = B;
    tr_sync<SM>();
    // ---- this thread's trial: its emission, if any
    if (tid < B) {
#pragma unroll
      for (int w = 0; w < kBatch / 32 - 1; ++w) v += w < (tid >> 5) ? sm.warp_tot[w] : 0u;
      const uint32_t ex = v - v0;
      const int at = rcnt + (int)(ex & 0xffffu), nf = (int)(ex >> 16);
      const bool full = m0 == kFull;
      const bool cross = !full && (at + (int)__popc(m0)) / P > at / P;
      const int ei = nf + at / P;
      sm.scan[tid] = ex;
      if (cross) sm.emit[at / P] = (uint32_t)ei;
      if ((full || cross) && ei == need - 1) sm.tstar = tid + 1;
    }
    tr_sync<SM>();
    // trials consumed, and the FIFO level and emissions after them
    const int Bu = sm.tstar;
    const uint32_t ml = sm.mask[Bu - 1], sl = sm.scan[Bu - 1];
    const int a_end = rcnt + (int)(sl & 0xffffu) + (ml == kFull ? 0 : __popc(ml));
    const int nf_end = (int)(sl >> 16) + (ml == kFull ? 1 : 0);
    const int qe = a_end / P;  // FIFO packets emitted
    auto put = [&](int at, uint64_t x) {
      if (RK == RK_BETA_SMALL) x = beta_post<DT == SD_F64>(x, d);
      if (DT == SD_I32H) {
        // BinomialGen returns trials - res when p > 1/2 (Discrete.h:1051)
        const int32_t q = (int32_t)u2f((uint32_t)x);
        x = (uint32_t)((RK == RK_BINOMIAL && d.ib) ? (int32_t)d.fh - q : q);
      }
      if (!CUT || at < count) out[at] = (V)x;
    };
    // ---- write outputs
    for (int e = tid; e < Bu * P; e += kTrThreads) {
      const int t = e / P, j = e % P;
      const uint32_t m = sm.mask[t];
      if (!((m >> j) & 1u)) continue;
      const uint32_t s = sm.scan[t];
      const int at = rcnt + (int)(s & 0xffffu);
      if (m == kFull) {
        put(((int)(s >> 16) + at / P) * P + j, cand[e]);
      } else {
        const int f = at + __popc(m & ((1u << j) - 1u)), q = f / P;
        if (q < qe) put((int)sm.emit[q] * P + f % P, cand[e]);
        else sm.fifo[fsl ^ 1][f - qe * P] = cand[e];  // the FIFO keeps the plain draws
      }
    }
    // carried lanes: emitted with the batch's first FIFO packet, or still carried
    if (tid < rcnt) {
      if (qe > 0) put((int)sm.emit[0] * P + tid, sm.fifo[fsl][tid]);
      else sm.fifo[fsl ^ 1][tid] = sm.fifo[fsl][tid];
    }
    out += (int64_t)(nf_end + qe) * P;
    if (CUT) count -= (int64_t)(nf_end + qe) * P;
    left -= nf_end + qe;
    rcnt = a_end - qe * P;
    fsl ^= 1;
    ps.sp += Bu * Wt;
    ps.sp -= ps.sp >= kTrRing ? kTrRing : 0;
    ps.av -= Bu * Wt;
    tr_sync<SM>();
  }
  return true;
}

// The engine's state after a call that ends inside the newest block (a trial or
// unit is evaluated in the batch after the block that holds its last word).
template <bool HALF>
__device__ __forceinline__ void leave_engine(const EngSmem& sm, EngState* st, const TrialPos& ps) {
  const int tid = threadIdx.x;
  if (ps.nb > 0) {
    const int cur = (int)(ps.nb & 1);
    const int rr = kN - ps.av / 8;  // packets used of it; a half packet counts as used
    for (int t = tid; t < kLanes * kN; t += kTrThreads) {
      const int l = t / kN, i = t % kN;
      st->win[l][i] = i < kN - rr ? sm.raw[cur ^ 1][l][rr + i] : sm.raw[cur][l][i - (kN - rr)];
    }
  }
  if (tid == 0) {
    if (HALF && ps.nb > 0) {
      const bool half = (ps.av & 7) == 4;  // ends mid-packet: the upper half stays cached
      if (half)
        for (int q = 0; q < 4; ++q) st->half_cache[q] = sm.w[ps.sp + q];
      st->half_valid = half ? 1 : 0;
    }
    st->consumed += (uint64_t)(ps.nb * kN - ps.av / 8);
  }
}

// The row's kind picks a copy of the loop of its own: with the kind tested per
// trial in one loop 64 rows of 10^6 gamma(0.5) floats on 608 engines took 1 660
// us instead of 1 580, and 2 10^5 parameter sets 12.0 ms instead of 11.2.
template <int DT, bool CUT, class SM, class V>
__device__ __forceinline__ bool draw_kind(SM& sm, const TrialRow& row, V* out, const int64_t Npk, const int64_t count,
                                          TrialPos& ps, int& rcnt, int& fsl, const int64_t max_blocks) {
  if (row.rk == RK_GAMMA_GS)
    return draw_row<DT, RK_GAMMA_GS, CUT>(sm, row.d, row.rk, 3, row.per_packet, out, Npk, count, ps, rcnt, fsl, max_blocks);
  if (row.rk == RK_GAMMA_TAN)
    return draw_row<DT, RK_GAMMA_TAN, CUT>(sm, row.d, row.rk, 2, row.per_packet, out, Npk, count, ps, rcnt, fsl, max_blocks);
  return draw_row<DT, -1, CUT>(sm, row.d, row.rk, row.packets, row.per_packet, out, Npk, count, ps, rcnt, fsl, max_blocks);
}

// RK >= 0: one row (args) of that kind; RK < 0: `rows` rows from memory, row i
// written at out + i * row_stride elements.
template <int DT, int RK>
__global__ void __launch_bounds__(kTrThreads, 4) k_trials(Plan p, TrialRow args, const TrialRow* rows, int nrows,
                                                          int64_t row_stride, int64_t max_blocks) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  constexpr bool kHalf = DT == SD_I32H;
  using V = typename std::conditional<DT == SD_F64, uint64_t, uint32_t>::type;
  extern __shared__ __align__(16) uint8_t tr_dyn[];
  EngSmem& sm = *reinterpret_cast<EngSmem*>(tr_dyn);
  const int k = blockIdx.x, tid = threadIdx.x;
  EngState* st = p.eng + k;
  int64_t off, n;
  slice_left(p, k, off, n);
  if (n == 0) return;
  const int64_t Npk = n / P;  // output packets of a row

  const int c0w = (kHalf && st->half_valid) ? 4 : 0;
  for (int i = tid; i < kLanes * kN; i += kTrThreads) (&sm.raw[0][0][0])[i] = (&st->win[0][0])[i];
  // the engine's cached half packet goes before the first block's words
  if (kHalf && tid < 4) sm.w[kTrRing - 4 + tid] = st->half_cache[tid];
  TrialPos ps{c0w ? kTrRing - 4 : 0, c0w, 0};
  bool ok = true;
  for (int r = 0; r < (RK < 0 ? nrows : 1) && ok; ++r) {
    __syncthreads();  // the window is there; the last row's carried lanes are out
    if (RK < 0) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(rows + r);
      for (int i = tid; i < (int)(sizeof(TrialRow) / 4); i += kTrThreads) reinterpret_cast<uint32_t*>(&sm.row)[i] = src[i];
      __syncthreads();
    }
    const TrialRow& row = RK < 0 ? sm.row : args;
    const int rk = row.rk;
    GenSlot* gs = &row.gen[k].s[0];
    V* out = reinterpret_cast<V*>(p.out) + (RK < 0 ? (int64_t)r * row_stride : 0) + off;
    const bool carries = RK >= 0 || rk <= RK_GAMMA_TAN;
    int rcnt = carries ? gs->rest_cnt : 0, fsl = 0;
    if (tid < 16)
      sm.fifo[0][tid] = DT == SD_F64
                            ? ((uint64_t)gs->rest[2 * (tid & 7)] | ((uint64_t)gs->rest[2 * (tid & 7) + 1] << 32))
                            : (uint64_t)gs->rest[tid];
    if (RK >= 0)
      ok = draw_row<DT, RK, false>(sm, row.d, rk, row.packets, row.per_packet, out, Npk, 0, ps, rcnt, fsl, max_blocks);
    else
      ok = draw_kind<DT, false>(sm, row, out, Npk, 0, ps, rcnt, fsl, max_blocks);
    if (carries) {
      if (tid == 0) gs->rest_cnt = rcnt;
      if (DT == SD_F64) {
        if (tid < 8) {
          gs->rest[2 * tid] = (uint32_t)sm.fifo[fsl][tid];
          gs->rest[2 * tid + 1] = (uint32_t)(sm.fifo[fsl][tid] >> 32);
        }
      } else if (tid < 16) {
        gs->rest[tid] = (uint32_t)sm.fifo[fsl][tid];
      }
    }
  }

  if (tid == 0 && !ok) atomicOr(&st->status, (int)GR_DEV_REJECT_LIMIT);
  leave_engine<kHalf>(sm, st, ps);
}

// ---------------------------------------------------------------- fixed units
// Kinds whose unit of P outputs takes U packets (half packets for the int32
// kind): the units whose words exist, a thread per output.  Bound by instruction
// issue.  4096 x 4096 on 608 engines, us, with packets of 64-bit words found by
// 64-bit position / here: gamma(5) f32 213 / 154, f64 526 / 471, binomial(20) 842 /
// 474.
template <int KIND, int DT>
__global__ void __launch_bounds__(kTrThreads, 4) k_units(Plan p, DistParams d, int U) {
  constexpr int P = DT == SD_F32 ? 8 : 4;
  constexpr bool kHalf = DT == SD_I32H;
  extern __shared__ __align__(16) uint8_t tr_dyn[];
  EngSmem& sm = *reinterpret_cast<EngSmem*>(tr_dyn);
  const int k = blockIdx.x, tid = threadIdx.x;
  EngState* st = p.eng + k;
  const int64_t g0 = (int64_t)k * p.gran_per_k + min((int64_t)k, p.gran_rem);
  const int64_t ng = p.gran_per_k + ((int64_t)k < p.gran_rem ? 1 : 0);
  const int64_t off = g0 * p.gran, n = ng * p.gran;
  if (n == 0) return;
  const int Wt = (kHalf ? 4 : 8) * U;
  const int c0w = (kHalf && st->half_valid) ? 4 : 0;
  for (int i = tid; i < kLanes * kN; i += kTrThreads) (&sm.raw[0][0][0])[i] = (&st->win[0][0])[i];
  if (kHalf && tid < 4) sm.w[kTrRing - 4 + tid] = st->half_cache[tid];
  __syncthreads();
  TrialPos ps{c0w ? kTrRing - 4 : 0, c0w, 0};
  int64_t left = n / P, o = off;
  while (left > 0) {
    while (ps.av < Wt) next_block(sm, ps);
    const int B = (int)min((int64_t)(ps.av / Wt), left);
    for (int e = tid; e < B * P; e += kTrThreads) {
      const int t = e / P, j = e % P;
      int a = ps.sp + t * Wt;
      a -= a >= kTrRing ? kTrRing : 0;
      auto word = [&](int64_t q) -> uint32_t {
        int i = a + (int)q;
        i -= i >= kTrRing ? kTrRing : 0;
        return sm.w[i];
      };
      auto rword = [&](int64_t r) -> uint64_t {
        int i = a + 2 * (int)r;
        i -= i >= kTrRing ? kTrRing : 0;
        return *reinterpret_cast<const uint64_t*>(&sm.w[i]);
      };
      staged_value<KIND, DT>(p, d, U, 0, j, o + e, word, rword);
    }
    o += (int64_t)B * P;
    left -= B;
    ps.sp += B * Wt;
    ps.sp -= ps.sp >= kTrRing ? kTrRing : 0;
    ps.av -= B * Wt;
    __syncthreads();
  }
  leave_engine<kHalf>(sm, st, ps);
  // a call served from the cached half packet alone leaves none
  if (kHalf && tid == 0 && ps.nb == 0 && c0w) st->half_valid = ps.av ? 1 : 0;
}

template <int KIND, int DT>
cudaError_t run_units(const Plan& p, const DistParams& d, int U, cudaStream_t s) {
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (U < 1 || U > kTrRing / 2 / 8) return cudaErrorNotSupported;
  if (!attr[dev]) {
    cudaError_t e =
        cudaFuncSetAttribute(k_units<KIND, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EngSmem));
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  k_units<KIND, DT><<<p.K, kTrThreads, sizeof(EngSmem), s>>>(p, d, U);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- parameter sets
// Batched GammaGen<float> sets: set i from its own Vmt19937_64(seed + 4 i)
// with a fresh generator, ceil(count / 8) packets of which the first `count`
// values are kept.  Bound by instruction issue, like the rest of this file.  A
// CTA takes sets in turn; four threads of an eleventh warp seed the next set's
// engine (PacketRandomEngine.h:256-265: 311 dependent steps of a 64-bit
// multiply, 5 us) while the ten others draw from the current one.  2 10^5 sets
// of up to 4 096 values: 13.4 ms with a CTA per set that seeds first, 11.2 ms
// here (11.3 with three CTAs per SM and no spilled registers).
struct VopSmem {
  SetSmem t;
  uint64_t seeds[kLanes][kN];
};

__global__ void __launch_bounds__(kTrThreads + 32, 4) k_gamma_sets(VopArgs va) {
  extern __shared__ __align__(16) uint8_t tr_dyn[];
  VopSmem& vs = *reinterpret_cast<VopSmem*>(tr_dyn);
  SetSmem& sm = vs.t;
  const int tid = threadIdx.x;
  for (int64_t set = blockIdx.x; set < va.nsets; set += gridDim.x) {
    if (set == blockIdx.x) {
      if (tid >= kTrThreads && tid < kTrThreads + kLanes) {
        const int l = tid - kTrThreads;
        uint64_t v = va.seed + 4ull * (uint64_t)set + (uint64_t)l;
        vs.seeds[l][0] = v;
        for (int i = 1; i < kN; ++i) vs.seeds[l][i] = v = (v ^ (v >> 62)) * kSeedF + (uint64_t)i;
      }
      __syncthreads();
    }
    const int64_t count = va.counts[set];
    if (tid < kTrThreads) {
      for (int i = tid; i < kLanes * kN; i += kTrThreads) (&sm.raw[0][0][0])[i] = (&vs.seeds[0][0])[i];
      if (tid == 0) {
        // GammaGen's branch and constants, NormalExp.h:446-460, 533-604
        const float alpha = va.a[set];
        const int cnt = (int)alpha;
        TrialRow& r = sm.row;
        r.rk = alpha < 1 ? (int)RK_GAMMA_GS : alpha == 1 ? kRowExp : ((float)cnt == alpha && cnt < 20) ? kRowInt : (int)RK_GAMMA_TAN;
        r.packets = r.rk == RK_GAMMA_GS ? 3 : r.rk == kRowExp ? 1 : r.rk == kRowInt ? cnt : 2;
        // trials per output packet: e + a over e G(a + 1) is at most 1.39; the
        // tan proposal's falls from pi at 1 to 1.77
        r.per_packet = r.rk == RK_GAMMA_GS ? 1.4f : r.rk == RK_GAMMA_TAN ? 1.77f + 0.35f / (alpha - 0.75f) : 1.0f;
        r.d.fa = alpha;
        r.d.fb = va.b[set];
        r.d.fc = 1 / alpha;
        r.d.fd = alpha - 1;
        r.d.fe = (float)(2.7182818284590452 / (alpha + 2.7182818284590452));
        r.d.ff = sqrtf(2 * alpha - 1);
        r.d.fh = 0x1p-18f * (1.0f + 40.0f / alpha);
      }
    }
    __syncthreads();
    if (tid >= kTrThreads) {
      const int64_t next = set + gridDim.x;
      if (tid < kTrThreads + kLanes && next < va.nsets) {
        const int l = tid - kTrThreads;
        uint64_t v = va.seed + 4ull * (uint64_t)next + (uint64_t)l;
        vs.seeds[l][0] = v;
        for (int i = 1; i < kN; ++i) vs.seeds[l][i] = v = (v ^ (v >> 62)) * kSeedF + (uint64_t)i;
      }
    } else if (count > 0) {
      const TrialRow& r = sm.row;
      TrialPos ps{0, 0, 0};
      int rcnt = 0, fsl = 0;
      const int64_t Npk = (count + 7) / 8;
      const int64_t max_blocks = ((16 * Npk + 4096) * 8 * r.packets) / (kN * 8) + 64;
      const bool ok = draw_kind<SD_F32, true>(sm, r, reinterpret_cast<uint32_t*>(va.out) + va.offsets[set], Npk, count, ps,
                                              rcnt, fsl, max_blocks);
      if (!ok && tid == 0) atomicOr(va.status, (int)GR_DEV_REJECT_LIMIT);
    }
    __syncthreads();
  }
}

template <int DT, int RK>
cudaError_t run_trials(const Plan& p, const TrialRow& row, const TrialRow* rows, int nrows, int64_t row_stride,
                       int64_t max_blocks, cudaStream_t s) {
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  constexpr size_t smem = sizeof(EngSmem);
  if (!attr[dev]) {
    cudaError_t e = cudaFuncSetAttribute(k_trials<DT, RK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  k_trials<DT, RK><<<p.K, kTrThreads, smem, s>>>(p, row, rows, nrows, row_stride, max_blocks);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_reject(const Plan& p, const DistParams& d, int rk, float per_packet, int64_t max_blocks,
                          cudaStream_t s) {
  const int dt = d.dtype == GR_F32 ? SD_F32 : d.dtype == GR_F64 ? SD_F64 : SD_I32H;
  TrialRow row{};
  row.d = d;
  row.gen = p.gen;
  row.rk = rk;
  row.packets = rk == RK_GAMMA_GS ? 3 : (rk >= RK_POISSON ? 1 : 2);
  row.per_packet = per_packet;
#define GR_RJ(R)                                                                               \
  if (rk == R) {                                                                               \
    if (dt == SD_F32) return run_trials<SD_F32, R>(p, row, nullptr, 1, 0, max_blocks, s);      \
    if (dt == SD_F64) return run_trials<SD_F64, R>(p, row, nullptr, 1, 0, max_blocks, s);      \
  }
  GR_RJ(RK_GAMMA_GS)
  GR_RJ(RK_GAMMA_TAN)
  GR_RJ(RK_BETA_SMALL)
#undef GR_RJ
  if (rk == RK_POISSON && dt == SD_I32H) return run_trials<SD_I32H, RK_POISSON>(p, row, nullptr, 1, 0, max_blocks, s);
  if (rk == RK_BINOMIAL && dt == SD_I32H) return run_trials<SD_I32H, RK_BINOMIAL>(p, row, nullptr, 1, 0, max_blocks, s);
  return cudaErrorNotSupported;
}

cudaError_t launch_units(const Plan& p, const DistParams& d, int U, cudaStream_t s) {
  const bool f32 = d.dtype == GR_F32, f64 = d.dtype == GR_F64;
  if (d.kind == GR_GAMMA || d.kind == GR_CHI_SQUARED) {
    if (f32) return run_units<GR_GAMMA, SD_F32>(p, d, U, s);
    if (f64) return run_units<GR_GAMMA, SD_F64>(p, d, U, s);
  }
  if (d.kind == GR_STUDENT_T) {
    if (f32) return run_units<GR_STUDENT_T, SD_F32>(p, d, U, s);
    if (f64) return run_units<GR_STUDENT_T, SD_F64>(p, d, U, s);
  }
  if (d.kind == GR_BINOMIAL && d.dtype == GR_I32) return run_units<GR_BINOMIAL, SD_I32H>(p, d, U, s);
  return cudaErrorNotSupported;
}

cudaError_t launch_gamma_rows(const Plan& p, int dtype, const TrialRow* rows, int nrows, int64_t row_stride,
                              int64_t max_blocks, cudaStream_t s) {
  if (dtype == GR_F64) return run_trials<SD_F64, -1>(p, TrialRow{}, rows, nrows, row_stride, max_blocks, s);
  return run_trials<SD_F32, -1>(p, TrialRow{}, rows, nrows, row_stride, max_blocks, s);
}

cudaError_t launch_gamma_sets(const VopArgs& va, cudaStream_t s) {
  static int grid[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  constexpr size_t smem = sizeof(VopSmem);
  if (!grid[dev]) {
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gamma_sets, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    grid[dev] = 4 * sms;
  }
  k_gamma_sets<<<(unsigned)std::min<int64_t>(va.nsets, grid[dev]), kTrThreads + 32, smem, s>>>(va);
  return cudaGetLastError();
}

}  // namespace gr
