// CompressMask rejection samplers (gr_samplers.cuh: rej_trial) over raw words
// in memory, data parallel.
//
// Trial t of a call reads a fixed run of words, so every trial's accept mask
// can be made at once.  With NF_t the fully accepted trials before t and A_t
// the carried lanes plus the lanes of partial trials before t, the automaton
// (arch/AVX/PacketFilter.h:147-184) emits at trial t
//   a fully accepted trial as it is,       as output packet NF_t + A_t / P,
//   FIFO packet q = A_t / P when A_t + (its lanes) reaches (q + 1) P, likewise:
//   k_rw_masks   accept masks, and per tile of 256 trials the counts;
//   k_rw_scan    the counts before each tile;
//   k_rw_emit    per tile the emissions, then one thread per output lane: the
//                candidate of the trial, or of the FIFO lane found by walking
//                the trials backwards;
//   k_rw_finish  engine window, caches and carried lanes after the last trial.
// Bound by the arithmetic of the candidates.  One engine, gamma(0.5) double,
// 10^6: 0.57 ms in the count / scan / write / gather kernels this replaces,
// which ran 128 CTAs of 160 threads twice over the trials.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/gpurand.h"
#include "gr_samplers.cuh"

namespace gr {

namespace {

constexpr int kTileTrials = 256;

struct RwArgs {
  Plan p;
  DistParams d;
  const CallSnap* snap;
  RwLayout L;
  uint8_t* mask;    // [K][L.mstride]
  int2* cnt;        // [K][L.tiles] full trials, lanes of partial trials
  int64_t* start;   // [K][L.tiles][2] the same before the tile (lanes: with the carried ones)
  int64_t* end;     // [K][3] trials used, FIFO lanes after them, output packets
  int64_t* done;
};

template <int RK>
__host__ __device__ constexpr int trial_packets() {
  return RK == RK_GAMMA_GS ? 3 : (RK == RK_POISSON || RK == RK_BINOMIAL) ? 1 : 2;
}
template <int DT>
__host__ __device__ constexpr int lanes_of() {
  return DT == SD_F32 ? 8 : 4;
}

__device__ __forceinline__ int64_t limit_of(const RwArgs& a, int k) {
  const int64_t ng = a.p.gran_per_k + ((int64_t)k < a.p.gran_rem ? 1 : 0);
  return ng - min(a.done[k], ng);
}

// Words of engine k for rej_trial: 32-bit words of the call's stream (the
// int32 kinds' stream starts with the engine's cached half packet), 64-bit
// lanes by packet.
template <int DT>
struct Source {
  const uint64_t* w;
  int64_t stride;
  int c0w;
  const uint32_t* cw;
  __device__ __forceinline__ Source(const RwArgs& a, int k)
      : w(a.p.words + (size_t)k * kLanes * a.p.wstride + kN), stride(a.p.wstride),
        c0w(DT == SD_I32H && a.snap[k].half_valid ? 4 : 0), cw(a.snap[k].half_cache) {}
  __device__ __forceinline__ uint64_t lane64(int64_t packet, int l) const {
    return mt_temper(__ldg(w + (size_t)l * stride + packet));
  }
  __device__ __forceinline__ uint32_t word(int64_t q) const {
    if (DT == SD_I32H) {
      if (q < c0w) return cw[q];
      q -= c0w;
    }
    const uint64_t v = lane64(q >> 3, (int)((q & 7) >> 1));
    return (q & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
  }
};

template <int RK, int DT>
__device__ __forceinline__ bool accepted(const RwArgs& a, const Source<DT>& src, int64_t t, int j) {
  uint64_t c;
  return rej_trial<RK, DT, false>(
      a.d, t, j, [&](int64_t q) { return src.word(q); },
      [&](int64_t r) { return src.lane64(r >> 2, (int)(r & 3)); }, c);
}

// Accepted lane j of trial t; t < 0: lane j of those carried into the call.
template <int RK, int DT>
__device__ __forceinline__ uint64_t value_at(const RwArgs& a, const Source<DT>& src, int k, int64_t t, int j) {
  if (t < 0) {
    const GenSlot& gs = a.p.gen[k].s[0];
    return DT == SD_F64 ? ((uint64_t)gs.rest[2 * j] | ((uint64_t)gs.rest[2 * j + 1] << 32)) : (uint64_t)gs.rest[j];
  }
  return rej_value<RK, DT>(
      a.d, t, j, [&](int64_t q) { return src.word(q); },
      [&](int64_t r) { return src.lane64(r >> 2, (int)(r & 3)); });
}

constexpr int kRwThreads = 256;

template <int RK, int DT>
__global__ void __launch_bounds__(kRwThreads) k_rw_masks(RwArgs a) {
  constexpr int P = lanes_of<DT>();
  __shared__ int2 s_cnt[kRwThreads / 32];
  const int k = blockIdx.y, tid = threadIdx.x;
  const Source<DT> src(a, k);
  const int64_t t0 = (int64_t)blockIdx.x * kTileTrials;
  uint8_t* mk = a.mask + (size_t)k * a.L.mstride;
  int nf = 0, nl = 0;
  for (int e = tid; e < kTileTrials * P; e += kRwThreads) {
    const int64_t t = t0 + e / P;
    const int j = e % P;
    bool acc = false;
    if (t < a.L.T) acc = accepted<RK, DT>(a, src, t, j);
    const uint32_t bal = __ballot_sync(0xffffffffu, acc);
    const uint32_t m = (bal >> (tid & 31 & ~(P - 1))) & ((1u << P) - 1);
    if (j == 0 && t < a.L.T) {
      mk[t] = (uint8_t)m;
      const int cn = __popc(m);
      nf += cn == P ? 1 : 0;
      nl += cn == P ? 0 : cn;
    }
  }
  for (int o = 16; o; o >>= 1) {
    nf += __shfl_xor_sync(0xffffffffu, nf, o);
    nl += __shfl_xor_sync(0xffffffffu, nl, o);
  }
  if ((tid & 31) == 0) s_cnt[tid >> 5] = make_int2(nf, nl);
  __syncthreads();
  if (tid == 0) {
    int2 v = make_int2(0, 0);
    for (int w = 0; w < kRwThreads / 32; ++w) {
      v.x += s_cnt[w].x;
      v.y += s_cnt[w].y;
    }
    a.cnt[(size_t)k * a.L.tiles + blockIdx.x] = v;
  }
}

template <int P>
__global__ void __launch_bounds__(1024) k_rw_scan(RwArgs a) {
  __shared__ int64_t s_tot[2][32];
  __shared__ int64_t s_carry[2];
  const int k = blockIdx.x, tid = threadIdx.x, n = a.L.tiles, nw = blockDim.x >> 5;
  const int2* cnt = a.cnt + (size_t)k * n;
  int64_t* st = a.start + (size_t)k * n * 2;
  if (tid == 0) {
    s_carry[0] = 0;
    s_carry[1] = a.p.gen[k].s[0].rest_cnt;
  }
  __syncthreads();
  for (int b = 0; b < n; b += blockDim.x) {
    const int i = b + tid;
    const int2 c = i < n ? cnt[i] : make_int2(0, 0);
    int64_t v[2] = {c.x, c.y};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, v[q], o);
        if ((tid & 31) >= o) v[q] += y;
      }
      if ((tid & 31) == 31) s_tot[q][tid >> 5] = v[q];
    }
    __syncthreads();
    if (tid < 64) {
      const int q = tid >> 5, l = tid & 31;
      int64_t t = l < nw ? s_tot[q][l] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, t, o);
        if (l >= o) t += y;
      }
      s_tot[q][l] = t;
    }
    __syncthreads();
    const int64_t in0 = s_carry[0] + v[0] + ((tid >> 5) ? s_tot[0][(tid >> 5) - 1] : 0);
    const int64_t in1 = s_carry[1] + v[1] + ((tid >> 5) ? s_tot[1][(tid >> 5) - 1] : 0);
    if (i < n) {
      st[2 * i] = in0 - c.x;
      st[2 * i + 1] = in1 - c.y;
    }
    __syncthreads();
    if (tid == (int)blockDim.x - 1) {
      s_carry[0] = in0;
      s_carry[1] = in1;
    }
    __syncthreads();
  }
  if (tid == 0) {  // all planned trials; the trial that emits the call's last packet replaces it
    a.end[(size_t)k * 3] = a.L.T;
    a.end[(size_t)k * 3 + 1] = s_carry[1];
    a.end[(size_t)k * 3 + 2] = min(limit_of(a, k), s_carry[0] + s_carry[1] / P);
  }
}

// The FIFO lane `dist` places before the end of the FIFO as it is after trial
// t: its trial and lane (trial -1: one of the lanes carried into the call).
//
// fifo_far: the trials of t's tile are walked backwards, eight at a time where all
// are fully accepted; a lane of an earlier tile is found by its place in the FIFO,
// which the counts before each tile bracket.  Trial by trial all the way, shapes
// whose trials nearly all are fully accepted took up to 220 ms for 2^24 values
// (beta(1e-4, 1e-4) double; 1.7 ms so), gamma(1e-6) float 20 ms (0.38).
template <int P>
__device__ __noinline__ int2 fifo_far(const uint8_t* mk, const int64_t* st, int carried, int t, int dist) {
  constexpr uint64_t kAllFull = P == 8 ? ~0ull : 0x0f0f0f0f0f0f0f0full;
  for (;;) {
    const int tile = t >= 0 ? t / kTileTrials : 0, first = tile * kTileTrials;
    while (t >= first) {
      if ((t & 7) == 7 && __ldg(reinterpret_cast<const uint64_t*>(mk + t - 7)) == kAllFull) {
        t -= 8;
        continue;
      }
      uint32_t m = __ldg(mk + t);
      const int cn = __popc(m);
      if (cn != P) {
        if (dist <= cn) {
          for (int r = cn - dist; r > 0; --r) m &= m - 1;
          return make_int2(t, __ffs(m) - 1);
        }
        dist -= cn;
      }
      --t;
    }
    const int64_t q = st[2 * tile + 1] - dist;  // its place in the FIFO
    if (q < carried) return make_int2(-1, max((int)q, 0));
    int lo = 0, hi = tile;  // lanes before tile lo <= q < lanes before tile hi
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (st[2 * mid + 1] <= q) lo = mid;
      else hi = mid;
    }
    t = hi * kTileTrials - 1;
    dist = (int)(st[2 * hi + 1] - q);
  }
}
template <int P>
__device__ __forceinline__ void fifo_lane(const RwArgs& a, int k, int64_t& t, int64_t dist, int& j) {
  const uint8_t* mk = a.mask + (size_t)k * a.L.mstride;
  // ordinary shapes find it a few trials back, in the same tile
  const int64_t stop = max(t - 16, (t & ~(int64_t)(kTileTrials - 1)) - 1);
  for (; t > stop; --t) {
    uint32_t m = __ldg(mk + t);
    const int cn = __popc(m);
    if (cn == P) continue;
    if (dist <= cn) {
      for (int r = cn - (int)dist; r > 0; --r) m &= m - 1;
      j = __ffs(m) - 1;
      return;
    }
    dist -= cn;
  }
  const int2 f = fifo_far<P>(mk, a.start + (size_t)k * a.L.tiles * 2, a.p.gen[k].s[0].rest_cnt, (int)t, (int)dist);
  t = f.x;
  j = f.y;
}

template <int RK, int DT>
__global__ void __launch_bounds__(kRwThreads) k_rw_emit(RwArgs a) {
  constexpr int P = lanes_of<DT>();
  __shared__ int s_tot[2][kRwThreads / 32];
  __shared__ uint16_t s_em[kTileTrials];  // emission: trial | FIFO << 15
  __shared__ uint8_t s_back[kTileTrials]; // ... FIFO: lanes left after the packet
  const int k = blockIdx.y, tid = threadIdx.x;
  const int64_t limit = limit_of(a, k);
  const int64_t t0 = (int64_t)blockIdx.x * kTileTrials;
  const int64_t* st = a.start + ((size_t)k * a.L.tiles + blockIdx.x) * 2;
  const int64_t nf0 = st[0], a0 = st[1];
  const int64_t e0 = nf0 + a0 / P;  // the tile's first emission
  if (e0 >= limit) return;
  const int64_t t = t0 + tid;
  const uint32_t m = t < a.L.T ? a.mask[(size_t)k * a.L.mstride + t] : 0;
  const int cn = __popc(m);
  const bool full = t < a.L.T && cn == P;
  int v[2] = {full ? 1 : 0, full ? 0 : cn};
  const int c[2] = {v[0], v[1]};
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v[q], o);
      if ((tid & 31) >= o) v[q] += y;
    }
    if ((tid & 31) == 31) s_tot[q][tid >> 5] = v[q];
  }
  __syncthreads();
  int all[2] = {0, 0};
#pragma unroll
  for (int w = 0; w < kRwThreads / 32; ++w) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (w < (tid >> 5)) v[q] += s_tot[q][w];
      all[q] += s_tot[q][w];
    }
  }
  const int64_t at = a0 + v[1] - c[1];  // FIFO lanes before this trial
  const bool fifo = !full && (at + cn) / P > at / P;
  const int64_t E = nf0 + v[0] - c[0] + at / P;
  if (full || fifo) {
    s_em[E - e0] = (uint16_t)(tid | (fifo ? 0x8000 : 0));
    s_back[E - e0] = (uint8_t)((at + cn) % P);
    if (E == limit - 1) {
      a.end[(size_t)k * 3] = t + 1;
      a.end[(size_t)k * 3 + 1] = at + (full ? 0 : cn);
    }
  }
  __syncthreads();
  const int64_t ne = min(nf0 + all[0] + (a0 + all[1]) / P, limit) - e0;
  const Source<DT> src(a, k);
  const int64_t g0 = (int64_t)k * a.p.gran_per_k + min((int64_t)k, a.p.gran_rem) + a.done[k];
  for (int u0 = 0; u0 < ne * P; u0 += kRwThreads) {
    const int u = u0 + tid, i = u / P, j = u % P;
    int64_t tt = 0;
    int jj = j;
    if (u < ne * P) {
      tt = t0 + (s_em[i] & 0x7fff);
      if (s_em[i] & 0x8000) fifo_lane<P>(a, k, tt, (int64_t)s_back[i] + P - j, jj);
    }
    // the searches take different times: without this the warp's threads run
    // the long value code in groups (11 of 32 active, 332 us for 4.2 M doubles)
    __syncwarp();
    if (u >= ne * P) continue;
    uint64_t b = value_at<RK, DT>(a, src, k, tt, jj);
    if (RK == RK_BETA_SMALL) b = beta_post<DT == SD_F64>(b, a.d);
    const int64_t o = (g0 + e0 + i) * P + j;
    if (DT == SD_F64) {
      reinterpret_cast<uint64_t*>(a.p.out)[o] = b;
    } else if (DT == SD_I32H) {
      const int32_t r = (int32_t)u2f((uint32_t)b);
      // BinomialGen returns trials - res when p > 1/2 (Discrete.h:1051)
      reinterpret_cast<int32_t*>(a.p.out)[o] = (RK == RK_BINOMIAL && a.d.ib) ? (int32_t)a.d.fh - r : r;
    } else {
      reinterpret_cast<uint32_t*>(a.p.out)[o] = (uint32_t)b;
    }
  }
}

template <int RK, int DT>
__global__ void __launch_bounds__(256) k_rw_finish(RwArgs a) {
  constexpr int P = lanes_of<DT>();
  const int k = blockIdx.x, tid = threadIdx.x;
  if (limit_of(a, k) <= 0) return;
  EngState* st = a.p.eng + k;
  GenSlot* gs = &a.p.gen[k].s[0];
  const int64_t te = a.end[(size_t)k * 3], ae = a.end[(size_t)k * 3 + 1], emitted = a.end[(size_t)k * 3 + 2];
  const Source<DT> src(a, k);
  const int64_t np = te * trial_packets<RK>();
  const int f = (int)(ae % P);
  uint64_t v = 0;
  if (tid < f) {
    int64_t t = te - 1;
    int j;
    fifo_lane<P>(a, k, t, f - tid, j);
    v = value_at<RK, DT>(a, src, k, t, j);
  }
  __syncthreads();  // the lanes carried into the call are read before they are replaced
  if (tid < P) {
    if (DT == SD_F64) {
      gs->rest[2 * tid] = (uint32_t)v;
      gs->rest[2 * tid + 1] = (uint32_t)(v >> 32);
    } else {
      gs->rest[tid] = (uint32_t)v;
    }
  }
  if (np > 0) {
    const uint64_t* w = a.p.words + (size_t)k * kLanes * a.p.wstride;
    for (int t = tid; t < kLanes * kN; t += blockDim.x)
      st->win[t / kN][t % kN] = w[(size_t)(t / kN) * a.p.wstride + np + t % kN];
  }
  if (tid == 0) {
    gs->rest_cnt = f;
    if (DT == SD_I32H && np > 0) {
      // a trial is one packet's words: with a cached half packet first, the
      // last packet's upper half stays cached
      if (src.c0w) {
        const uint64_t lo = src.lane64(np - 1, 2), hi = src.lane64(np - 1, 3);
        st->half_cache[0] = (uint32_t)lo;
        st->half_cache[1] = (uint32_t)(lo >> 32);
        st->half_cache[2] = (uint32_t)hi;
        st->half_cache[3] = (uint32_t)(hi >> 32);
      }
    }
    st->consumed += (uint64_t)np;
    a.done[k] += emitted;
  }
}

constexpr size_t al(size_t x) { return (x + 255) / 256 * 256; }

template <int RK, int DT>
cudaError_t run_rw(const RwArgs& a, cudaStream_t s) {
  const dim3 grid((unsigned)a.L.tiles, (unsigned)a.p.K);
  k_rw_masks<RK, DT><<<grid, kRwThreads, 0, s>>>(a);
  k_rw_scan<lanes_of<DT>()><<<a.p.K, a.L.tiles > 256 ? 1024 : 256, 0, s>>>(a);
  k_rw_emit<RK, DT><<<grid, kRwThreads, 0, s>>>(a);
  k_rw_finish<RK, DT><<<a.p.K, 256, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

RwLayout reject_words_layout(int K, int64_t T) {
  RwLayout L{};
  L.T = T;
  L.tiles = (int32_t)((T + kTileTrials - 1) / kTileTrials);
  L.mstride = (int64_t)al((size_t)T);
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += al(b);
    return at;
  };
  L.o_mask = take((size_t)K * L.mstride);
  L.o_cnt = take((size_t)K * L.tiles * sizeof(int2));
  L.o_start = take((size_t)K * L.tiles * 16);
  L.o_end = take((size_t)K * 24);
  L.bytes = o;
  return L;
}

cudaError_t launch_reject_words(const Plan& p, const DistParams& d, int rk, const CallSnap* snap, const RwLayout& L,
                                char* scratch, int64_t* done, cudaStream_t s) {
  RwArgs a{};
  a.p = p;
  a.d = d;
  a.snap = snap;
  a.L = L;
  a.mask = reinterpret_cast<uint8_t*>(scratch + L.o_mask);
  a.cnt = reinterpret_cast<int2*>(scratch + L.o_cnt);
  a.start = reinterpret_cast<int64_t*>(scratch + L.o_start);
  a.end = reinterpret_cast<int64_t*>(scratch + L.o_end);
  a.done = done;
  if (L.tiles <= 0) return cudaSuccess;
  const int dt = d.dtype == GR_F32 ? SD_F32 : d.dtype == GR_F64 ? SD_F64 : SD_I32H;
#define GR_RW(R)                                       \
  if (rk == R) {                                       \
    if (dt == SD_F32) return run_rw<R, SD_F32>(a, s);  \
    if (dt == SD_F64) return run_rw<R, SD_F64>(a, s);  \
  }
  GR_RW(RK_GAMMA_GS)
  GR_RW(RK_GAMMA_TAN)
  GR_RW(RK_BETA_SMALL)
#undef GR_RW
  if (rk == RK_POISSON && dt == SD_I32H) return run_rw<RK_POISSON, SD_I32H>(a, s);
  if (rk == RK_BINOMIAL && dt == SD_I32H) return run_rw<RK_BINOMIAL, SD_I32H>(a, s);
  return cudaErrorNotSupported;
}

}  // namespace gr
