// BetaGen's general branch (NormalExp.h:970-975; FisherFGen over it) over raw
// words in memory, data parallel.
//
// Each output packet draws one packet from GammaGen(a), then one from
// GammaGen(b), from wherever the previous output packet stopped: a chain whose
// state at an output's start is the packet position x and the number of lanes
// each rejection component's CompressMask carries (arch/AVX/PacketFilter.h:
// 147-184).  A step of the chain needs only the accept masks, so:
//   k_chain_masks    the P-lane accept mask of every position;
//   k_chain_visits   per position and number of carried lanes, how many trials
//                    the draw starting there takes and the lanes it leaves;
//   k_chain_table    per segment of J positions, the state in which each
//                    possible entry state leaves it.  A warp follows all of
//                    them together; chains that reach the same state merge at
//                    boundaries 32, 64, 128, ... positions in, so that few are
//                    left after the first hundred positions;
//   k_chain_compose  the entry state of every segment from the call's first;
//   k_chain_walk     one warp per segment follows the true chain, one table
//                    read per component and output packet, and records each
//                    output packet's state;
//   k_chain_scan     output packets before each segment;
//   k_chain_emit     one thread per output lane: from the state recorded, the
//                    trials of each component's draw, then the lane's two
//                    values, from the draw's own trials or from an earlier
//                    output's trial that left the lane carried;
//   k_chain_finish   engine window and carried lanes after the last output.
// With few engines the chain runs in segments; with many, each engine's in one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/gpurand.h"
#include "gr_samplers.cuh"

namespace gr {

namespace {

constexpr int kEsc = 0xffff;         // no such state: the chain ran out of masks, or left the table
constexpr uint32_t kEntInit = 0xffffffu;  // entry position of the lanes carried into the call

template <bool R0, bool R1>
__host__ __device__ constexpr int entry_offsets() {
  // positions into a segment at which an output can start whose predecessor
  // started before it: a draw is at most 19 packets, and a component's trials
  // (accepted per lane with probability > 0.45) take a handful; a longer
  // overshoot ends the recorded chain, and the caller's fallback goes on
  return (R0 && R1) ? 32 : 64;
}
template <int P, bool R0, bool R1>
__host__ __device__ constexpr int entry_states() {
  return entry_offsets<R0, R1>() * (R0 ? P : 1) * (R1 ? P : 1);
}

// An output "adds" to a component's carried lanes unless its draw was one fully
// accepted trial.  adds[c]: the segment's last such output plus 1; prev[c]: the
// last segment before it that has one, plus 1 (0: none).
struct ChainSeg {
  int32_t nrec, bad, adds[2], prev[2];
};

struct ChainArgs {
  Plan p;
  BetaConsts bk;
  ChainLayout L;
  uint8_t* mask;   // [K][rejection components][L.mstride]
  uint8_t* vis;    // [K][rejection components][L.mstride][P]: trials - 1 << 3 | lanes left
  uint16_t* tab;
  uint16_t* gtab;
  int32_t* entry;
  ChainSeg* seg;
  int64_t* ebase;
  uint32_t* rec;   // per output packet: x | lanes carried << 24 (component 0), << 27 (component 1)
  uint16_t* prev;  // [rejection components][K * Sg][L.rcap] the segment's last output before it that adds, plus 1
  int64_t* done;
  int32_t M;       // positions with masks
};
// A visit entry: trials - 1 << 3 | lanes left; with nothing carried (P = 1,
// PoissonGen's chain) the step's half packets - 1.  kNoVisit: a draw that the
// positions in memory do not finish.
template <int P>
constexpr int kNoVisit = P == 1 ? 255 : 31;
template <int P>
__device__ __forceinline__ int visit_trials(uint32_t e) {
  return P == 1 ? (int)e : (int)(e >> 3);
}

__device__ __forceinline__ int64_t limit_of(const ChainArgs& a, int k) {
  const int64_t ng = a.p.gran_per_k + ((int64_t)k < a.p.gran_rem ? 1 : 0);
  return ng - min(a.done[k], ng);
}

// a tempered word of packet x, lane l of the engine's words w
__device__ __forceinline__ uint64_t tw(const uint64_t* w, int64_t stride, int x, int l) {
  return mt_temper(__ldg(w + (size_t)l * stride + kN + x));
}

// ---------------------------------------------------------------- masks
constexpr int kMaskThreads = 256;
template <int DT, int T0, int T1>
__global__ void __launch_bounds__(kMaskThreads) k_chain_masks(ChainArgs a) {
  constexpr int P = beta_lanes<DT>();
  __shared__ uint64_t sw[kLanes][kMaskThreads + 4];
  const int k = blockIdx.y, tid = threadIdx.x;
  const int x0 = blockIdx.x * kMaskThreads;
  const uint64_t* w = a.p.words + (size_t)k * kLanes * a.p.wstride;
  for (int i = tid; i < kLanes * (kMaskThreads + 2); i += kMaskThreads) {
    const int l = i / (kMaskThreads + 2), q = i % (kMaskThreads + 2);
    sw[l][q] = x0 + q < (int)a.L.n ? tw(w, a.p.wstride, x0 + q, l) : 0;
  }
  __syncthreads();
  const int x = x0 + tid;
  if (x >= a.M) return;
  const int ty0 = T0 >= 0 ? T0 : a.bk.c[0].type, ty1 = T1 >= 0 ? T1 : a.bk.c[1].type;
  const int nr = (ty0 >= 2) + (ty1 >= 2);
  int at = 0;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int ty = c == 0 ? ty0 : ty1;
    if (ty < 2) continue;
    const BetaComp& g = a.bk.c[c];
    // accepted lanes, and those the filters leave to the reference's expressions
    uint32_t m = 0, open = 0;
    if (ty == 2) {
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        const uint64_t w0 = sw[l][tid], w1 = sw[l][tid + 1], w2 = sw[l][tid + 2];
        if (DT == SD_F64) {
          const int f = gs_filter_f64(w0, w1, w2, g.f_px, g.f_inv, g.f_am1, g.f_band);
          m |= (f == 1 ? 1u : 0u) << l;
          open |= (f < 0 ? 1u : 0u) << l;
        } else {
          constexpr float e = 1.1920928955078125e-07f / 8;
          const int f0 = gs_filter(ur_f((uint32_t)w0), ur_f((uint32_t)w1) + e, ur_f((uint32_t)w2), g.f_px, g.f_inv,
                                   g.f_am1, g.f_band);
          const int f1 = gs_filter(ur_f((uint32_t)(w0 >> 32)), ur_f((uint32_t)(w1 >> 32)) + e,
                                   ur_f((uint32_t)(w2 >> 32)), g.f_px, g.f_inv, g.f_am1, g.f_band);
          m |= ((f0 == 1 ? 1u : 0u) | (f1 == 1 ? 2u : 0u)) << (2 * l);
          open |= ((f0 < 0 ? 1u : 0u) | (f1 < 0 ? 2u : 0u)) << (2 * l);
        }
      }
    } else {
#pragma unroll
      for (int l = 0; l < kLanes; ++l) {
        const uint64_t w0 = sw[l][tid], w1 = sw[l][tid + 1];
        if (DT == SD_F64) {
          const int f = tan_filter_f64(w0, w1, g.f_am1, g.f_sq);
          m |= (f == 1 ? 1u : 0u) << l;
          open |= (f < 0 ? 1u : 0u) << l;
        } else {
          const int f0 = tan_filter(ur_f((uint32_t)w0), ur_f((uint32_t)w1), g.f_am1, g.f_sq, kTanDeltaF);
          const int f1 = tan_filter(ur_f((uint32_t)(w0 >> 32)), ur_f((uint32_t)(w1 >> 32)), g.f_am1, g.f_sq, kTanDeltaF);
          m |= ((f0 == 1 ? 1u : 0u) | (f1 == 1 ? 2u : 0u)) << (2 * l);
          open |= ((f0 < 0 ? 1u : 0u) | (f1 < 0 ? 2u : 0u)) << (2 * l);
        }
      }
    }
    while (open) {
      const int j = __ffs(open) - 1;
      open &= open - 1;
      const int l = DT == SD_F64 ? j : (j >> 1);
      const uint64_t w0 = sw[l][tid], w1 = sw[l][tid + 1], w2 = sw[l][tid + 2];
      bool acc = false;
      auto uf = [&](int q) {
        const uint64_t v = q == 0 ? w0 : (q == 1 ? w1 : w2);
        return ur_f((j & 1) ? (uint32_t)(v >> 32) : (uint32_t)v);
      };
      auto ud = [&](int q) { return q == 0 ? w0 : (q == 1 ? w1 : w2); };
      if (c == 0) beta_comp_u<DT, true>(g, ty0, uf, ud, acc);
      else beta_comp_u<DT, true>(g, ty1, uf, ud, acc);
      m |= (acc ? 1u : 0u) << j;
    }
    a.mask[((size_t)k * nr + at) * a.L.mstride + x] = (uint8_t)m;
    ++at;
  }
}

// ---------------------------------------------------------------- visits
// One component's draw from position x with f lanes carried: trials until one
// is fully accepted or the carried lanes reach P.  One thread per position:
// the draws for all f read the same trials, and more carried lanes end no
// later, so the f's still open are [0, P - lanes so far).
constexpr int kVisThreads = 256;
template <int P, bool R0, bool R1>
__global__ void __launch_bounds__(kVisThreads) k_chain_visits(ChainArgs a) {
  constexpr int NR = (R0 ? 1 : 0) + (R1 ? 1 : 0);
  const int k = blockIdx.y / NR, r = blockIdx.y % NR;
  const int U = a.bk.c[(R0 && r == 0) ? 0 : 1].U;
  const int x = blockIdx.x * kVisThreads + threadIdx.x;
  if (x >= a.M) return;
  const uint8_t* mk = a.mask + ((size_t)k * NR + r) * a.L.mstride;
  uint64_t out = ~0ull;  // every f: no visit
  int cum = 0;
  for (int t = 0, y = x; t < kNoVisit<P> && y < a.M; ++t, y += U) {
    const int cn = __popc((uint32_t)__ldg(mk + y));
    const bool full = cn == P;
    const int top = P - cum;  // f below this are open
    if (!full) cum += cn;
    for (int f = full ? 0 : max(0, P - cum); f < top; ++f) {
      const uint64_t e = (uint64_t)((t << 3) | (full ? f + cum : f + cum - P));
      out = (out & ~(255ull << (8 * f))) | e << (8 * f);
    }
    if (full || cum >= P) break;
  }
  uint8_t* v = a.vis + (((size_t)k * NR + r) * a.L.mstride + x) * P;
  if (P == 8) *reinterpret_cast<uint64_t*>(v) = out;
  else *reinterpret_cast<uint32_t*>(v) = (uint32_t)out;
}

// ---------------------------------------------------------------- the chain
// One output packet from state (x, f0, f1); v0 / v1: the components' visit
// entries.  False: a draw the masks do not finish.
// adds0, adds1: whether the draws add to the carried lanes (one trial that leaves
// as many was fully accepted: entry == lanes carried).
template <int P, bool R0, bool R1, class V0, class V1>
__device__ __forceinline__ bool chain_step(int& x, int& f0, int& f1, int U0, int U1, V0&& v0, V1&& v1, bool& adds0,
                                           bool& adds1) {
  int y = x + U0, g0 = f0;
  if (R0) {
    const uint32_t e = v0(x, f0);
    const int t = visit_trials<P>(e);
    if (t == kNoVisit<P>) return false;
    y = x + (t + 1) * U0;
    g0 = P == 1 ? 0 : (int)(e & 7u);
    adds0 = e != (uint32_t)f0;
  }
  if (R1) {
    const uint32_t e = v1(y, f1);
    const int t = visit_trials<P>(e);
    if (t == kNoVisit<P>) return false;
    y += (t + 1) * U1;
    adds1 = e != (uint32_t)f1;
    f1 = (int)(e & 7u);
  } else {
    y += U1;
  }
  x = y;
  f0 = g0;
  return true;
}

template <int P, bool R0, bool R1>
__device__ __forceinline__ int state_code(int o, int f0, int f1) {
  constexpr int OM = entry_offsets<R0, R1>();
  if ((unsigned)o >= (unsigned)OM) return kEsc;
  return o + OM * ((R0 ? f0 : 0) + (R0 ? P : 1) * (R1 ? f1 : 0));
}
template <int P, bool R0, bool R1>
__device__ __forceinline__ void state_of(int code, int& o, int& f0, int& f1) {
  constexpr int OM = entry_offsets<R0, R1>();
  o = code % OM;
  const int f = code / OM;
  f0 = R0 ? f % P : 0;
  f1 = R1 ? f / (R0 ? P : 1) : 0;
}

// ---------------------------------------------------------------- tables
// One warp per segment.  Shared memory per warp: the visit entries of the
// segment's positions and a pad (draws past the end belong to outputs started
// before it), the chain each entry state is on, the chains' states, and per
// state the chain that claimed it.
constexpr int kPad = 192;
template <int P, bool R0, bool R1>
__host__ __device__ constexpr int table_warps() {
  return (R0 && R1) ? 1 : 4;
}
template <int P, bool R0, bool R1>
__host__ __device__ constexpr int table_vis_bytes(int J) {
  return (J + kPad) * P;
}
template <int P, bool R0, bool R1>
__host__ __device__ constexpr size_t table_smem(int J) {
  return (size_t)table_warps<P, R0, R1>() * ((size_t)table_vis_bytes<P, R0, R1>(J) * ((R0 ? 1 : 0) + (R1 ? 1 : 0)) +
                                             entry_states<P, R0, R1>() * (2 + 2 + 2 + 4));
}

// 16-byte copies of one warp: count bytes (a multiple of 16) of the visit
// array from position p0 on; what lies past the array's end is not read.
template <int P>
__device__ __forceinline__ const uint4* vis_at(const ChainArgs& a, int k, int NR, int r, int64_t p0) {
  return reinterpret_cast<const uint4*>(a.vis + (((size_t)k * NR + r) * a.L.mstride + p0) * P);
}

template <int P, bool R0, bool R1>
__global__ void __launch_bounds__(32 * table_warps<P, R0, R1>()) k_chain_table(ChainArgs a) {
  constexpr int NS = entry_states<P, R0, R1>();
  constexpr int W = table_warps<P, R0, R1>();
  constexpr int NR = (R0 ? 1 : 0) + (R1 ? 1 : 0);
  extern __shared__ __align__(16) uint8_t tb_dyn[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int J = a.L.J, vb = table_vis_bytes<P, R0, R1>(J);
  uint8_t* vs = tb_dyn + (size_t)warp * (NR * vb + NS * 10);  // [NR][J + kPad][P]
  uint32_t* st = reinterpret_cast<uint32_t*>(vs + NR * vb);   // chain -> x (relative) | f0 << 16 | f1 << 24
  uint16_t* on = reinterpret_cast<uint16_t*>(st + NS);        // entry state -> chain (kEsc: none)
  uint16_t* claim = on + NS;                                  // state -> a chain in it
  uint16_t* id = claim + NS;                                  // chain -> its number after merging
  const int64_t sg = (int64_t)blockIdx.x * W + warp;
  const int64_t total = (int64_t)a.p.K * a.L.Sg;
  if (sg >= total) return;
  const int k = (int)(sg / a.L.Sg), s = (int)(sg % a.L.Sg);
  const int lo = s * J;
  const int U0 = a.bk.c[0].U, U1 = a.bk.c[1].U;
  for (int r = 0; r < NR; ++r) {
    const uint4* src = vis_at<P>(a, k, NR, r, lo);
    const int64_t have = (int64_t)(a.M - lo) * P;  // entries that were written
    for (int i = lane; i < vb / 16; i += 32)
      reinterpret_cast<uint4*>(vs + r * vb)[i] = 16 * (int64_t)i < have ? __ldg(src + i) : make_uint4(~0u, ~0u, ~0u, ~0u);
  }
  // entry states: outputs start at multiples of the components' packets' gcd
  int g = U0, h = U1;
  while (h) {
    const int t = g % h;
    g = h;
    h = t;
  }
  int na = 0;
  for (int b = 0; b < NS; b += 32) {
    const int e = b + lane;
    int o, f0, f1;
    state_of<P, R0, R1>(e, o, f0, f1);
    const bool can = (lo + o) % g == 0;
    const uint32_t bal = __ballot_sync(0xffffffffu, can);
    const int i = na + __popc(bal & ((1u << lane) - 1u));
    on[e] = can ? (uint16_t)i : (uint16_t)kEsc;
    if (can) st[i] = (uint32_t)o | (uint32_t)f0 << 16 | (uint32_t)f1 << 24;
    na += __popc(bal);
  }
  __syncwarp();
  const int lim = min(J + kPad - 1, a.M - 1 - lo);  // last position with an entry here
  auto v0 = [&](int x, int f) -> uint32_t { return x <= lim ? vs[x * P + f] : 255u; };
  auto v1 = [&](int x, int f) -> uint32_t { return x <= lim ? vs[(R0 ? vb : 0) + x * P + f] : 255u; };
  for (int be = min(32, J);; be = min(2 * be, J)) {
    for (int e = lane; e < NS; e += 32) claim[e] = (uint16_t)kEsc;
    __syncwarp();
    for (int i = lane; i < na; i += 32) {
      const uint32_t v = st[i];
      int sx = (int)(v & 0xffffu), c0 = (int)((v >> 16) & 255), c1 = (int)(v >> 24);
      bool ok = v != 0xffffffffu, adds0, adds1;
      while (ok && sx < be) ok = chain_step<P, R0, R1>(sx, c0, c1, U0, U1, v0, v1, adds0, adds1);
      const int code = ok ? state_code<P, R0, R1>(sx - be, c0, c1) : kEsc;
      st[i] = code == kEsc ? 0xffffffffu : ((uint32_t)sx | (uint32_t)c0 << 16 | (uint32_t)c1 << 24);
      if (code != kEsc) claim[code] = (uint16_t)i;
    }
    __syncwarp();
    if (be == J) break;
    // number the chains that own their state, then move the others to them
    int nn = 0;
    for (int b = 0; b < na; b += 32) {
      const int i = b + lane;
      int code = kEsc;
      if (i < na && st[i] != 0xffffffffu) {
        const uint32_t v = st[i];
        code = state_code<P, R0, R1>((int)(v & 0xffffu) - be, (int)((v >> 16) & 255), (int)(v >> 24));
      }
      const bool win = code != kEsc && claim[code] == i;
      const uint32_t bal = __ballot_sync(0xffffffffu, win);
      if (win) id[i] = (uint16_t)(nn + __popc(bal & ((1u << lane) - 1u)));
      nn += __popc(bal);
    }
    __syncwarp();
    for (int e = lane; e < NS; e += 32) {
      const int i = on[e];
      if (i == kEsc) continue;
      const uint32_t v = st[i];
      on[e] = v == 0xffffffffu
                  ? (uint16_t)kEsc
                  : id[claim[state_code<P, R0, R1>((int)(v & 0xffffu) - be, (int)((v >> 16) & 255), (int)(v >> 24))]];
    }
    __syncwarp();
    // owners' numbers only go down, so they move in place, 32 at a time
    for (int b = 0; b < na; b += 32) {
      const int i = b + lane;
      bool win = false;
      uint32_t v = 0;
      if (i < na) {
        v = st[i];
        if (v != 0xffffffffu)
          win = claim[state_code<P, R0, R1>((int)(v & 0xffffu) - be, (int)((v >> 16) & 255), (int)(v >> 24))] == i;
      }
      __syncwarp();
      if (win) st[id[i]] = v;
      __syncwarp();
    }
    na = nn;
  }
  uint16_t* out = a.tab + (size_t)sg * NS;
  for (int e = lane; e < NS; e += 32) {
    int code = kEsc;
    if (on[e] != kEsc) {
      const uint32_t v = st[on[e]];
      if (v != 0xffffffffu)
        code = state_code<P, R0, R1>((int)(v & 0xffffu) - J, (int)((v >> 16) & 255), (int)(v >> 24));
    }
    out[e] = (uint16_t)code;
  }
}

// ---------------------------------------------------------------- composition
// Groups of gsz segments: up = 1 makes each group's table (grid groups, K)
// from its segments' in shared memory; up = 0 follows a group's true entry
// (from the groups' tables and the call's first state) through its segments.
template <int P, bool R0, bool R1>
__global__ void __launch_bounds__(512) k_chain_compose(ChainArgs a, int up) {
  constexpr int NS = entry_states<P, R0, R1>();
  extern __shared__ __align__(16) uint8_t cp_dyn[];
  uint16_t* t = reinterpret_cast<uint16_t*>(cp_dyn);  // [gsz][NS]
  __shared__ int s_entry;
  const int k = blockIdx.y, g = blockIdx.x, tid = threadIdx.x;
  const int Sg = a.L.Sg, gsz = a.L.gsz, ng = a.L.groups;
  const int s0 = g * gsz, cnt = min(gsz, Sg - s0);
  const uint16_t* src = a.tab + ((size_t)k * Sg + s0) * NS;
  for (int i = tid; i < cnt * NS / 8; i += blockDim.x)
    reinterpret_cast<uint4*>(t)[i] = reinterpret_cast<const uint4*>(src)[i];
  if (up) {
    __syncthreads();
    for (int e = tid; e < NS; e += blockDim.x) {
      int c = e;
      for (int s = 0; s < cnt && c != kEsc; ++s) c = t[s * NS + c];
      a.gtab[((size_t)k * ng + g) * NS + e] = (uint16_t)c;
    }
    return;
  }
  if (tid == 0) {
    const GenState& gs = a.p.gen[k];
    int c = state_code<P, R0, R1>(0, R0 && P > 1 ? gs.s[1].rest_cnt : 0, R1 ? gs.s[2].rest_cnt : 0);
    for (int q = 0; q < g && c != kEsc; ++q) c = a.gtab[((size_t)k * ng + q) * NS + c];
    s_entry = c;
  }
  __syncthreads();
  if (tid == 0) {
    int c = s_entry;
    for (int s = 0; s < cnt; ++s) {
      a.entry[(size_t)k * Sg + s0 + s] = c;
      if (c != kEsc) c = t[s * NS + c];
    }
  }
}

// ---------------------------------------------------------------- walk
// One warp per segment: lane 0 follows the true chain from the segment's entry
// state while the warp's copies of the next tile of visit entries are in
// flight.  Bound by the latency of the chain: one shared-memory read and a few
// dependent operations per component and output packet.
constexpr int kTile = 1024;
template <int P, bool R0, bool R1>
__global__ void __launch_bounds__(32) k_chain_walk(ChainArgs a) {
  constexpr int NR = (R0 ? 1 : 0) + (R1 ? 1 : 0);
  constexpr int VB = (kTile + kPad) * P;
  extern __shared__ __align__(16) uint8_t wk_dyn[];  // [2][NR][VB]
  __shared__ int s_x;
  const int Sg = a.L.Sg, lane = threadIdx.x;
  const int64_t sg = blockIdx.x;
  const int k = (int)(sg / Sg), s = (int)(sg % Sg);
  const int U0 = a.bk.c[0].U, U1 = a.bk.c[1].U;
  const int lo = s * a.L.J;
  const int hi = s == Sg - 1 ? INT32_MAX : lo + a.L.J;
  int o = 0, f0 = 0, f1 = 0;
  if (s == 0) {
    f0 = R0 && P > 1 ? a.p.gen[k].s[1].rest_cnt : 0;
    f1 = R1 ? a.p.gen[k].s[2].rest_cnt : 0;
  } else {
    const int code = a.entry[sg];
    if (code == kEsc) {
      if (lane == 0) a.seg[sg] = ChainSeg{0, 1, {0, 0}, {0, 0}};
      return;
    }
    state_of<P, R0, R1>(code, o, f0, f1);
  }
  auto fetch = [&](int tile, int buf) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const uint4* src = vis_at<P>(a, k, NR, r, (int64_t)tile * kTile);
      const int64_t have = ((int64_t)a.M - (int64_t)tile * kTile) * P;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(wk_dyn + (size_t)(buf * NR + r) * VB);
      for (int i = lane; i < VB / 16; i += 32)
        if (16 * (int64_t)i < have)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint32_t* rec = a.rec + (size_t)sg * a.L.rcap;
  const int want = (int)min(limit_of(a, k), (int64_t)a.L.rcap);
  // [0]: the first rejection component's, [1]: the second's
  uint16_t* prev0 = a.prev + (size_t)sg * a.L.rcap;
  uint16_t* prev1 = prev0 + (NR == 2 ? (size_t)a.p.K * Sg * a.L.rcap : 0);
  int x = lo + o, nrec = 0, bad = 0, last0 = 0, last1 = 0;
  int tile = x / kTile;
  fetch(tile, 0);
  for (int b = 0;; b ^= 1) {
    fetch(tile + 1, b ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      const int base = tile * kTile, stop = min(hi, base + kTile);
      const int lim = min(a.M - 1, base + kTile + kPad - 1);
      const uint8_t* vs = wk_dyn + (size_t)b * NR * VB;
      auto v0 = [&](int y, int f) -> uint32_t { return y <= lim ? vs[(y - base) * P + f] : 255u; };
      auto v1 = [&](int y, int f) -> uint32_t { return y <= lim ? vs[(R0 ? VB : 0) + (y - base) * P + f] : 255u; };
      while (x < stop && nrec < want) {
        const uint32_t r = (uint32_t)x | (uint32_t)f0 << 24 | (uint32_t)f1 << 27;
        int y = x;
        bool adds0 = false, adds1 = false;
        if (!chain_step<P, R0, R1>(y, f0, f1, U0, U1, v0, v1, adds0, adds1) || (R0 && !R1 && P > 1 && y > (int)a.L.n)) {
          bad = 1;
          break;
        }
        x = y;
        rec[nrec] = r;
        if (P > 1) {
          if (R0) prev0[nrec] = (uint16_t)last0;
          if (R1) prev1[nrec] = (uint16_t)last1;
        }
        ++nrec;
        if (adds0) last0 = nrec;
        if (adds1) last1 = nrec;
      }
      s_x = (bad || nrec >= want || x >= hi) ? -1 : x;
    }
    __syncwarp();
    const int nx = s_x;
    __syncwarp();
    if (nx < 0) break;
    ++tile;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (lane == 0) a.seg[sg] = ChainSeg{nrec, bad, {last0, last1}, {0, 0}};
}

// ---------------------------------------------------------------- scan
// A0, A1: the components whose outputs add to carried lanes.
template <bool A0, bool A1>
__global__ void __launch_bounds__(1024) k_chain_scan(ChainArgs a) {
  __shared__ int64_t s_tot[32];
  __shared__ int s_top[2][32];
  __shared__ int64_t s_carry;
  __shared__ int s_bad, s_last[2];
  const int k = blockIdx.x, tid = threadIdx.x, Sg = a.L.Sg;
  ChainSeg* seg = a.seg + (size_t)k * Sg;
  int64_t* eb = a.ebase + (size_t)k * (Sg + 1);
  if (tid == 0) {
    s_carry = 0;
    s_bad = INT32_MAX;
    s_last[0] = s_last[1] = 0;
  }
  __syncthreads();
  for (int s = tid; s < Sg; s += blockDim.x)
    if (seg[s].bad) atomicMin(&s_bad, s);
  __syncthreads();
  const int lastgood = s_bad;  // a chain that stopped in segment s says nothing about the later ones
  for (int b = 0; b < Sg; b += blockDim.x) {
    const int s = b + tid;
    const int64_t v = (s < Sg && s <= lastgood) ? seg[s].nrec : 0;
    int64_t x = v;
    int top[2];  // the last segment up to this one with an output that adds, plus 1
#pragma unroll
    for (int c = 0; c < 2; ++c) top[c] = ((c ? A1 : A0) && s < Sg && seg[s].adds[c]) ? s + 1 : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
      const int t0 = A0 ? __shfl_up_sync(0xffffffffu, top[0], o) : 0, t1 = A1 ? __shfl_up_sync(0xffffffffu, top[1], o) : 0;
      if ((tid & 31) >= o) {
        x += y;
        top[0] = max(top[0], t0);
        top[1] = max(top[1], t1);
      }
    }
    if ((tid & 31) == 31) {
      s_tot[tid >> 5] = x;
      s_top[0][tid >> 5] = top[0];
      s_top[1][tid >> 5] = top[1];
    }
    __syncthreads();
    if (tid < 32) {
      const bool have = tid < (int)(blockDim.x >> 5);
      int64_t t = have ? s_tot[tid] : 0;
      int p0 = have ? s_top[0][tid] : 0, p1 = have ? s_top[1][tid] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, t, o);
        const int t0 = A0 ? __shfl_up_sync(0xffffffffu, p0, o) : 0, t1 = A1 ? __shfl_up_sync(0xffffffffu, p1, o) : 0;
        if (tid >= o) {
          t += y;
          p0 = max(p0, t0);
          p1 = max(p1, t1);
        }
      }
      s_tot[tid] = t;
      s_top[0][tid] = p0;
      s_top[1][tid] = p1;
    }
    __syncthreads();
    const int64_t incl = s_carry + x + ((tid >> 5) ? s_tot[(tid >> 5) - 1] : 0);
    int before[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!(c ? A1 : A0)) {
        before[c] = 0;
        continue;
      }
      const int up = __shfl_up_sync(0xffffffffu, top[c], 1);
      before[c] = max(max(s_last[c], (tid >> 5) ? s_top[c][(tid >> 5) - 1] : 0), (tid & 31) ? up : 0);
    }
    if (s < Sg) {
      eb[s] = incl - v;
      if (A0) seg[s].prev[0] = before[0];
      if (A1) seg[s].prev[1] = before[1];
    }
    __syncthreads();
    if (tid == (int)blockDim.x - 1) {
      s_carry = incl;
      s_last[0] = max(before[0], top[0]);
      s_last[1] = max(before[1], top[1]);
    }
    __syncthreads();
  }
  if (tid == 0) eb[Sg] = s_carry;
}

// ---------------------------------------------------------------- emission
// A component's draw from position x with f lanes carried (a visit).
struct Visits {
  const uint8_t* mk;
  int U, P;
  // the trials of the visit: full: its last trial is fully accepted and *last
  // its position; pushed: accepted lanes its partial trials left in the FIFO;
  // where: position and lane of pushed lane `idx` (idx < 0: none)
  __device__ __forceinline__ bool scan(int x, int f, int idx, int& last, int& pushed, uint32_t& pos, int& lane) const {
    int acc = 0;
    for (int y = x;; y += U) {
      const uint32_t m = __ldg(mk + y);
      const int cn = __popc(m);
      last = y;
      if (cn == P) {
        pushed = acc;
        return true;
      }
      if ((unsigned)(idx - acc) < (unsigned)cn) {
        uint32_t mm = m;
        for (int r = idx - acc; r > 0; --r) mm &= mm - 1;
        pos = (uint32_t)y;
        lane = __ffs(mm) - 1;
      }
      acc += cn;
      if (f + acc >= P) {
        pushed = acc;
        return false;
      }
    }
  }
};

template <int DT>
__device__ __forceinline__ Visits visits_of(const ChainArgs& a, int k, int c, bool R0, bool R1) {
  const int NR = (R0 ? 1 : 0) + (R1 ? 1 : 0), r = (c == 1 && R0) ? 1 : 0;
  return Visits{a.mask + ((size_t)k * NR + r) * a.L.mstride, a.bk.c[c].U, beta_lanes<DT>()};
}

// Where the draw of component c of the output recorded as r starts.
template <int DT>
__device__ __forceinline__ int draw_start(const ChainArgs& a, int k, int c, bool R0, bool R1, uint32_t r) {
  const int x = (int)(r & 0xffffffu);
  if (c == 0) return x;
  if (!R0) return x + a.bk.c[0].U;
  constexpr int P = beta_lanes<DT>();
  const uint8_t e = __ldg(a.vis + ((size_t)k * (R1 ? 2 : 1) * a.L.mstride + x) * P + ((r >> 24) & 7u));
  return x + ((e >> 3) + 1) * a.bk.c[0].U;
}

// The lane `dist` places before the end of component c's FIFO as it is before
// output i of segment s: position and lane of its trial (kEntInit: a lane
// carried into the call).  A few outputs back one by one, where ordinary shapes find
// it, then from one output that adds lanes to the one before it: output by output all
// the way, the last lanes of a shape whose trials nearly all are fully accepted took
// milliseconds.
template <int DT>
__device__ __forceinline__ void carried_lane(const ChainArgs& a, int k, int c, bool R0, bool R1, int s, int64_t i, int dist,
                                             uint32_t& pos, int& lane) {
  const Visits v = visits_of<DT>(a, k, c, R0, R1);
  const ChainSeg* seg = a.seg + (size_t)k * a.L.Sg;
  const uint16_t* prev = a.prev + (c == 1 && R0 ? (size_t)a.p.K * a.L.Sg * a.L.rcap : 0) + (size_t)k * a.L.Sg * a.L.rcap;
  int q = (int)i;  // the output looked at next, plus 1
  for (int back = 0;; ++back) {
    if (q == 0) {
      s = seg[s].prev[c] - 1;
      if (s < 0) {
        pos = kEntInit;
        lane = max(a.p.gen[k].s[1 + c].rest_cnt - dist, 0);
        return;
      }
      q = seg[s].adds[c];
    }
    const size_t at = (size_t)s * a.L.rcap + q - 1;
    const uint32_t r = __ldg(a.rec + (size_t)k * a.L.Sg * a.L.rcap + at);
    const int x = draw_start<DT>(a, k, c, R0, R1, r), f = (int)((r >> (c ? 27 : 24)) & 7u);
    int last, pushed;
    v.scan(x, f, -1, last, pushed, pos, lane);
    if (dist <= pushed) {
      v.scan(x, f, pushed - dist, last, pushed, pos, lane);
      return;
    }
    dist -= pushed;
    q = back < 4 ? q - 1 : prev[at];
  }
}

template <int DT, int T0, int T1>
__device__ __forceinline__ uint64_t chain_value(const ChainArgs& a, const uint64_t* w, int k, int c, uint32_t pos,
                                                int j) {
  const int ty = c == 0 ? (T0 >= 0 ? T0 : a.bk.c[0].type) : (T1 >= 0 ? T1 : a.bk.c[1].type);
  const BetaComp& g = a.bk.c[c];
  if (pos == kEntInit) {
    const uint32_t* r = a.p.gen[k].s[1 + c].rest;
    return DT == SD_F64 ? ((uint64_t)r[2 * j] | ((uint64_t)r[2 * j + 1] << 32)) : (uint64_t)r[j];
  }
  const int x = (int)pos;
  auto word = [&](int q) {
    const uint64_t v = tw(w, a.p.wstride, x + q, j >> 1);
    return (j & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
  };
  auto uf = [&](int q) { return ur_f(word(q)); };
  auto ud = [&](int q) { return tw(w, a.p.wstride, x + q, j); };
  if (DT == SD_F64 && ty == 2)
    return d2u(1.0 * gs_value_f64(tw(w, a.p.wstride, x, j), tw(w, a.p.wstride, x + 1, j), g.tpx, g.d_inv));
  bool acc;
  return beta_comp_u<DT, false>(g, ty, uf, ud, acc);
}

// grid (parts of segments, engines); CLOSED: neither component rejects, output
// i draws at i (U0 + U1)
constexpr int kEmitThreads = 128;
template <int DT, int T0, int T1, bool R0, bool R1>
__global__ void __launch_bounds__(kEmitThreads) k_chain_emit(ChainArgs a, int parts) {
  constexpr int P = beta_lanes<DT>();
  constexpr bool CLOSED = !R0 && !R1;
  const int k = blockIdx.y, s = blockIdx.x / parts, part = blockIdx.x % parts;
  const int Sg = a.L.Sg;
  const int U0 = a.bk.c[0].U, U1 = a.bk.c[1].U;
  const int64_t limit = limit_of(a, k);
  const int64_t eb = CLOSED ? 0 : a.ebase[(size_t)k * (Sg + 1) + s];
  const int64_t all = CLOSED ? min(limit, a.L.n / (U0 + U1)) : min(limit, a.ebase[(size_t)k * (Sg + 1) + s + 1]) - eb;
  const int64_t per = (all + parts - 1) / parts;
  const int64_t i0 = per * part, i1 = min(all, i0 + per);
  const uint64_t* w = a.p.words + (size_t)k * kLanes * a.p.wstride;
  const int64_t g0 = (int64_t)k * a.p.gran_per_k + min((int64_t)k, a.p.gran_rem) + a.done[k];
  const uint32_t* rec = a.rec + ((size_t)k * Sg + s) * a.L.rcap;
  for (int64_t u0 = i0 * P; u0 < i1 * P; u0 += kEmitThreads) {
    const int64_t u = u0 + threadIdx.x, i = u / P;
    const bool valid = u < i1 * P;
    const int j = (int)(u % P);
    const uint32_t r = (CLOSED || !valid) ? 0 : __ldg(rec + i);
    int x = CLOSED ? (int)(i * (U0 + U1)) : (int)(r & 0xffffffu);
    uint32_t pos[2];
    int lane[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      pos[c] = (uint32_t)x;
      lane[c] = j;
      if (c ? R1 : R0) {
        if (valid) {
          const int f = (int)((r >> (c ? 27 : 24)) & 7u);
          const Visits vis = visits_of<DT>(a, k, c, R0, R1);
          int last, pushed;
          if (vis.scan(x, f, j - f, last, pushed, pos[c], lane[c])) {
            pos[c] = (uint32_t)last;
            lane[c] = j;
          } else if (j < f) {
            carried_lane<DT>(a, k, c, R0, R1, s, i, f - j, pos[c], lane[c]);
          }
          x = last + vis.U;
        }
      } else {
        x += c ? U1 : U0;
      }
    }
    // the searches take different times: the warp meets again before the
    // values, which are most of the work
    __syncwarp();
    if (!valid) continue;
    uint64_t v[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) v[c] = chain_value<DT, T0, T1>(a, w, k, c, pos[c], lane[c]);
    const int64_t at = (g0 + eb + i) * P + j;
    if (DT == SD_F32) {
      const float p1 = u2f((uint32_t)v[0]), p2 = u2f((uint32_t)v[1]);
      const float q = p1 / (p1 + p2);
      reinterpret_cast<float*>(a.p.out)[at] = a.bk.post == 1 ? (a.bk.fpost * q) / (1.0f - q) : q;
    } else {
      const double p1 = u2d(v[0]), p2 = u2d(v[1]);
      const double q = div_d(p1, p1 + p2);
      reinterpret_cast<double*>(a.p.out)[at] = a.bk.post == 1 ? (a.bk.dpost * q) / (1.0 - q) : q;
    }
  }
}

// ---------------------------------------------------------------- state
template <int DT, bool R0, bool R1>
__global__ void __launch_bounds__(256) k_chain_finish(ChainArgs a) {
  const int k = blockIdx.x, tid = threadIdx.x, Sg = a.L.Sg;
  EngState* st = a.p.eng + k;
  GenState* gs = a.p.gen + k;
  const int U0 = a.bk.c[0].U, U1 = a.bk.c[1].U;
  const int64_t limit = limit_of(a, k);
  const uint64_t* w = a.p.words + (size_t)k * kLanes * a.p.wstride;
  int64_t tot, np, i = 0;
  int f[2] = {0, 0};
  int s = 0;
  if (!R0 && !R1) {
    tot = min(limit, a.L.n / (U0 + U1));
    np = tot * (U0 + U1);
  } else {
    const int64_t* eb = a.ebase + (size_t)k * (Sg + 1);
    tot = min(limit, eb[Sg]);
    if (tot <= 0) return;
    int lo = 0, hi = Sg;  // the segment of output tot - 1: eb[lo] <= tot - 1 < eb[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (eb[mid] <= tot - 1) lo = mid;
      else hi = mid;
    }
    s = lo;
    i = tot - eb[s];  // outputs of the segment up to and with the last
    const uint32_t r = a.rec[((size_t)k * Sg + s) * a.L.rcap + i - 1];
    int x = (int)(r & 0xffffffu);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (c ? R1 : R0) {
        const int fc = (int)((r >> (c ? 27 : 24)) & 7u);
        const Visits vis = visits_of<DT>(a, k, c, R0, R1);
        int last, pushed, lane;
        uint32_t pos;
        const bool full = vis.scan(x, fc, -1, last, pushed, pos, lane);
        f[c] = fc + pushed - (full ? 0 : beta_lanes<DT>());
        x = last + vis.U;
      } else {
        x += c ? U1 : U0;
      }
    }
    np = x;
  }
  if (tot <= 0) return;
  uint64_t v = 0;
  const int c = tid / 8, j = tid % 8;
  const bool mine = tid < 16 && (c ? R1 : R0);
  if (mine && j < f[c]) {
    uint32_t pos = 0;
    int lane = 0;
    carried_lane<DT>(a, k, c, R0, R1, s, i, f[c] - j, pos, lane);
    v = chain_value<DT, -1, -1>(a, w, k, c, pos, lane);
  }
  __syncthreads();  // the lanes carried into the call are read before they are replaced
  if (mine) {
    GenSlot& g = gs->s[1 + c];
    if (DT == SD_F64) {
      g.rest[2 * j] = (uint32_t)v;
      g.rest[2 * j + 1] = (uint32_t)(v >> 32);
    } else {
      g.rest[j] = (uint32_t)v;
    }
    if (j == 0) g.rest_cnt = f[c];
  }
  for (int t = tid; t < kLanes * kN; t += blockDim.x)
    st->win[t / kN][t % kN] = w[(size_t)(t / kN) * a.p.wstride + np + t % kN];
  if (tid == 0) {
    st->consumed += (uint64_t)np;
    a.done[k] += tot;
  }
}

// ---------------------------------------------------------------- Poisson
// PoissonGen with mean < 12 (Discrete.h:870-882), also BinomialGen with trials
// min(p, 1 - p) < 1: one packetOp multiplies half packets of uniforms until
// every lane's product is <= exp(-mean) and returns, per lane, how many
// products stayed above it.  A step from half packet x takes L(x) half
// packets and the next output starts at x + L(x): a chain with nothing
// carried.  Position 0 is the engine's cached half packet when there is one.
struct PoisArgs {
  ChainArgs c;
  const CallSnap* snap;
  uint32_t* pos;  // [K][c.L.mstride] the four counts, 6 bits each
  float thr;      // exp(-mean)
  int trials, flip;
};
constexpr int kPoisLook = 64;  // half packets one step may read (so 6 bits hold a count)

constexpr int kStepThreads = 256;
__global__ void __launch_bounds__(kStepThreads) k_pois_steps(PoisArgs a) {
  __shared__ float4 su[kStepThreads + kPoisLook];
  const int k = blockIdx.y, tid = threadIdx.x;
  const int x0 = blockIdx.x * kStepThreads;
  const int cached = a.snap[k].half_valid ? 1 : 0;
  const uint64_t* w = a.c.p.words + (size_t)k * kLanes * a.c.p.wstride;
  const int nh = 2 * (int)a.c.p.wcount + cached;  // half packets that exist
  for (int i = tid; i < kStepThreads + kPoisLook; i += kStepThreads) {
    const int x = x0 + i;
    float4 u = make_float4(0, 0, 0, 0);
    if (x < cached) {
      const uint32_t* h = a.snap[k].half_cache;
      u = make_float4(ur_f(h[0]), ur_f(h[1]), ur_f(h[2]), ur_f(h[3]));
    } else if (x < nh) {
      const int h = x - cached, l = 2 * (h & 1);
      const uint64_t p = tw(w, a.c.p.wstride, h >> 1, l), q = tw(w, a.c.p.wstride, h >> 1, l + 1);
      u = make_float4(ur_f((uint32_t)p), ur_f((uint32_t)(p >> 32)), ur_f((uint32_t)q), ur_f((uint32_t)(q >> 32)));
    }
    su[i] = u;
  }
  __syncthreads();
  const int x = x0 + tid;
  if (x >= a.c.M) return;
  float v[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  uint32_t n[4] = {0, 0, 0, 0};
  bool any = true;
  int L = 0;
  while (any && L < kPoisLook) {
    const float4 u = su[tid + L];
    v[0] *= u.x;
    v[1] *= u.y;
    v[2] *= u.z;
    v[3] *= u.w;
    any = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool c = a.thr < v[j];
      n[j] += c ? 1u : 0u;
      any |= c;
    }
    ++L;
  }
  const size_t at = (size_t)k * a.c.L.mstride + x;
  // a step longer than the look-ahead, or past what exists, ends the chain
  a.c.vis[at] = (any || x + L > nh) ? (uint8_t)255 : (uint8_t)(L - 1);
  a.pos[at] = n[0] | n[1] << 6 | n[2] << 12 | n[3] << 18;
}

__global__ void __launch_bounds__(256) k_pois_emit(PoisArgs a) {
  const ChainArgs& c = a.c;
  const int k = blockIdx.y, s = blockIdx.x, Sg = c.L.Sg;
  const int64_t limit = limit_of(c, k);
  const int64_t eb = c.ebase[(size_t)k * (Sg + 1) + s];
  const int64_t all = min(limit, c.ebase[(size_t)k * (Sg + 1) + s + 1]) - eb;
  const int64_t g0 = (int64_t)k * c.p.gran_per_k + min((int64_t)k, c.p.gran_rem) + c.done[k] + eb;
  const uint32_t* rec = c.rec + ((size_t)k * Sg + s) * c.L.rcap;
  const uint32_t* pos = a.pos + (size_t)k * c.L.mstride;
  for (int64_t i = threadIdx.x; i < all; i += blockDim.x) {
    const uint32_t q = __ldg(pos + (rec[i] & 0xffffffu));
    int v[4] = {(int)(q & 63), (int)((q >> 6) & 63), (int)((q >> 12) & 63), (int)((q >> 18) & 63)};
    if (a.flip) {  // BinomialGen: trials - res when p > 1/2
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = a.trials - v[j];
    }
    reinterpret_cast<int4*>(c.p.out)[g0 + i] = make_int4(v[0], v[1], v[2], v[3]);
  }
}

__global__ void __launch_bounds__(256) k_pois_finish(PoisArgs a) {
  const ChainArgs& c = a.c;
  const int k = blockIdx.x, tid = threadIdx.x, Sg = c.L.Sg;
  const int64_t* eb = c.ebase + (size_t)k * (Sg + 1);
  const int64_t tot = min(limit_of(c, k), eb[Sg]);
  if (tot <= 0) return;
  int lo = 0, hi = Sg;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (eb[mid] <= tot - 1) lo = mid;
    else hi = mid;
  }
  const int x = (int)(c.rec[((size_t)k * Sg + lo) * c.L.rcap + (tot - 1 - eb[lo])] & 0xffffffu);
  const int cached = a.snap[k].half_valid ? 1 : 0;
  const int fresh = x + c.vis[(size_t)k * c.L.mstride + x] + 1 - cached;  // half packets drawn
  const int np = (fresh + 1) / 2;
  EngState* st = c.p.eng + k;
  const uint64_t* w = c.p.words + (size_t)k * kLanes * c.p.wstride;
  for (int t = tid; t < kLanes * kN; t += blockDim.x)
    st->win[t / kN][t % kN] = w[(size_t)(t / kN) * c.p.wstride + np + t % kN];
  if (tid == 0) {
    if (fresh & 1) {  // the last packet's upper half stays cached
      const uint64_t p = tw(w, c.p.wstride, np - 1, 2), q = tw(w, c.p.wstride, np - 1, 3);
      st->half_cache[0] = (uint32_t)p;
      st->half_cache[1] = (uint32_t)(p >> 32);
      st->half_cache[2] = (uint32_t)q;
      st->half_cache[3] = (uint32_t)(q >> 32);
    }
    st->half_valid = fresh & 1;
    st->consumed += (uint64_t)np;
    c.done[k] += tot;
  }
}

constexpr size_t al(size_t x) { return (x + 255) / 256 * 256; }

// From the visit entries to the recorded chain and the outputs before each
// segment.
template <int P, bool R0, bool R1>
cudaError_t run_core(const ChainArgs& a, cudaStream_t s) {
  constexpr int NR = (R0 ? 1 : 0) + (R1 ? 1 : 0);
  const int K = a.p.K, Sg = a.L.Sg;
  if (Sg > 1) {
    const size_t tsm = table_smem<P, R0, R1>(a.L.J);
    const size_t csm = (size_t)a.L.gsz * entry_states<P, R0, R1>() * 2;
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr[dev]) {
      cudaError_t e = cudaFuncSetAttribute(k_chain_table<P, R0, R1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 98304);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_chain_compose<P, R0, R1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 98304);
      if (e != cudaSuccess) return e;
      attr[dev] = true;
    }
    constexpr int W = table_warps<P, R0, R1>();
    const int64_t segs = (int64_t)K * Sg;
    k_chain_table<P, R0, R1><<<(unsigned)((segs + W - 1) / W), 32 * W, tsm, s>>>(a);
    if (a.L.groups > 1) k_chain_compose<P, R0, R1><<<dim3(a.L.groups, K), 512, csm, s>>>(a, 1);
    k_chain_compose<P, R0, R1><<<dim3(a.L.groups, K), 512, csm, s>>>(a, 0);
  }
  k_chain_walk<P, R0, R1><<<(unsigned)(K * Sg), 32, (size_t)2 * NR * (kTile + kPad) * P, s>>>(a);
  k_chain_scan<R0 && (P > 1), R1><<<K, Sg > 256 ? 1024 : 256, 0, s>>>(a);
  return cudaGetLastError();
}

template <int DT, bool R0, bool R1, int T0, int T1>
cudaError_t run_chain(const ChainArgs& a0, cudaStream_t s) {
  constexpr int P = beta_lanes<DT>();
  ChainArgs a = a0;
  const int K = a.p.K, Sg = a.L.Sg;
  constexpr bool CLOSED = !R0 && !R1;
  if constexpr (!CLOSED) {
    constexpr int NR = (R0 ? 1 : 0) + (R1 ? 1 : 0);
    k_chain_masks<DT, T0, T1><<<dim3((unsigned)((a.M + kMaskThreads - 1) / kMaskThreads), K), kMaskThreads, 0, s>>>(a);
    k_chain_visits<P, R0, R1><<<dim3((unsigned)((a.M + kVisThreads - 1) / kVisThreads), K * NR), kVisThreads, 0, s>>>(a);
    const cudaError_t e = run_core<P, R0, R1>(a, s);
    if (e != cudaSuccess) return e;
  }
  // about 400 output lanes per CTA
  const int64_t lanes = a.L.rcap * (int64_t)P;
  const int parts = (int)std::max<int64_t>(1, std::min<int64_t>(lanes / 512, 60000 / Sg));
  k_chain_emit<DT, T0, T1, R0, R1><<<dim3((unsigned)Sg * parts, K), kEmitThreads, 0, s>>>(a, parts);
  k_chain_finish<DT, R0, R1><<<K, 256, 0, s>>>(a);
  return cudaGetLastError();
}

template <int DT>
cudaError_t run_chain_types(const ChainArgs& a, cudaStream_t s) {
  const int t0 = a.bk.c[0].type, t1 = a.bk.c[1].type;
  if (t0 < 2 && t1 < 2) return run_chain<DT, false, false, -1, -1>(a, s);
  if (t0 >= 2 && t1 >= 2) return run_chain<DT, true, true, -1, -1>(a, s);
  // the GS + integral-alpha pairs have kernels without the other samplers' code
  if (t0 == 2 && t1 == 1) return run_chain<DT, true, false, 2, 1>(a, s);
  if (t0 == 1 && t1 == 2) return run_chain<DT, false, true, 1, 2>(a, s);
  if (t0 >= 2) return run_chain<DT, true, false, -1, -1>(a, s);
  return run_chain<DT, false, true, -1, -1>(a, s);
}

}  // namespace

namespace {
// M positions of visits, P entries each; NR rejection components, ns entry
// states per segment; minu: fewest positions of an output.
ChainLayout layout_of(int K, int64_t n, int64_t M, int32_t J, int P, int NR, int ns, int minu, int pos_bytes) {
  ChainLayout L{};
  L.n = n;
  L.Sg = (J > 0 && NR && M > J) ? (int32_t)((M + J - 1) / J) : 1;
  L.J = L.Sg > 1 ? J : (int32_t)std::max<int64_t>(n, M);
  L.rcap = (int32_t)(L.J / minu + 2);
  if (!NR) return L;
  L.ns = L.Sg > 1 ? ns : 0;
  L.gsz = L.ns ? std::max(1, 65536 / (L.ns * 2)) : 0;
  L.groups = L.ns ? (L.Sg + L.gsz - 1) / L.gsz : 0;
  L.mstride = (int64_t)al((size_t)std::max<int64_t>(M, 1) + 256);
  const size_t segs = (size_t)K * L.Sg;
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += al(b);
    return at;
  };
  L.o_mask = take(pos_bytes ? (size_t)K * L.mstride * pos_bytes : (size_t)K * NR * L.mstride);
  L.o_vis = take((size_t)K * NR * L.mstride * P);
  L.o_tab = take(segs * L.ns * 2);
  L.o_gtab = take((size_t)K * L.groups * L.ns * 2);
  L.o_entry = take(segs * 4);
  L.o_seg = take(segs * sizeof(ChainSeg));
  L.o_ebase = take((segs + K) * 8);
  L.o_rec = take(segs * L.rcap * 4);
  L.o_prev = take(P > 1 ? segs * L.rcap * 2 * NR : 0);
  L.bytes = o;
  return L;
}
}  // namespace

ChainLayout chain_layout(const DistParams& d, int K, int64_t n, int32_t J) {
  const int P = d.dtype == GR_F32 ? 8 : 4;
  const int U0 = d.ia & 255, U1 = d.ib & 255;
  const bool R0 = (d.ia >> 8) >= 2, R1 = (d.ib >> 8) >= 2, RR = R0 && R1;
  return layout_of(K, n, n - std::max({U0, U1, 3}) + 1, J, P, (R0 ? 1 : 0) + (R1 ? 1 : 0), RR ? 32 * P * P : 64 * P,
                   U0 + U1, 0);
}

ChainLayout poisson_layout(int K, int64_t n, int32_t J) {
  return layout_of(K, n, 2 * n, J, 1, 1, entry_states<1, true, false>(), 1, 4);
}

cudaError_t launch_poisson_words(const Plan& p, const DistParams& d, const CallSnap* snap, const ChainLayout& L,
                                 char* scratch, int64_t* done, cudaStream_t s) {
  PoisArgs a{};
  a.c.p = p;
  a.c.bk.c[0].U = 1;
  a.c.bk.c[1].U = 0;
  a.c.L = L;
  a.c.vis = reinterpret_cast<uint8_t*>(scratch + L.o_vis);
  a.c.tab = reinterpret_cast<uint16_t*>(scratch + L.o_tab);
  a.c.gtab = reinterpret_cast<uint16_t*>(scratch + L.o_gtab);
  a.c.entry = reinterpret_cast<int32_t*>(scratch + L.o_entry);
  a.c.seg = reinterpret_cast<ChainSeg*>(scratch + L.o_seg);
  a.c.ebase = reinterpret_cast<int64_t*>(scratch + L.o_ebase);
  a.c.rec = reinterpret_cast<uint32_t*>(scratch + L.o_rec);
  a.c.done = done;
  a.c.M = (int32_t)(2 * L.n);
  a.pos = reinterpret_cast<uint32_t*>(scratch + L.o_mask);
  a.snap = snap;
  a.thr = d.fe;
  a.trials = d.ia;
  a.flip = d.ic;
  k_pois_steps<<<dim3((unsigned)((a.c.M + kStepThreads - 1) / kStepThreads), p.K), kStepThreads, 0, s>>>(a);
  cudaError_t e = run_core<1, true, false>(a.c, s);
  if (e != cudaSuccess) return e;
  k_pois_emit<<<dim3((unsigned)L.Sg, p.K), 256, 0, s>>>(a);
  k_pois_finish<<<p.K, 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_chain(const Plan& p, const DistParams& d, const ChainLayout& L, char* scratch, int64_t* done,
                         cudaStream_t s) {
  ChainArgs a{};
  a.p = p;
  a.bk.c[0] = beta_component(d.ia, d.fa, d.da);
  a.bk.c[1] = beta_component(d.ib, d.fb, d.db);
  a.bk.post = d.post;
  a.bk.fpost = d.fh;
  a.bk.dpost = d.dh;
  a.L = L;
  a.mask = reinterpret_cast<uint8_t*>(scratch + L.o_mask);
  a.tab = reinterpret_cast<uint16_t*>(scratch + L.o_tab);
  a.gtab = reinterpret_cast<uint16_t*>(scratch + L.o_gtab);
  a.entry = reinterpret_cast<int32_t*>(scratch + L.o_entry);
  a.seg = reinterpret_cast<ChainSeg*>(scratch + L.o_seg);
  a.ebase = reinterpret_cast<int64_t*>(scratch + L.o_ebase);
  a.vis = reinterpret_cast<uint8_t*>(scratch + L.o_vis);
  a.rec = reinterpret_cast<uint32_t*>(scratch + L.o_rec);
  a.prev = reinterpret_cast<uint16_t*>(scratch + L.o_prev);
  a.done = done;
  a.M = (int32_t)(L.n - std::max({a.bk.c[0].U, a.bk.c[1].U, 3}) + 1);
  if (a.M <= 0) return cudaSuccess;
  if (L.ns == 0 && L.mstride && L.rcap > 0xfffe) return cudaErrorInvalidValue;  // 16-bit places (gr_api.cu splits long calls)
  return d.dtype == GR_F64 ? run_chain_types<SD_F64>(a, s) : run_chain_types<SD_F32>(a, s);
}

}  // namespace gr
