// Temporal neighbour sampling, two kernels per hop:
//
//   sample_count_kernel  search of the row's time-sorted timestamps for the candidate window [lo, cut) of every target;
//                        stores the window and min(fanout, cut-lo), and the total of the CTA
//   sample_fill_kernel   output offsets from the CTA totals and the counts.  Windows that are copied as they are (recent:
//                        the tail; uniform with no more candidates than the fan-out) and picks (uniform: Floyd's k-subset
//                        with Philox4x32-10, ranked ascending) are written one OUTPUT ELEMENT per thread -- every lane
//                        busy, stores coalesced, all loads of a thread independent of each other.
//
// Large launches are bound by sectors: 384,000 recent-20 targets take 140 us (180 with 8-ary searches and one element per
// thread in flight, 155 before the copy loop was driven from shared memory), uniform-10 217 us (300 with a warp drawing for one
// target after the other, 235 before the draws were kept in registers); small ones by the chain of dependent loads: 4,096
// recent-20 targets 15 us as a graph of their own (20.5 with an arrival counter to clear and a last-CTA scan).
// One fused kernel (offsets by a look-back over the CTAs) was slower from 16,000 targets on: the look-back has to wait for
// the slowest search before it.
//
// Algorithmic HBM bytes per target: 16 (indptr pair) + 16 (target id, time) + 8*ceil(log2 deg) (search
// probes) + k_eff*24 (nbr, ts, eid reads) + k_eff*36 (five output arrays) + 8 (offset).
#include "chain.cuh"
#include "common.cuh"
#include "sampler.cuh"
#include "scan.cuh"

namespace sgl {
namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kCtaThreads = kWarpsPerCta * 32;
constexpr int kFillUnroll = 2;   // elements of a thread in flight (four cost registers, that is resident CTAs)

// first position p in [lo, hi) with ts[p] >= bound (hi when none); all 32 lanes cooperate and agree
__device__ __forceinline__ int64_t warp_lower_bound(const int64_t* __restrict__ ts, int64_t lo, int64_t hi,
                                                    int64_t bound, int lane) {
  while (hi - lo > 32) {
    int64_t stride = (hi - lo + 31) >> 5;
    int64_t p = lo + (int64_t)(lane + 1) * stride - 1;
    if (p > hi - 1) p = hi - 1;
    bool less = __ldg(ts + p) < bound;
    unsigned b = __ballot_sync(0xffffffffu, less);
    int c = __popc(b);  // probes are monotone, so the true ones are lanes [0, c)
    if (c == 32) return hi;
    int64_t p_first_false = lo + (int64_t)(c + 1) * stride - 1;
    if (p_first_false > hi - 1) p_first_false = hi - 1;
    if (c > 0) {
      int64_t p_last_true = lo + (int64_t)c * stride - 1;
      if (p_last_true > hi - 1) p_last_true = hi - 1;
      lo = p_last_true + 1;
    }
    hi = p_first_false;
  }
  bool less = (lo + lane < hi) && (__ldg(ts + lo + lane) < bound);
  return lo + __popc(__ballot_sync(0xffffffffu, less));
}

struct Philox {
  uint32_t c[4];
  __device__ __forceinline__ Philox(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1) {
    c[0] = c0; c[1] = c1; c[2] = c2; c[3] = c3;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
      uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
      uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
      c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
  }
};

// first position p in [lo, hi) with ts[p] >= bound, one lane on its own.  Every probe of a lane is its own 32-byte sector,
// so what a search costs is probes when there are many lanes (WIDE = false: halving, one probe per bit; 384,000 targets
// took 67 us with the other form, the load/store units busy with 2.3 probes per bit) and rounds when there are few
// (WIDE = true: three, then seven independent probes per round).
template <bool WIDE>
__device__ __forceinline__ int64_t lane_lower_bound(const int64_t* __restrict__ ts, int64_t lo, int64_t hi, int64_t bound) {
  if (!WIDE) {
    while (hi > lo) {
      const int64_t mid = lo + ((hi - lo) >> 1);
      if (__ldg(ts + mid) < bound) lo = mid + 1; else hi = mid;
    }
    return lo;
  }
  while (hi - lo > 256) {
    const int64_t q = (hi - lo) >> 2;
    int c = 0;                          // the probes are monotone: the first c of them are "less"
#pragma unroll
    for (int j = 1; j < 4; ++j) c += (__ldg(ts + lo + j * q) < bound) ? 1 : 0;
    const int64_t nlo = c ? lo + c * q + 1 : lo;
    if (c < 3) hi = lo + (c + 1) * q;
    lo = nlo;
  }
  while (hi - lo > 8) {
    const int64_t q = (hi - lo) >> 3;   // >= 1, and lo + 7 q < hi
    int c = 0;
#pragma unroll
    for (int j = 1; j < 8; ++j) c += (__ldg(ts + lo + j * q) < bound) ? 1 : 0;
    const int64_t nlo = c ? lo + c * q + 1 : lo;
    if (c < 7) hi = lo + (c + 1) * q;
    lo = nlo;
  }
  int c = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) c += (lo + j < hi && __ldg(ts + lo + j) < bound) ? 1 : 0;
  return lo + c;
}

// The same bound through the fence of the row (timestamp of the last edge of every 32-edge block, see sgl_tcsr_fence):
// the block that holds the answer is found in the fence -- a small array that lives in L2 -- and only that block of the
// row is read: one or two 128-byte lines of the timestamps per search instead of 32 scattered sectors per round.
__device__ __forceinline__ int64_t warp_fenced_lower_bound(const int64_t* __restrict__ ts, const int64_t* __restrict__ fence_row,
                                                           int64_t s, int64_t e, int64_t bound, int lane) {
  int64_t p0 = s;
  if (e - s > 32) {
    const int64_t nb = (e - s + 31) >> 5;
    const int64_t j = warp_lower_bound(fence_row, 0, nb, bound, lane);
    if (j >= nb) return e;
    p0 = s + (j << 5);
  }
  const bool less = (p0 + lane < e) && (__ldg(ts + p0 + lane) < bound);
  return p0 + __popc(__ballot_sync(0xffffffffu, less));
}

template <bool WIDE>
__device__ __forceinline__ int64_t lane_fenced_lower_bound(const int64_t* __restrict__ ts, const int64_t* __restrict__ fence_row,
                                                           int64_t s, int64_t e, int64_t bound) {
  if (e - s <= 32) return lane_lower_bound<WIDE>(ts, s, e, bound);
  const int64_t nb = (e - s + 31) >> 5;
  const int64_t j = lane_lower_bound<WIDE>(fence_row, 0, nb, bound);
  if (j >= nb) return e;
  const int64_t p0 = s + (j << 5), p1 = p0 + 32 < e ? p0 + 32 : e;
  return lane_lower_bound<WIDE>(ts, p0, p1, bound);
}

struct SampleArgs {
  const int64_t *indptr, *nbr, *ts, *eid, *fence;
  int64_t num_nodes;
  const int64_t *targets, *target_ts;
  int64_t n_cap;
  const int64_t* d_n;
  int fanout, policy, equal_root_time, keep_root_time;
  int64_t allowed_offset;
  uint64_t seed;
  uint32_t rng_stream;
  int64_t *out_nbr, *out_dst, *out_ts;
  float* out_dt;
  int64_t *out_dt_i64, *out_eid, *out_offsets;
  int64_t *win_lo, *win_cut;   // [n_cap] candidate window of every target
  int32_t* cnt;                // [n_cap] edges of every target
  int64_t* cta_sums;           // [count CTAs] edges of the CTA, or (more than kDirectCtas of them) of the CTAs before it
  unsigned int* done;          // arrival counter of the count CTAs (more than kDirectCtas)
  int64_t* total_out;          // optional second place for the number of sampled edges
  int32_t* d_status;
};

// Up to this many count CTAs a fill CTA adds up the totals before its own by itself (16 KB of L2 reads at most): no
// arrival counter to clear, no last CTA that scans while the others are gone.
constexpr int64_t kDirectCtas = 2048;

__device__ __forceinline__ uint64_t draw_below(int64_t target, int d, uint32_t rng_stream, uint64_t seed, uint64_t bound) {
  Philox ph((uint32_t)target, (uint32_t)((uint64_t)target >> 32), (uint32_t)d, rng_stream, (uint32_t)seed, (uint32_t)(seed >> 32));
  return ((uint64_t)ph.c[0] | ((uint64_t)ph.c[1] << 32)) % bound;
}

// x mod b, exactly, by reciprocal estimate and correction (Barrett's method in two 32-bit steps, the reciprocal of a Newton step in
// double precision): the quotient estimate is off by at most one -- the reciprocal's relative error is below 2^-45, a step's quotient
// below 2^32 --, which the remainder's sign and size show.  The compiler's 64-bit remainder was a third of the instructions of a
// launch that draws.
__device__ __forceinline__ uint32_t remainder_step(uint32_t upper, uint32_t lower, uint32_t b, double db, double inv) {
  const uint64_t y = ((uint64_t)upper << 32) | lower;      // upper < b
  const uint32_t q = __double2uint_rz(fma((double)upper, 4294967296.0, (double)lower) * inv);     // (saturates)
  int64_t r = (int64_t)(y - (uint64_t)q * b);
  r += r < 0 ? (int64_t)b : 0;
  r -= r >= (int64_t)b ? (int64_t)b : 0;
  return (uint32_t)r;
}
__device__ __forceinline__ uint32_t remainder_u32(uint64_t x, uint32_t b) {
  const double db = (double)b, guess = (double)__frcp_rn((float)b), inv = fma(guess, fma(-db, guess, 1.0), guess);   // one Newton step
  return remainder_step(remainder_step(0u, (uint32_t)(x >> 32), b, db, inv), (uint32_t)x, b, db, inv);
}

__device__ __forceinline__ uint32_t draw_below_u32(int64_t target, int d, uint32_t rng_stream, uint64_t seed, uint32_t bound) {
  Philox ph((uint32_t)target, (uint32_t)((uint64_t)target >> 32), (uint32_t)d, rng_stream, (uint32_t)seed, (uint32_t)(seed >> 32));
  return remainder_u32((uint64_t)ph.c[0] | ((uint64_t)ph.c[1] << 32), bound);
}

// Floyd's subset selection of `fanout` <= kRegPicks out of cand > fanout positions by one lane: draw d picks uniformly in [0, cand -
// fanout + d], a repeat is replaced by cand - fanout + d.  Everything in registers (unrolled: the round keys and a round of the
// generator are shared by the draws); the picks are left in ascending order.
constexpr int kRegPicks = 16;
__device__ __forceinline__ void draw_sorted(int64_t target, uint32_t cand, int fanout, uint32_t rng_stream, uint64_t seed, uint32_t* picks) {
  uint32_t pick[kRegPicks];
  int rank[kRegPicks];
#pragma unroll
  for (int d = 0; d < kRegPicks; ++d) {
    if (d < fanout) {
      const uint32_t top = cand - (uint32_t)fanout + (uint32_t)d;
      Philox ph((uint32_t)target, (uint32_t)((uint64_t)target >> 32), (uint32_t)d, rng_stream, (uint32_t)seed, (uint32_t)(seed >> 32));
      uint32_t x = remainder_u32((uint64_t)ph.c[0] | ((uint64_t)ph.c[1] << 32), top + 1u);
      bool clash = false;
#pragma unroll
      for (int q = 0; q < d; ++q) clash |= pick[q] == x;
      x = clash ? top : x;
      rank[d] = 0;
#pragma unroll
      for (int q = 0; q < d; ++q) {
        const bool above = pick[q] < x;
        rank[d] += above ? 1 : 0;
        rank[q] += above ? 0 : 1;
      }
      pick[d] = x;
    }
  }
#pragma unroll
  for (int d = 0; d < kRegPicks; ++d)
    if (d < fanout) picks[rank[d]] = pick[d];
}

__device__ __forceinline__ void emit_edge(const SampleArgs& a, int64_t p, int64_t o, int64_t t, int64_t target) {
  const int64_t ets = __ldg(a.ts + p);
  a.out_nbr[o] = __ldg(a.nbr + p);
  a.out_eid[o] = __ldg(a.eid + p);
  a.out_ts[o] = a.keep_root_time ? t : ets;
  a.out_dt[o] = (float)(t - ets);
  if (a.out_dt_i64) a.out_dt_i64[o] = ets - t;
  a.out_dst[o] = target;
}

// Windows and counts.  TPC targets per CTA: 8 = one warp per target (32-ary search), 256 = one lane per target (8-ary).
template <int TPC, bool WIDE>
__global__ void __launch_bounds__(kCtaThreads)
sample_count_kernel(const SampleArgs a) {
  constexpr bool kWarpPerTarget = TPC == kWarpsPerCta;
  const int64_t n = eff_count(a.n_cap, a.d_n);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * TPC + (kWarpPerTarget ? warp : (int)threadIdx.x);
  int32_t c = 0;
  if (i < n) {
    const int64_t node = __ldg(a.targets + i), t = __ldg(a.target_ts + i);
    const int64_t bound = t + (a.equal_root_time ? 1 : 0), from = t - a.allowed_offset;
    int64_t lo = 0, cut = 0;
    if (node < 0 || node >= a.num_nodes) {
      if (!kWarpPerTarget || lane == 0) dev_flag(a.d_status, SGL_DEV_BAD_NODE);
    } else {
      const int64_t s = __ldg(a.indptr + node), e = __ldg(a.indptr + node + 1);
      const int64_t* frow = a.fence ? a.fence + (s >> 5) + node : nullptr;
      lo = cut = s;
      if (e > s) {
        if (kWarpPerTarget) {
          cut = frow ? warp_fenced_lower_bound(a.ts, frow, s, e, bound, lane) : warp_lower_bound(a.ts, s, e, bound, lane);
          if (a.allowed_offset >= 0 && cut > s)
            lo = frow ? warp_fenced_lower_bound(a.ts, frow, s, e, from, lane) : warp_lower_bound(a.ts, s, cut, from, lane);
        } else {
          cut = frow ? lane_fenced_lower_bound<WIDE>(a.ts, frow, s, e, bound) : lane_lower_bound<WIDE>(a.ts, s, e, bound);
          if (a.allowed_offset >= 0 && cut > s)
            lo = frow ? lane_fenced_lower_bound<WIDE>(a.ts, frow, s, e, from) : lane_lower_bound<WIDE>(a.ts, s, cut, from);
        }
        if (lo > cut) lo = cut;
      }
    }
    c = (int32_t)(cut - lo < a.fanout ? cut - lo : a.fanout);
    if (!kWarpPerTarget || lane == 0) {
      a.win_lo[i] = lo;
      a.win_cut[i] = cut;
      a.cnt[i] = c;
    }
  }
  int total;
  cta_exclusive_scan<kCtaThreads, int>(!kWarpPerTarget || lane == 0 ? c : 0, &total);
  if (gridDim.x <= kDirectCtas) {
    if (threadIdx.x == 0) a.cta_sums[blockIdx.x] = total;
  } else {
    publish_and_scan_cta_totals<kCtaThreads>((int64_t)total, a.cta_sums, a.done, a.out_offsets + a.n_cap);
  }
}

// Edges of FT targets (FT divides CT, the targets per CTA of the count kernel).  Up to kMapFanout edges per target, shared memory
// says for every output element which target it belongs to and, where targets draw, which candidate it is, in output order: the
// copy loop is then a handful of instructions around its three loads.  (It was issue bound: 100 - 170 instructions per edge,
// 384,000 x 20 recent 101 us, a drawn hop of 4.2 M x 10 targets 458 us.)
constexpr int kMapFanout = 32;
// Without draws the kernel needs few registers, and the copy wants CTAs (384,000 x 20 recent: one kernel for both, 62 registers, 90.6 us;
// bounded to six CTAs per SM 84.7, to eight 84.5, four elements in flight per thread 86 - 111; 32, 128 and 256 targets per CTA 85, 86, 90).
// Targets that draw, a lane each, were no faster with more CTAs and spills (in the code for both: uniform, 40,000 targets, fan-out 33
// 176 -> 191 us).  A warp per target wants the CTAs, and draws best in the code for both: 40 registers, by itself 62 (uniform, 16,384 targets,
// fan-out 33 59.4 us, so 53.6, 100 175 and 152).
enum Fill { kCopies, kDraws, kEither };
template <int CT, int FT, Fill MODE>
__global__ void __launch_bounds__(kCtaThreads, MODE == kCopies ? 6 : MODE == kDraws ? 4 : 0)
sample_fill_kernel(const SampleArgs a, int count_ctas) {
  static_assert(CT % FT == 0 && CT <= kCtaThreads && FT % kWarpsPerCta == 0, "fill CTAs tile the count CTAs");
  constexpr bool kLaneDraws = CT != kWarpsPerCta;          // picks by the target's lane instead of its warp
  constexpr uint32_t kNotHere = ~0u;                       // (a candidate window this large is drawn from by a warp, below)
  constexpr int64_t kDrawn = INT64_MIN;
  extern __shared__ uint64_t s_dyn[];
  __shared__ int32_t s_ex[FT + 1];   // offset of the target's first element inside the CTA's output; [FT] = end
  __shared__ int64_t s_src[FT], s_t[FT];                   // what a candidate number, or an output position, is added to
  __shared__ int64_t s_base[kWarpsPerCta];
  const int64_t n = eff_count(a.n_cap, a.d_n);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t first = (int64_t)blockIdx.x * FT;          // this CTA's first target
  const int64_t count_cta = first / CT;
  const int sub = (int)(first - count_cta * CT);           // where this CTA's targets start inside the count CTA
  const int fanout = a.fanout;
  const bool direct = count_ctas <= kDirectCtas;
  const int slot = (int)threadIdx.x - sub;
  const int64_t i = count_cta * CT + threadIdx.x;
  const bool in_ct = threadIdx.x < CT && i < n, mine = slot >= 0 && slot < FT && threadIdx.x < CT;
  const int c = in_ct ? a.cnt[i] : 0;
  int64_t lo = 0, cut = 0, t = 0;
  if (mine && in_ct) {
    lo = a.win_lo[i];
    cut = a.win_cut[i];
    t = a.target_ts[i];
  }
  int64_t before = 0;
  if (direct) {
    for (int64_t b = threadIdx.x; b < count_cta; b += kCtaThreads) before += a.cta_sums[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) s_base[warp] = before;
  }
  int ct_total;
  const int ex = cta_exclusive_scan<kCtaThreads, int>(c, &ct_total);    // (its barriers also publish s_base)
  int64_t base = 0;
  if (direct) {
#pragma unroll
    for (int w = 0; w < kWarpsPerCta; ++w) base += s_base[w];
    if (threadIdx.x == 0 && first + FT >= a.n_cap) {
      a.out_offsets[a.n_cap] = base + ct_total;
      if (a.total_out) *a.total_out = base + ct_total;
    }
  } else {
    base = a.cta_sums[count_cta];
    if (threadIdx.x == 0 && first + FT >= a.n_cap && a.total_out) *a.total_out = a.out_offsets[a.n_cap];
  }
  const bool draws = MODE == kEither ? a.policy == SGL_POLICY_UNIFORM : MODE == kDraws, has_map = fanout <= kMapFanout;
  const bool drawn = draws && cut - lo > fanout;           // (of this thread's target)
  if (mine) {
    s_ex[slot] = ex;
    // recent: tail of the window; uniform with no more candidates than edges: the whole window
    s_src[slot] = has_map && draws ? lo : (drawn ? kDrawn : cut - c - ex);
    s_t[slot] = t;
    if (slot == FT - 1) s_ex[FT] = ex + c;
    // offsets past the valid targets all equal the total, so out_offsets[n..n_cap] stays a valid prefix array
    if (i < a.n_cap) a.out_offsets[i] = base + ex;
  }
  __syncthreads();
  const int begin = s_ex[0], end = s_ex[FT];
  const int64_t out0 = base + begin;
  bool left = draws;                                       // targets that draw are left for the warps
  if (has_map) {
    uint32_t* s_pos = (uint32_t*)s_dyn;                    // [FT * fanout] candidate of every element, where targets draw
    uint8_t* s_map = (uint8_t*)(s_pos + (draws ? FT * fanout : 0));
    if (kLaneDraws) {
      if (mine) {
        const int e0 = ex - begin;
        for (int j = 0; j < c; ++j) s_map[e0 + j] = (uint8_t)slot;
        if (draws) {
          const int64_t cand = cut - lo;
          if (!drawn || cand > 0xffffffffll) {
            for (int j = 0; j < c; ++j) s_pos[e0 + j] = drawn ? kNotHere : (uint32_t)j;
          } else if (fanout <= kRegPicks) {
            draw_sorted(i, (uint32_t)cand, fanout, a.rng_stream, a.seed, s_pos + e0);
          } else {
            for (int d = 0; d < fanout; ++d) {
              const uint32_t top = (uint32_t)(cand - fanout + d);
              uint32_t pick = draw_below_u32(i, d, a.rng_stream, a.seed, top + 1u);
              bool clash = false;
              for (int q = 0; q < d; ++q) clash |= s_pos[e0 + q] == pick;
              if (clash) pick = top;
              int q = d;                                   // ascending
              for (; q > 0 && s_pos[e0 + q - 1] > pick; --q) s_pos[e0 + q] = s_pos[e0 + q - 1];
              s_pos[e0 + q] = pick;
            }
          }
        }
      }
    } else {
      // one warp per target
      const int e0 = s_ex[warp] - begin, cw = s_ex[warp + 1] - s_ex[warp];
      if (lane < cw) s_map[e0 + lane] = (uint8_t)warp;
      if (draws) {
        const int64_t wcand = __shfl_sync(0xffffffffu, lane == 0 && first + warp < n ? a.win_cut[first + warp] - a.win_lo[first + warp] : 0, 0);
        if (wcand <= fanout || wcand > 0xffffffffll) {
          if (lane < cw) s_pos[e0 + lane] = wcand <= fanout ? (uint32_t)lane : kNotHere;
        } else {
          uint32_t pick = 0;
          if (lane < fanout) pick = draw_below_u32(first + warp, lane, a.rng_stream, a.seed, (uint32_t)(wcand - fanout + lane) + 1u);
          for (int d = 1; d < fanout; ++d) {
            const uint32_t other = __shfl_sync(0xffffffffu, pick, d);
            const bool clash = __any_sync(0xffffffffu, lane < d && pick == other);
            if (clash && lane == d) pick = (uint32_t)(wcand - fanout + d);
          }
          int rank = 0;                                    // ascending
          for (int d = 0; d < fanout; ++d) rank += __shfl_sync(0xffffffffu, pick, d) < pick ? 1 : 0;
          if (lane < fanout) s_pos[e0 + rank] = pick;
        }
      }
    }
    left = __syncthreads_or(mine && drawn && cut - lo > 0xffffffffll);
    // one output element per thread: all lanes busy, stores coalesced; the loads of kFillUnroll elements of a thread are in
    // flight together
    const int m = end - begin;
    for (int o0 = (int)threadIdx.x; o0 < m; o0 += kCtaThreads * kFillUnroll) {
      int at[kFillUnroll];
      int64_t ets[kFillUnroll], nb[kFillUnroll], ei[kFillUnroll];
#pragma unroll
      for (int u = 0; u < kFillUnroll; ++u) {
        const int o = o0 + u * kCtaThreads;
        at[u] = -1;
        if (o >= m) continue;
        const int k = s_map[o];
        uint32_t off = (uint32_t)(o + begin);
        if (draws) off = s_pos[o];
        if (draws && off == kNotHere) continue;
        const int64_t p = s_src[k] + off;
        at[u] = k;
        ets[u] = __ldg(a.ts + p);
        nb[u] = __ldg(a.nbr + p);
        ei[u] = __ldg(a.eid + p);
      }
#pragma unroll
      for (int u = 0; u < kFillUnroll; ++u) {
        if (at[u] < 0) continue;
        const int64_t g = out0 + (o0 + u * kCtaThreads), tt = s_t[at[u]];
        a.out_nbr[g] = nb[u];
        a.out_eid[g] = ei[u];
        a.out_ts[g] = a.keep_root_time ? tt : ets[u];
        a.out_dt[g] = (float)(tt - ets[u]);
        if (a.out_dt_i64) a.out_dt_i64[g] = ets[u] - tt;
        a.out_dst[g] = first + at[u];
      }
    }
  } else {
    for (int o = begin + (int)threadIdx.x; o < end; o += kCtaThreads) {
      int k = 0, b = FT;                   // last slot with s_ex[slot] <= o (its next offset is > o, so it is not empty)
      while (b - k > 1) {
        const int m = (k + b) >> 1;
        if (s_ex[m] <= o) k = m; else b = m;
      }
      if (s_src[k] != kDrawn) emit_edge(a, s_src[k] + o, base + o, s_t[k], first + k);
    }
  }
  if (!left) return;
  // targets that draw and were not served above: one warp per target
#pragma unroll 1
  for (int wslot = warp; wslot < FT; wslot += kWarpsPerCta) {
    const int64_t i = first + wslot;
    if (i >= n) break;
    const int64_t lo = a.win_lo[i], cand = a.win_cut[i] - lo;
    if (cand <= fanout || (has_map && cand <= 0xffffffffll)) continue;
    const int64_t t = s_t[wslot];
    const int64_t off = base + s_ex[wslot];
    if (fanout > 32) {
      // more draws than lanes: the same selection, with the picks of the target kept in this warp's shared memory
      uint64_t* picks = s_dyn + (size_t)warp * fanout;
      for (int d = lane; d < fanout; d += 32) picks[d] = draw_below(i, d, a.rng_stream, a.seed, (uint64_t)(cand - fanout + d + 1));
      __syncwarp();
      for (int d = 1; d < fanout; ++d) {          // draw d against the (final) draws before it
        const uint64_t mine = picks[d];
        bool clash = false;
        for (int q = lane; q < d; q += 32) clash |= picks[q] == mine;
        clash = __any_sync(0xffffffffu, clash);
        __syncwarp();
        if (clash && lane == 0) picks[d] = (uint64_t)(cand - fanout + d);
        __syncwarp();
      }
      for (int d = lane; d < fanout; d += 32) {   // rank ascending, then copy
        const uint64_t pick = picks[d];
        int rank = 0;
        for (int q = 0; q < fanout; ++q) rank += picks[q] < pick ? 1 : 0;
        emit_edge(a, lo + (int64_t)pick, off + rank, t, i);
      }
      __syncwarp();
    } else {
      uint64_t pick = 0;
      if (lane < fanout) pick = draw_below(i, lane, a.rng_stream, a.seed, (uint64_t)(cand - fanout + lane + 1));
      for (int d = 1; d < fanout; ++d) {
        uint64_t mine = __shfl_sync(0xffffffffu, pick, d);
        bool clash = lane < d && pick == mine;
        if (__any_sync(0xffffffffu, clash) && lane == d) pick = (uint64_t)(cand - fanout + d);
      }
      // rank ascending
      int rank = 0;
      for (int d = 0; d < fanout; ++d) {
        uint64_t other = __shfl_sync(0xffffffffu, pick, d);
        rank += (other < pick) ? 1 : 0;
      }
      if (lane < fanout) emit_edge(a, lo + (int64_t)pick, off + rank, t, i);
    }
  }
}

__global__ void __launch_bounds__(kCtaThreads)
draws_below_kernel(int64_t first_target, int draw, uint32_t rng_stream, uint64_t seed, const uint32_t* __restrict__ bounds, int64_t n,
                   uint32_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * kCtaThreads + threadIdx.x;
  if (i < n) out[i] = draw_below_u32(first_target + i, draw, rng_stream, seed, bounds[i]);
}

// number of sampled edges -> pinned host memory, then `seq` behind it; sums: one per count CTA
__global__ void __launch_bounds__(kCtaThreads)
export_total_kernel(const int64_t* __restrict__ sums, int count, int64_t* host, int64_t seq) {
  int64_t x = 0;
  for (int i = threadIdx.x; i < count; i += kCtaThreads) x += sums[i];
  int64_t total;
  cta_exclusive_scan<kCtaThreads, int64_t>(x, &total);
  if (threadIdx.x == 0) {
    *(volatile int64_t*)host = total;
    __threadfence_system();
    *(volatile int64_t*)(host + 1) = seq;
  }
}

// roots and query times of a mini-batch out of pinned host memory
__global__ void __launch_bounds__(256)
stage_roots_kernel(const int64_t* __restrict__ roots, const int64_t* __restrict__ times, int64_t n, int64_t* __restrict__ d_roots,
                   int64_t* __restrict__ d_times) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i < n) {
    d_roots[i] = roots[i];
    d_times[i] = times[i];
  }
}

}  // namespace
}  // namespace sgl

using namespace sgl;

// Up to 16,384 targets a warp each hides the latency of the few dependent loads; above, a lane each; from 65,536 on
// throughput counts and not the latency of one search.
constexpr int64_t kWarpTargets = 16384;
constexpr int64_t kManyTargets = 65536;

extern "C" size_t sgl_sample_ws_bytes(int64_t n_targets) {
  if (n_targets < 1) n_targets = 1;
  return 2 * align_up((size_t)n_targets * 8) + align_up((size_t)n_targets * 4) +
         align_up((size_t)((n_targets + kWarpsPerCta - 1) / kWarpsPerCta) * 8) + align_up(sizeof(unsigned int));
}

template <int CT, int FT, bool WIDE>
static int launch_sample(const SampleArgs& a, cudaStream_t stream, int64_t* host_total, int64_t seq) {
  const unsigned ctas = (unsigned)((a.n_cap + CT - 1) / CT);
  if (ctas > kDirectCtas) SGL_CHECK_RC(zero_async(a.done, sizeof(unsigned int), stream));
  SGL_CHECK_RC(launch(sample_count_kernel<CT, WIDE>, ctas, kCtaThreads, 0, stream, a));
  LaunchScope* in = LaunchScope::current();
  if (host_total && in) {
    // on its way while the edges are copied (a second chain of the graph)
    cudaStream_t side = (cudaStream_t)(uintptr_t)3;
    SGL_CHECK_RC(in->follow(side, stream));
    const bool direct = ctas <= kDirectCtas;
    SGL_CHECK_RC(launch(export_total_kernel, 1, kCtaThreads, 0, side, direct ? a.cta_sums : a.out_offsets + a.n_cap, direct ? (int)ctas : 1,
                        host_total, seq));
  }
  size_t smem = 0;
  if (a.policy == SGL_POLICY_UNIFORM) {
    if (a.fanout > kMapFanout) smem = (size_t)kWarpsPerCta * a.fanout * sizeof(uint64_t);
    else smem = (size_t)FT * a.fanout * sizeof(uint32_t);
  }
  if (a.fanout <= kMapFanout) smem += (size_t)FT * a.fanout;
  const unsigned fill_ctas = (unsigned)((a.n_cap + FT - 1) / FT);
  constexpr Fill kUniform = CT == kWarpsPerCta ? kEither : kDraws;
  return a.policy == SGL_POLICY_UNIFORM ? launch(sample_fill_kernel<CT, FT, kUniform>, fill_ctas, kCtaThreads, smem, stream, a, (int)ctas)
                                        : launch(sample_fill_kernel<CT, FT, kCopies>, fill_ctas, kCtaThreads, smem, stream, a, (int)ctas);
}

int sgl::check_sampling(int fanout, int policy, int64_t n_targets) {
  SGL_REQUIRE(fanout >= 1, SGL_ERR_ARG, "sample_layer: fanout=%d must be >= 1", fanout);
  SGL_REQUIRE(policy == SGL_POLICY_RECENT || policy == SGL_POLICY_UNIFORM, SGL_ERR_ARG, "sample_layer: unknown policy %d", policy);
  SGL_REQUIRE(policy != SGL_POLICY_UNIFORM || fanout <= SGL_MAX_UNIFORM_FANOUT, SGL_ERR_UNSUPPORTED, "sample_layer: uniform fanout %d > %d", fanout,
              SGL_MAX_UNIFORM_FANOUT);
  SGL_REQUIRE(n_targets < ((int64_t)1 << 34), SGL_ERR_UNSUPPORTED, "sample_layer: too many targets");
  return SGL_OK;
}

int sgl::sample_layer(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                      int64_t num_nodes, const int64_t* targets, const int64_t* target_ts, int64_t n_targets, const int64_t* d_n,
                      int fanout, int policy, int equal_root_time, int64_t allowed_offset, int keep_root_time, uint64_t seed,
                      uint32_t rng_stream, int64_t* out_nbr, int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_dt_i64,
                      int64_t* out_eid, int64_t* out_offsets, int64_t* total_out, int32_t* d_status, void* ws, size_t ws_bytes,
                      void* stream_, int64_t* host_total, int64_t seq) {
  SGL_NVTX("sgl_sample_layer");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_targets >= 0 && num_nodes >= 0, SGL_ERR_ARG, "sample_layer: negative size");
  SGL_CHECK_RC(check_sampling(fanout, policy, n_targets));
  SGL_REQUIRE(out_offsets, SGL_ERR_ARG, "sample_layer: out_offsets is null");
  if (n_targets == 0) {
    SGL_CHECK_RC(zero_async(out_offsets, sizeof(int64_t), stream));
    if (total_out) SGL_CHECK_RC(zero_async(total_out, sizeof(int64_t), stream));
    if (host_total) {
      host_total[0] = 0;
      host_total[1] = seq;
    }
    return SGL_OK;
  }
  SGL_REQUIRE(indptr && nbr && ts && eid && targets && target_ts && out_nbr && out_dst && out_ts && out_dt && out_eid,
              SGL_ERR_ARG, "sample_layer: null array");
  SampleArgs a;
  a.indptr = indptr; a.nbr = nbr; a.ts = ts; a.eid = eid; a.fence = fence;
  a.num_nodes = num_nodes;
  a.targets = targets; a.target_ts = target_ts;
  a.n_cap = n_targets;
  a.d_n = d_n;
  a.fanout = fanout; a.policy = policy; a.equal_root_time = equal_root_time; a.keep_root_time = keep_root_time;
  a.allowed_offset = allowed_offset;
  a.seed = seed;
  a.rng_stream = rng_stream;
  a.out_nbr = out_nbr; a.out_dst = out_dst; a.out_ts = out_ts;
  a.out_dt = out_dt;
  a.out_dt_i64 = out_dt_i64; a.out_eid = out_eid; a.out_offsets = out_offsets;
  a.total_out = total_out;
  a.d_status = d_status;
  WsCarver c(ws, ws_bytes);
  a.win_lo = c.take<int64_t>(n_targets);
  a.win_cut = c.take<int64_t>(n_targets);
  a.cnt = c.take<int32_t>(n_targets);
  a.cta_sums = c.take<int64_t>((size_t)((n_targets + kWarpsPerCta - 1) / kWarpsPerCta));
  a.done = c.take<unsigned int>(1);
  SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "sample_layer: workspace %zu < %zu bytes", ws_bytes,
              sgl_sample_ws_bytes(n_targets));
  LaunchScope scope(stream);
  if (n_targets <= kWarpTargets) {
    SGL_CHECK_RC((launch_sample<kWarpsPerCta, kWarpsPerCta, true>(a, stream, host_total, seq)));
  } else if (policy == SGL_POLICY_UNIFORM) {
    // targets per fill CTA: a lane of the CTA draws for every target, so as many as there are threads once that leaves
    // several CTAs per SM; windows that are copied are spread thinner
    if (n_targets < kManyTargets) SGL_CHECK_RC((launch_sample<kCtaThreads, 128, true>(a, stream, host_total, seq)));
    else SGL_CHECK_RC((launch_sample<kCtaThreads, 256, false>(a, stream, host_total, seq)));
  } else {
    if (n_targets < kManyTargets) SGL_CHECK_RC((launch_sample<kCtaThreads, 64, true>(a, stream, host_total, seq)));
    else SGL_CHECK_RC((launch_sample<kCtaThreads, 64, false>(a, stream, host_total, seq)));
  }
  return scope.submit();
}

extern "C" int sgl_sample_layer(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                                int64_t num_nodes, const int64_t* targets, const int64_t* target_ts, int64_t n_targets,
                                const int64_t* d_n, int fanout, int policy, int equal_root_time, int64_t allowed_offset,
                                int keep_root_time, uint64_t seed, uint32_t rng_stream, int64_t* out_nbr,
                                int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_dt_i64,
                                int64_t* out_eid, int64_t* out_offsets, int32_t* d_status, void* ws, size_t ws_bytes,
                                void* stream) {
  return sgl::sample_layer(indptr, nbr, ts, eid, nullptr, num_nodes, targets, target_ts, n_targets, d_n, fanout, policy,
                           equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts, out_dt,
                           out_dt_i64, out_eid, out_offsets, nullptr, d_status, ws, ws_bytes, stream);
}

extern "C" int sgl_sample_layer_counted(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                                        const int64_t* fence, int64_t num_nodes, const int64_t* targets, const int64_t* target_ts,
                                        int64_t n_targets, const int64_t* d_n, int fanout, int policy, int equal_root_time,
                                        int64_t allowed_offset, int keep_root_time, uint64_t seed, uint32_t rng_stream,
                                        int64_t* out_nbr, int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_dt_i64,
                                        int64_t* out_eid, int64_t* out_offsets, int32_t* d_status, void* ws, size_t ws_bytes,
                                        int64_t* host_total, int64_t seq, void* stream) {
  return sgl::sample_layer(indptr, nbr, ts, eid, fence, num_nodes, targets, target_ts, n_targets, d_n, fanout, policy,
                           equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts, out_dt,
                           out_dt_i64, out_eid, out_offsets, nullptr, d_status, ws, ws_bytes, stream, host_total, seq);
}

extern "C" int sgl_sample_layer_fenced(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                                       const int64_t* fence, int64_t num_nodes, const int64_t* targets, const int64_t* target_ts,
                                       int64_t n_targets, const int64_t* d_n, int fanout, int policy, int equal_root_time,
                                       int64_t allowed_offset, int keep_root_time, uint64_t seed, uint32_t rng_stream,
                                       int64_t* out_nbr, int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_dt_i64,
                                       int64_t* out_eid, int64_t* out_offsets, int32_t* d_status, void* ws, size_t ws_bytes,
                                       void* stream) {
  return sgl::sample_layer(indptr, nbr, ts, eid, fence, num_nodes, targets, target_ts, n_targets, d_n, fanout, policy,
                           equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts, out_dt,
                           out_dt_i64, out_eid, out_offsets, nullptr, d_status, ws, ws_bytes, stream);
}

extern "C" int sgl_sample_gather_fenced(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                                        const int64_t* fence, int64_t num_nodes, const int64_t* targets, const int64_t* target_ts,
                                        int64_t n_targets, int fanout, int policy, int equal_root_time, int64_t allowed_offset,
                                        int keep_root_time, uint64_t seed, uint32_t rng_stream, int64_t* out_nbr, int64_t* out_dst,
                                        int64_t* out_ts, float* out_dt, int64_t* out_eid, int64_t* out_offsets,
                                        const void* feat_table, int64_t feat_rows, int64_t row_bytes, int64_t src_pitch,
                                        void* out_feats, int gather_mode, int32_t* d_status, void* ws, size_t ws_bytes, void* stream) {
  LaunchScope scope((cudaStream_t)stream);
  int rc = sgl::sample_layer(indptr, nbr, ts, eid, fence, num_nodes, targets, target_ts, n_targets, nullptr, fanout, policy,
                             equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts, out_dt,
                             nullptr, out_eid, out_offsets, nullptr, d_status, ws, ws_bytes, stream);
  if (rc != SGL_OK) return rc;
  if (n_targets == 0) return scope.submit();
  SGL_CHECK_RC(sgl_gather_rows(feat_table, feat_rows, row_bytes, src_pitch, out_eid, nullptr, 0, n_targets * fanout,
                         out_offsets + n_targets, out_feats, row_bytes, nullptr, nullptr, gather_mode, d_status, stream));
  return scope.submit();
}

// One graph launch per mini-batch.  Driven from Python as two copies, three kernels, two events and a read-back a batch cost
// 80 us of host time, four batches in flight 343 us for 100 us of kernels; small inputs are read by a kernel because a
// copy engine takes 4 us to start.
extern "C" int sgl_prefetch_batch(const int64_t* host_roots, const int64_t* host_ts, const int64_t* indptr, const int64_t* nbr,
                                  const int64_t* ts, const int64_t* eid, const int64_t* fence, int64_t num_nodes, int64_t* targets,
                                  int64_t* target_ts, int64_t n_targets, int fanout, int policy, int equal_root_time,
                                  int64_t allowed_offset, int keep_root_time, uint64_t seed, uint32_t rng_stream, int64_t* out_nbr,
                                  int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_eid, int64_t* out_offsets,
                                  const void* feat_table, int64_t feat_rows, int64_t row_bytes, int64_t src_pitch, void* out_feats,
                                  int gather_mode, int32_t* d_status, void* ws, size_t ws_bytes, int64_t* host_total, int64_t seq,
                                  void* consumer, void* stream_) {
  SGL_NVTX("sgl_prefetch_batch");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_targets >= 0 && host_total && (host_roots == nullptr) == (host_ts == nullptr), SGL_ERR_ARG, "prefetch_batch: bad argument");
  SGL_CHECK_RC(order_after(stream, (cudaStream_t)consumer));
  LaunchScope scope(stream);
  if (host_roots && n_targets > 0)
    SGL_CHECK_RC(launch(stage_roots_kernel, (unsigned)((n_targets + 255) / 256), 256, 0, stream, host_roots, host_ts, n_targets, targets,
                        target_ts));
  SGL_CHECK_RC(sgl::sample_layer(indptr, nbr, ts, eid, fence, num_nodes, targets, target_ts, n_targets, nullptr, fanout, policy,
                                 equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts, out_dt,
                                 nullptr, out_eid, out_offsets, nullptr, d_status, ws, ws_bytes, stream, host_total, seq));
  if (out_feats && n_targets > 0)
    SGL_CHECK_RC(sgl_gather_rows(feat_table, feat_rows, row_bytes, src_pitch, out_eid, nullptr, 0, n_targets * fanout,
                                 out_offsets + n_targets, out_feats, row_bytes, nullptr, nullptr, gather_mode, d_status, stream));
  return scope.submit();
}

extern "C" int sgl_sample_gather(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                                 int64_t num_nodes, const int64_t* targets, const int64_t* target_ts, int64_t n_targets,
                                 int fanout, int policy, int equal_root_time, int64_t allowed_offset, int keep_root_time,
                                 uint64_t seed, uint32_t rng_stream, int64_t* out_nbr, int64_t* out_dst, int64_t* out_ts,
                                 float* out_dt, int64_t* out_eid, int64_t* out_offsets, const void* feat_table,
                                 int64_t feat_rows, int64_t row_bytes, int64_t src_pitch, void* out_feats, int gather_mode,
                                 int32_t* d_status, void* ws, size_t ws_bytes, void* stream) {
  SGL_NVTX("sgl_sample_gather");
  LaunchScope scope((cudaStream_t)stream);
  int rc = sgl_sample_layer(indptr, nbr, ts, eid, num_nodes, targets, target_ts, n_targets, nullptr, fanout, policy,
                            equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts,
                            out_dt, nullptr, out_eid, out_offsets, d_status, ws, ws_bytes, stream);
  if (rc != SGL_OK) return rc;
  if (n_targets == 0) return scope.submit();
  SGL_CHECK_RC(sgl_gather_rows(feat_table, feat_rows, row_bytes, src_pitch, out_eid, nullptr, 0, n_targets * fanout,
                         out_offsets + n_targets, out_feats, row_bytes, nullptr, nullptr, gather_mode, d_status, stream));
  return scope.submit();
}

extern "C" int sgl_draws_below(int64_t first_target, int draw, uint32_t rng_stream, uint64_t seed, const uint32_t* bounds, int64_t n,
                               uint32_t* out, void* stream) {
  SGL_REQUIRE(n >= 0 && n < ((int64_t)1 << 38) && (n == 0 || (bounds && out)), SGL_ERR_ARG, "draws_below: bad argument");
  if (n == 0) return SGL_OK;
  return launch(draws_below_kernel, (unsigned)((n + kCtaThreads - 1) / kCtaThreads), kCtaThreads, 0, (cudaStream_t)stream, first_target, draw,
                rng_stream, seed, bounds, n, out);
}

// ---------------------------------------------------------------------------------------------------------------
// Sampling without caller-provided scratch.
//
// Some hosts of this library cannot hand it device memory on demand: a sampler thread that runs next to a training
// loop must not call cudaMalloc (it stalls every stream of the device while it runs), and a process whose HBM has
// been handed in full to another framework's pool has no allocator of its own to ask.  For them the scratch of one
// hop lives in a fixed array inside the library image instead.  Every GPU that loads the library carries the array
// (about 1.3 MB) until the process exits.
// ---------------------------------------------------------------------------------------------------------------
namespace {
constexpr int64_t kStaticMaxTargets = SGL_STATIC_SAMPLE_MAX_TARGETS;
// same layout as the caller-provided workspace of sgl_sample_layer for kStaticMaxTargets targets
constexpr size_t kStaticScratchBytes = 2 * ((kStaticMaxTargets * 8 + 255) / 256 * 256) + ((kStaticMaxTargets * 4 + 255) / 256 * 256) +
                                       ((kStaticMaxTargets / kWarpsPerCta * 8 + 255) / 256 * 256) + 256;
static __device__ __align__(256) unsigned char g_static_sample_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_static_scratch_addr[kMaxDevices];   // device address of the array, per device, filled on first use
}  // namespace

extern "C" int sgl_sample_layer_static(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                                       int64_t num_nodes, const int64_t* targets, const int64_t* target_ts,
                                       int64_t n_targets, int fanout, int policy, int equal_root_time,
                                       int64_t allowed_offset, int keep_root_time, uint64_t seed, uint32_t rng_stream,
                                       int64_t* out_nbr, int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_eid,
                                       int64_t* out_offsets, int32_t* d_status, void* stream) {
  SGL_REQUIRE(n_targets >= 0 && n_targets <= kStaticMaxTargets, SGL_ERR_ARG,
              "sample_layer_static: %lld targets exceed the built-in scratch (at most %lld per call); use sgl_sample_layer "
              "with your own workspace for larger batches", (long long)n_targets, (long long)kStaticMaxTargets);
  int dev = -1;
  SGL_CUDA_CHECK(cudaGetDevice(&dev));
  SGL_REQUIRE(dev >= 0 && dev < kMaxDevices, SGL_ERR_UNSUPPORTED, "sample_layer_static: device index %d not supported", dev);
  if (g_static_scratch_addr[dev] == nullptr) {
    // In host code the array's name is only a handle; the address kernels can use has to be asked for, once per
    // device, with that device current.
    void* p = nullptr;
    SGL_CUDA_CHECK(cudaGetSymbolAddress(&p, g_static_sample_scratch));
    SGL_REQUIRE(p != nullptr, SGL_ERR_CUDA, "sample_layer_static: no device address for the built-in scratch");
    g_static_scratch_addr[dev] = p;
  }
  // (no clearing: launches of this size leave the only word of the scratch that would need it alone)
  const PlainLaunches plain;
  return sgl_sample_layer(indptr, nbr, ts, eid, num_nodes, targets, target_ts, n_targets, nullptr, fanout, policy,
                          equal_root_time, allowed_offset, keep_root_time, seed, rng_stream, out_nbr, out_dst, out_ts,
                          out_dt, nullptr, out_eid, out_offsets, d_status, g_static_scratch_addr[dev], kStaticScratchBytes,
                          stream);
}
