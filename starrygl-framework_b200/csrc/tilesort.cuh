// Stable sort of mini-batch sized lists (up to 1,212,416 items) in TWO kernels, with the producer of the keys and the
// consumer of the sorted order fused into them:
//
//   ts_part_kernel<Source>    a CTA makes the keys of its tile (Source), sorts a sample of the whole list -- every CTA the
//                             same one -- takes one splitter per CTA from it and groups its items by bucket
//   ts_bucket_kernel<Sink>    a CTA collects its bucket's pieces from all tiles, sorts them and hands every item to the
//                             Sink with its global position -- and, for sinks that number distinct keys, the rank of its
//                             key among them
//   ts_single_kernel          lists of at most 2,048 items: one CTA
//
// An item is (key, position): the position breaks ties, so the order is the stable one, all items differ, and a bucket
// cannot grow with the number of equal keys.  Key and position share one 64-bit word when they fit, otherwise a 64-bit
// and a 32-bit word (WIDE).
//
// What bounds it: latency.  A list of 40 k - 300 k keys is 0.3 - 2 MB, a microsecond of bandwidth; the chain is two
// launches, a sample sort and an in-CTA sort.  The tile size is picked ON THE DEVICE from the item count, so that a
// list spreads over all 148 SMs even when the launch capacity is several times the actual count (multi-hop batches).
// Every instruction here is fetched once or twice per CTA, and that, not memory, was half of the time: loops over the item slots of a
// thread jump over the slots that the CTA's items do not reach, sums over warps are warp reductions instead of unrolled loads, and
// splitters are searched by one rolled loop for all items of a thread.  Both kernels together, unique (id, time) pairs of 44 bits:
// 4,096 pairs 12.3 us (17.9 before), 41,000 17.6 (23.1), 144,000 23.5 (32.6), 300,000 34.2 (50.5); with a power-law share of the ids
// 14.9 (18.4), 17.2 (22.9), 25.8 (32.2), 39.5 (50.1).  One CTA, 100 / 600 / 1,500 / 2,048 pairs: 4.2 / 5.6 / 7.4 / 8.5 us (4.5 / 7.3 /
// 10.9 / 13.5); power law 4.5 / 6.9 / 10.5 / 12.8 (4.5 / 7.2 / 11.0 / 13.5), thirty copies of every pair 4.5 / 7.1 / 10.4 / 12.1 (4.5 / 7.4 /
// 11.0 / 12.9): these go to the pivots at once (cut into bins two to four times they took 6.1 / 8.1 / 10.9 / 13.3 and 5.2 / 8.2 / 12.1 / 13.9).
// An LSD radix sort with one kernel per 11 key bits took 25, 84 and 95 us for 4,096, 41,000 and 160,000 pairs: few CTAs with large
// digit tables, and a dependent kernel per digit.
#pragma once
#include "common.cuh"
#include "launch.cuh"
#include "scan.cuh"

namespace sgl {
namespace tilesort {

constexpr int kMaxCtas = kNumSM;        // tiles, and buckets: one CTA per SM
constexpr int kThreadBits = 9;
constexpr int kThreads = 1 << kThreadBits;   // threads of every kernel here; at least kMaxCtas (1,024 were no faster)
constexpr int kWarps = kThreads / 32;
// The kernels' registers are bounded as if they had more threads: the whole register file of an SM would keep everything else off it
// (the CSC of a hop next to the merge of the next list: 11 us, 40 us when it had to wait for the merge's CTAs).
constexpr int kRegThreads = 640;
constexpr int kMinTile = 256;
constexpr int kMaxTile = 8192;
constexpr int kTileItems = kMaxTile / kThreads;
constexpr int kMaxSamples = 2048;       // sample of the whole list: about fourteen per bucket with 148 buckets
// (Capacity: what a launch holds at most.  Lists that really are that long have buckets beyond shared memory and sort them
// in L2, still no slower than the radix passes; multi-hop lists usually fill a third of their capacity.)
constexpr int64_t kMaxItems = (int64_t)kMaxCtas * kMaxTile;
constexpr int kSingleMax = 2048;
constexpr unsigned long long kWaitNs = 2000000000ull;

struct Item {
  uint64_t k;
  uint32_t p;
};

template <bool WIDE>
struct View {                           // items in shared or global memory
  uint64_t* k;
  uint32_t* p;
  __device__ __forceinline__ Item get(int i) const { return {k[i], WIDE ? p[i] : 0u}; }
  __device__ __forceinline__ void set(int i, const Item& x) const {
    k[i] = x.k;
    if (WIDE) p[i] = x.p;
  }
};

template <bool WIDE>
__device__ __forceinline__ bool less(const Item& a, const Item& b) {
  return WIDE ? (a.k < b.k || (a.k == b.k && a.p < b.p)) : a.k < b.k;
}
template <bool WIDE>
__device__ __forceinline__ Item make_item(uint64_t key, uint32_t pos, int pos_bits) {
  return WIDE ? Item{key, pos} : Item{(key << pos_bits) | pos, 0u};
}
template <bool WIDE>
__device__ __forceinline__ uint64_t key_of(const Item& x, int pos_bits) {
  return WIDE ? x.k : (x.k >> pos_bits);
}
template <bool WIDE>
__device__ __forceinline__ uint32_t pos_of(const Item& x, int pos_bits) {
  return WIDE ? x.p : (uint32_t)(x.k & ((1ull << pos_bits) - 1ull));
}

// one position out of the j-th of 2^sb equal parts of [0, m), m >= 2^sb
__device__ __forceinline__ int sample_at(int j, int sb, int m) {
  const uint32_t a = (uint32_t)(((uint64_t)j * (uint32_t)m) >> sb), b = (uint32_t)(((uint64_t)(j + 1) * (uint32_t)m) >> sb);
  return (int)(a + __umulhi((uint32_t)j * 0x9E3779B1u, b - a));
}

// Sort of m distinct items inside a CTA, in place; tmp, aux and grp are scratch of m entries.
//   1. q = 2^QB sampled items are put in order by counting, for each, the smaller ones among them (q * q comparisons)
//   2. every item finds its group between two of them; groups are counted and laid out
//   3. inside its group (about m / q items) an item's place is again the number of smaller ones
// Every step is wide and short.  A bitonic network has log^2 stages that depend on each other: 1,100 items took
// 11,000 - 18,000 cycles, most of it latency.  q is a compile-time number so that the counting loops of steps 1 and 2
// are straight loads and comparisons.
template <bool WIDE, int QB>
__device__ __forceinline__ void group_sort(const View<WIDE>& v, const View<WIDE>& tmp, uint32_t* aux, uint16_t* grp, int m) {
  constexpr int Q = 1 << QB, STEP = QB > 4 ? QB - 4 : 0;
  constexpr int PB = kThreadBits - QB < 5 ? kThreadBits - QB : 5;    // 2^PB lanes share one sample
  __shared__ uint64_t s_raw_k[Q], s_piv_k[Q];
  __shared__ uint32_t s_raw_p[WIDE ? Q : 1], s_piv_p[WIDE ? Q : 1];
  __shared__ int s_start[Q + 2], s_cnt[Q + 1], s_wsum[kWarps];
  const View<WIDE> raw{s_raw_k, s_raw_p}, piv{s_piv_k, s_piv_p};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();
  if (tid < Q) raw.set(tid, v.get(sample_at(tid, QB, m)));
  if (tid <= Q) s_cnt[tid] = 0;
  __syncthreads();
  if (tid < Q << PB) {
    const Item x = raw.get(tid >> PB);
    const int part = tid & ((1 << PB) - 1);
    int below = 0;
#pragma unroll
    for (int i = 0; i < Q >> PB; ++i) below += less<WIDE>(raw.get((i << PB) + part), x) ? 1 : 0;
#pragma unroll
    for (int o = 1; o < 1 << PB; o <<= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    if (part == 0) piv.set(below, x);
  }
  __syncthreads();
  for (int i = tid; i < m; i += kThreads) {
    // first against every 2^STEP-th pivot, which all lanes read at the same address, then a few probes of their own
    const Item x = v.get(i);
    int g = 0;
#pragma unroll
    for (int j = 0; j < Q >> STEP; ++j) g += less<WIDE>(x, piv.get(((j + 1) << STEP) - 1)) ? 0 : 1;
    g <<= STEP;
    if (g < Q) {
#pragma unroll
      for (int h = (1 << STEP) >> 1; h >= 1; h >>= 1) g += less<WIDE>(x, piv.get(g + h - 1)) ? 0 : h;
    }
    aux[i] = ((uint32_t)g << 21) | (uint32_t)atomicAdd(&s_cnt[g], 1);
  }
  __syncthreads();
  {
    const int c = tid <= Q ? s_cnt[tid] : 0;
    int x = warp_inclusive_scan(c, lane);
    if (lane == 31) s_wsum[warp] = x;
    __syncthreads();
    x += __reduce_add_sync(0xffffffffu, lane < warp && lane < kWarps ? s_wsum[lane] : 0);
    if (tid <= Q) s_start[tid + 1] = x;
    if (tid == 0) s_start[0] = 0;
    __syncthreads();
  }
  for (int i = tid; i < m; i += kThreads) {
    const uint32_t a = aux[i];
    const int g = (int)(a >> 21), at = s_start[g] + (int)(a & 0x1fffffu);
    tmp.set(at, v.get(i));
    grp[at] = (uint16_t)g;
  }
  __syncthreads();
  for (int i = tid; i < m; i += kThreads) {
    const Item x = tmp.get(i);
    const int g = grp[i], a = s_start[g], e = s_start[g + 1];
    int below = a, j = a;
    for (; j + 4 <= e; j += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) below += less<WIDE>(tmp.get(j + u), x) ? 1 : 0;
    }
    for (; j < e; ++j) below += less<WIDE>(tmp.get(j), x) ? 1 : 0;
    v.set(below, x);
  }
  __syncthreads();
}

// A few items: every item is compared with every other.
template <bool WIDE>
__device__ __forceinline__ void rank_sort(const View<WIDE>& v, const View<WIDE>& tmp, int m) {
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += kThreads) tmp.set(i, v.get(i));
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += kThreads) {
    const Item x = tmp.get(i);
    int below = 0;
#pragma unroll 4
    for (int j = 0; j < m; ++j) below += less<WIDE>(tmp.get(j), x) ? 1 : 0;
    v.set(below, x);
  }
  __syncthreads();
}

// smallest and largest of a warp's words, by halves (64-bit shuffles would be 20 dependent steps)
__device__ __forceinline__ uint64_t warp_min(uint64_t x) {
  const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(x >> 32));
  return ((uint64_t)hi << 32) | __reduce_min_sync(0xffffffffu, (uint32_t)(x >> 32) == hi ? (uint32_t)x : ~0u);
}
__device__ __forceinline__ uint64_t warp_max(uint64_t x) {
  const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(x >> 32));
  return ((uint64_t)hi << 32) | __reduce_max_sync(0xffffffffu, (uint32_t)(x >> 32) == hi ? (uint32_t)x : 0u);
}

// Sort of up to K * kThreads items inside a CTA by counting: the range of the items is cut into 2^b >= m equal bins; while a bin
// holds more than a few of its c items it is cut again, into 2^b >= c; inside a bin an item's place is the number of smaller
// ones.  A uniform list is done after one level, a list with a few ids that hold a large part of it after two or three.  One atomic
// and two loads of shared memory per item and level, and a scan of at most 2 m counters.  Copies of one key stay together until bins
// are as narrow as positions: where crowded bins are full of them (recent neighbours of the same few nodes), or after kSpreadLevels
// levels, it gives up and leaves the items as they were; returns whether they are sorted.
// ALONE (a list that one CTA sorts; buckets of a longer one are cut by its splitters already): a list whose items crowd is left to the
// pivots before anything is counted.  It shows in pairs of lanes that are close to each other: 3 % of the threads see one among five
// others if an id holds 8 % of the list or a pair has thirty copies of 1,500, and 0.2 % of them where all are alike.
// cnt: scratch of 2 m words, 16-byte aligned, and 16 bytes that may be written behind them; some: 2 m half words.
constexpr int kSpreadFew = 16, kSpreadLevels = 4;         // (16, 32, 64, 128 items of a bin are left to comparisons at levels 1 - 4)
constexpr int kSpreadCopies = 32;                         // threads that may hold a copy of a crowded bin's first key
template <bool WIDE, int K, bool ALONE>
__device__ __forceinline__ bool spread_sort(const View<WIDE>& v, uint32_t* cnt, uint16_t* some, int m, int pos_bits) {
  constexpr int R = K / 2;               // rounds of a scan: four counters per thread and round, 2 m counters
  static_assert(K % 2 == 0 && 2 * K * kThreads < (1 << 16), "items and bins are counted in 16 bits each");
  __shared__ uint64_t s_lo[kWarps], s_hi[kWarps];
  __shared__ uint32_t s_sum[R][kWarps], s_end;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Item x[K];
  uint32_t bin[K], in[K];                // bin of the item (upper half: bits of the key below what the bin says), its number in it
  __syncthreads();
  uint64_t lo = ~0ull, hi = 0;
#pragma unroll
  for (int c = 0; c < K; ++c) {
    if (c * kThreads >= m) break;
    const int i = tid + c * kThreads;
    if (i < m) {
      x[c] = v.get(i);
      lo = x[c].k < lo ? x[c].k : lo;
      hi = x[c].k > hi ? x[c].k : hi;
    }
  }
  lo = warp_min(lo);
  hi = warp_max(hi);
  bool near = false;                     // does one of five other lanes have its first item within 1 / 4,096 of the warp's range?
  if (ALONE) {
    const int bits = 64 - __clzll((long long)(hi - lo));
    const uint32_t part = tid < m ? (uint32_t)((x[0].k - lo) >> (bits > 12 ? bits - 12 : 0)) : 1u << 31 | lane;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) near |= __shfl_xor_sync(0xffffffffu, part, o) == part;
  }
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  const int first_bits = m > 1 ? 32 - __clz(m - 1) : 0;
  int bins = 1 << first_bits;
  for (int i = tid * 4; i < bins; i += kThreads * 4) *(uint4*)(cnt + i) = make_uint4(0, 0, 0, 0);
  if (ALONE) {
    if (__syncthreads_count(near) * 32 > (m < kThreads ? m : kThreads)) return false;
  } else {
    __syncthreads();
  }
  lo = warp_min(s_lo[lane & (kWarps - 1)]);
  hi = warp_max(s_hi[lane & (kWarps - 1)]);
  {
    const int bits = 64 - __clzll((long long)(hi - lo)), below = bits > first_bits ? bits - first_bits : 0;
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c * kThreads >= m) break;
      bin[c] = tid + c * kThreads < m ? (uint32_t)((x[c].k - lo) >> below) | (uint32_t)below << 16 : 0u;
    }
  }
  uint32_t few = kSpreadFew;
  for (int level = 1;; ++level, few *= 2) {
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c * kThreads >= m) break;
      if (tid + c * kThreads < m) in[c] = atomicAdd(&cnt[bin[c] & 0xffffu], 1u);
    }
    __syncthreads();
    // items before every bin (upper half), and bins of the next level before its own (lower half)
    uint4 own[R];
    uint32_t upto[R];
    bool many = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r * kThreads * 4 >= bins) break;
      const int i = (r * kThreads + tid) * 4;
      uint4 w = make_uint4(0, 0, 0, 0);
      if (i < bins) {
        w = *(const uint4*)(cnt + i);
        uint32_t* const p = &w.x;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t n = i + u < bins ? p[u] : 0u;
          many |= n > few;
          p[u] = (n << 16) | (n > 1 ? 1u << (32 - __clz(n - 1)) : n);
        }
      }
      own[r] = w;
      upto[r] = warp_inclusive_scan(w.x + w.y + w.z + w.w, lane);
      if (lane == 31) s_sum[r][warp] = upto[r];
    }
    many = __syncthreads_or(many);
    if (many) {
      // (the counters are as they were: the starts are written below)
      if (level == kSpreadLevels) return false;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c * kThreads >= m) break;
        if (tid + c * kThreads < m && in[c] == 0) some[bin[c] & 0xffffu] = (uint16_t)(tid + c * kThreads);
      }
      __syncthreads();
      bool copy = false;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c * kThreads >= m) break;
        if (tid + c * kThreads < m && in[c] > 0 && cnt[bin[c] & 0xffffu] > few)
          copy |= key_of<WIDE>(x[c], pos_bits) == key_of<WIDE>(v.get(some[bin[c] & 0xffffu]), pos_bits);
      }
      if (__syncthreads_count(copy) > kSpreadCopies) return false;
    }
    uint32_t base = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r * kThreads * 4 >= bins) break;
      const uint32_t n = lane < kWarps ? s_sum[r][lane] : 0u, before = base + __reduce_add_sync(0xffffffffu, lane < warp ? n : 0u);
      base += __reduce_add_sync(0xffffffffu, n);
      const int i = (r * kThreads + tid) * 4;
      if (i < bins) {
        uint4 s;
        s.x = before + upto[r] - (own[r].x + own[r].y + own[r].z + own[r].w);
        s.y = s.x + own[r].x;
        s.z = s.y + own[r].y;
        s.w = s.z + own[r].z;
        *(uint4*)(cnt + i) = s;
      }
    }
    if (tid == 0) s_end = base;
    __syncthreads();
    const uint32_t end = s_end;
    if (!many) {
      uint32_t at[K], e[K];
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c * kThreads >= m) break;
        if (tid + c * kThreads < m) {
          const int j = (int)(bin[c] & 0xffffu);
          at[c] = cnt[j] >> 16;
          e[c] = (j + 1 < bins ? cnt[j + 1] : end) >> 16;
          v.set(at[c] + in[c], x[c]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c * kThreads >= m) break;
        if (tid + c * kThreads < m) {
          uint32_t to = at[c];
#pragma unroll 4
          for (uint32_t j = at[c]; j < e[c]; ++j) to += less<WIDE>(v.get(j), x[c]) ? 1u : 0u;
          at[c] = to;
        }
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < K; ++c) {
        if (c * kThreads >= m) break;
        if (tid + c * kThreads < m) v.set(at[c], x[c]);
      }
      __syncthreads();
      return true;
    }
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c * kThreads >= m) break;
      if (tid + c * kThreads < m) {
        const int j = (int)(bin[c] & 0xffffu), left = (int)(bin[c] >> 16);
        const uint32_t s = cnt[j], n = ((j + 1 < bins ? cnt[j + 1] : end) >> 16) - (s >> 16);
        const int want = n > 1 ? 32 - __clz(n - 1) : 0, take = want < left ? want : left;
        bin[c] = ((s & 0xffffu) + ((uint32_t)((x[c].k - lo) >> (left - take)) & ((1u << take) - 1u))) | (uint32_t)(left - take) << 16;
      }
    }
    bins = (int)(end & 0xffffu);
    __syncthreads();
    for (int i = tid * 4; i < bins; i += kThreads * 4) *(uint4*)(cnt + i) = make_uint4(0, 0, 0, 0);
    __syncthreads();
  }
}

// By counting up to MOST * kThreads items (0: not at all), otherwise, or where that gave up, by pivots: q grows with m so that ordering
// q pivots and ranking inside groups of m / q cost about the same (measured at 300, 600, 1,600, 2,200 and 7,000 items).
template <bool WIDE, int MOST, bool ALONE = false>
__device__ __forceinline__ void block_sort(const View<WIDE>& v, const View<WIDE>& tmp, uint32_t* aux, uint16_t* grp, int m, int pos_bits) {
  if (m < 64) {
    rank_sort<WIDE>(v, tmp, m);
    return;
  }
  if constexpr (MOST > 0) {
    if (m <= 4 * kThreads) {
      if (spread_sort<WIDE, 4, ALONE>(v, (uint32_t*)tmp.k, (uint16_t*)aux, m, pos_bits)) return;
    } else if (m <= MOST * kThreads) {
      if (spread_sort<WIDE, MOST, ALONE>(v, (uint32_t*)tmp.k, (uint16_t*)aux, m, pos_bits)) return;
    }
  }
  if (m >= 3072) group_sort<WIDE, 8>(v, tmp, aux, grp, m);
  else if (m >= 768) group_sort<WIDE, 7>(v, tmp, aux, grp, m);
  else group_sort<WIDE, 5>(v, tmp, aux, grp, m);
}
static_assert(kMaxItems < (1 << 21), "rank inside a group: 21 bits");

// What a Sink is:
//   kUnique = false   item(at, key, pos): the item at global position `at`
//                     between(at, key, has_prev, prev_key): `key` is the first at or behind position `at`, `prev_key` the last before
//                     it; called once per item, not always by the item's own CTA
//   kUnique = true    item(at, key, pos, head, u, head2, u2): `head` = first item of its group (equal sink.group(key)), `u` =
//                     number of the group; with kLevels = 2 the same for sink.group2(key), coarser than group.  Items with
//                     counted(key) = false (sorted behind the others) belong to no group.
//   begin()           called once per thread before the rest (loads device-side counts)
//   finish(n, last_key, has_last, groups, groups2)   once, by all threads of the CTA of the last bucket
//   kAfter / after()  by one thread after every CTA has delivered its items
// A Source: begin() loads device-side counts and returns the number of items; key(load(i)) is the key of item i.  load() only reads,
// so that the loads of several items are in flight together; what is wrong with an item is flagged by key().  kOnDemand: where on_demand()
// says so the list mostly turns out to be empty.

// What a bucket publishes for a sink that numbers groups, in ctl[1 + b] (0: not known yet): whether the item behind it starts a group
// / a coarser group, and the groups that start in it, its own first item aside (that is for the bucket before to say).
constexpr unsigned long long kKnown = 1, kNext1 = 2, kNext2 = 4;
__device__ __forceinline__ unsigned long long groups_of(unsigned long long pub) {      // coarser groups in the upper half
  return ((pub >> 8) & 0xffffffull) + (pub & kNext1 ? 1ull : 0ull) + ((pub >> 32) << 32) + (pub & kNext2 ? 1ull << 32 : 0ull);
}
static_assert(kMaxItems < (1 << 24), "groups of a bucket: 24 bits");

// The items of one CTA in sorted order -> the sink.  `base` = global position of the first; `b` / `last` = which bucket this is and
// whether it is the last one; `next_key` (not the last): the first key of the bucket behind it.  A bucket but the first begins with
// its splitter, so only the first can be empty.
template <class Sink, bool WIDE>
__device__ __forceinline__ void deliver(const Sink& sink, const View<WIDE>& v, int m, int64_t n, int64_t base, uint64_t next_key,
                                        int pos_bits, int b, bool last, unsigned long long* ctl, int32_t* d_status) {
  auto key_at = [&](int i) { return key_of<WIDE>(v.get(i), pos_bits); };
  if constexpr (!Sink::kUnique) {
    for (int i = threadIdx.x; i < m; i += kThreads) {
      const Item x = v.get(i);
      const uint64_t k = key_of<WIDE>(x, pos_bits);
      sink.item(base + i, k, pos_of<WIDE>(x, pos_bits));
      if (i > 0 || b == 0) sink.between(base + i, k, i > 0, i > 0 ? key_at(i - 1) : 0);
    }
    if (!last && threadIdx.x == 0) sink.between(base + m, next_key, m > 0, m > 0 ? key_at(m - 1) : 0);
    if (last) sink.finish(n, m > 0 ? key_at(m - 1) : 0, m > 0, 0, 0);
  } else {
    constexpr bool kTwo = Sink::kLevels == 2;
    __shared__ unsigned long long s_warp[kWarps], s_before[kWarps];
    __shared__ int s_head;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // groups that start between two neighbours: bit 0, coarser groups: bit 1
    auto heads = [&](uint64_t p, uint64_t k) -> int {
      if (!sink.counted(k)) return 0;
      int h = sink.group(p) != sink.group(k) ? 1 : 0;
      if constexpr (kTwo) h |= sink.group2(p) != sink.group2(k) ? 2 : 0;
      return h;
    };
    auto first_heads = [&](uint64_t k) -> int { return sink.counted(k) ? (kTwo ? 3 : 1) : 0; };
    // a warp takes consecutive items; their groups are counted, published, and those of the buckets before added up
    const int span = ((m + kWarps * 32 - 1) / (kWarps * 32)) * 32, from = warp * span, to = from + span < m ? from + span : m;
    unsigned long long own = 0;
    for (int i0 = from; i0 < to; i0 += 32) {
      const int i = i0 + lane, h = i > 0 && i < to ? heads(key_at(i - 1), key_at(i)) : 0;
      own += (unsigned long long)__popc(__ballot_sync(0xffffffffu, h & 1));
      if (kTwo) own += (unsigned long long)__popc(__ballot_sync(0xffffffffu, h & 2)) << 32;
    }
    if (lane == 0) s_warp[warp] = own;
    if (threadIdx.x == 0) s_head = b == 0 && m > 0 ? first_heads(key_at(0)) : 0;
    __syncthreads();
    // (two counts below 2^32 each, summed apart)
    auto sum = [](unsigned long long x) -> unsigned long long {
      const unsigned lower = __reduce_add_sync(0xffffffffu, (unsigned)x);
      return (unsigned long long)lower | (kTwo ? (unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)(x >> 32)) << 32 : 0ull);
    };
    const unsigned long long share = lane < kWarps ? s_warp[lane] : 0;
    const unsigned long long total = sum(share);
    unsigned long long off = sum(lane < warp ? share : 0), others = 0;
    if (ctl != nullptr) {
      volatile unsigned long long* pub = ctl + 1;
      if (threadIdx.x == 0) {
        const int next = last ? 0 : (m > 0 ? heads(key_at(m - 1), next_key) : first_heads(next_key));
        const int first = b == 0 ? s_head : 0;       // (nobody before bucket 0 counts its first item)
        pub[b] = kKnown | (next & 1 ? kNext1 : 0) | (next & 2 ? kNext2 : 0) | (((total & 0xffffffffull) + (first & 1)) << 8) |
                 ((total >> 32) + (unsigned long long)(first >> 1)) << 32;
      }
      // lower buckets have taken their ticket before this one: their CTAs are running and wait only for still lower ones
      unsigned long long before = 0;
      for (int t = threadIdx.x; t < b; t += kThreads) {
        unsigned long long c = pub[t];
        // (the clock is read now and then only: a read takes longer than a poll)
        unsigned long long t0 = 0;
        for (unsigned spin = 1; c == 0; ++spin) {
          c = pub[t];
          if ((spin & 63u) != 0 || c != 0) continue;
          unsigned long long now;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (t0 == 0) t0 = now;
          if (now - t0 > kWaitNs) {
            dev_flag(d_status, SGL_DEV_TIMEOUT);
            break;
          }
        }
        before += groups_of(c);
        if (t == b - 1) s_head = (c & kNext1 ? 1 : 0) | (c & kNext2 ? 2 : 0);
      }
      before = sum(before);
      if (lane == 0) s_before[warp] = before;
      __syncthreads();
      others = sum(lane < kWarps ? s_before[lane] : 0);
      off += others;
    }
    // groups that start before the warp's first item: the bucket's first item is counted with the buckets before (b > 0)
    const int head0 = s_head;
    if (b == 0 ? warp > 0 : warp == 0) {
      const unsigned long long h = (unsigned long long)(head0 & 1) | ((unsigned long long)(head0 >> 1) << 32);
      if (b == 0) off += h; else off -= h;
    }
    for (int i0 = from; i0 < to; i0 += 32) {
      const int i = i0 + lane;
      int h = 0;
      Item x{0, 0};
      uint64_t k = 0;
      if (i < to) {
        x = v.get(i);
        k = key_of<WIDE>(x, pos_bits);
        h = i > 0 ? heads(key_at(i - 1), k) : head0;
      }
      const unsigned b1 = __ballot_sync(0xffffffffu, h & 1), b2 = kTwo ? __ballot_sync(0xffffffffu, h & 2) : 0u;
      if (i < to) {
        const unsigned upto = (2u << lane) - 1u;
        const int64_t u = (int64_t)(off & 0xffffffffull) + __popc(b1 & upto) - 1, u2 = (int64_t)(off >> 32) + __popc(b2 & upto) - 1;
        sink.item(base + i, k, pos_of<WIDE>(x, pos_bits), h & 1, u, h >> 1, u2);
      }
      off += (unsigned long long)__popc(b1) | ((unsigned long long)__popc(b2) << 32);
    }
    if (last) {
      // all groups: those before the bucket, and its own
      unsigned long long all = total + others;
      if (b == 0) all += (unsigned long long)(head0 & 1) | ((unsigned long long)(head0 >> 1) << 32);
      sink.finish(n, 0, false, (int64_t)(all & 0xffffffffull), (int64_t)(all >> 32));
    }
  }
}

// after(): once every CTA of the launch has delivered
template <class Sink>
__device__ __forceinline__ void arrive(const Sink& sink, unsigned long long* counter, int ctas) {
  if constexpr (Sink::kAfter) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (counter == nullptr || atomicAdd(counter, 1ull) == (unsigned long long)(ctas - 1)) {
        __threadfence();
        sink.after();
      }
    }
  }
}

// Tile size for n items on at most `ctas` CTAs: an even share, so that the list spreads over all SMs.
__host__ __device__ inline int tile_for(int64_t n, int ctas) {
  const int t = (int)(((uint32_t)n + (uint32_t)ctas - 1u) / (uint32_t)ctas);       // (lists are below 2^21)
  return t < kMinTile ? kMinTile : (t + 31) & ~31;
}

// Scratch of one sort (device pointers), see carve().
struct Scratch {
  uint64_t* tile_k;     // [n] items grouped by bucket inside every tile
  uint32_t* tile_p;     // [n] (WIDE)
  int32_t* start;       // [bucket][tile] where the bucket's piece starts inside the tile; row `tiles` = the tile's end
  uint64_t* split;      // [bucket] smallest key of the bucket (of all but the first)
  uint64_t* over_k;     // [2][n] buckets that do not fit shared memory
  uint32_t* over_p;     // [2][n] (WIDE)
  uint32_t* over_a;     // [n]
  uint16_t* over_g;     // [n]
  unsigned long long* ctl;   // [0] ticket, [1 + b] what bucket b has published, [kCtlWords - 1] arrivals
};

constexpr int kCtlWords = kMaxCtas + 3;
constexpr int kMatrix = (kMaxCtas + 1) * kMaxCtas;

inline size_t ws_bytes(int64_t n) {
  if (n < 1) n = 1;
  return align_up((size_t)n * 8) + align_up((size_t)n * 4) + align_up(kMatrix * 4) + align_up(kMaxCtas * 8) + align_up((size_t)n * 16) +
         align_up((size_t)n * 8) + align_up((size_t)n * 4) + align_up((size_t)n * 2) + align_up(kCtlWords * 8);
}

inline Scratch carve(WsCarver& c, int64_t n) {
  Scratch s;
  s.tile_k = c.take<uint64_t>(n);
  s.tile_p = c.take<uint32_t>(n);
  s.start = c.take<int32_t>(kMatrix);
  s.split = c.take<uint64_t>(kMaxCtas);
  s.over_k = c.take<uint64_t>(2 * (size_t)n);
  s.over_p = c.take<uint32_t>(2 * (size_t)n);
  s.over_a = c.take<uint32_t>(n);
  s.over_g = c.take<uint16_t>(n);
  s.ctl = c.take<unsigned long long>(kCtlWords);
  return s;
}

// block_sort's arrays for `cap` items in dynamic shared memory
template <bool WIDE>
struct Arrays {
  View<WIDE> v, tmp;
  uint32_t* aux;
  uint16_t* grp;
  static constexpr size_t bytes(int cap) { return (size_t)cap * (2 * (WIDE ? 12 : 8) + 4 + 2); }
  __device__ __forceinline__ Arrays(unsigned char* smem, int cap) {
    uint64_t* k = (uint64_t*)smem;
    aux = (uint32_t*)(k + 2 * cap);
    uint32_t* p = aux + cap;
    v = View<WIDE>{k, p};
    tmp = View<WIDE>{k + cap, p + cap};
    grp = (uint16_t*)(WIDE ? p + 2 * cap : p);
  }
};

// Tile [first, first + m) of K * kThreads items at most.  What a part costs is largely its instructions, fetched once each: those of
// item slots that no thread of a mini-batch has are jumped over.
template <class Source, bool WIDE, int K>
__device__ __forceinline__ void part_tile(const Source& src, int pos_bits, const Scratch& sc, int64_t n, int64_t first, int m, int tiles,
                                          const Arrays<WIDE>& sm) {
  constexpr int kBatch = 4;              // items of a thread whose loads, and searches, run side by side
  constexpr int kSplit = 256;            // splitters, filled up with largest words
  static_assert(kMaxCtas <= kSplit && K % kBatch == 0, "eight steps of the search");
  __shared__ int s_cnt[kMaxCtas], s_w[kWarps];
  __shared__ uint64_t s_split_k[kSplit];
  __shared__ uint32_t s_split_p[WIDE ? kSplit : 1];
  const View<WIDE> split{s_split_k, s_split_p};      // splitter b (b = 1 .. tiles - 1) at split[b - 1]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int buckets = tiles;             // one bucket per tile (two smaller ones were slower)
  // Samples: sorting more costs more, fewer leave larger buckets.  Measured with 148 buckets (512, 1,024, 2,048 samples): 41,000 pairs
  // 17, 20, - us; 100,000 19.5, 21.6, -; 144,000 24.4, 23.6, 30; 200,000 -, 26.3, 26.7 - 34; 300,000 -, 41, 34.6.  Buckets of 3.5 samples
  // are at most about four times the mean, of 14 about 1.7 times.  (With more than one tile the sample is smaller than the list.)
  const int sb = tiles <= 8 ? 8 : (n < 100000 ? 9 : (n < 220000 ? 10 : 11)), s = tiles > 1 ? 1 << sb : 0;
  typename Source::Raw sample[kMaxSamples / kThreads];
#pragma unroll
  for (int r = 0; r < kMaxSamples / kThreads; ++r) {
    if (r * kThreads >= s) break;        // (s is at least half the number of threads)
    sample[r] = src.load(sample_at((tid + r * kThreads) & (s - 1), sb, (int)n));
  }
  Item x[K];
#pragma unroll
  for (int r0 = 0; r0 < K; r0 += kBatch) {
    if (r0 * kThreads >= m) break;
    typename Source::Raw raw[kBatch];
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      if ((r0 + r) * kThreads >= m) break;
      const int i = tid + (r0 + r) * kThreads;
      raw[r] = src.load(first + (i < m ? i : m - 1));      // (no branch around a load)
    }
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      if ((r0 + r) * kThreads >= m) break;
      const int i = tid + (r0 + r) * kThreads;
      if (i < m) x[r0 + r] = make_item<WIDE>(src.key(raw[r]), (uint32_t)(first + i), pos_bits);
    }
  }
#pragma unroll
  for (int r = 0; r < kMaxSamples / kThreads; ++r) {
    if (r * kThreads >= s) break;
    const int j = tid + r * kThreads;
    if (j < s) sm.v.set(j, make_item<WIDE>(src.key(sample[r]), (uint32_t)sample_at(j, sb, (int)n), pos_bits));
  }
  if (tid < buckets) s_cnt[tid] = 0;
  if (tiles > 1) {
    block_sort<WIDE, 0>(sm.v, sm.tmp, sm.aux, sm.grp, s, pos_bits);
    if (tid < kSplit) {
      const Item none{~0ull, ~0u};
      split.set(tid, tid + 1 < buckets ? sm.v.get((int)((uint32_t)((tid + 1) * s) / (uint32_t)buckets)) : none);
      if (blockIdx.x == 0 && tid + 1 < buckets) sc.split[tid + 1] = key_of<WIDE>(split.get(tid), pos_bits);
    }
  }
  __syncthreads();
  int bucket[K], at[K];
#pragma unroll
  for (int r0 = 0; r0 < K; r0 += kBatch) {
    if (r0 * kThreads >= m) break;
    int lo[kBatch];
#pragma unroll
    for (int r = 0; r < kBatch; ++r) lo[r] = 0;
    if (tiles > 1) {
      // number of splitters that are not greater (the words that fill up count where an item is all ones: none of them is a bucket)
#pragma unroll 1
      for (int h = kSplit / 2; h >= 1; h >>= 1) {
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
          if ((r0 + r) * kThreads >= m) break;
          lo[r] += less<WIDE>(x[r0 + r], split.get(lo[r] + h - 1)) ? 0 : h;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      if ((r0 + r) * kThreads >= m) break;
      if (tid + (r0 + r) * kThreads < m) {
        const int bk = lo[r] < buckets ? lo[r] : buckets - 1;
        bucket[r0 + r] = bk;
        at[r0 + r] = atomicAdd(&s_cnt[bk], 1);
      }
    }
  }
  __syncthreads();
  const int c = tid < buckets ? s_cnt[tid] : 0;
  int off = warp_inclusive_scan(c, lane);
  if (lane == 31) s_w[warp] = off;
  __syncthreads();
  off += __reduce_add_sync(0xffffffffu, lane < warp && lane < kWarps ? s_w[lane] : 0) - c;
  if (tid < buckets) {
    s_cnt[tid] = off;
    sc.start[tid * tiles + blockIdx.x] = off;
  }
  if (tid == 0) sc.start[buckets * tiles + blockIdx.x] = m;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < K; ++r) {
    if (r * kThreads >= m) break;
    if (tid + r * kThreads < m) View<WIDE>{sc.tile_k, sc.tile_p}.set((int)first + s_cnt[bucket[r]] + at[r], x[r]);
  }
}

template <class Source, bool WIDE>
__global__ void __launch_bounds__(kRegThreads)
ts_part_kernel(Source src, int pos_bits, Scratch sc) {
  extern __shared__ __align__(16) unsigned char smem_ts[];
  const int64_t n = src.begin();
  const int tile = tile_for(n, (int)gridDim.x);
  const int tiles = (int)(((uint32_t)n + (uint32_t)tile - 1u) / (uint32_t)tile);
  if (blockIdx.x == 0)
    for (int t = threadIdx.x; t < kCtlWords; t += kThreads) sc.ctl[t] = 0;
  const int64_t first = (int64_t)blockIdx.x * tile;
  if (first >= n) return;
  const int m = (int)(n - first < tile ? n - first : tile);
  const Arrays<WIDE> sm(smem_ts, kMaxSamples);
  if (m <= 4 * kThreads) part_tile<Source, WIDE, 4>(src, pos_bits, sc, n, first, m, tiles, sm);
  else part_tile<Source, WIDE, kTileItems>(src, pos_bits, sc, n, first, m, tiles, sm);
}

// cap = items that fit this launch's shared memory
template <class Source, class Sink, bool WIDE>
__global__ void __launch_bounds__(kRegThreads)
ts_bucket_kernel(Source src, Sink sink, int pos_bits, int64_t n_cap, Scratch sc, int cap, int32_t* d_status) {
  extern __shared__ __align__(16) unsigned char smem_ts[];
  __shared__ int s_ticket;
  __shared__ int s_at[kMaxCtas + 1];
  __shared__ int s_from[kMaxCtas];
  __shared__ int s_w[kWarps];
  __shared__ int s_sum[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // (every CTA takes a ticket, next to the loads of begin(); those beyond the number of buckets leave)
  if (tid == 0) s_ticket = Sink::kUnique ? (int)atomicAdd(sc.ctl, 1ull) : (int)blockIdx.x;
  const int64_t n = src.begin();
  sink.begin();
  __syncthreads();
  const int b = s_ticket;
  if (n <= 0) {
    if (b == 0) {
      sink.finish(0, 0, false, 0, 0);
      arrive(sink, nullptr, 1);
    }
    return;
  }
  const int tile = tile_for(n, (int)gridDim.x);
  const int tiles = (int)(((uint32_t)n + (uint32_t)tile - 1u) / (uint32_t)tile);
  const int buckets = tiles;             // one bucket per tile (two smaller ones were slower)
  if (b >= buckets) return;
  const uint64_t next_key = b + 1 < buckets ? sc.split[b + 1] : 0;
  // thread t: the bucket's piece of tile t
  int lo = 0, len = 0;
  if (tid < tiles) {
    lo = sc.start[b * tiles + tid];
    len = sc.start[(b + 1) * tiles + tid] - lo;
  }
  const int off = warp_inclusive_scan(len, lane);
  const int before = (int)__reduce_add_sync(0xffffffffu, (unsigned)lo);
  if (lane == 31) s_w[warp] = off;
  if (lane == 0) s_sum[warp] = before;
  __syncthreads();
  const int share_w = lane < kWarps ? s_w[lane] : 0, woff = __reduce_add_sync(0xffffffffu, lane < warp ? share_w : 0);
  const int m = __reduce_add_sync(0xffffffffu, share_w);
  const int64_t base = __reduce_add_sync(0xffffffffu, lane < kWarps ? s_sum[lane] : 0);
  if (tid < tiles) {
    s_at[tid] = woff + off - len;
    s_from[tid] = tid * tile + lo - (woff + off - len);
  }
  if (tid == 0) s_at[tiles] = m;
  __syncthreads();
  const View<WIDE> from{sc.tile_k, sc.tile_p};
  // a few lanes copy one piece, all pieces at once (148 tiles of 1,000: about seven items a piece, two lanes)
  const int share = tiles > kThreads / 4 ? 1 : (tiles > kThreads / 8 ? 2 : (tiles > kThreads / 16 ? 3 : 4));
  auto collect = [&](const View<WIDE>& v) {
    const int a = tid >> share;
    if (a < tiles) {
      const int e = s_at[a + 1], f = s_from[a];
#pragma unroll 8
      for (int i = s_at[a] + (tid & ((1 << share) - 1)); i < e; i += 1 << share) v.set(i, from.get(f + i));
    }
  };
  const bool last = b == buckets - 1;
  if (m <= cap) {
    const Arrays<WIDE> sm(smem_ts, cap);
    collect(sm.v);
    block_sort<WIDE, 8>(sm.v, sm.tmp, sm.aux, sm.grp, m, pos_bits);
    deliver<Sink, WIDE>(sink, sm.v, m, n, base, next_key, pos_bits, b, last, sc.ctl, d_status);
  } else {
    // a bucket that shared memory does not hold (unevenly spread sample) is sorted in global memory
    const View<WIDE> v{sc.over_k + base, sc.over_p + base}, tmp{sc.over_k + n_cap + base, sc.over_p + n_cap + base};
    collect(v);
    block_sort<WIDE, 0>(v, tmp, sc.over_a + base, sc.over_g + base, m, pos_bits);
    deliver<Sink, WIDE>(sink, v, m, n, base, next_key, pos_bits, b, last, sc.ctl, d_status);
  }
  arrive(sink, sc.ctl + kCtlWords - 1, buckets);
}

template <class Source, class Sink, bool WIDE>
__global__ void __launch_bounds__(kRegThreads)
ts_single_kernel(Source src, Sink sink, int pos_bits, int32_t* d_status) {
  extern __shared__ __align__(16) unsigned char smem_ts[];
  const int m = (int)src.begin();
  sink.begin();
  const Arrays<WIDE> sm(smem_ts, kSingleMax);
  for (int i = threadIdx.x; i < m; i += kThreads) {
    sm.v.set(i, make_item<WIDE>(src.key(src.load(i)), (uint32_t)i, pos_bits));
  }
  block_sort<WIDE, kSingleMax / kThreads, true>(sm.v, sm.tmp, sm.aux, sm.grp, m, pos_bits);
  deliver<Sink, WIDE>(sink, sm.v, m, m, 0, 0, pos_bits, 0, true, nullptr, d_status);
  arrive(sink, nullptr, 1);
}

inline int launches(int64_t n_cap) { return n_cap <= 0 ? 0 : (n_cap <= kSingleMax ? 1 : 2); }

template <class Source, class Sink, bool WIDE>
int launch_as(const Source& src, const Sink& sink, int64_t n_cap, int pos_bits, const Scratch& sc, int32_t* d_status,
              cudaStream_t stream) {
  static std::atomic<uint64_t> single_done{0}, bucket_done{0}, part_done{0};
  if (n_cap <= kSingleMax) {
    constexpr size_t smem = Arrays<WIDE>::bytes(kSingleMax);
    SGL_CUDA_CHECK(allow_smem((const void*)ts_single_kernel<Source, Sink, WIDE>, single_done, smem));
    SGL_CHECK_RC(launch(ts_single_kernel<Source, Sink, WIDE>, 1, kThreads, smem, stream, src, sink, pos_bits, d_status));
    return SGL_OK;
  }
  const int64_t min_tiles = (n_cap + kMinTile - 1) / kMinTile;
  const int ctas = (int)(min_tiles < kMaxCtas ? min_tiles : kMaxCtas);
  const int tile = tile_for(n_cap, ctas);
  // a bucket is about a tile, up to twice that, and with few samples per bucket (more than 64 of them) up to five times; what does
  // not fit goes through global memory
  constexpr int kCapMost = WIDE ? 6912 : 9216;
  const int room = (ctas > 64 ? 8 : 4) * tile, cap = room < kCapMost ? room : kCapMost;
  SGL_CUDA_CHECK(allow_smem((const void*)ts_bucket_kernel<Source, Sink, WIDE>, bucket_done, Arrays<WIDE>::bytes(kCapMost)));
  SGL_CUDA_CHECK(allow_smem((const void*)ts_part_kernel<Source, WIDE>, part_done, Arrays<WIDE>::bytes(kMaxSamples)));
  SGL_CHECK_RC(launch(ts_part_kernel<Source, WIDE>, ctas, kThreads, Arrays<WIDE>::bytes(kMaxSamples), stream,
                      src, pos_bits, sc));
  SGL_CHECK_RC(launch(ts_bucket_kernel<Source, Sink, WIDE>, ctas, kThreads, Arrays<WIDE>::bytes(cap), stream, src, sink,
                      pos_bits, n_cap, sc, cap, d_status));
  return SGL_OK;
}

// Sorts the items of `src` (at most n_cap <= kMaxItems, keys of key_bits bits) and delivers them to `sink`.
template <class Source, class Sink>
int launch(const Source& src, const Sink& sink, int64_t n_cap, int key_bits, const Scratch& sc, int32_t* d_status,
           cudaStream_t stream) {
  int pos_bits = 0;
  while (((n_cap - 1) >> pos_bits) != 0) ++pos_bits;
  return key_bits + pos_bits > 64 ? launch_as<Source, Sink, true>(src, sink, n_cap, pos_bits, sc, d_status, stream)
                                  : launch_as<Source, Sink, false>(src, sink, n_cap, pos_bits, sc, d_status, stream);
}

}  // namespace tilesort
}  // namespace sgl
