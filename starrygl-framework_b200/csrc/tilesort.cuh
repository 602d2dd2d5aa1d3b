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
// Measured (44-bit keys): 4,096 keys 14 us, 41,000 20 us, 160,000 29 us, 480,000 61 us; an LSD radix sort with one kernel
// per 11 key bits took 25, 84, 95 and 140 us: few CTAs with large digit tables, and a dependent kernel per digit.
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

// Number of the `cnt` ascending items of v that are not greater than x.  The first step counts against every 2^step-th item,
// which all lanes read at the same address; only the last few probes differ between lanes (a plain binary search is bound
// by the bank conflicts of its middle levels).  1 << step = about cnt / 16.
template <bool WIDE>
__device__ __forceinline__ int not_above(const View<WIDE>& v, int cnt, int step, const Item& x) {
  int lo = 0;
#pragma unroll 4
  for (int i = (1 << step) - 1; i < cnt; i += 1 << step) lo += less<WIDE>(x, v.get(i)) ? 0 : 1;
  lo <<= step;
  int hi = lo + (1 << step) - 1;         // item hi is greater than x, or does not exist
  if (hi > cnt) hi = cnt;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (less<WIDE>(x, v.get(mid))) hi = mid; else lo = mid + 1;
  }
  return lo;
}
__device__ __forceinline__ int step_for(int cnt) {
  int s = 0;
  while ((16 << s) < cnt) ++s;
  return s;
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
#pragma unroll
    for (int w = 0; w < (Q + 32) / 32; ++w)
      if (w < warp) x += s_wsum[w];
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

// q grows with m so that ordering q pivots and ranking inside groups of m / q cost about the same (measured at 300, 600,
// 1,600, 2,200 and 7,000 items).
template <bool WIDE>
__device__ __forceinline__ void block_sort(const View<WIDE>& v, const View<WIDE>& tmp, uint32_t* aux, uint16_t* grp, int m) {
  if (m >= 3072) group_sort<WIDE, 8>(v, tmp, aux, grp, m);
  else if (m >= 768) group_sort<WIDE, 7>(v, tmp, aux, grp, m);
  else if (m >= 64) group_sort<WIDE, 5>(v, tmp, aux, grp, m);
  else rank_sort<WIDE>(v, tmp, m);
}
static_assert(kMaxItems < (1 << 21), "rank inside a group: 21 bits");

// What a Sink is:
//   kUnique = false   item(at, key, pos, has_prev, prev_key): the item at global position `at`, and the key before it
//   kUnique = true    item(at, key, pos, head, u, head2, u2): `head` = first item of its group (equal sink.group(key)), `u` =
//                     number of the group; with kLevels = 2 the same for sink.group2(key), coarser than group.  Items with
//                     counted(key) = false (sorted behind the others) belong to no group.
//   kPred             needs the key before a bucket's first item (prev_key, head)
//   begin()           called once per thread before the rest (loads device-side counts)
//   finish(n, last_key, has_last, groups, groups2)   once, by all threads of the CTA of the last bucket
//   kAfter / after()  by one thread after every CTA has delivered its items
// A Source: begin() loads device-side counts and returns the number of items; key(i); prepare(i) is called for every i in
// [0, n) before any item is delivered.

// The items of one CTA in sorted order -> the sink.  `base` = global position of the first, `pred_key` = the key before it
// (when has_pred), `b` / `last` = which bucket this is and whether it is the last one.
template <class Sink, bool WIDE>
__device__ __forceinline__ void deliver(const Sink& sink, const View<WIDE>& v, int m, int64_t n, int64_t base, uint64_t pred_key,
                                        bool has_pred, int pos_bits, int b, bool last, unsigned long long* ctl, int32_t* d_status) {
  if constexpr (!Sink::kUnique) {
    for (int i = threadIdx.x; i < m; i += kThreads) {
      const Item x = v.get(i);
      const bool hp = i > 0 || has_pred;
      const uint64_t pk = i > 0 ? key_of<WIDE>(v.get(i - 1), pos_bits) : pred_key;
      sink.item(base + i, key_of<WIDE>(x, pos_bits), pos_of<WIDE>(x, pos_bits), hp, pk);
    }
    if (last) sink.finish(n, m > 0 ? key_of<WIDE>(v.get(m - 1), pos_bits) : pred_key, m > 0 || has_pred, 0, 0);
  } else {
    constexpr bool kTwo = Sink::kLevels == 2;
    __shared__ unsigned long long s_warp[kWarps];
    __shared__ unsigned long long s_base;
    // heads of item i: bit 0 of its group, bit 32 of its coarser group
    auto heads_of = [&](int i) -> unsigned long long {
      const uint64_t k = key_of<WIDE>(v.get(i), pos_bits);
      if (!sink.counted(k)) return 0;
      if (i == 0 && !has_pred) return kTwo ? 0x100000001ull : 1ull;
      const uint64_t p = i > 0 ? key_of<WIDE>(v.get(i - 1), pos_bits) : pred_key;
      unsigned long long h = sink.group(p) != sink.group(k) ? 1ull : 0ull;
      if constexpr (kTwo) h |= sink.group2(p) != sink.group2(k) ? 0x100000000ull : 0ull;
      return h;
    };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto cta_sum = [&](unsigned long long x) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      __syncthreads();
      if (lane == 0) s_warp[warp] = x;
      __syncthreads();
      x = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) x += s_warp[w];
      return x;
    };
    // heads of the bucket -> published; the numbers of the earlier buckets are summed up by one thread each
    unsigned long long heads = 0, before = 0;
    for (int i = threadIdx.x; i < m; i += kThreads) heads += heads_of(i);
    heads = cta_sum(heads);
    if (ctl != nullptr) {
      volatile unsigned long long* pub = ctl + 1;
      if (threadIdx.x == 0) pub[b] = heads + 1ull;
      // lower buckets have taken their ticket before this one: their CTAs are running and wait only for still lower ones
      for (int t = threadIdx.x; t < b; t += kThreads) {
        unsigned long long c = pub[t];
        if (c == 0) {
          unsigned long long t0, t1;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
          do {
            c = pub[t];
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
          } while (c == 0 && t1 - t0 < kWaitNs);
          if (c == 0) {
            dev_flag(d_status, SGL_DEV_TIMEOUT);
            c = 1;
          }
        }
        before += c - 1ull;
      }
      before = cta_sum(before);
    }
    if (threadIdx.x == 0) s_base = before;
    __syncthreads();
    for (int i0 = 0; i0 < m; i0 += kThreads) {
      const int i = i0 + threadIdx.x;
      const unsigned long long h = i < m ? heads_of(i) : 0ull;
      const unsigned b1 = __ballot_sync(0xffffffffu, (h & 1ull) != 0), b2 = kTwo ? __ballot_sync(0xffffffffu, (h >> 32) != 0) : 0u;
      if (lane == 0) s_warp[warp] = (unsigned long long)__popc(b1) | ((unsigned long long)__popc(b2) << 32);
      __syncthreads();
      unsigned long long off = s_base, tot = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const unsigned long long c = s_warp[w];
        if (w < warp) off += c;
        tot += c;
      }
      __syncthreads();
      if (threadIdx.x == 0) s_base += tot;
      if (i < m) {
        const Item x = v.get(i);
        const unsigned upto = (2u << lane) - 1u;
        const int64_t u = (int64_t)(off & 0xffffffffull) + __popc(b1 & upto) - 1, u2 = (int64_t)(off >> 32) + __popc(b2 & upto) - 1;
        sink.item(base + i, key_of<WIDE>(x, pos_bits), pos_of<WIDE>(x, pos_bits), (h & 1ull) != 0, u, (h >> 32) != 0, u2);
      }
      __syncthreads();
    }
    if (last) sink.finish(n, 0, false, (int64_t)((before + heads) & 0xffffffffull), (int64_t)((before + heads) >> 32));
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
  const int t = (int)((n + ctas - 1) / ctas);
  return t < kMinTile ? kMinTile : (t + 31) & ~31;
}

// Scratch of one sort (device pointers), see carve().
struct Scratch {
  uint64_t* tile_k;     // [n] items grouped by bucket inside every tile
  uint32_t* tile_p;     // [n] (WIDE)
  int32_t* start;       // [bucket][tile] where the bucket's piece starts inside the tile; row `tiles` = the tile's end
  uint64_t* top;        // [bucket][tile] largest key of the piece (0 where it is empty)
  uint64_t* over_k;     // [2][n] buckets that do not fit shared memory
  uint32_t* over_p;     // [2][n] (WIDE)
  uint32_t* over_a;     // [n]
  uint16_t* over_g;     // [n]
  unsigned long long* ctl;   // [0] ticket, [1 + b] groups of bucket b plus one (0 = not known yet), [kCtlWords - 1] arrivals
};

constexpr int kCtlWords = kMaxCtas + 3;
constexpr int kMatrix = (kMaxCtas + 1) * kMaxCtas;

inline size_t ws_bytes(int64_t n) {
  if (n < 1) n = 1;
  return align_up((size_t)n * 8) + align_up((size_t)n * 4) + align_up(kMatrix * 4) + align_up(kMatrix * 8) + align_up((size_t)n * 16) +
         align_up((size_t)n * 8) + align_up((size_t)n * 4) + align_up((size_t)n * 2) + align_up(kCtlWords * 8);
}

inline Scratch carve(WsCarver& c, int64_t n) {
  Scratch s;
  s.tile_k = c.take<uint64_t>(n);
  s.tile_p = c.take<uint32_t>(n);
  s.start = c.take<int32_t>(kMatrix);
  s.top = c.take<uint64_t>(kMatrix);
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

template <class Source, bool WIDE, bool TOP>
__global__ void __launch_bounds__(kThreads)
ts_part_kernel(Source src, int pos_bits, Scratch sc) {
  extern __shared__ __align__(16) unsigned char smem_ts[];
  __shared__ int s_cnt[kMaxCtas], s_w[kWarps];
  __shared__ unsigned long long s_top[kMaxCtas];
  const int64_t n = src.begin();
  const int tile = tile_for(n, (int)gridDim.x);
  const int tiles = (int)((n + tile - 1) / tile);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.x == 0)
    for (int t = tid; t < kCtlWords; t += kThreads) sc.ctl[t] = 0;
  const int64_t first = (int64_t)blockIdx.x * tile;
  if (first >= n) return;
  const int m = (int)(n - first < tile ? n - first : tile);
  Item x[kTileItems];
#pragma unroll
  for (int r = 0; r < kTileItems; ++r) {
    const int i = tid + r * kThreads;
    x[r] = i < m ? make_item<WIDE>(src.key(first + i), (uint32_t)(first + i), pos_bits) : Item{0, 0};
    if (i < m) src.prepare(first + i);
  }
  const Arrays<WIDE> sm(smem_ts, kMaxSamples);
  const View<WIDE> split = sm.tmp;       // splitter b (b = 1 .. tiles - 1) at split[b - 1]
  const int buckets = tiles;             // one bucket per tile (two smaller ones were slower)
  if (tiles > 1) {
    // (more than one tile: n is above (tiles - 1) * 256, the sample is smaller than the list)
    // Samples: sorting more costs more, fewer leave larger buckets.  Measured with 148 buckets (512, 1,024, 2,048 samples): 60,000
    // keys 29, 31, 35 us; 144,000 keys 41, 37, 41 us; 300,000 keys (57), 57, 53 us.  Buckets of 3.5 samples are at most about
    // four times the mean, of 14 about 1.7 times.
    const int sb = tiles <= 8 ? 8 : (n < 70000 ? 9 : (n < 220000 ? 10 : 11)), s = 1 << sb;
    for (int j = tid; j < s; j += kThreads) {
      const int i = sample_at(j, sb, (int)n);
      sm.v.set(j, make_item<WIDE>(src.key(i), (uint32_t)i, pos_bits));
    }
    block_sort<WIDE>(sm.v, sm.tmp, sm.aux, sm.grp, s);
    for (int b = 1 + tid; b < buckets; b += kThreads) split.set(b - 1, sm.v.get(b * s / buckets));
  }
  const int step = step_for(buckets - 1);
  for (int b = tid; b < buckets; b += kThreads) {
    s_cnt[b] = 0;
    s_top[b] = 0;
  }
  __syncthreads();
  int bucket[kTileItems], at[kTileItems];
#pragma unroll
  for (int r = 0; r < kTileItems; ++r) {
    bucket[r] = at[r] = 0;
    if (tid + r * kThreads < m) {
      bucket[r] = not_above<WIDE>(split, buckets - 1, step, x[r]);
      at[r] = atomicAdd(&s_cnt[bucket[r]], 1);
      if (TOP) atomicMax(&s_top[bucket[r]], (unsigned long long)key_of<WIDE>(x[r], pos_bits));
    }
  }
  __syncthreads();
  const int c = tid < buckets ? s_cnt[tid] : 0;
  int off = warp_inclusive_scan(c, lane);
  if (lane == 31) s_w[warp] = off;
  __syncthreads();
  for (int w = 0; w < warp; ++w) off += s_w[w];
  off -= c;
  if (tid < buckets) {
    s_cnt[tid] = off;
    sc.start[tid * tiles + blockIdx.x] = off;
    if (TOP) sc.top[tid * tiles + blockIdx.x] = s_top[tid];
  }
  if (tid == 0) sc.start[buckets * tiles + blockIdx.x] = m;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kTileItems; ++r)
    if (tid + r * kThreads < m) View<WIDE>{sc.tile_k, sc.tile_p}.set((int)first + s_cnt[bucket[r]] + at[r], x[r]);
}

// cap = items that fit this launch's shared memory
template <class Source, class Sink, bool WIDE>
__global__ void __launch_bounds__(kThreads)
ts_bucket_kernel(Source src, Sink sink, int pos_bits, int64_t n_cap, Scratch sc, int cap, int32_t* d_status) {
  extern __shared__ __align__(16) unsigned char smem_ts[];
  __shared__ int s_ticket;
  __shared__ int s_at[kMaxCtas + 1];
  __shared__ int s_from[kMaxCtas];
  __shared__ int s_w[kWarps];
  __shared__ long long s_sum[kWarps];
  __shared__ unsigned long long s_top;
  __shared__ int s_pred;
  const int64_t n = src.begin();
  sink.begin();
  if (n <= 0) {
    if (blockIdx.x == 0) {
      sink.finish(0, 0, false, 0, 0);
      arrive(sink, nullptr, 1);
    }
    return;
  }
  const int tile = tile_for(n, (int)gridDim.x);
  const int tiles = (int)((n + tile - 1) / tile);
  const int buckets = tiles;             // one bucket per tile (two smaller ones were slower)
  if ((int)blockIdx.x >= buckets) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_ticket = Sink::kUnique ? (int)atomicAdd(sc.ctl, 1ull) : (int)blockIdx.x;
    s_top = 0;
    s_pred = 0;
  }
  __syncthreads();
  const int b = s_ticket;
  // thread t: the bucket's piece of tile t
  long long before = 0;
  int lo = 0, len = 0;
  if (tid < tiles) {
    lo = sc.start[b * tiles + tid];
    len = sc.start[(b + 1) * tiles + tid] - lo;
    before = lo;
    if (Sink::kPred && b > 0) {
      // (a bucket after the first holds at least its splitter, so only bucket 0 can be an empty predecessor)
      const unsigned long long top = sc.top[(b - 1) * tiles + tid];
      if (lo > sc.start[(b - 1) * tiles + tid]) {
        s_pred = 1;
        atomicMax(&s_top, top);
      }
    }
  }
  const int off = warp_inclusive_scan(len, lane);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 31) s_w[warp] = off;
  if (lane == 0) s_sum[warp] = before;
  __syncthreads();
  int woff = 0, m = 0;
  int64_t base = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) woff += s_w[w];
    m += s_w[w];
    base += s_sum[w];
  }
  if (tid < tiles) {
    s_at[tid] = woff + off - len;
    s_from[tid] = tid * tile + lo - (woff + off - len);
  }
  if (tid == 0) s_at[tiles] = m;
  const bool has_pred = s_pred != 0;
  const uint64_t pred_key = s_top;
  __syncthreads();
  const View<WIDE> from{sc.tile_k, sc.tile_p};
  // four lanes copy one piece (about seven items at 148 tiles of 1,000)
  auto collect = [&](const View<WIDE>& v) {
    for (int a = tid >> 2; a < tiles; a += kThreads / 4) {
      const int e = s_at[a + 1], f = s_from[a];
#pragma unroll 4
      for (int i = s_at[a] + (tid & 3); i < e; i += 4) v.set(i, from.get(f + i));
    }
  };
  const bool last = b == buckets - 1;
  if (m <= cap) {
    const Arrays<WIDE> sm(smem_ts, cap);
    collect(sm.v);
    block_sort<WIDE>(sm.v, sm.tmp, sm.aux, sm.grp, m);
    deliver<Sink, WIDE>(sink, sm.v, m, n, base, pred_key, has_pred, pos_bits, b, last, sc.ctl, d_status);
  } else {
    // a bucket that shared memory does not hold (unevenly spread sample) is sorted in global memory
    const View<WIDE> v{sc.over_k + base, sc.over_p + base}, tmp{sc.over_k + n_cap + base, sc.over_p + n_cap + base};
    collect(v);
    block_sort<WIDE>(v, tmp, sc.over_a + base, sc.over_g + base, m);
    deliver<Sink, WIDE>(sink, v, m, n, base, pred_key, has_pred, pos_bits, b, last, sc.ctl, d_status);
  }
  arrive(sink, sc.ctl + kCtlWords - 1, buckets);
}

template <class Source, class Sink, bool WIDE>
__global__ void __launch_bounds__(kThreads)
ts_single_kernel(Source src, Sink sink, int pos_bits, int32_t* d_status) {
  extern __shared__ __align__(16) unsigned char smem_ts[];
  const int m = (int)src.begin();
  sink.begin();
  const Arrays<WIDE> sm(smem_ts, kSingleMax);
  for (int i = threadIdx.x; i < m; i += kThreads) {
    sm.v.set(i, make_item<WIDE>(src.key(i), (uint32_t)i, pos_bits));
    src.prepare(i);
  }
  block_sort<WIDE>(sm.v, sm.tmp, sm.aux, sm.grp, m);
  deliver<Sink, WIDE>(sink, sm.v, m, m, 0, 0, false, pos_bits, 0, true, nullptr, d_status);
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
  SGL_CUDA_CHECK(allow_smem((const void*)ts_part_kernel<Source, WIDE, Sink::kPred>, part_done, Arrays<WIDE>::bytes(kMaxSamples)));
  SGL_CHECK_RC(launch(ts_part_kernel<Source, WIDE, Sink::kPred>, ctas, kThreads, Arrays<WIDE>::bytes(kMaxSamples), stream,
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
