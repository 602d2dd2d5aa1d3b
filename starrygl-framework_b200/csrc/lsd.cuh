// Radix sort of lists beyond the mini-batch sort: least significant digit first, up to 9 bits a pass, ONE kernel per pass (the
// "onesweep" scheme of Adinets and Merrill, with Merrill and Garland's decoupled look-back):
//   1. lsd_hist_kernel   one read of the keys: digit totals of every pass
//   2. lsd_scan_kernel   start of every digit, all passes
//   3. lsd_pass_kernel   per pass: a CTA takes the next tile, ranks its keys stably, publishes its digit counts, adds up those of
//                        the tiles before it, and writes every digit's run with consecutive threads
//   4. lsd_deliver_kernel   hands every item with its place, and for sinks that number groups its group's number, to a Sink
// HBM traffic per pass and key: 16 B + twice the payload (a histogram kernel, a scan kernel and a scatter kernel per pass read
// the keys once more and took 1.0 ms per pass for 50 M keys).
#pragma once
#include <type_traits>

#include "launch.cuh"
#include "scan.cuh"
#include "sort.cuh"
#include "tilesort.cuh"

namespace sgl {
namespace {

constexpr int kBits = 9;
constexpr int kRadix = 1 << kBits;
constexpr int kMaxPasses = 8;
// Measured (50 M and 4.2 M keys of 44 bits, 256 - 1,024 threads, 8 - 20 keys each, 8 and 9 bits a pass): two CTAs of 512 threads per SM
// are the best of them; 9 bits take five passes instead of six.  A pass of 50 M keys with an 8-byte payload: 481 - 490 us, 3.3 TB/s;
// the first and the last of a T-CSR build, which read and write four arrays, 597 and 566 us.  The load/store pipe is busy two
// thirds of the time (ranks, staging), HBM half.
constexpr int kLsdThreads = 512;
constexpr int kLsdCtas = 2;
constexpr int kLsdWarps = kLsdThreads / 32;
template <class V>
constexpr int kLsdItems = sizeof(V) == 4 ? 14 : 12;      // keys per thread; more would spill
template <class V>
constexpr int kLsdTile = kLsdThreads * kLsdItems<V>;
template <class V>
constexpr int kLookWide = sizeof(V) == 4 ? 8 : 4;         // tiles a look-back step reads (measured: 2 - 16)
constexpr int kHistThreads = 512;

// a pass: `bits` <= kBits bits from `shift` on
struct Digit {
  int shift, bits;
  __device__ __forceinline__ uint32_t of(uint64_t key) const { return (uint32_t)(key >> shift) & ((1u << bits) - 1u); }
};

// Digit totals of every pass, each first.bits further up: one shared-memory counter table per pass.  A warp whose keys all carry the
// same digit (high digits of a hub, ordered input) adds once.  Items that are checked on the way (Items::kChecked, edges) have check(i)
// called once each and the words or-ed; where refuses() says so of the result, *stop is set and the passes do nothing.  Of their groups of
// 32 only the first that are alike are looked for.
// 50 M edges: 276 us with their ids read (466 with a look at every group; 274 with that and the ids left to the scan, which took 262 and
// not 184 us then); pairs of a batch, skewed in some groups and not in others, 14 M and 3.8 M: 181 us with a look at every group, 202.
template <class Items>
__global__ void __launch_bounds__(kHistThreads)
lsd_hist_kernel(Items items, Digit first, int passes, unsigned long long* __restrict__ hist, int64_t* d_count, unsigned int* stop) {
  __shared__ uint32_t s_hist[kMaxPasses * kRadix];
  const int64_t n = items.begin();
  if (d_count && blockIdx.x == 0 && threadIdx.x == 0) *d_count = n;      // for the kernels behind the first pass
  for (int j = threadIdx.x; j < passes * kRadix; j += kHistThreads) s_hist[j] = 0;
  __syncthreads();
  constexpr int kAhead = 4;              // keys in flight per thread
  const int64_t stride = (int64_t)gridDim.x * kHistThreads * kAhead;
  const int lane = threadIdx.x & 31;
  [[maybe_unused]] unsigned long long check = 0;
  for (int64_t i0 = (int64_t)blockIdx.x * kHistThreads * kAhead; i0 < n; i0 += stride) {
    uint64_t key[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t i = i0 + u * kHistThreads + threadIdx.x;
      key[u] = i < n ? items.key(i) : 0;
      if constexpr (Items::kChecked) check |= i < n ? items.check(i) : 0ull;
    }
    // are the digits of a warp's u-th keys alike?  Then they are counted.
    auto look = [&](int u, uint32_t* h, uint32_t d) -> bool {
      const bool valid = i0 + u * kHistThreads + threadIdx.x < n;
      const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
      if (!__all_sync(0xffffffffu, !valid || d == d0)) return false;
      const unsigned act = __ballot_sync(0xffffffffu, valid);
      if (lane == 0 && act) atomicAdd(&h[d0], (uint32_t)__popc(act));
      return true;
    };
    if constexpr (Items::kChecked) {
      for (int p = 0; p < passes; ++p) {
        const Digit digit{first.shift + p * first.bits, first.bits};
        uint32_t* const h = s_hist + p * kRadix;
        bool alike = true;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const uint32_t d = digit.of(key[u]);
          alike = alike && look(u, h, d);
          if (!alike && i0 + u * kHistThreads + threadIdx.x < n) atomicAdd(&h[d], 1u);
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        for (int p = 0; p < passes; ++p) {
          uint32_t* const h = s_hist + p * kRadix;
          const uint32_t d = Digit{first.shift + p * first.bits, first.bits}.of(key[u]);
          if (!look(u, h, d) && i0 + u * kHistThreads + threadIdx.x < n) atomicAdd(&h[d], 1u);
        }
      }
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < passes * kRadix; j += kHistThreads)
    if (s_hist[j]) atomicAdd(&hist[j], (unsigned long long)s_hist[j]);
  if constexpr (Items::kChecked)
    if (items.refuses(check)) *(volatile unsigned int*)stop = 1u;
}

// totals -> starts, one CTA per pass
static __global__ void __launch_bounds__(kRadix) lsd_scan_kernel(unsigned long long* __restrict__ hist) {
  unsigned long long* h = hist + blockIdx.x * kRadix;
  const unsigned long long v = h[threadIdx.x];
  h[threadIdx.x] = cta_exclusive_scan<kRadix, unsigned long long>(v, nullptr);
}

// Published by a tile per digit: value, pass number + 1, and whether the value is the tile's own or includes all
// tiles before it.  Words of an earlier pass count as not published, so the array is cleared once per sort.
constexpr uint64_t kOwn = 1ull << 62, kAll = 2ull << 62, kValue = (1ull << 56) - 1;
__device__ __forceinline__ uint64_t pass_tag(int pass) { return (uint64_t)(pass + 1) << 56; }

template <class V>
struct LsdSmem {
  union {
    uint64_t keys[kLsdTile<V>];               // the tile in digit order, and after that its payload
    uint32_t mask[kLsdWarps][kRadix];      // before that: lanes of the warp's current round that hold the digit
  };
  uint32_t cnt[kLsdWarps][kRadix];         // keys of the digit in the warp so far, then where the warp's start in the tile
  uint32_t out[kRadix];                    // global position of the tile's digit run minus its position in the tile (mod 2^32)
  int ticket;
  unsigned int stop;
};

// Sum of what the tiles before this one hold of digit threadIdx.x; publishes it with the tile's own.
template <int kWide>
__device__ __forceinline__ uint64_t look_back(uint64_t* state, int pass, int tile, uint32_t total, unsigned long long limit, unsigned int* gave_up,
                                              int32_t* d_status) {
  const uint64_t tag = pass_tag(pass);
  volatile uint64_t* st = state + threadIdx.x;
  uint64_t sum = 0;
  unsigned long long t0 = 0;
  if (limit == 0) {                      // (no patience: given up whether it would have waited or not; not in the loop, where it cost 3 %)
    dev_flag(d_status, SGL_DEV_TIMEOUT);
    *(volatile unsigned int*)gave_up = 1u;
    st[(size_t)tile * kRadix] = kAll | tag | total;
    return 0;
  }
  // (tiles are taken in order: those before this one are running or done)
  for (int t = tile - 1; t >= 0;) {
    uint64_t w[kWide];
#pragma unroll
    for (int u = 0; u < kWide; ++u) w[u] = t - u >= 0 ? st[(size_t)(t - u) * kRadix] : 0;
    bool done = false, stalled = false;
#pragma unroll
    for (int u = 0; u < kWide; ++u) {
      if (done || stalled || t < 0) continue;
      if ((w[u] & (0x3full << 56)) != tag) {
        stalled = true;
        continue;
      }
      sum += w[u] & kValue;
      done = (w[u] & kAll) != 0;
      --t;
    }
    if (done) break;
    if (stalled) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      if (now - t0 >= limit) {
        dev_flag(d_status, SGL_DEV_TIMEOUT);
        *(volatile unsigned int*)gave_up = 1u;
        break;
      }
    }
  }
  st[(size_t)tile * kRadix] = kAll | tag | (sum + total);
  return sum;
}

// where a pass reads its items from: the arrays of the pass before, or (first pass) the producer of the keys
template <class V>
struct ArrayItems {
  static constexpr bool kChecked = false;
  const uint64_t* keys;
  const V* vals;
  int64_t n_cap;
  const int64_t* d_n;
  __device__ __forceinline__ int64_t begin() const { return eff_count(n_cap, d_n); }
  __device__ __forceinline__ uint64_t key(int64_t i) const { return keys[i]; }
  __device__ __forceinline__ V val(int64_t i) const { return vals[i]; }
};

// where a pass writes them: the arrays of the next one, or (last pass, optionally) what the caller makes of sorted items
template <class V>
struct ArrayOut {
  uint64_t* keys;
  V* vals;
  __device__ __forceinline__ void key(uint32_t g, uint64_t k) const { keys[g] = k; }
  __device__ __forceinline__ void val(uint32_t g, V v) const { vals[g] = v; }
};

// a Source (see tilesort.cuh) with the position as payload
template <class Source>
struct SourceItems {
  static constexpr bool kChecked = false;
  Source src;
  __device__ __forceinline__ int64_t begin() { return src.begin(); }
  __device__ __forceinline__ uint64_t key(int64_t i) const { return src.key(src.load(i)); }
  __device__ __forceinline__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};

// kLoop: a CTA takes tile after tile instead of one, for sorts that mostly turn out not to be needed (a CTA per tile of 38 M entries that
// are not there took 8 us a pass, 38 us behind the last merge of a batch; a list that is there is faster without the loop, passes of a
// CSC of 1.3 M edges 84 and 80 us, 16 M 793 and 756).
template <class V, class Items, class Out, bool kLoop>
__global__ void __launch_bounds__(kLsdThreads, kLsdCtas)
lsd_pass_kernel(Items items, Digit digit, int pass,
                const unsigned long long* __restrict__ starts, unsigned int* __restrict__ ticket, uint64_t* state,
                Out out, unsigned long long limit, unsigned int* gave_up, const unsigned int* __restrict__ stop, int32_t* d_status) {
  extern __shared__ __align__(16) unsigned char smem[];
  LsdSmem<V>& sm = *(LsdSmem<V>*)smem;
  constexpr int kItems = kLsdItems<V>, kTile = kLsdTile<V>;
  const int64_t n = items.begin();
  if ((int64_t)blockIdx.x * kTile >= n) return;            // (capacity beyond the count; the others share the tickets)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    const unsigned int s = *stop;        // (on its way together with the ticket; the same for all CTAs of a pass)
    sm.ticket = (int)atomicAdd(ticket, 1u);
    sm.stop = s;
  }
  do {
    for (int j = tid; j < kLsdWarps * kRadix / 4; j += kLsdThreads) {
      ((uint4*)&sm.mask[0][0])[j] = make_uint4(0, 0, 0, 0);
      ((uint4*)&sm.cnt[0][0])[j] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    if (sm.stop) break;
    const int tile = sm.ticket;
    const int64_t tile_base = (int64_t)tile * kTile;
    if (kLoop && tile_base >= n) break;
    const int tile_n = (int)(n - tile_base < kTile ? n - tile_base : kTile);
    // a warp owns consecutive keys of the tile, 32 at a time: (warp, round, lane) order = key order
    const int first = warp * (kItems * 32) + lane;
    uint64_t k[kItems];
#pragma unroll
    for (int c = 0; c < kItems; ++c) {
      const int j = first + c * 32;
      k[c] = j < tile_n ? items.key(tile_base + j) : ~0ull;
    }
    // stable rank inside the warp: the lanes of a round that share a digit find each other through one word per digit
    uint16_t rank[kItems];
    uint32_t *mask = sm.mask[warp], *cnt = sm.cnt[warp];
    const uint32_t below = (1u << lane) - 1u;
#pragma unroll
    for (int c = 0; c < kItems; ++c) {
      const bool valid = first + c * 32 < tile_n;
      const uint32_t d = digit.of(k[c]);
      // through shared memory, or by ballots: one kind of round fills the load/store pipe, the other the integer pipe
      const bool by_ballot = c % 3 == 0;
      uint32_t peers;
      if (by_ballot) {
        peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < kBits; ++b) {
          const uint32_t m = __ballot_sync(0xffffffffu, (d >> b) & 1u);
          peers &= (d >> b) & 1u ? m : ~m;
        }
      } else {
        if (valid) atomicOr(&mask[d], 1u << lane);
        __syncwarp();
        peers = valid ? mask[d] : 0u;
      }
      const uint32_t before = valid ? cnt[d] : 0u;
      __syncwarp();
      if (valid && (peers & below) == 0) {   // the lowest lane of the digit
        if (!by_ballot) mask[d] = 0;
        cnt[d] = before + __popc(peers);
      }
      __syncwarp();
      rank[c] = (uint16_t)(before + __popc(peers & below));
    }
    __syncthreads();
    // per digit: counts of the warps -> starts of the warps; the tile's count is published, those of the tiles before added up
    static_assert(kRadix <= kLsdThreads && kTile < (1 << 16), "a thread per digit, 16-bit places");
    uint32_t total = 0;
    if (tid < kRadix) {
#pragma unroll
      for (int w = 0; w < kLsdWarps; ++w) total += sm.cnt[w][tid];
      ((volatile uint64_t*)state)[(size_t)tile * kRadix + tid] = (tile == 0 ? kAll : kOwn) | pass_tag(pass) | total;
    }
    const uint32_t start = cta_exclusive_scan<kLsdThreads, uint32_t>(total, nullptr);
    if (tid < kRadix) {
      uint32_t at = start;
#pragma unroll
      for (int w = 0; w < kLsdWarps; ++w) {
        const uint32_t c = sm.cnt[w][tid];
        sm.cnt[w][tid] = at;
        at += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kItems; ++c) {
      if (first + c * 32 < tile_n) {
        rank[c] += (uint16_t)cnt[digit.of(k[c])];      // place in the tile
        sm.keys[rank[c]] = k[c];
      }
    }
    if (tid < kRadix) {
      const uint64_t sum = tile > 0 ? look_back<kLookWide<V>>(state, pass, tile, total, limit, gave_up, d_status) : 0;
      sm.out[tid] = (uint32_t)(starts[tid] + sum) - start;
    }
    __syncthreads();
    // (everybody has read the ticket; its tile has published what others wait for)
    if (kLoop && tid == 0) sm.ticket = (int)atomicAdd(ticket, 1u);
    // consecutive threads take consecutive tile positions, i.e. runs of one digit -> consecutive addresses
    constexpr uint32_t kNone = ~0u;
    uint32_t g[kItems];
#pragma unroll
    for (int c = 0; c < kItems; ++c) {
      const int j = c * kLsdThreads + tid;
      g[c] = kNone;
      if (j < tile_n) {
        const uint64_t key = sm.keys[j];
        g[c] = sm.out[digit.of(key)] + j;
        if (g[c] >= n) g[c] = kNone;       // (only where a look-back gave up)
        if (g[c] != kNone) out.key(g[c], key);
      }
    }
    // the payload follows through the same shared memory (loaded late: keys and payload do not fit the registers)
    V v[kItems];
#pragma unroll
    for (int c = 0; c < kItems; ++c) {
      const int j = first + c * 32;
      v[c] = j < tile_n ? items.val(tile_base + j) : (V)0;
    }
    __syncthreads();
    V* vals = (V*)sm.keys;
#pragma unroll
    for (int c = 0; c < kItems; ++c)
      if (first + c * 32 < tile_n) vals[rank[c]] = v[c];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kItems; ++c)
      if (g[c] != kNone) out.val(g[c], vals[c * kLsdThreads + tid]);
    if (kLoop) __syncthreads();
  } while (kLoop);
}

// ---- delivery of a sorted list to a Sink (see tilesort.cuh) -------------------------------------------------------------
constexpr int kDeliverThreads = 256;
constexpr int kDeliverItems = 8;
template <class Sink>
constexpr int kDeliverCtas = Sink::kUnique ? 4 : 6;       // per SM (without numbering 32 registers, with the 56 of 4 CTAs 1.3 M edges took 44 us, not 33)
constexpr int kDeliverTile = kDeliverThreads * kDeliverItems;

// Sum of what the CTAs before this one (by ticket: they all run already) published; called by one whole warp.
__device__ __forceinline__ uint64_t deliver_prefix(uint64_t* state, int tile, uint64_t total, int lane, unsigned long long limit, int32_t* d_status) {
  volatile uint64_t* st = state;
  if (lane == 0) st[tile] = tile == 0 ? (kAll | total) : (kOwn | total);
  constexpr uint64_t kSum = (1ull << 62) - 1;
  uint64_t base = 0;
  unsigned long long t0 = 0;
  for (int look = tile - 1; look >= 0;) {
    const int p = look - lane;
    uint64_t v = kAll;                   // before the first tile: nothing
    if (p >= 0) v = st[p];
    if (__any_sync(0xffffffffu, v == 0)) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, now - t0 >= limit)) {
        if (lane == 0) dev_flag(d_status, SGL_DEV_TIMEOUT);
        break;
      }
      continue;
    }
    const unsigned all = __ballot_sync(0xffffffffu, (v & kAll) != 0);
    const int stop = all ? __ffs(all) - 1 : 31;
    uint64_t x = lane <= stop ? (v & kSum) : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    base += x;
    if (all) break;
    look -= 32;
  }
  if (lane == 0 && tile > 0) st[tile] = kAll | (base + total);
  return base;
}

// ctl[0] ticket, ctl[1] arrivals; state: one word per tile, cleared
template <class Sink>
__global__ void __launch_bounds__(kDeliverThreads, kDeliverCtas<Sink>)
lsd_deliver_kernel(Sink sink, const uint64_t* __restrict__ keys, const uint32_t* __restrict__ pos, int64_t n_cap, const int64_t* d_count,
                   unsigned long long* ctl, uint64_t* state, unsigned long long limit, const unsigned int* gave_up, int32_t* d_status) {
  const int64_t n = *gave_up ? 0 : eff_count(n_cap, d_count);     // (a pass that gave up left places unwritten)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  sink.begin();
  if (n <= 0) {
    if (blockIdx.x == 0) {
      sink.finish(0, 0, false, 0, 0);
      tilesort::arrive(sink, nullptr, 1);
    }
    return;
  }
  const int tiles = (int)((n + kDeliverTile - 1) / kDeliverTile);
  if constexpr (!Sink::kUnique) {
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int64_t base = (int64_t)tile * kDeliverTile;
#pragma unroll
      for (int c = 0; c < kDeliverItems; ++c) {
        const int64_t i = base + c * kDeliverThreads + tid;
        if (i < n) {
          sink.item(i, keys[i], pos[i]);
          sink.between(i, keys[i], i > 0, i > 0 ? keys[i - 1] : 0ull);
        }
      }
      if (tile == tiles - 1) sink.finish(n, keys[n - 1], true, 0, 0);
      tilesort::arrive(sink, ctl + 1, tiles);
    }
  } else {
    constexpr bool kTwo = Sink::kLevels == 2;
    constexpr int kShift = 31;           // two counts share the word: 31 bits each
    __shared__ int s_ticket;
    __shared__ uint64_t s_cnt[kDeliverItems * (kDeliverThreads / 32)], s_scan[kDeliverItems * (kDeliverThreads / 32)];
    __shared__ uint64_t s_base;
    if ((int)blockIdx.x >= tiles) return;
    for (;;) {                           // tile after tile (14 M entries of 42 M at most: 252 us, with a CTA per tile of the capacity 284)
      if (tid == 0) s_ticket = (int)atomicAdd(ctl, 1ull);
      __syncthreads();
      const int tile = s_ticket;
      if (tile >= tiles) break;
      const int64_t first = (int64_t)tile * kDeliverTile;
      uint64_t k[kDeliverItems];
      uint32_t p[kDeliverItems];
      unsigned h1 = 0, h2 = 0;             // bit c: item c of the thread starts a group / a coarser group
      unsigned up1[kDeliverItems], up2[kDeliverItems];
#pragma unroll
      for (int c = 0; c < kDeliverItems; ++c) {
        const int64_t i = first + c * kDeliverThreads + tid;
        k[c] = i < n ? __ldcs(keys + i) : 0;     // (streamed: the cache is for what the sink scatters)
        p[c] = i < n ? __ldcs(pos + i) : 0u;
      }
#pragma unroll
      for (int c = 0; c < kDeliverItems; ++c) {
        const int64_t i = first + c * kDeliverThreads + tid;
        bool a = false, b = false;
        if (i < n && sink.counted(k[c])) {
          const uint64_t q = i > 0 ? keys[i - 1] : 0ull;
          a = i == 0 || sink.group(q) != sink.group(k[c]);
          if constexpr (kTwo) b = i == 0 || sink.group2(q) != sink.group2(k[c]);
        }
        const unsigned ba = __ballot_sync(0xffffffffu, a), bb = kTwo ? __ballot_sync(0xffffffffu, b) : 0u;
        h1 |= (a ? 1u : 0u) << c;
        h2 |= (b ? 1u : 0u) << c;
        const unsigned upto = (2u << lane) - 1u;
        up1[c] = __popc(ba & upto);
        up2[c] = __popc(bb & upto);
        if (lane == 0) s_cnt[c * (kDeliverThreads / 32) + warp] = (uint64_t)__popc(ba) | ((uint64_t)__popc(bb) << kShift);
      }
      __syncthreads();
      constexpr int kCells = kDeliverItems * (kDeliverThreads / 32);
      const uint64_t mine = tid < kCells ? s_cnt[tid] : 0;
      uint64_t total;
      const uint64_t ex = cta_exclusive_scan<kDeliverThreads, uint64_t>(mine, &total);
      if (tid < kCells) s_scan[tid] = ex;
      if (warp == 0) {
        const uint64_t base = deliver_prefix(state, tile, total, lane, limit, d_status);
        if (lane == 0) s_base = base;
      }
      __syncthreads();
      const uint64_t base = s_base, low = kTwo ? (1ull << kShift) - 1 : ~0ull;
#pragma unroll
      for (int c = 0; c < kDeliverItems; ++c) {
        const int64_t i = first + c * kDeliverThreads + tid;
        if (i >= n) continue;
        const uint64_t off = base + s_scan[c * (kDeliverThreads / 32) + warp];
        const int64_t u = (int64_t)(off & low) + up1[c] - 1, u2 = kTwo ? (int64_t)(off >> kShift) + up2[c] - 1 : 0;
        sink.item(i, k[c], p[c], (h1 >> c) & 1u, u, (h2 >> c) & 1u, u2);
      }
      if (tile == tiles - 1) sink.finish(n, 0, false, (int64_t)((base + total) & low), kTwo ? (int64_t)((base + total) >> kShift) : 0);
      tilesort::arrive(sink, ctl + 1, tiles);
      __syncthreads();
    }
  }
}

inline int lsd_passes(int first_bit, int num_bits) { return num_bits <= first_bit + kBits ? 1 : (num_bits - first_bit + kBits - 1) / kBits; }
template <class V>
inline int64_t lsd_tiles(int64_t n) { return (n + kLsdTile<V> - 1) / kLsdTile<V>; }

template <class V>
inline size_t lsd_ws_bytes(int64_t n) {
  return align_up((kMaxPasses * kRadix + kMaxPasses) * 8) + align_up((size_t)lsd_tiles<V>(n < 1 ? 1 : n) * kRadix * 8);
}

// Sorts on key bits [first_bit, num_bits), at least one pass; the first pass reads from `items`, writes to (k1, v1), the next to
// (k0, v0) and so on; *in_first says whether the result ends in (k1, v1).  With a `last` of another type than ArrayOut the last
// pass writes there instead and its arrays stay free.  Items that are refused (see lsd_hist_kernel) are not sorted.  **gave_up on the device: a look-back ran into its time limit, the result
// is not to be used as positions.  d_n: number of items on the device (<= n); d_count: the count kernel writes it there, from items.
template <class V, class Items, class Last, bool kLoop = false>
int lsd_sort(const Items& items, uint64_t* k1, V* v1, uint64_t* k0, V* v0, int64_t n, const int64_t* d_n, int64_t* d_count, int first_bit, int num_bits,
             const Last& last, bool* in_first, unsigned int** gave_up, WsCarver& c, int32_t* d_status, cudaStream_t stream) {
  using Array = ArrayOut<V>;
  constexpr bool kArray = std::is_same<Last, Array>::value;
  const int passes = lsd_passes(first_bit, num_bits);
  const int bits = num_bits > first_bit ? (num_bits - first_bit + passes - 1) / passes : 1;     // an even share each
  const int64_t tiles = lsd_tiles<V>(n);
  unsigned long long* hist = c.take<unsigned long long>(kMaxPasses * kRadix + kMaxPasses);
  unsigned int* tickets = (unsigned int*)(hist + kMaxPasses * kRadix);
  *gave_up = tickets + kMaxPasses;
  unsigned int* const stop = *gave_up + 1;
  uint64_t* state = c.take<uint64_t>((size_t)tiles * kRadix);
  SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "radix sort: workspace too small for %lld keys", (long long)n);
  SGL_CHECK_RC(zero_async(hist, (size_t)((char*)(state + (size_t)tiles * kRadix) - (char*)hist), stream));     // (one behind the other)
  SGL_CHECK_RC(launch(lsd_hist_kernel<Items>, stream_grid(n, kHistThreads * 16, 4), kHistThreads, 0, stream, items, Digit{first_bit, bits},
                      passes, hist, d_count, stop));
  SGL_CHECK_RC(launch(lsd_scan_kernel, passes, kRadix, 0, stream, hist));
  for (int p = 0; p < passes; ++p) {
    const Array out{p & 1 ? k0 : k1, p & 1 ? v0 : v1};
    const ArrayItems<V> in{p & 1 ? k1 : k0, p & 1 ? v1 : v0, n, d_n};
    auto pass = [&](const auto& from, const auto& to) -> int {
      using From = std::decay_t<decltype(from)>;
      using To = std::decay_t<decltype(to)>;
      static std::atomic<uint64_t> done{0};
      SGL_CUDA_CHECK(allow_smem((const void*)lsd_pass_kernel<V, From, To, kLoop>, done, sizeof(LsdSmem<V>)));
      const unsigned ctas = (unsigned)(kLoop && tiles > kNumSM * kLsdCtas ? kNumSM * kLsdCtas : tiles);
      return launch(lsd_pass_kernel<V, From, To, kLoop>, ctas, kLsdThreads, sizeof(LsdSmem<V>), stream, from, Digit{first_bit + p * bits, bits}, p,
                    hist + p * kRadix, tickets + p, state, to, look_back_ns(), *gave_up, stop, d_status);
    };
    const bool to_last = !kArray && p == passes - 1;
    if (p == 0) SGL_CHECK_RC(to_last ? pass(items, last) : pass(items, out));
    else SGL_CHECK_RC(to_last ? pass(in, last) : pass(in, out));
  }
  *in_first = passes & 1;
  return SGL_OK;
}

inline size_t list_ws_bytes(int64_t n) {
  if (n < 1) n = 1;
  if (n <= tilesort::kMaxItems) return tilesort::ws_bytes(n);
  return 2 * align_up((size_t)n * 8) + 2 * align_up((size_t)n * 4) + lsd_ws_bytes<uint32_t>(n) + align_up(8) +
         align_up(((size_t)((n + kDeliverTile - 1) / kDeliverTile) + 2) * 8);
}

// Sorts the items of `src` (at most n_cap, keys of key_bits bits) and delivers them to `sink`: the mini-batch sort, or the
// radix passes and a delivery kernel for longer lists.
template <class Source, class Sink>
int sort_list(const Source& src, const Sink& sink, int64_t n_cap, int key_bits, void* ws, size_t ws_bytes, int32_t* d_status,
              cudaStream_t stream) {
  WsCarver c(ws, ws_bytes);
  if (n_cap <= tilesort::kMaxItems) {
    const tilesort::Scratch sc = tilesort::carve(c, n_cap);
    SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "sort: workspace %zu < %zu bytes", ws_bytes, list_ws_bytes(n_cap));
    return tilesort::launch(src, sink, n_cap, key_bits, sc, d_status, stream);
  }
  SGL_REQUIRE(n_cap < ((int64_t)1 << 32), SGL_ERR_UNSUPPORTED, "sort: %lld entries need a 64-bit position", (long long)n_cap);
  uint64_t *k0 = c.take<uint64_t>(n_cap), *k1 = c.take<uint64_t>(n_cap);
  uint32_t *v0 = c.take<uint32_t>(n_cap), *v1 = c.take<uint32_t>(n_cap);
  int64_t* count = c.take<int64_t>(1);
  const int64_t tiles = (n_cap + kDeliverTile - 1) / kDeliverTile;
  unsigned long long* ctl = c.take<unsigned long long>((size_t)tiles + 2);
  SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "sort: workspace %zu < %zu bytes", ws_bytes, list_ws_bytes(n_cap));
  SGL_CHECK_RC(zero_async(ctl, (size_t)(tiles + 2) * 8, stream));
  bool in_first;
  unsigned int* gave_up;
  auto sort = [&](auto loop) -> int {
    return lsd_sort<uint32_t, SourceItems<Source>, ArrayOut<uint32_t>, decltype(loop)::value>(
        SourceItems<Source>{src}, k1, v1, k0, v0, n_cap, count, count, 0, key_bits, ArrayOut<uint32_t>{}, &in_first, &gave_up, c, d_status, stream);
  };
  bool loop = Sink::kUnique;             // (delivery without numbering, as many CTAs as there is room for or one per tile: CSC of 16 M edges
                                         // 1,301, 1,208 us)
  if constexpr (Source::kOnDemand) {
    SGL_CHECK_RC(src.on_demand() ? sort(std::true_type{}) : sort(std::false_type{}));
    loop = loop || src.on_demand();
  } else {
    SGL_CHECK_RC(sort(std::false_type{}));
  }
  constexpr int kRoom = kNumSM * kDeliverCtas<Sink>;
  const unsigned ctas = (unsigned)(loop && tiles > kRoom ? kRoom : tiles);
  return launch(lsd_deliver_kernel<Sink>, ctas, kDeliverThreads, 0, stream, sink, in_first ? k1 : k0, in_first ? v1 : v0, n_cap, count, ctl,
                (uint64_t*)(ctl + 2), look_back_ns(), gave_up, d_status);
}

}  // namespace
}  // namespace sgl
