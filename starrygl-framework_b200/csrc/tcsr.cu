// T-CSR construction: rows keyed by node id, inside a row ascending timestamp, ties in input order.
//
//   1. tcsr_scan_kernel   one pass over keys and times: timestamp range, keys out of range, is it in time order already, do the
//                         first and last neighbour and edge ids fit 32 bits each (the sort's counts look at all of them); the last CTA
//                         hands the answer to the host
//   2. stable sort by (node << ts_bits) | (ts - ts_min), only the populated bits:
//        up to tilesort::kMaxItems edges   the mini-batch sort, whose sink writes the rows
//        more                              radix passes (lsd.cuh).  Neighbour and edge id travel as the payload (8 bytes) when
//                                          they fit, so that nothing is gathered through a permutation at the end: two random
//                                          8-byte reads per edge took 2.6 of the 8.1 ms of a 50 M edge build.  Input in time
//                                          order, as event streams are, is sorted on the node bits alone.
//        node and timestamp bits above 64  by timestamp, then stably by node
//   3. the last pass writes the edges to their places, tcsr_rows_kernel the row pointer from the row boundaries (no atomics, no
//      prefix sum); with positions as payload tcsr_emit_gather_kernel does both
//
// 50 M edges, 1 M nodes in no particular order: bound by the radix passes' traffic, 264 B per edge.
#include <stddef.h>

#include "chain.cuh"
#include "lsd.cuh"

namespace sgl {
namespace {

// All maxima of unsigned words, so that the block starts as zeros.
struct InputScan {
  unsigned long long late, early;    // largest timestamp, largest complement of a timestamp (sign bit flipped)
  unsigned long long bad_keys;
  unsigned long long flags;          // kUnordered | kWideIds
  unsigned long long arrived;
  long long status;                  // (low half) status word of the sort: a look-back that gave up
};
constexpr unsigned long long kUnordered = 1, kWideIds = 2, kSign = 1ull << 63;

constexpr int kScanThreads = 256;

__global__ void __launch_bounds__(kScanThreads)
tcsr_scan_kernel(const int64_t* __restrict__ key, const int64_t* __restrict__ nbr, const int64_t* __restrict__ ts,
                 const int64_t* __restrict__ eid, int64_t m, int64_t num_nodes, int check_ids, InputScan* out, int64_t* host) {
  unsigned long long late = 0, early = 0, wide = 0;
  unsigned bad = 0, unordered = 0;
  const int64_t stride = (int64_t)gridDim.x * kScanThreads;
#pragma unroll 2
  for (int64_t i = (int64_t)blockIdx.x * kScanThreads + threadIdx.x; i < m; i += stride) {
    const int64_t t = ts[i], k = key[i];
    const unsigned long long u = (unsigned long long)t ^ kSign;
    late = u > late ? u : late;
    early = ~u > early ? ~u : early;
    if (i + 1 < m) unordered |= ts[i + 1] < t ? 1u : 0u;
    bad += (k < 0 || k >= num_nodes) ? 1u : 0u;
    // (a look at the first and the last of them, where ids that ascend are largest; the counts of the sort see all)
    if (check_ids && (i < stride || i >= m - stride)) {
      wide |= (unsigned long long)nbr[i];
      if (eid) wide |= (unsigned long long)eid[i];
    }
  }
  __shared__ unsigned long long s_late[kScanThreads / 32], s_early[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, late, o), b = __shfl_xor_sync(0xffffffffu, early, o);
    late = a > late ? a : late;
    early = b > early ? b : early;
  }
  if (lane == 0) {
    s_late[warp] = late;
    s_early[warp] = early;
  }
  const int bad_cta = __syncthreads_or((int)bad) ? 1 : 0;
  const int flags = (__syncthreads_or((int)unordered) ? (int)kUnordered : 0) | (__syncthreads_or((wide >> 32) != 0) ? (int)kWideIds : 0);
  if (bad_cta) {
    const unsigned w = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0 && w) atomicAdd(&out->bad_keys, (unsigned long long)w);
  }
  if (threadIdx.x == 0) {
    for (int w = 1; w < kScanThreads / 32; ++w) {
      late = s_late[w] > late ? s_late[w] : late;
      early = s_early[w] > early ? s_early[w] : early;
    }
    atomicMax(&out->late, late);
    atomicMax(&out->early, early);
    if (flags) atomicOr(&out->flags, (unsigned long long)flags);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&out->arrived, 1ull) == gridDim.x - 1) {
      __threadfence();
      volatile InputScan* s = out;
      host[0] = (int64_t)(~s->early ^ kSign);
      host[1] = (int64_t)(s->late ^ kSign);
      host[2] = (int64_t)s->bad_keys;
      host[3] = (int64_t)s->flags;
      __threadfence_system();
      *(volatile int64_t*)(host + 4) = 1;
    }
  }
}

// key = (node << ts_bits) | (ts - ts_min)
struct EdgeKey {
  const int64_t *key, *ts;
  long long ts_min;
  int ts_bits;
  __device__ __forceinline__ uint64_t of(int64_t i) const { return make({key[i], ts[i]}); }
  __device__ __forceinline__ uint64_t make(const longlong2& x) const {
    const uint64_t dt = (uint64_t)x.y - (uint64_t)ts_min;
    return ts_bits >= 64 ? dt : (((uint64_t)x.x << ts_bits) | dt);
  }
  __device__ __forceinline__ int64_t node(uint64_t k) const { return ts_bits >= 64 ? 0 : (int64_t)(k >> ts_bits); }
  __device__ __forceinline__ int64_t time(uint64_t k) const {
    return (int64_t)((ts_bits >= 64 ? k : (k & ((1ull << ts_bits) - 1ull))) + (uint64_t)ts_min);
  }
};

// row pointer: every node in (prev, node] starts at position i
__device__ __forceinline__ void start_rows(int64_t* __restrict__ indptr, int64_t prev, int64_t node, int64_t i) {
  for (int64_t v = prev + 1; v <= node; ++v) indptr[v] = i;
}

// ---- up to the mini-batch limit -----------------------------------------------------------------------------------------
// The sort is enqueued together with the scan and reads the time range where the scan leaves it; node, time and position share a word of
// 64 bits then, or there is nothing to sort, nothing is written, and the host, which learns the same a little later, raises or starts over
// with what it knows.
struct ScannedRange {
  const InputScan* scan;                 // nullptr: the key is complete
  int id_bits, pos_bits;
  // false: node ids out of range, or key and position need more than a word
  __device__ __forceinline__ bool read(EdgeKey& k) const {
    if (scan == nullptr) return true;
    const unsigned long long early = scan->early, late = scan->late;
    k.ts_min = (long long)(~early ^ kSign);
    k.ts_bits = 64 - __clzll((long long)(late - ~early));
    return scan->bad_keys == 0 && k.ts_bits + id_bits + pos_bits <= 64;
  }
};

struct EdgeSource {
  static constexpr bool kOnDemand = false;
  EdgeKey k;
  int64_t m;
  ScannedRange range;
  using Raw = longlong2;
  __device__ __forceinline__ int64_t begin() { return range.read(k) ? m : 0; }
  __device__ __forceinline__ Raw load(int64_t i) const { return {k.key[i], k.ts[i]}; }
  __device__ __forceinline__ uint64_t key(const Raw& x) const { return k.make(x); }
};

struct EdgeSink {
  static constexpr bool kUnique = false, kAfter = false;
  EdgeKey k;
  const int64_t *nbr, *eid;
  int64_t num_nodes;
  int64_t *indptr, *out_nbr, *out_ts, *out_eid, *out_perm;
  ScannedRange range;
  bool sorted;
  __device__ __forceinline__ void begin() { sorted = range.read(k); }
  __device__ __forceinline__ void item(int64_t at, uint64_t key, uint32_t p) const {
    out_nbr[at] = nbr[p];
    out_ts[at] = k.time(key);
    out_eid[at] = eid ? eid[p] : (int64_t)p;
    if (out_perm) out_perm[at] = p;
  }
  __device__ __forceinline__ void between(int64_t at, uint64_t key, bool has_prev, uint64_t prev) const {
    start_rows(indptr, has_prev ? k.node(prev) : -1, k.node(key), at);
  }
  __device__ __forceinline__ void finish(int64_t m, uint64_t last, bool has_last, int64_t, int64_t) const {
    if (!sorted) return;
    for (int64_t v = (has_last ? k.node(last) + 1 : 0) + threadIdx.x; v <= num_nodes; v += blockDim.x) indptr[v] = m;
  }
};

// ---- above: items of the first radix pass ---------------------------------------------------------------------------------
struct EdgePairs {                    // neighbour and edge id as payload
  static constexpr bool kChecked = true;
  EdgeKey k;
  const int64_t *nbr, *eid;
  int64_t m;
  InputScan* scan;
  __device__ __forceinline__ unsigned long long check(int64_t i) const { return (unsigned long long)nbr[i] | (unsigned long long)(eid ? eid[i] : 0); }
  __device__ __forceinline__ bool refuses(unsigned long long bits) const {
    const bool wide = (bits >> 32) != 0;
    if (wide) atomicOr(&scan->flags, kWideIds);
    return wide;
  }
  __device__ __forceinline__ int64_t begin() const { return m; }
  __device__ __forceinline__ uint64_t key(int64_t i) const { return k.of(i); }
  __device__ __forceinline__ uint64_t val(int64_t i) const {
    return (uint64_t)(uint32_t)nbr[i] | ((uint64_t)(uint32_t)(eid ? eid[i] : i) << 32);
  }
};

struct EdgePositions {                // position as payload
  static constexpr bool kChecked = false;
  EdgeKey k;
  int64_t m;
  __device__ __forceinline__ int64_t begin() const { return m; }
  __device__ __forceinline__ uint64_t key(int64_t i) const { return k.of(i); }
  __device__ __forceinline__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};

// The last radix pass writes the edges where they belong; the node of every edge stays for the row pointer.
struct EdgeOut {
  EdgeKey k;
  uint32_t* node;
  int64_t *nbr, *ts, *eid;
  __device__ __forceinline__ void key(uint32_t g, uint64_t key) const {
    node[g] = (uint32_t)k.node(key);
    ts[g] = k.time(key);
  }
  __device__ __forceinline__ void val(uint32_t g, uint64_t v) const {
    nbr[g] = (int64_t)(uint32_t)v;
    eid[g] = (int64_t)(v >> 32);
  }
};

__global__ void __launch_bounds__(256)
tcsr_rows_kernel(const InputScan* scan, const uint32_t* __restrict__ node, int64_t m, int64_t num_nodes, int64_t* __restrict__ indptr) {
  const int64_t stride = (int64_t)gridDim.x * 256;
  if (scan->status || (scan->flags & kWideIds)) {      // (the host reports it, or does it again; no rows rather than wrong ones)
    for (int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x; v <= num_nodes; v += stride) indptr[v] = 0;
    return;
  }
  for (int64_t i0 = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4; i0 <= m; i0 += stride * 4) {
    uint32_t x[4] = {0, 0, 0, 0};
    if (i0 + 4 <= m) {
      const uint4 q = *(const uint4*)(node + i0);
      x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
    } else {
      for (int u = 0; u < 4; ++u)
        if (i0 + u < m) x[u] = node[i0 + u];
    }
    int64_t prev = i0 > 0 ? (int64_t)node[i0 - 1] : -1;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i0 + u > m) break;
      const int64_t cur = i0 + u < m ? (int64_t)x[u] : num_nodes;
      start_rows(indptr, prev, cur, i0 + u);
      prev = cur;
    }
  }
}

// combined == 0: the keys are node ids and the timestamps are gathered too
__global__ void __launch_bounds__(256)
tcsr_emit_gather_kernel(const InputScan* scan, const uint64_t* __restrict__ keys, const uint32_t* __restrict__ perm, int combined, EdgeKey k,
                        const int64_t* __restrict__ nbr, const int64_t* __restrict__ eid, int64_t m, int64_t num_nodes,
                        int64_t* __restrict__ indptr, int64_t* __restrict__ out_nbr, int64_t* __restrict__ out_ts,
                        int64_t* __restrict__ out_eid, int64_t* __restrict__ out_perm) {
  if (scan->status) {
    for (int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x; v <= num_nodes; v += (int64_t)gridDim.x * 256) indptr[v] = 0;
    return;
  }
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < m; i += (int64_t)gridDim.x * 256) {
    const uint32_t p = perm[i];
    const uint64_t key = keys[i];
    out_nbr[i] = nbr[p];
    out_ts[i] = combined ? k.time(key) : k.ts[p];
    out_eid[i] = eid ? eid[p] : (int64_t)p;
    if (out_perm) out_perm[i] = (int64_t)p;
    const int64_t node = combined ? k.node(key) : (int64_t)key;
    start_rows(indptr, i > 0 ? (combined ? k.node(keys[i - 1]) : (int64_t)keys[i - 1]) : -1, node, i);
    if (i == m - 1)
      for (int64_t r = node + 1; r <= num_nodes; ++r) indptr[r] = m;
  }
}

// keys of the two rounds when node and timestamp do not share a word
__global__ void __launch_bounds__(256)
tcsr_round_keys_kernel(EdgeKey k, const uint32_t* __restrict__ perm, int64_t m, uint64_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < m; i += (int64_t)gridDim.x * 256)
    out[i] = perm ? (uint64_t)k.key[perm[i] < m ? perm[i] : 0u] : (uint64_t)k.ts[i] - (uint64_t)k.ts_min;
}

__global__ void fill_i64_kernel(int64_t* p, int64_t n, int64_t v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = v;
}

int launch_fence(const int64_t* indptr, const int64_t* ts, int64_t num_nodes, int64_t m, int64_t* out_fence, const ScannedRange& range,
                 cudaStream_t stream);

}  // namespace
}  // namespace sgl

using namespace sgl;

extern "C" size_t sgl_tcsr_build_ws_bytes(int64_t num_nodes, int64_t m) {
  (void)num_nodes;
  if (m < 1) m = 1;
  const size_t pairs = 4 * align_up((size_t)m * 8) + lsd_ws_bytes<uint64_t>(m);
  const size_t rounds = 2 * align_up((size_t)m * 8) + 2 * align_up((size_t)m * 4) + radix_sort_ws_bytes(m);
  size_t most = m <= tilesort::kMaxItems ? list_ws_bytes(m) : pairs;
  most = most > rounds ? most : rounds;
  return align_up(sizeof(InputScan)) + most;
}

extern "C" int sgl_tcsr_build_fenced(int64_t num_nodes, int64_t m, const int64_t* key, const int64_t* nbr, const int64_t* ts,
                                     const int64_t* eid, int64_t* indptr, int64_t* out_nbr, int64_t* out_ts, int64_t* out_eid,
                                     int64_t* out_perm, int64_t* out_fence, int64_t* h_ts_range, void* ws, size_t ws_bytes,
                                     void* stream_) {
  SGL_NVTX("sgl_tcsr_build");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(num_nodes >= 0 && m >= 0, SGL_ERR_ARG, "tcsr_build: negative size");
  SGL_REQUIRE(m < ((int64_t)1 << 32), SGL_ERR_UNSUPPORTED, "tcsr_build: m=%lld needs a 64-bit permutation", (long long)m);
  SGL_REQUIRE(indptr, SGL_ERR_ARG, "tcsr_build: indptr is null");
  if (m == 0) {
    fill_i64_kernel<<<stream_grid(num_nodes + 1, 256, 4), 256, 0, stream>>>(indptr, num_nodes + 1, 0);
    SGL_LAUNCH_CHECK();
    if (h_ts_range) h_ts_range[0] = h_ts_range[1] = 0;
    return SGL_OK;
  }
  SGL_REQUIRE(key && nbr && ts && out_nbr && out_ts && out_eid, SGL_ERR_ARG, "tcsr_build: null array");
  SGL_REQUIRE(ws && ws_bytes >= sgl_tcsr_build_ws_bytes(num_nodes, m), SGL_ERR_WORKSPACE, "tcsr_build: workspace %zu < %zu bytes", ws_bytes,
              sgl_tcsr_build_ws_bytes(num_nodes, m));
  InputScan* d_scan = (InputScan*)ws;
  void* rest = (char*)ws + align_up(sizeof(InputScan));
  const size_t rest_bytes = ws_bytes - align_up(sizeof(InputScan));
  const bool small = m <= tilesort::kMaxItems;
  int32_t* const d_status = (int32_t*)&d_scan->status;
  void* words = nullptr;
  SGL_CHECK_RC(sgl_host_words(&words));
  int64_t* h = (int64_t*)words;
  h[4] = 0;
  const int id_bits = bits_for(num_nodes > 0 ? (uint64_t)(num_nodes - 1) : 0);
  int pos_bits = 0;
  while (((m - 1) >> pos_bits) != 0) ++pos_bits;
  {
    LaunchScope scope(stream);
    SGL_CHECK_RC(zero_async(d_scan, sizeof(InputScan), stream));
    // (the mini-batch sort gathers through the position anyway: its scan leaves the ids alone)
    SGL_CHECK_RC(launch(tcsr_scan_kernel, stream_grid(m, kScanThreads * 4, 8), kScanThreads, 0, stream, key, nbr, ts, eid, m, num_nodes, small ? 0 : 1,
                        d_scan, h));
    // 160,000 edges: 14 of 49 us passed between the scan and a sort that waited for the host to know its result.
    if (small) {
      const EdgeKey k{key, ts, 0, 0};
      const ScannedRange range{d_scan, id_bits, pos_bits};
      SGL_CHECK_RC(sort_list(EdgeSource{k, m, range}, EdgeSink{k, nbr, eid, num_nodes, indptr, out_nbr, out_ts, out_eid, out_perm, range, false}, m,
                             64 - pos_bits, rest, rest_bytes, nullptr, stream));
      if (out_fence && num_nodes > 0) SGL_CHECK_RC(launch_fence(indptr, out_ts, num_nodes, m, out_fence, range, stream));
    }
    SGL_CHECK_RC(scope.submit());
  }
  SGL_CHECK_RC(sgl_wait_word(h + 4, 1, stream));
  const long long ts_min = h[0], ts_max = h[1];
  const unsigned long long bad = (unsigned long long)h[2], flags = (unsigned long long)h[3];
  SGL_REQUIRE(bad == 0, SGL_ERR_RANGE, "tcsr_build: %llu edge keys outside [0, %lld)", bad, (long long)num_nodes);
  if (h_ts_range) {
    h_ts_range[0] = ts_min;
    h_ts_range[1] = ts_max;
  }
  const int ts_bits = bits_for((uint64_t)ts_max - (uint64_t)ts_min);
  if (small && ts_bits + id_bits + pos_bits <= 64) return SGL_OK;
  const EdgeKey k{key, ts, ts_min, ts_bits};
  const int grid = stream_grid(m, 256 * 4, 8);
  // Neighbour and edge id as payload, as far as the scan saw; the sort's counts see all ids, and where some do not fit the passes behind them
  // do nothing and the host starts over with positions (a wide id in the middle of 2 M edges in no order: 250 us, at either end 200, with the
  // edges sorted before anybody asked 393; 50 M edges 5.68, 5.23, 8.36 ms).
  bool narrow = !small && ts_bits + id_bits <= 64 && !(flags & kWideIds) && out_perm == nullptr && num_nodes <= ((int64_t)1 << 32);
  for (;;) {
    LaunchScope scope(stream);
    WsCarver c(rest, rest_bytes);
    if (ts_bits + id_bits > 64) {
      // two stable rounds: by timestamp, then by node id
      uint64_t *k0 = c.take<uint64_t>(m), *k1 = c.take<uint64_t>(m);
      uint32_t *v0 = c.take<uint32_t>(m), *v1 = c.take<uint32_t>(m);
      const size_t sort_bytes = radix_sort_ws_bytes(m);
      char* sort_ws = c.take<char>(sort_bytes);
      SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "tcsr_build: workspace too small");
      SGL_CHECK_RC(launch(tcsr_round_keys_kernel, grid, 256, 0, stream, k, nullptr, m, k0));
      int in_alt = 0;
      SGL_CHECK_RC(radix_sort_pairs(k0, v0, k1, v1, m, nullptr, ts_bits, true, &in_alt, d_status, sort_ws, sort_bytes, stream));
      uint32_t *perm = in_alt ? v1 : v0, *other = in_alt ? v0 : v1;
      uint64_t *kk = in_alt ? k1 : k0, *kk_alt = in_alt ? k0 : k1;     // (the sorted timestamps are no longer needed)
      SGL_CHECK_RC(launch(tcsr_round_keys_kernel, grid, 256, 0, stream, k, perm, m, kk));
      SGL_CHECK_RC(radix_sort_pairs(kk, perm, kk_alt, other, m, nullptr, id_bits, false, &in_alt, d_status, sort_ws, sort_bytes, stream));
      SGL_CHECK_RC(launch(tcsr_emit_gather_kernel, grid, 256, 0, stream, d_scan, in_alt ? kk_alt : kk, in_alt ? other : perm, 0, k, nbr, eid, m,
                          num_nodes, indptr, out_nbr, out_ts, out_eid, out_perm));
    } else if (small) {
      const ScannedRange known{nullptr, 0, 0};
      SGL_CHECK_RC(sort_list(EdgeSource{k, m, known}, EdgeSink{k, nbr, eid, num_nodes, indptr, out_nbr, out_ts, out_eid, out_perm, known, false}, m,
                             ts_bits + id_bits, rest, rest_bytes, nullptr, stream));
    } else {
      const int first_bit = flags & kUnordered ? 0 : (ts_bits < 56 ? ts_bits : 56);   // in time order: only the node bits are left
      bool in_first;
      unsigned int* gave_up;
      if (narrow) {
        uint64_t *k1 = c.take<uint64_t>(m), *k0 = c.take<uint64_t>(m), *v1 = c.take<uint64_t>(m), *v0 = c.take<uint64_t>(m);
        uint32_t* node = (uint32_t*)(lsd_passes(first_bit, ts_bits + id_bits) & 1 ? k1 : k0);      // the last pass's own array
        const EdgeOut out{k, node, out_nbr, out_ts, out_eid};
        SGL_CHECK_RC((lsd_sort<uint64_t, EdgePairs>(EdgePairs{k, nbr, eid, m, d_scan}, k1, v1, k0, v0, m, nullptr, nullptr, first_bit, ts_bits + id_bits, out,
                                                    &in_first, &gave_up, c, d_status, stream)));
        SGL_CHECK_RC(launch(tcsr_rows_kernel, stream_grid(m, 256 * 4, 8), 256, 0, stream, d_scan, node, m, num_nodes, indptr));
      } else {
        uint64_t *k1 = c.take<uint64_t>(m), *k0 = c.take<uint64_t>(m);
        uint32_t *v1 = c.take<uint32_t>(m), *v0 = c.take<uint32_t>(m);
        SGL_CHECK_RC((lsd_sort<uint32_t, EdgePositions>(EdgePositions{k, m}, k1, v1, k0, v0, m, nullptr, nullptr, first_bit, ts_bits + id_bits,
                                                        ArrayOut<uint32_t>{}, &in_first, &gave_up, c, d_status, stream)));
        SGL_CHECK_RC(launch(tcsr_emit_gather_kernel, grid, 256, 0, stream, d_scan, in_first ? k1 : k0, in_first ? v1 : v0, 1, k, nbr, eid, m, num_nodes,
                            indptr, out_nbr, out_ts, out_eid, out_perm));
      }
    }
    if (out_fence && num_nodes > 0) SGL_CHECK_RC(launch_fence(indptr, out_ts, num_nodes, m, out_fence, {nullptr, 0, 0}, stream));
    if (small) return scope.submit();
    // The radix passes wait for each other's tiles, for a limited time: the graph is handed out once they are known to have come through.
    int64_t* const result = h + 8;
    constexpr int kStatus = (offsetof(InputScan, status) - offsetof(InputScan, flags)) / 8;
    SGL_CHECK_RC(export_words((const int64_t*)&d_scan->flags, result, kStatus + 1, stream));
    SGL_CHECK_RC(scope.submit());
    SGL_CHECK_RC(sgl_wait_word(result + kStatus + 1, 1, stream));
    SGL_REQUIRE(result[kStatus] == 0, SGL_ERR_CUDA, "tcsr_build: a look-back over the tiles of the sort ran into its time limit");
    if (!narrow || !(result[0] & (int64_t)kWideIds)) return SGL_OK;
    narrow = false;
  }
}

extern "C" int sgl_tcsr_build(int64_t num_nodes, int64_t m, const int64_t* key, const int64_t* nbr, const int64_t* ts, const int64_t* eid,
                              int64_t* indptr, int64_t* out_nbr, int64_t* out_ts, int64_t* out_eid, int64_t* out_perm,
                              int64_t* h_ts_range, void* ws, size_t ws_bytes, void* stream) {
  return sgl_tcsr_build_fenced(num_nodes, m, key, nbr, ts, eid, indptr, out_nbr, out_ts, out_eid, out_perm, nullptr, h_ts_range, ws, ws_bytes,
                               stream);
}

// ---------------------------------------------------------------------------------------------------------------
// Search index over the time-sorted rows ("fence"): for every block of 32 consecutive edges of a row the timestamp of
// the block's last edge.  Row r (edges [s, e)) owns the entries fence[(s >> 5) + r + j], j < ceil((e - s) / 32) -- a
// placement that needs no pointer array of its own: consecutive rows never overlap because
// floor((s + d) / 32) - floor(s / 32) >= ceil(d / 32) - 1.  About 1.6 % of the adjacency's size, so it stays in L2 while
// the timestamps themselves (8 bytes per edge) do not; a time-range search walks the fence and then reads ONE block of
// the row.
// ---------------------------------------------------------------------------------------------------------------
namespace sgl {
namespace {
// The row of fence entry x is the last r with (indptr[r] >> 5) + r <= x; that start position is strictly increasing in r, so kSpan
// consecutive entries lie in at most kSpan consecutive rows.  A CTA finds the first of them with one 32-ary search, fetches the row
// pointers in one go and looks every entry up in shared memory; a hub row's tens of thousands of entries have as many threads.
// Bound by latency below 300,000 entries (a binary search of the row pointer per entry was up to 20 dependent loads: 160,000 edges of
// 10,000 nodes 7.1 us, now 5.0), above by the sector that is read for every 32nd timestamp (50 M edges of 1 M nodes 70 us, now 50).
constexpr int kFenceThreads = 256;
template <int kPer>
__global__ void __launch_bounds__(kFenceThreads)
tcsr_fence_kernel(const int64_t* __restrict__ indptr, const int64_t* __restrict__ ts, int64_t num_nodes, int64_t len,
                  int64_t* __restrict__ fence, const ScannedRange range) {
  constexpr int kSpan = kFenceThreads * kPer;
  __shared__ int64_t s_ptr[kSpan + 1], s_row;
  EdgeKey unused{};
  if (!range.read(unused)) return;
  const int tid = threadIdx.x, lane = tid & 31;
  for (int64_t x0 = (int64_t)blockIdx.x * kSpan; x0 < len; x0 += (int64_t)gridDim.x * kSpan) {
    if (tid < 32) {
      int64_t lo = 0, hi = num_nodes;      // invariant: start(lo) <= x0; rows >= hi start after x0
      while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) >> 5, mid = lo + (lane + 1) * step;
        const bool upto = mid < hi && (__ldg(indptr + mid) >> 5) + mid <= x0;
        const int c = __popc(__ballot_sync(0xffffffffu, upto));
        const int64_t end = lo + (c + 1) * step;
        hi = end < hi ? end : hi;
        lo += c * step;
      }
      if (lane == 0) s_row = lo;
    }
    __syncthreads();
    const int64_t r0 = s_row;
    const int rows = num_nodes - r0 < kSpan ? (int)(num_nodes - r0) : kSpan;
#pragma unroll
    for (int j = tid; j <= kSpan; j += kFenceThreads)
      if (j <= rows) s_ptr[j] = __ldg(indptr + r0 + j);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int64_t x = x0 + u * kFenceThreads + tid;
      if (x >= len) break;
      int lo = 0, hi = rows;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if ((s_ptr[mid] >> 5) + r0 + mid <= x) lo = mid; else hi = mid;
      }
      const int64_t s = s_ptr[lo], e = s_ptr[lo + 1], j = x - ((s >> 5) + r0 + lo);
      if (j < ((e - s + 31) >> 5)) {
        const int64_t last = s + (j << 5) + 31;
        fence[x] = __ldg(ts + (last < e ? last : e - 1));
      }
    }
    __syncthreads();
  }
}

int launch_fence(const int64_t* indptr, const int64_t* ts, int64_t num_nodes, int64_t m, int64_t* out_fence, const ScannedRange& range,
                 cudaStream_t stream) {
  const int64_t len = sgl_tcsr_fence_len(num_nodes, m);
  // (four entries a thread once that leaves every SM its eight CTAs)
  if (len < (int64_t)kNumSM * 8 * kFenceThreads * 4)
    return launch(tcsr_fence_kernel<1>, stream_grid(len, kFenceThreads, 16), kFenceThreads, 0, stream, indptr, ts, num_nodes, len, out_fence, range);
  return launch(tcsr_fence_kernel<4>, stream_grid(len, kFenceThreads * 4, 16), kFenceThreads, 0, stream, indptr, ts, num_nodes, len, out_fence, range);
}
}  // namespace
}  // namespace sgl

extern "C" int64_t sgl_tcsr_fence_len(int64_t num_nodes, int64_t m) { return (m >> 5) + num_nodes + 1; }

extern "C" int sgl_tcsr_fence(const int64_t* indptr, const int64_t* ts, int64_t num_nodes, int64_t m, int64_t* out_fence,
                              void* stream_) {
  SGL_REQUIRE(num_nodes >= 0 && m >= 0, SGL_ERR_ARG, "tcsr_fence: negative size");
  if (num_nodes == 0 || m == 0) return SGL_OK;
  SGL_REQUIRE(indptr && ts && out_fence, SGL_ERR_ARG, "tcsr_fence: null array");
  return launch_fence(indptr, ts, num_nodes, m, out_fence, {nullptr, 0, 0}, (cudaStream_t)stream_);
}
