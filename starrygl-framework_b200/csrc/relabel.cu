// Dedup / relabel kernels of the mini-batch builder.  Everything is sort based so that local ids come out in
// the deterministic order the CPU builder produces (sorted unique), not in hash-table order:
//
// key = (id << ts_bits) | (ts - ts_base), stable sort, numbers of the distinct keys -> unique list and inverse map, with the
// producer of the keys and the consumer of the order fused into the sort (lists.cuh, sort_list in lsd.cuh).
//
// Algorithmic HBM bytes: 16 read + 8 write per input pair, 16 per unique pair, plus the sort passes
// (32 B per pair and populated key byte).
#include <limits.h>

#include "launch.cuh"
#include "sort.cuh"
#include "lists.cuh"
#include "lsd.cuh"
#include "rowcsc.cuh"

namespace sgl {
namespace {

constexpr int kThreads = 256;

// CSC of edges that already are in (dst, ts) order -- the first hop of a batch, whose targets are the layer list
// itself: target i is row i, and a target's samples come out in ascending time.  No sort: a copy plus the row pointer.
__global__ void __launch_bounds__(kThreads)
csc_emit_sorted_kernel(const int64_t* __restrict__ dst, int64_t n_cap, const int64_t* d_n, int64_t num_dst_cap,
                       const int64_t* d_num_dst, const int64_t* __restrict__ src_local, const int64_t* __restrict__ ts,
                       const float* __restrict__ dt, const int64_t* __restrict__ eid, int64_t* __restrict__ indptr,
                       int64_t* __restrict__ out_indices, int64_t* __restrict__ out_ts, float* __restrict__ out_dt,
                       int64_t* __restrict__ out_eid, int32_t* d_status) {
  const int64_t n = eff_count(n_cap, d_n);
  const int64_t num_dst = eff_count(num_dst_cap, d_num_dst);
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  if (n == 0) {
    for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v <= num_dst; v += stride) indptr[v] = 0;
    return;
  }
  for (int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x; j < n; j += stride) {
    out_indices[j] = src_local[j];
    out_ts[j] = ts[j];
    out_dt[j] = dt[j];
    out_eid[j] = eid[j];
    const int64_t d = dst[j];
    const int64_t prev = j == 0 ? -1 : dst[j - 1];
    if (d < prev || d < 0 || (d == prev && ts[j] < ts[j - 1])) dev_flag(d_status, SGL_DEV_BAD_INDEX);   // not in (dst, ts) order
    for (int64_t v = prev + 1; v <= d && v <= num_dst; ++v) indptr[v] = j;
    if (j == n - 1)
      for (int64_t v = d + 1; v <= num_dst; ++v) indptr[v] = n;
  }
}

// CSC by sort; gate: see CscSource
int csc_sort(const int64_t* src_local, const int64_t* dst, const int64_t* dst_map, const int64_t* ts, const float* dt, const int64_t* eid,
             int64_t n_edges, const int64_t* d_n_edges, int64_t num_dst, const int64_t* d_num_dst, int dst_bits, int ts_bits, int64_t ts_base,
             int64_t* out_indptr, int64_t* out_indices, int64_t* out_ts, float* out_dt, int64_t* out_eid, const int* gate, int32_t* d_status,
             void* ws, size_t ws_bytes, cudaStream_t stream) {
  return sort_list(CscSource{dst, dst_map, ts, d_n_edges, n_edges, dst_bits, ts_bits, ts_base, gate, d_status},
                   CscSink{num_dst, d_num_dst, ts_bits, src_local, ts, dt, eid, out_indptr, out_indices, out_ts, out_dt, out_eid, gate},
                   n_edges < 1 ? 1 : n_edges, dst_bits + ts_bits, ws, ws_bytes, d_status, stream);
}

// ---- CSC in list order (rowcsc.cuh) --------------------------------------------------------------------------------------
constexpr int kRowItems = 8;             // list items per thread of the count kernel
constexpr int kRowTile = kThreads * kRowItems;
constexpr int64_t kMaxRowTargets = 32;
constexpr int kMapFanout = 32;
inline int64_t rows_ctas(int64_t cap) { return (cap + kRowTile - 1) / kRowTile < 1 ? 1 : (cap + kRowTile - 1) / kRowTile; }

// start[at]: edges of the items before `at` in its tile; sums: edges before the tile; from[at]: first edge of the item, and their number
// (32 bits each: build_csc_rows takes fewer than 2^32 edges).
// Targets of `drawn` or more edges may have drawn them.
__global__ void __launch_bounds__(kThreads)
csc_rows_count_kernel(const RowOrder ro, const int64_t* d_rows, const int64_t* __restrict__ offsets, int drawn, uint32_t* __restrict__ start,
                      uint2* __restrict__ from, int64_t* sums, unsigned int* done, int* gate) {
  __shared__ uint32_t s_w[kThreads / 32];
  const int64_t n = ro.first[*d_rows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t first = (int64_t)blockIdx.x * kRowTile + warp * (32 * kRowItems) + lane;
  uint32_t o[kRowItems], c[kRowItems];
  bool crowded = false;
#pragma unroll
  for (int r = 0; r < kRowItems; ++r) {
    const int64_t at = first + r * 32;
    o[r] = at < n ? ro.order[at] : ~0u;
  }
#pragma unroll
  for (int r = 0; r < kRowItems; ++r) {
    const int64_t at = first + r * 32;
    uint2 f = make_uint2(0u, 0u);
    if (o[r] != ~0u) {
      const int64_t a = offsets[o[r]];
      f = make_uint2((uint32_t)a, (uint32_t)(offsets[o[r] + 1] - a));
    }
    c[r] = f.y;
    if (at < n) from[at] = f;
  }
#pragma unroll
  for (int r = 0; r < kRowItems; ++r) {
    const int64_t at = first + r * 32;
    if (c[r] >= (uint32_t)drawn && at + kMaxRowTargets < n) crowded |= ro.row[at] == ro.row[at + kMaxRowTargets];
  }
  uint32_t carry = 0;
#pragma unroll
  for (int r = 0; r < kRowItems; ++r) {
    const uint32_t x = warp_inclusive_scan(c[r], lane), own = c[r];
    c[r] = carry + x - own;
    carry += __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) s_w[warp] = carry;
  if (crowded) *gate = 1;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    if (w < warp) before += s_w[w];
    total += s_w[w];
  }
#pragma unroll
  for (int r = 0; r < kRowItems; ++r)
    if (first + r * 32 < n) start[first + r * 32] = before + c[r];
  publish_and_scan_cta_totals<kThreads>((int64_t)total, sums, done, nullptr);
}

// Edges of kThreads list items; consecutive threads take consecutive edges.  Bound by sectors: a target's few edges lie anywhere in every
// array that they are read from, so where they start comes in list order from the count, and the time difference is that of the row's
// time (row_ts) instead of a read of its own (10 M edges of 4.2 M targets: 290 us, so 214, next to
// the digit counts of the next list).
__global__ void __launch_bounds__(kThreads)
csc_rows_copy_kernel(const RowOrder ro, const int64_t* d_rows, const int64_t* __restrict__ row_ts, const int64_t* __restrict__ offsets,
                     const uint2* __restrict__ from, const int64_t* __restrict__ ts, const int64_t* __restrict__ eid, int fanout, int drawn,
                     const uint32_t* __restrict__ start,
                     const int64_t* __restrict__ sums, const int* gate, int64_t* __restrict__ indptr, int64_t* __restrict__ indices,
                     int64_t* __restrict__ out_ts, float* __restrict__ out_dt, int64_t* __restrict__ out_eid) {
  extern __shared__ uint8_t s_map[];       // item of every edge (fan-outs up to kMapFanout)
  __shared__ int s_ex[kThreads + 1];
  __shared__ int64_t s_src[kThreads], s_to[kThreads], s_t[kThreads];
  __shared__ uint32_t s_q0[kThreads], s_q1[kThreads];
  if (*gate) return;
  const int64_t rows = *d_rows, n = ro.first[rows];
  const int tid = threadIdx.x;
  const int64_t first = (int64_t)blockIdx.x * kThreads, at = first + tid;
  if (n == 0 && at == 0) indptr[0] = 0;
  if (first >= n) return;
  int c = 0;
  if (at < n) {
    const uint2 f = from[at];
    const uint32_t u = ro.row[at], q0 = ro.first[u], q1 = ro.first[u + 1];
    const int64_t begin = sums[q0 / kRowTile] + start[q0];
    c = (int)f.y;
    s_src[tid] = (int64_t)f.x;
    s_t[tid] = row_ts[u];
    s_to[tid] = begin;
    s_q0[tid] = q0;
    s_q1[tid] = q1;
    if (q0 == at) indptr[u] = begin;
    if (at == n - 1) indptr[rows] = sums[at / kRowTile] + start[at] + c;
  }
  int total;
  const int ex = cta_exclusive_scan<kThreads, int>(c, &total);
  const bool has_map = fanout <= kMapFanout;
  s_ex[tid] = ex;
  if (tid == kThreads - 1) s_ex[kThreads] = total;
  if (has_map)
    for (int j = 0; j < c; ++j) s_map[ex + j] = (uint8_t)tid;
  __syncthreads();
  for (int o = tid; o < total; o += kThreads) {
    int k;
    if (has_map) {
      k = s_map[o];
    } else {
      int b = kThreads;                    // last item with s_ex[item] <= o
      k = 0;
      while (b - k > 1) {
        const int m = (k + b) >> 1;
        if (s_ex[m] <= o) k = m; else b = m;
      }
    }
    const int j = o - s_ex[k];
    const int64_t e = s_src[k] + j, t = ts[e];
    const float d = (float)(s_t[k] - t);
    const int64_t id = eid[e];
    int64_t to = s_to[k] + j;
    const uint32_t me = (uint32_t)(first + k), q0 = s_q0[k], q1 = s_q1[k];
    if (s_ex[k + 1] - s_ex[k] < drawn) {
      // the row's targets have this same list: before the edge come the earlier ones of every target, the equal ones of the targets
      // before, and its own equal ones before it
      const uint32_t others = ro.order[q0] == ~0u ? q0 + 1 : q0;         // the row's first target
      if (q1 - others > 1) {
        const int64_t end = s_src[k] + s_ex[k + 1] - s_ex[k];
        int64_t lo = e, hi = e + 1;
        while (lo > s_src[k] && __ldg(ts + lo - 1) == t) --lo;
        while (hi < end && __ldg(ts + hi) == t) ++hi;
        to += (lo - s_src[k]) * (int64_t)(q1 - others - 1) + (hi - lo) * (int64_t)(me - others);
      }
    } else for (uint32_t q = q0; q < q1; ++q) {
      if (q == me) continue;
      const uint32_t other = ro.order[q];
      if (other == ~0u) continue;
      // edges of the other target before this one: earlier ones, and equal ones of an earlier target
      const int64_t s0 = __ldg(offsets + other);
      int64_t a = s0, b = __ldg(offsets + other + 1);
      while (a < b) {
        const int64_t mid = (a + b) >> 1, x = __ldg(ts + mid);
        if (x < t || (x == t && q < me)) a = mid + 1; else b = mid;
      }
      to += a - s0;
    }
    indices[to] = e;
    out_ts[to] = t;
    out_dt[to] = d;
    out_eid[to] = id;
  }
}

// ---- node relabel by bitmap ----------------------------------------------------------------------------------------------
// Ids without a time need no sort: the new ones of a list are marked in a bitmap of the nodes, their ascending order is the bitmap's, and
// an entry's local id is its node's.  Three kernels of 2 - 5 us; kernels of a list, the sort -> the bitmap (entries over 50,000 nodes, all
// nodes alike / a power law with its hubs next to each other / one node): 2,049 entries 21 -> 11 us; 20,000 24 / 24 / 26 -> 12 / 13 / 10;
// 80,000 31 / 31 / 38 -> 17 / 20 / 12; 300,000 54 / 56 / 75 -> 30 / 43 / 17; 1.2 M 250 / 234 / 224 -> 78 / 107 / 37; 4 M 208 / 198 / 161 ->
// 145 / 223 / 62.  Over 2^19 nodes: 2,049 entries 21 -> 13, 80,000 33 / 32 / 38 -> 15 / 22 / 14, 4 M 250 / 238 / 201 -> 95 / 218 / 64.
// A CTA of the middle kernel counts the marks before its own by itself, so the bitmap is bounded: 2^19 nodes are 64 KB, at most 64 loads a
// thread; up to 2,048 entries one CTA sorts in a single launch.
constexpr int64_t kBitmapNodes = 1 << 19;
static_assert(kBitmapNodes / 8 <= tilesort::kMatrix * 4, "the bitmap lies in the scratch of a sort");
inline bool by_bitmap(int64_t n, int64_t num_nodes) { return n > tilesort::kSingleMax && num_nodes > 0 && num_nodes <= kBitmapNodes; }

// Lists have hubs, and an atomic on a hot word takes 0.65 ns: lanes of a warp that share a word set their marks together (looked for only
// where some of 48 pairs of lanes do), and a mark that is there already is not set again (one atomic per entry: 300,000 entries 133 us with
// a power law, 202 us of one node; 4 M entries 1.6 and 2.6 ms).
__global__ void __launch_bounds__(kThreads)
nodes_mark_kernel(const int64_t* __restrict__ ids, int64_t n_cap, const int64_t* d_n, int64_t num_nodes, const int64_t* __restrict__ mask,
                  int64_t epoch, uint32_t* bits, int32_t* d_status) {
  __shared__ uint32_t s_marks[kThreads];   // of the lanes that share a word, at the first of them
  const int64_t n = eff_count(n_cap, d_n), stride = (int64_t)gridDim.x * kThreads;
  const int lane = threadIdx.x & 31;
  uint32_t* const marks = s_marks + (threadIdx.x & ~31);
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i - lane < n; i += stride) {
    int word = -1;
    uint32_t mark = 0;
    if (i < n) {
      const int64_t g = ids[i];
      if (g < 0 || g >= num_nodes) {
        dev_flag(d_status, SGL_DEV_BAD_NODE);
      } else {
        // (not in the first round: there is nothing to find, and reading behind everybody's marks took 2 of 7 us)
        const uint32_t there = i >= stride ? __ldcg(bits + (g >> 5)) : 0u, own = 1u << (g & 31);
        if (mask[g] != epoch && !(there & own)) {
          word = (int)(g >> 5);
          mark = own;
        }
      }
    }
    const int w16 = __shfl_xor_sync(0xffffffffu, word, 16), w8 = __shfl_xor_sync(0xffffffffu, word, 8), w4 = __shfl_xor_sync(0xffffffffu, word, 4);
    if (__any_sync(0xffffffffu, word >= 0 && (word == w16 || word == w8 || word == w4))) {
      const int first = __ffs(__match_any_sync(0xffffffffu, word)) - 1;
      marks[lane] = 0;
      __syncwarp();
      if (word >= 0) atomicOr(marks + first, mark);
      __syncwarp();
      mark = marks[lane];
      if (lane != first) word = -1;
      __syncwarp();
    }
    if (word >= 0) atomicOr(bits + word, mark);
  }
}

// a thread takes eight nodes
__global__ void __launch_bounds__(kThreads)
nodes_emit_kernel(const uint32_t* __restrict__ bits, int words, int64_t* __restrict__ mapper, int64_t* __restrict__ mask, int64_t epoch,
                  const int64_t* d_next_local, int64_t* out_new_ids, int64_t* d_n_new, const int64_t* d_start) {
  const int first = blockIdx.x * (kThreads / 4), tid = threadIdx.x, w = first + (tid >> 2);
  uint32_t mine = w < words ? (bits[w] >> ((tid & 3) * 8)) & 0xffu : 0u;
  int before = 0;
#pragma unroll 8
  for (int j = tid; j < first; j += kThreads) before += __popc(bits[j]);
  const int64_t next = *d_next_local;
  if (d_start) out_new_ids += next - *d_start;
  int earlier, total;
  cta_exclusive_scan<kThreads, int>(before, &earlier);
  int64_t u = earlier + cta_exclusive_scan<kThreads, int>(__popc(mine), &total);
  if (blockIdx.x == gridDim.x - 1 && tid == 0) *d_n_new = earlier + total;
  for (; mine; mine &= mine - 1, ++u) {
    const int64_t g = (int64_t)w * 32 + (tid & 3) * 8 + (__ffs(mine) - 1);
    mapper[g] = next + u;
    mask[g] = epoch;
    out_new_ids[u] = g;
  }
}

__global__ void __launch_bounds__(kThreads)
nodes_map_kernel(const int64_t* __restrict__ ids, int64_t n_cap, const int64_t* d_n, int64_t num_nodes, const int64_t* __restrict__ mapper,
                 int64_t* __restrict__ out_local, int64_t* d_next_local, const int64_t* d_n_new) {
  const int64_t n = eff_count(n_cap, d_n), stride = (int64_t)gridDim.x * kThreads;
  if (blockIdx.x == 0 && threadIdx.x == 0) *d_next_local += *d_n_new;
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += stride) {
    const int64_t g = ids[i];
    out_local[i] = g >= 0 && g < num_nodes ? __ldg(mapper + g) : -1;
  }
}

// first position with sorted[pos] >= value, one thread per value
__global__ void lower_bound_kernel(const int64_t* __restrict__ sorted, int64_t n, const int64_t* __restrict__ values,
                                   int k, int64_t* __restrict__ out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  int64_t v = values[i], lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = lo + ((hi - lo) >> 1);
    if (sorted[mid] < v) lo = mid + 1; else hi = mid;
  }
  out[i] = lo;
}


}  // namespace
}  // namespace sgl

using namespace sgl;

extern "C" size_t sgl_unique_pairs_ws_bytes(int64_t n_total) { return list_ws_bytes(n_total); }

int sgl::unique_pairs(const int64_t* a_id, const int64_t* a_ts, int64_t n_a, const int64_t* d_n_a,
                                const int64_t* b_id, const int64_t* b_ts, int64_t n_b, const int64_t* d_n_b, int id_bits,
                                int ts_bits, int64_t ts_base, int64_t* out_id, int64_t* out_ts, int64_t* inv_a,
                                int64_t* inv_b, uint32_t* inv_b32, int64_t* d_n_unique, const RowOrder& ro, int32_t* d_status, void* ws,
                                size_t ws_bytes, void* stream_) {
  SGL_NVTX("sgl_unique_pairs");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_a >= 0 && n_b >= 0, SGL_ERR_ARG, "unique_pairs: negative size");
  SGL_REQUIRE(id_bits >= 0 && ts_bits >= 0 && id_bits + ts_bits <= 64, SGL_ERR_UNSUPPORTED,
              "unique_pairs: id_bits %d + ts_bits %d exceed the 64-bit sort key", id_bits, ts_bits);
  SGL_REQUIRE(d_n_unique, SGL_ERR_ARG, "unique_pairs: d_n_unique is null");
  const int64_t n = n_a + n_b;
  if (n == 0) {
    SGL_CHECK_RC(zero_async(d_n_unique, sizeof(int64_t), stream));
    if (ro.first) SGL_CHECK_RC(zero_async(ro.first, sizeof(uint32_t), stream));
    return SGL_OK;
  }
  SGL_REQUIRE((n_a == 0 || (a_id && a_ts)) && (n_b == 0 || (b_id && b_ts)) && out_id && out_ts, SGL_ERR_ARG,
              "unique_pairs: null array");
  LaunchScope scope(stream);
  SGL_CHECK_RC(sort_list(PairSource{a_id, a_ts, d_n_a, b_id, b_ts, d_n_b, n_a, n_b, id_bits, ts_bits, ts_base, d_status},
                         PairSink{n_a, d_n_a, ts_bits, ts_base, out_id, out_ts, inv_a, inv_b, d_n_unique, ro.order, ro.row, ro.first, inv_b32}, n,
                         id_bits + ts_bits, ws, ws_bytes, d_status, stream));
  return scope.submit();
}

extern "C" int sgl_unique_pairs(const int64_t* a_id, const int64_t* a_ts, int64_t n_a, const int64_t* d_n_a, const int64_t* b_id,
                                const int64_t* b_ts, int64_t n_b, const int64_t* d_n_b, int id_bits, int ts_bits, int64_t ts_base,
                                int64_t* out_id, int64_t* out_ts, int64_t* inv_a, int64_t* inv_b, int64_t* d_n_unique, int32_t* d_status,
                                void* ws, size_t ws_bytes, void* stream) {
  return unique_pairs(a_id, a_ts, n_a, d_n_a, b_id, b_ts, n_b, d_n_b, id_bits, ts_bits, ts_base, out_id, out_ts, inv_a, inv_b, nullptr,
                      d_n_unique, RowOrder{}, d_status, ws, ws_bytes, stream);
}

extern "C" size_t sgl_build_csc_ws_bytes(int64_t n_edges, int64_t num_dst) {
  (void)num_dst;
  return list_ws_bytes(n_edges);
}

extern "C" int sgl_build_csc(const int64_t* src_local, const int64_t* dst, const int64_t* dst_map, const int64_t* ts,
                             const float* dt, const int64_t* eid, int64_t n_edges, const int64_t* d_n_edges,
                             int64_t num_dst, const int64_t* d_num_dst, int dst_bits, int ts_bits, int64_t ts_base,
                             int64_t* out_indptr, int64_t* out_indices, int64_t* out_ts, float* out_dt, int64_t* out_eid,
                             int presorted, int32_t* d_status, void* ws, size_t ws_bytes, void* stream_) {
  SGL_NVTX("sgl_build_csc");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_edges >= 0 && num_dst >= 0, SGL_ERR_ARG, "build_csc: negative size");
  if (presorted) {
    SGL_REQUIRE(dst_map == nullptr, SGL_ERR_ARG, "build_csc: presorted input cannot go through a dst_map");
    SGL_REQUIRE(out_indptr, SGL_ERR_ARG, "build_csc: out_indptr is null");
    SGL_REQUIRE(n_edges == 0 || (src_local && dst && ts && dt && eid && out_indices && out_ts && out_dt && out_eid), SGL_ERR_ARG,
                "build_csc: null array");
    const int64_t work_s = n_edges > num_dst + 1 ? n_edges : num_dst + 1;
    SGL_CHECK_RC(launch(csc_emit_sorted_kernel, stream_grid(work_s, kThreads, 16), kThreads, 0, stream, dst, n_edges,
                        d_n_edges, num_dst, d_num_dst, src_local, ts, dt, eid, out_indptr, out_indices, out_ts, out_dt,
                        out_eid, d_status));
    return SGL_OK;
  }
  SGL_REQUIRE(dst_bits >= 0 && ts_bits >= 0 && dst_bits + ts_bits <= 64, SGL_ERR_UNSUPPORTED,
              "build_csc: dst_bits %d + ts_bits %d exceed the 64-bit sort key", dst_bits, ts_bits);
  SGL_REQUIRE(out_indptr, SGL_ERR_ARG, "build_csc: out_indptr is null");
  SGL_REQUIRE(n_edges == 0 || (dst && ts && dt && eid && out_indices && out_ts && out_dt && out_eid), SGL_ERR_ARG,
              "build_csc: null array");
  LaunchScope scope(stream);
  SGL_CHECK_RC(csc_sort(src_local, dst, dst_map, ts, dt, eid, n_edges, d_n_edges, num_dst, d_num_dst, dst_bits, ts_bits, ts_base, out_indptr,
                        out_indices, out_ts, out_dt, out_eid, nullptr, d_status, ws, ws_bytes, stream));
  return scope.submit();
}

size_t sgl::build_csc_rows_ws_bytes(int64_t n_edges, int64_t list_cap) {
  return align_up((size_t)list_cap * 4) + align_up((size_t)list_cap * sizeof(uint2)) + align_up((size_t)rows_ctas(list_cap) * 8) + align_up(8) +
         list_ws_bytes(n_edges);
}

int sgl::build_csc_rows(const RowOrder& ro, int64_t list_cap, const int64_t* row_ts, const int64_t* offsets, int fanout, bool draws,
                        const int64_t* dst, const int64_t* dst_map, const int64_t* ts, const float* dt, const int64_t* eid, int64_t n_edges,
                        const int64_t* d_n_edges, int64_t num_dst, const int64_t* d_num_dst, int dst_bits, int ts_bits, int64_t ts_base, int64_t* out_indptr, int64_t* out_indices,
                        int64_t* out_ts, float* out_dt, int64_t* out_eid, int32_t* d_status, void* ws, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  // (list items and, in `from`, first edges of targets are 32-bit words; the sort of a row with too many targets has the same limit)
  SGL_REQUIRE(n_edges >= 0 && n_edges < ((int64_t)1 << 32) && list_cap < ((int64_t)1 << 32), SGL_ERR_UNSUPPORTED,
              "build_csc: %lld edges of %lld list items need 64-bit positions", (long long)n_edges, (long long)list_cap);
  SGL_REQUIRE(dst_bits >= 0 && ts_bits >= 0 && dst_bits + ts_bits <= 64, SGL_ERR_UNSUPPORTED,
              "build_csc: dst_bits %d + ts_bits %d exceed the 64-bit sort key", dst_bits, ts_bits);
  LaunchScope scope(stream);
  WsCarver c(ws, ws_bytes);
  uint32_t* start = c.take<uint32_t>(list_cap);
  uint2* from = c.take<uint2>(list_cap);
  const int64_t ctas = rows_ctas(list_cap);
  int64_t* sums = c.take<int64_t>(ctas);
  unsigned int* words = c.take<unsigned int>(2);           // arrivals, gate
  const size_t sort_bytes = list_ws_bytes(n_edges);
  char* sort_ws = c.take<char>(sort_bytes);
  SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "build_csc: workspace %zu < %zu bytes", ws_bytes, build_csc_rows_ws_bytes(n_edges, list_cap));
  int* gate = (int*)(words + 1);
  SGL_CHECK_RC(zero_async(words, 8, stream));
  SGL_CHECK_RC(launch(csc_rows_count_kernel, (unsigned)ctas, kThreads, 0, stream, ro, d_num_dst, offsets, draws ? fanout : INT_MAX, start,
                      from, sums, words, gate));
  // the copy and the sort side by side: the gate lets one of them do something (the sort's kernels that find nothing to do took 8 us behind
  // the copy of 100,000 edges)
  LaunchScope* in = LaunchScope::current();
  cudaStream_t other = in ? (cudaStream_t)(uintptr_t)7 : stream;
  if (in) SGL_CHECK_RC(in->follow(other, stream));
  SGL_CHECK_RC(launch(csc_rows_copy_kernel, (unsigned)((list_cap + kThreads - 1) / kThreads), kThreads,
                      fanout <= kMapFanout ? (size_t)kThreads * fanout : 0, stream, ro, d_num_dst, row_ts, offsets, from, ts, eid, fanout,
                      draws ? fanout : INT_MAX, start, sums, gate, out_indptr, out_indices, out_ts, out_dt, out_eid));
  SGL_CHECK_RC(csc_sort(nullptr, dst, dst_map, ts, dt, eid, n_edges, d_n_edges, num_dst, d_num_dst, dst_bits, ts_bits, ts_base, out_indptr,
                        out_indices, out_ts, out_dt, out_eid, gate, d_status, sort_ws, sort_bytes, other));
  if (in) SGL_CHECK_RC(in->follow(stream, other));
  return scope.submit();
}

extern "C" size_t sgl_relabel_nodes_ws_bytes(int64_t n) { return list_ws_bytes(n); }

int sgl::check_relabel(int64_t n, int64_t num_nodes) {
  SGL_REQUIRE(n >= 0 && num_nodes >= 0, SGL_ERR_ARG, "relabel_nodes: negative size");
  SGL_REQUIRE(bits_for(num_nodes > 0 ? (uint64_t)(num_nodes - 1) : 0) < 63, SGL_ERR_UNSUPPORTED, "relabel_nodes: num_nodes too large");
  SGL_REQUIRE(by_bitmap(n, num_nodes) || n < ((int64_t)1 << 32), SGL_ERR_UNSUPPORTED, "relabel_nodes: %lld entries need a 64-bit position", (long long)n);
  return SGL_OK;
}

int sgl::relabel_nodes(const int64_t* ids, int64_t n, const int64_t* d_n, int64_t num_nodes, int64_t* mapper,
                                 int64_t* mask, int64_t epoch, int64_t* d_next_local, int64_t* out_local,
                                 int64_t* out_new_ids, int64_t* d_n_new, const int64_t* d_start, int32_t* d_status, void* ws, size_t ws_bytes,
                                 void* stream_) {
  SGL_NVTX("sgl_relabel_nodes");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_CHECK_RC(check_relabel(n, num_nodes));
  SGL_REQUIRE(d_next_local && d_n_new, SGL_ERR_ARG, "relabel_nodes: null counter");
  if (n == 0) {
    SGL_CHECK_RC(zero_async(d_n_new, sizeof(int64_t), stream));
    return SGL_OK;
  }
  SGL_REQUIRE(ids && mapper && mask && out_local && out_new_ids, SGL_ERR_ARG, "relabel_nodes: null array");
  const int id_bits = bits_for(num_nodes > 0 ? (uint64_t)(num_nodes - 1) : 0);
  LaunchScope scope(stream);
  if (by_bitmap(n, num_nodes)) {
    WsCarver c(ws, ws_bytes);
    const int words = (int)((num_nodes + 31) / 32);
    uint32_t* bits = c.take<uint32_t>(words);
    SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "relabel_nodes: workspace %zu < %zu bytes", ws_bytes, sgl_relabel_nodes_ws_bytes(n));
    const int grid = stream_grid(n, kThreads, 8);
    SGL_CHECK_RC(zero_async(bits, (size_t)words * 4, stream));
    SGL_CHECK_RC(launch(nodes_mark_kernel, grid, kThreads, 0, stream, ids, n, d_n, num_nodes, mask, epoch, bits, d_status));
    SGL_CHECK_RC(launch(nodes_emit_kernel, (words + kThreads / 4 - 1) / (kThreads / 4), kThreads, 0, stream, bits, words, mapper, mask, epoch,
                        d_next_local, out_new_ids, d_n_new, d_start));
    SGL_CHECK_RC(launch(nodes_map_kernel, grid, kThreads, 0, stream, ids, n, d_n, num_nodes, mapper, out_local, d_next_local, d_n_new));
    return scope.submit();
  }
  SGL_CHECK_RC(sort_list(NodesSource{ids, d_n, n, num_nodes, mask, epoch, id_bits, d_status},
                         NodesSink{ids, num_nodes, id_bits, mapper, mask, epoch, d_next_local, out_local, out_new_ids, d_n_new, d_start, 0},
                         n, id_bits + 1, ws, ws_bytes, d_status, stream));
  return scope.submit();
}

extern "C" int sgl_relabel_nodes(const int64_t* ids, int64_t n, const int64_t* d_n, int64_t num_nodes, int64_t* mapper,
                                 int64_t* mask, int64_t epoch, int64_t* d_next_local, int64_t* out_local,
                                 int64_t* out_new_ids, int64_t* d_n_new, int32_t* d_status, void* ws, size_t ws_bytes,
                                 void* stream) {
  return relabel_nodes(ids, n, d_n, num_nodes, mapper, mask, epoch, d_next_local, out_local, out_new_ids, d_n_new, nullptr, d_status, ws,
                       ws_bytes, stream);
}

extern "C" int sgl_lower_bound_i64(const int64_t* sorted, int64_t n, const int64_t* values, int k, int64_t* out,
                                   void* stream_) {
  SGL_REQUIRE(n >= 0 && k >= 0, SGL_ERR_ARG, "lower_bound: negative size");
  if (k == 0) return SGL_OK;
  SGL_REQUIRE((n == 0 || sorted) && values && out, SGL_ERR_ARG, "lower_bound: null array");
  SGL_CHECK_RC(launch(lower_bound_kernel, (k + 127) / 128, 128, 0, (cudaStream_t)stream_, sorted, n, values, k, out));
  return SGL_OK;
}

extern "C" size_t sgl_seeds_ws_bytes(int64_t n_events) { return align_up(8) + list_ws_bytes(n_events); }

extern "C" int sgl_seeds_in_window(const int64_t* ev_src, const int64_t* ev_ts, const int64_t* ev_eid, int64_t n_events,
                                   const int64_t* node_chunk, const uint8_t* chunk_mask, int64_t num_chunks,
                                   int64_t num_nodes, int id_bits, int ts_bits, int64_t ts_base, int64_t* out_roots,
                                   int64_t* out_ts_ptr, int64_t* out_ts, int64_t* out_q_ptr, int64_t* out_q_eid,
                                   int64_t* d_counts, int32_t* d_status, void* ws, size_t ws_bytes, void* stream_) {
  SGL_NVTX("sgl_seeds_in_window");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_events >= 0 && num_nodes >= 0, SGL_ERR_ARG, "seeds_in_window: negative size");
  SGL_REQUIRE(id_bits >= 0 && ts_bits >= 0 && id_bits + ts_bits < 64, SGL_ERR_UNSUPPORTED,
              "seeds_in_window: id_bits %d + ts_bits %d leave no room for the sentinel key", id_bits, ts_bits);
  SGL_REQUIRE(d_counts && out_ts_ptr && out_q_ptr, SGL_ERR_ARG, "seeds_in_window: null output");
  if (n_events == 0) {
    SGL_CHECK_RC(zero_async(d_counts, 3 * sizeof(int64_t), stream));
    SGL_CHECK_RC(zero_async(out_ts_ptr, sizeof(int64_t), stream));
    SGL_CHECK_RC(zero_async(out_q_ptr, sizeof(int64_t), stream));
    return SGL_OK;
  }
  SGL_REQUIRE(ev_src && ev_ts && ev_eid && out_roots && out_ts && out_q_eid, SGL_ERR_ARG, "seeds_in_window: null array");
  const int64_t n = n_events;
  SGL_REQUIRE(n < ((int64_t)1 << 31), SGL_ERR_UNSUPPORTED, "seeds_in_window: too many events");
  const int key_bits = id_bits + ts_bits;
  SGL_REQUIRE(ws && ws_bytes >= sgl_seeds_ws_bytes(n), SGL_ERR_WORKSPACE, "seeds_in_window: workspace %zu < %zu bytes", ws_bytes,
              sgl_seeds_ws_bytes(n));
  unsigned long long* valid = (unsigned long long*)ws;
  LaunchScope scope(stream);
  SGL_CHECK_RC(zero_async(valid, sizeof(*valid), stream));
  SGL_CHECK_RC(sort_list(
      SeedsSource{ev_src, ev_ts, n, nullptr, node_chunk, chunk_mask, num_chunks, num_nodes, id_bits, ts_bits, ts_base, d_status},
      SeedsSink{nullptr, key_bits, ts_bits, ts_base, ev_eid, out_roots, out_ts_ptr, out_ts, out_q_ptr, out_q_eid, d_counts, nullptr, valid},
      n, key_bits + 1, (char*)ws + align_up(8), ws_bytes - align_up(8), d_status, stream));
  return scope.submit();
}
