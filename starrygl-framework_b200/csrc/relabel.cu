// Dedup / relabel kernels of the mini-batch builder.  Everything is sort based so that local ids come out in
// the deterministic order the CPU builder produces (sorted unique), not in hash-table order:
//
// key = (id << ts_bits) | (ts - ts_base), stable sort, numbers of the distinct keys -> unique list and inverse map, with the
// producer of the keys and the consumer of the order fused into the sort (lists.cuh, sort_list in lsd.cuh).
//
// Algorithmic HBM bytes: 16 read + 8 write per input pair, 16 per unique pair, plus the sort passes
// (32 B per pair and populated key byte).
#include "launch.cuh"
#include "sort.cuh"
#include "lists.cuh"
#include "lsd.cuh"

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

extern "C" int sgl_unique_pairs(const int64_t* a_id, const int64_t* a_ts, int64_t n_a, const int64_t* d_n_a,
                                const int64_t* b_id, const int64_t* b_ts, int64_t n_b, const int64_t* d_n_b, int id_bits,
                                int ts_bits, int64_t ts_base, int64_t* out_id, int64_t* out_ts, int64_t* inv_a,
                                int64_t* inv_b, int64_t* d_n_unique, int32_t* d_status, void* ws, size_t ws_bytes,
                                void* stream_) {
  SGL_NVTX("sgl_unique_pairs");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_a >= 0 && n_b >= 0, SGL_ERR_ARG, "unique_pairs: negative size");
  SGL_REQUIRE(id_bits >= 0 && ts_bits >= 0 && id_bits + ts_bits <= 64, SGL_ERR_UNSUPPORTED,
              "unique_pairs: id_bits %d + ts_bits %d exceed the 64-bit sort key", id_bits, ts_bits);
  SGL_REQUIRE(d_n_unique, SGL_ERR_ARG, "unique_pairs: d_n_unique is null");
  const int64_t n = n_a + n_b;
  if (n == 0) {
    SGL_CHECK_RC(zero_async(d_n_unique, sizeof(int64_t), stream));
    return SGL_OK;
  }
  SGL_REQUIRE((n_a == 0 || (a_id && a_ts)) && (n_b == 0 || (b_id && b_ts)) && out_id && out_ts, SGL_ERR_ARG,
              "unique_pairs: null array");
  LaunchScope scope(stream);
  SGL_CHECK_RC(sort_list(PairSource{a_id, a_ts, d_n_a, b_id, b_ts, d_n_b, n_a, n_b, id_bits, ts_bits, ts_base, d_status},
                         PairSink{n_a, d_n_a, ts_bits, ts_base, out_id, out_ts, inv_a, inv_b, d_n_unique}, n, id_bits + ts_bits, ws,
                         ws_bytes, d_status, stream));
  return scope.submit();
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
  const int64_t cap = n_edges < 1 ? 1 : n_edges;
  SGL_REQUIRE(n_edges == 0 || (dst && ts && dt && eid && out_indices && out_ts && out_dt && out_eid), SGL_ERR_ARG,
              "build_csc: null array");
  LaunchScope scope(stream);
  SGL_CHECK_RC(sort_list(
      CscSource{dst, dst_map, ts, d_n_edges, n_edges, dst_bits, ts_bits, ts_base, d_status},
      CscSink{num_dst, d_num_dst, ts_bits, src_local, ts, dt, eid, out_indptr, out_indices, out_ts, out_dt, out_eid}, cap,
      dst_bits + ts_bits, ws, ws_bytes, d_status, stream));
  return scope.submit();
}

extern "C" size_t sgl_relabel_nodes_ws_bytes(int64_t n) { return list_ws_bytes(n); }

int sgl::relabel_nodes(const int64_t* ids, int64_t n, const int64_t* d_n, int64_t num_nodes, int64_t* mapper,
                                 int64_t* mask, int64_t epoch, int64_t* d_next_local, int64_t* out_local,
                                 int64_t* out_new_ids, int64_t* d_n_new, const int64_t* d_start, int32_t* d_status, void* ws, size_t ws_bytes,
                                 void* stream_) {
  SGL_NVTX("sgl_relabel_nodes");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n >= 0 && num_nodes >= 0, SGL_ERR_ARG, "relabel_nodes: negative size");
  SGL_REQUIRE(d_next_local && d_n_new, SGL_ERR_ARG, "relabel_nodes: null counter");
  if (n == 0) {
    SGL_CHECK_RC(zero_async(d_n_new, sizeof(int64_t), stream));
    return SGL_OK;
  }
  SGL_REQUIRE(ids && mapper && mask && out_local && out_new_ids, SGL_ERR_ARG, "relabel_nodes: null array");
  const int id_bits = bits_for(num_nodes > 0 ? (uint64_t)(num_nodes - 1) : 0);
  SGL_REQUIRE(id_bits < 63, SGL_ERR_UNSUPPORTED, "relabel_nodes: num_nodes too large");
  LaunchScope scope(stream);
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
