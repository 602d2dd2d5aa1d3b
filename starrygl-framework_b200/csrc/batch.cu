// The whole mini-batch in one call: (node, time) relabel of the roots, every hop, relabel and CSC per hop -- enqueued
// back to back with all sizes on the device, results in one arena that the caller allocates with a single allocation.
//
// What this replaces is host time: driven entry point by entry point from Python a two-hop batch of 4,096 roots cost 37
// allocations and 20 foreign calls, and its 200 us of kernels took 490 us to issue.
//
// Results: sections of 8-byte words in the order of batch_sections(), each rounded up to 32 words, one behind the other in an
// arena or (sgl_build_batch_at) wherever the caller wants each to lie:
//   roots            gids[n], ts[n], inverse map[n]
//   hop l            nbr, dst, ts, dt (fp32), eid [T_l k_l], offsets[T_l + 1]; merged list gids, ts [C_l + T_l k_l], column
//                    indices of the hop's edges in it [T_l k_l]; from the second hop on: CSC row pointer [C_l + 1], indices,
//                    ts, dt (fp32), eid [T_l k_l]
//   with T_0 = C_0 = n, T_(l+1) = T_l k_l, C_(l+1) = C_l + T_l k_l.  The first hop needs no CSC of its own: its targets are the
//   list itself and its edges come out in (row, time) order, so its offsets ARE the row pointer.
// Meta (8-byte words): entries of the root list, then per hop sampled edges and entries of the merged list, then a status
// word (used when the caller has none of its own).

#include <memory>
#include <new>

#include "chain.cuh"
#include "rowcsc.cuh"
#include "sampler.cuh"
#include "sort.cuh"
#include "tilesort.cuh"

using namespace sgl;

namespace {

constexpr int kHostWords = 512;   // of sgl_host_words
constexpr int kRootSections = 3, kHopSections = 14;

inline int64_t words(int64_t n) { return ((n < 1 ? 1 : n) + 31) / 32 * 32; }

// sizes of the sections in words; returns the number of sections
int batch_sections(int64_t n, const int32_t* fanouts, int hops, int64_t* out) {
  int s = 0;
  for (int i = 0; i < kRootSections; ++i) out[s++] = words(n);
  int64_t t = n, c = n;
  for (int l = 0; l < hops; ++l) {
    const int64_t e = t * fanouts[l];
    out[s++] = words(e);                         // 0 nbr
    out[s++] = words(e);                         // 1 dst
    out[s++] = words(e);                         // 2 ts
    out[s++] = words((e + 1) / 2);               // 3 dt
    out[s++] = words(e);                         // 4 eid
    out[s++] = words(t + 1);                     // 5 offsets
    out[s++] = words(c + e);                     // 6 gids
    out[s++] = words(c + e);                     // 7 ts
    out[s++] = words(e);                         // 8 column index of an edge
    const bool csc = l > 0;
    out[s++] = csc ? words(c + 1) : 0;           // 9 indptr
    out[s++] = csc ? words(e) : 0;               // 10 indices
    out[s++] = csc ? words(e) : 0;               // 11 ts
    out[s++] = csc ? words((e + 1) / 2) : 0;     // 12 dt
    out[s++] = csc ? words(e) : 0;               // 13 eid
    t = e;
    c += e;
  }
  return s;
}

size_t sample_ws(int64_t n, const int32_t* fanouts, int hops) {
  size_t most = 0;
  for (int l = 0; l < hops; ++l) {
    const size_t b = align_up(sgl_sample_ws_bytes(n));
    most = most > b ? most : b;
    n *= fanouts[l];
  }
  return most;
}

size_t list_ws(int64_t n, const int32_t* fanouts, int hops) {
  size_t most = sgl_unique_pairs_ws_bytes(n);
  int64_t t = n, c = n;
  for (int l = 0; l < hops; ++l) {
    t *= fanouts[l];
    c += t;
    const size_t b = sgl_unique_pairs_ws_bytes(c);
    most = most > b ? most : b;
  }
  return align_up(most);
}

// Edges of a hop go to their rows along the order of the layer list (rowcsc.cuh), but for lists that one CTA sorts.
inline bool by_rows(int64_t edges) { return edges > tilesort::kSingleMax; }

// orders of the layer lists that a CSC is made along: kept per hop, the next list is merged while it is read
size_t order_ws(int64_t n, const int32_t* fanouts, int hops) {
  size_t sum = 0;
  int64_t t = n, c = n;
  for (int l = 0; l + 1 < hops; ++l) {
    t *= fanouts[l];
    c += t;
    if (by_rows(t * fanouts[l + 1])) sum += RowOrder::bytes(c);
  }
  return sum;
}

size_t csc_ws(int64_t n, const int32_t* fanouts, int hops) {
  size_t most = 0;
  int64_t t = n, c = n;
  for (int l = 0; l < hops; ++l) {
    const int64_t e = t * fanouts[l];
    const size_t b = l > 0 ? (by_rows(e) ? build_csc_rows_ws_bytes(e, c) : sgl_build_csc_ws_bytes(e, c)) : 0;
    most = most > b ? most : b;
    t = e;
    c += e;
  }
  return align_up(most);
}

// indices[j] = col[indices[j]]: edge numbers -> positions in the merged list.  A batch with ids or times that were flagged and
// replaced can leave entries of `indices` unwritten (targets of one list entry then have different edges, which build_csc_rows
// rules out): they are not followed.
__global__ void __launch_bounds__(256)
map_columns_kernel(int64_t* __restrict__ indices, const int64_t* __restrict__ col, int64_t n_cap, const int64_t* d_n, int32_t* d_status) {
  const int64_t n = eff_count(n_cap, d_n), stride = (int64_t)gridDim.x * 256;
  for (int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x; j < n; j += stride) {
    const int64_t e = indices[j];
    if ((uint64_t)e < (uint64_t)n) indices[j] = __ldg(col + e);
    else dev_flag(d_status, SGL_DEV_BAD_INDEX);
  }
}

// The same from 32-bit positions, which also become the list's 64-bit ones.
__global__ void __launch_bounds__(256)
map_columns_narrow_kernel(int64_t* __restrict__ indices, const uint32_t* __restrict__ narrow, int64_t* __restrict__ col, int64_t n_cap,
                          const int64_t* d_n, int32_t* d_status) {
  const int64_t n = eff_count(n_cap, d_n), stride = (int64_t)gridDim.x * 256;
  for (int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x; j < n; j += stride) {
    const int64_t e = indices[j];
    if ((uint64_t)e < (uint64_t)n) indices[j] = (int64_t)__ldg(narrow + e);
    else dev_flag(d_status, SGL_DEV_BAD_INDEX);
    __stcs((long long*)col + j, (long long)__ldg(narrow + j));
  }
}

// The merge of a list scatters the edges' positions in it.  Beyond half of L2 as 64-bit words every store is a sector read and
// written in HBM; as 32-bit words they stay in L2 longer (15 M edges: 437 -> 290 us for the delivery).
inline bool narrow_columns(int64_t edges) { return edges > (int64_t)8 << 20; }

size_t narrow_ws(int64_t n, const int32_t* fanouts, int hops) {
  int64_t t = n;
  size_t most = 0;
  for (int l = 0; l < hops; ++l) {
    t *= fanouts[l];
    if (l > 0 && narrow_columns(t)) most = align_up((size_t)t * 4);        // (sizes grow)
  }
  return most;
}

}  // namespace

extern "C" int64_t sgl_build_batch_layout(int64_t n_roots, const int32_t* fanouts, int n_hops, int64_t* section_words) {
  if (n_roots < 0 || n_hops < 0 || (n_hops && !fanouts) || !section_words) return -1;
  const int s = batch_sections(n_roots, fanouts, n_hops, section_words);
  int64_t total = 0;
  for (int i = 0; i < s; ++i) total += section_words[i];
  return total;
}

extern "C" size_t sgl_build_batch_ws_bytes(int64_t n_roots, const int32_t* fanouts, int n_hops) {
  return sample_ws(n_roots, fanouts, n_hops) + list_ws(n_roots, fanouts, n_hops) + csc_ws(n_roots, fanouts, n_hops) +
         order_ws(n_roots, fanouts, n_hops) + narrow_ws(n_roots, fanouts, n_hops);
}

// host_early, host_ready: see sgl_build_batch_staged, sgl_build_batch_ready
static int build_batch(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                                  int64_t num_nodes, const int64_t* roots, const int64_t* root_ts, int64_t n_roots,
                                  const int32_t* fanouts, int n_hops, int policy, int equal_root_time, int64_t allowed_offset,
                                  uint64_t seed, int id_bits, int ts_bits, int64_t ts_base, const int64_t* section_at, int64_t* base,
                                  int64_t* other_base, int64_t* meta, int32_t* d_status, int64_t* host_meta, int64_t* host_early,
                                  int64_t* host_ready, void* ws, size_t ws_bytes, void* side_stream, void* stream_) {
  SGL_NVTX("sgl_build_batch");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n_roots >= 0 && n_hops >= 0 && (n_hops == 0 || fanouts), SGL_ERR_ARG, "build_batch: bad size");
  for (int l = 0; l < n_hops; ++l) SGL_REQUIRE(fanouts[l] >= 1, SGL_ERR_ARG, "build_batch: fanout=%d must be >= 1", fanouts[l]);
  SGL_REQUIRE(meta, SGL_ERR_ARG, "build_batch: meta is null");
  // The root list starts before the hops are set up (flush, below): what a hop refuses is refused here, before anything runs.
  struct Hop {
    int64_t *nbr, *dst, *ts, *eid, *offs, *gids, *gts, *col, *indptr, *indices, *cts, *ceid;
    float *dt, *cdt;
  };
  const std::unique_ptr<Hop[]> hop(new (std::nothrow) Hop[n_hops + 1]);
  SGL_REQUIRE(hop, SGL_ERR_ARG, "build_batch: no host memory for %d hops", n_hops);
  int64_t *cur_id = nullptr, *cur_ts = nullptr, *inv = nullptr;
  if (n_roots > 0) {
    SGL_REQUIRE(section_at && roots && root_ts && (n_hops == 0 || (indptr && nbr && ts && eid)), SGL_ERR_ARG, "build_batch: null array");
    constexpr int64_t kMost = (int64_t)1 << 32;
    int64_t t = n_roots, c = n_roots;
    for (int l = 0; l < n_hops; ++l) {
      SGL_CHECK_RC(check_sampling(fanouts[l], policy, t));
      SGL_REQUIRE(t < kMost && fanouts[l] <= kMost / t && c + t * fanouts[l] < kMost, SGL_ERR_UNSUPPORTED,
                  "build_batch: hop %d: edges and list entries need 64-bit positions", l);
      SGL_REQUIRE(l == 0 || bits_for((uint64_t)c) + ts_bits <= 64, SGL_ERR_UNSUPPORTED,
                  "build_batch: hop %d: rows and times (%d bits) exceed the 64-bit sort key", l, ts_bits);
      t *= fanouts[l];
      c += t;
    }
    SGL_REQUIRE(ws_bytes >= sgl_build_batch_ws_bytes(n_roots, fanouts, n_hops), SGL_ERR_WORKSPACE, "build_batch: workspace %zu < %zu bytes",
                ws_bytes, sgl_build_batch_ws_bytes(n_roots, fanouts, n_hops));
    int sec = 0;
    auto take = [&]() -> int64_t* {
      const int64_t at = section_at[sec++];
      return (int64_t*)(at >= 0 ? (uintptr_t)base + (uintptr_t)at * 8 : (uintptr_t)other_base + (uintptr_t)(-1 - at) * 8);
    };
    cur_id = take(); cur_ts = take(); inv = take();
    bool all = cur_id && cur_ts;
    for (int l = 0; l < n_hops; ++l) {
      Hop& h = hop[l];
      h.nbr = take(); h.dst = take(); h.ts = take(); h.dt = (float*)take(); h.eid = take(); h.offs = take();
      h.gids = take(); h.gts = take(); h.col = take();
      h.indptr = take(); h.indices = take(); h.cts = take(); h.cdt = (float*)take(); h.ceid = take();
      all = all && h.nbr && h.dst && h.ts && h.dt && h.eid && h.offs && h.gids && h.gts && (h.col || n_hops == 1) &&
            (l == 0 || (h.indptr && h.indices && h.cts && h.cdt && h.ceid));
    }
    SGL_REQUIRE(all, SGL_ERR_ARG, "build_batch: null section");
  }
  LaunchScope scope(stream);
  SGL_CHECK_RC(zero_async(meta, (size_t)(2 + 2 * n_hops) * sizeof(int64_t), stream));
  auto done = [&]() -> int {
    if (host_early) SGL_CHECK_RC(export_words(meta, host_early, 1 + 2 * n_hops, stream));      // (no roots, or no hops)
    if (host_ready) SGL_CHECK_RC(export_words(meta, host_ready, 0, stream));
    if (host_meta) SGL_CHECK_RC(export_words(meta, host_meta, 2 + 2 * n_hops, stream));
    return scope.submit();
  };
  if (n_roots == 0) return done();
  if (d_status == nullptr) d_status = (int32_t*)(meta + 1 + 2 * n_hops);
  const size_t swb = sample_ws(n_roots, fanouts, n_hops), lwb = list_ws(n_roots, fanouts, n_hops), cwb = csc_ws(n_roots, fanouts, n_hops);
  void *sws = ws, *lws = (char*)ws + swb, *cws = (char*)lws + lwb;
  char* ows = (char*)cws + cwb;
  uint32_t* const cols32 = (uint32_t*)(ows + order_ws(n_roots, fanouts, n_hops));
  RowOrder order_of{};                   // of the layer list merged last, where the next CSC goes along it
  int rc = sgl_unique_pairs(roots, root_ts, n_roots, nullptr, nullptr, nullptr, 0, nullptr, id_bits, ts_bits, ts_base, cur_id, cur_ts, inv,
                            nullptr, meta, d_status, lws, lwb, stream);
  if (rc) return rc;
  if (n_hops > 0) SGL_CHECK_RC(scope.flush());             // (600 roots 50.3 -> 46.5 us a batch, 4,096 roots two hops 143 -> 134)
  auto sample = [&](int l, const int64_t* tgt, const int64_t* tgt_ts, int64_t n, const int64_t* d_n, cudaStream_t on) {
    const Hop& h = hop[l];
    return sample_layer(indptr, nbr, ts, eid, fence, num_nodes, tgt, tgt_ts, n, d_n, fanouts[l], policy, equal_root_time, allowed_offset, 0,
                        seed, (uint32_t)l, h.nbr, h.dst, h.ts, h.dt, nullptr, h.eid, h.offs, meta + 1 + 2 * l, d_status, sws, swb, on);
  };
  // Hop l + 1 queries one target per edge sampled by hop l at that edge's time and waits for no relabel but the first; the
  // CSC of a hop needs the relabel before it but not its own (its columns are translated at the end).  Where they can
  // both run on a second stream, next to the relabels: 4,096 roots uniform [10, 10], kernels of 170 us end after 107.
  if (n_hops > 0 && (rc = sample(0, cur_id, cur_ts, n_roots, meta, stream))) return rc;
  const bool forked = n_hops > 1 && (LaunchScope::current() != nullptr || (side_stream != nullptr && side_stream != stream_));
  // (inside a launch scope a stream is only a name for a chain of kernels)
  cudaStream_t side = forked ? (side_stream ? (cudaStream_t)side_stream : (cudaStream_t)(uintptr_t)3) : stream;
  enum { kFork, kSampled, kRelabelled, kCsc };
  Order order;
  if (forked) {
    SGL_CHECK_RC(order.init(LaunchScope::current()));
    SGL_CHECK_RC(order.mark(kFork, stream));
    SGL_CHECK_RC(order.wait(kFork, side));
  }
  int64_t t = n_roots, c = n_roots;
  const int64_t* d_cur = meta;
  const int64_t* last_col = nullptr;
  for (int l = 0; l < n_hops; ++l) {
    const Hop& h = hop[l];
    const int64_t e = t * fanouts[l];
    int64_t *d_edges = meta + 1 + 2 * l, *d_next = meta + 2 + 2 * l;
    if (forked && l > 0) SGL_CHECK_RC(order.wait(kSampled, stream));
    if (l + 1 < n_hops) {
      if ((rc = sample(l + 1, h.nbr, h.ts, e, d_edges, side))) return rc;
      if (forked) SGL_CHECK_RC(order.mark(kSampled, side));
    }
    if (l > 0) {
      if (forked) SGL_CHECK_RC(order.wait(kRelabelled, side));
      rc = by_rows(e) ? build_csc_rows(order_of, c, cur_ts, h.offs, fanouts[l], policy == SGL_POLICY_UNIFORM, h.dst, last_col, h.ts, h.dt, h.eid, e,
                                       d_edges, c, d_cur, bits_for((uint64_t)c), ts_bits, ts_base, h.indptr, h.indices, h.cts, h.cdt, h.ceid, d_status, cws, cwb,
                                       side)
                      : sgl_build_csc(nullptr, h.dst, last_col, h.ts, h.dt, h.eid, e, d_edges, c, d_cur, bits_for((uint64_t)c), ts_bits,
                                      ts_base, h.indptr, h.indices, h.cts, h.cdt, h.ceid, 0, d_status, cws, cwb, side);
      if (rc) return rc;
      if (forked) SGL_CHECK_RC(order.mark(kCsc, side));
    }
    if (host_ready && l + 1 == n_hops) {
      // (behind the columns of the hop before too: they are translated on the main stream, next to this hop's CSC)
      if (forked && l > 0) {
        SGL_CHECK_RC(order.mark(kFork, stream));
        SGL_CHECK_RC(order.wait(kFork, side));
      }
      SGL_CHECK_RC(export_words(meta, host_ready, 0, l > 0 ? side : stream));
      host_ready = nullptr;
      // (launched one by one, a stream of the caller's: it has to be joined behind this too; a chain of a graph needs no end)
      if (forked && l > 0 && LaunchScope::current() == nullptr) SGL_CHECK_RC(order.mark(kCsc, side));
    }
    order_of = RowOrder{};
    if (l + 1 < n_hops && by_rows(e * fanouts[l + 1])) {
      order_of = RowOrder::carve(ows, c + e);
      ows += RowOrder::bytes(c + e);
    }
    if (host_early && l + 1 == n_hops) {
      cudaStream_t on = stream;
      if (LaunchScope::current() != nullptr) {
        on = (cudaStream_t)(uintptr_t)5;       // a third chain of the graph, next to the last merge
        SGL_CHECK_RC(LaunchScope::current()->follow(on, stream));
      }
      SGL_CHECK_RC(export_words(meta, host_early, 1 + 2 * n_hops, on));
      host_early = nullptr;
    }
    rc = unique_pairs(cur_id, cur_ts, c, d_cur, h.nbr, h.ts, e, d_edges, id_bits, ts_bits, ts_base, h.gids, h.gts, nullptr, h.col,
                      l > 0 && narrow_columns(e) ? cols32 : nullptr, d_next, order_of, d_status, lws, lwb, stream);
    if (rc) return rc;
    const bool narrow = l > 0 && narrow_columns(e);
    if (forked && l + 1 < n_hops && !narrow) SGL_CHECK_RC(order.mark(kRelabelled, stream));
    if (l > 0) {
      if (forked) SGL_CHECK_RC(order.wait(kCsc, stream));
      if (narrow) SGL_CHECK_RC(launch(map_columns_narrow_kernel, stream_grid(e, 256 * 4, 8), 256, 0, stream, h.indices, cols32, h.col, e, d_edges,
                                       d_status));
      else SGL_CHECK_RC(launch(map_columns_kernel, stream_grid(e, 256 * 4, 8), 256, 0, stream, h.indices, h.col, e, d_edges, d_status));
    }
    if (forked && l + 1 < n_hops && narrow) SGL_CHECK_RC(order.mark(kRelabelled, stream));     // (the next CSC may read h.col)
    cur_id = h.gids;
    cur_ts = h.gts;
    d_cur = d_next;
    last_col = h.col;
    t = e;
    c += e;
  }
  return done();
}

extern "C" int sgl_build_batch_at(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                                  int64_t num_nodes, const int64_t* roots, const int64_t* root_ts, int64_t n_roots,
                                  const int32_t* fanouts, int n_hops, int policy, int equal_root_time, int64_t allowed_offset,
                                  uint64_t seed, int id_bits, int ts_bits, int64_t ts_base, const int64_t* section_at, int64_t* base,
                                  int64_t* other_base, int64_t* meta, int32_t* d_status, int64_t* host_meta, void* ws, size_t ws_bytes,
                                  void* side_stream, void* stream) {
  return build_batch(indptr, nbr, ts, eid, fence, num_nodes, roots, root_ts, n_roots, fanouts, n_hops, policy, equal_root_time, allowed_offset, seed,
                     id_bits, ts_bits, ts_base, section_at, base, other_base, meta, d_status, host_meta, nullptr, nullptr, ws, ws_bytes, side_stream,
                     stream);
}

extern "C" int sgl_build_batch_staged(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                                      int64_t num_nodes, const int64_t* roots, const int64_t* root_ts, int64_t n_roots,
                                      const int32_t* fanouts, int n_hops, int policy, int equal_root_time, int64_t allowed_offset,
                                      uint64_t seed, int id_bits, int ts_bits, int64_t ts_base, const int64_t* section_at, int64_t* base,
                                      int64_t* other_base, int64_t* meta, int32_t* d_status, int64_t* host_meta, int64_t* host_early,
                                      void* ws, size_t ws_bytes, void* side_stream, void* stream) {
  return build_batch(indptr, nbr, ts, eid, fence, num_nodes, roots, root_ts, n_roots, fanouts, n_hops, policy, equal_root_time, allowed_offset, seed,
                     id_bits, ts_bits, ts_base, section_at, base, other_base, meta, d_status, host_meta, host_early, nullptr, ws, ws_bytes,
                     side_stream, stream);
}

extern "C" int sgl_build_batch_ready(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                                      int64_t num_nodes, const int64_t* roots, const int64_t* root_ts, int64_t n_roots,
                                      const int32_t* fanouts, int n_hops, int policy, int equal_root_time, int64_t allowed_offset,
                                      uint64_t seed, int id_bits, int ts_bits, int64_t ts_base, const int64_t* section_at, int64_t* base,
                                      int64_t* other_base, int64_t* meta, int32_t* d_status, int64_t* host_meta, int64_t* host_early,
                                      int64_t* host_ready, void* ws, size_t ws_bytes, void* side_stream, void* stream) {
  return build_batch(indptr, nbr, ts, eid, fence, num_nodes, roots, root_ts, n_roots, fanouts, n_hops, policy, equal_root_time, allowed_offset, seed,
                     id_bits, ts_bits, ts_base, section_at, base, other_base, meta, d_status, host_meta, host_early, host_ready, ws, ws_bytes,
                     side_stream, stream);
}

extern "C" int sgl_build_batch(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                               int64_t num_nodes, const int64_t* roots, const int64_t* root_ts, int64_t n_roots,
                               const int32_t* fanouts, int n_hops, int policy, int equal_root_time, int64_t allowed_offset,
                               uint64_t seed, int id_bits, int ts_bits, int64_t ts_base, int64_t* arena, int64_t* meta,
                               int32_t* d_status, int64_t* host_meta, void* ws, size_t ws_bytes, void* side_stream, void* stream) {
  const std::unique_ptr<int64_t[]> at(n_hops >= 0 ? new (std::nothrow) int64_t[kRootSections + (size_t)n_hops * kHopSections] : nullptr);
  SGL_REQUIRE(at && sgl_build_batch_layout(n_roots, fanouts, n_hops, at.get()) >= 0, SGL_ERR_ARG, "build_batch: bad size");
  SGL_REQUIRE(arena || n_roots == 0, SGL_ERR_ARG, "build_batch: null array");
  int64_t next = 0;
  for (int s = 0; s < kRootSections + n_hops * kHopSections; ++s) {
    const int64_t size = at[s];
    at[s] = next;
    next += size;
  }
  return sgl_build_batch_at(indptr, nbr, ts, eid, fence, num_nodes, roots, root_ts, n_roots, fanouts, n_hops, policy, equal_root_time,
                            allowed_offset, seed, id_bits, ts_bits, ts_base, at.get(), arena, nullptr, meta, d_status, host_meta, ws, ws_bytes,
                            side_stream, stream);
}

// Up to kMaxExport arrays packed one behind the other (16-byte aligned offsets) and copied to the host in one go, or in two
// when the bytes from `split` on go to a second buffer.
namespace {
constexpr int kMaxExport = 96;
struct Export {
  const char* src[kMaxExport];
  int64_t bytes[kMaxExport], at[kMaxExport];
};
__global__ void __launch_bounds__(256) pack_kernel(const __grid_constant__ Export x, char* __restrict__ dst) {
  const int a = blockIdx.y;
  const char* s = x.src[a];
  char* d = dst + x.at[a];
  const int64_t bytes = x.bytes[a], tid = (int64_t)blockIdx.x * 256 + threadIdx.x, stride = (int64_t)gridDim.x * 256;
  const int64_t quads = ((uintptr_t)s & 15) == 0 ? bytes >> 4 : 0;
  for (int64_t i = tid; i < quads; i += stride) ((uint4*)d)[i] = ((const uint4*)s)[i];
  for (int64_t i = quads * 4 + tid; i < bytes >> 2; i += stride) ((uint32_t*)d)[i] = ((const uint32_t*)s)[i];
}
}  // namespace

extern "C" int sgl_export_arrays(int n, const void* const* src, const int64_t* bytes, const int64_t* at, void* staging, void* host,
                                 int64_t total, void* host2, int64_t split, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n >= 0 && n <= kMaxExport && (n == 0 || (src && bytes && at)) && total >= 0, SGL_ERR_ARG, "export_arrays: at most %d arrays",
              kMaxExport);
  if (n == 0 || total == 0) return SGL_OK;
  SGL_REQUIRE(staging && (host || split == 0), SGL_ERR_ARG, "export_arrays: null buffer");
  Export x;
  memset(&x, 0, sizeof(x));
  int64_t most = 1;
  for (int i = 0; i < n; ++i) {
    SGL_REQUIRE((src[i] || bytes[i] == 0) && bytes[i] >= 0 && bytes[i] % 4 == 0 && at[i] % 16 == 0 && at[i] >= 0 && at[i] + bytes[i] <= total,
                SGL_ERR_ARG, "export_arrays: bad array %d", i);
    x.src[i] = (const char*)src[i];
    x.bytes[i] = bytes[i];
    x.at[i] = at[i];
    most = bytes[i] > most ? bytes[i] : most;
  }
  SGL_CHECK_RC(launch(pack_kernel, dim3((unsigned)stream_grid(most / 16 + 1, 256 * 4, 4), (unsigned)n), 256, 0, stream, x, (char*)staging));
  if (host2 == nullptr) split = total;
  SGL_REQUIRE(split >= 0 && split <= total, SGL_ERR_ARG, "export_arrays: bad split");
  if (split > 0) SGL_CUDA_CHECK(cudaMemcpyAsync(host, staging, (size_t)split, cudaMemcpyDeviceToHost, stream));
  if (split < total)
    SGL_CUDA_CHECK(cudaMemcpyAsync(host2, (char*)staging + split, (size_t)(total - split), cudaMemcpyDeviceToHost, stream));
  return SGL_OK;
}

// One copy per array.
extern "C" int sgl_copy_arrays(int n, const void* const* src, const int64_t* bytes, void* const* dst, void* stream) {
  SGL_REQUIRE(n >= 0 && (n == 0 || (src && bytes && dst)), SGL_ERR_ARG, "copy_arrays: null table");
  for (int i = 0; i < n; ++i) {
    SGL_REQUIRE(bytes[i] >= 0 && (bytes[i] == 0 || (src[i] && dst[i])), SGL_ERR_ARG, "copy_arrays: bad array %d", i);
    if (bytes[i] > 0) SGL_CUDA_CHECK(cudaMemcpyAsync(dst[i], src[i], (size_t)bytes[i], cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  }
  return SGL_OK;
}

// Pinned buffer of the calling thread (4,096 bytes) for results that the host waits for.
extern "C" int sgl_host_words(void** out) {
  SGL_REQUIRE(out, SGL_ERR_ARG, "host_words: out is null");
  struct Pinned {
    void* p = nullptr;
    ~Pinned() {                          // (with the thread; at the end of the process the driver may be gone already)
      if (p) cudaFreeHost(p);
    }
  };
  static thread_local Pinned words;
  if (words.p == nullptr) SGL_CUDA_CHECK(cudaHostAlloc(&words.p, kHostWords * 8, cudaHostAllocPortable));
  *out = words.p;
  return SGL_OK;
}

// Waits until work on the stream has set *flag to at_least or more: the host looks at the word itself for a while (a stream
// synchronisation costs 5 us more than the kernel that it waits for), then waits for the stream, which also reports errors.
extern "C" int sgl_wait_word(const int64_t* flag, int64_t at_least, void* stream) {
  SGL_REQUIRE(flag, SGL_ERR_ARG, "wait_word: flag is null");
  const volatile int64_t* f = flag;
  for (int i = 0; i < 2000000; ++i) {
    if (*f >= at_least) return SGL_OK;
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
  }
  SGL_CUDA_CHECK(cudaStreamSynchronize((cudaStream_t)stream));
  SGL_REQUIRE(*f >= at_least, SGL_ERR_CUDA, "wait_word: the stream ended without setting the word");
  return SGL_OK;
}

// Copies up to 4,088 bytes of device memory (whole 8-byte words) to the host and waits for them.
extern "C" int sgl_read_back(const void* src, void* dst, size_t bytes, void* stream) {
  SGL_REQUIRE(src && dst && bytes % 8 == 0 && bytes / 8 < (size_t)kHostWords, SGL_ERR_ARG, "read_back: at most %d words", kHostWords - 1);
  void* p = nullptr;
  SGL_CHECK_RC(sgl_host_words(&p));
  int64_t* host = (int64_t*)p;
  const int words = (int)(bytes / 8);
  SGL_CHECK_RC(export_words((const int64_t*)src, host, words, (cudaStream_t)stream));
  SGL_CHECK_RC(sgl_wait_word(host + words, 1, stream));
  memcpy(dst, host, bytes);
  return SGL_OK;
}
