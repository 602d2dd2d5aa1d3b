// One query of the graph API in one call: roots of a time window, negatives behind them, every hop, and the node-level
// relabel of roots and neighbours -- enqueued back to back with every size on the device.
//
// Driven entry point by entry point a two-layer query of 1,000 events was 55 kernels and copies with 10 synchronisations,
// 1.0 ms, most of it host time in two threads that wait for each other's interpreter lock.
//
// Arena (8-byte words, sections rounded up to 32 words), C = capacity of the window, Q = C + negatives:
//   roots[C] (global ids), roots[C] (local ids), ts_ptr[C + 1], q_ptr[C + 1], q_eid[C], query node[Q], query time[Q],
//   per hop (T_0 = Q, T_(l+1) = T_l k): nbr, dst, ts, dt (fp32), dt (int64), eid, local ids [T_l k], offsets[T_l + 1];
//   new global ids [C + sum of T_l k]
// Meta: 0 roots, 1 (root, time) pairs, 2 events, 3 queries, 4 first local id, 5 status, 6 - 7 window, 8 valid events,
//   9 + l edges of hop l, 9 + hops + j new ids of list j (roots, hop 0, ...).
#include "chain.cuh"
#include "lists.cuh"
#include "lsd.cuh"
#include "sampler.cuh"
#include "sort.cuh"

namespace sgl {
namespace {

constexpr int kMaxHops = 8;
constexpr int kHead = 7, kPerHop = 8, kMetaHead = 9;

inline int64_t words(int64_t n) { return ((n < 1 ? 1 : n) + 31) / 32 * 32; }

int query_sections(int64_t c, int64_t n_neg, int fanout, int hops, int64_t* out) {
  int s = 0;
  const int64_t q = c + n_neg;
  out[s++] = words(c);
  out[s++] = words(c);
  out[s++] = words(c + 1);
  out[s++] = words(c + 1);
  out[s++] = words(c);
  out[s++] = words(q);
  out[s++] = words(q);
  int64_t t = q, ids = c;
  for (int l = 0; l < hops; ++l) {
    const int64_t e = t * fanout;
    for (int i = 0; i < 3; ++i) out[s++] = words(e);     // nbr, dst, ts
    out[s++] = words((e + 1) / 2);                       // dt
    for (int i = 0; i < 3; ++i) out[s++] = words(e);     // dt (int64), eid, local ids
    out[s++] = words(t + 1);
    t = e;
    ids += e;
  }
  out[s++] = words(ids);
  return s;
}

// Bounds of [t0, t1) in the time-ordered events, known on the host to lie in [from, from + cap].  One warp, both searches 32-ary.
__global__ void window_kernel(const int64_t* __restrict__ ev_ts, int64_t from, int64_t cap, int64_t t0, int64_t t1, int64_t* meta) {
  const int lane = threadIdx.x & 31;
  int64_t bound[2];
  for (int g = 0; g < 2; ++g) {
    const int64_t v = g ? t1 : t0;
    int64_t lo = from, hi = from + cap;                  // first position with ts >= v in [lo, hi]
    while (hi - lo > 32) {
      const int64_t q = (hi - lo) / 33;
      const bool below = ev_ts[lo + (lane + 1) * q] < v;
      const int c = __popc(__ballot_sync(0xffffffffu, below));
      if (c < 32) hi = lo + (c + 1) * q;
      if (c > 0) lo = lo + c * q + 1;
    }
    const bool below = lo + lane < hi && ev_ts[lo + lane] < v;
    bound[g] = lo + __popc(__ballot_sync(0xffffffffu, below));
  }
  if (lane == 0) {
    meta[6] = bound[0];
    meta[7] = bound[1] > bound[0] ? bound[1] - bound[0] : 0;
    meta[5] = 0;
    meta[8] = 0;
  }
}

// negatives behind the pairs of the window; first local id of the query (0 when the numbering restarts)
__global__ void __launch_bounds__(256)
append_kernel(const int64_t* __restrict__ neg, const int64_t* __restrict__ neg_ts, int64_t n_neg, int64_t* q_node, int64_t* q_ts,
              int reset, int64_t* d_next_local, int64_t* meta) {
  const int64_t at = meta[1];
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i == 0) {
    meta[3] = at + n_neg;
    if (reset) *d_next_local = 0;
    meta[4] = *d_next_local;
  }
  if (i < n_neg) {
    q_node[at + i] = neg[i];
    q_ts[at + i] = neg_ts[i];
  }
}

}  // namespace
}  // namespace sgl

using namespace sgl;

extern "C" int64_t sgl_query_layout(int64_t cap, int64_t n_neg, int fanout, int n_hops, int64_t* section_words) {
  if (cap < 0 || n_neg < 0 || fanout < 1 || n_hops < 0 || n_hops > kMaxHops || !section_words) return -1;
  const int s = query_sections(cap, n_neg, fanout, n_hops, section_words);
  int64_t total = 0;
  for (int i = 0; i < s; ++i) total += section_words[i];
  return total;
}

extern "C" size_t sgl_query_ws_bytes(int64_t cap, int64_t n_neg, int fanout, int n_hops) {
  size_t seeds = align_up(sgl_seeds_ws_bytes(cap)), sample = 0, nodes = align_up(sgl_relabel_nodes_ws_bytes(cap));
  int64_t t = cap + n_neg;
  for (int l = 0; l < n_hops; ++l) {
    const size_t a = align_up(sgl_sample_ws_bytes(t)), b = align_up(sgl_relabel_nodes_ws_bytes(t * fanout));
    sample = sample > a ? sample : a;
    nodes = nodes > b ? nodes : b;
    t *= fanout;
  }
  return seeds + sample + nodes;
}

extern "C" int sgl_query_at(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                         int64_t num_nodes, const int64_t* ev_src, const int64_t* ev_ts, const int64_t* ev_eid, int64_t ev_from,
                         int64_t cap, int64_t t_begin, int64_t t_end, const int64_t* node_chunk, const uint8_t* chunk_mask,
                         int64_t num_chunks, const int64_t* neg, const int64_t* neg_ts, int64_t n_neg, int fanout, int n_hops, int policy,
                         int equal_root_time, int64_t allowed_offset, int keep_root_time, int id_bits, int ts_bits, int64_t ts_base,
                         int64_t* mapper, int64_t* mask, int64_t epoch, int restart, int64_t* d_next_local,
                            const int64_t* section_at, int64_t* base, int64_t* meta,
                         int64_t* host_meta, void* ws, size_t ws_bytes, void* producer, void* stream_) {
  SGL_NVTX("sgl_query");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(cap >= 1 && cap < ((int64_t)1 << 31) && n_neg >= 0 && n_hops >= 0 && n_hops <= kMaxHops, SGL_ERR_UNSUPPORTED,
              "query: at most 2^31 events and %d hops", kMaxHops);
  SGL_REQUIRE(id_bits >= 0 && ts_bits >= 0 && id_bits + ts_bits < 64, SGL_ERR_UNSUPPORTED,
              "query: id_bits %d + ts_bits %d leave no room for the sentinel key", id_bits, ts_bits);
  SGL_REQUIRE(ev_src && ev_ts && ev_eid && mapper && mask && d_next_local && section_at && meta && host_meta && (n_neg == 0 || (neg && neg_ts)),
              SGL_ERR_ARG, "query: null array");
  SGL_REQUIRE(ws_bytes >= sgl_query_ws_bytes(cap, n_neg, fanout, n_hops), SGL_ERR_WORKSPACE, "query: workspace %zu < %zu bytes", ws_bytes,
              sgl_query_ws_bytes(cap, n_neg, fanout, n_hops));
  // The seeds start before the hops are set up (flush, below): what a hop refuses is refused here, before anything runs.
  SGL_REQUIRE(n_hops == 0 || (indptr && nbr && ts && eid), SGL_ERR_ARG, "query: null array");
  SGL_CHECK_RC(check_relabel(cap, num_nodes));
  for (int64_t l = 0, q = cap + n_neg; l < n_hops; ++l, q *= fanout) {
    SGL_CHECK_RC(check_sampling(fanout, policy, q));
    SGL_REQUIRE(fanout <= INT64_MAX / (q > 0 ? q : 1), SGL_ERR_UNSUPPORTED, "query: too many edges");
    SGL_CHECK_RC(check_relabel(q * fanout, num_nodes));
  }
  SGL_CHECK_RC(order_after(stream, (cudaStream_t)producer));
  int sec = 0;
  auto take = [&]() -> int64_t* { return (int64_t*)((uintptr_t)base + (uintptr_t)section_at[sec++] * 8); };
  int64_t *roots = take(), *roots_local = take(), *ts_ptr = take(), *q_ptr = take(), *q_eid = take(), *q_node = take(), *q_ts = take();
  struct Hop {
    int64_t *nbr, *dst, *ts, *dti, *eid, *local, *offs;
    float* dt;
  } hop[kMaxHops];
  for (int l = 0; l < n_hops; ++l) {
    Hop& h = hop[l];
    h.nbr = take(); h.dst = take(); h.ts = take(); h.dt = (float*)take(); h.dti = take(); h.eid = take(); h.local = take(); h.offs = take();
  }
  int64_t* new_ids = take();
  int32_t* d_status = (int32_t*)(meta + 5);
  size_t sample_b = 0;
  int64_t t = cap + n_neg;
  for (int l = 0; l < n_hops; ++l, t *= fanout) {
    const size_t a = align_up(sgl_sample_ws_bytes(t));
    sample_b = sample_b > a ? sample_b : a;
  }
  const size_t seeds_b = align_up(sgl_seeds_ws_bytes(cap)), nodes_b = ws_bytes - seeds_b - sample_b;
  char *seeds_ws = (char*)ws, *sample_ws = seeds_ws + seeds_b, *nodes_ws = sample_ws + sample_b;

  LaunchScope scope(stream);
  SGL_CHECK_RC(launch(window_kernel, 1, 32, 0, stream, ev_ts, ev_from, cap, t_begin, t_end, meta));
  const int key_bits = id_bits + ts_bits;
  SGL_CHECK_RC(sort_list(
      SeedsSource{ev_src, ev_ts, cap, meta + 6, node_chunk, chunk_mask, num_chunks, num_nodes, id_bits, ts_bits, ts_base, d_status},
      SeedsSink{meta + 6, key_bits, ts_bits, ts_base, ev_eid, roots, ts_ptr, q_ts, q_ptr, q_eid, meta, q_node,
                (unsigned long long*)(meta + 8)},
      cap, key_bits + 1, seeds_ws, seeds_b, d_status, stream));
  SGL_CHECK_RC(scope.flush());             // (nothing of it outlives a call that is refused below; 1,000 events 184 -> 173 us for two queries)
  SGL_CHECK_RC(launch(append_kernel, (unsigned)((n_neg + 255) / 256 < 1 ? 1 : (n_neg + 255) / 256), 256, 0, stream, neg, neg_ts, n_neg,
                      q_node, q_ts, restart, d_next_local, meta));
  // the hops next to the relabels: hop l + 1 needs the raw neighbours of hop l, their relabel comes whenever it comes
  LaunchScope* in = LaunchScope::current();
  cudaStream_t side = in ? (cudaStream_t)(uintptr_t)3 : stream;      // (a second chain of the graph)
  if (in) SGL_CHECK_RC(in->follow(side, stream));
  auto relabel = [&](const int64_t* ids, int64_t n, const int64_t* d_ids, int64_t* local, int64_t* d_new) -> int {
    return relabel_nodes(ids, n, d_ids, num_nodes, mapper, mask, epoch, d_next_local, local, new_ids, d_new, meta + 4, d_status, nodes_ws,
                         nodes_b, stream);
  };
  SGL_CHECK_RC(relabel(roots, cap, meta, roots_local, meta + kMetaHead + n_hops));
  const int64_t *tgt = q_node, *tgt_ts = q_ts, *d_n = meta + 3;
  t = cap + n_neg;
  for (int l = 0; l < n_hops; ++l) {
    const Hop& h = hop[l];
    SGL_CHECK_RC(sample_layer(indptr, nbr, ts, eid, fence, num_nodes, tgt, tgt_ts, t, d_n, fanout, policy, equal_root_time, allowed_offset,
                              keep_root_time, 0, (uint32_t)l, h.nbr, h.dst, h.ts, h.dt, h.dti, h.eid, h.offs, meta + kMetaHead + l,
                              d_status, sample_ws, sample_b, side));
    if (in) SGL_CHECK_RC(in->follow(stream, side));
    const int64_t e = t * fanout;
    SGL_CHECK_RC(relabel(h.nbr, e, meta + kMetaHead + l, h.local, meta + kMetaHead + n_hops + 1 + l));
    tgt = h.nbr;
    tgt_ts = h.ts;
    d_n = meta + kMetaHead + l;
    t = e;
  }
  if (in) SGL_CHECK_RC(in->follow(stream, side));
  SGL_CHECK_RC(export_words(meta, host_meta, kMetaHead + 2 * n_hops + 1, stream));
  return scope.submit();
}

extern "C" int sgl_query(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                         int64_t num_nodes, const int64_t* ev_src, const int64_t* ev_ts, const int64_t* ev_eid, int64_t ev_from,
                         int64_t cap, int64_t t_begin, int64_t t_end, const int64_t* node_chunk, const uint8_t* chunk_mask,
                         int64_t num_chunks, const int64_t* neg, const int64_t* neg_ts, int64_t n_neg, int fanout, int n_hops, int policy,
                         int equal_root_time, int64_t allowed_offset, int keep_root_time, int id_bits, int ts_bits, int64_t ts_base,
                         int64_t* mapper, int64_t* mask, int64_t epoch, int restart, int64_t* d_next_local, int64_t* arena, int64_t* meta,
                         int64_t* host_meta, void* ws, size_t ws_bytes, void* producer, void* stream) {
  int64_t at[kHead + kMaxHops * kPerHop + 1], next = 0;
  SGL_REQUIRE(arena && sgl_query_layout(cap, n_neg, fanout, n_hops, at) >= 0, SGL_ERR_ARG, "query: bad shape or null arena");
  for (int s = 0; s < kHead + n_hops * kPerHop + 1; ++s) {
    const int64_t size = at[s];
    at[s] = next;
    next += size;
  }
  return sgl_query_at(indptr, nbr, ts, eid, fence, num_nodes, ev_src, ev_ts, ev_eid, ev_from, cap, t_begin, t_end, node_chunk, chunk_mask,
                      num_chunks, neg, neg_ts, n_neg, fanout, n_hops, policy, equal_root_time, allowed_offset, keep_root_time, id_bits, ts_bits,
                      ts_base, mapper, mask, epoch, restart, d_next_local, at, arena, meta, host_meta, ws, ws_bytes, producer, stream);
}

// Source side of message-flow blocks for the hops of a query: block l has the D_l destinations (queries of the hop) followed
// by its N_l neighbours; column indices of its edges are D_l + j.  The queries of hop 0 are the (root, time) pairs under
// their root's local id and the negatives as they are, those of hop l the neighbours of hop l - 1.
namespace sgl {
namespace {
struct BlockHop {
  const int64_t *prev_node, *prev_ts, *node, *ts;
  int64_t d, n;
  int64_t *out_node, *out_ts, *out_index;
};
struct Blocks {
  BlockHop hop[kMaxHops];
  const int64_t *ts_ptr, *roots_local, *neg, *neg_ts;
  int64_t n_roots, n_pairs;
};

__global__ void __launch_bounds__(256) blocks_kernel(const __grid_constant__ Blocks b) {
  const BlockHop& h = b.hop[blockIdx.y];
  const int64_t stride = (int64_t)gridDim.x * 256;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < h.d + h.n; i += stride) {
    int64_t node, t;
    if (i >= h.d) {
      const int64_t j = i - h.d;
      node = h.node[j];
      t = h.ts[j];
      h.out_index[j] = i;
    } else {
      if (blockIdx.y > 0) {
        node = h.prev_node[i];
        t = h.prev_ts[i];
      } else if (i >= b.n_pairs) {
        node = b.neg[i - b.n_pairs];
        t = b.neg_ts[i - b.n_pairs];
      } else {
        t = h.prev_ts[i];
        int64_t lo = 0, hi = b.n_roots;      // root whose pairs hold pair i
        while (hi - lo > 1) {
          const int64_t mid = (lo + hi) >> 1;
          if (b.ts_ptr[mid] <= i) lo = mid; else hi = mid;
        }
        node = b.roots_local[lo];
      }
    }
    h.out_node[i] = node;
    h.out_ts[i] = t;
  }
}
}  // namespace
}  // namespace sgl

extern "C" int sgl_query_blocks(int n_hops, const int64_t* const* node, const int64_t* const* ts, const int64_t* counts,
                                const int64_t* q_ts, const int64_t* ts_ptr, const int64_t* roots_local, const int64_t* neg, const int64_t* neg_ts,
                                int64_t n_roots, int64_t n_pairs, int64_t n_queries, int64_t* out, void* stream_) {
  SGL_REQUIRE(n_hops >= 1 && n_hops <= kMaxHops && node && ts && counts && q_ts && ts_ptr && out &&
                  (n_queries <= n_pairs || (neg && neg_ts)), SGL_ERR_ARG, "query_blocks: bad argument");
  Blocks b;
  memset(&b, 0, sizeof(b));
  b.ts_ptr = ts_ptr;
  b.roots_local = roots_local;
  b.neg = neg;
  b.neg_ts = neg_ts;
  b.n_roots = n_roots;
  b.n_pairs = n_pairs;
  int64_t d = n_queries, most = 1;
  for (int l = 0; l < n_hops; ++l) {
    BlockHop& h = b.hop[l];
    h.prev_node = l ? node[l - 1] : nullptr;
    h.prev_ts = l ? ts[l - 1] : q_ts;
    h.node = node[l];
    h.ts = ts[l];
    h.d = d;
    h.n = counts[l];
    h.out_node = out;
    h.out_ts = out + (d + h.n);
    h.out_index = out + 2 * (d + h.n);
    out += 2 * (d + h.n) + h.n;
    most = d + h.n > most ? d + h.n : most;
    d = h.n;
  }
  SGL_CHECK_RC(launch(blocks_kernel, dim3((unsigned)stream_grid(most, 256 * 2, 8), (unsigned)n_hops), 256, 0, (cudaStream_t)stream_, b));
  return SGL_OK;
}
