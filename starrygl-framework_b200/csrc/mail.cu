// Mailbox update of a mini-batch: "latest message per node" reduce, row assembly and the write into the mailbox.
//
// The reference concatenates the batch's source and destination nodes, builds one mail row per entry
// ([own memory | other end's memory | edge feature]), and keeps for every distinct node the entry with the largest
// timestamp (unique + scatter_max + index).  Here the 2B x width mail matrix is never materialised: the entries are sorted
// by (node, latest time first, position; sources first, then destinations), so that a node's winner -- the largest
// timestamp and, among equal timestamps, the FIRST entry -- is the first of its run, and mail_emit_kernel gathers the
// winners' rows straight from the per-event tables.
//
// Timestamps are compared as fp32, like the reference, which converts them to the mailbox dtype before the reduce.
// Algorithmic HBM bytes: 8 + 4|8 read per entry + sort passes (32 B per entry and populated key byte), and per
// unique node 2 * row bytes + 20 written / read.
#include "chain.cuh"
#include "lsd.cuh"

namespace sgl {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxSeg = 4;

struct Segs {
  const float* a[kMaxSeg];   // source of the segment for entries of the first list (row = entry position)
  const float* b[kMaxSeg];   // ... of the second list (row = position - n_a)
  int64_t dim[kMaxSeg];
  int n;
};

__device__ __forceinline__ float ts_at(const void* ts, int64_t ts_len, int is_i64, int64_t pos) {
  const int64_t k = pos < ts_len ? pos : pos - ts_len;   // cat(ts, ts) when one value per event is given
  return is_i64 ? (float)((const int64_t*)ts)[k] : ((const float*)ts)[k];
}

// monotone map fp32 -> uint32 (larger float, larger integer)
__device__ __forceinline__ uint32_t orderable(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct Words4 {
  using T = float4;
};
struct Words1 {
  using T = float;
};

// One warp per unique node: the winner's position and timestamp, and its mail row out of the per-event tables, in pieces of
// 16 bytes when every segment allows it (W = Words4; 7,000 rows of 372 values: 10.8 us in pieces of 4 bytes).
template <class W>
__global__ void __launch_bounds__(kThreads)
mail_emit_kernel(const uint32_t* __restrict__ winner, int64_t n_cap, const int64_t* d_num_unique, int64_t n_a,
                 const void* ts, int64_t ts_len, int ts_is_i64, Segs segs, int64_t width,
                 int64_t* __restrict__ out_pos, float* __restrict__ out_ts, float* __restrict__ out_mail) {
  using T = typename W::T;
  constexpr int kPer = sizeof(T) / 4;
  const int64_t n = eff_count(n_cap, d_num_unique);
  const int lane = threadIdx.x & 31;
  const int64_t n_warps = (int64_t)gridDim.x * (kThreads / 32);
  for (int64_t u = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5; u < n; u += n_warps) {
    const int64_t pos = winner[u];
    if (lane == 0) {
      if (out_pos) out_pos[u] = pos;
      if (out_ts) out_ts[u] = ts_at(ts, ts_len, ts_is_i64, pos);
    }
    if (!out_mail) continue;
    const bool first = pos < n_a;
    const int64_t row = first ? pos : pos - n_a;
    T* dst = (T*)(out_mail + u * width);
    int64_t off = 0;
    for (int s = 0; s < segs.n; ++s) {
      const int64_t words = segs.dim[s] / kPer;
      const T* src = (const T*)((first ? segs.a[s] : segs.b[s]) + row * segs.dim[s]);
      for (int64_t e = lane; e < words; e += 32) dst[off + e] = __ldg(src + e);
      off += words;
    }
  }
}

// mailbox[node, next_pos[node], :] = mail[u, :], the timestamp alongside, and the ring position advanced.
// One warp per row; `index` holds distinct nodes (the output of the reduce), so no two warps touch one node.
template <class W>
__global__ void __launch_bounds__(kThreads)
mailbox_write_kernel(const int64_t* __restrict__ index, int64_t n_cap, const int64_t* d_n, const float* __restrict__ mail,
                     const float* __restrict__ mail_ts, int64_t width, float* __restrict__ mailbox,
                     float* __restrict__ mailbox_ts, int64_t* __restrict__ next_pos, int64_t num_nodes, int64_t mailbox_size,
                     int advance, int32_t* d_status) {
  using T = typename W::T;
  const int64_t n = eff_count(n_cap, d_n), words = width / (int64_t)(sizeof(T) / 4);
  const int lane = threadIdx.x & 31;
  const int64_t n_warps = (int64_t)gridDim.x * (kThreads / 32);
  for (int64_t u = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5; u < n; u += n_warps) {
    const int64_t g = index[u];
    if (g < 0 || g >= num_nodes) {
      if (lane == 0) dev_flag(d_status, SGL_DEV_BAD_NODE);
      continue;
    }
    int64_t p = next_pos ? next_pos[g] : 0;
    if (p < 0 || p >= mailbox_size) {
      if (lane == 0) dev_flag(d_status, SGL_DEV_BAD_INDEX);
      continue;
    }
    T* dst = (T*)(mailbox + (g * mailbox_size + p) * width);
    const T* src = (const T*)(mail + u * width);
#pragma unroll 4
    for (int64_t e = lane; e < words; e += 32) dst[e] = __ldg(src + e);
    __syncwarp();   // every lane has read next_pos[g] before lane 0 advances it
    if (lane == 0) {
      mailbox_ts[g * mailbox_size + p] = mail_ts[u];
      if (advance && next_pos && mailbox_size > 1) next_pos[g] = (p + 1) % mailbox_size;
    }
  }
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

struct MailSource {
  static constexpr bool kOnDemand = false;
  const int64_t *ids_a, *ids_b;
  int64_t n_a, n, num_nodes;
  const void* ts;
  int64_t ts_len;
  int ts_is_i64;
  int32_t* d_status;
  __device__ __forceinline__ int64_t begin() const { return n; }
  struct Raw {
    int64_t g;
    uint32_t late;
  };
  __device__ __forceinline__ Raw load(int64_t j) const { return {j < n_a ? ids_a[j] : ids_b[j - n_a], late_first(j)}; }
  __device__ __forceinline__ uint64_t key(const Raw& x) const {
    int64_t g = x.g;
    if (g < 0 || g >= num_nodes) {
      dev_flag(d_status, SGL_DEV_BAD_NODE);
      g = 0;
    }
    return ((uint64_t)g << 32) | x.late;
  }
  __device__ __forceinline__ uint32_t late_first(int64_t j) const { return ~orderable(ts_at(ts, ts_len, ts_is_i64, j)); }
};

// Node ids beyond 32 bits leave no room for the time in the key: sorted by time first, then stably by node.
struct MailTimes {
  static constexpr bool kOnDemand = false;
  MailSource m;
  __device__ __forceinline__ int64_t begin() const { return m.n; }
  using Raw = uint32_t;
  __device__ __forceinline__ Raw load(int64_t j) const { return m.late_first(j); }
  __device__ __forceinline__ uint64_t key(Raw x) const { return x; }
};
struct OrderSink {
  static constexpr bool kUnique = false, kAfter = false;
  uint32_t* order;
  __device__ __forceinline__ void begin() const {}
  __device__ __forceinline__ void item(int64_t at, uint64_t, uint32_t pos) const { order[at] = pos; }
  __device__ __forceinline__ void between(int64_t, uint64_t, bool, uint64_t) const {}
  __device__ __forceinline__ void finish(int64_t, uint64_t, bool, int64_t, int64_t) const {}
};
struct MailNodes {
  static constexpr bool kOnDemand = false;
  MailSource m;
  const uint32_t* order;
  __device__ __forceinline__ int64_t begin() const { return m.n; }
  using Raw = int64_t;
  __device__ __forceinline__ Raw load(int64_t i) const {
    const int64_t j = order[i];
    return j < m.n_a ? m.ids_a[j] : m.ids_b[j - m.n_a];
  }
  __device__ __forceinline__ uint64_t key(Raw g) const {
    if (g >= 0 && g < m.num_nodes) return (uint64_t)g;
    dev_flag(m.d_status, SGL_DEV_BAD_NODE);
    return 0;
  }
};

struct MailSink {
  static constexpr bool kUnique = true, kAfter = false;
  static constexpr int kLevels = 1;
  int64_t* out_index;
  uint32_t* winner;
  int64_t* d_num_unique;
  const uint32_t* order;     // what the positions count (nullptr: the entries themselves)
  int node_shift;
  __device__ __forceinline__ void begin() const {}
  __device__ __forceinline__ bool counted(uint64_t) const { return true; }
  __device__ __forceinline__ uint64_t group(uint64_t k) const { return k >> node_shift; }
  __device__ __forceinline__ void item(int64_t, uint64_t k, uint32_t pos, bool head, int64_t u, bool, int64_t) const {
    if (!head) return;
    out_index[u] = (int64_t)(k >> node_shift);
    winner[u] = order ? order[pos] : pos;
  }
  __device__ __forceinline__ void finish(int64_t, uint64_t, bool, int64_t groups, int64_t) const {
    if (threadIdx.x == 0) *d_num_unique = groups;
  }
};


}  // namespace
}  // namespace sgl

using namespace sgl;

extern "C" size_t sgl_mail_reduce_ws_bytes(int64_t n_entries) {
  const int64_t n = n_entries < 1 ? 1 : n_entries;
  return 2 * align_up((size_t)n * 4) + list_ws_bytes(n);
}

extern "C" int sgl_mail_reduce_counted(const int64_t* ids_a, int64_t n_a, const int64_t* ids_b, int64_t n_b, int64_t num_nodes,
                               const void* ts, int64_t ts_len, int ts_is_i64, int n_seg, const float* const* seg_a,
                               const float* const* seg_b, const int64_t* seg_dim, int64_t* out_index, int64_t* out_pos,
                               float* out_ts, float* out_mail, int64_t* d_num_unique, int32_t* d_status, void* ws,
                               size_t ws_bytes, int64_t* host_unique, int64_t seq, void* stream_) {
  SGL_NVTX("sgl_mail_reduce");
  cudaStream_t stream = (cudaStream_t)stream_;
  const int64_t n = n_a + n_b;
  SGL_REQUIRE(n_a >= 0 && n_b >= 0 && num_nodes >= 0 && n <= 0xffffffffll, SGL_ERR_ARG, "mail_reduce: bad size");
  SGL_REQUIRE(d_num_unique, SGL_ERR_ARG, "mail_reduce: null counter");
  SGL_REQUIRE(n_seg >= 0 && n_seg <= kMaxSeg, SGL_ERR_ARG, "mail_reduce: at most %d row segments", kMaxSeg);
  if (n == 0) {
    SGL_CHECK_RC(zero_async(d_num_unique, sizeof(int64_t), stream));
    if (host_unique) {
      host_unique[0] = 0;
      host_unique[1] = seq;
    }
    return SGL_OK;
  }
  SGL_REQUIRE((n_a == 0 || ids_a) && (n_b == 0 || ids_b) && ts && out_index, SGL_ERR_ARG, "mail_reduce: null array");
  SGL_REQUIRE(ts_len == n || (ts_len == n_a && n_a == n_b), SGL_ERR_ARG,
              "mail_reduce: ts must hold one value per entry, or one per event when both lists have that length");
  Segs segs;
  memset(&segs, 0, sizeof(segs));
  segs.n = out_mail ? n_seg : 0;
  int64_t width = 0;
  for (int s = 0; s < segs.n; ++s) {
    SGL_REQUIRE(seg_dim && seg_a && seg_b && seg_dim[s] >= 0, SGL_ERR_ARG, "mail_reduce: bad segment table");
    SGL_REQUIRE(seg_dim[s] == 0 || ((n_a == 0 || seg_a[s]) && (n_b == 0 || seg_b[s])), SGL_ERR_ARG,
                "mail_reduce: segment %d has a null source", s);
    segs.a[s] = seg_a[s];
    segs.b[s] = seg_b[s];
    segs.dim[s] = seg_dim[s];
    width += seg_dim[s];
  }
  const int id_bits = bits_for(num_nodes > 0 ? (uint64_t)(num_nodes - 1) : 0);
  bool quads = aligned16(out_mail);
  for (int s = 0; s < segs.n; ++s) quads = quads && segs.dim[s] % 4 == 0 && aligned16(segs.a[s]) && aligned16(segs.b[s]);
  SGL_REQUIRE(ws && ws_bytes >= sgl_mail_reduce_ws_bytes(n), SGL_ERR_WORKSPACE, "mail_reduce: workspace %zu < %zu bytes", ws_bytes,
              sgl_mail_reduce_ws_bytes(n));
  uint32_t *winner = (uint32_t*)ws, *order = (uint32_t*)((char*)ws + align_up((size_t)n * 4));
  void* sort_ws = (char*)ws + 2 * align_up((size_t)n * 4);
  const size_t sort_bytes = ws_bytes - 2 * align_up((size_t)n * 4);
  const MailSource entries{ids_a, ids_b, n_a, n, num_nodes, ts, ts_len, ts_is_i64, d_status};
  LaunchScope scope(stream);
  if (id_bits <= 32) {
    SGL_CHECK_RC(sort_list(entries, MailSink{out_index, winner, d_num_unique, nullptr, 32}, n, id_bits + 32, sort_ws, sort_bytes, d_status,
                           stream));
  } else {
    SGL_CHECK_RC(sort_list(MailTimes{entries}, OrderSink{order}, n, 32, sort_ws, sort_bytes, d_status, stream));
    SGL_CHECK_RC(sort_list(MailNodes{entries, order}, MailSink{out_index, winner, d_num_unique, order, 0}, n, id_bits, sort_ws, sort_bytes,
                           d_status, stream));
  }
  if (LaunchScope* in = host_unique ? LaunchScope::current() : nullptr) {
    // the number of nodes is on its way while the rows are put together (a second chain of the graph)
    cudaStream_t side = (cudaStream_t)(uintptr_t)3;
    SGL_CHECK_RC(in->follow(side, stream));
    SGL_CHECK_RC(launch(export_words_kernel, 1, 32, 0, side, d_num_unique, host_unique, 1, seq));
  }
  const int grid = stream_grid(n, kThreads / 32, 8);
  if (quads)
    SGL_CHECK_RC(launch(mail_emit_kernel<Words4>, grid, kThreads, 0, stream, winner, n, d_num_unique, n_a, ts, ts_len, ts_is_i64, segs,
                        width, out_pos, out_ts, out_mail));
  else
    SGL_CHECK_RC(launch(mail_emit_kernel<Words1>, grid, kThreads, 0, stream, winner, n, d_num_unique, n_a, ts, ts_len, ts_is_i64, segs,
                        width, out_pos, out_ts, out_mail));
  return scope.submit();
}

extern "C" int sgl_mail_reduce(const int64_t* ids_a, int64_t n_a, const int64_t* ids_b, int64_t n_b, int64_t num_nodes, const void* ts,
                               int64_t ts_len, int ts_is_i64, int n_seg, const float* const* seg_a, const float* const* seg_b,
                               const int64_t* seg_dim, int64_t* out_index, int64_t* out_pos, float* out_ts, float* out_mail,
                               int64_t* d_num_unique, int32_t* d_status, void* ws, size_t ws_bytes, void* stream) {
  return sgl_mail_reduce_counted(ids_a, n_a, ids_b, n_b, num_nodes, ts, ts_len, ts_is_i64, n_seg, seg_a, seg_b, seg_dim, out_index, out_pos,
                                 out_ts, out_mail, d_num_unique, d_status, ws, ws_bytes, nullptr, 0, stream);
}

extern "C" int sgl_mailbox_write(const int64_t* index, int64_t n, const int64_t* d_n, const float* mail, const float* mail_ts,
                                 int64_t width, float* mailbox, float* mailbox_ts, int64_t* next_mail_pos, int64_t num_nodes,
                                 int64_t mailbox_size, int advance, int32_t* d_status, void* stream_) {
  SGL_NVTX("sgl_mailbox_write");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n >= 0 && width >= 1 && num_nodes >= 0 && mailbox_size >= 1, SGL_ERR_ARG, "mailbox_write: bad size");
  if (n == 0) return SGL_OK;
  SGL_REQUIRE(index && mail && mail_ts && mailbox && mailbox_ts, SGL_ERR_ARG, "mailbox_write: null array");
  SGL_REQUIRE(mailbox_size == 1 || next_mail_pos, SGL_ERR_ARG, "mailbox_write: a mailbox of several slots needs next_mail_pos");
  const int grid = stream_grid(n, kThreads / 32, 8);
  if (width % 4 == 0 && aligned16(mail) && aligned16(mailbox))
    SGL_CHECK_RC(launch(mailbox_write_kernel<Words4>, grid, kThreads, 0, stream, index, n, d_n, mail, mail_ts, width,
                        mailbox, mailbox_ts, next_mail_pos, num_nodes, mailbox_size, advance, d_status));
  else
    SGL_CHECK_RC(launch(mailbox_write_kernel<Words1>, grid, kThreads, 0, stream, index, n, d_n, mail, mail_ts, width,
                        mailbox, mailbox_ts, next_mail_pos, num_nodes, mailbox_size, advance, d_status));
  return SGL_OK;
}
