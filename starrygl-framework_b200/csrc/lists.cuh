#pragma once
#include "tilesort.cuh"

namespace sgl {

__device__ __forceinline__ uint64_t low_mask(int bits) { return bits >= 64 ? ~0ull : ((1ull << bits) - 1ull); }

// Producers and consumers of sorted lists: the dedup / relabel operations, fused into the sort's kernels (sort_list in lsd.cuh;
// pack, sort passes, head scan and emit were 8 - 9 kernels and a memset).
struct PairSource {
  static constexpr bool kOnDemand = false;
  const int64_t *a_id, *a_ts, *d_n_a, *b_id, *b_ts, *d_n_b;
  int64_t n_a, n_b;
  int id_bits, ts_bits;
  int64_t ts_base;
  int32_t* d_status;
  __device__ __forceinline__ int64_t begin() {
    n_a = eff_count(n_a, d_n_a);
    n_b = eff_count(n_b, d_n_b);
    return n_a + n_b;
  }
  using Raw = longlong2;
  __device__ __forceinline__ Raw load(int64_t i) const {
    const bool a = i < n_a;              // (selects addresses, not values: loads without branches overlap)
    const int64_t j = a ? i : i - n_a;
    return {(a ? a_id : b_id)[j], (a ? a_ts : b_ts)[j]};
  }
  __device__ __forceinline__ uint64_t key(const Raw& x) const {
    int64_t id = x.x;
    const int64_t t = x.y;
    uint64_t dt = (uint64_t)t - (uint64_t)ts_base;
    if (id < 0 || ((uint64_t)id & ~low_mask(id_bits))) { dev_flag(d_status, SGL_DEV_BAD_NODE); id = 0; }
    if (t < ts_base || (dt & ~low_mask(ts_bits))) { dev_flag(d_status, SGL_DEV_BAD_TS); dt = 0; }
    return ts_bits >= 64 ? dt : (((uint64_t)id << ts_bits) | dt);
  }
};

struct PairSink {
  static constexpr bool kUnique = true, kAfter = false;
  static constexpr int kLevels = 1;
  int64_t n_a;
  const int64_t* d_n_a;
  int ts_bits;
  int64_t ts_base;
  int64_t *out_id, *out_ts, *inv_a, *inv_b, *d_n_unique;
  uint32_t *order, *row, *first;         // optional: see RowOrder
  uint32_t* inv_b32;                     // optional: in place of inv_b
  __device__ __forceinline__ void begin() { n_a = eff_count(n_a, d_n_a); }
  __device__ __forceinline__ bool counted(uint64_t) const { return true; }
  __device__ __forceinline__ uint64_t group(uint64_t k) const { return k; }
  __device__ __forceinline__ void item(int64_t at, uint64_t k, uint32_t pos, bool head, int64_t u, bool, int64_t) const {
    if (order) {
      order[at] = (int64_t)pos < n_a ? ~0u : (uint32_t)(pos - n_a);
      row[at] = (uint32_t)u;
      if (head) first[u] = (uint32_t)at;
    }
    if (head) {
      __stcs((long long*)out_id + u, ts_bits >= 64 ? 0ll : (long long)(k >> ts_bits));
      __stcs((long long*)out_ts + u, (long long)((int64_t)(k & low_mask(ts_bits)) + ts_base));
    }
    if ((int64_t)pos < n_a) {
      if (inv_a) inv_a[pos] = u;
    } else if (inv_b32) {
      inv_b32[(int64_t)pos - n_a] = (uint32_t)u;
    } else if (inv_b) {
      inv_b[(int64_t)pos - n_a] = u;
    }
  }
  __device__ __forceinline__ void finish(int64_t n, uint64_t, bool, int64_t groups, int64_t) const {
    if (threadIdx.x == 0) {
      *d_n_unique = groups;
      if (order) first[groups] = (uint32_t)n;
    }
  }
};

struct CscSource {
  static constexpr bool kOnDemand = true;
  const int64_t *dst, *dst_map, *ts, *d_n;
  int64_t n_cap;
  int dst_bits, ts_bits;
  int64_t ts_base;
  const int* gate;                       // optional: 0 = another kernel has done the work
  int32_t* d_status;
  bool on_demand() const { return gate != nullptr; }
  __device__ __forceinline__ int64_t begin() const { return gate && *gate == 0 ? 0 : eff_count(n_cap, d_n); }
  using Raw = longlong2;
  __device__ __forceinline__ Raw load(int64_t e) const { return {dst_map ? dst_map[dst[e]] : dst[e], ts[e]}; }
  __device__ __forceinline__ uint64_t key(const Raw& x) const {
    int64_t d = x.x;
    const int64_t t = x.y;
    uint64_t dt = (uint64_t)t - (uint64_t)ts_base;
    if (d < 0 || ((uint64_t)d & ~low_mask(dst_bits))) { dev_flag(d_status, SGL_DEV_BAD_NODE); d = 0; }
    if (t < ts_base || (dt & ~low_mask(ts_bits))) { dev_flag(d_status, SGL_DEV_BAD_TS); dt = 0; }
    return ts_bits >= 64 ? dt : (((uint64_t)d << ts_bits) | dt);
  }
};

struct CscSink {
  static constexpr bool kUnique = false, kAfter = false;
  int64_t num_dst;
  const int64_t* d_num_dst;
  int ts_bits;
  const int64_t *src_local, *ts;
  const float* dt;
  const int64_t* eid;
  int64_t *indptr, *out_indices, *out_ts;
  float* out_dt;
  int64_t* out_eid;
  const int* gate;                       // as in CscSource
  __device__ __forceinline__ void begin() { num_dst = gate && *gate == 0 ? -1 : eff_count(num_dst, d_num_dst); }
  __device__ __forceinline__ int64_t row(uint64_t k) const { return ts_bits >= 64 ? 0 : (int64_t)(k >> ts_bits); }
  __device__ __forceinline__ void item(int64_t at, uint64_t, uint32_t p) const {
    out_indices[at] = src_local ? src_local[p] : (int64_t)p;
    out_ts[at] = ts[p];
    out_dt[at] = dt[p];
    out_eid[at] = eid[p];
  }
  __device__ __forceinline__ void between(int64_t at, uint64_t k, bool has_prev, uint64_t prev) const {
    const int64_t d = row(k);
    for (int64_t v = has_prev ? row(prev) + 1 : 0; v <= d && v <= num_dst; ++v) indptr[v] = at;
  }
  __device__ __forceinline__ void finish(int64_t n, uint64_t last, bool has_last, int64_t, int64_t) const {
    for (int64_t v = (has_last ? row(last) + 1 : 0) + threadIdx.x; v <= num_dst; v += blockDim.x) indptr[v] = n;
  }
};

struct NodesSource {
  static constexpr bool kOnDemand = false;
  const int64_t *ids, *d_n;
  int64_t n_cap, num_nodes;
  const int64_t* mask;
  int64_t epoch;
  int id_bits;
  int32_t* d_status;
  __device__ __forceinline__ int64_t begin() const { return eff_count(n_cap, d_n); }
  using Raw = longlong2;                 // id, epoch of the node
  __device__ __forceinline__ Raw load(int64_t i) const {
    const int64_t g = ids[i];
    return {g, g >= 0 && g < num_nodes ? mask[g] : 0};
  }
  __device__ __forceinline__ uint64_t key(const Raw& x) const {
    const int64_t g = x.x;
    if (g < 0 || g >= num_nodes) {
      dev_flag(d_status, SGL_DEV_BAD_NODE);
      return 1ull << id_bits;            // invalid and already known ids sort behind every new id
    }
    return x.y != epoch ? (uint64_t)g : 1ull << id_bits;
  }
};

struct NodesSink {
  static constexpr bool kUnique = true, kAfter = true;
  static constexpr int kLevels = 1;
  const int64_t* ids;
  int64_t num_nodes;
  int id_bits;
  int64_t *mapper, *mask;
  int64_t epoch;
  int64_t *d_next_local, *out_local, *out_new_ids, *d_n_new;
  const int64_t* d_start;    // optional: out_new_ids[0] is the id of local number *d_start (lists that continue each other)
  int64_t next;
  __device__ __forceinline__ void begin() {
    next = *(volatile int64_t*)d_next_local;
    if (d_start) out_new_ids += next - *d_start;
  }
  __device__ __forceinline__ bool counted(uint64_t k) const { return (k >> id_bits) == 0; }
  __device__ __forceinline__ uint64_t group(uint64_t k) const { return k; }
  __device__ __forceinline__ void item(int64_t, uint64_t k, uint32_t pos, bool head, int64_t u, bool, int64_t) const {
    if (counted(k)) {
      if (head) {
        mapper[k] = next + u;
        mask[k] = epoch;
        out_new_ids[u] = (int64_t)k;
      }
      out_local[pos] = next + u;
    } else {
      const int64_t g = ids[pos];        // known before this call: its entry does not change during it
      out_local[pos] = (g >= 0 && g < num_nodes) ? mapper[g] : -1;
    }
  }
  __device__ __forceinline__ void finish(int64_t, uint64_t, bool, int64_t groups, int64_t) const {
    if (threadIdx.x == 0) *d_n_new = groups;
  }
  __device__ __forceinline__ void after() const { *d_next_local = next + *(volatile int64_t*)d_n_new; }
};

// Events of the window by (source, time); events outside the chosen chunks sort behind.  Groups: (source, time) pairs;
// coarser groups: sources.
struct SeedsSource {
  static constexpr bool kOnDemand = false;
  const int64_t *ev_src, *ev_ts;
  int64_t n;
  const int64_t* win;        // optional: {first event, number of events} on the device; n is the capacity then
  const int64_t* node_chunk;
  const uint8_t* chunk_mask;
  int64_t num_chunks, num_nodes;
  int id_bits, ts_bits;
  int64_t ts_base;
  int32_t* d_status;
  __device__ __forceinline__ int64_t begin() {
    if (win) {
      ev_src += win[0];
      ev_ts += win[0];
      n = eff_count(n, win + 1);
    }
    return n;
  }
  struct Raw {
    int64_t s, t;
    bool take;
  };
  __device__ __forceinline__ Raw load(int64_t j) const {
    Raw x{ev_src[j], ev_ts[j], true};
    if (chunk_mask && x.s >= 0 && x.s < num_nodes) {
      const int64_t c = node_chunk ? node_chunk[x.s] : 0;
      x.take = c >= 0 && c < num_chunks && chunk_mask[c];
    }
    return x;
  }
  __device__ __forceinline__ uint64_t key(const Raw& x) const {
    const int64_t s = x.s, t = x.t;
    const uint64_t dt = (uint64_t)t - (uint64_t)ts_base;
    if (s < 0 || s >= num_nodes) {
      dev_flag(d_status, SGL_DEV_BAD_NODE);
    } else if (t < ts_base || (dt & ~low_mask(ts_bits))) {
      dev_flag(d_status, SGL_DEV_BAD_TS);
    } else {
      if (x.take) return ((uint64_t)s << ts_bits) | dt;
    }
    return 1ull << (id_bits + ts_bits);
  }
};

struct SeedsSink {
  static constexpr bool kUnique = true, kAfter = true;
  static constexpr int kLevels = 2;
  const int64_t* win;        // as in SeedsSource
  int key_bits, ts_bits;
  int64_t ts_base;
  const int64_t* ev_eid;
  int64_t *out_roots, *out_ts_ptr, *out_ts, *out_q_ptr, *out_q_eid, *d_counts;
  int64_t* out_pair_node;    // optional: the node of every pair
  unsigned long long* d_valid;
  __device__ __forceinline__ void begin() {
    if (win) ev_eid += win[0];
  }
  __device__ __forceinline__ bool counted(uint64_t k) const { return (k >> key_bits) == 0; }
  __device__ __forceinline__ uint64_t group(uint64_t k) const { return k; }
  __device__ __forceinline__ uint64_t group2(uint64_t k) const { return k >> ts_bits; }
  __device__ __forceinline__ void item(int64_t at, uint64_t k, uint32_t pos, bool head, int64_t u, bool head2, int64_t u2) const {
    if (!counted(k)) return;
    out_q_eid[at] = ev_eid[pos];
    if (head) {
      out_ts[u] = (int64_t)(k & low_mask(ts_bits)) + ts_base;
      out_q_ptr[u] = at;
      if (out_pair_node) out_pair_node[u] = (int64_t)(k >> ts_bits);
    }
    if (head2) {
      out_roots[u2] = (int64_t)(k >> ts_bits);
      out_ts_ptr[u2] = u;
    }
    // number of selected events: they come first (one atomic per warp)
    const unsigned act = __activemask(), upto = __reduce_max_sync(act, (unsigned)at + 1u);
    if ((threadIdx.x & 31) == (unsigned)__ffs(act) - 1u) atomicMax(d_valid, (unsigned long long)upto);
  }
  __device__ __forceinline__ void finish(int64_t, uint64_t, bool, int64_t groups, int64_t groups2) const {
    if (threadIdx.x == 0) {
      d_counts[0] = groups2;
      d_counts[1] = groups;
    }
  }
  __device__ __forceinline__ void after() const {
    volatile int64_t* c = d_counts;
    const int64_t valid = (int64_t)*(volatile unsigned long long*)d_valid;
    out_q_ptr[c[1]] = valid;
    out_ts_ptr[c[0]] = c[1];
    c[2] = valid;
  }
};

// What relabel_nodes refuses whatever its arrays: for entry points that start work before they set up the relabels.
int check_relabel(int64_t n, int64_t num_nodes);

// sgl_relabel_nodes for lists that continue each other: with d_start, out_new_ids[0] is the id of local number *d_start.
int relabel_nodes(const int64_t* ids, int64_t n, const int64_t* d_n, int64_t num_nodes, int64_t* mapper, int64_t* mask, int64_t epoch,
                  int64_t* d_next_local, int64_t* out_local, int64_t* out_new_ids, int64_t* d_n_new, const int64_t* d_start,
                  int32_t* d_status, void* ws, size_t ws_bytes, void* stream);

}  // namespace sgl
