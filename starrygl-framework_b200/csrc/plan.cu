// Route plan of one layer on the GPU: which rows of the layer's (id, ts) list this partition must push to which
// other ranks, and where they land there.
//
// Input: the layer list sorted by (id, ts) (what the batch builder produces), the owner partition of every node and
// the replica table (CSR over node id of (rank, slot)).  For every distinct node id the row with the latest timestamp
// is the last row of its run.  Rows of nodes owned here are expanded to one entry per replica on another rank, then
// ordered by rank (stable: ascending list row inside a rank).
//
// Up to 32 ranks (three kernels): entries counted per (rank, CTA), one scan of those counts, every entry written straight
// to its place -- no sort over the capacity (rows x (ranks - 1), ten kernels and 250 us for the last list of an 8,000-root
// two-hop slot with 90,000 rows).  More ranks:
//
//   plan_count_kernel   per row: is it the run's last row and owned here? how many foreign replicas? CTA scan,
//                       last CTA scans the CTA totals; per-rank sizes by atomic add (order independent)
//   plan_expand_kernel  writes (rank, row, slot) triplets in row order
//   radix sort on the rank (one 8-bit pass) + plan_emit_kernel gathers rows and slots in sorted order
#include "launch.cuh"
#include "scan.cuh"
#include "sort.cuh"

namespace sgl {
namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads)
plan_count_kernel(const int64_t* __restrict__ ids, int64_t n_cap, const int64_t* d_n, const int64_t* __restrict__ node_parts,
                  int64_t num_nodes, int64_t pid, const int64_t* __restrict__ indptr, const int64_t* __restrict__ ranks,
                  int64_t num_parts, int64_t* __restrict__ local_off, int64_t* __restrict__ cta_sums,
                  unsigned int* done_counter, int64_t* d_total, unsigned long long* __restrict__ send_sizes, int32_t* d_status) {
  const int64_t n = eff_count(n_cap, d_n);
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  int64_t len = 0;
  if (i < n) {
    const int64_t id = ids[i];
    if (id < 0 || id >= num_nodes) {
      dev_flag(d_status, SGL_DEV_BAD_NODE);
    } else {
      if (i + 1 < n && ids[i + 1] < id) dev_flag(d_status, SGL_DEV_BAD_INDEX);   // list must be sorted by id
      const bool tail = (i == n - 1) || ids[i + 1] != id;
      if (tail && node_parts[id] == pid) {
        for (int64_t p = indptr[id]; p < indptr[id + 1]; ++p) {
          const int64_t r = ranks[p];
          if (r != pid && r >= 0 && r < num_parts) {
            ++len;
            atomicAdd(send_sizes + r, 1ull);
          }
        }
      }
    }
  }
  int64_t total;
  int64_t ex = cta_exclusive_scan<kThreads, int64_t>(len, &total);
  if (i < n) local_off[i] = ex;
  publish_and_scan_cta_totals<kThreads>(total, cta_sums, done_counter, d_total);
}

__global__ void __launch_bounds__(kThreads)
plan_expand_kernel(const int64_t* __restrict__ ids, int64_t n_cap, const int64_t* d_n, const int64_t* __restrict__ node_parts,
                   int64_t num_nodes, int64_t pid, const int64_t* __restrict__ indptr, const int64_t* __restrict__ ranks,
                   const int64_t* __restrict__ locs, int64_t num_parts, const int64_t* __restrict__ local_off,
                   const int64_t* __restrict__ cta_sums, int64_t cap, uint64_t* __restrict__ keys,
                   int64_t* __restrict__ tmp_rows, int64_t* __restrict__ tmp_locs, int32_t* d_status) {
  const int64_t n = eff_count(n_cap, d_n);
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const int64_t id = ids[i];
  if (id < 0 || id >= num_nodes) return;
  const bool tail = (i == n - 1) || ids[i + 1] != id;
  if (!tail || node_parts[id] != pid) return;
  int64_t off = cta_sums[blockIdx.x] + local_off[i];
  for (int64_t p = indptr[id]; p < indptr[id + 1]; ++p) {
    const int64_t r = ranks[p];
    if (r == pid || r < 0 || r >= num_parts) continue;
    if (off >= cap) {
      dev_flag(d_status, SGL_DEV_OVERFLOW);
      return;
    }
    keys[off] = (uint64_t)r;
    tmp_rows[off] = i;
    tmp_locs[off] = locs[p];
    ++off;
  }
}

__global__ void __launch_bounds__(kThreads)
plan_emit_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ perm, int64_t cap, const int64_t* d_total,
                 const int64_t* __restrict__ tmp_rows, const int64_t* __restrict__ tmp_locs, int64_t* __restrict__ out_ranks,
                 int64_t* __restrict__ out_rows, int64_t* __restrict__ out_locs) {
  const int64_t n = eff_count(cap, d_total);
  for (int64_t j = (int64_t)blockIdx.x * kThreads + threadIdx.x; j < n; j += (int64_t)gridDim.x * kThreads) {
    const uint32_t p = perm[j] < n ? perm[j] : 0u;      // (a sort that ran into its time limit leaves any value)
    out_ranks[j] = (int64_t)keys[j];
    out_rows[j] = tmp_rows[p];
    out_locs[j] = tmp_locs[p];
  }
}

// ---- up to kFewParts ranks: entries counted per (rank, CTA), placed by rank without a sort --------------------------------
constexpr int kFewParts = 32;
constexpr int kMaxLayers = 9;

// Layer lists whose plans are made side by side (grid.y), one after the other a two-hop slot's three plans took 55 us of kernels.
struct PlanLayer {
  const int64_t *ids, *d_n;
  int64_t n_cap, cap;
  int32_t* tally;
  int64_t *out_ranks, *out_rows, *out_locs, *send_sizes, *total;
};
struct PlanLayers {
  PlanLayer l[kMaxLayers];
};

// does row i send its node's row, and to which copies?  [*s, *e) of the replica lists; false: nothing
__device__ __forceinline__ bool plan_row(const int64_t* __restrict__ ids, int64_t n, int64_t i, const int64_t* __restrict__ node_parts,
                                         int64_t num_nodes, int64_t pid, const int64_t* __restrict__ indptr, int32_t* d_status,
                                         int64_t* s, int64_t* e) {
  const int64_t id = ids[i];
  if (id < 0 || id >= num_nodes) {
    dev_flag(d_status, SGL_DEV_BAD_NODE);
    return false;
  }
  if (i + 1 < n) {
    const int64_t next = ids[i + 1];
    if (next < id) dev_flag(d_status, SGL_DEV_BAD_INDEX);   // list must be sorted by id
    if (next == id) return false;
  }
  if (node_parts[id] != pid) return false;
  *s = indptr[id];
  *e = indptr[id + 1];
  return true;
}

__global__ void __launch_bounds__(kThreads)
plan_tally_kernel(const __grid_constant__ PlanLayers layers, const int64_t* __restrict__ node_parts, int64_t num_nodes, int64_t pid,
                  const int64_t* __restrict__ indptr, const int64_t* __restrict__ ranks, int num_parts, int32_t* d_status) {
  __shared__ int s_cnt[kFewParts];
  const PlanLayer& l = layers.l[blockIdx.y];
  const int64_t* __restrict__ ids = l.ids;
  int32_t* __restrict__ tally = l.tally;
  const int64_t n = eff_count(l.n_cap, l.d_n);
  if ((int64_t)blockIdx.x * kThreads >= n) return;
  if (threadIdx.x < num_parts) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  int64_t s, e;
  if (i < n && plan_row(ids, n, i, node_parts, num_nodes, pid, indptr, d_status, &s, &e))
    for (int64_t p = s; p < e; ++p) {
      const int64_t r = ranks[p];
      if (r != pid && r >= 0 && r < num_parts) atomicAdd(&s_cnt[r], 1);
    }
  __syncthreads();
  const int64_t ctas = (n + kThreads - 1) / kThreads;
  if (threadIdx.x < num_parts) tally[threadIdx.x * ctas + blockIdx.x] = s_cnt[threadIdx.x];
}

// exclusive scan of the (rank, CTA) counts in place, rank by rank; sizes per rank and the total.  One CTA per layer.  The counts of a rank
// lie behind those of the rank before: one scan of all of them, four to a thread (7.4 us with a scan per rank for 4 ranks, 3.9 now).
// Sizes and total are exact whatever they are; a place beyond kLastPlace is kept as kLastPlace, and nothing is written there.
constexpr int32_t kLastPlace = INT32_MAX;
__global__ void __launch_bounds__(1024)
plan_place_kernel(const __grid_constant__ PlanLayers layers, int num_parts) {
  __shared__ int64_t s_carry, s_begin[kFewParts + 1];
  const PlanLayer& l = layers.l[blockIdx.x];
  int32_t* tally = l.tally;
  int64_t *d_send_sizes = l.send_sizes, *d_total = l.total;
  const int64_t n = eff_count(l.n_cap, l.d_n);
  const uint32_t ctas = (uint32_t)((n + kThreads - 1) / kThreads), all = ctas * (uint32_t)num_parts;      // (below 2^24, see few_parts)
  if (threadIdx.x == 0) s_carry = 0;
  if (threadIdx.x <= num_parts) s_begin[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t b = 0; b < all; b += 4 * 1024) {
    const uint32_t j = b + 4 * threadIdx.x;
    int64_t v[4], sum = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = j + u < all ? tally[j + u] : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t x = v[u];
      v[u] = sum;
      sum += x;
    }
    const int64_t carry = s_carry;       // (the barriers of the scan lie between this read and the write below)
    int64_t tot;
    const int64_t at = carry + cta_exclusive_scan<1024, int64_t>(sum, &tot);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j + u >= all) break;
      const int64_t place = at + v[u];
      tally[j + u] = place < kLastPlace ? (int32_t)place : kLastPlace;
      const uint32_t r = (j + u) / ctas;
      if (r * ctas == j + u) s_begin[r] = place;
    }
    if (threadIdx.x == 0) s_carry = carry + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) *d_total = s_begin[num_parts] = s_carry;
  __syncthreads();
  if (threadIdx.x < num_parts) d_send_sizes[threadIdx.x] = s_begin[threadIdx.x + 1] - s_begin[threadIdx.x];
}

// Four ranks at a time share a scan, 16 bits each (three layers, 4 ranks: 11.4 -> 10.9 us), unless a node has more copies than that allows.
// (46 registers, 11.4 us: with the 57 that it would take there is a CTA per SM less, 12.1 us)
__global__ void __launch_bounds__(kThreads, 5)
plan_write_kernel(const __grid_constant__ PlanLayers layers, const int64_t* __restrict__ node_parts, int64_t num_nodes, int64_t pid,
                  const int64_t* __restrict__ indptr, const int64_t* __restrict__ ranks, const int64_t* __restrict__ locs, int num_parts,
                  int32_t* d_status) {
  const PlanLayer& l = layers.l[blockIdx.y];
  const int64_t* __restrict__ ids = l.ids;
  const int32_t* __restrict__ tally = l.tally;
  const int64_t cap = l.cap;
  int64_t *__restrict__ out_ranks = l.out_ranks, *__restrict__ out_rows = l.out_rows, *__restrict__ out_locs = l.out_locs;
  const int64_t n = eff_count(l.n_cap, l.d_n);
  if ((int64_t)blockIdx.x * kThreads >= n) return;
  const int64_t ctas = (n + kThreads - 1) / kThreads;
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  int64_t s = 0, e = 0;
  if (!(i < n && plan_row(ids, n, i, node_parts, num_nodes, pid, indptr, nullptr, &s, &e))) s = e = 0;
  constexpr int64_t kMostCopies = 65535 / kThreads;
  const int width = __syncthreads_or(e - s > kMostCopies) ? 1 : 4;      // ranks per scan
  const int bits = 64 / width;
  for (int r0 = 0; r0 < num_parts; r0 += width) {
    int64_t before[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int32_t place = u < width && r0 + u < num_parts ? tally[(r0 + u) * ctas + blockIdx.x] : 0;
      before[u] = place == kLastPlace ? cap : place;
    }
    uint64_t mine = 0;
    for (int64_t p = s; p < e; ++p) {
      const int64_t r = ranks[p];
      if (r != pid && r >= r0 && r < r0 + width && r < num_parts) mine += 1ull << ((int)(r - r0) * bits);
    }
    uint64_t at = cta_exclusive_scan<kThreads, uint64_t>(mine, nullptr);
    if (mine == 0) continue;
    bool over = false;
    const uint64_t low = width == 1 ? ~0ull : 0xffffull;
    for (int64_t p = s; p < e; ++p) {
      const int64_t r = ranks[p];
      if (r == pid || r < r0 || r >= r0 + width || r >= num_parts) continue;
      const int u = (int)(r - r0);
      const int64_t first = u == 0 ? before[0] : (u == 1 ? before[1] : (u == 2 ? before[2] : before[3]));
      const int64_t to = first + (int64_t)((at >> (u * bits)) & low);
      at += 1ull << (u * bits);
      if (to >= cap) {
        over = true;
        continue;
      }
      out_ranks[to] = r;
      out_rows[to] = i;
      out_locs[to] = locs[p];
    }
    if (over) dev_flag(d_status, SGL_DEV_OVERFLOW);
  }
}

inline int64_t ctas_for(int64_t n) { return (n + kThreads - 1) / kThreads < 1 ? 1 : (n + kThreads - 1) / kThreads; }

bool few_parts(int64_t n, int64_t num_parts) { return num_parts <= kFewParts && n * num_parts < ((int64_t)1 << 31); }

int plan_few(const PlanLayers& layers, int count, int64_t most_n, const int64_t* node_parts, int64_t num_nodes, int64_t pid,
             const int64_t* rep_indptr, const int64_t* rep_ranks, const int64_t* rep_locs, int num_parts, int32_t* d_status,
             cudaStream_t stream) {
  const dim3 grid((unsigned)ctas_for(most_n), (unsigned)count);
  SGL_CHECK_RC(launch(plan_tally_kernel, grid, kThreads, 0, stream, layers, node_parts, num_nodes, pid, rep_indptr, rep_ranks, num_parts,
                      d_status));
  SGL_CHECK_RC(launch(plan_place_kernel, (unsigned)count, 1024, 0, stream, layers, num_parts));
  return launch(plan_write_kernel, grid, kThreads, 0, stream, layers, node_parts, num_nodes, pid, rep_indptr, rep_ranks, rep_locs, num_parts,
                d_status);
}

}  // namespace
}  // namespace sgl

using namespace sgl;

extern "C" size_t sgl_plan_route_ws_bytes(int64_t n, int64_t cap) {
  if (n < 1) n = 1;
  if (cap < 1) cap = 1;
  return align_up((size_t)kFewParts * ctas_for(n) * 4) + align_up((size_t)n * 8) + align_up((size_t)ctas_for(n) * 8) + align_up(8) + 2 * align_up((size_t)cap * 8) +
         2 * align_up((size_t)cap * 4) + 2 * align_up((size_t)cap * 8) + radix_sort_ws_bytes(cap);
}

extern "C" int sgl_plan_route(const int64_t* layer_ids, int64_t n, const int64_t* d_n, const int64_t* node_parts,
                              int64_t num_nodes, int64_t pid, const int64_t* rep_indptr, const int64_t* rep_ranks,
                              const int64_t* rep_locs, int64_t num_parts, int64_t cap, int64_t* out_ranks, int64_t* out_rows,
                              int64_t* out_locs, int64_t* d_send_sizes, int64_t* d_total, int32_t* d_status, void* ws,
                              size_t ws_bytes, void* stream_) {
  SGL_NVTX("sgl_plan_route");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(n >= 0 && cap >= 0 && num_nodes >= 0 && num_parts >= 1 && num_parts <= 256 && pid >= 0 && pid < num_parts,
              SGL_ERR_ARG, "plan_route: bad size (1 <= num_parts <= 256, 0 <= pid < num_parts)");
  SGL_REQUIRE(d_send_sizes && d_total, SGL_ERR_ARG, "plan_route: null counter");
  LaunchScope scope(stream);
  if (n == 0) {
    SGL_CHECK_RC(zero_async(d_send_sizes, (size_t)num_parts * sizeof(int64_t), stream));
    SGL_CHECK_RC(zero_async(d_total, sizeof(int64_t), stream));
    return scope.submit();
  }
  SGL_REQUIRE(layer_ids && node_parts && rep_indptr && rep_ranks && rep_locs && out_ranks && out_rows && out_locs, SGL_ERR_ARG,
              "plan_route: null array");
  const int64_t capc = cap < 1 ? 1 : cap;
  if (few_parts(n, num_parts)) {
    WsCarver c(ws, ws_bytes);
    int32_t* tally = c.take<int32_t>((size_t)(num_parts * ctas_for(n)));
    SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "plan_route: workspace %zu < %zu bytes", ws_bytes, sgl_plan_route_ws_bytes(n, cap));
    PlanLayers layers;
    memset(&layers, 0, sizeof(layers));
    layers.l[0] = PlanLayer{layer_ids, d_n, n, cap, tally, out_ranks, out_rows, out_locs, d_send_sizes, d_total};
    SGL_CHECK_RC(plan_few(layers, 1, n, node_parts, num_nodes, pid, rep_indptr, rep_ranks, rep_locs, (int)num_parts, d_status, stream));
    return scope.submit();
  }
  SGL_CHECK_RC(zero_async(d_send_sizes, (size_t)num_parts * sizeof(int64_t), stream));
  WsCarver c(ws, ws_bytes);
  int64_t* local_off = c.take<int64_t>(n);
  int64_t* cta_sums = c.take<int64_t>(ctas_for(n));
  unsigned int* done = c.take<unsigned int>(1);
  uint64_t* k0 = c.take<uint64_t>(capc);
  uint64_t* k1 = c.take<uint64_t>(capc);
  uint32_t* v0 = c.take<uint32_t>(capc);
  uint32_t* v1 = c.take<uint32_t>(capc);
  int64_t* tmp_rows = c.take<int64_t>(capc);
  int64_t* tmp_locs = c.take<int64_t>(capc);
  size_t sort_bytes = radix_sort_ws_bytes(capc);
  char* sort_ws = c.take<char>(sort_bytes);
  SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "plan_route: workspace %zu < %zu bytes", ws_bytes, sgl_plan_route_ws_bytes(n, cap));
  SGL_CHECK_RC(zero_async(done, sizeof(unsigned int), stream));
  SGL_CHECK_RC(launch(plan_count_kernel, (unsigned)ctas_for(n), kThreads, 0, stream, layer_ids, n, d_n, node_parts,
                      num_nodes, pid, rep_indptr, rep_ranks, num_parts, local_off, cta_sums, done, d_total, (unsigned long
                      long*)d_send_sizes, d_status));
  SGL_CHECK_RC(launch(plan_expand_kernel, (unsigned)ctas_for(n), kThreads, 0, stream, layer_ids, n, d_n, node_parts,
                      num_nodes, pid, rep_indptr, rep_ranks, rep_locs, num_parts, local_off, cta_sums, cap, k0, tmp_rows,
                      tmp_locs, d_status));

  int in_alt = 0;
  int rc = radix_sort_pairs(k0, v0, k1, v1, capc, d_total, bits_for((uint64_t)(num_parts - 1)), true, &in_alt, d_status, sort_ws, sort_bytes,
                            stream);
  if (rc) return rc;
  SGL_CHECK_RC(launch(plan_emit_kernel, stream_grid(capc, kThreads, 8), kThreads, 0, stream, in_alt ? k1 : k0, in_alt ? v1 :
                      v0, capc, d_total, tmp_rows, tmp_locs, out_ranks, out_rows, out_locs));
  return scope.submit();
}

extern "C" size_t sgl_plan_routes_ws_bytes(int layers, const int64_t* n, const int64_t* cap) {
  size_t sum = 0, most = 0;
  for (int i = 0; i < layers; ++i) {
    const size_t one = align_up(sgl_plan_route_ws_bytes(n[i], cap[i]));
    most = one > most ? one : most;
    sum += align_up((size_t)kFewParts * ctas_for(n[i]) * 4);
  }
  return sum > most ? sum : most;
}

extern "C" int sgl_plan_routes(int layers, const int64_t* const* layer_ids, const int64_t* n, const int64_t* const* d_n,
                               const int64_t* node_parts, int64_t num_nodes, int64_t pid, const int64_t* rep_indptr,
                               const int64_t* rep_ranks, const int64_t* rep_locs, int64_t num_parts, const int64_t* cap,
                               int64_t* const* out, int64_t* const* d_counts, int32_t* d_status, void* ws, size_t ws_bytes, void* stream_) {
  SGL_NVTX("sgl_plan_routes");
  cudaStream_t stream = (cudaStream_t)stream_;
  SGL_REQUIRE(layers >= 0 && (layers == 0 || (layer_ids && n && d_n && cap && out && d_counts)), SGL_ERR_ARG, "plan_routes: null table");
  LaunchScope scope(stream);
  bool few = layers <= kMaxLayers && num_parts >= 1 && pid >= 0 && pid < num_parts && num_nodes >= 0 && node_parts && rep_indptr && rep_ranks &&
             rep_locs;
  for (int i = 0; i < layers && few; ++i) few = n[i] > 0 && cap[i] > 0 && few_parts(n[i], num_parts) && layer_ids[i] && out[i] && d_counts[i];
  if (few && layers > 0) {
    WsCarver c(ws, ws_bytes);
    PlanLayers l;
    memset(&l, 0, sizeof(l));
    int64_t most = 1;
    for (int i = 0; i < layers; ++i) {
      int32_t* tally = c.take<int32_t>((size_t)(num_parts * ctas_for(n[i])));
      l.l[i] = PlanLayer{layer_ids[i], d_n[i], n[i], cap[i], tally, out[i], out[i] + cap[i], out[i] + 2 * cap[i], d_counts[i],
                         d_counts[i] + num_parts};
      most = n[i] > most ? n[i] : most;
    }
    SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "plan_routes: workspace %zu < %zu bytes", ws_bytes, sgl_plan_routes_ws_bytes(layers, n, cap));
    SGL_CHECK_RC(plan_few(l, layers, most, node_parts, num_nodes, pid, rep_indptr, rep_ranks, rep_locs, (int)num_parts, d_status, stream));
  } else {
    for (int i = 0; i < layers; ++i)
      SGL_CHECK_RC(sgl_plan_route(layer_ids[i], n[i], d_n[i], node_parts, num_nodes, pid, rep_indptr, rep_ranks, rep_locs, num_parts, cap[i],
                                  out[i], out[i] + cap[i], out[i] + 2 * cap[i], d_counts[i], d_counts[i] + num_parts, d_status, ws, ws_bytes,
                                  stream_));
  }
  return scope.submit();
}
