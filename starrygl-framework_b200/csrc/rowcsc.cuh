// CSC of a hop from what is known already: a hop's edges lie target by target, each target's in ascending time, and the sort that
// merged the targets into the layer list left them row by row.  So the edges need no sort of their own:
//   1. csc_rows_count_kernel   edges of every list item in list order, their exclusive sum; rows with too many targets are noticed
//   2. csc_rows_copy_kernel    every edge to its row.  The targets of a row are the same node at the same time, reached along several
//                              edges: they have one candidate window.  Where they took all of it or its tail their edges are the
//                              same, and an edge's place follows from its own list; where they drew, it is the number of edges of
//                              the others that come before it
// A row of more than kMaxRowTargets targets that drew would make step 2 quadratic: then it writes nothing and the sort does all of
// it (sgl_build_csc with the gate as its condition).
//
// Bound by HBM: 28 B read and 36 B written per edge, and the reads of a row's other targets.  14 M edges over 4.2 M targets: the sort
// and its delivery read and wrote every edge's key and position seven times, 1.2 ms next to the merge of the next list.
#pragma once
#include "lists.cuh"

namespace sgl {

// list items in sorted order: number of the target (~0: an item of the list before), its row, and the first item of every row
struct RowOrder {
  uint32_t *order, *row, *first;
  static size_t bytes(int64_t cap) { return 2 * align_up((size_t)cap * 4) + align_up((size_t)(cap + 1) * 4); }
  static RowOrder carve(void* p, int64_t cap) {
    RowOrder r;
    r.order = (uint32_t*)p;
    r.row = (uint32_t*)((char*)p + align_up((size_t)cap * 4));
    r.first = (uint32_t*)((char*)p + 2 * align_up((size_t)cap * 4));
    return r;
  }
};

// sgl_unique_pairs that also leaves the order of its list, and (inv_b32) the inverse of the second part in 32-bit words instead of
// inv_b
int unique_pairs(const int64_t* a_id, const int64_t* a_ts, int64_t n_a, const int64_t* d_n_a, const int64_t* b_id, const int64_t* b_ts,
                 int64_t n_b, const int64_t* d_n_b, int id_bits, int ts_bits, int64_t ts_base, int64_t* out_id, int64_t* out_ts, int64_t* inv_a,
                 int64_t* inv_b, uint32_t* inv_b32, int64_t* d_n_unique, const RowOrder& ro, int32_t* d_status, void* ws, size_t ws_bytes,
                 void* stream);

size_t build_csc_rows_ws_bytes(int64_t n_edges, int64_t list_cap);
// `list_cap` / d_num_dst: capacity of the list's order and its number of rows; row_ts: time of every row; offsets[i]: first edge of target
// i; dt: the row's time minus the edge's, as the sampler writes it
int build_csc_rows(const RowOrder& ro, int64_t list_cap, const int64_t* row_ts, const int64_t* offsets, int fanout, bool draws,
                   const int64_t* dst, const int64_t* dst_map, const int64_t* ts, const float* dt, const int64_t* eid, int64_t n_edges, const int64_t* d_n_edges, int64_t num_dst,
                   const int64_t* d_num_dst, int dst_bits, int ts_bits, int64_t ts_base, int64_t* out_indptr, int64_t* out_indices,
                   int64_t* out_ts, float* out_dt, int64_t* out_eid, int32_t* d_status, void* ws, size_t ws_bytes, void* stream);

}  // namespace sgl
