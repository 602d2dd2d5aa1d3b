// One hop of temporal sampling (sampler.cu) for the other translation units: sgl_sample_layer_fenced with a second place for
// the number of sampled edges, and (host_total, see sgl_sample_layer_counted) a third.
#pragma once
#include "common.cuh"

namespace sgl {
// What sample_layer refuses whatever its arrays: for entry points that start work before they set up the hops.
int check_sampling(int fanout, int policy, int64_t n_targets);

int sample_layer(const int64_t* indptr, const int64_t* nbr, const int64_t* ts, const int64_t* eid, const int64_t* fence,
                 int64_t num_nodes, const int64_t* targets, const int64_t* target_ts, int64_t n_targets, const int64_t* d_n, int fanout,
                 int policy, int equal_root_time, int64_t allowed_offset, int keep_root_time, uint64_t seed, uint32_t rng_stream,
                 int64_t* out_nbr, int64_t* out_dst, int64_t* out_ts, float* out_dt, int64_t* out_dt_i64, int64_t* out_eid,
                 int64_t* out_offsets, int64_t* total_out, int32_t* d_status, void* ws, size_t ws_bytes, void* stream,
                 int64_t* host_total = nullptr, int64_t seq = 0);
}  // namespace sgl
