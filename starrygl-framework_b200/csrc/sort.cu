// Stable radix sort of (uint64 key, uint32 payload) pairs in memory: the two-kernel sort of tilesort.cuh for mini-batch sizes,
// the radix passes of lsd.cuh above.
#include "lsd.cuh"

namespace sgl {

namespace {

// ---------------------------------------------------------------------------------------------------------------
// Mini-batch sizes: the two-kernel sort of tilesort.cuh with plain keys in and plain (key, payload) out.
// ---------------------------------------------------------------------------------------------------------------
struct RawSource {
  const uint64_t* keys;
  int64_t n_cap;
  const int64_t* d_n;
  uint64_t mask;        // only the sorted bits take part
  __device__ __forceinline__ int64_t begin() const { return eff_count(n_cap, d_n); }
  using Raw = uint64_t;
  __device__ __forceinline__ Raw load(int64_t i) const { return keys[i]; }
  __device__ __forceinline__ uint64_t key(Raw x) const { return x & mask; }
};

struct RawSink {
  static constexpr bool kUnique = false, kAfter = false;
  __device__ __forceinline__ void begin() const {}
  const uint64_t* keys;
  const uint32_t* vals;  // nullptr: the payload is the input position
  uint64_t* out_keys;
  uint32_t* out_vals;
  uint64_t mask;
  __device__ __forceinline__ void item(int64_t at, uint64_t key, uint32_t pos) const {
    out_keys[at] = mask == ~0ull ? key : keys[pos];
    out_vals[at] = vals ? vals[pos] : pos;
  }
  __device__ __forceinline__ void between(int64_t, uint64_t, bool, uint64_t) const {}
  __device__ __forceinline__ void finish(int64_t, uint64_t, bool, int64_t, int64_t) const {}
};

// first pass over pairs without a payload of their own
struct IotaItems {
  static constexpr bool kChecked = false;
  const uint64_t* keys;
  int64_t n_cap;
  const int64_t* d_n;
  __device__ __forceinline__ int64_t begin() const { return eff_count(n_cap, d_n); }
  __device__ __forceinline__ uint64_t key(int64_t i) const { return keys[i]; }
  __device__ __forceinline__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};

}  // namespace

size_t radix_sort_ws_bytes(int64_t n) {
  return align_up(8) + (n <= tilesort::kMaxItems ? tilesort::ws_bytes(n) : lsd_ws_bytes<uint32_t>(n));     // (8: a status word)
}

int radix_sort_pairs(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, int64_t n,
                     const int64_t* d_n, int num_bits, bool iota_vals, int* result_in_alt, int32_t* d_status, void* ws,
                     size_t ws_bytes, cudaStream_t stream) {
  SGL_REQUIRE(n >= 0 && n < ((int64_t)1 << 32), SGL_ERR_ARG, "radix sort: n=%lld outside [0, 2^32)", (long long)n);
  SGL_REQUIRE(num_bits >= 0 && num_bits <= 64, SGL_ERR_ARG, "radix sort: num_bits=%d", num_bits);
  *result_in_alt = 0;
  if (n == 0 || (num_bits == 0 && !iota_vals)) return SGL_OK;
  SGL_REQUIRE(keys && vals && keys_alt && vals_alt, SGL_ERR_ARG, "radix sort: null buffer");
  LaunchScope scope(stream);
  WsCarver c(ws, ws_bytes);
  if (n <= tilesort::kMaxItems) {
    const tilesort::Scratch sc = tilesort::carve(c, n);
    SGL_REQUIRE(c.ok(), SGL_ERR_WORKSPACE, "radix sort: workspace %zu < %zu bytes", ws_bytes, radix_sort_ws_bytes(n));
    const uint64_t mask = num_bits >= 64 ? ~0ull : ((1ull << num_bits) - 1ull);
    *result_in_alt = 1;
    SGL_CHECK_RC(tilesort::launch(RawSource{keys, n, d_n, mask}, RawSink{keys, iota_vals ? nullptr : vals, keys_alt, vals_alt, mask}, n,
                                  num_bits, sc, d_status, stream));
    return scope.submit();
  }
  bool alt = false;
  unsigned int* gave_up;
  if (iota_vals)
    SGL_CHECK_RC((lsd_sort<uint32_t, IotaItems>(IotaItems{keys, n, d_n}, keys_alt, vals_alt, keys, vals, n, d_n, nullptr, 0, num_bits, ArrayOut<uint32_t>{}, &alt, &gave_up, c,
                                                d_status, stream)));
  else
    SGL_CHECK_RC((lsd_sort<uint32_t, ArrayItems<uint32_t>>(ArrayItems<uint32_t>{keys, vals, n, d_n}, keys_alt, vals_alt, keys, vals, n,
                                                           d_n, nullptr, 0, num_bits, ArrayOut<uint32_t>{}, &alt, &gave_up, c, d_status, stream)));
  *result_in_alt = alt ? 1 : 0;
  return scope.submit();
}

}  // namespace sgl

extern "C" size_t sgl_radix_sort_ws_bytes(int64_t n) { return sgl::radix_sort_ws_bytes(n); }

// number of kernels one sort of n keys of num_bits bits launches (for launch accounting; memsets are not kernels)
extern "C" int sgl_radix_sort_launches(int64_t n, int num_bits) {
  if (n <= 0) return 0;
  if (n <= sgl::tilesort::kMaxItems) return sgl::tilesort::launches(n);
  return 2 + sgl::lsd_passes(0, num_bits);
}

extern "C" int sgl_radix_sort_u64_u32(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, int64_t n,
                                      int num_bits, int* h_result_in_alt, void* ws, size_t ws_bytes, void* stream) {
  int dummy = 0;
  int* const in_alt = h_result_in_alt ? h_result_in_alt : &dummy;
  if (n <= sgl::tilesort::kMaxItems)     // (nothing in it waits)
    return sgl::radix_sort_pairs(keys, vals, keys_alt, vals_alt, n, nullptr, num_bits, false, in_alt, nullptr, ws, ws_bytes, (cudaStream_t)stream);
  const size_t head = sgl::align_up(8);
  SGL_REQUIRE(ws && ws_bytes >= sgl::radix_sort_ws_bytes(n), SGL_ERR_WORKSPACE, "radix sort: workspace %zu < %zu bytes", ws_bytes,
              sgl::radix_sort_ws_bytes(n));
  int64_t* status = (int64_t*)ws;
  SGL_CUDA_CHECK(cudaMemsetAsync(status, 0, 8, (cudaStream_t)stream));
  SGL_CHECK_RC(sgl::radix_sort_pairs(keys, vals, keys_alt, vals_alt, n, nullptr, num_bits, false, in_alt, (int32_t*)status, (char*)ws + head,
                                     ws_bytes - head, (cudaStream_t)stream));
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  SGL_CUDA_CHECK(cudaStreamIsCapturing((cudaStream_t)stream, &st));
  if (st != cudaStreamCaptureStatusNone) return SGL_OK;
  int64_t bits = 0;
  SGL_CHECK_RC(sgl_read_back(status, &bits, 8, stream));
  SGL_REQUIRE(bits == 0, SGL_ERR_CUDA, "radix sort: a look-back over the tiles ran into its time limit");
  return SGL_OK;
}
