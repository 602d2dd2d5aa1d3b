// Helpers of the entry points that enqueue a whole batch or query.
#pragma once
#include "launch.cuh"

namespace sgl {

// N events per device of the calling thread, made on first use and given back when the thread ends.
template <int N>
struct ThreadEvents {
  cudaEvent_t ev[64][N] = {};
  ~ThreadEvents() {
    for (auto& d : ev)
      for (cudaEvent_t e : d)
        if (e) cudaEventDestroy(e);
  }
  int of_device(cudaEvent_t** out) {
    int dev = 0;
    SGL_CUDA_CHECK(cudaGetDevice(&dev));
    for (cudaEvent_t& e : ev[dev & 63])
      if (e == nullptr) SGL_CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    *out = ev[dev & 63];
    return SGL_OK;
  }
};

// Order between the two streams of an entry point: nodes of the launch scope, or (captured calls) events of this thread, recorded
// and waited for at once and so reusable.
struct Order {
  static constexpr int kMarks = 4;
  LaunchScope* scope;
  std::vector<int> nodes[kMarks];
  cudaEvent_t* ev;

  int init(LaunchScope* s) {
    scope = s;
    if (scope) return SGL_OK;
    static thread_local ThreadEvents<kMarks> pool;
    return pool.of_device(&ev);
  }
  int mark(int i, cudaStream_t s) {
    if (scope) return scope->mark(s, &nodes[i]);
    SGL_CUDA_CHECK(cudaEventRecord(ev[i], s));
    return SGL_OK;
  }
  int wait(int i, cudaStream_t s) {
    if (scope) return scope->wait(s, nodes[i]);
    SGL_CUDA_CHECK(cudaStreamWaitEvent(s, ev[i], 0));
    return SGL_OK;
  }
};

// what `stream` is given from here on comes after everything `producer` has been given so far
inline int order_after(cudaStream_t stream, cudaStream_t producer) {
  if (producer == stream) return SGL_OK;
  static thread_local ThreadEvents<1> pool;
  cudaEvent_t* e = nullptr;
  const int rc = pool.of_device(&e);
  if (rc != SGL_OK) return rc;
  SGL_CUDA_CHECK(cudaEventRecord(*e, producer));
  SGL_CUDA_CHECK(cudaStreamWaitEvent(stream, *e, 0));
  return SGL_OK;
}

// words of device memory -> pinned host memory, then the flag behind them
static __global__ void export_words_kernel(const int64_t* __restrict__ src, int64_t* dst, int words, int64_t flag) {
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) *(volatile int64_t*)(dst + words) = flag;
}

inline int export_words(const int64_t* src, int64_t* dst, int words, cudaStream_t stream) {
  *(volatile int64_t*)(dst + words) = 0;
  return launch(export_words_kernel, 1, 32, 0, stream, src, dst, words, (int64_t)1);
}

}  // namespace sgl
