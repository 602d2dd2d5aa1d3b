// Kernel launches of an entry point that issues several: collected, then submitted as ONE CUDA graph launch.
//
// A kernel launch costs the host about 4 us here; an executable graph whose kernel nodes get new parameters and grid sizes
// costs 1.1 us + 0.3 us per node (14 kernels: 58 us of launches, 5 us as a graph), and its kernels follow each other more
// closely.  The graph depends only on which kernels follow which, not on sizes or pointers, so a handful of them per
// thread and stream serves every call:
//
//   LaunchScope scope(stream);                                   // collects from here on, on this thread
//   SGL_CHECK_RC(launch(kernel, grid, block, smem, stream, args...));
//   return scope.submit();
//
// Scopes nest: an entry point called inside another's scope adds to it.  The first call of a sequence on a stream launches
// its kernels one by one (a sequence that never comes back is not worth a graph), so do calls on a capturing stream.
#pragma once
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <new>
#include <vector>

#include "common.cuh"

namespace sgl {

// Nothing may throw across the library's C functions: what allocates host memory on the way runs in here.
template <class F>
int no_throw(F&& f) {
  try {
    return f();
  } catch (const std::bad_alloc&) {
    set_error("out of host memory");
    return SGL_ERR_CUDA;
  }
}

struct LaunchNode {
  const void* func;
  dim3 grid, block;
  unsigned smem;
  cudaStream_t on;
  uint32_t arg_first, arg_count;      // into LaunchList::arg_at
  std::vector<int> deps;
};

struct LaunchList {
  std::vector<LaunchNode> nodes;
  size_t used = 0;                    // nodes of this list in use (the vectors inside are kept)
  std::vector<unsigned char> bytes;   // argument values, 16-byte aligned
  std::vector<uint32_t> arg_at;
  void clear() {
    used = 0;
    bytes.clear();
    arg_at.clear();
  }
};

// While one exists, the calling thread launches its kernels one by one: for calls that must not make the driver allocate, as an
// executable graph does.
class PlainLaunches {
 public:
  PlainLaunches();
  ~PlainLaunches();
};

class LaunchScope {
 public:
  explicit LaunchScope(cudaStream_t main);
  ~LaunchScope();
  // Adds a kernel to the scope that is open on this thread; false when there is none (or it launches one by one).
  static LaunchScope* current();
  int add(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t on, const void* const* args, const size_t* sizes, int n);
  // what is added to stream s after wait(s, m) comes after everything that was on the marked stream at mark(marked, &m)
  int mark(cudaStream_t s, std::vector<int>* nodes) {
    return no_throw([&] {
      *nodes = tail(s).nodes;
      return SGL_OK;
    });
  }
  int wait(cudaStream_t s, const std::vector<int>& nodes);
  // ... after everything that is on the other stream by now
  int follow(cudaStream_t s, cudaStream_t other) {
    std::vector<int> nodes;
    const int rc = mark(other, &nodes);
    return rc != SGL_OK ? rc : wait(s, nodes);
  }
  int submit();
  // Submits what was collected so far and goes on collecting (nothing in an inner scope): the device starts on it while the host
  // still adds and sets up the rest, which takes 0.6 us a kernel and 5 us a launch.  For a beginning of 10 - 15 us that everything else
  // waits for.  Arguments are checked before it, those of what follows too: a call that is refused has started nothing.
  int flush();

 private:
  int submit_list(bool ahead);
  bool owner_;
  cudaStream_t main_;
  struct Tail {
    cudaStream_t stream;
    std::vector<int> nodes;           // what the next kernel on the stream waits for
  };
  std::vector<Tail> tails_;
  Tail& tail(cudaStream_t s);
};

template <class... KArgs, class... Args>
int launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const Args&... args) {
  LaunchScope* s = LaunchScope::current();
  if (s == nullptr) {
    kernel<<<grid, block, smem, stream>>>(static_cast<KArgs>(args)...);
    SGL_LAUNCH_CHECK();
    return SGL_OK;
  }
  auto add = [&](const KArgs&... a) -> int {
    const void* p[] = {(const void*)&a...};
    const size_t n[] = {sizeof(KArgs)...};
    return s->add((const void*)kernel, grid, block, smem, stream, p, n, (int)sizeof...(KArgs));
  };
  return add(static_cast<KArgs>(args)...);
}

// A kernel that a call launches by itself may be set up while the one before it on the stream still runs (programmatic stream
// serialization): a gather of 22 us and a scatter of 6 were 1.8 us apart, and
// a pass of both took 32.8 us, 27.1 so (31.7 when a kernel let the next one in at its start: it holds what the running one needs).  Such a kernel calls after_predecessor()
// before it touches memory, reads what others may have written through pointers that current() has handed out behind that, and not
// through the read-only path, which may be served from before.  In a scope the launch is an ordinary one.
template <class... KArgs, class... Args>
int launch_early(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const Args&... args) {
  if (LaunchScope::current() != nullptr) return launch(kernel, grid, block, smem, stream, args...);
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  SGL_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...));
  return SGL_OK;
}

#ifdef __CUDACC__
__device__ __forceinline__ void after_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// p, in a form that the compiler knows only from here on
template <class T>
__device__ __forceinline__ T* current(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
#endif

// Zero bytes (a multiple of four, four-byte aligned) in stream order, in a launch scope or not.
int zero_async(void* p, size_t bytes, cudaStream_t stream);

// How long the look-backs of lsd.cuh wait for the tiles before them, see sgl_look_back_limit.
unsigned long long look_back_ns();

// kernels that need more than 48 KB of shared memory say so once per device
inline cudaError_t allow_smem(const void* kernel, std::atomic<uint64_t>& done, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

#define SGL_CHECK_RC(expr)     \
  do {                         \
    const int rc_ = (expr);    \
    if (rc_ != SGL_OK) return rc_; \
  } while (0)

}  // namespace sgl
