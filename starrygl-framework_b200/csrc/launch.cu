#include "launch.cuh"

#include <memory>

namespace sgl {
namespace {

// per thread and kind (whole calls or the rest of one, beginnings that were submitted ahead): the least recently used one makes room
constexpr size_t kMaxGraphs = 32;

struct Cached {
  bool ahead;                         // the beginning of a call
  int device;
  cudaStream_t stream;
  std::vector<const void*> funcs;
  std::vector<std::vector<int>> deps;
  cudaGraph_t graph = nullptr;        // kept: the executable graph's nodes are named by its nodes
  cudaGraphExec_t exec = nullptr;     // nullptr: the sequence was seen once
  ~Cached() {                         // (launches that are still running finish first)
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
  }
  std::vector<cudaGraphNode_t> nodes;
  std::vector<std::vector<unsigned char>> set;     // grid, block, shared memory and arguments that a node has
  uint64_t last_use = 0;
  bool refused = false;               // no graph could be made of it (no memory, say): launched one by one
};

struct Thread {
  LaunchScope* open = nullptr;
  int plain = 0;
  LaunchList list;
  std::vector<Cached*> graphs;        // of both kinds
  uint64_t clock = 0;
  std::vector<void*> params;
  ~Thread() {
    for (Cached* c : graphs) delete c;
  }
};

thread_local Thread t_state;

bool same(const Cached& c, bool ahead, int device, cudaStream_t stream, const LaunchList& l) {
  if (c.ahead != ahead || c.device != device || c.stream != stream || c.funcs.size() != l.used) return false;
  for (size_t i = 0; i < l.used; ++i)
    if (c.funcs[i] != l.nodes[i].func || c.deps[i] != l.nodes[i].deps) return false;
  return true;
}

void** params_of(const LaunchNode& n) {
  Thread& t = t_state;
  t.params.resize(n.arg_count);
  for (uint32_t i = 0; i < n.arg_count; ++i) t.params[i] = t.list.bytes.data() + t.list.arg_at[n.arg_first + i];
  return t.params.data();
}

cudaKernelNodeParams node_params(const LaunchNode& n) {
  cudaKernelNodeParams p;
  memset(&p, 0, sizeof(p));
  p.func = const_cast<void*>(n.func);
  p.gridDim = n.grid;
  p.blockDim = n.block;
  p.sharedMemBytes = n.smem;
  p.kernelParams = params_of(n);
  return p;
}

// Notes what node i of the list is given; false: its node in the graph has just that.
bool changed(Cached& c, size_t i) {
  const LaunchList& l = t_state.list;
  const LaunchNode& n = l.nodes[i];
  const size_t from = n.arg_count ? l.arg_at[n.arg_first] : 0,
               to = n.arg_count ? (i + 1 < l.used && l.nodes[i + 1].arg_count ? l.arg_at[l.nodes[i + 1].arg_first] : l.bytes.size()) : 0;
  const unsigned shape[] = {n.grid.x, n.grid.y, n.grid.z, n.block.x, n.block.y, n.block.z, n.smem};
  std::vector<unsigned char>& set = c.set[i];
  if (set.size() == sizeof(shape) + (to - from) && memcmp(set.data(), shape, sizeof(shape)) == 0 &&
      memcmp(set.data() + sizeof(shape), l.bytes.data() + from, to - from) == 0)
    return false;
  set.resize(sizeof(shape) + (to - from));
  memcpy(set.data(), shape, sizeof(shape));
  memcpy(set.data() + sizeof(shape), l.bytes.data() + from, to - from);
  return true;
}

int one_by_one(cudaStream_t stream) {
  const LaunchList& l = t_state.list;
  for (size_t i = 0; i < l.used; ++i) {
    const LaunchNode& n = l.nodes[i];
    SGL_CUDA_CHECK(cudaLaunchKernel(n.func, n.grid, n.block, params_of(n), n.smem, stream));
  }
  return SGL_OK;
}

int build(Cached& c) {
  const LaunchList& l = t_state.list;
  std::vector<cudaGraphNode_t> nodes(l.used), deps;
  // (before there is a graph: an entry with one has all of its notes, also after a failed allocation)
  c.set.assign(l.used, {});
  for (size_t i = 0; i < l.used; ++i) changed(c, i);
  cudaGraph_t graph = nullptr;
  SGL_CUDA_CHECK(cudaGraphCreate(&graph, 0));
  std::unique_ptr<CUgraph_st, decltype(&cudaGraphDestroy)> made(graph, &cudaGraphDestroy);
  cudaError_t e = cudaSuccess;
  for (size_t i = 0; i < l.used && e == cudaSuccess; ++i) {
    deps.clear();
    for (int d : l.nodes[i].deps) deps.push_back(nodes[d]);
    const cudaKernelNodeParams p = node_params(l.nodes[i]);
    e = cudaGraphAddKernelNode(&nodes[i], graph, deps.data(), deps.size(), &p);
  }
  cudaGraphExec_t exec = nullptr;
  if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
  if (e != cudaSuccess) {
    cudaGetLastError();
    c.refused = true;
    return SGL_OK;
  }
  c.graph = made.release();
  c.exec = exec;
  c.nodes = std::move(nodes);
  return SGL_OK;
}

__global__ void zero_words_kernel(uint32_t* p, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = 0;
}

thread_local int64_t t_look_back_ns = 2000000000;

}  // namespace

unsigned long long look_back_ns() { return (unsigned long long)t_look_back_ns; }

int zero_async(void* p, size_t bytes, cudaStream_t stream) {
  if (LaunchScope::current() == nullptr) {
    SGL_CUDA_CHECK(cudaMemsetAsync(p, 0, bytes, stream));
    return SGL_OK;
  }
  return launch(zero_words_kernel, stream_grid((int64_t)(bytes / 4), 256, 8), 256, 0, stream, (uint32_t*)p, bytes / 4);
}

PlainLaunches::PlainLaunches() { ++t_state.plain; }
PlainLaunches::~PlainLaunches() { --t_state.plain; }

LaunchScope* LaunchScope::current() { return t_state.open; }

LaunchScope::LaunchScope(cudaStream_t main) : owner_(false), main_(main) {
  Thread& t = t_state;
  if (t.open != nullptr || t.plain > 0) return;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(main, &st) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (st != cudaStreamCaptureStatusNone) return;
  owner_ = true;
  t.list.clear();
  t.open = this;
}

LaunchScope::~LaunchScope() {
  if (owner_ && t_state.open == this) t_state.open = nullptr;
}

LaunchScope::Tail& LaunchScope::tail(cudaStream_t s) {
  for (Tail& t : tails_)
    if (t.stream == s) return t;
  tails_.push_back(Tail{s, {}});
  return tails_.back();
}

int LaunchScope::add(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t on, const void* const* args,
                     const size_t* sizes, int n) {
  return no_throw([&] {
    LaunchList& l = t_state.list;
    if (l.used == l.nodes.size()) l.nodes.emplace_back();
    LaunchNode& node = l.nodes[l.used];
    node.func = func;
    node.grid = grid;
    node.block = block;
    node.smem = (unsigned)smem;
    node.on = on;
    node.arg_first = (uint32_t)l.arg_at.size();
    node.arg_count = (uint32_t)n;
    for (int i = 0; i < n; ++i) {
      const size_t at = (l.bytes.size() + 15) & ~(size_t)15;
      l.bytes.resize(at + sizes[i]);
      memcpy(l.bytes.data() + at, args[i], sizes[i]);
      l.arg_at.push_back((uint32_t)at);
    }
    Tail& t = tail(on);
    node.deps = t.nodes;
    t.nodes.assign(1, (int)l.used);
    ++l.used;
    return SGL_OK;
  });
}

int LaunchScope::wait(cudaStream_t s, const std::vector<int>& nodes) {
  return no_throw([&] {
    Tail& t = tail(s);
    for (int d : nodes) {
      bool known = false;
      for (int k : t.nodes) known = known || k == d;
      if (!known) t.nodes.push_back(d);
    }
    return SGL_OK;
  });
}

int LaunchScope::submit() {
  if (!owner_) return SGL_OK;
  owner_ = false;
  t_state.open = nullptr;
  return no_throw([&] { return submit_list(false); });
}

int LaunchScope::flush() {
  if (!owner_) return SGL_OK;
  return no_throw([&] {
    const int rc = submit_list(true);
    t_state.list.clear();
    tails_.clear();                      // (what follows comes after all of it, in stream order)
    return rc;
  });
}

int LaunchScope::submit_list(bool ahead) {
  Thread& t = t_state;
  LaunchList& l = t.list;
  if (l.used == 0) return SGL_OK;
  if (l.used == 1) return one_by_one(main_);
  int device = 0;
  SGL_CUDA_CHECK(cudaGetDevice(&device));
  ++t.clock;
  Cached* c = nullptr;
  for (Cached* g : t.graphs)
    if (same(*g, ahead, device, main_, l)) {
      c = g;
      break;
    }
  if (c == nullptr) {
    size_t kind = 0, oldest = t.graphs.size();
    for (size_t i = 0; i < t.graphs.size(); ++i) {
      if (t.graphs[i]->ahead != ahead) continue;
      ++kind;
      if (oldest == t.graphs.size() || t.graphs[i]->last_use < t.graphs[oldest]->last_use) oldest = i;
    }
    if (kind >= kMaxGraphs) {
      Cached* old = t.graphs[oldest];
      delete old;
      t.graphs.erase(t.graphs.begin() + oldest);
    }
    c = new Cached;
    c->ahead = ahead;
    c->device = device;
    c->stream = main_;
    for (size_t i = 0; i < l.used; ++i) {
      c->funcs.push_back(l.nodes[i].func);
      c->deps.push_back(l.nodes[i].deps);
    }
    c->last_use = t.clock;
    t.graphs.push_back(c);
    return one_by_one(main_);
  }
  c->last_use = t.clock;
  if (c->exec == nullptr && !c->refused) SGL_CHECK_RC(build(*c));
  else if (!c->refused) {
    for (size_t i = 0; i < l.used; ++i) {
      if (!changed(*c, i)) continue;
      const cudaKernelNodeParams p = node_params(l.nodes[i]);
      const cudaError_t e = cudaGraphExecKernelNodeSetParams(c->exec, c->nodes[i], &p);
      if (e != cudaSuccess) c->set[i].clear();         // (who knows what it has)
      SGL_CUDA_CHECK(e);
    }
  }
  if (c->refused) return one_by_one(main_);
  SGL_CUDA_CHECK(cudaGraphLaunch(c->exec, main_));
  return SGL_OK;
}

}  // namespace sgl

extern "C" int sgl_launch_graphs(void) {
  int n = 0;
  for (const sgl::Cached* c : sgl::t_state.graphs) n += c->exec != nullptr && !c->ahead ? 1 : 0;
  return n;
}

extern "C" int64_t sgl_look_back_limit(int64_t ns) {
  const int64_t before = sgl::t_look_back_ns;
  if (ns >= 0) sgl::t_look_back_ns = ns;
  return before;
}
