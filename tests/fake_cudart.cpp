// A CUDA runtime for host tests: linked with the library's objects in place of
// the real one, it lets the library's host code run without a GPU.  Device
// memory is host memory, copies and fills happen at the call (in a graph, at its
// launch), and kernels do nothing, except:
//   k_scan       stores the total given by fake_scan_total
//   k_finalize   stores the step result queued by fake_step (else an empty one)
//   k_composite  checks that the arrays it got are live, and counts those that
//                are not (fake_bad)
// fake_fail(n) makes the n-th allocation from now on fail, once.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace {
std::map<const void*, size_t> g_live, g_room;
std::multimap<size_t, void*> g_free;
std::map<const void*, std::string> g_names;
using Graph = std::vector<std::function<void()>>;
Graph* g_capture = nullptr;
int g_fail = 0;
cudaError_t g_last = cudaSuccess;
struct Step { double loss; unsigned long long pairs, items; uint32_t err, chunks; };
std::deque<Step> g_steps;
uint64_t g_scan_total = 0;
uint64_t g_bad = 0, g_composites = 0, g_replays = 0, g_pool_cap = 0;

// the kernels' parameters that are looked at, as the library declares them
struct Lists { const uint32_t *ids, *ranges, *keys; uint32_t super_per_view, super_x; };
struct Takers { uint32_t *ids, *prev, *head, *drawn, *heavy, *n_heavy; uint8_t* is_heavy; uint32_t pool_cap; };

size_t size_of(const void* p) {
  auto it = g_live.find(p);
  return it == g_live.end() ? 0 : it->second;
}
void enqueue(std::function<void()> f) {
  if (g_capture) g_capture->push_back(std::move(f));
  else f();
}
cudaError_t alloc(void** p, size_t n) {
  *p = nullptr;
  if (g_fail > 0 && --g_fail == 0) return g_last = cudaErrorMemoryAllocation;
  // a freed array's memory goes to the next one that fits, as a device's does
  auto it = g_free.lower_bound(n);
  if (it != g_free.end()) {
    *p = it->second;
    g_free.erase(it);
  } else {
    g_room[*p = std::malloc(n + (1u << 20))] = n + (1u << 20);
  }
  std::memset(*p, 0, n);
  g_live[*p] = n;
  return cudaSuccess;
}
cudaError_t release(void* p) {
  if (p && g_live.erase(p)) g_free.emplace(g_room[p], p);
  return cudaSuccess;
}
cudaError_t launch(const void* func, void** args) {
  const std::string& n = g_names[func];
  if (n.find("11k_composite") != std::string::npos) {
    const Lists l = *static_cast<Lists*>(args[1]);
    const Takers t = *static_cast<Takers*>(args[11]);
    enqueue([l, t] {
      ++g_composites;
      // the lists are read in groups of four words
      if (size_of(l.ids) == 0 || size_of(l.ids) % 16) ++g_bad;
      if (l.keys && (size_of(l.keys) == 0 || size_of(l.keys) % 16)) ++g_bad;
      g_pool_cap = t.pool_cap;
      if (t.head && (t.pool_cap == 0 || size_of(t.ids) < (size_t)t.pool_cap * 64 * 128 ||
                     size_of(t.prev) < (size_t)t.pool_cap * 64 * 4))
        ++g_bad;
    });
  } else if (n.find("6k_scan") != std::string::npos) {
    uint64_t* total = *static_cast<uint64_t**>(args[4]);
    enqueue([total] { if (total) *total = g_scan_total; });
  } else if (n.find("10k_finalize") != std::string::npos) {
    Step* out = *static_cast<Step**>(args[9]);
    enqueue([out] {
      *out = Step{};
      if (g_steps.empty()) return;
      *out = g_steps.front();
      g_steps.pop_front();
    });
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_fail(int n) { g_fail = n; }
void fake_scan_total(uint64_t n) { g_scan_total = n; }
void fake_step(uint64_t pairs, uint64_t items, uint32_t err, uint32_t chunks) {
  g_steps.push_back(Step{0.0, pairs, items, err, chunks});
}
uint64_t fake_bad() { return g_bad; }
uint64_t fake_composites() { return g_composites; }
uint64_t fake_replays() { return g_replays; }
uint64_t fake_pool_cap() { return g_pool_cap; }
uint64_t fake_live() { return g_live.size(); }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) {
  g_names[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
struct Config { dim3 grid, block; size_t smem; void* stream; };
static Config g_config;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void* s) { g_config = {g, b, m, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = g_config.grid; *b = g_config.block; *m = g_config.smem; *static_cast<void**>(s) = g_config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) { return launch(f, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { return launch(f, args); }

cudaError_t cudaMalloc(void** p, size_t n) { return alloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return alloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return alloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return alloc(p, n); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return release(p); }
cudaError_t cudaFreeHost(void* p) { return release(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  enqueue([=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  enqueue([=] { if (n) std::memset(d, v, n); });
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = 1ull << 34; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char page[1 << 20]; *p = page; return cudaSuccess; }

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
static cudaError_t handle(void** h) { *h = std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle((void**)s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free((void*)s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle((void**)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle((void**)e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free((void*)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { g_capture = new Graph; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)g_capture;
  g_capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t) new Graph(*(Graph*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete (Graph*)e; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  ++g_replays;
  for (auto& f : *(Graph*)e) f();
  return cudaSuccess;
}
}  // extern "C"
