// The CUDA runtime calls libfk's host code makes, on plain memory: device and
// pinned buffers are host allocations that are never handed out again, copies
// run at once, kernels do nothing -- except that the ordering kernels "find"
// the number of outputs a test asks for.  A stream capture records its copies
// and the ordering kernels' arguments; a graph launch runs them again.  Every
// address used is looked up, so work on a freed buffer is counted instead of
// corrupting anything.
#include "fake_cuda.h"

#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../../first-knowns_b200/csrc/fk_types.h"

namespace {

struct Alloc { size_t bytes; bool live; };
std::map<uintptr_t, Alloc> g_alloc;
std::map<const void*, std::string> g_name;   // kernel stubs
Fake g;
bool g_capturing = false;
int64_t g_fail_at = -1;                      // allocations left until one fails
cudaError_t g_last = cudaSuccess;

cudaError_t fail(cudaError_t e) { return g_last = e; }

cudaError_t allocate(void** p, size_t n) {
  if (g_fail_at == 0) {
    g_fail_at = -1;
    return fail(cudaErrorMemoryAllocation);
  }
  if (g_fail_at > 0) --g_fail_at;
  ++g.allocations;
  *p = std::calloc(n ? n : 1, 1);
  g_alloc[(uintptr_t)*p] = {n ? n : 1, true};
  return cudaSuccess;
}

void release(void* p) {
  if (p) g_alloc[(uintptr_t)p].live = false;
}

// An address inside a buffer that has been freed (host memory of the caller's
// own is not a buffer), or null.
bool dead(const void* p, size_t n) {
  if (!p) return true;
  auto it = g_alloc.upper_bound((uintptr_t)p);
  if (it == g_alloc.begin()) return false;
  --it;
  if ((uintptr_t)p >= it->first + it->second.bytes) return false;
  return !it->second.live || (uintptr_t)p + n > it->first + it->second.bytes;
}

struct Node {
  std::string kernel;          // empty: a copy, a fill or an event
  uint64_t* event = nullptr;
  void* dst = nullptr;
  const void* src = nullptr;
  size_t bytes = 0;
  std::vector<uint64_t> args;
};

// Arguments of the kernels a test looks at: p pointer, w 64 bits, u 32 bits.
const std::pair<const char*, const char*> kKernels[] = {
    {"k_order_prep", "pupppppp"},   {"k_bucket_count", "ppwppppp"},
    {"k_scan", "ppp"},              {"k_bucket_scatter", "ppwppppppp"},
    {"k_sort_seg", "pppp"},
};

void run(const Node& n) {
  if (n.event) {
    *n.event = g.kernels;
    return;
  }
  if (n.kernel.empty()) {
    if (dead(n.dst, n.bytes) || (n.src && dead(n.src, n.bytes))) {
      ++g.dead;
      return;
    }
    if (n.src) std::memcpy(n.dst, n.src, n.bytes);
    else std::memset(n.dst, 0, n.bytes);
    return;
  }
  ++g.kernels;
  for (const auto& k : kKernels) {
    if (n.kernel != k.first) continue;
    for (size_t i = 0; k.second[i]; ++i)
      if (k.second[i] == 'p' && dead((const void*)n.args[i], 1)) {
        ++g.dead;
        return;
      }
  }
  if (n.kernel == "k_bucket_count" && g.overflows) {
    fk::DevCounters* c = (fk::DevCounters*)n.args[1];
    c->overflow = 1;
    c->ncand = n.args[2] + 1;
    --g.overflows;
  } else if (n.kernel == "k_order_prep") {   // every output is the last item's
    const uint32_t ni = (uint32_t)n.args[1];
    uint64_t* off = (uint64_t*)n.args[2];
    for (uint32_t i = 0; i < ni; ++i) off[i] = 0;
    off[ni] = ni ? g.outputs : 0;
  } else if (n.kernel == "k_sort_seg") {
    uint64_t* sorted = (uint64_t*)n.args[0];
    if (dead(sorted, 8 * g.outputs)) ++g.dead;
    else
      for (uint64_t k = 0; k < g.outputs; ++k) sorted[k] = k << 8 | 7;
  }
}

struct Graph { std::vector<Node> nodes; };
Graph* g_graph = nullptr;

cudaError_t issue(Node n) {
  if (g_capturing) g_graph->nodes.push_back(std::move(n));
  else run(n);
  return cudaSuccess;
}

struct Event { uint64_t at; };
struct Config { dim3 grid, block; size_t smem; cudaStream_t stream; } g_config;

}  // namespace

Fake& fake() { return g; }
void fake_fail_allocation(int64_t skip) { g_fail_at = skip; }
void fake_kernel() {
  Node n;
  n.kernel = "k_sieve";
  issue(n);
}

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name,
                            int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_name[stub] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem,
                                     cudaStream_t s) {
  g_config = {grid, block, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem,
                                       void* s) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *(cudaStream_t*)s = g_config.stream;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { release(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { release(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  Node c;
  c.dst = d; c.src = s; c.bytes = n;
  run(c);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k,
                            cudaStream_t) {
  Node c;
  c.dst = d; c.src = s; c.bytes = n;
  if (k == cudaMemcpyDeviceToHost && !g_capturing) g.d2h += n;
  return issue(c);
}
cudaError_t cudaMemset(void* d, int, size_t n) {
  Node c;
  c.dst = d; c.bytes = n;
  run(c);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int, size_t n, cudaStream_t) {
  Node c;
  c.dst = d; c.bytes = n;
  return issue(c);
}
cudaError_t cudaLaunchKernel(const void* stub, dim3, dim3, void** args, size_t,
                             cudaStream_t) {
  Node n;
  n.kernel = "other";
  for (const auto& k : kKernels) {
    if (g_name[stub].find(k.first) == std::string::npos) continue;
    n.kernel = k.first;
    for (size_t i = 0; k.second[i]; ++i)
      n.args.push_back(k.second[i] == 'u' ? *(uint32_t*)args[i]
                                          : *(uint64_t*)args[i]);
    break;
  }
  return issue(n);
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  g_capturing = true;
  g_graph = new Graph;
  ++g.captures;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* out) {
  g_capturing = false;
  *out = (cudaGraph_t)g_graph;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t gr,
                                 unsigned long long) {
  *e = (cudaGraphExec_t) new Graph(*(Graph*)gr);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (const Node& n : ((Graph*)e)->nodes) run(n);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t gr) { delete (Graph*)gr; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete (Graph*)e;
  return cudaSuccess;
}

// an event's time: the kernels launched before it
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t) new Event{0};
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  Node n;
  n.event = &((Event*)e)->at;
  return issue(n);
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned) {
  return cudaEventRecord(e, s);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)((Event*)b)->at - (float)((Event*)a)->at;
  return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
}  // extern "C"
