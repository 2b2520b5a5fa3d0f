// A stand-in for the CUDA runtime, for tests of the host code's error paths
// without a GPU: device memory is host memory, kernels and streams do nothing,
// and the calls named by the fake_* controls fail.  Linked with the library's
// own objects instead of the runtime.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <vector>

namespace {
std::mutex mu;
std::map<void *, size_t> live;
std::vector<long long> sizes;
std::set<void *> events;
long long fail_bytes = 0, fail_skip = 0, launches = 0, instantiations = 0;
bool fail_events = false, capturing = false, memset_node = false;
int captured_nodes = 0;
cudaError_t last = cudaSuccess;
char device_symbol[64 << 20];

cudaError_t fail(cudaError_t e) {
  last = e;
  return e;
}
cudaError_t take(void **p, size_t n) {
  std::lock_guard<std::mutex> lk(mu);
  sizes.push_back((long long)n);
  *p = nullptr;
  if (fail_bytes && (long long)n == fail_bytes && fail_skip-- <= 0) return fail(cudaErrorMemoryAllocation);
  *p = std::calloc(n ? n : 1, 1);
  live[*p] = n;
  return cudaSuccess;
}
cudaError_t give(void *p) {
  std::lock_guard<std::mutex> lk(mu);
  if (!p) return cudaSuccess;
  if (!live.erase(p)) return fail(cudaErrorInvalidValue);
  std::free(p);
  return cudaSuccess;
}
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
};
thread_local Config config;
}  // namespace

extern "C" {
// ---- controls -----------------------------------------------------------------
// allocations of this size fail but for the first few (0: none fails)
void fake_fail_bytes(long long n, long long skip) { fail_bytes = n, fail_skip = skip; }
void fake_fail_events(int on) { fail_events = on != 0; }
void fake_memset_node(int on) { memset_node = on != 0; }  // captured bodies hold a memset
long long fake_launches() { return launches; }
long long fake_instantiations() { return instantiations; }
int fake_last_error() { return (int)last; }
long long fake_live() { return (long long)live.size(); }
void fake_forget_sizes() { sizes.clear(); }
int fake_sizes(long long *out, int cap) {  // of the allocations since
  for (int k = 0; k < cap && k < (int)sizes.size(); ++k) out[k] = sizes[k];
  return (int)sizes.size();
}

// ---- memory --------------------------------------------------------------------
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void **p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  if (!capturing) std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = *t = size_t(1) << 38;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) {
  *p = reinterpret_cast<cudaMemPool_t>(device_symbol);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  *p = device_symbol;
  return cudaSuccess;
}

// ---- device, errors --------------------------------------------------------------
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *least, int *greatest) {
  *least = 0, *greatest = -5;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "error of the stand-in runtime"; }

// ---- streams, events ----------------------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return take((void **)s, 8); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return take((void **)s, 8); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return give(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) {
  return events.count(e) ? cudaSuccess : fail(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  *e = nullptr;
  if (fail_events) return fail(cudaErrorMemoryAllocation);
  const cudaError_t r = take((void **)e, 8);
  events.insert(*e);
  return r;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  events.erase(e);
  return give(e);
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  return events.count(e) ? cudaSuccess : fail(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}

// ---- kernels --------------------------------------------------------------------------
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
  config = {grid, block, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st) {
  *grid = config.grid, *block = config.block, *smem = config.smem;
  *static_cast<cudaStream_t *>(st) = config.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3 g, dim3 b, void **, size_t, cudaStream_t) {
  if (!g.x || !g.y || !g.z || !b.x || !b.y || !b.z || b.x * b.y * b.z > 1024) return fail(cudaErrorInvalidConfiguration);
  if (capturing)
    ++captured_nodes;
  else
    ++launches;
  return cudaSuccess;
}

// ---- graphs -----------------------------------------------------------------------------
cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) { return take((void **)g, 8); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return give(g); }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) {
  *h = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t g, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                             cudaGraphNodeParams *par) {
  static cudaGraph_t body[1];
  body[0] = g;
  *n = reinterpret_cast<cudaGraphNode_t>(g);
  par->conditional.phGraph_out = body;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *,
                                          size_t, cudaStreamCaptureMode) {
  capturing = true;
  captured_nodes = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  capturing = false;
  *g = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *nodes, size_t *n) {
  if (nodes)
    for (size_t k = 0; k < *n; ++k) nodes[k] = reinterpret_cast<cudaGraphNode_t>(k + 1);
  else
    *n = (size_t)captured_nodes;
  return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t node, cudaGraphNodeType *t) {
  *t = memset_node && node == reinterpret_cast<cudaGraphNode_t>(1) ? cudaGraphNodeTypeMemset : cudaGraphNodeTypeKernel;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  ++instantiations;
  return take((void **)e, 8);
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return give(e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
}
