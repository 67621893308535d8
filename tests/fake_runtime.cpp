// A stand-in for the CUDA runtime with which the engine's host code runs on the CPU
// (tests/test_host_runtime.py links the engine's objects against it): device memory is
// host memory, copies copy, kernels do nothing, and every launch, stream, pinned
// allocation and graph is recorded.  Two devices of 148 SMs; a stream belongs to the
// device that was current when it was made, and as the runtime documents, a kernel
// launch into a stream of another device than the current one fails.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

struct Launch {
  std::string kernel;
  unsigned grid, block;
  bool programmatic;
  cudaStream_t stream;
};
struct CUstream_st { int device; bool capturing; };
struct CUevent_st { int device; bool captured; };
struct CUgraph_st { std::vector<Launch> nodes; };
struct CUgraphExec_st { std::vector<Launch> nodes; };

namespace {
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
thread_local struct { dim3 grid, block; size_t shared; cudaStream_t stream; } pushed;
std::map<const void*, std::string> names;
std::vector<Launch> launches, captured;   // run so far; nodes of the graph being captured
std::set<cudaStream_t> streams;
bool capture = false;
int fail_instantiations = 0;
long host_allocs, streams_made, instantiated, updated, nodes, device_bytes;

cudaError_t fail(cudaError_t e) { last = e; return e; }

cudaError_t launch(const void* f, dim3 grid, dim3 block, cudaStream_t s, bool programmatic) {
  if (s && s->device != device) return fail(cudaErrorInvalidResourceHandle);
  Launch l{names[f], grid.x, block.x, programmatic, s};
  (s && s->capturing ? captured : launches).push_back(l);
  return cudaSuccess;
}

// streams by their order of first use, so that two captures of one topology compare equal
std::vector<int> topology(const std::vector<Launch>& v) {
  std::map<cudaStream_t, int> order;
  std::vector<int> t;
  for (const Launch& l : v) t.push_back(order.emplace(l.stream, (int)order.size()).first->second);
  return t;
}
}  // namespace

extern "C" {
// ---- the record, read by the tests
void fake_fail_instantiations(int n) { fail_instantiations = n; }
void fake_reset() {
  launches.clear();
  host_allocs = streams_made = instantiated = updated = nodes = device_bytes = 0;
}
long fake_count(const char* what) {
  const std::string w = what;
  return w == "host_allocs" ? host_allocs : w == "streams_made" ? streams_made : w == "instantiated" ? instantiated
         : w == "updated" ? updated : w == "nodes" ? nodes : w == "device_bytes" ? device_bytes : w == "launches" ? (long)launches.size() : -1;
}
const char* fake_launch(int i, int* grid, int* block, int* programmatic, int* stream) {
  const Launch& l = launches[i];
  *grid = (int)l.grid;
  *block = (int)l.block;
  *programmatic = l.programmatic;
  *stream = topology(launches)[i];
  return l.kernel.c_str();
}

// ---- what the compiler's registration code calls
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, struct CUstream_st* s) {
  pushed = {grid, block, shared, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* s) {
  *grid = pushed.grid;
  *block = pushed.block;
  *shared = pushed.shared;
  *(cudaStream_t*)s = pushed.stream;
  return cudaSuccess;
}

// ---- devices and errors
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d > 1) return fail(cudaErrorInvalidDevice);
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidResourceHandle ? "invalid resource handle" : "error"; }

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); device_bytes += (long)n; return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(1, n); host_allocs++; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }

// ---- streams and events
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = new CUstream_st{device, false};
  streams.insert(*s);
  streams_made++;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { streams.erase(s); delete s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new CUevent_st{device, false}; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  if (s && s->device != e->device) return fail(cudaErrorInvalidResourceHandle);
  e->captured = s && s->capturing;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  if (e->captured) s->capturing = true;
  return cudaSuccess;
}

// ---- launches and graphs
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t, cudaStream_t s) {
  return launch(f, grid, block, s, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  bool programmatic = false;
  for (unsigned k = 0; k < c->numAttrs; k++)
    if (c->attrs[k].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      programmatic = c->attrs[k].val.programmaticStreamSerializationAllowed != 0;
  return launch(f, c->gridDim, c->blockDim, c->stream, programmatic);
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  if (capture) return fail(cudaErrorIllegalState);
  capture = s->capturing = true;
  captured.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capture = false;
  for (cudaStream_t s : streams) s->capturing = false;
  *g = new CUgraph_st{captured};
  nodes = (long)captured.size();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete g; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  if (fail_instantiations > 0) {
    fail_instantiations--;
    return fail(cudaErrorMemoryAllocation);
  }
  *x = new CUgraphExec_st{g->nodes};
  instantiated++;
  return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t x, cudaGraph_t g, cudaGraphExecUpdateResultInfo*) {
  if (topology(x->nodes) != topology(g->nodes)) return fail(cudaErrorGraphExecUpdateFailure);
  x->nodes = g->nodes;
  updated++;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete x; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  launches.insert(launches.end(), x->nodes.begin(), x->nodes.end());
  return cudaSuccess;
}
}
