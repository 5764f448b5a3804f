// A CUDA runtime without a GPU, for tests of the library's host code: memory is
// host memory and kernels do nothing.  Copies and fills are queued and happen
// when something waits for them, as late as an asynchronous call may take place;
// a cooperative launch takes the queue first (stream order) and is then handed
// to g_fake_cooperative.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <vector>

struct Queued {
  void* dst;
  const void* src;  // nullptr: fill
  int value;
  size_t n;
};
static std::vector<Queued> g_queue;
static std::map<char*, size_t> g_allocs;
static size_t g_log_bytes = 0;
static std::vector<char> g_log;

extern "C" {
void (*g_fake_cooperative)(const void* func, dim3 grid, dim3 block, void** args, size_t smem) = nullptr;
void (*g_fake_forget)(const void* p, size_t n) = nullptr;  // memory allocated, freed or filled
// Contents, at the time they were read, of every copy of `bytes` bytes.
void fake_log_copies(size_t bytes) {
  g_log_bytes = bytes;
  g_log.clear();
}
size_t fake_logged(char* out, size_t cap) {
  memcpy(out, g_log.data(), g_log.size() < cap ? g_log.size() : cap);
  return g_log.size();
}
}

static cudaError_t drain() {
  for (const Queued& q : g_queue) {
    if (!q.src) {
      memset(q.dst, q.value, q.n);
      if (g_fake_forget) g_fake_forget(q.dst, q.n);
      continue;
    }
    memmove(q.dst, q.src, q.n);
    if (q.n == g_log_bytes) g_log.insert(g_log.end(), (const char*)q.dst, (const char*)q.dst + q.n);
  }
  g_queue.clear();
  return cudaSuccess;
}
static cudaError_t allocate(void** p, size_t n) {
  *p = calloc(n ? n : 1, 1);
  g_allocs[(char*)*p] = n;
  if (g_fake_forget) g_fake_forget(*p, n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
static cudaError_t release(void* p) {
  drain();
  auto it = g_allocs.find((char*)p);
  if (it == g_allocs.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  if (g_fake_forget) g_fake_forget(p, it->second);
  g_allocs.erase(it);
  free(p);
  return cudaSuccess;
}
template <typename T>
static cudaError_t handle(T* h) {
  static size_t next = 1;
  *h = (T)(next++);
  return cudaSuccess;
}

extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return allocate(p, n); }
cudaError_t cudaMallocManaged(void** p, size_t n, unsigned) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaFreeHost(void* p) { return release(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  g_queue.push_back({d, s, 0, n});
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  cudaMemcpyAsync(d, s, n, k, nullptr);
  return drain();
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  g_queue.push_back({d, nullptr, v, n});
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return drain(); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return drain(); }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** a, size_t s, cudaStream_t) {
  drain();
  if (g_fake_cooperative) g_fake_cooperative(f, g, b, a, s);
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148
     : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448
     : a == cudaDevAttrL2CacheSize ? 126 << 20 : 0;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeDevice;
  a->devicePointer = (void*)p;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = (void*)s;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake CUDA runtime"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamGetDevice(cudaStream_t, int* d) { return cudaGetDevice(d); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return handle(e); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) {
  *n = 0;
  return cudaSuccess;
}
}
