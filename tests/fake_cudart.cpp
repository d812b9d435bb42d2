// Stand-in for the CUDA runtime behind the library's launchers: it records every
// launch and copy and returns the errors a test asks for, so that the choice of
// kernels and what a refused launch leaves behind are checked without a GPU.
// Linked with the library's own object files; no kernel runs.
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string> g_names;
std::string g_log;
cudaError_t g_last = cudaSuccess;
unsigned g_max_cluster = 16;  // clusters of more CTAs are refused
int g_launches_to_fail = 0, g_attrs_to_fail = 0, g_sms = 148;
bool g_host_pointers = false;  // what cudaPointerGetAttributes says of every pointer

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
void note(const char* fmt, ...) {
  char line[512];
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(line, sizeof line, fmt, ap);
  va_end(ap);
  g_log += line;
}
}  // namespace

extern "C" {
// ---- what a test sets and reads ----------------------------------------------------
void fake_reset() {
  g_log.clear();
  g_last = cudaSuccess;
  g_max_cluster = 16;
  g_launches_to_fail = g_attrs_to_fail = 0;
  g_sms = 148;
  g_host_pointers = false;
}
void fake_max_cluster(unsigned n) { g_max_cluster = n; }
void fake_fail_launches(int n) { g_launches_to_fail = n; }
void fake_fail_attributes(int n) { g_attrs_to_fail = n; }
void fake_sms(int n) { g_sms = n; }
void fake_host_pointers() { g_host_pointers = true; }
const char* fake_log() { return g_log.c_str(); }
int fake_pending_error() { return (int)g_last; }

// ---- registration (written by nvcc into every object) --------------------------------
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, void*, void*, void*, void*, int*) {
  g_names[fn] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

// ---- launches ------------------------------------------------------------------------
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
  unsigned cluster = 0;  // an ordinary launch
  for (unsigned i = 0; i < c->numAttrs; i++)
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
  cudaError_t e = cudaSuccess;
  if (cluster > g_max_cluster) e = cudaErrorInvalidClusterSize;
  if (g_launches_to_fail > 0) {
    g_launches_to_fail--;
    e = cudaErrorLaunchOutOfResources;
  }
  if (c->gridDim.x == 0) e = cudaErrorInvalidConfiguration;
  note("%s %s grid %u block %u smem %zu cluster %u\n", e == cudaSuccess ? "launch" : "refused", g_names[fn].c_str(),
       c->gridDim.x, c->blockDim.x, c->dynamicSmemBytes, cluster);
  return done(e);
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
  note("launch %s grid %u block %u smem %zu cluster 0\n", g_names[fn].c_str(), g.x, b.x, smem);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) {
  if (g_attrs_to_fail <= 0) return cudaSuccess;
  g_attrs_to_fail--;
  return done(cudaErrorInvalidValue);
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes*, const void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }

// ---- device, streams, memory: everything is host memory, every stream is idle -----------
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? g_sms : 0;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::malloc(n)) ? cudaSuccess : done(cudaErrorMemoryAllocation); }
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  note("copy %s %zu\n", k == cudaMemcpyHostToDevice ? "h2d" : k == cudaMemcpyDeviceToHost ? "d2h" : "d2d", n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof *a);
  a->type = g_host_pointers ? cudaMemoryTypeUnregistered : cudaMemoryTypeDevice;
  a->devicePointer = const_cast<void*>(p);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
}
