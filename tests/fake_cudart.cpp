// A CUDA runtime without a GPU for tests of the library's host code: preloaded
// before libcudart, it keeps a log of the calls the library makes, counts
// device memory against a limit, refuses launches whose grid or block no GPU
// takes, and runs nothing.  Device pointers are numbers that nobody reads.
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::string g_log;
std::map<uintptr_t, size_t> g_live;            // device allocations
std::map<const void*, std::string> g_kernels;  // host stub -> device name
size_t g_limit = (size_t)1 << 62, g_used = 0;
uintptr_t g_next = (uintptr_t)1 << 40;
intptr_t g_handle = 0x1000;
bool g_capturing = false;
cudaError_t g_last = cudaSuccess;
struct { dim3 grid, block; size_t smem; cudaStream_t st; } g_config;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
const char* name(cudaStream_t s) {
  static char buf[32];
  if (!s) return "legacy";
  snprintf(buf, sizeof buf, "%p", (void*)s);
  return buf;
}
void note(const char* what, cudaStream_t s, const char* more = "") {
  g_log += std::string(what) + " " + name(s) + " " + more + "\n";
}
cudaError_t take(void** p, size_t n) {
  const size_t held = (n + 511) / 512 * 512;
  if (held > g_limit - g_used) return ret(cudaErrorMemoryAllocation);
  *p = (void*)g_next;
  g_live[g_next] = held;
  g_next += held + 4096;
  g_used += held;
  return cudaSuccess;
}
cudaError_t give(void* p) {
  if (!p) return cudaSuccess;
  auto it = g_live.find((uintptr_t)p);
  if (it == g_live.end()) return ret(cudaErrorInvalidValue);
  g_used -= it->second;
  g_live.erase(it);
  return cudaSuccess;
}
cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  char more[512];
  const auto it = g_kernels.find(f);
  snprintf(more, sizeof more, "%s grid %u,%u,%u block %u,%u,%u smem %zu", it == g_kernels.end() ? "?" : it->second.c_str(),
           g.x, g.y, g.z, b.x, b.y, b.z, smem);
  if (g.x == 0 || g.y == 0 || g.z == 0 || g.x > 0x7fffffffu || g.y > 65535 || g.z > 65535 || b.x * b.y * b.z == 0 ||
      b.x * b.y * b.z > 1024 || b.z > 64 || smem > 232448) {
    note("refused", s, more);
    return ret(cudaErrorInvalidConfiguration);
  }
  note("launch", s, more);
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- for the tests ----
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_limit(size_t bytes) { g_limit = bytes; }
size_t fake_used() { return g_used; }

// ---- the runtime ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* device, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_kernels[host] = device;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  g_config = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = g_config.grid;
  *b = g_config.block;
  *smem = g_config.smem;
  *(cudaStream_t*)st = g_config.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t smem, cudaStream_t s) {
  return launch(f, g, b, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1 << 20;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetLimit(size_t* v, cudaLimit) { *v = 0; return cudaSuccess; }
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorName(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
const char* cudaGetErrorString(cudaError_t e) { return cudaGetErrorName(e); }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof *a);
  a->numRegs = 64;
  a->maxThreadsPerBlock = 1024;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 8; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 8;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = (void*)((uintptr_t)1 << 39); return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) {
  char more[64];
  snprintf(more, sizeof more, "%zu", n);
  note("malloc", nullptr, more);
  return take(p, n);
}
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return take(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *t = g_limit;
  *f = g_limit - g_used;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)g_handle++; return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { note("memset", nullptr); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t s) { note("memset", s); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void*, size_t n, cudaMemcpyKind k, cudaStream_t s) {
  if (k == cudaMemcpyDeviceToHost) memset(dst, 0, n);
  note("memcpy", s);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind k) {
  return cudaMemcpyAsync(dst, src, n, k, nullptr);
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(g_handle++ * 16); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { note("sync", s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { g_capturing = true; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  g_capturing = false;
  *g = (cudaGraph_t)g_handle++;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)g_handle++;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { note("graph", s); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)g_handle++; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
}
