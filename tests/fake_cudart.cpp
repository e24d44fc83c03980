// A CUDA runtime without a GPU, preloaded ahead of libcudart by the host-side
// tests: device memory is host memory, kernels do nothing, and every call is
// written to a log ("absent": a copy to host pages that nothing has touched).
// The n-th allocation can be made to fail, and the device's free memory to be
// what a test wants.
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <unistd.h>

#include <map>
#include <string>
#include <vector>

namespace {
std::string g_log;
std::map<const void*, std::string> g_names;
std::map<void*, size_t> g_live;
size_t g_total = (size_t)288 << 30, g_used = 0;
long g_fail = -1;  // allocations until one fails; negative: none does
cudaError_t g_last = cudaSuccess;
std::string g_watch;
int g_arg = 0;
uintptr_t g_streams = 0x1000;

void put(const char* what, const void* p, size_t n, const void* stream) {
  char b[512];
  snprintf(b, sizeof b, "%s %p %zu %p\n", what, p, n, stream);
  g_log += b;
}
cudaError_t fail(cudaError_t e) { return g_last = e; }
struct Config {
  dim3 g, b;
  size_t sm;
  cudaStream_t s;
} g_conf;
// whether some page of host memory has not been touched yet
bool absent(const void* p, size_t n) {
  const uintptr_t page = sysconf(_SC_PAGESIZE), lo = (uintptr_t)p / page * page;
  std::vector<unsigned char> v(((uintptr_t)p + n - lo + page - 1) / page);
  if (n == 0 || mincore((void*)lo, (uintptr_t)p + n - lo, v.data())) return false;
  for (unsigned char c : v)
    if (!(c & 1)) return true;
  return false;
}
int encode_tiled(...) { return 0; }
int ctx_current(void** c) {
  *c = (void*)0x10;
  return 0;
}
int ctx_id(void*, unsigned long long* id) {
  *id = 1;
  return 0;
}
}  // namespace

extern "C" {
// ---- the tests' handles
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_fail(long n) { g_fail = n; }
void fake_total(size_t n) { g_total = n; }
size_t fake_used() { return g_used; }
// log argument `arg` (8 bytes) of launches whose kernel's name contains `name`
void fake_watch(const char* name, int arg) {
  g_watch = name;
  g_arg = arg;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_fail == 0 || n > g_total - g_used) {
    g_fail = -1;
    put("nomem", nullptr, n, nullptr);
    return fail(cudaErrorMemoryAllocation);
  }
  if (g_fail > 0) --g_fail;
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  if (n <= (1u << 20)) memset(*p, 0, n);
  g_live[*p] = n;
  g_used += n;
  put("malloc", *p, n, nullptr);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  auto it = g_live.find(p);
  if (it == g_live.end()) return fail(cudaErrorInvalidValue);
  g_used -= it->second;
  put("free", p, it->second, nullptr);
  g_live.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
  put("register", p, n, nullptr);
  return cudaSuccess;
}
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = g_total - g_used;
  *t = g_total;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  put(k == cudaMemcpyHostToDevice ? "h2d" : k == cudaMemcpyDeviceToHost ? "d2h" : "d2d",
      k == cudaMemcpyDeviceToHost ? s : d, n, st);
  if (k == cudaMemcpyDeviceToHost && absent(d, n)) put("absent", d, n, st);
  if (k != cudaMemcpyDeviceToDevice) memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, 0); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  put("memset", d, n, st);
  if (n <= (1u << 20)) memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, 0); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof *a);
  a->type = cudaMemoryTypeDevice;
  a->devicePointer = (void*)p;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = (void*)s;
  return cudaSuccess;
}

// ---- devices, errors, streams, events
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)(g_streams += 0x10);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  put("sync", nullptr, 0, s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)0x20;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)0x30;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
  *g = (cudaGraph_t)0x20;
  return cudaSuccess;
}
cudaError_t cudaGraphAddChildGraphNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraph_t) {
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)0x40;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *p = !strcmp(name, "cuCtxGetCurrent") ? (void*)ctx_current : !strcmp(name, "cuCtxGetId") ? (void*)ctx_id : (void*)encode_tiled;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

// ---- kernels
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t s) {
  g_conf = {g, b, sm, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* s) {
  *g = g_conf.g, *b = g_conf.b, *sm = g_conf.sm, *(cudaStream_t*)s = g_conf.s;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t s) {
  const std::string& n = g_names[f];
  const void* a = nullptr;
  if (!g_watch.empty() && n.find(g_watch) != std::string::npos) memcpy(&a, args[g_arg], sizeof a);
  put(("launch:" + n).c_str(), a, 0, s);
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** args, size_t sm, cudaStream_t s) {
  return cudaLaunchKernel((const void*)k, g, b, args, sm, s);
}
}
