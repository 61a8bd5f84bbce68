// A CUDA runtime of host memory, preloaded in front of the real one
// (LD_PRELOAD) so that the library's host code runs without a GPU: kernels do
// nothing, device memory is host memory with a limit, and what was called is
// logged.  Only what the library calls is defined.
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>

namespace {

struct Block {
  size_t bytes;
  int device;
};

std::map<void*, Block> g_blocks;
std::map<const void*, cudaPointerAttributes> g_ptr;   // attributes told by a test
std::string g_log;
size_t g_used = 0, g_limit = ~size_t(0);
size_t g_pool_used = 0, g_pool_idle = 0;
unsigned long long g_pool_keep = 0;
int g_device = 0, g_fail_launch = 0;
cudaError_t g_last = cudaSuccess;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}

template <class... A>
void say(const char* fmt, A... a) {
  char line[256];
  snprintf(line, sizeof(line), fmt, a...);
  g_log += line;
  g_log += '\n';
}

cudaError_t launch(const void* f) {
  Dl_info info;
  const char* name = (dladdr(f, &info) && info.dli_sname) ? info.dli_sname : "?";
  if (g_fail_launch > 0 && --g_fail_launch == 0) return done(cudaErrorLaunchOutOfResources);
  say("launch %.120s device %d", name, g_device);
  return cudaSuccess;
}

void* take(size_t n) { return aligned_alloc(256, (n + 255) / 256 * 256 + 256); }

}  // namespace

extern "C" {

// ------------------------------------------------------------ for the tests
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_limit(size_t bytes) { g_limit = bytes; }
void fake_device(int d) { g_device = d; }
void fake_fail_launch(int nth) { g_fail_launch = nth; }
void fake_pointer(const void* p, int type, int device) {
  cudaPointerAttributes a;
  memset(&a, 0, sizeof(a));
  a.type = (cudaMemoryType)type;
  a.device = device;
  g_ptr[p] = a;
}
size_t fake_used() { return g_used; }
// double i of every block = i
void fake_count() {
  for (auto& b : g_blocks)
    for (size_t i = 0; i < b.second.bytes / sizeof(double); ++i) ((double*)b.first)[i] = (double)i;
}
size_t fake_pool_idle() { return g_pool_idle; }

// ------------------------------------------------------------ memory
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  if (g_used + g_pool_used + g_pool_idle + n > g_limit) return done(cudaErrorMemoryAllocation);
  *p = take(n);
  g_blocks[*p] = Block{n, g_device};
  g_used += n;
  say("malloc %zu device %d", n, g_device);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  auto it = g_blocks.find(p);
  if (it == g_blocks.end()) return cudaSuccess;
  g_used -= it->second.bytes;
  free(p);
  g_blocks.erase(it);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = take(n);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  say("memcpy %p %p %zu", d, s, n);
  memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof(*a));
  auto t = g_ptr.find(p);
  auto b = g_blocks.find(const_cast<void*>(p));
  if (t != g_ptr.end()) *a = t->second;
  else if (b != g_blocks.end()) {
    a->type = cudaMemoryTypeDevice;
    a->device = b->second.device;
  }
  return cudaSuccess;
}

// one pool; a block given back stays with it up to the release threshold
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*) {
  *pool = (cudaMemPool_t)&g_pool_keep;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr attr, void* v) {
  if (attr == cudaMemPoolAttrReleaseThreshold) g_pool_keep = *(unsigned long long*)v;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep) {
  if (g_pool_idle > keep) g_pool_idle = keep;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  *p = nullptr;
  const size_t from_idle = n < g_pool_idle ? n : g_pool_idle;
  if (g_used + g_pool_used + g_pool_idle - from_idle + n > g_limit) return done(cudaErrorMemoryAllocation);
  g_pool_idle -= from_idle;
  g_pool_used += n;
  *p = take(n);
  g_blocks[*p] = Block{0, g_device};
  say("pool malloc %zu", n);
  // the block's size, for cudaFreeAsync
  *(size_t*)*p = n;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  const size_t n = *(size_t*)p;
  g_blocks.erase(p);
  free(p);
  g_pool_used -= n;
  g_pool_idle += n;
  if (g_pool_idle > g_pool_keep) g_pool_idle = (size_t)g_pool_keep;
  return cudaSuccess;
}

// ------------------------------------------------------------ launches, streams, the rest
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) { return launch(f); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaGetDevice(int* d) {
  *d = g_device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  g_device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  say("stream device %d", g_device);
  *s = (cudaStream_t)take(8);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)take(8);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

}  // extern "C"
