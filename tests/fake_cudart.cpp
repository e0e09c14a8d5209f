// A CUDA runtime for tests of the library's host code on a machine without a
// GPU: device memory is host memory filled with the double 1.0, copies and
// fills happen at once, kernels do not run.  It records what the tests ask
// about: allocations (and makes a chosen one fail), work given to the legacy
// default stream, and null pointers among the arguments of chosen kernels.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <string>
#include <vector>

namespace {
struct Watch {
  std::string kernel;
  int arg, n;   // n pointers from the start of argument arg
  size_t room;  // bytes that have to be left in their allocations
};
std::map<char *, size_t> g_mem;        // live allocations, device and page-locked
std::map<char *, size_t> g_dev;        // the device ones
std::map<const void *, std::string> g_name;
std::map<std::string, int> g_count;    // launches by kernel
std::string g_fast, g_last_kernel;
int g_fast_ctas, g_last_ctas;
std::vector<Watch> g_watch;
int g_allocs, g_fail_at, g_legacy, g_null, g_launches, g_bad_frees, g_short;
cudaError_t g_last;

cudaError_t err(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
cudaError_t alloc(void **p, size_t n, bool dev) {
  if (++g_allocs == g_fail_at) return err(cudaErrorMemoryAllocation);
  char *q = (char *)aligned_alloc(512, (n + 511) / 512 * 512 + 512);
  for (size_t i = 0; i + 8 <= n; i += 8) *(double *)(q + i) = 1.0;
  g_mem[q] = n;
  if (dev) g_dev[q] = n;
  *p = q;
  return cudaSuccess;
}
cudaError_t release(void *p) {
  if (!p) return cudaSuccess;
  if (!g_mem.erase((char *)p)) return g_bad_frees++, err(cudaErrorInvalidValue);
  g_dev.erase((char *)p);
  free(p);
  return cudaSuccess;
}
// bytes from p to the end of its allocation; the whole address space if it is not one
size_t room(const void *p) {
  auto it = g_mem.upper_bound((char *)p);
  if (it == g_mem.begin()) return (size_t)-1;
  --it;
  const size_t off = (char *)p - it->first;
  return off < it->second ? it->second - off : (size_t)-1;
}
cudaError_t copy(void *d, const void *s, size_t n) {
  if (!d || !s || n > room(d) || n > room(s)) return err(cudaErrorInvalidValue);
  memmove(d, s, n);
  return cudaSuccess;
}
struct Config {
  dim3 g, b;
  size_t sm;
  cudaStream_t st;
};
std::vector<Config> g_config;
}  // namespace

extern "C" {
// ------------------------------------------------------- what the tests use
void fake_fail_at(int n) { g_allocs = 0, g_fail_at = n; }   // the n-th allocation from now on; 0: none
int fake_allocs() { return g_allocs; }
int fake_live() { return (int)g_mem.size(); }
int fake_legacy() { return g_legacy; }
int fake_launches() { return g_launches; }
// the times that events measure: half as long after a launch of this kernel with up to so many CTAs
void fake_fast(const char *kernel, int ctas) { g_fast = kernel, g_fast_ctas = ctas; }
void fake_watch(const char *kernel, int arg, int n) { g_watch.push_back({kernel, arg, n, 0}); }
void fake_watch_room(const char *kernel, int arg, size_t room) { g_watch.push_back({kernel, arg, 1, room}); }
void fake_unwatch() { g_watch.clear(); }
int fake_short_args() { return g_short; }
int fake_launched(const char *kernel) {
  int n = 0;
  for (const auto &k : g_count)
    if (k.first.find(kernel) != std::string::npos) n += k.second;
  return n;
}
int fake_null_args() { return g_null; }
int fake_bad_frees() { return g_bad_frees; }

// -------------------------------------------------------------- the runtime
cudaError_t cudaMalloc(void **p, size_t n) { return alloc(p, n, true); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return alloc(p, n, true); }
cudaError_t cudaMallocHost(void **p, size_t n) { return alloc(p, n, false); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return alloc(p, n, false); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaFree(void *p) { return release(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return release(p); }
cudaError_t cudaFreeHost(void *p) { return release(p); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  g_legacy += st == nullptr;
  return copy(d, s, n);
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return g_legacy++, copy(d, s, n); }
cudaError_t cudaMemset(void *d, int v, size_t n) { return g_legacy++, memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  g_legacy += st == nullptr;
  if (!d || n > room(d)) return err(cudaErrorInvalidValue);
  return memset(d, v, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t st) {
  g_legacy += st == nullptr;
  for (size_t i = 0; i < h; i++)
    if (copy((char *)d + i * dp, (const char *)s + i * sp, w) != cudaSuccess) return cudaErrorInvalidValue;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  memset(a, 0, sizeof(*a));
  auto it = g_dev.upper_bound((char *)p);
  const bool dev = it != g_dev.begin() && (char *)p < std::prev(it)->first + std::prev(it)->second;
  a->type = dev ? cudaMemoryTypeDevice : room(p) != (size_t)-1 ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
static int address_range(unsigned long long *base, size_t *n, unsigned long long p) {
  auto it = g_dev.upper_bound((char *)p);
  if (it == g_dev.begin() || (char *)p >= std::prev(it)->first + std::prev(it)->second) return 1;
  *base = (unsigned long long)std::prev(it)->first;
  *n = std::prev(it)->second;
  return 0;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *) {
  *f = strcmp(name, "cuMemGetAddressRange") ? nullptr : (void *)address_range;
  return *f ? cudaSuccess : err(cudaErrorInvalidValue);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = nullptr, cudaErrorInvalidValue; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  static char some[64];
  static int n;
  return *s = (cudaStream_t)(some + n++ % 64), cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = !g_fast.empty() && g_last_kernel.find(g_fast) != std::string::npos && g_last_ctas <= g_fast_ctas ? 0.5f : 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  return *e = nullptr, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaProfilerStart() { return cudaSuccess; }
cudaError_t cudaProfilerStop() { return cudaSuccess; }

// ----------------------------------------------------------------- launches
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t st) {
  g_config.push_back({g, b, sm, st});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *sm, void *st) {
  const Config c = g_config.back();
  g_config.pop_back();
  *g = c.g, *b = c.b, *sm = c.sm, *(cudaStream_t *)st = c.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t, cudaStream_t st) {
  g_launches++;
  g_legacy += st == nullptr;
  if (!g.x || !g.y || !g.z || !b.x || b.x * b.y * b.z > 1024) return err(cudaErrorInvalidConfiguration);
  const std::string &name = g_name[f];
  g_count[name]++;
  g_last_kernel = name;
  g_last_ctas = g.x;
  for (const Watch &w : g_watch)
    if (name.find(w.kernel) != std::string::npos)
      for (int i = 0; i < w.n; i++) {
        const void *p = ((void **)args[w.arg])[i];
        g_null += p == nullptr;
        g_short += room(p) < w.room;
      }
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  g_name[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
