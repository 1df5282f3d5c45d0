// fake_cudart.cpp -- a CUDA runtime without a GPU, for CPU tests of the host
// side of libeagb.so: the library's own objects are linked with this file in
// place of the CUDA runtime.
//
// Device memory is host memory, copies and fills are done at once, kernels do
// nothing.  What the runtime refuses by itself is refused here too: dynamic
// shared memory beyond what a kernel was opted in to, block and grid sizes out
// of range.  An error stays pending for cudaGetLastError, as it does there.
// fake_* functions inject allocation failures and count what was called.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
struct State {
  std::recursive_mutex m;
  std::map<char *, size_t> mem;          // live device memory
  std::map<const void *, int> smem;      // dynamic SMEM a kernel is opted in to
  std::map<const void *, std::string> name;
  std::map<std::string, long> calls;
  long fail_in = -1;                     // allocations until one fails
  std::string refused;                   // launches refused, one a line
};
State &S() {  // kernels are registered before this file's own objects exist
  static State *s = new State;
  return *s;
}
struct Lock {
  std::lock_guard<std::recursive_mutex> l{S().m};
};
thread_local cudaError_t g_last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
};
thread_local Config g_config;
constexpr size_t kBlockSmem = 227 * 1024;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
void count(const char *what) {
  Lock l;
  ++S().calls[what];
}
cudaError_t launch(const void *f, dim3 g, dim3 b, size_t smem) {
  Lock l;
  const auto it = S().smem.find(f);
  const size_t lim = it == S().smem.end() ? 48 * 1024 : (size_t)it->second;
  const std::string name = S().name.count(f) ? S().name[f] : "?";
  ++S().calls["launch " + name];
  if (smem > lim || b.x * b.y * b.z > 1024 || !b.x || !g.x || !g.y || g.y > 65535 || g.z > 65535) {
    S().refused += name + " grid " + std::to_string(g.x) + " x " + std::to_string(g.y) + " block " + std::to_string(b.x) +
                 " smem " + std::to_string(smem) + " of " + std::to_string(lim) + "\n";
    return done(cudaErrorInvalidValue);
  }
  return cudaSuccess;
}
void *fresh() {
  static uintptr_t next = 0x1000;
  Lock l;
  return (void *)(next += 16);
}
}  // namespace

extern "C" {

// The n-th allocation from now on fails (0: the next one; negative: none does).
void fake_fail_in(long n) {
  Lock l;
  S().fail_in = n;
}
long fake_live(void) {
  Lock l;
  return (long)S().mem.size();
}
unsigned long long fake_live_bytes(void) {
  Lock l;
  unsigned long long s = 0;
  for (auto &p : S().mem) s += p.second;
  return s;
}
// Calls whose name begins with `what` (kernels: "launch " and the mangled name).
long fake_calls(const char *what) {
  Lock l;
  long n = 0;
  for (auto &c : S().calls)
    if (!c.first.compare(0, std::strlen(what), what)) n += c.second;
  return n;
}
const char *fake_refused(void) { return S().refused.c_str(); }
void fake_reset(void) {
  Lock l;
  S().calls.clear();
  S().refused.clear();
  S().fail_in = -1;
}

// Memory
cudaError_t cudaMalloc(void **p, size_t n) {
  Lock l;
  if (S().fail_in >= 0 && S().fail_in-- == 0) return done(cudaErrorMemoryAllocation);
  n = (n + 4095) & ~(size_t)4095;
  void *q = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (q == MAP_FAILED) return done(cudaErrorMemoryAllocation);
  S().mem[(char *)q] = n;
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  Lock l;
  if (!p) return cudaSuccess;
  const auto it = S().mem.find((char *)p);
  if (it == S().mem.end()) return done(cudaErrorInvalidValue);
  munmap(p, it->second);
  S().mem.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
  *p = ::operator new(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  ::operator delete(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = *t = (size_t)256 << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  count(k == cudaMemcpyHostToDevice ? "cudaMemcpy to device" : "cudaMemcpy");
  if (n && (!d || !s)) return done(cudaErrorInvalidValue);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (n && (!d || !s)) return done(cudaErrorInvalidValue);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
static cudaError_t fill(void *p, int v, size_t n) {
  if (n && !p) return done(cudaErrorInvalidValue);
  char *a = (char *)(((uintptr_t)p + 4095) & ~(uintptr_t)4095), *e = (char *)(((uintptr_t)p + n) & ~(uintptr_t)4095);
  if (v || e <= a) {
    std::memset(p, v, n);
    return cudaSuccess;
  }
  std::memset(p, 0, a - (char *)p);
  madvise(a, e - a, MADV_DONTNEED);  // whole pages: zero again without being touched
  std::memset(e, 0, (char *)p + n - e);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  count("cudaMemset");
  return fill(p, v, n);
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return fill(p, v, n); }

// Device, streams, events, graphs
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
  std::memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = (cudaStream_t)fresh(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)fresh(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = (cudaEvent_t)fresh(), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = (cudaGraph_t)fresh(), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  count("cudaGraphInstantiate");
  return *x = (cudaGraphExec_t)fresh(), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  count("cudaGraphLaunch");
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *) {
  return done(cudaErrorNotSupported);
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return done(cudaErrorNotSupported); }

// Errors
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError(void) { return g_last; }
const char *cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaErrorInvalidValue ? "invalid argument" : "error";
}

// Kernels
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  Lock l;
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  if (v < 0 || (size_t)v > kBlockSmem) return done(cudaErrorInvalidValue);
  S().smem[f] = v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
  std::memset(a, 0, sizeof(*a));
  a->maxThreadsPerBlock = 1024;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t smem, unsigned) {
  *n = smem <= kBlockSmem ? 1 : 0;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
  return *n = 8, cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **, size_t smem, cudaStream_t) {
  return launch(f, g, b, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st *st) {
  g_config = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = g_config.grid;
  *b = g_config.block;
  *smem = g_config.smem;
  *(cudaStream_t *)st = g_config.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { return *k = (cudaKernel_t)f, cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **, size_t smem, cudaStream_t) {
  return launch((const void *)k, g, b, smem);
}
void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  Lock l;
  S().name[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

// cuRAND host calls (the device probe's): none here
int curandCreateGenerator(void *, int) { return 1; }
int curandDestroyGenerator(void *) { return 1; }
int curandGenerateUniformDouble(void *, double *, size_t) { return 1; }
int curandSetGeneratorOffset(void *, unsigned long long) { return 1; }
int curandSetPseudoRandomGeneratorSeed(void *, unsigned long long) { return 1; }

}  // extern "C"
