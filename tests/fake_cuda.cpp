// A CUDA runtime without a GPU, for tests of the library's host code: linked
// with the library's own objects in place of the real runtime.  "Device" memory
// is the host's, copies happen at once, kernels are counted and not run.  The
// calls that a test names fail, and leave the pending error that a failing call
// of the runtime leaves.
#include <cuda_runtime_api.h>
#include <sys/syscall.h>
#include <time.h>
#include <unistd.h>

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

namespace {
thread_local cudaError_t g_last = cudaSuccess;
std::mutex g_mu;
struct Failure { int from, times; cudaError_t code; };
std::map<std::string, Failure> g_failures;    // call -> the calls of it that fail
std::map<const void *, std::string> g_names;  // host stub -> kernel
std::map<const void *, std::pair<void *, size_t>> g_vars;
std::vector<std::string> g_launched;
int g_slow_ms = 0, g_busy_ms = 0;
struct Patch { size_t bytes, offset; unsigned long long value; } g_patch = {};

// The fake's own containers always have memory.
thread_local int g_inside = 0;
struct Inside {
  Inside() { g_inside++; }
  ~Inside() { g_inside--; }
};

cudaError_t result(const char *call) {
  Inside inside;
  std::lock_guard<std::mutex> lock(g_mu);
  auto f = g_failures.find(call);
  if (f == g_failures.end()) return cudaSuccess;
  if (--f->second.from >= 0 || f->second.times-- <= 0) return cudaSuccess;
  return g_last = f->second.code;
}
bool g_no_host_memory = false;
struct Launch { dim3 grid, block; size_t smem; cudaStream_t stream; };
thread_local std::vector<Launch> g_config;
}  // namespace

void *operator new(size_t n) {
  void *p = g_no_host_memory && !g_inside ? nullptr : malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" {
// ---- the test's side -------------------------------------------------------------
// After `skip` more calls of `call`, the next `times` of them return `code`.
void fake_fail(const char *call, int skip, int times, int code) {
  std::lock_guard<std::mutex> lock(g_mu);
  g_failures[call] = Failure{skip, times, (cudaError_t)code};
}
int fake_launches(void) { return (int)g_launched.size(); }
// The next copy to the device takes this long.
void fake_slow_copy(int ms) { g_slow_ms = ms; }
// An event takes this long to come, from the wait for it on.
void fake_busy_device(int ms) { g_busy_ms = ms; }
// How often a thread has slept for a time (not until it is woken).
std::atomic<int> g_sleeps{0};
int fake_sleeps(void) { return g_sleeps; }
int nanosleep(const timespec *t, timespec *left) {
  g_sleeps++;
  return (int)syscall(SYS_nanosleep, t, left);
}
// The next copy of `bytes` bytes back to the host has `value` at `offset`.
void fake_read_back(size_t bytes, size_t offset, unsigned long long value) {
  g_patch = Patch{bytes, offset, value};
}

// operator new fails, as when the host has no memory left.
void fake_no_host_memory(int on) { g_no_host_memory = on != 0; }

// ---- the runtime's --------------------------------------------------------------
#define FAKE(name, args, ...)                       \
  cudaError_t name args {                           \
    const cudaError_t e = result(#name);            \
    if (e != cudaSuccess) return e;                 \
    __VA_ARGS__;                                    \
    return cudaSuccess;                             \
  }
FAKE(cudaGetDeviceCount, (int *n), *n = 1)
FAKE(cudaGetDevice, (int *d), *d = 0)
FAKE(cudaSetDevice, (int), )
FAKE(cudaGetDeviceProperties, (cudaDeviceProp * p, int), memset(p, 0, sizeof(*p));
     p->multiProcessorCount = 148)
FAKE(cudaDeviceGetAttribute, (int *v, cudaDeviceAttr, int), *v = 148)
FAKE(cudaMemGetInfo, (size_t * f, size_t *t), *f = *t = (size_t)1 << 30)
FAKE(cudaMalloc, (void **p, size_t n), *p = calloc(1, n ? n : 1))
FAKE(cudaHostAlloc, (void **p, size_t n, unsigned), *p = calloc(1, n ? n : 1))
FAKE(cudaFree, (void *p), free(p))
FAKE(cudaFreeHost, (void *p), free(p))
FAKE(cudaMemcpy, (void *d, const void *s, size_t n, cudaMemcpyKind), memcpy(d, s, n))
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  const cudaError_t e = result("cudaMemcpyAsync");
  if (e != cudaSuccess) return e;
  memcpy(d, s, n);
  if (kind == cudaMemcpyDeviceToHost && n == g_patch.bytes) {
    memcpy((char *)d + g_patch.offset, &g_patch.value, sizeof(g_patch.value));
    g_patch.bytes = 0;
  }
  int ms = 0;
  if (kind == cudaMemcpyHostToDevice) {
    std::lock_guard<std::mutex> lock(g_mu);
    std::swap(ms, g_slow_ms);
  }
  if (ms) std::this_thread::sleep_for(std::chrono::milliseconds(ms));
  return cudaSuccess;
}
FAKE(cudaMemsetAsync, (void *d, int v, size_t n, cudaStream_t), memset(d, v, n))
FAKE(cudaMemcpyToSymbol, (const void *, const void *, size_t, size_t, cudaMemcpyKind), )
FAKE(cudaGetSymbolAddress, (void **p, const void *v), *p = g_vars[v].first)
FAKE(cudaStreamCreateWithFlags, (cudaStream_t * s, unsigned), *s = (cudaStream_t)malloc(1))
FAKE(cudaStreamDestroy, (cudaStream_t s), free(s))
FAKE(cudaStreamSynchronize, (cudaStream_t), )
FAKE(cudaStreamWaitEvent, (cudaStream_t, cudaEvent_t, unsigned), )
FAKE(cudaEventCreate, (cudaEvent_t * v), *v = (cudaEvent_t)malloc(1))
FAKE(cudaEventCreateWithFlags, (cudaEvent_t * v, unsigned), *v = (cudaEvent_t)malloc(1))
FAKE(cudaEventDestroy, (cudaEvent_t v), free(v))
FAKE(cudaEventRecord, (cudaEvent_t, cudaStream_t), )
FAKE(cudaEventRecordWithFlags, (cudaEvent_t, cudaStream_t, unsigned), )
FAKE(cudaEventQuery, (cudaEvent_t), )
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  const cudaError_t e = result("cudaEventSynchronize");
  // the runtime's wait spins, by default
  const auto until = std::chrono::steady_clock::now() + std::chrono::milliseconds(g_busy_ms);
  while (std::chrono::steady_clock::now() < until) {}
  return e;
}
FAKE(cudaEventElapsedTime, (float *ms, cudaEvent_t, cudaEvent_t), *ms = 0)
FAKE(cudaFuncSetAttribute, (const void *, cudaFuncAttribute, int), )
FAKE(cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags,
     (int *n, const void *, int, size_t, unsigned), *n = 3)
// no graphs: the library then issues the work as plain launches
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  return g_last = cudaErrorNotSupported;
}
FAKE(cudaStreamEndCapture, (cudaStream_t, cudaGraph_t *g), *g = nullptr)
FAKE(cudaGraphInstantiate, (cudaGraphExec_t *, cudaGraph_t, unsigned long long), )
FAKE(cudaGraphLaunch, (cudaGraphExec_t, cudaStream_t), )
FAKE(cudaGraphDestroy, (cudaGraph_t), )
FAKE(cudaGraphExecDestroy, (cudaGraphExec_t), )
cudaError_t cudaPeekAtLastError(void) { return g_last; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "an error of the test's"; }

cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t, cudaStream_t) {
  const cudaError_t e = result("cudaLaunchKernel");
  if (e != cudaSuccess) return e;
  Inside inside;
  std::lock_guard<std::mutex> lock(g_mu);
  g_launched.push_back(g_names[f]);
  return cudaSuccess;
}

// what the compiler's stubs call
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  Inside inside;
  g_config.push_back(Launch{grid, block, smem, s});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
  const Launch l = g_config.back();
  g_config.pop_back();
  *grid = l.grid;
  *block = l.block;
  *smem = l.smem;
  *(cudaStream_t *)s = l.stream;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {
  g_names[f] = name;
}
void __cudaRegisterVar(void **, char *v, char *, const char *, int, size_t n, int, int) {
  g_vars[v] = {calloc(1, n), n};
}
}
