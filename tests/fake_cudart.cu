// A CUDA runtime on the host, for tests of what the library does when a call fails.
//
// The library's objects are linked against this file instead of the runtime: device
// memory is host memory, streams run at once and kernels do nothing, but for a few
// whose outcome the host code acts on.  Tests set what is to fail through the fake_*
// functions.
// (Only the host pass: the device pass has some of these names as its own.)
#ifndef __CUDA_ARCH__
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <map>
#include <mutex>
#include <string>

#include "../lauematching_b200/csrc/kernels.cuh"

namespace {

std::mutex mu;
std::map<void *, size_t> device_mem, host_mem;
size_t device_used = 0, device_limit = ~(size_t)0, host_used = 0, host_limit = ~(size_t)0;
long device_mallocs = 0;
std::map<const void *, std::string> &kernels() {  // filled before this file's own objects are made
  static auto *m = new std::map<const void *, std::string>;
  return *m;
}
std::map<std::string, long> launched;
std::string fail_kernel;
long fail_copies_of = 0;  // copies of at least this many bytes fail (0: none)
unsigned long long hist[256];
unsigned survivors = 0, fractional = 0;
cudaError_t last = cudaSuccess;

cudaError_t result(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

cudaError_t take(std::map<void *, size_t> &mem, size_t &used, size_t limit, void **p, size_t n) {
  std::lock_guard<std::mutex> l(mu);
  n = n ? n : 1;
  if (n > limit || used > limit - n) return result(cudaErrorMemoryAllocation);
  void *m = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (m == MAP_FAILED) return result(cudaErrorMemoryAllocation);
  mem[m] = n;
  used += n;
  *p = m;
  return cudaSuccess;
}

cudaError_t give(std::map<void *, size_t> &mem, size_t &used, void *p) {
  if (!p) return cudaSuccess;
  std::lock_guard<std::mutex> l(mu);
  auto it = mem.find(p);
  if (it == mem.end()) return result(cudaErrorInvalidValue);
  used -= it->second;
  munmap(p, it->second);
  mem.erase(it);
  return cudaSuccess;
}

bool inside(const std::map<void *, size_t> &mem, const void *p) {
  auto it = mem.upper_bound(const_cast<void *>(p));
  if (it == mem.begin()) return false;
  --it;
  return static_cast<const char *>(p) < static_cast<const char *>(it->first) + it->second;
}

cudaError_t copy(void *d, const void *s, size_t n) {
  if (fail_copies_of && n >= (size_t)fail_copies_of) return result(cudaErrorUnknown);
  memmove(d, s, n);
  return cudaSuccess;
}

// The kernels whose outcome decides what the host does next.
void act(const std::string &name, void **args) {
  if (name.find("glist_total_kernel") != std::string::npos) {
    memcpy(*static_cast<unsigned long long **>(args[2]), hist, sizeof(hist));
  } else if (name.find("listed_kernel") != std::string::npos) {  // survivors in slot 0
    static_cast<lmb::CmpArgs *>(args[0])->surv_cnt[0] += survivors;
  } else if (name.find("whole_kernel") != std::string::npos) {
    **static_cast<unsigned **>(args[2]) |= fractional;
  } else if (name.find("order_kernel") != std::string::npos && name.find("noalloc") == std::string::npos) {
    const lmb::OrderArgs &a = *static_cast<lmb::OrderArgs *>(args[0]);
    for (int i = 0; i < a.nslots; i++) {
      const int k = a.slots[i];
      a.host_status[k] = a.status[k];
      a.status[k] = 0;
    }
  }
}

struct Shape {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
};
thread_local Shape pushed;
int handle[64];

}  // namespace

extern "C" {

// ---- what tests set and read ----------------------------------------------------
void fake_reset() {
  device_limit = host_limit = ~(size_t)0;
  device_mallocs = 0;
  launched.clear();
  fail_kernel.clear();
  fail_copies_of = 0;
  memset(hist, 0, sizeof(hist));
  survivors = fractional = 0;
  last = cudaSuccess;
}
void fake_limits(size_t device, size_t host) {
  device_limit = device;
  host_limit = host;
}
size_t fake_device_used() { return device_used; }
size_t fake_host_used() { return host_used; }
long fake_device_mallocs() { return device_mallocs; }
void fake_fail_kernel(const char *part) { fail_kernel = part; }
void fake_fail_copies(long bytes) { fail_copies_of = bytes; }
void fake_counts(int count, unsigned long long records) { hist[count] = records; }
void fake_survivors(unsigned n) { survivors = n; }
void fake_fractional(unsigned yes) { fractional = yes; }  // frames and backgrounds as 16-bit numbers
long fake_launched(const char *part) {
  long n = 0;
  for (const auto &k : launched)
    if (k.first.find(part) != std::string::npos) n += k.second;
  return n;
}

// ---- the runtime ------------------------------------------------------------------
void **__cudaRegisterFatBinary(void *) { return reinterpret_cast<void **>(handle); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {
  kernels()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *st) {
  pushed = Shape{g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = pushed.grid;
  *b = pushed.block;
  *smem = pushed.smem;
  *static_cast<cudaStream_t *>(st) = pushed.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **args, size_t, cudaStream_t) {
  const std::string &name = kernels()[f];
  if (!fail_kernel.empty() && name.find(fail_kernel) != std::string::npos)
    return result(cudaErrorLaunchOutOfResources);
  launched[name]++;
  act(name, args);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  device_mallocs++;
  return take(device_mem, device_used, device_limit, p, n);
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) { return give(device_mem, device_used, p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  return take(host_mem, host_used, host_limit, p, n);
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void *p) { return give(host_mem, host_used, p); }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *t = device_limit;
  *f = device_limit - device_used;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  std::lock_guard<std::mutex> l(mu);
  memset(a, 0, sizeof(*a));
  a->type = inside(device_mem, p) ? cudaMemoryTypeDevice
            : inside(host_mem, p) ? cudaMemoryTypeHost
                                  : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return copy(d, s, n);
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char *cudaGetErrorString(cudaError_t) { return "a failure that the test asked for"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10 : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
  memset(a, 0, sizeof(*a));
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                   unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return result(cudaErrorInvalidSymbol); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(handle);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = reinterpret_cast<cudaGraph_t>(handle);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  *x = reinterpret_cast<cudaGraphExec_t>(handle);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = reinterpret_cast<cudaEvent_t>(handle);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}

}  // extern "C"
#endif
