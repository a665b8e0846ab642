// A CUDA runtime without a device, for host-side tests (LD_PRELOADed before the library):
// memory is host memory, kernels do nothing but are logged, streams and events are numbers.
// A test asks for the failures of interest:
//   fake_devices(n)         n devices; what is set for one device does not hold on another
//   fake_limit(bytes)       allocations beyond that many bytes in all fail (0: none does)
//   fake_fail_alloc(k, n)   after k more allocations, n fail
//   fake_fail_launch(name)  launches of kernels whose name contains it fail ("": none does)
//   fake_contents(v)        what fingerprints say of every array from here on
//   fake_log(buf, n)        the launches since the last call, one "device kernel note" a line
// A launch with more than 48 KB of dynamic shared memory fails, as on a device, unless the
// kernel's limit was raised on the current one.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

#include "kernels.hpp"

namespace {
std::recursive_mutex mu;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
int ndevices = 1;
size_t limit = 0, used = 0;
int fail_after = 0, fail_count = 0;
unsigned long long contents = 1;
constexpr size_t kTotal = size_t(64) << 30;
std::map<void*, size_t> blocks;
std::map<const void*, std::string> names;
std::map<std::pair<int, const void*>, int> smem;
std::string fail_name, text;
std::set<cudaStream_t> capturing;

struct Config {
  dim3 grid, block;
  size_t shared;
  cudaStream_t st;
};
thread_local std::vector<Config> pushed;

cudaError_t result(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}

cudaError_t launch(const void* f, dim3 grid, size_t shared, void** args) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const std::string& n = names[f];
  if (!fail_name.empty() && n.find(fail_name) != std::string::npos) return result(cudaErrorInvalidValue);
  const auto it = smem.find({device, f});
  if (shared > 48 * 1024 && (it == smem.end() || size_t(it->second) < shared)) return result(cudaErrorInvalidValue);
  text += std::to_string(device) + " " + n;
  if (n.find("oz_pack_kernel") != std::string::npos) {
    const auto* j = static_cast<const mpsxx::OzPackJobs*>(args[0]);
    text += " " + std::to_string(j->n);
  }
  if (n.find("fingerprint_kernel") != std::string::npos) {
    const auto* j = static_cast<const mpsxx::PrintJobs*>(args[0]);
    for (unsigned i = 0; i < grid.y; ++i) j->out[i]->h[0] = j->out[i]->h[1] = contents;
  }
  text += "\n";
  return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_devices(int n) { ndevices = n; }
void fake_limit(size_t b) { limit = b; }
void fake_fail_alloc(int k, int n) {
  fail_after = k;
  fail_count = n;
}
void fake_fail_launch(const char* n) { fail_name = n; }
void fake_contents(unsigned long long v) { contents = v; }
size_t fake_used() { return used; }
int fake_log(char* buf, int n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const int len = static_cast<int>(text.size());
  if (buf && n > 0) {
    snprintf(buf, size_t(n), "%s", text.c_str());
    text.clear();
  }
  return len;
}

cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= ndevices) return result(cudaErrorInvalidDevice);
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = ndevices;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "invalid"; }
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (fail_after > 0) {
    --fail_after;
  } else if (fail_count > 0) {
    --fail_count;
    return result(cudaErrorMemoryAllocation);
  }
  if (used + n > kTotal || (limit && used + n > limit)) return result(cudaErrorMemoryAllocation);
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  blocks[*p] = n;
  used += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  const auto it = blocks.find(p);
  if (it == blocks.end()) return p ? result(cudaErrorInvalidValue) : cudaSuccess;
  used -= it->second;
  blocks.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  const size_t all = limit ? limit : kTotal;
  *t = all;
  *f = all > used ? all - used : 0;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = aligned_alloc(4096, (n + 4095) / 4096 * 4096);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  static long next = 0;
  *s = reinterpret_cast<cudaStream_t>(++next * 16);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(16);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode) {
  return capturing.insert(st).second ? cudaSuccess : result(cudaErrorIllegalState);
}
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(16);
  return capturing.erase(st) ? cudaSuccess : result(cudaErrorIllegalState);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(16);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  return launch(f, c->gridDim, c->dynamicSmemBytes, args);
}

// what the compiler's launch syntax and module registration call
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  std::lock_guard<std::recursive_mutex> lk(mu);
  names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  pushed.push_back({g, b, s, st});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  const Config c = pushed.back();
  pushed.pop_back();
  *g = c.grid;
  *b = c.block;
  *s = c.shared;
  *static_cast<cudaStream_t*>(st) = c.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void** args, size_t s, cudaStream_t) {
  return launch(reinterpret_cast<const void*>(k), grid, s, args);
}

int cusolverDnCreate(void** h) {
  *h = &mu;
  return 0;
}
int cusolverDnSetStream(void*, cudaStream_t) { return 0; }
int cusolverDnDestroy(void*) { return 0; }
int cusolverDnDestroyParams(void*) { return 0; }
}
