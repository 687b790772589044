// A CUDA runtime for the library's host code on a machine without a GPU:
// device memory is host memory, kernels do nothing, and every copy, launch and
// wait is checked against the order CUDA promises. A copy from pageable host
// memory may return before its data is on the device (a synchronous one on the
// legacy stream too), so it stays pending until something waits for it; a
// kernel launched on another stream meanwhile may read the old contents.
#include <cuda_runtime_api.h>
#include <driver_types.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

struct CUstream_st {
  bool blocking;
};
struct CUevent_st {
  cudaStream_t stream = nullptr;
  long seq = 0;
};

namespace {
struct Pending {
  cudaStream_t stream;
  size_t bytes;
  long seq;
  std::set<cudaStream_t> ordered;  // streams that wait for it
};
std::mutex mu;
long seq = 0;
std::vector<Pending> pending;
std::map<void*, size_t> live, pinned;
std::map<const void*, std::string> kernels;
std::map<std::string, long> launches;
std::string unordered;

// What runs in stream b comes after what stream a holds: the same stream, or
// the legacy stream (null) and a blocking one.
bool in_order(cudaStream_t a, cudaStream_t b) {
  return a == b || (!a && b->blocking) || (a && !b && a->blocking);
}
void wait(cudaStream_t s, long until) {
  std::vector<Pending> left;
  for (const Pending& p : pending)
    if (p.seq > until || !in_order(p.stream, s)) left.push_back(p);
  pending.swap(left);
}
bool is_pinned(const void* p) {
  for (auto& [base, n] : pinned)
    if (p >= base && p < (char*)base + n) return true;
  return false;
}
void copied(cudaStream_t s, const void* src, size_t n, cudaMemcpyKind kind) {
  if (kind == cudaMemcpyHostToDevice && n && !(s == nullptr && is_pinned(src))) pending.push_back({s, n, ++seq, {}});
}
cudaError_t allocate(void** p, size_t n) {
  std::lock_guard<std::mutex> g(mu);
  *p = std::calloc(1, n ? n : 1);
  if (!*p) return cudaErrorMemoryAllocation;
  live[*p] = n;
  return cudaSuccess;
}
cudaError_t give_back(void* p) {
  std::lock_guard<std::mutex> g(mu);
  live.erase(p);
  std::free(p);
  return cudaSuccess;
}
struct Config {
  dim3 g, b;
  size_t sh;
  cudaStream_t s;
};
thread_local std::vector<Config> configs;
}  // namespace

#define FAKE extern "C" __attribute__((visibility("default")))

// What the tests ask.
FAKE const char* fake_unordered() { return unordered.c_str(); }
FAKE void fake_forget() { unordered.clear(); }
FAKE unsigned long fake_live_bytes() {
  std::lock_guard<std::mutex> g(mu);
  unsigned long n = 0;
  for (auto& [p, b] : live) n += b;
  return n;
}
FAKE long fake_launches(const char* part) {
  std::lock_guard<std::mutex> g(mu);
  long n = 0;
  for (auto& [name, k] : launches)
    if (name.find(part) != std::string::npos) n += k;
  return n;
}

// Modules.
extern "C" void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
extern "C" void __cudaRegisterFatBinaryEnd(void**) {}
extern "C" void __cudaUnregisterFatBinary(void**) {}
extern "C" void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*,
                                       dim3*, int*) {
  kernels[host] = name;
}
extern "C" void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
extern "C" unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sh, cudaStream_t s) {
  configs.push_back({g, b, sh, s});
  return 0;
}
extern "C" cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sh, void* s) {
  const Config c = configs.back();
  configs.pop_back();
  *g = c.g, *b = c.b, *sh = c.sh, *(cudaStream_t*)s = c.s;
  return cudaSuccess;
}
extern "C" cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  launches[kernels[f]]++;
  for (const Pending& p : pending)
    if (!in_order(p.stream, s) && !p.ordered.count(s))
      unordered += kernels[f] + " beside a copy of " + std::to_string(p.bytes) + " bytes\n";
  return cudaSuccess;
}

// Memory.
extern "C" cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
extern "C" cudaError_t cudaFree(void* p) { return give_back(p); }
extern "C" cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n ? n : 1);
  std::lock_guard<std::mutex> g(mu);
  pinned[*p] = n;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> g(mu);
  pinned.erase(p);
  std::free(p);
  return cudaSuccess;
}
extern "C" cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  std::lock_guard<std::mutex> g(mu);
  wait(nullptr, seq);  // it runs in the legacy stream after what was put there
  std::memcpy(d, s, n);
  copied(nullptr, s, n, k);
  return cudaSuccess;
}
extern "C" cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  std::lock_guard<std::mutex> g(mu);
  std::memcpy(d, s, n);
  copied(st, s, n, k);
  return cudaSuccess;
}
extern "C" cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
extern "C" cudaError_t cudaMemcpyToSymbol(const void* d, const void* s, size_t n, size_t at, cudaMemcpyKind k) {
  return cudaMemcpy((char*)d + at, s, n, k);
}
extern "C" cudaError_t cudaMemcpyFromSymbol(void* d, const void* s, size_t n, size_t at, cudaMemcpyKind k) {
  return cudaMemcpy(d, (const char*)s + at, n, k);
}
extern "C" cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}
extern "C" cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  *p = nullptr;
  return cudaSuccess;
}
extern "C" cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
extern "C" cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
extern "C" cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return allocate(p, n); }
extern "C" cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give_back(p); }

// Streams and events.
extern "C" cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) {
  *s = new CUstream_st{!(flags & cudaStreamNonBlocking)};
  return cudaSuccess;
}
extern "C" cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  wait(s, seq);
  return cudaSuccess;
}
extern "C" cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::mutex> g(mu);
  pending.clear();
  return cudaSuccess;
}
extern "C" cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = new CUevent_st;
  return cudaSuccess;
}
extern "C" cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
extern "C" cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete e;
  return cudaSuccess;
}
extern "C" cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> g(mu);
  e->stream = s, e->seq = seq;
  return cudaSuccess;
}
extern "C" cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> g(mu);
  wait(e->stream, e->seq);
  return cudaSuccess;
}
extern "C" cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
extern "C" cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
extern "C" cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::mutex> g(mu);
  for (Pending& p : pending)
    if (in_order(p.stream, e->stream) && p.seq <= e->seq) p.ordered.insert(s);
  return cudaSuccess;
}
extern "C" cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
extern "C" cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(&seq);
  return cudaSuccess;
}
extern "C" cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
extern "C" cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
extern "C" cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }

// The device: one B200.
extern "C" cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
extern "C" cudaError_t cudaSetDevice(int) { return cudaSuccess; }
extern "C" cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10 : 65536;
  if (a == cudaDevAttrComputeCapabilityMinor) *v = 0;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  a->ptxVersion = a->binaryVersion = 100;
  a->maxThreadsPerBlock = 1024;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "fake"; }
