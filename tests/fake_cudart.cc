// A CUDA runtime without a GPU, for host-side tests: the library's own objects are linked against it, so that a
// test can let an allocation fail and look at what the library allocates, frees, waits for and launches.
// Device memory is host memory that is never touched by a kernel: kernels do not run, their launches are recorded.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {
std::map<const void*, std::string> kernels;     // host stub -> kernel name
std::map<void*, size_t> device, pinned;         // live allocations
size_t fail_above = SIZE_MAX;                   // a larger allocation fails ...
long fail_nth = -1;                             // ... and so does the n-th from now (0: the next)
std::vector<std::string> events;                // "malloc 123", "free", "pin 123", "unpin", "chunk", "sync", "launch name"
std::string watch_name;
int watch_arg = -1;
void* watched = nullptr;
dim3 push_grid, push_block;
size_t push_smem;
cudaStream_t push_stream;

const size_t TOUCH = 16u << 20;                 // larger memsets and copies are left out

bool refused(size_t bytes)
{
  if (bytes > fail_above) return true;
  return fail_nth >= 0 && fail_nth-- == 0;
}
void* map(size_t bytes)
{
  void* p = mmap(nullptr, bytes ? bytes : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  return p == MAP_FAILED ? nullptr : p;
}
cudaError_t launch(const void* f, void** args)
{
  const auto k = kernels.find(f);
  const std::string name = k == kernels.end() ? "?" : k->second;
  events.push_back("launch " + name);
  if (watch_arg >= 0 && name.find(watch_name) != std::string::npos) watched = *static_cast<void**>(args[watch_arg]);
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- for the tests
void fake_fail_above(size_t bytes) { fail_above = bytes; }
void fake_fail_nth(long n) { fail_nth = n; }
void fake_clear() { events.clear(); }
int fake_count(const char* what)   // events that begin so
{
  int n = 0;
  for (const auto& e : events) n += e.compare(0, strlen(what), what) == 0;
  return n;
}
int fake_first(const char* what)   // position of the first such event, -1 if there is none
{
  for (size_t k = 0; k < events.size(); ++k)
    if (events[k].compare(0, strlen(what), what) == 0) return (int)k;
  return -1;
}
size_t fake_device_bytes()
{
  size_t n = 0;
  for (const auto& a : device) n += a.second;
  return n;
}
size_t fake_device_allocations() { return device.size(); }
size_t fake_pinned_allocations() { return pinned.size(); }
void fake_watch(const char* name, int arg) { watch_name = name; watch_arg = arg; watched = nullptr; }
// the last watched argument (a pointer), and whether it lies in `bytes` live device bytes
void* fake_watched() { return watched; }
int fake_is_device(void* p, size_t bytes)
{
  for (const auto& a : device) {
    const char *b = static_cast<char*>(a.first), *q = static_cast<char*>(p);
    if (q >= b && q + bytes <= b + a.second) return 1;
  }
  return 0;
}

// ---- what the compiler's stubs call
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*)
{
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st* q)
{
  push_grid = g; push_block = b; push_smem = s; push_stream = q;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* q)
{
  *g = push_grid; *b = push_block; *s = push_smem; *static_cast<cudaStream_t*>(q) = push_stream;
  return cudaSuccess;
}

// ---- the runtime
cudaError_t cudaMalloc(void** p, size_t n)
{
  if (refused(n)) return cudaErrorMemoryAllocation;   // *p is left alone
  *p = map(n);
  device[*p] = n;
  events.push_back("malloc " + std::to_string(n));
  return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
  const auto a = device.find(p);
  if (a == device.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  munmap(p, a->second ? a->second : 1);
  device.erase(a);
  events.push_back("free");
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
  if (refused(n)) return cudaErrorMemoryAllocation;
  if (pinned.empty()) events.push_back("chunk");   // the driver maps one for the first and keeps it to the last
  *p = map(n);
  pinned[*p] = n;
  events.push_back("pin " + std::to_string(n));
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
  const auto a = pinned.find(p);
  if (a == pinned.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  munmap(p, a->second ? a->second : 1);
  pinned.erase(a);
  events.push_back("unpin");
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n)
{
  if (!p) return cudaErrorInvalidValue;
  if (n <= TOUCH) memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
  if (!d || !s) return cudaErrorInvalidValue;
  if (n <= TOUCH) memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) { return launch(f, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { return launch(f, args); }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { events.push_back("sync"); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(0x100); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(0x200); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
}
