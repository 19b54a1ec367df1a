// A CUDA runtime for tests of the engine's host side on the CPU: device memory is host memory, kernels do nothing, streams and
// events are names.  Preloaded in front of the real one.  It keeps count of what the engine asks for, refuses memory when it is
// told to, and checks that every copy and fill stays inside one live allocation.
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <pthread.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>

namespace {
std::recursive_mutex mu;
std::map<const char*, size_t> live;               // device allocations
std::map<const void*, std::string> names;         // kernels by host stub
std::map<std::string, long> launched, value;      // `value`: what a test sets and reads (fake_set, fake_get)
thread_local cudaError_t pending = cudaSuccess;   // what cudaGetLastError returns
thread_local int device = 0;
struct Call { dim3 grid, block; size_t smem; void* stream; };
thread_local Call call;

const pthread_t main_thread = pthread_self();

long& v(const char* key) { return value[key]; }

// Whether a request for memory is refused: beyond `limit` bytes in all, as the `refuse_one`-th from now on, or when the countdown
// `refuse_after` has run out.
bool refused(size_t bytes) {
  if (v("limit") && v("used") + (long)bytes > v("limit")) return true;
  if (v("refuse_one") && --v("refuse_one") == 0) return true;
  return v("refusing") && v("refuse_after")-- <= 0;
}
bool inside(const void* p, size_t bytes) {
  auto it = live.upper_bound(static_cast<const char*>(p));
  if (it == live.begin()) return false;
  --it;
  return static_cast<const char*>(p) + bytes <= it->first + it->second;
}
// `bytes` of device memory from p on are touched
bool touch(const void* p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (!bytes || inside(p, bytes)) return true;
  ++v("violations");
  return false;
}
cudaError_t copy(void* d, const void* s, size_t bytes, cudaMemcpyKind kind) {
  const bool ok_d = kind == cudaMemcpyDeviceToHost || touch(d, bytes), ok_s = kind == cudaMemcpyHostToDevice || touch(s, bytes);
  if (ok_d && ok_s && bytes) std::memmove(d, s, bytes);
  return cudaSuccess;
}
cudaError_t launch(const void* f, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (!s) ++v("legacy");
  if (v("throw_launch") && --v("throw_launch") == 0) throw std::bad_alloc();      // (as `throw_at`)
  ++launched[names[f]];
  if (v("unordered")) ++v("races");     // a fill of the legacy stream, which this launch does not wait for, is under way
  return cudaSuccess;
}
CUresult encode_tiled(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void* p, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                      const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  touch(p, 1);
  return CUDA_SUCCESS;
}
template <class T>
cudaError_t fresh(T* out) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (refused(0)) return pending = cudaErrorMemoryAllocation;
  *out = reinterpret_cast<T>(std::malloc(1));
  return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_set(const char* key, long x) { std::lock_guard<std::recursive_mutex> lock(mu); value[key] = x; }
long fake_get(const char* key) { std::lock_guard<std::recursive_mutex> lock(mu); return value[key]; }
// Launches of kernels whose (mangled) name contains `part`.
long fake_launches(const char* part) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  long n = 0;
  for (auto& k : launched) if (k.first.find(part) != std::string::npos) n += k.second;
  return n;
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  ++v(pthread_equal(pthread_self(), main_thread) ? "requests" : "requests_beside");
  if (refused(bytes)) return pending = cudaErrorMemoryAllocation;
  *p = std::calloc(bytes ? bytes : 1, 1);
  live[static_cast<char*>(*p)] = bytes;
  v("used") += (long)bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (!p) return cudaSuccess;
  auto it = live.find(static_cast<char*>(p));
  if (it == live.end()) { ++v("violations"); return cudaErrorInvalidValue; }
  v("used") -= (long)it->second;
  live.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  ++v(pthread_equal(pthread_self(), main_thread) ? "requests" : "requests_beside");
  if (refused(0)) return pending = cudaErrorMemoryAllocation;
  *p = std::calloc(bytes ? bytes : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) { return cudaHostAlloc(p, bytes, 0); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  *total = v("limit") ? (size_t)v("limit") : (size_t)180 << 30;
  *free_bytes = *total - (size_t)v("used");
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int c, size_t bytes) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (touch(p, bytes)) std::memset(p, c, bytes);
  v("unordered") = 1;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int c, size_t bytes, cudaStream_t) {
  if (touch(p, bytes) && bytes) std::memset(p, c, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemset2DAsync(void* p, size_t pitch, int c, size_t width, size_t height, cudaStream_t) {
  if (height && touch(p, pitch * (height - 1) + width))
    for (size_t y = 0; y < height; ++y) std::memset(static_cast<char*>(p) + y * pitch, c, width);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { fake_set("unordered", 0); return copy(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  {
    std::lock_guard<std::recursive_mutex> lock(mu);
    if (v("throw_at") && --v("throw_at") == 0) throw std::bad_alloc();      // (stands for the engine's own host memory)
  }
  return copy(d, s, n, k);
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k) {
  for (size_t y = 0; y < h; ++y) copy(static_cast<char*>(d) + y * dp, static_cast<const char*>(s) + y * sp, w, k);
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> lock(mu);
  v("unordered") = 0;
  ++v("device_waits");
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* out, cudaDeviceAttr a, int) {
  *out = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrL2CacheSize ? 126 << 20 : 0;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  ++v("streams");
  return fresh(s);
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return fresh(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return fresh(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = pending; pending = cudaSuccess; return e; }
const char* cudaGetErrorName(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "cudaErrorMemoryAllocation" : "error"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 74; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *f = reinterpret_cast<void*>(&encode_tiled);
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) { return launch(f, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->stream); }

void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, void*, void*, void*, void*, int*) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  names[stub] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) { call = Call{g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = call.grid; *b = call.block; *smem = call.smem; *static_cast<void**>(s) = call.stream;
  return cudaSuccess;
}
}
