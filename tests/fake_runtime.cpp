// A CUDA runtime and cuFFT without a device, for CPU tests of the library's host side: the
// library's own objects are linked with this file instead of the CUDA libraries
// (tests/test_engine_host.py).  Device memory is address space that reads as zeros and is only
// written by copies; kernels are counted by name and not run.  fake_*: what the tests set and
// ask for.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cufft.h>
#include <sys/mman.h>

#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

namespace {
struct Block {
  size_t bytes;
  bool pool;
};
std::map<void*, Block> g_blocks;
std::map<const void*, std::string>& names() {  // filled while the library is loaded
  static std::map<const void*, std::string> m;
  return m;
}
std::map<std::string, int> g_launches;
size_t g_live = 0, g_limit = 0;
int g_capturing = 0, g_capture_broken = 0, g_symbol = 0, g_symbol_at = -1, g_symbol_reads = 0;
int g_pool_allocs = 0, g_launched = 0;
cudaStreamCaptureMode g_mode = cudaStreamCaptureModeGlobal;
std::vector<std::pair<cudaHostFn_t, void*>> g_user_objects;

// calls that a capture in global mode does not allow
cudaError_t unsafe_call() {
  if (!g_capturing || g_mode == cudaStreamCaptureModeRelaxed) return cudaSuccess;
  g_capture_broken = 1;
  return cudaErrorStreamCaptureUnsupported;
}
cudaError_t take(void** p, size_t n, bool pool) {
  *p = nullptr;
  if (g_limit && g_live + n > g_limit) return cudaErrorMemoryAllocation;
  void* m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE,
                 MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
  g_blocks[m] = Block{n, pool};
  g_live += n;
  *p = m;
  return cudaSuccess;
}
cudaError_t give(void* p) {
  if (!p) return cudaSuccess;
  auto it = g_blocks.find(p);
  if (it == g_blocks.end()) return cudaErrorInvalidValue;
  munmap(p, it->second.bytes ? it->second.bytes : 1);
  g_live -= it->second.bytes;
  g_blocks.erase(it);
  return cudaSuccess;
}
CUresult encode_tiled(...) { return CUDA_SUCCESS; }
cudaError_t launched(const void* f) {
  ++g_launched;
  ++g_launches[names().count(f) ? names()[f] : std::string("?")];
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ------------------------------------------------------------------ for the tests
long long fake_live_bytes() { return (long long)g_live; }
void fake_set_limit(long long bytes) { g_limit = (size_t)bytes; }  // 0: no limit
void fake_set_capturing(int on) {
  g_capturing = on;
  g_capture_broken = 0;
}
int fake_capture_broken() { return g_capture_broken; }
// every captured graph goes, and the user objects they held with them
void fake_destroy_graphs() {
  std::vector<std::pair<cudaHostFn_t, void*>> objects;
  objects.swap(g_user_objects);
  for (auto& o : objects) o.first(o.second);
}
// device variables read as `value`, from their `at`-th read on
void fake_set_symbol(int value, int at) {
  g_symbol = value;
  g_symbol_at = at;
  g_symbol_reads = 0;
}
int fake_symbol_reads() { return g_symbol_reads; }
void fake_reset_counts() {
  g_launches.clear();
  g_launched = g_pool_allocs = 0;
}
int fake_pool_allocs() { return g_pool_allocs; }
// launches of the kernels whose mangled name contains `part`
int fake_launches(const char* part) {
  int n = 0;
  for (const auto& kv : g_launches)
    if (kv.first.find(part) != std::string::npos) n += kv.second;
  return n;
}

// ------------------------------------------------------------------ kernels
void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t) {
  return launched((const void*)k);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) {
  return launched(f);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
  *n = 2;
  return cudaSuccess;
}

// ------------------------------------------------------------------ memory
cudaError_t cudaMalloc(void** p, size_t n) {
  const cudaError_t e = unsafe_call();
  return e == cudaSuccess ? take(p, n, false) : e;
}
cudaError_t cudaFree(void* p) {
  const cudaError_t e = unsafe_call();
  return e == cudaSuccess ? give(p) : e;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
  ++g_pool_allocs;
  return take(p, n, true);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset2DAsync(void*, size_t, int, size_t, size_t, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbolAsync(void* d, const void*, size_t n, size_t, cudaMemcpyKind,
                                      cudaStream_t) {
  const int v = g_symbol_at >= 0 && g_symbol_reads >= g_symbol_at ? g_symbol : 0;
  ++g_symbol_reads;
  memcpy(d, &v, n < sizeof(v) ? n : sizeof(v));
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* d, const void* s, size_t n, size_t at, cudaMemcpyKind k) {
  return cudaMemcpyFromSymbolAsync(d, s, n, at, k, nullptr);
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) {
  g_symbol_at = -1;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static char area[64];
  *p = area;
  return cudaSuccess;
}

// ------------------------------------------------------------------ device, streams, events
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount                    ? 152
       : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472
       : a == cudaDevAttrReservedSharedMemoryPerBlock     ? 1024
                                                           : 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
  *f = (void*)encode_tiled;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus* s,
                                     unsigned long long*, cudaGraph_t* g, const cudaGraphNode_t**,
                                     const cudaGraphEdgeData**, size_t*) {
  if (g) *g = (cudaGraph_t)1;
  return cudaStreamIsCapturing(nullptr, s);
}
cudaError_t cudaUserObjectCreate(cudaUserObject_t* o, void* p, cudaHostFn_t f, unsigned, unsigned) {
  g_user_objects.emplace_back(f, p);
  *o = (cudaUserObject_t)1;
  return cudaSuccess;
}
cudaError_t cudaGraphRetainUserObject(cudaGraph_t, cudaUserObject_t, unsigned, unsigned) {
  return cudaSuccess;
}
cudaError_t cudaUserObjectRelease(cudaUserObject_t, unsigned) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
  std::swap(*m, g_mode);
  return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) {
  *id = (unsigned long long)s;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)1;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }

// ------------------------------------------------------------------ cuFFT
cufftResult cufftCreate(cufftHandle* h) {
  *h = 1;
  return CUFFT_SUCCESS;
}
cufftResult cufftDestroy(cufftHandle) { return CUFFT_SUCCESS; }
cufftResult cufftPlan3d(cufftHandle* h, int, int, int, cufftType) { return cufftCreate(h); }
cufftResult cufftMakePlan3d(cufftHandle, int, int, int, cufftType, size_t* ws) {
  *ws = 1 << 20;
  return CUFFT_SUCCESS;
}
cufftResult cufftMakePlanMany(cufftHandle, int, int*, int*, int, int, int*, int, int, cufftType, int,
                              size_t* ws) {
  *ws = 1 << 20;
  return CUFFT_SUCCESS;
}
cufftResult cufftMakePlanMany64(cufftHandle, int, long long int*, long long int*, long long int,
                                long long int, long long int*, long long int, long long int,
                                cufftType, long long int, size_t* ws) {
  *ws = 1 << 20;
  return CUFFT_SUCCESS;
}
cufftResult cufftSetAutoAllocation(cufftHandle, int) { return CUFFT_SUCCESS; }
cufftResult cufftSetWorkArea(cufftHandle, void*) { return CUFFT_SUCCESS; }
cufftResult cufftSetStream(cufftHandle, cudaStream_t) { return CUFFT_SUCCESS; }
cufftResult cufftExecR2C(cufftHandle, cufftReal*, cufftComplex*) { return CUFFT_SUCCESS; }
cufftResult cufftExecC2R(cufftHandle, cufftComplex*, cufftReal*) { return CUFFT_SUCCESS; }
cufftResult cufftExecZ2D(cufftHandle, cufftDoubleComplex*, cufftDoubleReal*) {
  return CUFFT_SUCCESS;
}
}
