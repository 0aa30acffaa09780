// A CUDA runtime without a GPU for the library's host code: device memory is
// reserved address space of a settable capacity, copies are memcpy, launches
// are checked against the limits of a launch and counted but do not run.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
size_t capacity = (size_t)280 << 30, used = 0, largest = ~(size_t)0;
std::map<void*, size_t> blocks;
std::map<const void*, std::string> names;
std::map<const void*, int> raised;  // dynamic shared memory a kernel was given leave for
std::map<std::string, int> launches;
int refused = 0;
bool mute = false;
cudaError_t last = cudaSuccess;

cudaError_t put(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem) {
  if (g.x == 0 || g.y == 0 || g.z == 0 || g.x > 0x7fffffffu || g.y > 65535 || g.z > 65535 ||
      (size_t)b.x * b.y * b.z > 1024 || smem > 227 * 1024 || (smem > 48 * 1024 && (int)smem > raised[f]))
    return put(cudaErrorInvalidValue);
  ++launches[names.count(f) ? names[f] : std::string("?")];
  return cudaSuccess;
}
cudaError_t make(void** p) {
  *p = std::malloc(1);
  return cudaSuccess;
}
int encode_tiled(...) { return 0; }
}  // namespace

extern "C" {
// Capacity, and the largest block that is free in one piece.
void fake_reset(size_t bytes, size_t block) {
  capacity = bytes;
  largest = block;
  launches.clear();
  refused = 0;
}
size_t fake_used() { return used; }
// Whether cudaMemGetInfo fails.
void fake_mute(int on) { mute = on != 0; }
// Allocations that found no room since the reset.
int fake_refused() { return refused; }
// Launches of the kernels whose name holds part.
int fake_launches(const char* part) {
  int n = 0;
  for (const auto& l : launches)
    if (l.first.find(part) != std::string::npos) n += l.second;
  return n;
}

void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(std::malloc(8)); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(const void** k, const void* f) {
  *k = f;
  return cudaSuccess;
}
static dim3 cfg_grid, cfg_block;
static size_t cfg_smem;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void*) {
  cfg_grid = g;
  cfg_block = b;
  cfg_smem = smem;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = cfg_grid;
  *b = cfg_block;
  *smem = cfg_smem;
  *static_cast<void**>(st) = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(const void* k, dim3 g, dim3 b, void**, size_t smem, void*) { return launch(k, g, b, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  if (used + n > capacity || n > largest) {
    ++refused;
    return put(cudaErrorMemoryAllocation);
  }
  void* m = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (m == MAP_FAILED) return put(cudaErrorMemoryAllocation);
  blocks[m] = n;
  used += n;
  *p = m;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  const auto it = blocks.find(p);
  if (it == blocks.end()) return put(cudaErrorInvalidValue);
  munmap(p, it->second);
  used -= it->second;
  blocks.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  if (mute) return put(cudaErrorUnknown);
  *f = capacity > used ? capacity - used : 0;
  *t = capacity;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc3DArray(cudaArray_t* a, const cudaChannelFormatDesc*, cudaExtent, unsigned) {
  return make(reinterpret_cast<void**>(a));
}
cudaError_t cudaFreeArray(cudaArray_t) { return cudaSuccess; }
cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f) {
  return cudaChannelFormatDesc{x, y, z, w, f};
}
cudaError_t cudaCreateTextureObject(cudaTextureObject_t* t, const cudaResourceDesc*, const cudaTextureDesc*,
                                    const cudaResourceViewDesc*) {
  *t = 1;
  return cudaSuccess;
}
cudaError_t cudaDestroyTextureObject(cudaTextureObject_t) { return cudaSuccess; }

cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  switch (a) {
    case cudaDevAttrMultiProcessorCount: *v = 152; break;
    case cudaDevAttrMaxSharedMemoryPerMultiprocessor: *v = 228 * 1024; break;
    case cudaDevAttrReservedSharedMemoryPerBlock: *v = 1024; break;
    case cudaDevAttrMaxRegistersPerMultiprocessor: *v = 65536; break;
    case cudaDevAttrMaxThreadsPerMultiProcessor: *v = 2048; break;
    case cudaDevAttrL2CacheSize: *v = 129 << 20; break;
    default: return put(cudaErrorInvalidValue);
  }
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  a->numRegs = 64;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > 227 * 1024) return put(cudaErrorInvalidValue);
    raised[f] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
  *f = reinterpret_cast<void*>(&encode_tiled);
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : (e == cudaSuccess ? "no error" : "error");
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}

cudaError_t cudaEventCreate(cudaEvent_t* e) { return make(reinterpret_cast<void**>(e)); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make(reinterpret_cast<void**>(e)); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make(reinterpret_cast<void**>(s)); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return make(reinterpret_cast<void**>(g)); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  return make(reinterpret_cast<void**>(x));
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  std::free(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  std::free(x);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
}
