// A CUDA runtime without a GPU, for tests of the library's host code: it is
// linked with the library's object files in place of the real one. Devices are
// numbers, device memory is host memory that kernels never touch, launches are
// written to a log. Launches are checked as a device checks them: dynamic
// shared memory beyond 48 KB needs the kernel's limit raised on the device that
// is current.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>

namespace {

int g_devices = 1, g_current = 0;
size_t g_free = size_t(64) << 30, g_largest = ~size_t(0);
cudaError_t g_last = cudaSuccess;
std::string g_log;
std::map<const void*, std::string> g_names;
std::map<std::pair<int, const void*>, size_t> g_limits;
std::map<void*, size_t> g_blocks;
std::set<void*> g_capturing;
size_t g_next = 0x1000;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_config;

void line(const char* fmt, auto... args) {
  char buf[1024];
  std::snprintf(buf, sizeof(buf), fmt, args...);
  g_log += buf;
  g_log += '\n';
}
cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  size_t limit = 48 * 1024;
  const auto it = g_limits.find({g_current, f});
  if (it != g_limits.end() && it->second > limit) limit = it->second;
  if (smem > limit || !grid.x || !grid.y || !grid.z || grid.y > 65535 || grid.z > 65535 || block.x * block.y * block.z > 1024)
    return set(cudaErrorInvalidValue);
  line("launch device=%d stream=%p grid=%u,%u,%u block=%u smem=%zu %s", g_current, (void*)s, grid.x, grid.y, grid.z,
       block.x, smem, g_names[f].c_str());
  return cudaSuccess;
}
void* handle() { return reinterpret_cast<void*>(g_next += 16); }

int encode_tiled(...) { return 0; }

}  // namespace

extern "C" {

// ---- what tests set and read ----
void fake_devices(int n) { g_devices = n; }
void fake_memory(size_t bytes) { g_free = bytes; }
void fake_largest_block(size_t bytes) { g_largest = bytes; }
void fake_capturing(void* stream, int on) {
  if (on)
    g_capturing.insert(stream);
  else
    g_capturing.erase(stream);
}
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }

// ---- kernels ----
void** __cudaRegisterFatBinary(void* p) { return static_cast<void**>(p); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
  g_config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *static_cast<cudaStream_t*>(stream) = g_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* out, const void* f) {
  *out = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t s) {
  return launch(f, grid, block, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int value) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || value < 0 || value > 227 * 1024)
    return set(cudaErrorInvalidValue);
  g_limits[{g_current, f}] = size_t(value);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t smem, unsigned) {
  *n = smem ? int(227 * 1024 / smem) : 2;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  const auto it = g_limits.find({g_current, f});
  if (c->dynamicSmemBytes > 48 * 1024 && (it == g_limits.end() || it->second < c->dynamicSmemBytes))
    return set(cudaErrorInvalidValue);
  *n = 76;
  return cudaSuccess;
}

// ---- devices and errors ----
cudaError_t cudaGetDeviceCount(int* n) {
  *n = g_devices;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= g_devices) return set(cudaErrorInvalidDevice);
  g_current = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = g_current;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return std::exchange(g_last, cudaSuccess); }
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaErrorInvalidValue ? "invalid argument" : "error";
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** fn, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult* r) {
  *fn = reinterpret_cast<void*>(encode_tiled);
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = handle();
  return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t bytes) {
  if (bytes > g_free || bytes > g_largest) {
    line("malloc %zu failed", bytes);
    return set(cudaErrorMemoryAllocation);
  }
  *p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (*p == MAP_FAILED) return set(cudaErrorMemoryAllocation);
  g_blocks[*p] = bytes;
  g_free -= bytes;
  line("malloc %zu", bytes);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  const auto it = g_blocks.find(p);
  if (it == g_blocks.end()) return p ? set(cudaErrorInvalidValue) : cudaSuccess;
  munmap(p, it->second);
  g_free += it->second;
  line("free %zu", it->second);
  g_blocks.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_b, size_t* total) {
  *free_b = g_free;
  *total = size_t(280) << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  line("memset stream=%p %zu", (void*)s, n);
  std::memset(p, v, n);
  return cudaSuccess;
}

// ---- streams, events, graphs ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = static_cast<cudaStream_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  line("synchronize stream=%p", (void*)s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  line("wait stream=%p event=%p", (void*)s, (void*)e);
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* v) {
  *v = g_capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = static_cast<cudaGraph_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = static_cast<cudaGraphExec_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = static_cast<cudaEvent_t>(handle());
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  line("record stream=%p event=%p", (void*)s, (void*)e);
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.f;
  return cudaSuccess;
}

}  // extern "C"
