// A stand-in for the CUDA runtime on a machine without a GPU, preloaded in front of it: two
// devices of 152 SMs, memory from the host's heap, no kernel runs. What the library asks for
// is checked and written down: a launch whose dynamic shared memory is beyond 48 KB and
// beyond what the kernel was opted in for on the current device is refused, as by the real
// runtime, and every accepted launch is logged with its kernel, grid, block and shared memory.
#include <cuda_runtime_api.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>

namespace {
int device = 0;
std::map<const void*, std::string> name;                    // host stub -> kernel
std::map<std::pair<int, const void*>, size_t> opted;        // (device, stub) -> opt-in
std::string launches;
std::map<void*, size_t> held;  // device memory
bool capturing = false;
long mallocs_left = -1;        // the device's memory is full after so many more (-1: never)
struct Config {
  dim3 grid, block;
  size_t smem;
  void* stream;
} pushed;

cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem) {
  const auto it = opted.find({device, f});
  const size_t most = it == opted.end() ? 48 * 1024 : it->second;
  if (smem > 48 * 1024 && smem > most) return cudaErrorInvalidValue;
  if (!g.x || !g.y || !g.z || g.y > 65535 || g.z > 65535 || !b.x || b.x * b.y * b.z > 1024)
    return cudaErrorInvalidConfiguration;
  launches += name[f] + " " + std::to_string(g.x) + " " + std::to_string(g.y) + " " + std::to_string(g.z) + " " +
              std::to_string(b.x) + " " + std::to_string(b.y) + " " + std::to_string(smem) + "\n";
  return cudaSuccess;
}
CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
void* handle() { return calloc(1, 8); }
cudaError_t last = cudaSuccess;
}  // namespace

extern "C" {
const char* fake_launches() { return launches.c_str(); }
void fake_mallocs_left(long n) { mallocs_left = n; }
void fake_clear() { launches.clear(); }
size_t fake_held() {
  size_t n = 0;
  for (const auto& m : held) n += m.second;
  return n;
}
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }

void** __cudaRegisterFatBinary(void*) { return (void**)handle(); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* kernel, int, void*, void*, void*, void*, int*) {
  name[stub] = kernel;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) {
  pushed = Config{g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = pushed.grid; *b = pushed.block; *smem = pushed.smem;
  *(void**)s = pushed.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* stub) { *k = (cudaKernel_t)stub; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
  const cudaError_t e = launch((const void*)k, g, b, smem);
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : "error"; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > 227 * 1024) return cudaErrorInvalidValue;
    opted[{device, f}] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
// blocks an SM by the sub-step kernels' launch bounds, else by 128 registers a thread and the
// shared memory; clusters by SMs
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t smem,
                                                                   unsigned) {
  const std::string& k = name[f];
  const auto has = [&](const char* s) { return k.find(s) != std::string::npos; };
  if (has("k_spg_p2")) *n = has("k_spg_p2_ene") || has("Li5E") ? 5 : has("IdL") ? 2 : 4;
  else *n = std::min(512 / threads, (int)(228 * 1024 / (smem + 4096)));
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  *n = 128 / (int)c->attrs[0].val.clusterDim.x;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *f = (void*)encode;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) {
  if (capturing) return last = cudaErrorStreamCaptureUnsupported;
  if (mallocs_left == 0) return last = cudaErrorMemoryAllocation;
  if (mallocs_left > 0) --mallocs_left;
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  held[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  held.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = calloc(1, 1 << 20); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)handle(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
// a captured launch is logged like any other, its graph's launch as "graph"
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  *g = (cudaGraph_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = (cudaGraphExec_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  launches += "graph 0 0 0 0 0 0\n";
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)handle(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)handle(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
// every interval a little shorter than the one before
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  static int n = 0;
  *ms = 100.0f / (float)(++n + 100);
  return cudaSuccess;
}
}
