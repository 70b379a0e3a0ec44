// A CUDA runtime for the library's host code on a machine without a GPU: two devices of 148 SMs whose memory is the host's and whose kernels do nothing.  It keeps
// what belongs to one device apart (allocations, kernels' limits of dynamic shared memory), refuses the launches that a device would
// refuse for their shared memory, and writes down every other.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {
constexpr int DEVICES = 2;
constexpr size_t DEFAULT_SMEM = 48 * 1024, MOST_SMEM = 227 * 1024;
std::recursive_mutex mu;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
std::map<const void*, std::string>& names() { static std::map<const void*, std::string> m; return m; }
std::map<std::pair<const void*, int>, size_t> limits;
std::map<std::pair<const void*, int>, int> shares;      // of an SM's L1 that a kernel asks for as shared memory, in percent
std::map<void*, std::pair<int, size_t>> blocks;
size_t held[DEVICES];
int attributes_to_refuse = 0, last_share = cudaSharedmemCarveoutDefault;
std::string launches;
struct Call { dim3 grid, block; size_t smem; cudaStream_t stream; };
thread_local std::vector<Call> calls;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem) {
  std::lock_guard<std::recursive_mutex> g(mu);
  const auto it = limits.find({f, device});
  if (smem > (it == limits.end() ? DEFAULT_SMEM : it->second) || grid.x == 0 || block.x * block.y * block.z > 1024) return done(cudaErrorInvalidValue);
  const auto share = shares.find({f, device});
  last_share = share == shares.end() ? cudaSharedmemCarveoutDefault : share->second;
  launches += std::to_string(device) + " " + names()[f] + " " + std::to_string(grid.x * grid.y * grid.z) + "\n";
  return cudaSuccess;
}
CUresult encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  memset(m, 0, sizeof(*m));
  return CUDA_SUCCESS;
}
cudaError_t take(void** p, size_t n) {
  std::lock_guard<std::recursive_mutex> g(mu);
  *p = aligned_alloc(256, (n + 255) / 256 * 256 + 256);
  if (!*p) return done(cudaErrorMemoryAllocation);
  blocks[*p] = {device, n};
  held[device] += n;
  return cudaSuccess;
}
cudaError_t give(void* p) {
  std::lock_guard<std::recursive_mutex> g(mu);
  const auto it = blocks.find(p);
  if (it != blocks.end()) {
    held[it->second.first] -= it->second.second;
    blocks.erase(it);
    free(p);
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- what a test asks and sets ----
const char* fake_launches() { return launches.c_str(); }      // "device kernel blocks" per line, since the last fake_clear
void fake_clear() { launches.clear(); }
int fake_share() { return last_share; }                        // the last launch's
size_t fake_held(int dev) { return held[dev]; }
void fake_refuse_attributes(int n) { attributes_to_refuse = n; }

// ---- the runtime ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names()[host] = name; }
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) { calls.push_back({grid, block, smem, stream}); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  const Call c = calls.back();
  calls.pop_back();
  *grid = c.grid; *block = c.block; *smem = c.smem; *static_cast<cudaStream_t*>(stream) = c.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) { return launch(f, grid, block, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes); }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::recursive_mutex> g(mu);
  if (attributes_to_refuse > 0) { --attributes_to_refuse; return done(cudaErrorInvalidValue); }
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) limits[{f, device}] = v;
  if (a == cudaFuncAttributePreferredSharedMemoryCarveout) shares[{f, device}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t smem, unsigned) { *n = smem <= MOST_SMEM ? 1 : 0; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= DEVICES) return done(cudaErrorInvalidDevice);
  device = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *fn = reinterpret_cast<void*>(&encode);
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  const cudaError_t e = take(p, n);
  if (e == cudaSuccess) memset(*p, 0, n);
  return e;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = size_t(180) << 30; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memmove(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
  for (size_t i = 0; i < h; ++i) memmove(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy2D(d, dp, s, sp, w, h, k); }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = reinterpret_cast<cudaGraph_t>(8); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = reinterpret_cast<cudaGraphExec_t>(8); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(8); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
}
