// Test harness (tests only): stands in for the CUDA runtime on a machine
// without a GPU (LD_PRELOAD). Device memory is host memory of a settable
// amount, beyond which cudaMalloc returns cudaErrorMemoryAllocation; kernels do
// nothing. tests/test_memory_limit.py runs the library's host side on it to see
// which calls still succeed when device memory is short, tests/test_host_state.py
// what the host side captures and launches.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>

static std::map<void*, size_t> g_blocks;
static size_t g_used = 0, g_peak = 0, g_limit = ~size_t(0) / 2;
static thread_local cudaError_t g_last = cudaSuccess;
static int g_captures = 0;       // stream captures begun
static unsigned g_cluster = 16;  // largest cluster that can be placed

static cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}

extern "C" {
void fake_limit(size_t bytes) { g_limit = bytes; }
void fake_max_cluster(unsigned n) { g_cluster = n; }
int fake_captures() { return g_captures; }
size_t fake_used() { return g_used; }
size_t fake_peak() {
  const size_t p = g_peak;
  g_peak = g_used;
  return p;
}

cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_used + n > g_limit) return set(cudaErrorMemoryAllocation);
  *p = std::calloc(1, n ? n : 1);
  g_blocks[*p] = n;
  g_used += n;
  if (g_used > g_peak) g_peak = g_used;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  auto it = g_blocks.find(p);
  if (it == g_blocks.end()) return set(cudaErrorInvalidValue);
  g_used -= it->second;
  g_blocks.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = g_limit - g_used;
  *t = g_limit;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = std::calloc(1, n ? n : 1), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memmove(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return std::memmove(d, s, n), cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
static bool placeable(const cudaLaunchConfig_t* c) {
  for (unsigned k = 0; k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributeClusterDimension && c->attrs[k].val.clusterDim.x > g_cluster) return false;
  return true;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
  return placeable(c) ? cudaSuccess : set(cudaErrorInvalidClusterSize);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  return *n = placeable(c) ? 1 : 0, cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return ++g_captures, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  return *g = reinterpret_cast<cudaGraph_t>(16), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  return *e = reinterpret_cast<cudaGraphExec_t>(16), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(16), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = reinterpret_cast<cudaEvent_t>(16), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.0f, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
}
