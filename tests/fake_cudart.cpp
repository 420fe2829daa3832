// Stand-in for the CUDA runtime, preloaded by tests of the library's host side
// on machines without a GPU: device memory is host memory, copies and fills
// happen at once, kernels do nothing.  Tests set what shall fail and read what
// was asked for through the fake_* functions.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
size_t g_limit = ~(size_t)0, g_largest = ~(size_t)0, g_held = 0;
std::map<void *, size_t> g_mem;
struct Fill {
  void *at;
  size_t bytes;
};
std::vector<Fill> g_fills;
int g_graphs = 0, g_graph_launches = 0, g_launches = 0, g_coop = 0;
bool g_capturing = false;
std::map<const void *, const char *> g_names;
std::string g_ran;
cudaError_t g_last = cudaSuccess;
cudaError_t err(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
cudaError_t launched(const void *kernel) {
  if (!g_capturing) ++g_launches;
  g_ran += std::string(g_names.count(kernel) ? g_names[kernel] : "?") + "\n";
  return cudaSuccess;
}
// the stream that cannot be captured
bool legacy(cudaStream_t st) { return st == nullptr || st == cudaStreamLegacy; }
void *token() {
  static char t;
  return &t;
}
}  // namespace

extern "C" {
// device memory that may be held at a time
void fake_limit(size_t bytes) { g_limit = bytes; }
// and in one piece
void fake_largest(size_t bytes) { g_largest = bytes; }
size_t fake_held() { return g_held; }
// the latest fill of `bytes` bytes
void *fake_filled(size_t bytes) {
  for (size_t i = g_fills.size(); i-- > 0;)
    if (g_fills[i].bytes == bytes) return g_fills[i].at;
  return nullptr;
}
int fake_graphs() { return g_graphs; }
int fake_graph_launches() { return g_graph_launches; }
int fake_launches() { return g_launches; }
int fake_cooperative() { return g_coop; }
// (mangled) names of the kernels launched since the last call, a line each
const char *fake_ran() {
  static std::string r;
  r.swap(g_ran);
  g_ran.clear();
  return r.c_str();
}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *,
                            dim3 *, int *) {
  g_names[host] = name;
}

cudaError_t cudaMalloc(void **p, size_t n) {
  if (n > g_largest || n > g_limit || g_held > g_limit - n) return err(cudaErrorMemoryAllocation);
  *p = aligned_alloc(512, (n + 511) / 512 * 512);
  if (!*p) return err(cudaErrorMemoryAllocation);
  memset(*p, 0xff, n);
  g_mem[*p] = n;
  g_held += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  const auto it = g_mem.find(p);
  if (it == g_mem.end()) return err(cudaErrorInvalidValue);
  g_held -= it->second;
  g_mem.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = malloc(n)) ? cudaSuccess : err(cudaErrorMemoryAllocation); }
cudaError_t cudaFreeHost(void *p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t i = 0; i < h; ++i) memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  g_fills.push_back({d, n});
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1);
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
  memset(a, 0, sizeof *a);
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaLaunchKernel(const void *k, dim3, dim3, void **, size_t, cudaStream_t) { return launched(k); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *k, void **) { return launched(k); }
cudaError_t cudaLaunchCooperativeKernel(const void *k, dim3, dim3, void **, size_t, cudaStream_t) {
  ++g_coop;
  return launched(k);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)token();
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return g_capturing ? err(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)token();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) {
  *t = 0.f;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t st, cudaStreamCaptureMode) {
  if (legacy(st)) return err(cudaErrorStreamCaptureUnsupported);
  g_capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  g_capturing = false;
  *g = (cudaGraph_t)token();
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  ++g_graphs;
  *x = (cudaGraphExec_t)token();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  ++g_graph_launches;
  return cudaSuccess;
}
}
