// A CUDA runtime in host memory for testing the library's host code without a GPU: allocations are
// calloc'd, copies run at once, kernels do not run.  A test can make the n-th allocation or the
// launch of a named kernel fail, and read how many launches, captures and graph launches there were.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

static std::map<const void *, std::string> &names() {
  static std::map<const void *, std::string> n;
  return n;
}
static cudaError_t last_error = cudaSuccess;
static long fail_malloc = 0, n_malloc = 0, n_clear_bytes = 0, n_bytes = 0, max_bytes = 0;
static std::map<void *, size_t> sizes;
static std::string fail_kernel;
static std::map<std::string, long> launched;
static long n_captures = 0, n_graph_launches = 0;
static bool capturing = false;

static cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last_error = e;
  return e;
}

extern "C" {
// ---- control of the tests
void fake_reset() {
  fail_malloc = max_bytes = n_malloc = n_clear_bytes = n_captures = n_graph_launches = 0;
  fail_kernel.clear();
  launched.clear();
  last_error = cudaSuccess;
}
void fake_fail_malloc(long nth) { fail_malloc = nth; }  // the nth allocation from now on and all after it (0: none)
void fake_limit(long bytes) { max_bytes = bytes; }  // allocations past this total fail (0: none)
long fake_allocated() { return n_bytes; }
void fake_fail_kernel(const char *name) { fail_kernel = name; }
long fake_launches(const char *name) {
  long n = 0;
  for (auto &l : launched) if (l.first.find(name) != std::string::npos) n += l.second;
  return n;
}
long fake_mallocs() { return n_malloc; }
long fake_cleared_bytes() { return n_clear_bytes; }
long fake_captures() { return n_captures; }
long fake_graph_launches() { return n_graph_launches; }

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n) {
  n_malloc++;
  *p = nullptr;
  if (fail_malloc && --fail_malloc <= 0) { fail_malloc = 1; return done(cudaErrorMemoryAllocation); }
  if (max_bytes && n_bytes + (long)n > max_bytes) return done(cudaErrorMemoryAllocation);
  *p = calloc(n ? n : 1, 1);
  sizes[*p] = n;
  n_bytes += (long)n;
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) {
  auto it = sizes.find(p);
  if (it != sizes.end()) { n_bytes -= (long)it->second; sizes.erase(it); }
  free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = calloc(n, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (!d || !s) return done(cudaErrorInvalidValue);
  if (!capturing) memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  if (!d) return done(cudaErrorInvalidValue);
  n_clear_bytes += (long)n;
  if (!capturing) memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = size_t(1) << 34; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { *p = const_cast<void *>(s); return cudaSuccess; }

// ---- device, errors, streams, events
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
  memset(p, 0, sizeof(*p));
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last_error; }
const char *cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }

// ---- kernels
struct Config { dim3 g, b; size_t smem; cudaStream_t s; };
static Config pushed;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { pushed = Config{g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
  *g = pushed.g; *b = pushed.b; *smem = pushed.smem; *(cudaStream_t *)s = pushed.s;
  return cudaSuccess;
}
static cudaError_t launch(const void *f) {
  const std::string &n = names()[f];
  if (!fail_kernel.empty() && n.find(fail_kernel) != std::string::npos) return done(cudaErrorLaunchOutOfResources);
  launched[n]++;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *f, void **) { return launch(f); }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) { memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { static void *h[1]; return h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
  names()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

// ---- graphs
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; n_captures++; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; capturing = false; *g = (cudaGraph_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                                          cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) { *st = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus *st, unsigned long long *, cudaGraph_t *g,
                                     const cudaGraphNode_t **d, size_t *n) {
  *st = cudaStreamCaptureStatusActive;
  if (g) *g = nullptr;
  if (d) *d = nullptr;
  if (n) *n = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) { *h = 1; return cudaSuccess; }
cudaError_t cudaGraphAddNode(cudaGraphNode_t *n, cudaGraph_t, const cudaGraphNode_t *, size_t, cudaGraphNodeParams *p) {
  static cudaGraph_t body[1];
  *n = nullptr;
  p->conditional.phGraph_out = body;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { n_graph_launches++; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(e); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
}
