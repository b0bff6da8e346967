// A CUDA runtime for the tests of the library's host side without a GPU:
// "device" memory is host memory, copies are memcpy, kernels do not run but
// are recorded (name, grid, first argument) and a chosen allocation fails.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
// bytes kept of a launch's first argument: what every one has on the caller's
// stack, more of the stages' argument block
constexpr size_t kArgBytes = 48, kStageBytes = 160;
struct Launch {
  std::string name;
  unsigned grid;
  unsigned char arg[kStageBytes];
};
// (filled by the objects' static constructors)
std::map<const void *, std::string> &names() {
  static std::map<const void *, std::string> m;
  return m;
}
std::map<char *, size_t> g_live;
std::vector<Launch> g_launches;
int g_fail_at = 0;  // > 0: this many allocations on, one fails
struct Config {
  dim3 grid, block;
  size_t smem;
  void *stream;
} g_config;

void record(const void *f, unsigned grid, void **args) {
  Launch l = {names()[f], grid, {}};
  const bool stage = l.name.find("stage_kernel") != std::string::npos &&
                     l.name.find("batch") == std::string::npos;
  std::memcpy(l.arg, args[0], stage ? kStageBytes : kArgBytes);
  g_launches.push_back(l);
}
void *handle() {
  static size_t next = 1000;
  return reinterpret_cast<void *>(++next);
}
}  // namespace

extern "C" {
void fake_fail_malloc(int nth) { g_fail_at = nth; }
void fake_clear() { g_launches.clear(); }
int fake_launches() { return (int)g_launches.size(); }
const char *fake_name(int i) { return g_launches[i].name.c_str(); }
unsigned fake_grid(int i) { return g_launches[i].grid; }
void fake_arg(int i, void *out) { std::memcpy(out, g_launches[i].arg, kStageBytes); }
int fake_live(void *p) {
  auto it = g_live.upper_bound((char *)p);
  if (it == g_live.begin()) return 0;
  --it;
  return (char *)p < it->first + it->second;
}

void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *,
                            void *, void *, int *) {
  names()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *st) {
  g_config = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = g_config.grid;
  *b = g_config.block;
  *smem = g_config.smem;
  *(void **)st = g_config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3, void **args, size_t, cudaStream_t) {
  record(f, g.x, args);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
  record(f, c->gridDim.x, args);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  if (g_fail_at > 0 && --g_fail_at == 0) return cudaErrorMemoryAllocation;
  *p = std::calloc(n ? n : 1, 1);
  g_live[(char *)*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  g_live.erase((char *)p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = std::calloc(n, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  if (n) std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  if (n) std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) {
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static void *scratch = std::calloc(16 << 20, 1);
  *p = scratch;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)handle();
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = (cudaGraph_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
  *x = (cudaGraphExec_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)handle();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
}
