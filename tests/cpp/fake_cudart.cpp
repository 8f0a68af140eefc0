// A CUDA runtime without a device: what the library's host code calls, on host memory.  "Device"
// memory is host memory (zeroed), copies are memcpy, kernels do nothing (but what a test does for
// them) and are recorded by name with their grid and block, and any call or launch can be made to fail.  A virtual clock gives
// kernels and first uses a duration, for code that decides by timing.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>

namespace fake {
std::vector<Launch> launches;
std::string fail_kernel, fail_call;
size_t allocated = 0;
std::set<const void *> device_only;
std::function<void(const std::string &, void **)> on_launch;
std::function<double(const std::string &, const Launch &)> kernel_ms;
std::function<double(const std::string &)> first_use_ms;
std::map<void **, std::vector<std::string>> &modules() {  // filled before main
  static std::map<void **, std::vector<std::string>> m;
  return m;
}
}  // namespace fake

namespace {
std::map<const void *, std::string> &names() {  // filled before main
  static std::map<const void *, std::string> m;
  return m;
}
std::set<const void *> g_used;
std::map<void *, size_t> g_sizes;
double g_host = 0.0, g_stream = 0.0;  // ms
cudaError_t g_last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_config;

cudaError_t check(const char *call) {
  return fake::fail_call == call ? cudaErrorUnknown : cudaSuccess;
}
void use(const void *fn) {
  if (g_used.insert(fn).second && fake::first_use_ms) g_host += fake::first_use_ms(names()[fn]);
}
cudaError_t launch(const void *fn, dim3 grid, dim3 block, void **args) {
  const std::string &name = names()[fn];
  if (!fake::fail_kernel.empty() && name.find(fake::fail_kernel) != std::string::npos)
    return g_last = cudaErrorCooperativeLaunchTooLarge;
  use(fn);
  fake::Launch l{name, (int)grid.x, (int)grid.y, (int)block.x};
  fake::launches.push_back(l);
  if (fake::on_launch) fake::on_launch(name, args);
  g_stream = (g_stream > g_host ? g_stream : g_host) +
             (fake::kernel_ms ? fake::kernel_ms(name, l) : 0.01);
  return cudaSuccess;
}
cudaError_t copy(void *d, const void *s, size_t n, cudaMemcpyKind kind) {
  if (cudaError_t e = check("cudaMemcpy")) return e;
  if (kind == cudaMemcpyDeviceToHost && fake::device_only.count(d)) return cudaErrorInvalidValue;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
}  // namespace

struct CUevent_st {
  double t;
};

extern "C" {
void **__cudaRegisterFatBinary(void *) { return new void *; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **module, const char *host, char *, const char *name, int, uint3 *,
                            uint3 *, dim3 *, dim3 *, int *) {
  names()[host] = name;
  fake::modules()[module].push_back(name);
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  g_config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *static_cast<cudaStream_t *>(stream) = g_config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *fn, dim3 grid, dim3 block, void **args, size_t,
                             cudaStream_t) {
  return launch(fn, grid, block, args);
}
cudaError_t cudaLaunchCooperativeKernel(const void *fn, dim3 grid, dim3 block, void **args, size_t,
                                        cudaStream_t) {
  return launch(fn, grid, block, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args) {
  return launch(fn, c->gridDim, c->blockDim, args);
}
cudaError_t cudaMalloc(void **p, size_t n) {
  if (cudaError_t e = check("cudaMalloc")) return e;
  *p = std::calloc(n ? n : 1, 1);
  g_sizes[*p] = n;
  fake::allocated += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  fake::allocated -= g_sizes[p];
  g_sizes.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = std::calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  return copy(d, s, n, k);
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return copy(d, s, n, k);
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
  for (size_t i = 0; i < h; i++)
    std::memcpy(static_cast<char *>(d) + i * dp, static_cast<const char *>(s) + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = *t = (size_t)180 << 30;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  std::memset(a, 0, sizeof(*a));
  a->type = fake::device_only.count(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148
       : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
  std::memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 148;
  p->major = 10;
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  *p = nullptr;
  return cudaErrorInvalidSymbol;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *fn) {
  use(fn);
  std::memset(a, 0, sizeof(*a));
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *fn, cudaFuncAttribute, int) {
  use(fn);
  return cudaSuccess;
}
// 1,024 threads to an SM, of any kernel
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int threads,
                                                          size_t) {
  *n = 1024 / threads;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *c) {
  *n = 148 * (1024 / (int)c->blockDim.x) / (int)c->gridDim.x;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(&g_config);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  if (g_host < g_stream) g_host = g_stream;
  return check("cudaStreamSynchronize");
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = new CUevent_st{0.0};
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete e;
  return cudaSuccess;
}
// an event is reached when the stream gets to it: at once on an idle one
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  if (cudaError_t c = check("cudaEventRecord")) return c;
  if (g_stream < g_host) g_stream = g_host;
  e->t = g_stream;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (g_host < e->t) g_host = e->t;
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(b->t - a->t);
  return cudaSuccess;
}
}
