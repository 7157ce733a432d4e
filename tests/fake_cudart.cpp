// TEST INFRASTRUCTURE: a CUDA runtime without a GPU, which the library's objects are linked with so
// that its host side can be tested: which kernels a call launches, on which device, and what it does
// when a call of the runtime fails. Device memory is host memory; launches are recorded, not run.
//
// As in the real runtime, a kernel's dynamic shared memory above 48 KB needs its opt-in attribute on
// the device it is launched on, a cooperative grid has to fit the SMs, and the error of a failed
// launch stays the last error until cudaGetLastError takes it.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#undef cudaGetDeviceProperties

namespace {

constexpr int kSms = 148, kSharedOptIn = 232448;

std::mutex g_mu;
std::map<const void*, std::string> g_names;             // kernels by host address
std::map<std::pair<int, const void*>, int> g_dynamic;   // opted-in shared memory, by device
std::string g_log;  // "<device> <kernel>\n" for each launch, "+dependent" behind a dependent one
int g_cooperative = kSms;                               // CTAs of a cooperative grid that fit
int g_pass = 0, g_fail = 0;                             // launches until the one that fails, its error

thread_local int t_device = 0;
thread_local cudaError_t t_last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local Config t_config{};

cudaError_t result(cudaError_t e) {
  if (e != cudaSuccess) t_last = e;
  return e;
}

cudaError_t launch(const void* f, dim3 grid, size_t smem, bool cooperative, bool dependent) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (g_fail != 0 && g_pass-- == 0) {
    const auto e = static_cast<cudaError_t>(g_fail);
    g_fail = 0;
    return result(e);
  }
  const auto it = g_dynamic.find({t_device, f});
  if (smem > (size_t)(it == g_dynamic.end() ? 48 << 10 : it->second))
    return result(cudaErrorInvalidValue);
  if (cooperative && (long long)grid.x * grid.y * grid.z > g_cooperative)
    return result(cudaErrorCooperativeLaunchTooLarge);
  g_log += std::to_string(t_device) + " " + g_names[f] + (dependent ? "+dependent\n" : "\n");
  return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- What the tests set and read.

// The launches since the last call, one a line; valid until the next call.
const char* fake_take_log() {
  static std::string out;
  std::lock_guard<std::mutex> lock(g_mu);
  out.swap(g_log);
  g_log.clear();
  return out.c_str();
}
void fake_set_cooperative_limit(int ctas) { g_cooperative = ctas < 0 ? kSms : ctas; }
void fake_fail_launch(int after, int error) { g_pass = after, g_fail = error; }
void fake_set_device(int device) { t_device = device; }

// ---- Kernels.

void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
  g_names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  t_config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = t_config.grid;
  *block = t_config.block;
  *smem = t_config.smem;
  *static_cast<cudaStream_t*>(stream) = t_config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) {
  return launch(f, grid, smem, false, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  bool cooperative = false, dependent = false;
  for (unsigned k = 0; k < c->numAttrs; ++k) {
    if (c->attrs[k].id == cudaLaunchAttributeCooperative) cooperative = c->attrs[k].val.cooperative;
    if (c->attrs[k].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      dependent = c->attrs[k].val.programmaticStreamSerializationAllowed;
  }
  return launch(f, c->gridDim, c->dynamicSmemBytes, cooperative, dependent);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v > kSharedOptIn) return result(cudaErrorInvalidValue);
    g_dynamic[{t_device, f}] = v;
  }
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* blocks, const void*, int,
                                                                   size_t, unsigned) {
  *blocks = 1;
  return cudaSuccess;
}

// ---- Devices and errors.

cudaError_t cudaGetDevice(int* d) {
  *d = t_device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  t_device = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount            ? kSms
       : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kSharedOptIn
                                                      : 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = t_last;
  t_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
const char* cudaGetErrorName(cudaError_t) { return "error"; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long,
                                    cudaDriverEntryPointQueryResult* r) {
  *f = nullptr;
  if (r) *r = cudaDriverEntryPointSymbolNotFound;
  return cudaErrorUnknown;
}

// ---- Memory.

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : result(cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  if (v != 0 || n < (64u << 10)) std::memset(d, v, n);  // large arrays are zero since cudaMalloc
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) {
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind) {
  std::memset(d, 0, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return result(cudaErrorInvalidSymbol); }

// ---- Streams and graphs (whose replays are not recorded).

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(&g_mu);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(&g_mu);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"
