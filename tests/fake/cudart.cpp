// A stand-in for the CUDA runtime, for tests of the library's host side on machines
// without a GPU: two devices, memory on the host heap, launches that are checked and
// noted but compute nothing.  Linked with the library's own objects (fake_runtime in
// tests/fake/__init__.py); failures that a GPU must not be made to have are made here.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <utility>
#include <vector>

namespace {
constexpr int DEVICES = 2;
int g_dev = 0, g_sms[DEVICES] = {152, 152};
cudaError_t g_last = cudaSuccess;
std::map<const void*, std::string> g_name;               // host stub -> kernel
std::map<std::pair<int, const void*>, int> g_optin;      // (device, kernel) -> dynamic shared memory
std::vector<std::string>* g_capture = nullptr;
std::string g_log, g_fail;
int g_status = 0;
struct Config {
  dim3 grid, block;
  size_t smem;
  void* stream;
} g_config;
cudaError_t fail(cudaError_t e) { return g_last = e; }
void* fresh(size_t n) { return calloc(1, n ? n : 1); }
cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == sizeof(int) && g_status) *(int*)d |= g_status;
  return cudaSuccess;
}
}  // namespace

// the tests' side
extern "C" {
void fake_device(int d) { g_dev = d; }
void fake_sms(int d, int n) { g_sms[d] = n; }
void fake_pending(int e) { g_last = (cudaError_t)e; }
void fake_fail(const char* part) { g_fail = part; }       // launches of kernels so named are refused
void fake_status(int bits) { g_status = bits; }           // or-ed into every int read back
void fake_clear() { g_log.clear(); }
const char* fake_log() { return g_log.c_str(); }          // launches, one per line: kernel@grid x,grid y
}

extern "C" {
void** __cudaRegisterFatBinary(void*) { return (void**)fresh(8); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_name[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
  *k = (cudaKernel_t)host;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
  g_config = Config{g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = g_config.grid;
  *b = g_config.block;
  *smem = g_config.smem;
  *(void**)s = g_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t) {
  const std::string& name = g_name[(const void*)k];
  if (!g_fail.empty() && name.find(g_fail) != std::string::npos) return fail(cudaErrorLaunchOutOfResources);
  if (smem > 48 * 1024 && (int)smem > g_optin[{g_dev, (const void*)k}]) return fail(cudaErrorInvalidValue);
  if (!g.x || !g.y || !g.z || g.y > 65535 || g.z > 65535 || !b.x || b.x * b.y * b.z > 1024)
    return fail(cudaErrorInvalidConfiguration);
  const std::string note = name + "@" + std::to_string(g.x) + "," + std::to_string(g.y);
  if (g_capture) g_capture->push_back(note);
  else g_log += note + "\n";
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v > 227 * 1024) return fail(cudaErrorInvalidValue);
  g_optin[{g_dev, f}] = v;
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = DEVICES, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = g_dev, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { return *v = g_sms[d], cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "an error of the test's making"; }
cudaError_t cudaPeekAtLastError() { return g_last; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) { return fail(cudaErrorInvalidValue); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = nullptr, fail(cudaErrorInvalidValue); }

cudaError_t cudaMalloc(void** p, size_t n) { return *p = fresh(n), cudaSuccess; }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = fresh(n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return copy(d, s, n, k); }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  for (size_t i = 0; i < h; ++i) memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind) { return memset(d, 0, n), cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)fresh(8), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)fresh(8), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }

// a graph is the list of the kernels captured
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  g_capture = new std::vector<std::string>();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)g_capture;
  g_capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t) new std::vector<std::string>(*(std::vector<std::string>*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete (std::vector<std::string>*)g, cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return delete (std::vector<std::string>*)e, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (const std::string& n : *(std::vector<std::string>*)e) g_log += n + "\n";
  return cudaSuccess;
}
}
