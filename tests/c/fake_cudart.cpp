// fake_cudart.cpp -- a CUDA runtime without a device: memory is the host's,
// copies are memcpy, kernels are not run.  Every call that queues or waits is
// written to a log, and a test can have the n-th call of one name fail, so
// that the library's error paths run on the CPU (tests/test_error_paths.py
// links its objects against this file).
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::string g_log, g_fail_name;
std::map<const void*, std::string>& names() {  // filled while the library is loaded
  static std::map<const void*, std::string> m;
  return m;
}
int g_fail_at = 0, g_int = 0;
cudaError_t g_fail_code = cudaSuccess, g_last = cudaSuccess;
long g_next = 16;
struct {
  dim3 grid, block;
  size_t smem;
  void* stream;
} g_cfg;

cudaError_t call(const char* name, const void* stream, const std::string& what = "") {
  if (g_fail_name == name && --g_fail_at == 0) {
    g_last = g_fail_code;
    g_log += std::string("fail ") + name + "\n";
    return g_fail_code;
  }
  g_log += std::string(name) + " " + std::to_string((long)stream) + (what.empty() ? "" : " " + what) + "\n";
  return cudaSuccess;
}
template <class T>
cudaError_t give(const char* name, T* out) {
  const cudaError_t e = call(name, nullptr);
  if (e == cudaSuccess) *out = (T)(g_next += 16);
  return e;
}
cudaError_t room(const char* name, void** p, size_t n) {
  const cudaError_t e = call(name, nullptr);
  *p = e == cudaSuccess ? std::calloc(n + 64, 1) : nullptr;
  return e;
}
cudaError_t copy(const char* name, void* d, const void* s, size_t n, cudaMemcpyKind k, void* stream) {
  const cudaError_t e = call(name, stream);
  if (e != cudaSuccess) return e;
  std::memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == sizeof(int) && g_int) std::memcpy(d, &g_int, n);
  return e;
}
}  // namespace

extern "C" {
// for the test: the n-th call of `name` from now on fails; single ints read
// back from the device are v (0: what is there)
void fake_fail(const char* name, int n, int code) {
  g_fail_name = name;
  g_fail_at = n;
  g_fail_code = (cudaError_t)code;
}
void fake_int(int v) { g_int = v; }
void fake_clear() { g_log.clear(); }
const char* fake_log() { return g_log.c_str(); }

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
  g_cfg = {g, b, s, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = g_cfg.grid;
  *b = g_cfg.block;
  *s = g_cfg.smem;
  *(void**)st = g_cfg.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) {
  return call("cudaLaunchKernel", s, names()[f]);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) {
  return call("cudaLaunchCooperativeKernel", s, names()[f]);
}
cudaError_t cudaMalloc(void** p, size_t n) { return room("cudaMalloc", p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return room("cudaMallocHost", p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return room("cudaMallocHost", p, n); }
cudaError_t cudaFree(void* p) {
  std::free(p);
  return call("cudaFree", nullptr);
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy("cudaMemcpy", d, s, n, k, nullptr); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  return copy("cudaMemcpyAsync", d, s, n, k, st);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
  const cudaError_t e = call("cudaMemsetAsync", s);
  if (e == cudaSuccess) std::memset(d, v, n);
  return e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return give("cudaStreamCreateWithFlags", s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return call("cudaStreamSynchronize", s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  return call("cudaStreamWaitEvent", s, std::to_string((long)e));
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return give("cudaEventCreate", e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return give("cudaEventCreate", e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return call("cudaEventRecord", s, std::to_string((long)e)); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return call("cudaEventSynchronize", e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return call("cudaDeviceSynchronize", nullptr); }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount      ? 148
       : a == cudaDevAttrComputeCapabilityMajor ? 10
       : a == cudaDevAttrMaxGridDimX            ? 0x7fffffff
                                                : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof(*a));
  a->ptxVersion = a->binaryVersion = 100;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return room("cudaMalloc", p, 1 << 20); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
// graphs are not part of what is tested here
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, cudaStreamCaptureMode) {
  return cudaErrorNotSupported;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;
  return cudaErrorNotSupported;
}
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus*, unsigned long long*, cudaGraph_t*,
                                        const cudaGraphNode_t**, size_t*) {
  return cudaErrorNotSupported;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, size_t, unsigned) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams*) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
