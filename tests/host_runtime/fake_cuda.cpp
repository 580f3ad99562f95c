// fake_cuda.cpp -- the CUDA runtime as the engine's host code sees it, on host
// memory, for tests of the host code on a machine without a GPU
// (fake_launchers.cu has the kernel launchers).
//
// Copies and clears happen when they are issued, kernels do nothing.  What is
// modelled is who waits for whom: work issued to a stream, and work the legacy default stream may still
// be doing when its call returns (a device memset; a copy from pageable
// memory), stays pending until the host waits for it.  The engine's streams
// do not order with the legacy stream, so an operation on one while the other
// has work pending is a missing wait; so is a launch on a stream whose device
// is not the calling thread's.  Both are recorded and counted.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>

namespace {

struct Stream {
  int device;
  bool pending = false;
};

std::set<Stream*> g_streams;
bool g_legacy_pending = false;
int g_device = 0, g_faults = 0;
std::string g_first;

void fault(const std::string& what) {
  if (g_faults++ == 0) g_first = what;
}

bool any_pending() {
  for (Stream* s : g_streams)
    if (s->pending) return true;
  return false;
}

void waited_for_streams() {
  for (Stream* s : g_streams) s->pending = false;  // a step's streams join before its last kernel
}

void legacy(const char* what, bool waits) {
  if (any_pending()) fault(std::string(what) + " on the legacy stream while the engine's streams have work pending");
  g_legacy_pending = !waits;
}

void issue(const char* what, cudaStream_t stream, bool launch) {
  if (!stream) return legacy(what, false);
  Stream* s = reinterpret_cast<Stream*>(stream);
  if (g_legacy_pending) fault(std::string(what) + " while the legacy stream has work pending");
  if (launch && s->device != g_device) fault(std::string(what) + " on a stream of another device");
  s->pending = true;
}

}  // namespace

extern "C" {

int fake_faults() { return g_faults; }
const char* fake_first_fault() { return g_first.c_str(); }
void fake_reset() { g_faults = 0, g_first.clear(); }
void fake_launch(const char* what, cudaStream_t s) { issue(what, s, true); }

cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemset(void* p, int v, size_t n) {
  legacy("cudaMemset", false);
  return std::memset(p, v, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  issue("cudaMemsetAsync", s, false);
  return std::memset(p, v, n), cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind kind) {
  legacy("cudaMemcpy", kind == cudaMemcpyDeviceToHost);
  return std::memcpy(to, from, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t s) {
  issue("cudaMemcpyAsync", s, false);
  return std::memcpy(to, from, n), cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  waited_for_streams();
  g_legacy_pending = false;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (s) waited_for_streams();
  else g_legacy_pending = false;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) {
  auto* made = new Stream{g_device};
  g_streams.insert(made);
  *s = reinterpret_cast<cudaStream_t>(made);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned flags) { return cudaStreamCreateWithPriority(s, flags, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  g_streams.erase(reinterpret_cast<Stream*>(s));
  delete reinterpret_cast<Stream*>(s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { return *least = 0, *greatest = -1, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return waited_for_streams(), cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return *x = nullptr, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { return issue("cudaGraphLaunch", s, true), cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 2, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return g_device = d, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }

}  // extern "C"
