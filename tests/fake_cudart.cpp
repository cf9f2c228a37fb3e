// A stand-in for the CUDA runtime that runs the library's host code on a machine
// without a GPU (preloaded before libcudart; test_host_order.py).  Device memory is
// host memory, kernels do nothing, and two kinds of facts are recorded:
//
//  - uploads in flight: a copy from pageable memory or a memset on the legacy stream
//    may return before it lands, and non-blocking streams do not wait for it.  The
//    next legacy copy waits for the earlier ones, a synchronisation for all; work
//    given to another stream while one is in flight is counted as a fault;
//  - one-launch Krylov solves: a launch of persist_kernel reports the end of its
//    solve in the flags, or, where the test says so, that its barrier ran out of time;
//    the plans made for them are counted (each asks once whether the device can do
//    cooperative launches);
//  - what the streams are given: a graph (G), one-cluster solves of a batch (C), a
//    cluster (P) or a grid (R) that solves one system, a wait of the host (S);
//  - frees, each of which waits for the whole device.
//
// A device-to-host copy of a single double reads 1.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <string>

#include "persist.h"

namespace {
int g_pending = 0, g_faults = 0;
int g_launches = 0, g_late_at = -1, g_iters = 1, g_plans = 0, g_frees = 0, g_clusters = 8;
std::string g_log;
constexpr uintptr_t kTestStream = 4096;  // the stream that tests pass
void landed() { g_pending = 0; }
void uses(cudaStream_t s) {
  if (s != nullptr && g_pending > 0) ++g_faults;
}
// upper case on the test's stream, lower case on another
void note(char c, cudaStream_t s) { g_log += reinterpret_cast<uintptr_t>(s) == kTestStream ? c : char(c + 32); }
}  // namespace

extern "C" {

// --- the test's side
int fake_pending() { return g_pending; }
int fake_faults() {
  const int f = g_faults;
  g_faults = 0;
  return f;
}
int fake_launches() { return g_launches; }
int fake_plans() {
  const int n = g_plans;
  g_plans = 0;
  return n;
}
int fake_frees() {
  const int n = g_frees;
  g_frees = 0;
  return n;
}
// Clusters that the device can run at once.
void fake_clusters(int n) { g_clusters = n; }
const char* fake_log() {
  static std::string out;
  out.swap(g_log);
  g_log.clear();
  return out.c_str();
}
// The launches of one-launch solves from now on report `iters` iterations and the end
// of the solve; the one numbered late_at (from 0; -1: none) a late barrier instead.
void fake_solves(int iters, int late_at) {
  g_launches = 0;
  g_iters = iters;
  g_late_at = late_at;
}

// --- the runtime's side
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::calloc(n + 32, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) {
  if (p) ++g_frees;
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  uses(st);
  std::memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost && n == sizeof(double)) *static_cast<double*>(d) = 1.0;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  landed();
  std::memcpy(d, s, n);
  if (k == cudaMemcpyHostToDevice) g_pending = 1;
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  ++g_pending;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  uses(st);
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  landed();
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (s == nullptr) landed();
  note('S', s);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t st) {
  uses(st);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void** args) {
  uses(c->stream);
  if (*static_cast<int*>(args[1]) != int(c->dynamicSmemBytes)) {  // not persist_kernel: its form for batches
    note('C', c->stream);
    return cudaSuccess;
  }
  const ufem::PersistSolve& a = *static_cast<const ufem::PersistSolve*>(args[0]);
  note(c->attrs[0].id == cudaLaunchAttributeCooperative ? 'R' : 'P', c->stream);
  const bool late = g_launches++ == g_late_at;
  if (late) a.ictl[ufem::kFlagLate] = 1;
  a.ictl[0] = late ? 0 : 1;
  a.ictl[2] = 0;
  a.ictl[3] = g_iters;
  a.dctl[ufem::kBnorm] = 1.0;
  a.dctl[ufem::kTrue] = 0.0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
  if (a == cudaDevAttrCooperativeLaunch) ++g_plans;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = g_clusters;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static void* scratch = std::calloc(size_t(16) << 20, 1);
  *p = scratch;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(std::malloc(8));
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamGetPriority(cudaStream_t, int* p) {
  *p = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(std::malloc(8));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(std::malloc(8));
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(std::malloc(8));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  std::free(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  uses(s);
  note('G', s);
  return cudaSuccess;
}

}  // extern "C"
