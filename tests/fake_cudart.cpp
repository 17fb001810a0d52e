// A CUDA runtime for the CPU tests of rg_stage.cpp: devices are a range of addresses each, streams
// and events know their device as the real ones do, copies happen at once.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "rg_host.h"

namespace {
constexpr size_t kBytes = size_t(64) << 20;  // memory of a device
unsigned char* g_mem[4] = {};
std::atomic<int> g_registered{0}, g_streams{0};
std::atomic<bool> g_captureFails{false};
thread_local int t_device = 0;
thread_local cudaError_t t_last = cudaSuccess;

cudaError_t fail(cudaError_t e) {
  t_last = e;
  return e;
}
struct Obj {
  int device;
};
int deviceOf(const void* p) {
  for (int d = 0; d < 4; ++d)
    if (g_mem[d] && p >= g_mem[d] && p < g_mem[d] + kBytes) return d;
  return -1;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = t_last; t_last = cudaSuccess; return e; }
cudaError_t cudaHostRegister(void*, size_t, unsigned int) { g_registered++; return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof(*a));
  const int d = deviceOf(p);
  a->type = d < 0 ? cudaMemoryTypeUnregistered : cudaMemoryTypeDevice;
  a->device = d < 0 ? cudaInvalidDeviceId : d;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) {
  g_streams++;
  *s = (cudaStream_t) new Obj{t_device};
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete (Obj*)s; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { *e = (cudaEvent_t) new Obj{t_device}; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Obj*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return ((Obj*)e)->device == ((Obj*)s)->device ? cudaSuccess : fail(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = cudaStreamCaptureStatusNone;
  return g_captureFails ? fail(cudaErrorStreamCaptureImplicit) : cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}

// ---- what the tests call (a thread's current device is set by the caller)
rg::StageUser* fake_user() { return new rg::StageUser(); }
void fake_user_end(rg::StageUser* u) { delete u; }
void* fake_device(int d) {
  if (!g_mem[d]) g_mem[d] = (unsigned char*)std::malloc(kBytes);
  return g_mem[d];
}
void fake_current(int d) { t_device = d; }
void fake_capture_fails(int on) { g_captureFails = on != 0; }
int fake_sets_made() { return g_registered; }
int fake_last_error() { return (int)cudaGetLastError(); }
// copy to device `d` and back into `back`, on a stream of that device; the first error
int fake_round_trip(int d, const void* src, void* back, size_t n) {
  Obj stream{d};
  cudaError_t e = rg::copyToDevice(fake_device(d), src, n, (cudaStream_t)&stream);
  if (e == cudaSuccess) e = rg::copyToHost(back, fake_device(d), n, (cudaStream_t)&stream);
  return (int)e;
}
int fake_upload(int d, const void* src, size_t n) {
  Obj stream{d};
  return (int)rg::copyToDevice(fake_device(d), src, n, (cudaStream_t)&stream);
}
}
