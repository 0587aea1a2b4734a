// The runtime of fake_cudart.h, and the registration entry points nvcc's objects call.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <deque>
#include <set>
#include <utility>
#include <vector>

namespace fake {
std::recursive_mutex mu;
bool device_runs = true, capturing = false;
int fail_queries = 0, refused = 0, frees_while_busy = 0;
}  // namespace fake

namespace {
struct Stream {
  std::deque<std::function<void()>> ops;
};
struct Event {
  Stream* stream = nullptr;
  bool pending = false;
};
std::set<Stream*> g_streams;
thread_local cudaStreamCaptureMode t_mode = cudaStreamCaptureModeGlobal;

Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
void run(Stream* s) {
  while (!s->ops.empty()) {
    auto f = std::move(s->ops.front());
    s->ops.pop_front();
    f();
  }
}
cudaError_t unsafe() {  // a call that a global-mode capture of any thread forbids
  if (!fake::capturing || t_mode == cudaStreamCaptureModeRelaxed) return cudaSuccess;
  ++fake::refused;
  return cudaErrorStreamCaptureUnsupported;
}
#define LOCK std::lock_guard<std::recursive_mutex> lock_(fake::mu)
}  // namespace

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
  std::swap(*m, t_mode);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  LOCK;
  if (cudaError_t e = unsafe()) return e;
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  LOCK;
  if (p && fake::busy()) ++fake::frees_while_busy;  // and lost: the work may use it
  else std::free(p);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  LOCK;
  Stream* n = new Stream();
  g_streams.insert(n);
  *s = reinterpret_cast<cudaStream_t>(n);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {  // its work goes on
  LOCK;
  if (of(s)->ops.empty()) {
    g_streams.erase(of(s));
    delete of(s);
  }
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  LOCK;
  if (cudaError_t e = unsafe()) return e;
  run(of(s));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new Event());
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  LOCK;
  Event* v = reinterpret_cast<Event*>(e);
  if (!v->pending) delete v;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  LOCK;
  Event* v = reinterpret_cast<Event*>(e);
  v->stream = of(s);
  v->pending = true;
  of(s)->ops.push_back([v] { v->pending = false; });
  return cudaSuccess;
}
static void run_to(Event* v) {
  while (v->pending && !v->stream->ops.empty()) {
    auto f = std::move(v->stream->ops.front());
    v->stream->ops.pop_front();
    f();
  }
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
  LOCK;
  if (cudaError_t r = unsafe()) return r;
  if (fake::fail_queries > 0) {
    --fake::fail_queries;
    return cudaErrorUnknown;
  }
  Event* v = reinterpret_cast<Event*>(e);
  if (fake::device_runs) run_to(v);
  return v->pending ? cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  LOCK;
  if (cudaError_t r = unsafe()) return r;
  run_to(reinterpret_cast<Event*>(e));
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  LOCK;
  if (k == cudaMemcpyHostToDevice) {  // the copies up are of pageable memory: staged at once
    std::vector<char> data((const char*)s, (const char*)s + n);
    of(st)->ops.push_back([d, data] { std::memcpy(d, data.data(), data.size()); });
  } else {
    of(st)->ops.push_back([d, s, n] { std::memcpy(d, s, n); });
  }
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  LOCK;
  of(st)->ops.push_back([d, v, n] { std::memset(d, v, n); });
  return cudaSuccess;
}
}  // extern "C"


namespace fake {
void enqueue(cudaStream_t s, std::function<void()> f) {
  LOCK;
  of(s)->ops.push_back(std::move(f));
}
int busy() {
  LOCK;
  int n = 0;
  for (Stream* s : g_streams) n += s->ops.empty() ? 0 : 1;
  return n;
}
}  // namespace fake

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, unsigned long, int, int) {}
int __cudaPopCallConfiguration(void*, void*, unsigned long*, void*) { return 1; }
int __cudaGetKernel(void*, const void*) { return 1; }
int __cudaLaunchKernel() { return 1; }
}
