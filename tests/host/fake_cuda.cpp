// fake_cuda.cpp -- see fake_cuda.h.  Only what the host layer calls.
#include "fake_cuda.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

namespace {

std::map<const char *, size_t> live;  // base -> bytes
size_t in_use = 0, limit = (size_t)1 << 40;
bool hidden = false;
int dead = 0, ncapture = 0, nlaunch = 0;
cudaError_t last = cudaSuccess;
cudaStream_t capturing = nullptr;
std::vector<const void *> recorded;
long next_handle = 0x1000;

struct Graph {
  std::vector<const void *> ptrs;
};

bool is_live(const void *p) {
  auto it = live.upper_bound((const char *)p);
  if (it == live.begin()) return false;
  --it;
  return (const char *)p < it->first + it->second;
}
cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
template <class T>
T handle() {
  return (T)(next_handle += 16);
}

}  // namespace

namespace fake {
void set_free_bytes(size_t n) { limit = in_use + n; }
void hide_free(bool on) { hidden = on; }
size_t bytes_in_use() { return in_use; }
int dead_uses() { return dead; }
int captures() { return ncapture; }
int graph_launches() { return nlaunch; }
void use(const void *p, void *s) {
  if (capturing && s == (void *)capturing) recorded.push_back(p);
  if (!is_live(p)) dead++;
}
}  // namespace fake

extern "C" {

cudaError_t cudaMalloc(void **p, size_t n) {
  *p = nullptr;
  if (in_use + n > limit) return done(cudaErrorMemoryAllocation);
  char *q = (char *)calloc(n ? n : 1, 1);
  live[q] = n ? n : 1;
  in_use += n ? n : 1;
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {  // the memory stays: a dead pointer is never handed out again
  if (!p) return cudaSuccess;
  auto it = live.find((const char *)p);
  if (it == live.end()) return done(cudaErrorInvalidValue);
  in_use -= it->second;
  live.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = hidden ? (size_t)1 << 40 : limit - in_use;
  *t = limit;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  if (k != cudaMemcpyDeviceToHost) fake::use(d, nullptr);
  if (k != cudaMemcpyHostToDevice) fake::use(s, nullptr);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemset(void *p, int v, size_t n) {
  fake::use(p, nullptr);
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int, size_t, cudaStream_t s) {
  fake::use(p, s);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  memset(a, 0, sizeof *a);
  a->type = is_live(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  capturing = s;
  recorded.clear();
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  capturing = nullptr;
  ncapture++;
  *g = (cudaGraph_t) new Graph{recorded};
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t) new Graph(*(Graph *)g);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph *)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { delete (Graph *)g; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t g, cudaStream_t s) {
  nlaunch++;
  for (const void *p : ((Graph *)g)->ptrs) fake::use(p, s);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = handle<cudaStream_t>(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = handle<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

}  // extern "C"
