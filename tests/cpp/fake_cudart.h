// A stand-in for the CUDA runtime calls that the library's host code makes
// (an executable that includes it takes them over from libcudart): launches
// do nothing and are counted, device memory is host memory, copies copy. A
// test can make a launch or an allocation fail, and it can see when a captured graph is
// replayed after memory that was there at its capture has been freed.  Freed
// memory is given out again, the longest free first, separately for requests
// of up to 64 KB and for larger ones: addresses come back as from a device.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <set>

namespace fake {
inline cudaError_t last = cudaSuccess;
inline long launches = 0, fail_at = -1;      // the launch with this number fails
inline long allocs = 0, fail_alloc_at = -1;  // the allocation with this number fails
inline int graphs = 0, stale_replays = 0;    // captures so far; replays of graphs whose memory was freed
inline uint32_t read_back = 0;               // every device-to-host copy gives these words
inline std::set<void*> live;
struct Graph {
  std::set<void*> memory;
  bool stale = false;
};
inline std::set<Graph*> instances;
inline bool capturing = false;

constexpr size_t kSmall = 64 << 10, kLarge = 512 << 20;  // (pages nobody touches cost nothing)
inline std::map<void*, bool> small;
inline std::deque<void*> unused[2];

inline cudaError_t alloc(void** p, size_t n) {
  *p = nullptr;
  if (allocs++ == fail_alloc_at || n > kLarge) return cudaErrorMemoryAllocation;
  const bool s = n <= kSmall;
  if (!unused[s].empty()) {
    *p = unused[s].front();
    unused[s].pop_front();
  } else if ((*p = malloc(s ? kSmall : kLarge)) == nullptr) {
    return cudaErrorMemoryAllocation;
  }
  small[*p] = s;
  live.insert(*p);
  return cudaSuccess;
}
inline cudaError_t release(void* p) {
  if (!p) return cudaSuccess;
  for (Graph* g : instances)
    if (g->memory.count(p)) g->stale = true;
  live.erase(p);
  unused[small[p]].push_back(p);
  return cudaSuccess;
}
inline cudaError_t launch() {
  if (launches++ == fail_at) return last = cudaErrorLaunchOutOfResources;
  return cudaSuccess;
}
template <typename T>
cudaError_t handle(T* out) {
  static long next = 0x1000;
  *out = reinterpret_cast<T>(next += 16);
  return cudaSuccess;
}
inline int null_copies = 0;  // copies and fills at a null pointer
inline cudaError_t copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
  if (!dst || !src) return null_copies++, cudaSuccess;
  if (kind != cudaMemcpyDeviceToHost) {
    if (kind == cudaMemcpyHostToDevice) memcpy(dst, src, n);
    return cudaSuccess;
  }
  for (size_t i = 0; i + 4 <= n; i += 4) memcpy(static_cast<char*>(dst) + i, &read_back, 4);
  return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaGetLastError() {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void*) { return fake::handle(k); }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return fake::launch(); }
cudaError_t cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return fake::launch(); }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 2, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  return *n = 2, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { return *p = const_cast<void*>(s), cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return fake::alloc(p, n); }
cudaError_t cudaFree(void* p) { return fake::release(p); }
cudaError_t cudaFreeHost(void* p) { return fake::release(p); }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  return fake::copy(dst, src, n, kind);
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) { return fake::copy(dst, src, n, kind); }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = (size_t)1 << 38, cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { return fake::handle(p); }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return fake::alloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake::release(p); }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int, size_t, cudaStream_t) { return fake::null_copies += !p, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return fake::handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return fake::handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return fake::handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = fake::capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return fake::capturing = true, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  fake::capturing = false;
  fake::graphs++;
  fake::Graph* f = new fake::Graph;
  f->memory = fake::live;
  *g = reinterpret_cast<cudaGraph_t>(f);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  fake::Graph* f = new fake::Graph(*reinterpret_cast<fake::Graph*>(g));
  fake::instances.insert(f);
  *x = reinterpret_cast<cudaGraphExec_t>(f);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete reinterpret_cast<fake::Graph*>(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  fake::Graph* f = reinterpret_cast<fake::Graph*>(x);
  fake::instances.erase(f);
  return delete f, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  if (reinterpret_cast<fake::Graph*>(x)->stale) fake::stale_replays++;
  return cudaSuccess;
}
}
