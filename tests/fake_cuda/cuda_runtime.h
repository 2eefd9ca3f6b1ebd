// The few CUDA runtime calls of asr_b200/csrc/devmem.h on a made-up device of `total` bytes, for its test without a device.
#pragma once
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>

typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
typedef struct Fake_stream* cudaStream_t;
typedef struct Fake_event* cudaEvent_t;
struct FakePool { size_t reserved = 0, used = 0; };
typedef FakePool* cudaMemPool_t;
enum { cudaMemAllocationTypePinned = 1, cudaMemLocationTypeDevice = 1, cudaEventDisableTiming = 2 };
enum cudaMemPoolAttr { cudaMemPoolAttrReleaseThreshold, cudaMemPoolAttrReservedMemCurrent, cudaMemPoolAttrUsedMemCurrent };
struct cudaMemPoolProps { int allocType; struct { int type, id; } location; };

struct FakeDevice {
  std::mutex lock;
  size_t total = (size_t)180 << 30, others = 0, used = 0;   // others: what other users of the device hold
  std::map<void*, size_t> blocks;
  std::map<void*, std::pair<FakePool*, size_t>> pooled;
  uintptr_t next = 4096;
  int asked = 0, mallocs = 0, frees = 0, events = 0;
  size_t free_bytes() const { return total > others + used ? total - others - used : 0; }
};
inline FakeDevice& fake() { static FakeDevice d; return d; }

inline cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> g(fake().lock);
  if (n > fake().free_bytes()) return cudaErrorMemoryAllocation;
  *p = (void*)(fake().next += 4096);
  fake().blocks[*p] = n;
  fake().used += n;
  ++fake().mallocs;
  return cudaSuccess;
}
template <typename T> cudaError_t cudaMalloc(T** p, size_t n) { return cudaMalloc((void**)p, n); }
inline cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> g(fake().lock);
  if (!p) return cudaSuccess;
  auto it = fake().blocks.find(p);
  if (it == fake().blocks.end()) return 1;
  fake().used -= it->second;
  fake().blocks.erase(it);
  ++fake().frees;
  return cudaSuccess;
}
inline cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  std::lock_guard<std::mutex> g(fake().lock);
  ++fake().asked;
  *f = fake().free_bytes();
  *t = fake().total;
  return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, int) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  std::lock_guard<std::mutex> g(fake().lock);
  ++fake().events;
  *e = (cudaEvent_t)(fake().next += 4096);
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t) {
  std::lock_guard<std::mutex> g(fake().lock);
  --fake().events;
  return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = new FakePool; return cudaSuccess; }
inline cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  std::lock_guard<std::mutex> g(fake().lock);
  fake().used -= p->reserved;
  delete p;
  return cudaSuccess;
}
inline cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
inline cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  std::lock_guard<std::mutex> g(fake().lock);
  *(uint64_t*)v = a == cudaMemPoolAttrReservedMemCurrent ? p->reserved : p->used;
  return cudaSuccess;
}
inline cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t most) {
  std::lock_guard<std::mutex> g(fake().lock);
  const size_t to = p->used > most ? p->used : most;
  if (p->reserved > to) { fake().used -= p->reserved - to; p->reserved = to; }
  return cudaSuccess;
}
inline cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  std::lock_guard<std::mutex> g(fake().lock);
  if (pool->reserved - pool->used < n) {
    const size_t more = n - (pool->reserved - pool->used);
    if (more > fake().free_bytes()) return cudaErrorMemoryAllocation;
    fake().used += more;
    pool->reserved += more;
  }
  pool->used += n;
  *p = (void*)(fake().next += 4096);
  fake().pooled[*p] = {pool, n};
  return cudaSuccess;
}
inline cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  std::lock_guard<std::mutex> g(fake().lock);
  auto it = fake().pooled.find(p);
  if (it == fake().pooled.end()) return 1;
  it->second.first->used -= it->second.second;
  fake().pooled.erase(it);
  return cudaSuccess;
}
