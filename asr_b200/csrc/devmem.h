// Device memory of a call's temporaries, kept between calls.  Host code on the CUDA runtime's calls alone, so that its rules
// can be tested without a device.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <mutex>

namespace asrb {

// The memory of a call's temporaries (DevMem) stays with the library, so that a call neither maps nor unmaps device memory
// (cudaMalloc and cudaFree of a chain batch's vectors took 10-50 ms a call, a second when the device's other processes did
// the same).  Arrays of BIG bytes or more are blocks of the device's allocator, at most `keep` bytes of them held between
// calls (the least recently used go first); smaller ones come from a stream-ordered pool that holds at most POOL_KEEP.  (The
// pool for all sizes: mapping a 20 GB array that it had given back took a second.)  One store serves all contexts of a
// device, so that several hold no more than one and an allocation of one that would fail gets what another has left.  What a
// context's calls left goes back with the context, and everything when a context's hold_workspace is switched off, when an
// allocation would fail, and at the end of a call that found less than a quarter of the device free or this store's
// (MemScope).  A call finds out when it takes new memory, and every LOOK-th that plans.
struct DevStore {
  static constexpr size_t BIG = (size_t)32 << 20, POOL_KEEP = (size_t)256 << 20;
  static constexpr int MOST = 64;   // held blocks
  static constexpr int LOOK = 64;   // 0.1 to 1 ms a question: at most some 15 us a call (4 % of a 0.9 ms call at 8)
  struct Block {
    void* p;
    size_t bytes;
    cudaEvent_t done;   // after the last use
    uint64_t used;
    const void* owner;   // context of the last use
  };
  std::mutex lock;
  int users = 0;        // contexts
  Block blocks[MOST];   // held, not in use
  int n = 0;
  uint64_t uses = 0;
  size_t keep = 0, out = 0;   // out: bytes of the blocks in use
  int plans = 0;              // served without asking the device, since it was asked last
  std::atomic<bool> scarce{false};
  cudaMemPool_t pool = nullptr;

  // the first and every further context of the device
  void open(int device, size_t total) {
    std::lock_guard<std::mutex> g(lock);
    if (users++) return;
    keep = total / 8;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
      uint64_t most = POOL_KEEP;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &most);
    } else {
      pool = nullptr;   // no pools on this device: small arrays from the device
      cudaGetLastError();
    }
  }
  // a context goes, with what its calls left
  void close(cudaStream_t s, const void* owner) {
    cudaStreamSynchronize(s);
    std::lock_guard<std::mutex> g(lock);
    for (int q = n - 1; q >= 0; --q)
      if (blocks[q].owner == owner) release(q);
    if (pool) cudaMemPoolTrimTo(pool, 0);
    if (--users) return;
    if (pool) cudaMemPoolDestroy(pool);
    pool = nullptr;
  }
  // a block of at least `bytes` for work on stream s: the smallest held one of up to twice that (a larger one is wanted by a
  // larger array of the same call), else a new one (false: out of memory)
  bool get(size_t bytes, cudaStream_t s, Block& b) {
    {
      std::lock_guard<std::mutex> g(lock);
      const bool taken[MOST] = {};
      const int at = fit(bytes, taken);
      if (at >= 0) {
        if (cudaStreamWaitEvent(s, blocks[at].done, 0) != cudaSuccess) {
          cudaGetLastError();
          return false;
        }
        b = blocks[at];
        blocks[at] = blocks[--n];
        out += b.bytes;
        return true;
      }
    }
    b = Block{nullptr, bytes, nullptr, 0, nullptr};
    if (cudaMalloc(&b.p, bytes) != cudaSuccess) {
      cudaGetLastError();
      trim();
      if (cudaMalloc(&b.p, bytes) != cudaSuccess) return false;
    }
    if (cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming) != cudaSuccess) {
      cudaFree(b.p);
      return false;
    }
    {
      std::lock_guard<std::mutex> g(lock);
      out += bytes;
    }
    look();
    return true;
  }
  // back from a call whose work on stream s still uses it
  void put(Block b, cudaStream_t s, const void* owner) {
    std::lock_guard<std::mutex> g(lock);
    out -= b.bytes;
    if (scarce || b.bytes > keep || cudaEventRecord(b.done, s) != cudaSuccess) {
      cudaGetLastError();
      cudaFree(b.p);   // waits for the work
      cudaEventDestroy(b.done);
      return;
    }
    drop(keep - b.bytes, MOST - 1);
    b.used = ++uses;
    b.owner = owner;
    blocks[n++] = b;
  }
  // what is held unused back to the device
  void trim() {
    if (pool) cudaMemPoolTrimTo(pool, 0);
    std::lock_guard<std::mutex> g(lock);
    drop(0, 0);
  }
  // asks the device; bytes free there or held unused here
  size_t look() {
    size_t freeb = pool_unused(), devb = 0, totb = 0;
    cudaMemGetInfo(&devb, &totb);
    std::lock_guard<std::mutex> g(lock);
    for (int q = 0; q < n; ++q) freeb += blocks[q].bytes;
    freeb += devb;
    scarce = freeb + out < totb / 4;
    plans = 0;
    return freeb;
  }
  // Bytes a call may plan with: free device memory and what is held unused.  need: the arrays of its largest batch, in the order
  // in which it will take them.  The call plans the same with any figure of twice their sum or more, so the device (0.1 to 1 ms)
  // is not asked every time where what is held will serve every one of them (a block that serves a small array may leave no
  // room for the others).
  size_t plan(std::initializer_list<size_t> need) {
    {
      std::lock_guard<std::mutex> g(lock);
      bool taken[MOST] = {}, ok = true;
      size_t sum = 0, small = 0;
      for (size_t bytes : need) {
        sum += bytes;
        if (bytes < BIG) { small += bytes; continue; }
        const int at = fit(bytes, taken);
        if (at >= 0) taken[at] = true;
        else ok = false;
      }
      if (ok && pool_unused() / 2 >= small && ++plans < LOOK) return 2 * sum;
    }
    return look();
  }
  // before a call takes `need` of the freeb bytes that it may plan with: where that is most of them, what is held goes back,
  // so that no array sits in a block of up to twice its size and leaves too little for the others
  void room(size_t need, size_t freeb) {
    if (need > freeb / 2) trim();
  }

 private:
  size_t pool_unused() const {
    uint64_t held = 0, used = 0;
    if (!pool || cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess || held <= used)
      return 0;
    return (size_t)(held - used);
  }
  // the held block that serves an array (-1: none), of those not taken
  int fit(size_t bytes, const bool* taken) const {
    int at = -1;
    for (int q = 0; q < n; ++q)
      if (!taken[q] && blocks[q].bytes >= bytes && blocks[q].bytes / 2 <= bytes && (at < 0 || blocks[q].bytes < blocks[at].bytes)) at = q;
    return at;
  }
  // held blocks down to `most` bytes and `count` (under the lock)
  void drop(size_t most, int count) {
    size_t sum = 0;
    for (int q = 0; q < n; ++q) sum += blocks[q].bytes;
    while (sum > most || n > count) {
      int old = 0;
      for (int q = 1; q < n; ++q)
        if (blocks[q].used < blocks[old].used) old = q;
      sum -= blocks[old].bytes;
      release(old);
    }
  }
  void release(int q) {
    cudaFree(blocks[q].p);
    cudaEventDestroy(blocks[q].done);
    blocks[q] = blocks[--n];
  }
};

// the store of a device (up to 64 in a machine); never destroyed
inline DevStore* dev_store(int device) {
  static DevStore* st = new DevStore[64];
  return st + (device & 63);
}

// An array that outlives the call (an operator's tables, a supercell's, a context's slab) from the device: where there is
// no room for it, what the store holds unused goes back first.
template <typename T>
bool dev_alloc(DevStore* st, cudaStream_t s, T** p, size_t bytes) {
  if (cudaMalloc(p, bytes) == cudaSuccess) return true;
  cudaGetLastError();
  if (st) {
    cudaStreamSynchronize(s);
    st->trim();
    if (cudaMalloc(p, bytes) == cudaSuccess) return true;
    cudaGetLastError();
  }
  *p = nullptr;
  return false;
}

// the store, stream and context that the calling thread's temporaries belong to (set for the length of an entry point)
struct CallMem {
  DevStore* store = nullptr;
  cudaStream_t stream = nullptr;
  const void* owner = nullptr;
};
inline CallMem& call_mem() {
  static thread_local CallMem c;
  return c;
}
struct MemScope {
  CallMem prev;
  MemScope(DevStore* store, cudaStream_t s, const void* owner) : prev(call_mem()) { call_mem() = CallMem{store, s, owner}; }
  ~MemScope() {
    DevStore* st = call_mem().store;
    if (st && st != prev.store && st->scarce) {   // the call's own arrays have gone back before
      cudaStreamSynchronize(call_mem().stream);
      st->trim();
    }
    call_mem() = prev;
  }
  MemScope(const MemScope&) = delete;
  MemScope& operator=(const MemScope&) = delete;
};

// one device allocation of a call, from the call's store (in the order of its stream, and given back to it), else from the
// device
struct DevMem {
  void* p = nullptr;
  CallMem c;
  DevStore::Block b{};
  bool get(size_t bytes) {
    c = call_mem();
    b = DevStore::Block{};
    if (c.store && bytes >= DevStore::BIG) {
      if (c.store->get(bytes, c.stream, b)) { p = b.p; return true; }
    } else if (c.store && c.store->pool) {
      if (cudaMallocFromPoolAsync(&p, bytes, c.store->pool, c.stream) == cudaSuccess) return true;
      cudaGetLastError();
      cudaStreamSynchronize(c.stream);   // what is held unused back to the device, then once more
      c.store->trim();
      if (cudaMallocFromPoolAsync(&p, bytes, c.store->pool, c.stream) == cudaSuccess) return true;
    } else {
      c.store = nullptr;
      if (cudaMalloc(&p, bytes) == cudaSuccess) return true;
    }
    cudaGetLastError();
    p = nullptr;
    return false;
  }
  void put() {
    if (!p) return;
    if (!c.store) cudaFree(p);
    else if (b.p) c.store->put(b, c.stream, c.owner);
    else cudaFreeAsync(p, c.stream);
    p = nullptr;
  }
};

}  // namespace asrb
