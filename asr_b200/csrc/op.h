// Internal types of the asr_b200 library: context, operator (device node tables) and the kernel-side views.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <vector>

#include "common.cuh"

struct asr_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;      // the stream every call runs on
  cudaStream_t own_stream = nullptr;  // created by asr_ctx_create
  int num_sms = 148;
  int64_t nchain = 0, nlev = 0, nfall = 0;
  int64_t launches = 0;   // kernels launched by this context
  int* d_err = nullptr;   // device error word
  // kernel timing (asr_ctx_profile): device time, launches and algorithmic work per kernel kind (ASR_KERNEL_*)
  struct ProfStat {
    double ms = 0.0, bytes = 0.0, flops = 0.0;
    int64_t launches = 0;
  };
  int profile = 0;
  ProfStat prof[ASR_KERNEL_KINDS];
  std::vector<cudaEvent_t> ev_pool;   // pairs (start, end) of the timed launches
  std::vector<int> ev_kind;           // kernel kind of every recorded pair
  int ev_used = 0;                    // pairs recorded and not yet read
  // starts a timed region on stream s (returns its pair index, -1 when profiling is off); regions may nest (a level of
  // the reverse sweep and its kernels); no synchronisation
  int prof_start(cudaStream_t s) {
    if (!profile) return -1;
    while ((int)ev_pool.size() < 2 * (ev_used + 1)) {
      cudaEvent_t e;
      if (cudaEventCreate(&e) != cudaSuccess) return -1;
      ev_pool.push_back(e);
    }
    if ((int)ev_kind.size() < ev_used + 1) ev_kind.resize(ev_used + 1);
    if (cudaEventRecord(ev_pool[2 * ev_used], s) != cudaSuccess) return -1;
    ev_kind[ev_used] = -1;   // open until prof_stop
    return ev_used++;
  }
  // ends the region `slot` of prof_start as one launch of `kind` with the given algorithmic bytes and flops
  void prof_stop(cudaStream_t s, int slot, int kind, double bytes, double flops) {
    if (slot < 0 || slot >= ev_used || ev_kind[slot] != -1) return;
    if (cudaEventRecord(ev_pool[2 * slot + 1], s) != cudaSuccess) return;
    ev_kind[slot] = kind;
    prof[kind].bytes += bytes;
    prof[kind].flops += flops;
    prof[kind].launches += 1;
  }
  unsigned char* cf_scratch = nullptr;   // device address of asr_cf_eval_noalloc's static array (resolved on first use)
  // the adjoint's vector slab, kept between calls while ws_hold is set (asr_ctx_hold_workspace)
  int ws_hold = 0;
  void* ws = nullptr;
  size_t ws_bytes = 0;
  // The memory of a call's temporaries (DevMem) stays with the context, so that a call neither maps nor unmaps device memory
  // (cudaMalloc and cudaFree of a chain batch's vectors took 10-50 ms a call, a second when the device's other processes did
  // the same).  Arrays of BIG bytes or more are blocks of the device's allocator, at most `keep` bytes of them held between
  // calls (the least recently used go first); smaller ones come from a stream-ordered pool that holds at most POOL_KEEP.  (The
  // pool for all sizes: mapping a 20 GB array that it had given back took a second.)  All of it goes back with the context,
  // when hold_workspace is switched off, when an allocation would fail, and after a call that found less than a quarter of
  // the device free.
  static constexpr size_t BIG = (size_t)32 << 20, POOL_KEEP = (size_t)256 << 20;
  struct Block {
    void* p;
    size_t bytes;
    cudaEvent_t done;   // after the last use
    uint64_t used;
  };
  std::mutex mem_lock;
  std::vector<Block> blocks;   // held, not in use
  uint64_t uses = 0;
  size_t keep = 0;
  bool scarce = false;
  cudaMemPool_t pool = nullptr;
  // a block of at least `bytes` for work on stream s: the smallest held one of up to twice that (a larger one is wanted by a
  // larger array of the same call), else a new one (false: out of memory)
  bool block_get(size_t bytes, cudaStream_t s, Block& b) {
    {
      std::lock_guard<std::mutex> g(mem_lock);
      int at = -1;
      for (int q = 0; q < (int)blocks.size(); ++q)
        if (blocks[q].bytes >= bytes && blocks[q].bytes / 2 <= bytes && (at < 0 || blocks[q].bytes < blocks[at].bytes)) at = q;
      if (at >= 0) {
        b = blocks[at];
        blocks.erase(blocks.begin() + at);
        if (cudaStreamWaitEvent(s, b.done, 0) == cudaSuccess) return true;
        cudaGetLastError();
        blocks.push_back(b);
        return false;
      }
    }
    b = Block{nullptr, bytes, nullptr, 0};
    if (cudaMalloc(&b.p, bytes) != cudaSuccess) {
      cudaGetLastError();
      mem_trim(0);
      if (cudaMalloc(&b.p, bytes) != cudaSuccess) return false;
    }
    if (cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming) == cudaSuccess) return true;
    cudaFree(b.p);
    return false;
  }
  // back from a call whose work on stream s still uses it
  void block_put(Block b, cudaStream_t s) {
    const size_t most = scarce ? 0 : keep;
    if (b.bytes > most || cudaEventRecord(b.done, s) != cudaSuccess) {
      cudaGetLastError();
      cudaFree(b.p);   // waits for the work
      cudaEventDestroy(b.done);
      return;
    }
    mem_trim(most - b.bytes, false);
    std::lock_guard<std::mutex> g(mem_lock);
    b.used = ++uses;
    blocks.push_back(b);
  }
  // held memory down to `most` bytes of blocks
  void mem_trim(size_t most, bool with_pool = true) {
    if (with_pool && pool) cudaMemPoolTrimTo(pool, 0);
    std::lock_guard<std::mutex> g(mem_lock);
    size_t sum = 0;
    for (const Block& b : blocks) sum += b.bytes;
    while (sum > most) {
      size_t old = 0;
      for (size_t q = 1; q < blocks.size(); ++q)
        if (blocks[q].used < blocks[old].used) old = q;
      sum -= blocks[old].bytes;
      cudaFree(blocks[old].p);
      cudaEventDestroy(blocks[old].done);
      blocks.erase(blocks.begin() + old);
    }
  }
  // Bytes a call may plan with: free device memory and what the context holds unused, the held slab with it.  A call that
  // needs at most `need` bytes for its largest batch plans the same with any figure of twice that or more, so the device (0.1
  // to 1 ms) is asked only where what is held would not do.
  size_t plan_bytes(size_t need = SIZE_MAX / 2) {
    size_t freeb = 0, devb = 0, totb = 0;
    {
      std::lock_guard<std::mutex> g(mem_lock);
      for (const Block& b : blocks) {
        freeb += b.bytes;
        if (b.bytes >= need && b.bytes / 2 <= need) return 2 * need;
      }
    }
    uint64_t held = 0, used = 0;
    if (pool && cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && held > used) {
      if ((size_t)(held - used) / 2 >= need) return 2 * need;
      freeb += (size_t)(held - used);
    }
    cudaMemGetInfo(&devb, &totb);
    freeb += devb;
    scarce = freeb < totb / 4;
    return freeb + ws_bytes;
  }
  void ws_release() {
    if (ws) cudaFree(ws);
    ws = nullptr;
    ws_bytes = 0;
  }
};

namespace asrb {

// the context whose pool the calling thread's temporaries come from (set for the length of an entry point)
inline asr_ctx*& pool_ctx() {
  static thread_local asr_ctx* c = nullptr;
  return c;
}
struct PoolScope {
  asr_ctx* prev;
  explicit PoolScope(asr_ctx* c) : prev(pool_ctx()) { pool_ctx() = c; }
  ~PoolScope() { pool_ctx() = prev; }
  PoolScope(const PoolScope&) = delete;
  PoolScope& operator=(const PoolScope&) = delete;
};
#define ASR_ENTER(ctx_)          \
  ASR_ON_DEVICE((ctx_)->device); \
  ::asrb::PoolScope pool_call_(ctx_)

// one device allocation of a call, from the context (in the order of its stream, and given back to it), else from the device
struct DevMem {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  asr_ctx* c = nullptr;
  asr_ctx::Block b{};
  bool get(size_t bytes) {
    c = pool_ctx();
    b = asr_ctx::Block{};
    s = c ? c->stream : nullptr;
    if (c && bytes >= asr_ctx::BIG) {
      if (c->block_get(bytes, s, b)) { p = b.p; return true; }
    } else if (c && c->pool) {
      if (cudaMallocFromPoolAsync(&p, bytes, c->pool, s) == cudaSuccess) return true;
      cudaGetLastError();
      cudaStreamSynchronize(s);   // what the context holds unused back to the device, then once more
      c->mem_trim(0);
      if (cudaMallocFromPoolAsync(&p, bytes, c->pool, s) == cudaSuccess) return true;
    } else {
      c = nullptr;
      if (cudaMalloc(&p, bytes) == cudaSuccess) return true;
    }
    cudaGetLastError();
    p = nullptr;
    return false;
  }
  void put() {
    if (!p) return;
    if (!c) cudaFree(p);
    else if (b.p) c->block_put(b, s);
    else cudaFreeAsync(p, s);
    p = nullptr;
  }
};

// Device view of the node tables, passed by value to the kernels.  Node indices are 0-based, -1 = absent link;
// operation indices 0-based.  Layouts follow the reference: flipr/flipg (nsmax, nn) and hopr/hopg (nslot, nn) with the
// state / slot index fastest, i.e. hopr[k + nslot * i].
struct OpView {
  int nn, nslot, nsmax, nop, ncls, nsp, ntype;
  const int* site;        // (nn) 1-based graph site
  const int8_t* lst;      // (nn) own local state
  const int8_t* ncl;      // (nn) 0-based class
  const int8_t* typ;      // (nn) 0-based site type (stype of the site)
  const int8_t* start;    // (nn) 1 if the node sits on the start site
  const int8_t* frozen;   // (nn) operator-level frozen species (0: none)
  const double* sq;       // (nn) sqrt(orbit size)
  const double* isq;      // (nn) 1 / sqrt(orbit size)
  const int8_t* nflip;    // (nn) flip links to other nodes
  const int* flipr;       // (nsmax, nn)
  const uint8_t* flipg;
  const int* hopr;        // (nslot, nn)
  const uint8_t* hopg;
  const int* stab_ptr;    // (nn + 1) 0-based offsets
  const uint8_t* stab;    // (nstab)
  const int8_t* nsc;      // (ncls) species per class
  const uint8_t* pi;      // (9, nop) 0-based orbital permutation: D(g)[pi(l), l] = sg(l)
  const uint16_t* sgm;    // (nop) bit l set: sg(l, g) = -1
};

}  // namespace asrb

struct asr_op {
  asr_ctx* ctx = nullptr;
  int nn = 0, nslot = 0, nsmax = 0, nop = 0, ncls = 0, nsp = 0, ntype = 1, nsite = 0, nstab = 0, start_site = 1;
  int start_l = 1;
  // batch shape chosen by asr_autotune per precision (index 0 FP64, 1 FP32); 0: the built-in defaults
  int tuned_tpb[2] = {0, 0}, tuned_npw[2] = {0, 0};
  int tuned_link[2] = {0, 0};             // 1: the step kernel's fixed-offset link gathers (chosen by asr_autotune)
  double tuned_link_ms[2][2] = {{-1.0, -1.0}, {-1.0, -1.0}};   // device ms of the general / fixed-offset step at the tuned shape
  // host copies of the model and group
  std::vector<int> nsc, spc;       // spc(ldspc, ncls)
  int ldspc = 1;
  std::vector<double> mt;          // (nsm, nsm, nsm, ncls)
  std::vector<int> pi;             // (9, nop) 1-based
  std::vector<double> sg, chi, dmat;
  std::vector<double> block;       // (9, 9, nslot, ntype) unrotated bond blocks
  std::vector<double> block0;      // (9, 9, ntype)
  std::vector<double> c, d, o, e;  // (9, nsp) current operator parameters
  std::vector<int8_t> frozen_h;    // (nn) operator-level frozen species
  // host copies of what a freeze reads (device node order), fetched from the device tables on the first freeze: the site,
  // the own local state and the number of flip links of every node, and the class of the start node
  std::vector<int> site_h;
  std::vector<int8_t> lst_h, nflip_h;
  int start_class = -1;
  // device node order: the tables live in a locality order (reverse Cuthill-McKee of the hop graph, start node first);
  // old_of_new[n] is the reference (build) index of device node n, new_of_old its inverse; empty: the build order
  std::vector<int> old_of_new, new_of_old;
  int dev_node(int old) const { return new_of_old.empty() ? old : new_of_old[old]; }
  int ref_node(int dev) const { return old_of_new.empty() ? dev : old_of_new[dev]; }
  // device tables
  int* d_site = nullptr;
  int* d_level = nullptr;
  int* d_orb = nullptr;
  int8_t *d_lst = nullptr, *d_ncl = nullptr, *d_typ = nullptr, *d_start = nullptr, *d_frozen = nullptr, *d_nflip = nullptr;
  double *d_sq = nullptr, *d_isq = nullptr;
  int *d_flipr = nullptr, *d_hopr = nullptr, *d_stab_ptr = nullptr;
  uint8_t *d_flipg = nullptr, *d_hopg = nullptr, *d_stab = nullptr;
  int8_t* d_nsc = nullptr;
  uint8_t* d_pi = nullptr;
  uint16_t* d_sgm = nullptr;
  double* d_blocks = nullptr;   // [t][kk][l][l'] kk = 0: on-site block, kk = 1 + slot
  float* d_blocks_f = nullptr;
  asrb::OpView view() const {
    return asrb::OpView{nn, nslot, nsmax, nop, ncls, nsp, ntype, d_site, d_lst, d_ncl, d_typ, d_start, d_frozen,
                        d_sq, d_isq, d_nflip, d_flipr, d_flipg, d_hopr, d_hopg, d_stab_ptr, d_stab, d_nsc, d_pi, d_sgm};
  }
};

namespace asrb {
// graph_build.cu
int build_operator(asr_ctx* ctx, int nsite, const int* nbr_ptr, const int* nbr, int ncls, const int* nsc, const int* cls,
                   const int* perm, int nop, int start, int maxlevel, int maxrank, const int* flippable, const int* stype,
                   asr_op* op, const int* tsite = nullptr, int ntarget = 0, int* tnode = nullptr, int* tgop = nullptr);
// flip links of every node (graph_build.cu), from the tables and classes on the device
int count_flips(asr_ctx* ctx, asr_op* op);
// host helpers (capi.cu)
void class_mt(const double* conc, int nsc, int nsm, double* mt);
}  // namespace asrb
