// nq_handle.h -- the handle behind the C ABI (include/nqueens_gb300.h) and the
// device buffers it owns; shared by the translation units that implement the
// ABI (nq_capi.cu, nq_unique.cu).  Not installed.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/nqueens_gb300.h"

namespace nq {

// Device buffer.  With a stream set, allocation and release are stream-ordered on
// that stream, from the handle's pool, so building or freeing one batch never
// waits for kernels of other batches still running.
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  cudaStream_t ordered = nullptr;
  cudaMemPool_t pool = nullptr;
  cudaError_t ensure(size_t n) {
    if (n <= cap) return cudaSuccess;
    release();
    size_t want = std::max<size_t>(n, 256);
    cudaError_t e = ordered ? cudaMallocFromPoolAsync(&p, want, pool, ordered) : cudaMalloc(&p, want);
    if (e == cudaSuccess) cap = want; else p = nullptr;
    return e;
  }
  void release() {
    if (p) { if (ordered) cudaFreeAsync(p, ordered); else cudaFree(p); }
    p = nullptr; cap = 0;
  }
};

// Control block of a batch run: totals (u64 per job), then the queue cursor
// (u64), the error word (u32) and the blocks that have ended (u32) at
// totals_bytes + 0 / + 8 / + 12.
struct Ctrl {
  static size_t bytes(int njobs) { return (size_t)njobs * 8 + 16; }
};

// Control block of a single-N run (device, zeroed before each run):
//   job total (u64), queue cursor (u64), error word (u32), deepest schedule (u32),
//   split queue length (u64), blocks of the DFS that have ended (u32), pad, device clock (ns, u64 x 3) at the start
//   of prepare, the start of the DFS and its end; behind them, zeroed when a list is
//   generated on the device: the states of each level (u32 x 7) and its error word (u32).
namespace ctl {
constexpr size_t kTotal = 0, kCursor = 8, kErr = 16, kTmax = 20, kSplit = 24, kDone = 32, kStamp = 40, kBytes = 64;
constexpr size_t kGen = 64, kGenErr = 92, kAll = 96;
}

// What a completion query runs on: a stream, a buffer and a pinned block for its control block.  Up to kSmall bytes the
// buffer is plain memory, in powers of two; what takes more comes from the handle's pool (which takes 32 MiB from the
// device at a time) and is given back to it without waiting for other streams.
struct QueryRun {
  static constexpr size_t kSmall = 16ull << 20;
  cudaStream_t stream = nullptr;
  DevBuf small, large;
  uint64_t* host = nullptr;
  cudaError_t ensure(size_t n, unsigned char** p) {
    size_t s = 256 << 10;
    while (s < n && s <= kSmall) s *= 2;
    DevBuf& b = s <= kSmall ? small : large;
    const cudaError_t e = b.ensure(s <= kSmall ? s : n);
    *p = (unsigned char*)b.p;
    return e;
  }
};

}  // namespace nq

struct nq_handle {
  int device = 0;
  int sms = 0;
  cudaStream_t stream = nullptr;
  int block = 64, grid = 0, split = -1;    // split: -1 automatic, 0..3 fixed depth
  std::string err;
  nq::DevBuf rec, root, info, sched, per_task, ctrl, sroot;
  nq::DevBuf gen, starts;                // device generator: the other state buffer, the start list
  nq::DevBuf utasks, uconfs, uctl;       // unique counter (nq_count_unique)
  // Completion queries: each runs on a stream and buffers of its own, so queries of several threads, and one beside an
  // asynchronous count, do not wait for each other.  Up to kQueryRuns of them are kept for the next queries, one of
  // them with what its largest query took.
  static constexpr size_t kQueryRuns = 8;
  std::vector<nq::QueryRun*> q_free;
  std::mutex q_mu;
  cudaError_t query_get(nq::QueryRun** out) {
    {
      std::lock_guard<std::mutex> lk(q_mu);
      if (!q_free.empty()) { *out = q_free.back(); q_free.pop_back(); return cudaSuccess; }
    }
    cudaError_t e = ensure_pool();
    if (e != cudaSuccess) return e;
    nq::QueryRun* q = new (std::nothrow) nq::QueryRun();
    if (!q) return cudaErrorMemoryAllocation;
    e = cudaStreamCreateWithFlags(&q->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess && !(q->host = (uint64_t*)pin_get(256))) e = cudaErrorMemoryAllocation;
    if (e != cudaSuccess) { query_free(q); return e; }
    q->large.ordered = q->stream; q->large.pool = pool;
    *out = q;
    return cudaSuccess;
  }
  void query_put(nq::QueryRun* q) {
    {
      std::lock_guard<std::mutex> lk(q_mu);
      if (q_free.size() < kQueryRuns) {
        for (nq::QueryRun* f : q_free)
          if (f->large.p) q->large.release();
        q_free.insert(q->large.p ? q_free.end() : q_free.begin(), q);     // the one with a large buffer is taken next
        return;
      }
    }
    query_free(q);
  }
  void query_free(nq::QueryRun* q) {
    q->large.release();
    if (q->stream) { cudaStreamSynchronize(q->stream); cudaStreamDestroy(q->stream); }
    q->small.release();
    pin_put(q->host);
    delete q;
  }
  nq::DevBuf okeys, oorder, ohist;       // queue order (nq_set_queue_order)
  int queue_order = 0;                   // 0: generator / split order, 1: largest estimated subtree first
  int64_t chunk_records = 0;             // records per chunk of nq_count (0: the library default)
  int64_t last_chunks = 0, last_records = 0;   // chunks and records of the last nq_count
  cudaEvent_t done = nullptr;            // recorded after the last asynchronous count (nq_sync waits on it)
  uint64_t* h_ctrl = nullptr;   // pinned read-back of the control block
  size_t h_ctrl_cap = 0;
  uint32_t* h_result = nullptr; // pinned, the control block as the last run's DFS left it, ...
  bool result_written = false;  // ... if that run launched one
  bool stamped = false;         // the last run's times stand in h_result, not in ev
  // Device memory of batches: a pool of the handle's own that keeps up to kPoolKeep bytes between batches (what
  // is above goes back to the device when a stream of it synchronises, all of it with the handle).  From the
  // device's default pool, which keeps nothing, each batch mapped its memory anew: build + run +
  // release of 4 jobs of N=8..10 177 + 35 + 92 us against 85 + 26 + 17 now, of 64 mixed jobs of N=9..16 490 + 765 + 189
  // against 307 + 765 + 22.
  static constexpr uint64_t kPoolKeep = 256ull << 20;
  cudaMemPool_t pool = nullptr;
  std::mutex pool_mu;
  cudaError_t ensure_pool() {
    std::lock_guard<std::mutex> lk(pool_mu);
    if (pool) return cudaSuccess;
    cudaMemPoolProps p{};
    p.allocType = cudaMemAllocationTypePinned;
    p.location.type = cudaMemLocationTypeDevice;
    p.location.id = device;
    cudaError_t e = cudaMemPoolCreate(&pool, &p);
    if (e != cudaSuccess) { pool = nullptr; return e; }
    uint64_t keep = kPoolKeep;
    return cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  // pinned read-back blocks for batches, reused (freeing pinned memory can
  // synchronise the device, which would stall other batches in flight)
  std::mutex pin_mu;
  std::vector<std::pair<void*, size_t>> pin_free;
  void* pin_get(size_t bytes) {
    {
      std::lock_guard<std::mutex> lk(pin_mu);
      for (size_t i = 0; i < pin_free.size(); i++)
        if (pin_free[i].second >= bytes) {
          void* q = pin_free[i].first;
          pin_free.erase(pin_free.begin() + (long)i);
          pinned_sizes[q] = bytes;
          return q;
        }
    }
    const size_t want = std::max<size_t>(bytes, 65536);
    void* q = nullptr;
    if (cudaMallocHost(&q, want) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(pin_mu);
    pinned_cap[q] = want;
    pinned_sizes[q] = bytes;
    return q;
  }
  void pin_put(void* q) {
    if (!q) return;
    std::lock_guard<std::mutex> lk(pin_mu);
    pin_free.push_back({q, pinned_cap[q]});
  }
  std::map<void*, size_t> pinned_cap, pinned_sizes;
  bool pending = false;
  int last_split = 0;        // split depth and queue length of the last run
  int64_t last_queue = 0;
  bool queue_on_device = false;   // its length stands in the control block, not yet in last_queue
  // events around the last run's kernels (same stream as the launches)
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};

  int fail(int status, const char* fmt, ...) {
    char buf[512];
    va_list ap; va_start(ap, fmt); vsnprintf(buf, sizeof buf, fmt, ap); va_end(ap);
    err = buf;
    return status;
  }
  int cuda_fail(cudaError_t e, const char* where) {
    return fail(e == cudaErrorMemoryAllocation ? NQ_ENOMEM : NQ_ECUDA, "%s: %s", where, cudaGetErrorString(e));
  }
  int ensure_pinned(size_t bytes) {
    if (bytes <= h_ctrl_cap) return NQ_OK;
    if (h_ctrl) cudaFreeHost(h_ctrl);
    h_ctrl = nullptr; h_ctrl_cap = 0;
    bytes = std::max<size_t>(bytes, 4096);
    cudaError_t e = cudaMallocHost((void**)&h_ctrl, bytes);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMallocHost");
    h_ctrl_cap = bytes;
    return NQ_OK;
  }
};

#define NQ_CUDA(h, call)                                     \
  do {                                                       \
    cudaError_t _e = (call);                                 \
    if (_e != cudaSuccess) return (h)->cuda_fail(_e, #call); \
  } while (0)
