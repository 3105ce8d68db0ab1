// nq_internal.h -- internal interface between the C-ABI layer (nq_capi.cu),
// the host task builders (nq_host.cpp) and the sm_103a kernels
// (nq_kernels.cu).  Not installed; the public interface is
// include/nqueens_gb300.h.
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace nq {

// Device-side error bits (OR-ed into a device word, read back by the host).
constexpr uint32_t DERR_SHIFT = 1u;      // a record needs a negative shift (reference would raise)
constexpr uint32_t DERR_DEPTH = 2u;      // a task's schedule is deeper than the launch's stack
constexpr uint32_t DERR_NOTERM = 4u;     // a schedule never reaches a base frame
constexpr uint32_t DERR_BADN = 8u;       // N outside 6..27 in a task
constexpr uint32_t DERR_FORMAT = 16u;    // a schedule op does not fit the compact word's fields

// Levels every task is expanded by before the DFS.  `rows`: rows left below the shallowest start (N - 2 -
// start row), which sets a task's work (about 4x per row).  Lanes of a warp share their work at the end of
// the queue, so splitting only has to even out the warps and give a short list more items than lanes:
// us of a whole call on GB300 at D = 0 / 1 / 2 / 3, m tasks:
//   8 rows (N=12):    m=4300   48 / 46 / 46 / 52
//   9 rows (N=13):    m=7731   62 / 54 / 55 / 62
//   10 rows (N=14):   m=1000   57 / 47 / 46 / 62       m=13233 80 / 67 / 70 / 127
//   12 rows (N=16):   m=4000  161 / 126 / 113 / 145    m=33046 601 / 343 / 322 / 421
//   13 rows (N=17):   m=49207 3326 / 1570 / 1450 / 1655
//   13 rows (N=18):   m=16000 903 / 696 / 420 / 475    m=200000 4864 / 3522 / 3661 / 4390
//   14 rows (N=19):   m=100   749 / 192 / 122 / 149    m=4000 1544 / 1161 / 703 / 543
//                     m=50000 9.9 / 4.7 / 4.0 / 4.4 ms    m=897071 67.2 / 64.4 / 67.4 ms
//   15 rows (N=20):   m=1000  4.1 / 1.7 / 1.5 / 0.75 ms   m=16000 20.6 / 12.4 / 7.4 / 6.7 ms
// A level makes 4.5 (N=14) to 8 (N=20 and more) times the items, and an item costs its loading; lists of 10^5 tasks and more are balanced at D = 1.
inline int choose_split(int64_t m, int rows) {
  if (rows <= 8) return 0;
  if (m > 100000) return m > 400000000 ? 0 : 1;   // ~7 subtasks a task stay within the u32 subtask queue
  if (rows >= 15 ? m < 20000 : rows == 14 && m >= 512 && m < 8192) return 3;
  return 2;
}

template <bool WIDE> struct QueryWord { using type = uint32_t; };
template <> struct QueryWord<true> { using type = uint2; };

// Prepared task arrays (structure of arrays, one entry per task).
struct TaskArrays {
  uint4* root = nullptr;      // {ld, rd, col, avail} of the root frame
  uint32_t* info = nullptr;   // info word (T, wexp, root count, N, status)
  void* sched = nullptr;      // per-task schedule words, stride `sw` words
  int sw = 0;                 // schedule words per task (>= T+1 of every task)
  bool wide = false;          // uint2 words (queries with far-reaching steps) instead of uint32
  bool ra_words = false;      // compact words carry RA (else it is in the roots' rd)
};

struct DfsLaunch {
  TaskArrays tasks;
  const uint4* sroot = nullptr;         // split queue: subtask frames ...
  const uint2* sinfo = nullptr;         // ... and {task, depth | job << 5}; nullptr: the task stands in the frames' w
  uint32_t depth = 0;                   // and all are at this depth (job 0); no sroot either: the queue holds the tasks
  int64_t m = 0;                        // queue length ...
  const unsigned long long* m_dev = nullptr;   // ... or where it stands on the device; above qcap the DFS does nothing
  unsigned long long qcap = 0;
  int64_t m_bound = 0;                  // bound of a length on the device, 0: none
  const uint32_t* order = nullptr;      // optional queue order (task index per slot)
  unsigned long long* cursor = nullptr; // queue cursor (device, zeroed before launch; 64-bit, so it never wraps)
  unsigned long long* job_totals = nullptr;  // weighted totals, slot (job id - job_base) (device)
  uint32_t job_base = 0;
  unsigned long long* per_task = nullptr;    // optional weighted count per task (device)
  unsigned int* err = nullptr;          // device error word
  int maxt = 0;                         // stack frames per lane (>= T of every task; words: maxt+1)
  bool big = false;                     // u64 per-task counters (some task has N >= 24)
  int block = 128;
  int grid = 0;                         // 0: one wave of resident blocks
  // Optional: the last block to end copies ctl_words u64 of the control block to pinned host memory (blocks_done:
  // zeroed before), so the caller only waits for the stream.
  const uint32_t* ctl = nullptr;
  unsigned ctl_words = 0;
  unsigned int* blocks_done = nullptr;
  uint32_t* host_ctl = nullptr;
  unsigned long long* stamp = nullptr;  // optional: the device clock at its start and (with host_ctl) at its end
  bool chained = false;                 // the kernel before it in the stream calls chain_next
};

// Prepare: records {ld, rd, col, startijkl} (the reference's 16-byte task
// record) -> task arrays at `offset`.  m_dev: the records' number stands on the
// device and m bounds it.  tmax: atomicMax of the schedule depth T over the
// launch's tasks; n_out: their number.
cudaError_t launch_prepare(int N, int64_t m, const unsigned int* m_dev, const uint4* records, const TaskArrays& out,
                           int64_t offset, unsigned int* err, cudaStream_t st, unsigned int* tmax, unsigned int* n_out);

// Prepare and split a single-N list (compact words) in one launch: tasks, and for D = 1..3 the queue of their
// depth-D frames {ld, rd, col, task} (qn counts them, also past qcap, where nothing is written any more) and the counts settled
// above depth D.  D = 0 writes the tasks' roots instead, which are the queue.
struct PrepareSplit {
  int N = 0;
  int64_t m = 0;                        // records ...
  const unsigned int* m_dev = nullptr;  // ... or where their number stands on the device (the launch covers m_max)
  const uint4* rec = nullptr;
  uint4* root = nullptr;                // D = 0
  uint32_t* info = nullptr;
  uint32_t* sched = nullptr;
  int sw = 0;
  bool ra_words = false;                // RA in the words; else (ra_in_rd holds) in the queue frames' rd
  unsigned int* err = nullptr;
  unsigned int* tmax = nullptr;         // optional
  unsigned long long* per_task = nullptr;    // optional; set for every task
  uint4* sroot = nullptr;               // D > 0
  unsigned long long qcap = 0;
  unsigned long long* qn = nullptr;     // zeroed before
  unsigned long long* total = nullptr;
  unsigned long long* stamp = nullptr;  // optional: the device clock at its start
};
cudaError_t launch_prepare_split(int D, int64_t m_max, const PrepareSplit& a, cudaStream_t st);

cudaError_t launch_dfs(const DfsLaunch& L, cudaStream_t st);

// Records of start constellations at a preset of 4..8, on the device: `starts` (device array of packed ijkl),
// or all of a board's where it is null (n_starts then bounds them).  gn[0..] receives the states of each
// level, gn[gen_levels(preset)] the records, which end in buf0 when the level count is even, else in buf1
// (`cap` records each; the caller bounds them).  gn zeroed before.
inline int gen_levels(int preset) { return preset - 3; }     // start constellations hold 3 or 4 queens
constexpr int kGenFused = 2;     // up to so many levels one launch makes the records: into the last buffer, the other stays untouched
cudaError_t launch_generate(int N, int preset, unsigned n_starts, const int* starts, uint4* buf0, uint4* buf1, unsigned cap,
                            unsigned* gn, unsigned* err, int sms, cudaStream_t st);

// A completion query as one task: root frame, terminal depth and device words (wide; compact queries use x).
struct QueryParam {
  uint4 root;
  uint32_t N, T;
  unsigned target;              // frames that are enough
  uint32_t words_wide;          // the words' form
  uint2 words[28];
};
// Its control block (u64 words): total, queue cursor, error word and DFS blocks that have ended, queue length
// after each level.
struct QueryCtl {
  static constexpr unsigned kTotal = 0, kCursor = 1, kErr = 2, kQueue = 3, kWords = 7;
};
struct QueryBuffers {
  unsigned long long* ctl;
  uint32_t* info;               // one task
  void* sched;
  uint4* tmp;                   // cap[0] frames
  uint4* sroot[4];              // the queue from one block, and after one to three levels over the whole GPU
  uint2* sinfo[4];
  unsigned cap[4];              // items each holds; the block's own, [0], always fits
};
// Writes the task, its queue and the control block, the queue expanded by `levels` (0..3) more levels.  A
// level longer than its buffer leaves its ctl[kQueue + ..] above its cap: what comes behind it does nothing.
cudaError_t launch_query(const QueryParam& p, const QueryBuffers& b, bool wide, int levels, int sms, cudaStream_t st);

// Batches.  A list holds sources: the tasks of a board's records (depth 0), or the frames a query was expanded
// to.  Jobs of one board share a list.
struct BatchList {
  uint32_t src0;                // its first source in src
  uint32_t task0;               // its first task, or the query's one
  uint32_t query, D;            // D: levels to expand the sources by
};
struct ListState {              // on the device, zeroed before the build
  unsigned int n, depth;        // sources, their depth
  unsigned long long items, settled;   // queue items, weighted counts settled above them
};
struct BatchJob { unsigned long long base; uint32_t off0, list, job, pad; };   // items from base on; off0: the list's first source in off
struct ListArgs {
  int n;                        // ranges (lists, or jobs)
  unsigned long long total;     // sources in them, padded to warps
  const unsigned long long* ends;
  const BatchList* lists;
  ListState* state;
  const uint4* src;
  const uint32_t* info;
  const void* sched;
  int sw;
  uint32_t* off;                // per source: its first item in the list's queue
};
cudaError_t launch_list_count(const ListArgs& a, bool wide, cudaStream_t st);
cudaError_t launch_list_write(const ListArgs& a, const BatchJob* jobs, uint4* sroot, uint2* sinfo, bool wide, cudaStream_t st);
// The queries' tasks and frames (state n and depth), one block each; frames in src and tmp (no level has more than cap).
struct BatchQuery { QueryParam p; uint32_t list, src0, tmp0, task, cap; };
cudaError_t launch_batch_queries(int n, const BatchQuery* q, uint4* src, uint4* tmp, ListState* state, const TaskArrays& ta,
                                 cudaStream_t st);

// Queue order, largest estimated subtree first: order[0..m) receives the queue
// indices (subtasks when sroot is set, else tasks); keys: m bytes of scratch,
// hist_offs: 512 u32 of scratch.
cudaError_t launch_order(int64_t m, const uint4* sroot, const TaskArrays& ta, uint8_t* keys,
                         unsigned int* hist_offs, uint32_t* order, cudaStream_t st);

// Largest block count per SM for a given stack depth (occupancy query).
int dfs_blocks_per_sm(bool wide, int block, int maxt);

// INT32 throughput probe: grid x 256 threads x iters x 128 instructions of
// one kind (0 lop3, 1 add, 2 shf, 3 mix).
cudaError_t int_peak(int kind, int iters, int grid, uint32_t* out, cudaStream_t st);
size_t dfs_smem_bytes(bool wide, int block, int maxt);

#ifdef __CUDACC__
// Chains of short kernels: launch_after lets a kernel's blocks be placed while the kernel before it in the stream
// still runs.  They wait at chain_wait, which every such kernel calls before it touches memory (in a plain launch
// it returns at once), until that kernel has ended and its writes are visible; what it writes is read through
// pointers without __restrict__, which would promise that nobody writes it while they run.  chain_next, at the top of a
// kernel, lets the launch behind it be placed once all of its own blocks have been.  A boundary between two
// kernels costs 1 to 2.5 us less so: a completion query of N=10 / N=17 31.7 / 106 us, 29.5 / 99 chained; a
// unique count of N=12 79 us, 57.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid); c.blockDim = dim3(block); c.dynamicSmemBytes = smem; c.stream = st;
  c.attrs = &at; c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void chain_next() { cudaTriggerProgrammaticLaunchCompletion(); }

// The device's clock in ns.
__device__ __forceinline__ unsigned long long device_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Called by all threads of all blocks as their last step: the last block to end copies `words` u64 of the control
// block `ctl` to pinned host memory (`done`: zeroed before).  A copy queued behind the kernel instead takes the
// copy engine's start and end: completion query of N=10 / N=17 36 / 129 us with one, 31.7 / 106 so.  `end`:
// optional, a word of ctl that receives the device's clock.
__device__ __forceinline__ void hand_over(const uint32_t* ctl, unsigned words, unsigned* done, uint32_t* host,
                                          unsigned long long* end = nullptr) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x >= 32u) return;
  unsigned n = 0;
  if (threadIdx.x == 0u) {
    n = atomicAdd(done, 1u);
    if (n == gridDim.x - 1u && end) *(volatile unsigned long long*)end = device_ns();
    __threadfence();
  }
  if (__shfl_sync(0xFFFFFFFFu, n, 0) != gridDim.x - 1u) return;
  __syncwarp();
  const volatile unsigned long long* from = (const volatile unsigned long long*)ctl;
  volatile unsigned long long* to = (volatile unsigned long long*)host;
  constexpr unsigned kAtOnce = 8;         // loads in flight a lane: a batch's block (258 of them) copied one by one took 15 us
  for (unsigned w0 = threadIdx.x; w0 < words; w0 += 32u * kAtOnce) {
    unsigned long long v[kAtOnce];
#pragma unroll
    for (unsigned k = 0; k < kAtOnce; k++) v[k] = w0 + 32u * k < words ? from[w0 + 32u * k] : 0ull;
#pragma unroll
    for (unsigned k = 0; k < kAtOnce; k++)
      if (w0 + 32u * k < words) to[w0 + 32u * k] = v[k];
  }
}

// position of the r-th set bit of m (r < popc(m))
__device__ __forceinline__ uint32_t nth_set(uint32_t m, uint32_t r) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t w = 16; w; w >>= 1) {
    const uint32_t c = __popc(m & ((1u << w) - 1u));
    if (r >= c) { r -= c; m >>= w; pos += w; }
  }
  return pos;
}
#endif

}  // namespace nq
