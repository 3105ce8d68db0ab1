// nq_capi.cu -- the extern "C" boundary of libnqgpu.so (include/nqueens_gb300.h).
//
// Owns device memory, streams, error reporting and the launch sequence:
//   records (host or device) -> prepare_kernel -> dfs_kernel -> totals.
// The library has no CPU counting path: every count is computed by the
// kernels in nq_kernels.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <map>
#include <mutex>
#include <cstdarg>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/nqueens_gb300.h"
#include "nq_common.cuh"
#include "nq_host.h"
#include "nq_handle.h"
#include "nq_internal.h"

using namespace nq;

namespace {

int preset_for(int N) {
  if (N >= 5 && N <= 17) return 5;
  if (N >= 18 && N <= 21) return 6;
  if (N >= 22 && N <= 24) return 7;
  if (N >= 25 && N <= 27) return 8;
  return 5;
}

int derr_to_status(uint32_t e) {
  if (e & DERR_DEPTH) return NQ_ESTACK;
  if (e & DERR_SHIFT) return NQ_EPRESET;
  if (e) return NQ_EINVAL;
  return NQ_OK;
}

const char* derr_text(uint32_t e) {
  if (e & DERR_DEPTH) return "a task's schedule is deeper than the launch's stack";
  if (e & DERR_SHIFT) return "a record needs a negative shift (preset too deep for N)";
  if (e & DERR_NOTERM) return "a task's schedule never reaches a base frame";
  if (e & DERR_BADN) return "task with N outside 6..27";
  if (e & DERR_FORMAT) return "a schedule op does not fit the compact schedule word";
  return "ok";
}

// Records per chunk of a whole-board count (nq_count): one chunk up to N=21
// (2.0 M records), four at N=22 (28.7 M), about 32 MB of host records each.
constexpr int64_t kChunkRecords = 8 << 20;
constexpr size_t kStage = 4096;      // pinned read-back block: uploads are staged behind its first bytes

int maxt_for(int N, int start_min) {
  // Terminal-parent depth T <= N - 3 - start; one frame of margin.
  int s = start_min < 0 ? 1 : start_min;
  int m = N - 2 - s;
  return std::max(1, std::min(m, kMaxDepth - 1));
}

}  // namespace

namespace {


// Lists up to this length run without a read-back between the launches: the DFS takes the queue's length
// from the device and stacks for the deepest task the start rows allow.  Longer ones read the queue's length
// and the deepest schedule first (18 us with the events), which buys a tighter stack (more resident warps).
// us without / with, records of N=15 16385 95 / 112, 21270 107 / 125, N=16 20000 216 / 234, 33046 305 / 314 (rows
// left up to 12); N=17 16385 583 / 585, 30000 952 / 930, 49207 1468 / 1412, N=19 20000 1858 / 1787.
int64_t no_read_back(int rows) { return rows <= 12 ? 65536 : 16384; }
constexpr int64_t kQueueBytes = 256 << 20;   // queue buffer a short list may bound its queue by

// records (device) -> counts on st; totals land in ctrl[0].  One launch prepares and splits, one counts.
// start_min bounds the records' schedules; t_max, where the caller knows it, is the deepest one's T.
// m_dev: the list's length stands there (u32) and m bounds it.
int run_records(nq_handle* h, int N, const uint4* d_rec, int64_t m, int start_min, unsigned long long* d_per_task,
                cudaStream_t st, int t_max = kMaxDepth, const unsigned int* m_dev = nullptr) {
  const int maxt = maxt_for(N, start_min);
  const int D = h->split >= 0 ? h->split : choose_split(m, maxt);
  NQ_CUDA(h, cudaSetDevice(h->device));
  NQ_CUDA(h, h->info.ensure((size_t)m * sizeof(uint32_t)));
  NQ_CUDA(h, h->sched.ensure((size_t)m * (maxt + 1) * sizeof(uint32_t)));
  NQ_CUDA(h, h->ctrl.ensure(ctl::kAll));
  if (int s = h->ensure_pinned(ctl::kAll)) return s;
  if (!h->h_result) NQ_CUDA(h, cudaMallocHost((void**)&h->h_result, ctl::kAll));
  h->result_written = false;
  unsigned char* c = (unsigned char*)h->ctrl.p;
  PrepareSplit P;
  P.N = N; P.m = m; P.m_dev = m_dev; P.rec = d_rec; P.info = (uint32_t*)h->info.p; P.sched = (uint32_t*)h->sched.p; P.sw = maxt + 1;
  P.ra_words = !ra_in_rd(N, start_min, D);
  P.err = (unsigned int*)(c + ctl::kErr); P.tmax = (unsigned int*)(c + ctl::kTmax);
  P.per_task = d_per_task; P.qn = (unsigned long long*)(c + ctl::kSplit); P.total = (unsigned long long*)(c + ctl::kTotal);
  // Queue capacity: a bound (each level places a queen in one of at most N - 2, N - 3, ... columns) where that
  // is small, else 8 a level (measured: up to 8), built again if it was too small.  Where the device has not that
  // much, the first launch only counts the queue, and it is built at its length.
  uint64_t bound = (uint64_t)m, guess = (uint64_t)m + 1024;
  for (int d = 0; d < D; d++) { bound *= (uint64_t)(N - 2 - d); guess *= 8; }
  bool read_back = (m > no_read_back(maxt) && !m_dev) || h->queue_order == 1 || (D > 0 && bound * sizeof(uint4) > (uint64_t)kQueueBytes);
  if (D > 0) {
    const uint64_t q = std::max(read_back ? std::min(bound, guess) : bound, (uint64_t)(h->sroot.cap / sizeof(uint4)));
    cudaError_t e = h->sroot.ensure((size_t)q * sizeof(uint4));
    if (e == cudaErrorMemoryAllocation) { cudaGetLastError(); read_back = true; e = cudaSuccess; }
    NQ_CUDA(h, e);
  } else {
    NQ_CUDA(h, h->root.ensure((size_t)m * sizeof(uint4)));
    P.root = (uint4*)h->root.p;
  }
  DfsLaunch L;
  L.tasks.root = (uint4*)h->root.p; L.tasks.info = P.info; L.tasks.sched = P.sched; L.tasks.sw = P.sw; L.tasks.wide = false; L.tasks.ra_words = P.ra_words;
  L.cursor = (unsigned long long*)(c + ctl::kCursor); L.job_totals = P.total;
  L.per_task = d_per_task; L.err = P.err; L.block = h->block; L.grid = h->grid;
  L.m = m;
  // Where nothing is read back between the launches, the kernels stamp their times themselves and the DFS's blocks
  // are placed while the first launch runs: an event between two launches keeps them apart by 3.5 us (counts of
  // 8 boards of 6..13: 380 us with the three events, 291 without).
  h->stamped = !read_back;
  if (read_back) NQ_CUDA(h, cudaEventRecord(h->ev[0], st));
  else P.stamp = (unsigned long long*)(c + ctl::kStamp);
  for (bool zeroed = m_dev != nullptr;; zeroed = false) {   // with m_dev, by the list's generator
    P.sroot = (uint4*)h->sroot.p;
    P.qcap = h->sroot.cap / sizeof(uint4);
    if (!zeroed) NQ_CUDA(h, cudaMemsetAsync(c, 0, ctl::kBytes, st));
    NQ_CUDA(h, launch_prepare_split(D, m, P, st));
    if (D > 0) { L.sroot = P.sroot; L.depth = (uint32_t)D; }
    if (!read_back) {
      if (D > 0 || m_dev) { L.m_dev = P.qn; L.qcap = D > 0 ? P.qcap : ~0ull; L.m_bound = (int64_t)std::min<uint64_t>(bound, 1ull << 40); }
      L.maxt = std::max(1, std::min(maxt, t_max) - D);
      break;
    }
    // Subtasks start at depth D with an empty stack, so the DFS needs T - D frames and T - D + 1 schedule
    // words per lane; the kernel still rejects any task deeper than that.
    NQ_CUDA(h, cudaMemcpyAsync(h->h_ctrl, c, ctl::kBytes, cudaMemcpyDeviceToHost, st));
    NQ_CUDA(h, cudaStreamSynchronize(st));
    const unsigned char* hc = (const unsigned char*)h->h_ctrl;
    L.maxt = std::max(1, std::min(maxt, (int)*(const uint32_t*)(hc + ctl::kTmax) - D));
    const uint64_t ns = *(const uint64_t*)(hc + ctl::kSplit);     // D = 0: the list's length
    if (D == 0) { L.m = (int64_t)ns; break; }
    if (ns > 0xFFFFFFFFull) return h->fail(NQ_ENOMEM, "split: %llu subtasks", (unsigned long long)ns);
    L.m = (int64_t)ns;
    if (ns <= P.qcap) break;
    NQ_CUDA(h, h->sroot.ensure((size_t)ns * sizeof(uint4)));
  }
  L.big = counts_need_u64(N, D > 0 && !read_back ? m : L.m);
  if (h->queue_order == 1) {
    NQ_CUDA(h, h->okeys.ensure((size_t)std::max<int64_t>(L.m, 1)));
    NQ_CUDA(h, h->oorder.ensure((size_t)std::max<int64_t>(L.m, 1) * sizeof(uint32_t)));
    NQ_CUDA(h, h->ohist.ensure(512 * sizeof(unsigned int)));
    NQ_CUDA(h, launch_order(L.m, L.sroot, L.tasks, (uint8_t*)h->okeys.p, (unsigned int*)h->ohist.p,
                            (uint32_t*)h->oorder.p, st));
    L.order = (const uint32_t*)h->oorder.p;
  }
  h->last_split = D; h->last_queue = L.m; h->queue_on_device = L.m_dev != nullptr;
  if (read_back) NQ_CUDA(h, cudaEventRecord(h->ev[1], st));
  else { L.chained = true; L.stamp = P.stamp + 1; }
  L.ctl = (const uint32_t*)c; L.ctl_words = ctl::kAll / 8; L.blocks_done = (unsigned int*)(c + ctl::kDone); L.host_ctl = h->h_result;
  NQ_CUDA(h, launch_dfs(L, st));
  h->result_written = L.m > 0 || L.m_dev;
  if (read_back) NQ_CUDA(h, cudaEventRecord(h->ev[2], st));
  return NQ_OK;
}

int read_ctrl(nq_handle* h, cudaStream_t st, uint64_t* total) {
  if (int s = h->ensure_pinned(ctl::kAll)) return s;
  if (!h->result_written) NQ_CUDA(h, cudaMemcpyAsync(h->h_ctrl, h->ctrl.p, ctl::kAll, cudaMemcpyDeviceToHost, st));
  NQ_CUDA(h, cudaStreamSynchronize(st));
  if (h->result_written) std::memcpy(h->h_ctrl, h->h_result, ctl::kAll);
  const unsigned char* hc = (const unsigned char*)h->h_ctrl;
  const uint32_t e = *(const uint32_t*)(hc + ctl::kErr);
  if (h->queue_on_device) h->last_queue = (int64_t)*(const uint64_t*)(hc + ctl::kSplit);
  if (e) return h->fail(derr_to_status(e), "device: %s", derr_text(e));
  if (total) *total = *(const uint64_t*)(hc + ctl::kTotal);
  return NQ_OK;
}

// Queue of a completion query: one block expands it to a target of frames and more, then the whole GPU by another
// one to three levels where the rows left make the frames large.  One block writes its 2,000 to 20,000 frames no
// faster than the whole GPU writes ten times as many, so it stops early where three levels are enough for the lanes.
// us of a query (mean of six), target 2048 and levels 0 / 1 / 2 / 3 from 0 / 11 / 13 / 16 rows against target 512 and
// 0 / 10 / 11 / 13 rows: N=12 two queens (10 rows) 35 / 35, N=14 one (13) 52 / 51, N=15 one 80 / 75, N=16 two 66 / 62,
// N=17 two (15) 122 / 120, N=18 four 54 / 51; with 16 rows and more 2048 stays: N=19 three 250 / 258, N=20 three 965 /
// 985.  Two levels there took 2118 us at N=19 with two queens (three 1630), one level
// 42 us at N=12 with two queens where none took 36 (from the target of 2048).
constexpr unsigned kQueryCap = 65536;
constexpr unsigned kQueryTarget = 2048;      // ... and of each query of a batch
unsigned query_target(int rows) { return rows >= 16 ? kQueryTarget : 512u; }
// The queue has room for the frames expected after each level (query_estimate), up to this many: a level less where
// more come, or the device has no room.  After three levels 0.04 to 5 10^6 items of 24 bytes are in it for N=15..23, 8
// to 20 10^6 for N=24..27 with two queens, and the level before them has a quarter at most.
constexpr unsigned kQueryMost = 5 << 20, kQueryMost2 = kQueryMost / 4;
int query_levels(int rows) { return rows >= 13 ? 3 : rows >= 11 ? 2 : rows >= 10 ? 1 : 0; }
// A batch's queries share the lanes with its other jobs, so the same need not be cut as fine.
int batch_query_levels(int rows) { return rows >= 15 ? 2 : rows >= 12 ? 1 : 0; }

// The most frames a level of a query's expansion has: only levels below the target are expanded, and a frame of
// depth d has at most as many candidates as columns are left there.
uint64_t query_frames(const QueryParam& p) {
  const uint64_t columns = (uint64_t)p.T + 2;      // left at the root
  uint64_t n = 1, most = 1;
  for (uint32_t d = 0; d < p.T; d++) {
    n = std::min<uint64_t>(n, p.target) * (columns - d);
    most = std::max(most, n);
  }
  return most;
}

// Frames expected at each depth 0..T of a query's expansion: a row's squares off the pre-placed queens' lines, less
// those that each queen of the rows above takes at random (its column and, on the board, two diagonals).  Diagonals that
// meet on a square count twice, so the product stands a little above the frames there are: from the first depth with
// the target's number on, 5,572 queries of N=8..27 had at most 0.88 / 0.78 / 0.66 of it after one / two / three levels.
void query_estimate(const QueryParam& p, double est[kMaxDepth]) {
  const double inv = 1.0 / p.N;
  double left[kMaxN];                        // of a row's squares, after a queen so many rows above
  for (uint32_t r = 1; r < p.N; r++) left[r] = 1.0 - (3.0 - 2.0 * r * inv) * inv;
  const uint32_t bm = (1u << p.N) - 1u;
  uint32_t ld = p.root.x, rd = p.root.y, row = 0, at[kMaxDepth];
  est[0] = 1.0;
  for (uint32_t d = 0; d < p.T; d++) {
    at[d] = row;
    double a = __builtin_popcount(bm & ~(ld | rd | p.root.z));
    for (uint32_t j = 0; j < d; j++) a *= left[row - at[j]];
    est[d + 1] = est[d] * a;
    const uint32_t x = p.words[d].x, step = x & W_S;         // both forms of the words hold the step and LA alike
    ld = (ld << step) | (x >> (32 - step));
    rd = (rd >> step) | p.words[d].y;
    row += step;
  }
}

// Room for the queue after 0..levels levels over the GPU.  The block stops at the first depth with `target` frames: the
// first with that many expected or, where fewer come there, the next, from less than the target.
void query_caps(const QueryParam& p, const double est[kMaxDepth], int levels, unsigned cap[4]) {
  uint32_t d = 0;
  while (d < p.T && est[d] < p.target) d++;
  cap[0] = (unsigned)query_frames(p);
  for (int l = 1; l <= levels; l++) {
    double n = 0.0;                    // at the terminal depth, which frames do not pass, the ones before it
    for (uint32_t k = d; k <= std::min(d + l, p.T); k++) n = std::max(n, est[k]);
    for (uint32_t k = d; k <= std::min(d + l + 1, p.T); k++) n = std::max(n, est[k] * std::min(1.0, p.target / est[d]));
    const double most = l == 2 && levels == 3 ? kQueryMost2 : kQueryMost;
    cap[l] = (unsigned)std::min(n + 512.0, most);
  }
}

// The query as a device task.  Returns 1, 0 when the count is settled here (*fixed), or -1 on bad arguments.
// The last free row holds one column for every board, so its parent row is the task's terminal depth (count
// the child if its row has a free square), as in constellation tasks.
int query_task(int N, int k, const int* rows, const int* cols, QueryParam* p, bool* wide, uint64_t* fixed) {
  uint32_t root[4];
  Op ops[kMaxDepth + 1];
  int n = 0;
  *fixed = 0;
  const int s = completion_root(N, k, rows, cols, root, ops, &n);
  if (s < 0) return -1;
  if (s != 0 || n == 1) {
    *fixed = s == 2 ? 1 : s == 0 ? (uint64_t)__builtin_popcount(root[3]) : 0;
    return 0;
  }
  p->root = make_uint4(root[0], root[1], root[2], root[3]);
  p->N = (uint32_t)N; p->T = (uint32_t)(n - 2); p->target = 0;
  *wide = false;
  for (int d = 0; d <= n - 2; d++) *wide = *wide || ops[d].ra != 0u || !compact_fits(ops[d], N);   // no RA in compact words
  p->words_wide = *wide ? 1u : 0u;
  for (int d = 0; d <= n - 2; d++)
    p->words[d] = *wide ? make_uint2(device_wide_x(ops[d]), ops[d].ra) : make_uint2(device_compact(ops[d], false), 0u);
  return 1;
}

// A compact query's words in the wide form.
void widen_query(QueryParam* p) {
  for (uint32_t d = 0; d <= p->T; d++) {
    const Op o = unpack_compact(p->words[d].x ^ C_NOLOOK, (int)p->N, false);
    p->words[d] = make_uint2(device_wide_x(o), 0u);
  }
  p->words_wide = 1;
}

}  // namespace

// ---------------------------------------------------------------------------
extern "C" {

const char* nq_version(void) { return "nqueens-gb300 0.1 (sm_103a)"; }

const char* nq_strerror(int s) {
  switch (s) {
    case NQ_OK: return "ok";
    case NQ_EINVAL: return "invalid argument";
    case NQ_ESTACK: return "task deeper than the launch's stack";
    case NQ_ETIMEOUT: return "bounded wait ran out";
    case NQ_ECUDA: return "CUDA error";
    case NQ_ENOMEM: return "out of memory";
    case NQ_EPRESET: return "preset too deep for N";
    case NQ_EBUSY: return "still running";
    default: return "unknown status";
  }
}

int nq_create(nq_handle** out, int device) {
  if (!out) return NQ_EINVAL;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) return NQ_ECUDA;
  nq_handle* h = new (std::nothrow) nq_handle();
  if (!h) return NQ_ENOMEM;
  h->device = device;
  if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaEventCreate(&h->ev[0]) != cudaSuccess || cudaEventCreate(&h->ev[1]) != cudaSuccess ||
      cudaEventCreate(&h->ev[2]) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->done, cudaEventDisableTiming) != cudaSuccess) {
    nq_destroy(h);
    return NQ_ECUDA;
  }
  *out = h;
  return NQ_OK;
}

void nq_destroy(nq_handle* h) {
  if (!h) return;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (QueryRun* q : h->q_free) h->query_free(q);
  h->rec.release(); h->root.release(); h->info.release(); h->sched.release(); h->per_task.release(); h->ctrl.release();
  h->sroot.release(); h->gen.release(); h->starts.release();
  h->okeys.release(); h->oorder.release(); h->ohist.release();
  h->utasks.release(); h->uconfs.release(); h->uctl.release();
  if (h->h_ctrl) cudaFreeHost(h->h_ctrl);
  if (h->h_result) cudaFreeHost(h->h_result);
  for (auto& q : h->pinned_cap) cudaFreeHost(q.first);
  for (auto& e : h->ev) if (e) cudaEventDestroy(e);
  if (h->done) cudaEventDestroy(h->done);
  if (h->pool) cudaMemPoolDestroy(h->pool);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

int nq_int32_peak(nq_handle* h, int kind, double* ops_per_s) {
  if (!h || !ops_per_s || kind < 0 || kind > 3) return NQ_EINVAL;
  NQ_CUDA(h, cudaSetDevice(h->device));
  NQ_CUDA(h, h->ctrl.ensure(Ctrl::bytes(1)));
  int per = 0;
  NQ_CUDA(h, cudaDeviceGetAttribute(&per, cudaDevAttrMaxThreadsPerMultiProcessor, h->device));
  const int grid = h->sms * std::max(1, per / 256);
  const int iters = 4096;
  cudaStream_t st = h->stream;
  NQ_CUDA(h, int_peak(kind, 64, grid, (uint32_t*)h->ctrl.p, st));   // warm-up
  double best = 0.0;
  for (int rep = 0; rep < 3; rep++) {
    NQ_CUDA(h, cudaEventRecord(h->ev[0], st));
    NQ_CUDA(h, int_peak(kind, iters, grid, (uint32_t*)h->ctrl.p, st));
    NQ_CUDA(h, cudaEventRecord(h->ev[1], st));
    NQ_CUDA(h, cudaEventSynchronize(h->ev[1]));
    float ms = 0.f;
    NQ_CUDA(h, cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]));
    const double ops = (double)grid * 256.0 * (double)iters * 128.0;
    best = std::max(best, ops / (ms * 1e-3));
  }
  *ops_per_s = best;
  return NQ_OK;
}

int nq_last_run_info(const nq_handle* h, int* split_depth, int64_t* queued) {
  if (!h) return NQ_EINVAL;
  if (split_depth) *split_depth = h->last_split;
  if (!queued) return NQ_OK;
  *queued = h->last_queue;
  if (h->pending && h->queue_on_device) {      // its length comes with the run's result
    if (cudaSetDevice(h->device) != cudaSuccess || cudaEventSynchronize(h->done) != cudaSuccess) return NQ_ECUDA;
    *queued = (int64_t)*(const uint64_t*)((const unsigned char*)h->h_result + ctl::kSplit);
  }
  return NQ_OK;
}

int nq_last_kernel_ms(nq_handle* h, float* prepare_ms, float* dfs_ms) {
  if (!h) return NQ_EINVAL;
  NQ_CUDA(h, cudaSetDevice(h->device));
  float a = 0.f, b = 0.f;
  if (h->stamped) {                       // asynchronous runs have recorded `done`; the others have ended
    if (h->pending) NQ_CUDA(h, cudaEventSynchronize(h->done));
    uint64_t t[3];
    std::memcpy(t, (const unsigned char*)h->h_result + ctl::kStamp, sizeof t);
    if (prepare_ms) *prepare_ms = (float)((double)(t[1] - t[0]) * 1e-6);
    if (dfs_ms) *dfs_ms = (float)((double)(t[2] - t[1]) * 1e-6);
    return NQ_OK;
  }
  NQ_CUDA(h, cudaEventSynchronize(h->ev[2]));
  NQ_CUDA(h, cudaEventElapsedTime(&a, h->ev[0], h->ev[1]));
  NQ_CUDA(h, cudaEventElapsedTime(&b, h->ev[1], h->ev[2]));
  if (prepare_ms) *prepare_ms = a;
  if (dfs_ms) *dfs_ms = b;
  return NQ_OK;
}

int nq_device_sms(const nq_handle* h, int* sms) {
  if (!h || !sms) return NQ_EINVAL;
  *sms = h->sms;
  return NQ_OK;
}

int nq_device_name(const nq_handle* h, char* buf, size_t cap) {
  if (!h || !buf || cap == 0) return NQ_EINVAL;
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, h->device) != cudaSuccess) return NQ_ECUDA;
  snprintf(buf, cap, "%s", p.name);
  return NQ_OK;
}

int nq_last_error(const nq_handle* h, char* buf, size_t cap) {
  if (!h || !buf || cap == 0) return NQ_EINVAL;
  snprintf(buf, cap, "%s", h->err.c_str());
  return NQ_OK;
}

int nq_set_config(nq_handle* h, int block, int grid, int split_depth) {
  if (!h) return NQ_EINVAL;
  if (block != 64 && block != 128 && block != 256) return h->fail(NQ_EINVAL, "block must be 64, 128 or 256");
  if (grid < 0 || split_depth < -1 || split_depth > 3) return h->fail(NQ_EINVAL, "bad grid or split depth");
  h->block = block; h->grid = grid; h->split = split_depth;
  return NQ_OK;
}

int nq_set_queue_order(nq_handle* h, int mode) {
  if (!h) return NQ_EINVAL;
  if (mode != 0 && mode != 1) return h->fail(NQ_EINVAL, "queue order must be 0 or 1");
  h->queue_order = mode;
  return NQ_OK;
}

int nq_get_queue_order(const nq_handle* h, int* mode) {
  if (!h || !mode) return NQ_EINVAL;
  *mode = h->queue_order;
  return NQ_OK;
}

int nq_get_config(const nq_handle* h, int* block, int* grid, int* split_depth) {
  if (!h) return NQ_EINVAL;
  if (block) *block = h->block;
  if (grid) *grid = h->grid;
  if (split_depth) *split_depth = h->split;
  return NQ_OK;
}

int nq_preset_for(int N) { return preset_for(N); }

int64_t nq_gen_constellations(int N, int preset, nq_record* out, int64_t cap) {
  std::vector<GenRecord> v;
  const int s = gen_constellations(N, preset, v, 0);
  if (s == -1) return NQ_EINVAL;
  if (s == -2) return NQ_EPRESET;
  const int64_t n = (int64_t)v.size();
  if (out && cap >= n)
    for (int64_t i = 0; i < n; i++)
      out[i] = nq_record{(uint32_t)v[i].ld, (uint32_t)v[i].rd, (uint32_t)v[i].col, v[i].startijkl};
  return n;
}

int64_t nq_gen_constellations_wide(int N, int preset, uint64_t* ld, uint64_t* rd, uint64_t* col, uint32_t* sijkl,
                                   int64_t cap) {
  std::vector<GenRecord> v;
  const int s = gen_constellations(N, preset, v, 0);
  if (s == -1) return NQ_EINVAL;
  if (s == -2) return NQ_EPRESET;
  const int64_t n = (int64_t)v.size();
  if (ld && rd && col && sijkl && cap >= n)
    for (int64_t i = 0; i < n; i++) { ld[i] = v[i].ld; rd[i] = v[i].rd; col[i] = v[i].col; sijkl[i] = v[i].startijkl; }
  return n;
}

int nq_exec_solutions(nq_handle* h, int N, const nq_record* records, int64_t m, uint64_t* solutions, uint64_t* total) {
  if (!h || !total || m < 0 || (m > 0 && !records)) return h ? h->fail(NQ_EINVAL, "null argument") : NQ_EINVAL;
  if (N < 6 || N > kMaxN) return h->fail(NQ_EINVAL, "exec_solutions: N=%d outside 6..27", N);
  if (m > (int64_t)0x7FFFFFFF) return h->fail(NQ_EINVAL, "too many records");
  *total = 0;
  if (m == 0) return NQ_OK;
  cudaStream_t st = h->stream;
  NQ_CUDA(h, cudaSetDevice(h->device));
  const int smin = (int)start_row_min(&records[0].startijkl, m, 4);
  NQ_CUDA(h, h->rec.ensure((size_t)m * sizeof(nq_record)));
  NQ_CUDA(h, cudaMemcpyAsync(h->rec.p, records, (size_t)m * sizeof(nq_record), cudaMemcpyHostToDevice, st));
  unsigned long long* pt = nullptr;
  if (solutions) {
    NQ_CUDA(h, h->per_task.ensure((size_t)m * 8));
    pt = (unsigned long long*)h->per_task.p;
  }
  if (int s = run_records(h, N, (const uint4*)h->rec.p, m, smin, pt, st)) return s;
  if (solutions) NQ_CUDA(h, cudaMemcpyAsync(solutions, pt, (size_t)m * 8, cudaMemcpyDeviceToHost, st));
  return read_ctrl(h, st, total);
}

int nq_exec_solutions_device(nq_handle* h, int N, const nq_record* d_records, int64_t m, int start_min,
                             uint64_t* d_solutions, uint64_t* d_total, void* stream) {
  if (!h || !d_total || m < 0 || (m > 0 && !d_records)) return h ? h->fail(NQ_EINVAL, "null argument") : NQ_EINVAL;
  if (N < 6 || N > kMaxN) return h->fail(NQ_EINVAL, "exec_solutions: N=%d outside 6..27", N);
  if (m > (int64_t)0x7FFFFFFF) return h->fail(NQ_EINVAL, "too many records");
  cudaStream_t st = stream ? (cudaStream_t)stream : h->stream;
  NQ_CUDA(h, cudaSetDevice(h->device));
  if (m == 0) {
    NQ_CUDA(h, cudaMemsetAsync(d_total, 0, 8, st));
    return NQ_OK;
  }
  // A captured call would have no run for nq_sync to wait for, and long lists synchronise: none is captured.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  NQ_CUDA(h, cudaStreamIsCapturing(st, &cap));
  if (cap != cudaStreamCaptureStatusNone) return h->cuda_fail(cudaErrorStreamCaptureUnsupported, "exec_solutions_device");
  if (int s = run_records(h, N, (const uint4*)d_records, m, start_min, (unsigned long long*)d_solutions, st)) return s;
  NQ_CUDA(h, cudaMemcpyAsync(d_total, h->ctrl.p, 8, cudaMemcpyDeviceToDevice, st));
  NQ_CUDA(h, cudaEventRecord(h->done, st));
  h->pending = true;
  return NQ_OK;
}

int nq_sync(nq_handle* h) {
  if (!h) return NQ_EINVAL;
  NQ_CUDA(h, cudaSetDevice(h->device));
  if (!h->pending) {                      // nothing asynchronous outstanding: the handle's own stream
    NQ_CUDA(h, cudaStreamSynchronize(h->stream));
    return NQ_OK;
  }
  // waits for this handle's last count only (its event), not for other handles, batches or streams
  NQ_CUDA(h, cudaEventSynchronize(h->done));
  h->pending = false;
  return read_ctrl(h, h->stream, nullptr);
}

int nq_debug_task_schedule(int N, nq_record rec, uint32_t root[4], uint32_t* info, uint32_t* words, int cap) {
  if (N < 6 || N > kMaxN || !root || !info || (cap > 0 && !words) || cap < 0) return NQ_EINVAL;
  const TaskHead t = decode_record(N, rec.ld, rec.rd, rec.col, rec.startijkl);
  if (t.status != TS_OK) return NQ_EPRESET;
  Root rt;
  uint32_t rc = 0;
  Op ops[kMaxDepth];
  const int T = walk_schedule(N, t, &rt, &rc, ops, std::min(cap, kMaxDepth));
  if (T == -2) return NQ_ESTACK;
  root[0] = rt.ld; root[1] = rt.rd; root[2] = rt.col; root[3] = (T < 0) ? 0u : rt.avail;
  *info = info_pack(T < 0 ? INFO_NO_DFS : (uint32_t)T, (uint32_t)t.wexp, rc, (uint32_t)N, TS_OK);
  if (T < 0) return 0;
  for (int d = 0; d <= T; d++) {
    if (!compact_fits(ops[d], N)) return NQ_EINVAL;
    words[d] = pack_compact(ops[d]);
  }
  return T + 1;
}

int64_t nq_debug_board_states(int N, int preset) { return (int64_t)board_states(N, preset); }

int64_t nq_debug_completion_tasks(int N, int k, const int* rows, const int* cols, int min_tasks, uint32_t* roots,
                                  uint32_t* infos, uint32_t* words, int stride, int64_t cap, uint64_t* fixed_count) {
  if (k < 0 || k > 8 || (k > 0 && (!rows || !cols)) || stride < 1) return NQ_EINVAL;
  std::vector<HostTask> v;
  int mt = 0;
  const int s = build_completion_tasks(N, k, rows, cols, min_tasks, 0, v, &mt);
  if (s < 0) return NQ_EINVAL;
  if (fixed_count) *fixed_count = (s == 2) ? 1 : 0;
  const int64_t n = (int64_t)v.size();
  if (cap >= n && n > 0) {
    if (!roots || !infos || !words) return NQ_EINVAL;
    for (int64_t i = 0; i < n; i++) {
      if (v[i].T + 1 > stride) return NQ_ESTACK;
      for (int q = 0; q < 4; q++) roots[i * 4 + q] = v[i].root[q];
      infos[i] = v[i].info;
      for (int d = 0; d <= v[i].T; d++) {
        words[(i * stride + d) * 2] = v[i].sched[2 * d];
        words[(i * stride + d) * 2 + 1] = v[i].sched[2 * d + 1];
      }
    }
  }
  return n;
}

int nq_count_completions(nq_handle* h, int N, int k, const int* rows, const int* cols, uint64_t* count);

int nq_tune(nq_handle* h, int N, int repeats, int* best_block, int* best_split, float* best_ms) {
  if (!h || repeats < 1) return h ? h->fail(NQ_EINVAL, "tune: bad arguments") : NQ_EINVAL;
  if (N < 6 || N > kMaxN) return h->fail(NQ_EINVAL, "tune: N=%d outside 6..27", N);
  std::vector<GenRecord> v;
  const int g = gen_constellations(N, preset_for(N), v, 0);
  if (g != 0) return h->fail(g == -2 ? NQ_EPRESET : NQ_EINVAL, "tune: generator failed for N=%d", N);
  const int64_t m = (int64_t)v.size();
  if (m == 0) return h->fail(NQ_EINVAL, "tune: no tasks for N=%d", N);
  std::vector<nq_record> r((size_t)m);
  for (int64_t i = 0; i < m; i++) r[i] = nq_record{(uint32_t)v[i].ld, (uint32_t)v[i].rd, (uint32_t)v[i].col, v[i].startijkl};
  cudaStream_t st = h->stream;
  NQ_CUDA(h, cudaSetDevice(h->device));
  const int smin = (int)start_row_min(&r[0].startijkl, m, 4);
  NQ_CUDA(h, h->rec.ensure((size_t)m * sizeof(nq_record)));
  NQ_CUDA(h, cudaMemcpyAsync(h->rec.p, r.data(), (size_t)m * sizeof(nq_record), cudaMemcpyHostToDevice, st));
  const int old_block = h->block, old_split = h->split;
  float best = 1e30f;
  int bb = old_block, bs = old_split;
  uint64_t want = 0;
  bool have_total = false;
  for (int b : {64, 128, 256})
    for (int s = 0; s <= 3; s++) {
      h->block = b; h->split = s;
      for (int k = 0; k <= repeats; k++) {           // first run warms up, then `repeats` timed runs
        uint64_t total = 0;
        int st_run = run_records(h, N, (const uint4*)h->rec.p, m, smin, nullptr, st);
        if (st_run == NQ_OK) st_run = read_ctrl(h, st, &total);
        if (st_run != NQ_OK) { h->block = old_block; h->split = old_split; return st_run; }
        if (!have_total) { want = total; have_total = true; }
        if (total != want) {
          h->block = old_block; h->split = old_split;
          return h->fail(NQ_ECUDA, "tune: N=%d count changed between configurations", N);
        }
        if (k == 0) continue;
        float ms = 0.f;
        float prep = 0.f;
        if (int e = nq_last_kernel_ms(h, &prep, &ms)) { h->block = old_block; h->split = old_split; return e; }
        ms += prep;
        if (ms < best) { best = ms; bb = b; bs = s; }
      }
    }
  h->block = bb; h->split = bs;                       // the handle keeps the fastest configuration
  if (best_block) *best_block = bb;
  if (best_split) *best_split = bs;
  if (best_ms) *best_ms = best;
  return NQ_OK;
}

int nq_set_chunk_records(nq_handle* h, int64_t records) {
  if (!h) return NQ_EINVAL;
  if (records < 0) return h->fail(NQ_EINVAL, "chunk size must be >= 0");
  h->chunk_records = records;
  return NQ_OK;
}

}  // extern "C"

namespace {

// The records of start constellations [s_begin, s_end), generated and counted
// chunk by chunk so host memory stays bounded for the largest boards (the
// reference streams its task list to a .bin file for the same reason,
// gen_constellations_stream_to_bin, 356Py_savesp_narrow.py:2988-3084): each
// chunk of starts is expanded into records on the host threads while the
// previous chunk's DFS runs on the GPU.
int count_generated(nq_handle* h, int N, int p, const std::vector<int>& starts, size_t s_begin, size_t s_end,
                    uint64_t* total);

int count_start_range(nq_handle* h, int N, int p, const std::vector<int>& starts, size_t s_begin, size_t s_end,
                      uint64_t* total) {
  // a chunk size set by the caller bounds the host list, deeper presets make more records than a buffer holds
  if (h->chunk_records == 0 && p <= 8) return count_generated(h, N, p, starts, s_begin, s_end, total);
  const int64_t chunk = h->chunk_records > 0 ? h->chunk_records : kChunkRecords;
  size_t next = s_begin;
  double per_start = 0.0;                  // records per start constellation seen so far
  std::vector<GenRecord> g;
  // Blocks of starts are expanded and packed into 16-byte records at once, so the
  // 32-byte generator records of at most an eighth of a chunk are alive at a time.
  auto gen_chunk = [&](std::vector<nq_record>& out) -> int {
    out.clear();
    if (per_start > 0.0)   // expected size of this chunk, so the vector does not double past it
      out.reserve((size_t)std::min((double)(chunk + chunk / 8), per_start * (double)(s_end - next) + 1024.0));
    while (next < s_end && (int64_t)out.size() < chunk) {
      const double want = std::min((double)(chunk - (int64_t)out.size()), (double)chunk / 8.0);
      const size_t take = per_start > 0.0 ? (size_t)std::max(1.0, want / per_start) : (size_t)16;
      const size_t s1 = std::min(s_end, next + take);
      g.clear();
      const int e = expand_starts(N, p, starts, next, s1, g, 0);
      if (e == -1) return h->fail(NQ_EINVAL, "generator: bad arguments N=%d preset=%d", N, p);
      if (e == -2) return h->fail(NQ_EPRESET, "generator: preset %d too deep for N=%d", p, N);
      per_start = 0.5 * per_start + 0.5 * (double)g.size() / (double)(s1 - next);
      if (per_start <= 0.0) per_start = 0.25;
      next = s1;
      const size_t o = out.size();
      out.resize(o + g.size());
      for (size_t i = 0; i < g.size(); i++)
        out[o + i] = nq_record{(uint32_t)g[i].ld, (uint32_t)g[i].rd, (uint32_t)g[i].col, g[i].startijkl};
    }
    std::vector<GenRecord>().swap(g);
    return NQ_OK;
  };
  cudaStream_t st = h->stream;
  NQ_CUDA(h, cudaSetDevice(h->device));
  std::vector<nq_record> cur, nxt;
  if (int e = gen_chunk(cur)) return e;
  uint64_t acc = 0;
  int64_t chunks = 0, records = 0;
  while (!cur.empty()) {
    const int64_t m = (int64_t)cur.size();
    const int smin = (int)start_row_min(&cur[0].startijkl, m, 4);
    NQ_CUDA(h, h->rec.ensure((size_t)m * sizeof(nq_record)));
    NQ_CUDA(h, cudaMemcpyAsync(h->rec.p, cur.data(), (size_t)m * sizeof(nq_record), cudaMemcpyHostToDevice, st));
    if (int s = run_records(h, N, (const uint4*)h->rec.p, m, smin, nullptr, st)) return s;
    if (int e = gen_chunk(nxt)) { cudaStreamSynchronize(st); return e; }   // overlaps the DFS just launched
    uint64_t t = 0;
    if (int s = read_ctrl(h, st, &t)) return s;
    acc += t; chunks++; records += m;
    cur.swap(nxt);
  }
  h->last_chunks = chunks;
  h->last_records = records;
  *total = acc;
  return NQ_OK;
}

// The same with the records generated on the device (presets 4..8): chunks of start constellations whose
// records are bounded by the buffers, one launch a queen, then the usual run over the list that never left
// the device.  The host generator above spends 0.9 ms on its threads alone at N=9..13 (a count of N=13 took
// 1.3 ms, 0.1 of it on the GPU) and 8 ms on N=19's 897,071 records.
constexpr uint64_t kGenRecords = 8 << 20;         // records a chunk may have (bound), 128 MiB a buffer
constexpr uint64_t kGenBoard = 2 << 20;           // states a board in one chunk may have
// The list's length stays on the device up to this many records: by the bound of a range of start constellations
// (2 to 4 times its records), or by a board's states.
constexpr uint64_t kGenNoReadBack = 65536, kGenNoReadBackBoard = 32768;

// At most this many states on any level from one start constellation to its records: it holds 3 or 4 queens, and its
// first free row has N - 3 or N - 4 columns left, the next one fewer, ...  Where the columns run out (N=7 at preset 8)
// a level before has more states than the records' own bound.
uint64_t start_bound(int N, int preset, int start) {
  const uint32_t col = 1u | (1u << (N - 1)) | ((1u << (N - 1)) >> geti(start)) | ((1u << (N - 1)) >> getj(start));
  uint64_t b = 1, most = 1;
  int c = N - __builtin_popcount(col);
  for (int q = getj(start) == N - 1 ? 3 : 4; q < preset; q++) {
    b *= (uint64_t)std::max(0, c--);
    most = std::max(most, b);
  }
  return most;
}

// One generated chunk on the handle's stream: starts (host list, or null: the whole board of at most n), counted; no
// level of it has more than `bound` states.
int count_chunk(nq_handle* h, int N, int p, const int* starts, size_t n, uint64_t bound, uint64_t* total, int64_t* records) {
  cudaStream_t st = h->stream;
  NQ_CUDA(h, cudaSetDevice(h->device));
  NQ_CUDA(h, h->ctrl.ensure(ctl::kAll));
  unsigned char* c = (unsigned char*)h->ctrl.p;
  unsigned int* gn = (unsigned int*)(c + ctl::kGen);
  const int levels = gen_levels(p);
  if (bound > 0x7FFFFFFFull) return h->fail(NQ_ENOMEM, "generator: too many records from one start constellation");
  const size_t cap = std::max<size_t>((size_t)bound, n);
  NQ_CUDA(h, h->rec.ensure(cap * sizeof(uint4)));
  if (levels > kGenFused) NQ_CUDA(h, h->gen.ensure(cap * sizeof(uint4)));
  if (int e = h->ensure_pinned(kStage + (starts ? n * sizeof(int) : 0))) return e;
  if (starts) {
    NQ_CUDA(h, h->starts.ensure(n * sizeof(int)));
    std::memcpy((unsigned char*)h->h_ctrl + kStage, starts, n * sizeof(int));
    NQ_CUDA(h, cudaMemcpyAsync(h->starts.p, (unsigned char*)h->h_ctrl + kStage, n * sizeof(int), cudaMemcpyHostToDevice, st));
  }
  NQ_CUDA(h, cudaMemsetAsync(c, 0, ctl::kAll, st));
  h->result_written = false;
  uint4* buf[2] = {(uint4*)h->rec.p, (uint4*)(levels > kGenFused ? h->gen.p : h->rec.p)};
  NQ_CUDA(h, launch_generate(N, p, (unsigned)n, starts ? (const int*)h->starts.p : nullptr, buf[0], buf[1], (unsigned)cap, gn,
                             (unsigned int*)(c + ctl::kGenErr), h->sms, st));
  const uint4* rec = buf[levels & 1];
  const int t_max = std::max(1, N - p - 2);        // a queen a depth, one column left in the base row
  const bool on_device = bound <= (starts ? kGenNoReadBack : kGenNoReadBackBoard) && h->queue_order == 0;
  int64_t m = (int64_t)bound;
  if (!on_device) {
    NQ_CUDA(h, cudaMemcpyAsync(h->h_ctrl, c, ctl::kAll, cudaMemcpyDeviceToHost, st));
    NQ_CUDA(h, cudaStreamSynchronize(st));
    m = *(const uint32_t*)((const unsigned char*)h->h_ctrl + ctl::kGen + 4 * levels);
  }
  if (m > 0)
    if (int e = run_records(h, N, rec, m, p - 3, nullptr, st, t_max, on_device ? gn + levels : nullptr)) return e;
  if (int e = read_ctrl(h, st, total)) return e;
  const unsigned char* hc = (const unsigned char*)h->h_ctrl;
  if (*(const uint32_t*)(hc + ctl::kGenErr)) return h->fail(NQ_EPRESET, "generator: preset %d too deep for N=%d", p, N);
  *records = *(const uint32_t*)(hc + ctl::kGen + 4 * levels);
  return NQ_OK;
}

int count_generated(nq_handle* h, int N, int p, const std::vector<int>& starts, size_t s_begin, size_t s_end,
                    uint64_t* total) {
  uint64_t acc = 0;
  int64_t chunks = 0, records = 0;
  for (size_t s0 = s_begin; s0 < s_end;) {
    size_t s1 = s0;
    uint64_t bound = 0;
    do { bound += start_bound(N, p, starts[s1++]); }
    while (s1 < s_end && bound + start_bound(N, p, starts[s1]) <= kGenRecords);
    uint64_t t = 0;
    int64_t r = 0;
    if (int e = count_chunk(h, N, p, &starts[s0], s1 - s0, bound, &t, &r)) return e;
    acc += t; chunks++; records += r;
    s0 = s1;
  }
  h->last_chunks = records == 0 ? 0 : chunks;
  h->last_records = records;
  *total = acc;
  return NQ_OK;
}

}  // namespace

extern "C" {

// Whole-board count: in one go where the device makes the whole board's list, else the start constellations
// are listed (cheap) and counted as one range.
int nq_count(nq_handle* h, int N, int preset, uint64_t* total) {
  if (!h || !total) return NQ_EINVAL;
  if (N < 1 || N > kMaxN) return h->fail(NQ_EINVAL, "N=%d outside 1..27", N);
  if (N <= 5) return nq_count_completions(h, N, 0, nullptr, nullptr, total);
  const int p = preset > 0 ? preset : preset_for(N);
  if (p < 4) return h->fail(NQ_EPRESET, "generator: preset %d below 4", p);
  if (h->chunk_records == 0 && p <= 8 && board_states(N, p) <= kGenBoard) {
    int64_t records = 0;
    if (int e = count_chunk(h, N, p, nullptr, board_states(N, 4), board_states(N, p), total, &records)) return e;
    h->last_chunks = records ? 1 : 0;
    h->last_records = records;
    return NQ_OK;
  }
  std::vector<int> starts;
  if (start_constellations(N, starts) != 0) return h->fail(NQ_EINVAL, "generator: bad arguments N=%d", N);
  return count_start_range(h, N, p, starts, 0, starts.size(), total);
}

int64_t nq_start_constellations(int N, int32_t* out, int64_t cap) {
  if (N < 6 || N > kMaxN) return NQ_EINVAL;
  std::vector<int> starts;
  if (start_constellations(N, starts) != 0) return NQ_EINVAL;
  const int64_t n = (int64_t)starts.size();
  if (out && cap >= n)
    for (int64_t i = 0; i < n; i++) out[i] = (int32_t)starts[i];
  return n;
}

int64_t nq_gen_constellations_starts(int N, int preset, int64_t first, int64_t count, nq_record* out, int64_t cap) {
  if (N < 6 || N > kMaxN) return NQ_EINVAL;
  const int p = preset > 0 ? preset : preset_for(N);
  if (p < 4) return NQ_EPRESET;
  std::vector<int> starts;
  if (start_constellations(N, starts) != 0) return NQ_EINVAL;
  const int64_t ns = (int64_t)starts.size();
  if (first < 0 || count < 0 || first > ns || count > ns - first) return NQ_EINVAL;
  std::vector<GenRecord> v;
  const int e = expand_starts(N, p, starts, (size_t)first, (size_t)(first + count), v, 0);
  if (e == -1) return NQ_EINVAL;
  if (e == -2) return NQ_EPRESET;
  const int64_t n = (int64_t)v.size();
  if (out && cap >= n)
    for (int64_t i = 0; i < n; i++)
      out[i] = nq_record{(uint32_t)v[i].ld, (uint32_t)v[i].rd, (uint32_t)v[i].col, v[i].startijkl};
  return n;
}

int nq_count_starts(nq_handle* h, int N, int preset, int64_t first, int64_t count, uint64_t* total) {
  if (!h || !total) return NQ_EINVAL;
  if (N < 6 || N > kMaxN) return h->fail(NQ_EINVAL, "count_starts: N=%d outside 6..27", N);
  const int p = preset > 0 ? preset : preset_for(N);
  if (p < 4) return h->fail(NQ_EPRESET, "generator: preset %d below 4", p);
  std::vector<int> starts;
  if (start_constellations(N, starts) != 0) return h->fail(NQ_EINVAL, "generator: bad arguments N=%d", N);
  const int64_t ns = (int64_t)starts.size();
  if (first < 0 || count < 0 || first > ns || count > ns - first)
    return h->fail(NQ_EINVAL, "count_starts: range [%lld, +%lld) outside the %lld start constellations",
                   (long long)first, (long long)count, (long long)ns);
  return count_start_range(h, N, p, starts, (size_t)first, (size_t)(first + count), total);
}

int nq_last_count_info(const nq_handle* h, int64_t* chunks, int64_t* records) {
  if (!h) return NQ_EINVAL;
  if (chunks) *chunks = h->last_chunks;
  if (records) *records = h->last_records;
  return NQ_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// batches
// ---------------------------------------------------------------------------
struct nq_batch {
  nq_handle* h = nullptr;
  std::vector<nq_job> jobs;
  cudaStream_t stream = nullptr;
  cudaEvent_t done = nullptr;
  DevBuf info, sched, ctrl, sroot, sinfo;  // tasks (jobs of one board share them), and the queue
  int64_t m = 0;        // sources of all jobs (records, query frames)
  int64_t ms = 0;       // queued items (every job's split output, job after job)
  int maxt = 1, sw = 2, grid = 0, block = 128;
  bool big = false;                        // some job's queue items may count 2^32: u64 per-lane counters
  bool wide = false;                       // 8-byte schedule words (a query with far-reaching steps); compact otherwise
  bool ra_words = false;                   // some board's compact words carry RA (too large to keep it in rd)
  std::vector<int64_t> sub_off, sub_m;     // queue range per job
  std::vector<int> job_maxt;
  std::vector<uint64_t> fixed_total;       // counts settled at build time (small tasks, full boards)
  uint64_t* h_out = nullptr;               // pinned: totals per job + cursor/err
  unsigned char* stage = nullptr;          // pinned: the build's uploads
  cudaGraphExec_t graph = nullptr;
  bool submitted = false;
  int64_t device_bytes = 0;
  int64_t h2d_bytes = 0;                   // host->device bytes of the build (queries, tables)
};

namespace {

// Jobs up to which the search's last block hands the totals over (one warp, 256 of them at a time); above, a copy.
// us of a replay, so / by a copy: 4 jobs of N=6..8 19.3 / 27.5, 256 24.0 / 28.9, 1024 25.5 / 28.0.
constexpr int kHandOver = 2048;

int batch_enqueue(nq_batch* b, int use_graph) {
  nq_handle* h = b->h;
  const int nj = (int)b->jobs.size();
  const size_t cb = Ctrl::bytes(nj);
  unsigned char* c = (unsigned char*)b->ctrl.p;
  auto enqueue = [&](cudaStream_t st) -> cudaError_t {
    cudaError_t e = cudaMemsetAsync(c, 0, cb, st);
    if (e != cudaSuccess) return e;
    TaskArrays ta;
    ta.info = (uint32_t*)b->info.p; ta.sched = b->sched.p; ta.sw = b->sw; ta.wide = b->wide; ta.ra_words = b->ra_words;
    DfsLaunch L;
    L.tasks = ta; L.sroot = (const uint4*)b->sroot.p; L.sinfo = (const uint2*)b->sinfo.p;
    L.m = b->ms; L.cursor = (unsigned long long*)(c + (size_t)nj * 8);
    L.job_totals = (unsigned long long*)c; L.err = (unsigned int*)(c + (size_t)nj * 8 + 8);
    L.maxt = b->maxt; L.block = b->block; L.grid = b->grid; L.big = b->big;
    const bool hand = b->ms > 0 && nj <= kHandOver;
    if (hand) {
      L.ctl = (const uint32_t*)c; L.ctl_words = (unsigned)(cb / 8); L.host_ctl = (uint32_t*)b->h_out;
      L.blocks_done = L.err + 1;
    }
    e = launch_dfs(L, st);
    if (e != cudaSuccess || hand) return e;
    return cudaMemcpyAsync(b->h_out, c, cb, cudaMemcpyDeviceToHost, st);
  };
  NQ_CUDA(h, cudaSetDevice(h->device));
  if (use_graph) {
    if (!b->graph) {
      cudaGraph_t g = nullptr;
      NQ_CUDA(h, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
      cudaError_t e = enqueue(b->stream);
      cudaError_t e2 = cudaStreamEndCapture(b->stream, &g);
      if (e != cudaSuccess) { if (g) cudaGraphDestroy(g); return h->cuda_fail(e, "batch capture"); }
      if (e2 != cudaSuccess) return h->cuda_fail(e2, "cudaStreamEndCapture");
      e = cudaGraphInstantiate(&b->graph, g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) { b->graph = nullptr; return h->cuda_fail(e, "cudaGraphInstantiate"); }
    }
    NQ_CUDA(h, cudaGraphLaunch(b->graph, b->stream));
  } else {
    NQ_CUDA(h, enqueue(b->stream));
  }
  NQ_CUDA(h, cudaEventRecord(b->done, b->stream));
  b->submitted = true;
  return NQ_OK;
}

int batch_collect(nq_batch* b, uint64_t* totals) {
  nq_handle* h = b->h;
  const int nj = (int)b->jobs.size();
  const uint32_t e = ((const uint32_t*)(b->h_out + nj))[2];
  b->submitted = false;
  if (e) return h->fail(derr_to_status(e), "device: %s", derr_text(e));
  if (totals)
    for (int j = 0; j < nj; j++) totals[j] = b->h_out[j] + b->fixed_total[j];
  return NQ_OK;
}

}  // namespace

extern "C" {

void nq_batch_destroy(nq_batch* b) {
  if (!b) return;
  cudaSetDevice(b->h->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  if (b->graph) cudaGraphExecDestroy(b->graph);
  for (DevBuf* d : {&b->info, &b->sched, &b->ctrl, &b->sroot, &b->sinfo}) d->release();
  if (b->stream) cudaStreamSynchronize(b->stream);   // this batch's own frees only
  b->h->pin_put(b->h_out);
  b->h->pin_put(b->stage);
  if (b->done) cudaEventDestroy(b->done);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

// Boards whose list the device makes: the deeper presets' outgrow the generator's buffers.
bool board_on_device(int N, int p) { return p <= 8 && board_states(N, p) <= kGenBoard; }

// A board's tasks in a batch go unsplit where the batch's counts give every lane at least a quarter of such a task:
// splitting then only adds items (the queue's end is evened out by the other jobs and within the warps).  us of a
// replay, split once (as any list above 10^5 tasks) / so: 64 jobs of N=12..15 1212 / 938, of N=10..14 271 / 174, 256
// 760 / 429, 16 of N=13..16 1012 / 978.  With an eighth 4 jobs of N=13..15 173 for 125.  Up to 11 rows left: at 12
// (N=16) an unsplit list saves 1 % in large batches, and the same job launched alone takes 550 us for 340.
double task_nodes(int rows) { return 100.0 * std::pow(4.0, rows - 9); }   // about: N=13..16 at preset 5 100, 350, 1300, 5500
constexpr double kLanes = 1024.0;                                          // resident an SM, about
bool unsplit_in_batch(int rows, double work, int sms) {
  return rows <= 11 && work >= 0.25 * task_nodes(rows) * kLanes * sms;
}

// Build, one synchronisation in all: the boards' records are generated on the device and prepared, each
// query is expanded by one block (queries and tables are the only uploads), every
// list's split is counted, the queue is allocated, and the jobs' items are written job after job.  Jobs of
// one board share its tasks and its counted list; each has its own items.  Building 64 mixed jobs of N=9..16
// on the host (generator, breadth-first searches, staging, two split launches a job) took 19 ms.
int nq_batch_create(nq_handle* h, const nq_job* jobs, int njobs, nq_batch** out) {
  if (!h || !out || njobs <= 0 || !jobs) return h ? h->fail(NQ_EINVAL, "batch: bad arguments") : NQ_EINVAL;
  *out = nullptr;
  NQ_CUDA(h, cudaSetDevice(h->device));
  nq_batch* b = new (std::nothrow) nq_batch();
  if (!b) return NQ_ENOMEM;
  b->h = h;
  b->jobs.assign(jobs, jobs + njobs);
  b->block = h->block;
  b->job_maxt.assign(njobs, 1); b->fixed_total.assign(njobs, 0);
  b->sub_off.assign(njobs, 0); b->sub_m.assign(njobs, 0);
  auto bad = [&](int status, const char* what, int j) {
    nq_batch_destroy(b);
    return h->fail(status, "batch job %d: %s", j, what);
  };
  // ---- the lists: one per board (N, preset) and one per query
  // weight: the list's length as the rules below count it
  struct List { int N = 0, rows = 0, T = 0; uint64_t cap = 0, weight = 0; bool query = false; int D = 0; uint32_t src0 = 0, task0 = 0; };
  struct Board { int p; uint32_t list; bool device; std::vector<GenRecord> recs; };
  std::vector<List> lists;
  std::vector<Board> boards;
  std::vector<BatchQuery> queries;
  std::vector<int> job_list(njobs, -1);
  std::map<std::pair<int, int>, uint32_t> board_list;
  uint64_t sources = 0;                          // all jobs' sources, roughly
  double work = 0.0;                             // and the counts' search nodes
  for (int j = 0; j < njobs; j++) {
    const nq_job& J = jobs[j];
    if (J.N < 1 || J.N > kMaxN || J.k < 0 || J.k > 8) return bad(NQ_EINVAL, "bad N or k", j);
    if (J.kind != NQ_JOB_COUNT && J.kind != NQ_JOB_COMPLETION) return bad(NQ_EINVAL, "unknown kind", j);
    if (J.kind == NQ_JOB_COUNT && J.N >= 6) {
      const int p = J.preset > 0 ? J.preset : preset_for(J.N);
      if (p < 4) return bad(NQ_EPRESET, "generator failed (preset below 4)", j);
      auto it = board_list.find({J.N, p});
      if (it == board_list.end()) {
        Board bd;
        bd.p = p; bd.list = (uint32_t)lists.size();
        List l;
        l.N = J.N; l.cap = board_states(J.N, p); l.rows = maxt_for(J.N, p - 3);
        b->ra_words = b->ra_words || !ra_in_rd(J.N, p - 3, 0);
        bd.device = board_on_device(J.N, p);
        if (!bd.device) {                        // the host's list
          const int s = gen_constellations(J.N, p, bd.recs, 0);
          if (s != 0) return bad(s == -2 ? NQ_EPRESET : NQ_EINVAL, "generator failed", j);
          l.cap = bd.recs.size();
        }
        l.weight = bd.device ? l.cap * (p == 4 ? 2 : 3) : l.cap;
        it = board_list.emplace(std::make_pair(J.N, p), bd.list).first;
        lists.push_back(l);
        boards.push_back(std::move(bd));
      }
      job_list[j] = (int)it->second;
      sources += lists[it->second].weight / 4;
      work += (double)(lists[it->second].weight / 4) * task_nodes(lists[it->second].rows);
    } else {
      int rows[8], cols[8];
      const int k = (J.kind == NQ_JOB_COUNT) ? 0 : J.k;
      for (int q = 0; q < k; q++) { rows[q] = J.rows[q]; cols[q] = J.cols[q]; }
      BatchQuery q{};
      bool wide = false;
      const int s = query_task(J.N, k, rows, cols, &q.p, &wide, &b->fixed_total[j]);
      if (s < 0) return bad(NQ_EINVAL, "bad pre-placed queens", j);
      if (s == 0) continue;
      b->wide = b->wide || wide;
      List l;
      l.N = J.N; l.T = (int)q.p.T; l.rows = l.T + 2; l.query = true;
      q.list = (uint32_t)lists.size();
      job_list[j] = (int)lists.size();
      lists.push_back(l);
      queries.push_back(q);
    }
  }
  const unsigned target = queries.size() > 64 ? kQueryTarget / 4 : kQueryTarget;
  for (BatchQuery& q : queries) {
    q.p.target = std::min(target, kQueryCap / q.p.N);
    lists[q.list].cap = query_frames(q.p);
    lists[q.list].weight = (uint64_t)q.p.target * q.p.N;
    sources += 4 * q.p.target;
    if (b->wide != (q.p.words_wide != 0)) widen_query(&q.p);
  }
  // ---- offsets, split depths, table sizes
  const size_t nl = lists.size(), nb = boards.size(), nq = queries.size();
  std::vector<unsigned long long> ends(nl);
  uint64_t src = 0, ntask = 0, words = 1, rec_cap = 0, gen_cap = 0, tmp_cap = 0;
  for (size_t i = 0; i < nl; i++) {
    List& l = lists[i];
    l.src0 = (uint32_t)src; l.task0 = (uint32_t)ntask;
    src += (l.cap + 31) & ~31ull;                // warps stay within a list
    ends[i] = src;
    ntask += l.query ? 1 : l.cap;
    words = std::max<uint64_t>(words, l.query ? l.T + 1 : l.rows + 1);
    const int levels = l.query ? batch_query_levels(l.rows) : choose_split((int64_t)std::max(sources, l.weight), l.rows);
    const bool whole = !l.query && unsplit_in_batch(l.rows, work, h->sms);
    // queries of the larger target are cut once in a batch with that many sources, of the smaller one twice: 256 mixed
    // jobs of N=9..16 3628 us with one, 3070 so; 64 718 so, 986 uncut
    const bool once = l.query && sources > 100000 && target == kQueryTarget;
    l.D = l.N <= 12 ? 0 : h->split >= 0 ? h->split : whole ? 0 : once ? std::min(levels, 1) : levels;
  }
  for (const Board& bd : boards) {
    rec_cap = std::max(rec_cap, lists[bd.list].cap);
    if (bd.device && gen_levels(bd.p) > kGenFused) gen_cap = std::max(gen_cap, lists[bd.list].cap);
  }
  if (src > 0xFFFFFFFFull || words > (uint64_t)kMaxDepth) { nq_batch_destroy(b); return h->fail(NQ_ENOMEM, "batch: too many tasks"); }
  b->sw = (int)words;
  const size_t word = b->wide ? sizeof(uint2) : sizeof(uint32_t), cb = Ctrl::bytes(njobs);
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t o_lists = up(nl * 8), o_q = o_lists + up(nl * sizeof(BatchList));
  const size_t o_jends = o_q + up(nq * sizeof(BatchQuery)), o_jobs = o_jends + up((size_t)njobs * 8);
  const size_t tab_bytes = o_jobs + up((size_t)njobs * sizeof(BatchJob));
  // state: list states, generated levels and deepest schedule per board, error words of generator and prepare
  const size_t o_gn = up(nl * sizeof(ListState)), o_tmax = o_gn + up(nb * 32), o_err = o_tmax + up(nb * 4);
  const size_t state_bytes = o_err + 8;
  cudaError_t e = cudaSuccess;
  cudaStream_t st = nullptr;
  DevBuf tab, state, rec, gen, frames, tmp, off;
  int status = NQ_OK;
  do {
    if ((e = h->ensure_pool()) != cudaSuccess ||
        (e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming)) != cudaSuccess) break;
    st = b->stream;
    for (DevBuf* d : {&b->info, &b->sched, &b->ctrl, &b->sroot, &b->sinfo, &tab, &state, &rec, &gen, &frames, &tmp, &off}) {
      d->ordered = st; d->pool = h->pool;
    }
    b->h_out = (uint64_t*)h->pin_get(std::max(cb, state_bytes));
    b->stage = (unsigned char*)h->pin_get(tab_bytes);
    if (!b->h_out || !b->stage) { e = cudaErrorMemoryAllocation; break; }
    if ((e = b->ctrl.ensure(cb)) != cudaSuccess || (e = tab.ensure(tab_bytes)) != cudaSuccess ||
        (e = state.ensure(state_bytes)) != cudaSuccess || (e = b->info.ensure(std::max<uint64_t>(ntask, 1) * 4)) != cudaSuccess ||
        (e = b->sched.ensure(std::max<uint64_t>(ntask, 1) * words * word)) != cudaSuccess ||
        (e = frames.ensure(std::max<uint64_t>(src, 1) * sizeof(uint4))) != cudaSuccess ||
        (e = off.ensure(std::max<uint64_t>(src, 1) * 4)) != cudaSuccess ||
        (nb && (e = rec.ensure(std::max<uint64_t>(rec_cap, 1) * sizeof(uint4))) != cudaSuccess) ||
        (gen_cap && (e = gen.ensure(gen_cap * sizeof(uint4))) != cudaSuccess)) break;
    unsigned char *dt = (unsigned char*)tab.p, *ds = (unsigned char*)state.p;
    // ---- upload the lists and queries
    BatchList* hl = (BatchList*)(b->stage + o_lists);
    if (nl) std::memcpy(b->stage, ends.data(), nl * 8);
    for (size_t i = 0; i < nl; i++) hl[i] = BatchList{lists[i].src0, lists[i].task0, lists[i].query ? 1u : 0u, (uint32_t)lists[i].D};
    BatchQuery* hq = (BatchQuery*)(b->stage + o_q);
    for (size_t i = 0; i < nq; i++) {
      hq[i] = queries[i];
      const List& l = lists[queries[i].list];
      hq[i].src0 = l.src0; hq[i].task = l.task0; hq[i].cap = (uint32_t)l.cap; hq[i].tmp0 = (uint32_t)tmp_cap;
      tmp_cap += l.cap;
    }
    if (nq && (e = tmp.ensure(tmp_cap * sizeof(uint4))) != cudaSuccess) break;
    if ((e = cudaMemcpyAsync(dt, b->stage, o_jends, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (e = cudaMemsetAsync(ds, 0, state_bytes, st)) != cudaSuccess) break;
    b->h2d_bytes = (int64_t)o_jends;
    ListState* dstate = (ListState*)ds;
    unsigned int* derr = (unsigned int*)(ds + o_err);
    TaskArrays ta;
    ta.info = (uint32_t*)b->info.p; ta.sched = b->sched.p; ta.sw = b->sw; ta.wide = b->wide; ta.ra_words = b->ra_words;
    // ---- boards: generate (or upload) the records, prepare them into the board's tasks
    for (size_t i = 0; i < nb && e == cudaSuccess; i++) {
      const Board& bd = boards[i];
      const List& l = lists[bd.list];
      const uint4* drec = (const uint4*)rec.p;
      const unsigned int* dn = nullptr;
      std::vector<nq_record> packed;
      if (bd.device) {
        const int levels = gen_levels(bd.p);
        uint4* buf[2] = {(uint4*)rec.p, (uint4*)(levels > kGenFused ? gen.p : rec.p)};
        unsigned int* gn = (unsigned int*)(ds + o_gn + i * 32);
        e = launch_generate(l.N, bd.p, (unsigned)board_states(l.N, 4), nullptr, buf[0], buf[1],
                            (unsigned)l.cap, gn, derr, h->sms, st);
        drec = buf[levels & 1];
        dn = gn + levels;
      } else if (l.cap) {
        packed.resize(l.cap);
        for (size_t r = 0; r < l.cap; r++)
          packed[r] = nq_record{(uint32_t)bd.recs[r].ld, (uint32_t)bd.recs[r].rd, (uint32_t)bd.recs[r].col, bd.recs[r].startijkl};
        e = cudaMemcpyAsync(rec.p, packed.data(), l.cap * sizeof(nq_record), cudaMemcpyHostToDevice, st);
        b->h2d_bytes += (int64_t)(l.cap * sizeof(nq_record));
      }
      ta.root = (uint4*)frames.p + ((int64_t)l.src0 - (int64_t)l.task0);      // task t's root is its list's source
      // Each board by its own size, whatever the search's form: a board with RA in rd has none in its words, and where
      // the step looks for it there it finds nothing.  In the words of a small board RA would meet the count flag.
      ta.ra_words = !ra_in_rd(l.N, bd.p - 3, 0);
      if (e == cudaSuccess)
        e = launch_prepare(l.N, (int64_t)l.cap, dn, drec, ta, l.task0, derr + 1, st, (unsigned int*)(ds + o_tmax) + i, &dstate[bd.list].n);
      if (e == cudaSuccess && !packed.empty()) e = cudaStreamSynchronize(st);   // the host list goes out of scope
    }
    if (e != cudaSuccess) break;
    ta.root = nullptr; ta.ra_words = b->ra_words;
    if ((e = launch_batch_queries((int)nq, (const BatchQuery*)(dt + o_q), (uint4*)frames.p, (uint4*)tmp.p, dstate, ta, st)) !=
        cudaSuccess) break;
    // ---- count every list's items, read the sizes back
    ListArgs a;
    a.n = (int)nl; a.total = src; a.ends = (const unsigned long long*)dt; a.lists = (const BatchList*)(dt + o_lists);
    a.state = dstate; a.src = (const uint4*)frames.p; a.info = ta.info; a.sched = ta.sched; a.sw = ta.sw; a.off = (uint32_t*)off.p;
    if ((e = launch_list_count(a, b->wide, st)) != cudaSuccess) break;
    if ((e = cudaMemcpyAsync(b->h_out, ds, state_bytes, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess) break;
    const unsigned char* hs = (const unsigned char*)b->h_out;
    const unsigned int* herr = (const unsigned int*)(hs + o_err);
    if (herr[0]) { status = h->fail(NQ_EPRESET, "batch: generator failed (preset too deep)"); break; }
    if (herr[1]) { status = h->fail(derr_to_status(herr[1]), "batch prepare: %s", derr_text(herr[1])); break; }
    const ListState* hst = (const ListState*)hs;
    for (size_t i = 0; i < nl; i++)          // a source's first slot is kept in 32 bits
      if (hst[i].items > 0xFFFFFFFFull) status = h->fail(NQ_ENOMEM, "batch: %llu items of one list", hst[i].items);
    if (status != NQ_OK) break;
    // Stacks sized to the deepest item: items start `depth` + D down, so they need (deepest T) less that.
    std::vector<int> deep(nl, 1);
    for (size_t i = 0; i < nb; i++)
      deep[boards[i].list] = std::max(1, (int)((const unsigned int*)(hs + o_tmax))[i] - lists[boards[i].list].D);
    for (const BatchQuery& q : queries)
      deep[q.list] = std::max(1, lists[q.list].T - (int)hst[q.list].depth - lists[q.list].D);
    unsigned long long* je = (unsigned long long*)(b->stage + o_jends);
    BatchJob* jt = (BatchJob*)(b->stage + o_jobs);
    int nj = 0;
    uint64_t items = 0, jsrc = 0;
    b->maxt = 1;
    for (int j = 0; j < njobs; j++) {
      b->sub_off[j] = (int64_t)items;
      const int li = job_list[j];
      if (li < 0) continue;
      const ListState& s = hst[li];
      b->fixed_total[j] += s.settled;
      b->sub_m[j] = (int64_t)s.items;
      b->job_maxt[j] = deep[li];
      b->m += s.n;
      if (s.items == 0) continue;
      b->maxt = std::max(b->maxt, deep[li]);
      b->big = b->big || counts_need_u64(jobs[j].N, (int64_t)s.items);
      jsrc += s.n;
      je[nj] = jsrc;
      jt[nj++] = BatchJob{items, (uint32_t)(li ? ends[li - 1] : 0ull), (uint32_t)li, (uint32_t)j, 0};
      items += s.items;
    }
    b->ms = (int64_t)items;
    for (DevBuf* d : {&rec, &gen, &tmp}) d->release();       // the queue may take their place
    if ((e = b->sroot.ensure(std::max<uint64_t>(items, 1) * sizeof(uint4))) != cudaSuccess ||
        (e = b->sinfo.ensure(std::max<uint64_t>(items, 1) * sizeof(uint2))) != cudaSuccess) break;
    // ---- write the jobs' items
    if (nj) {
      if ((e = cudaMemcpyAsync(dt + o_jends, b->stage + o_jends, tab_bytes - o_jends, cudaMemcpyHostToDevice, st)) != cudaSuccess) break;
      b->h2d_bytes += (int64_t)(tab_bytes - o_jends);
      a.n = nj; a.total = jsrc; a.ends = (const unsigned long long*)(dt + o_jends);
      if ((e = launch_list_write(a, (const BatchJob*)(dt + o_jobs), (uint4*)b->sroot.p, (uint2*)b->sinfo.p, b->wide, st)) !=
          cudaSuccess) break;
    }
  } while (0);
  if (st) for (DevBuf* d : {&tab, &state, &rec, &gen, &frames, &tmp, &off}) d->release();   // after the launches above, on the stream
  if (e != cudaSuccess) status = h->cuda_fail(e, "batch build");
  if (status != NQ_OK) { nq_batch_destroy(b); return status; }
  b->device_bytes = (int64_t)(b->info.cap + b->sched.cap + b->ctrl.cap + b->sroot.cap + b->sinfo.cap);
  *out = b;
  return NQ_OK;
}

int64_t nq_job_device_bytes(const nq_job* job, int sms, int split_depth) {
  if (!job || sms < 1 || split_depth < -1 || split_depth > 3) return NQ_EINVAL;
  const nq_job& J = *job;
  if (J.N < 1 || J.N > kMaxN || J.k < 0 || J.k > 8) return NQ_EINVAL;
  int64_t m = 0, tasks = 1;
  int rows = 1, levels = 0;
  int64_t word = sizeof(uint2), list = sizeof(uint4);        // bytes a schedule word, and a source while its list is made
  if (J.kind == NQ_JOB_COUNT && J.N >= 6) {
    const int p = J.preset > 0 ? J.preset : preset_for(J.N);
    if (p < 4) return NQ_EPRESET;
    m = (int64_t)board_states(J.N, p);
    if (m == 0 || J.N < p) {               // no figure, or a preset that may be too deep
      std::vector<GenRecord> v;
      const int s = gen_constellations(J.N, p, v, 0);
      if (s != 0) return s == -2 ? NQ_EPRESET : NQ_EINVAL;
      m = std::max(m, (int64_t)v.size());
    }
    tasks = m;
    rows = maxt_for(J.N, p - 3);
    levels = choose_split(m, rows);
    word = sizeof(uint32_t);
    if (board_on_device(J.N, p) && gen_levels(p) > kGenFused) list *= 2;
  } else if (J.kind == NQ_JOB_COUNT || J.kind == NQ_JOB_COMPLETION) {
    int r[8], c[8];
    const int k = (J.kind == NQ_JOB_COUNT) ? 0 : J.k;
    for (int q = 0; q < k; q++) { r[q] = J.rows[q]; c[q] = J.cols[q]; }
    QueryParam p;
    bool wide = false;
    uint64_t fixed = 0;
    const int s = query_task(J.N, k, r, c, &p, &wide, &fixed);
    if (s < 0) return NQ_EINVAL;
    if (s > 0) {
      p.target = std::min(kQueryTarget, kQueryCap / (unsigned)J.N);
      m = (int64_t)query_frames(p);
      rows = (int)p.T + 2;
      levels = batch_query_levels(rows);
    }
  } else {
    return NQ_EINVAL;
  }
  // split queue: each level multiplies the items by at most ~8 (measured 6.2-8x); it takes the place of the list
  const int D = (J.N <= 12) ? 0 : (split_depth >= 0 ? split_depth : levels);
  int64_t ns = m;
  for (int d = 0; d < D; d++) ns *= 8;
  const int64_t per_source = 16 /*frame*/ + 4 /*slot*/;
  return m * per_source + tasks * (4 /*info*/ + (int64_t)(rows + 1) * word) + std::max(m * list, ns * (16 + 8)) +
         (int64_t)Ctrl::bytes(1) + 4096;
}

int nq_batch_set_grid(nq_batch* b, int grid) {
  if (!b || grid < 0) return NQ_EINVAL;
  if (b->submitted) return b->h->fail(NQ_EBUSY, "batch is running");
  if (b->graph) { cudaGraphExecDestroy(b->graph); b->graph = nullptr; }   // the captured launch used the old grid
  b->grid = grid;
  return NQ_OK;
}

int nq_resident_blocks(nq_handle* h, int wide, int maxt, int* blocks) {
  if (!h || !blocks || maxt < 1 || maxt >= kMaxDepth) return NQ_EINVAL;
  *blocks = h->sms * std::max(1, dfs_blocks_per_sm(wide != 0, h->block, maxt));
  return NQ_OK;
}

int nq_batch_resident_blocks(const nq_batch* b, int* blocks) {
  if (!b || !blocks) return NQ_EINVAL;
  *blocks = b->h->sms * std::max(1, dfs_blocks_per_sm(b->wide, b->block, b->maxt));
  return NQ_OK;
}

int64_t nq_batch_tasks(const nq_batch* b) { return b ? b->m : NQ_EINVAL; }
int64_t nq_batch_device_bytes(const nq_batch* b) { return b ? b->device_bytes : NQ_EINVAL; }
int64_t nq_batch_h2d_bytes(const nq_batch* b) { return b ? b->h2d_bytes : NQ_EINVAL; }

int nq_batch_submit(nq_batch* b, int use_graph) {
  if (!b) return NQ_EINVAL;
  if (b->submitted) return b->h->fail(NQ_EBUSY, "batch already submitted");
  return batch_enqueue(b, use_graph);
}

int nq_batch_poll(nq_batch* b, uint64_t* totals, int64_t max_wait_us) {
  if (!b) return NQ_EINVAL;
  if (!b->submitted) return b->h->fail(NQ_EINVAL, "batch not submitted");
  const auto t0 = std::chrono::steady_clock::now();
  for (;;) {
    cudaError_t q = cudaEventQuery(b->done);
    if (q == cudaSuccess) break;
    if (q != cudaErrorNotReady) return b->h->cuda_fail(q, "cudaEventQuery");
    const int64_t us = std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - t0).count();
    if (us >= max_wait_us) return NQ_EBUSY;
    std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
  return batch_collect(b, totals);
}

int nq_batch_run(nq_batch* b, int use_graph, uint64_t* totals) {
  if (!b) return NQ_EINVAL;
  if (int s = nq_batch_submit(b, use_graph)) return s;
  NQ_CUDA(b->h, cudaEventSynchronize(b->done));
  return batch_collect(b, totals);
}

int nq_batch_run_plain(nq_batch* b, uint64_t* totals) {
  if (!b) return NQ_EINVAL;
  nq_handle* h = b->h;
  const int nj = (int)b->jobs.size();
  unsigned char* c = (unsigned char*)b->ctrl.p;
  NQ_CUDA(h, cudaSetDevice(h->device));
  for (int j = 0; j < nj; j++) {
    uint64_t t = 0;
    if (b->sub_m[j] > 0) {
      NQ_CUDA(h, cudaMemsetAsync(c, 0, 24, b->stream));
      TaskArrays ta;
      ta.info = (uint32_t*)b->info.p; ta.sched = b->sched.p; ta.sw = b->sw; ta.wide = b->wide; ta.ra_words = b->ra_words;
      // One job per launch over its subtask range; its tasks carry job id j, which lands in slot 0.
      DfsLaunch L;
      L.tasks = ta; L.sroot = (const uint4*)b->sroot.p + b->sub_off[j]; L.sinfo = (const uint2*)b->sinfo.p + b->sub_off[j];
      L.m = b->sub_m[j]; L.cursor = (unsigned long long*)(c + 8);
      L.job_totals = (unsigned long long*)c; L.job_base = (uint32_t)j; L.err = (unsigned int*)(c + 16);
      L.maxt = b->job_maxt[j]; L.block = b->block; L.grid = b->grid; L.big = counts_need_u64(b->jobs[j].N, b->sub_m[j]);
      NQ_CUDA(h, launch_dfs(L, b->stream));
      NQ_CUDA(h, cudaMemcpyAsync(b->h_out, c, 24, cudaMemcpyDeviceToHost, b->stream));
      NQ_CUDA(h, cudaStreamSynchronize(b->stream));
      const uint32_t e = ((const uint32_t*)b->h_out)[4];
      if (e) return h->fail(derr_to_status(e), "device: %s", derr_text(e));
      t = b->h_out[0];
    }
    if (totals) totals[j] = t + b->fixed_total[j];
  }
  return NQ_OK;
}

// One launch builds the query's queue from its root frame (a parameter, so nothing is uploaded), larger boards
// take one to three more over the whole GPU, one counts and hands the count over.  Building the tasks on the host
// and running them as a batch of one took 340 us at N=10 and 990 us of 1.1 ms at N=17 (two queens).
int nq_count_completions(nq_handle* h, int N, int k, const int* rows, const int* cols, uint64_t* count) {
  if (!h || !count || k < 0 || k > 8 || (k > 0 && (!rows || !cols))) return h ? h->fail(NQ_EINVAL, "bad arguments") : NQ_EINVAL;
  if (N < 1 || N > kMaxN) return h->fail(NQ_EINVAL, "N=%d outside 1..27", N);
  for (int q = 0; q < k; q++)
    if (rows[q] < 0 || rows[q] >= N || cols[q] < 0 || cols[q] >= N) return h->fail(NQ_EINVAL, "queen outside the board");
  QueryParam p;
  bool wide = false;
  uint64_t fixed = 0;
  const int s = query_task(N, k, rows, cols, &p, &wide, &fixed);
  if (s < 0) return h->fail(NQ_EINVAL, "bad pre-placed queens");
  if (s == 0) { *count = fixed; return NQ_OK; }
  NQ_CUDA(h, cudaSetDevice(h->device));
  struct Lease {                             // its stream and buffers are this call's alone
    nq_handle* h;
    QueryRun* q = nullptr;
    ~Lease() { if (q) h->query_put(q); }
  } lease{h};
  NQ_CUDA(h, h->query_get(&lease.q));
  QueryRun& q = *lease.q;
  cudaStream_t st = q.stream;
  p.target = std::min(query_target((int)p.T + 2), kQueryCap / (unsigned)N);
  int levels = query_levels((int)p.T + 2);
  double est[kMaxDepth] = {0.0};
  if (levels > 0) query_estimate(p, est);
  for (;; levels--) {                        // a level less where the queue did not fit
    QueryBuffers b{};
    query_caps(p, est, levels, b.cap);
    size_t items = 0;
    for (int l = 0; l <= levels; l++) items += b.cap[l];
    unsigned char* c = nullptr;
    const cudaError_t room = q.ensure(1024 + (b.cap[0] + items) * sizeof(uint4) + items * sizeof(uint2), &c);
    if (room == cudaErrorMemoryAllocation && levels > 0) { cudaGetLastError(); continue; }
    NQ_CUDA(h, room);
    b.ctl = (unsigned long long*)c; b.info = (uint32_t*)(c + 128); b.sched = c + 256;
    b.tmp = (uint4*)(c + 1024);
    b.sroot[0] = b.tmp + b.cap[0];
    b.sinfo[0] = (uint2*)(b.sroot[0] + items);
    for (int l = 1; l <= levels; l++) { b.sroot[l] = b.sroot[l - 1] + b.cap[l - 1]; b.sinfo[l] = b.sinfo[l - 1] + b.cap[l - 1]; }
    NQ_CUDA(h, launch_query(p, b, wide, levels, h->sms, st));
    DfsLaunch L;
    L.tasks.info = b.info; L.tasks.sched = b.sched; L.tasks.sw = kMaxDepth; L.tasks.wide = wide;
    L.sroot = b.sroot[levels]; L.sinfo = b.sinfo[levels];
    L.m_dev = b.ctl + QueryCtl::kQueue + levels; L.qcap = b.cap[levels];
    L.cursor = b.ctl + QueryCtl::kCursor; L.job_totals = b.ctl + QueryCtl::kTotal; L.err = (unsigned int*)(b.ctl + QueryCtl::kErr);
    // Frames in the queue stand at the terminal depth or at least as deep as N^depth reaches the target.
    int depth = levels;
    for (uint64_t f = 1; f < p.target; f *= (uint64_t)N) depth++;
    L.maxt = std::max(1, (int)p.T - depth); L.block = h->block; L.grid = h->grid;
    L.big = counts_need_u64(N, p.target);      // a queue below the target stands at its terminal depth
    L.ctl = (const uint32_t*)b.ctl; L.ctl_words = QueryCtl::kWords; L.host_ctl = (uint32_t*)q.host;
    L.blocks_done = (unsigned int*)(b.ctl + QueryCtl::kErr) + 1;
    L.chained = true;
    NQ_CUDA(h, launch_dfs(L, st));
    NQ_CUDA(h, cudaStreamSynchronize(st));
    bool fits = true;
    for (int l = 1; l <= levels; l++) fits = fits && q.host[QueryCtl::kQueue + l] <= b.cap[l];
    if (fits) break;
  }
  const uint32_t e = (uint32_t)q.host[QueryCtl::kErr];
  if (e) return h->fail(derr_to_status(e), "device: %s", derr_text(e));
  *count = q.host[QueryCtl::kTotal] + fixed;
  return NQ_OK;
}

}  // extern "C"
