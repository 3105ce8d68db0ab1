// nq_noalloc.cu -- exec_solutions for callers that cannot allocate device memory.
//
// Some callers of this library must not call cudaMalloc/cudaFree after they
// start: a serving process whose device memory is owned and pre-reserved by
// another allocator (a framework's caching allocator, a fixed per-tenant
// budget), or a latency-critical loop where an allocation's implicit device
// synchronisation would stall every other stream.  This entry point runs the
// same prepare and DFS kernels as nq_exec_solutions_device, but its scratch
// (control words, task info, per-depth schedules, and the split queue in what
// is left) lives in one file-scope __device__ array of fixed size, which every
// GPU that loads the library holds until the process exits.  Nothing here
// allocates.
//
// Limits: at most kMaxRecords records per call (N <= 17 at the default
// presets) and schedules of at most kMaxWords depths.  All calls share the
// one array, so calls that overlap on the GPU (different streams or host
// threads at the same time) race: the caller must serialise them.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../../include/nqueens_gb300.h"
#include "nq_common.cuh"
#include "nq_internal.h"

namespace {

constexpr int64_t kMaxRecords = 131072;
constexpr int kMaxWords = 24;                        // schedule words per task (depths 0..23)
constexpr size_t kCtrlBytes = 256;                   // totals, queue cursor, error word, queue length
constexpr size_t kRootBytes = (size_t)kMaxRecords * sizeof(uint4);
constexpr size_t kInfoBytes = (size_t)kMaxRecords * sizeof(uint2);   // info words, and room to round the parts to 16 bytes
constexpr size_t kSchedBytes = (size_t)kMaxRecords * kMaxWords * sizeof(uint32_t);
constexpr size_t kScratchBytes = kCtrlBytes + kRootBytes + kInfoBytes + kSchedBytes;   // 15.0 MiB + 256 B
constexpr int kMaxDevices = 64;

std::mutex g_setup_mu;
void* g_scratch[kMaxDevices] = {nullptr};

}  // namespace

// The scratch itself.  In host code this name is only a stand-in for the
// symbol, not a device address: the address each device uses comes from
// cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char nq_noalloc_scratch[kScratchBytes];

namespace {

// Set-up, once per device, with that device current.
int scratch_for_current_device(void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return NQ_ECUDA;
  std::lock_guard<std::mutex> lk(g_setup_mu);
  if (!g_scratch[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, nq_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) return NQ_ECUDA;
    g_scratch[dev] = p;
  }
  *out = g_scratch[dev];
  return NQ_OK;
}

}  // namespace

extern "C" int nq_exec_solutions_noalloc(int N, const nq_record* d_records, int64_t m, int start_min,
                                         uint64_t* d_solutions, uint64_t* d_total, void* stream) {
  using namespace nq;
  if (N < 6 || N > kMaxN || m < 0 || !d_total || (m > 0 && !d_records)) return NQ_EINVAL;
  if (m > kMaxRecords) return NQ_EINVAL;                // beyond the fixed scratch: rejected, never truncated
  const int s = start_min < 0 ? 1 : start_min;
  const int maxt = N - 2 - s < 1 ? 1 : N - 2 - s;       // stack frames; schedule words maxt + 1
  if (maxt + 1 > kMaxWords) return NQ_EINVAL;
  void* base = nullptr;
  if (int st = scratch_for_current_device(&base)) return st;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* c = (unsigned char*)base;
  unsigned long long* totals = (unsigned long long*)c;
  unsigned long long* cursor = (unsigned long long*)(c + 8);
  unsigned int* err = (unsigned int*)(c + 16);
  if (m == 0) {
    if (cudaMemsetAsync(d_total, 0, 8, st) != cudaSuccess) return NQ_ECUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? NQ_OK : NQ_ECUDA;
  }
  // info and schedules first, then the roots (unsplit) or as many queue items as fit
  PrepareSplit P;
  P.N = N; P.m = m; P.rec = (const uint4*)d_records; P.sw = maxt + 1; P.err = err; P.total = totals;
  P.per_task = (unsigned long long*)d_solutions; P.qn = (unsigned long long*)(c + 24);
  size_t used = kCtrlBytes;
  P.info = (uint32_t*)(c + used);
  used += ((size_t)m * sizeof(uint32_t) + 15) & ~(size_t)15;
  P.sched = (uint32_t*)(c + used);
  used += ((size_t)m * P.sw * sizeof(uint32_t) + 15) & ~(size_t)15;
  P.qcap = (kScratchBytes - used) / sizeof(uint4);
  // Split as deep as the usual rule says while the queue should fit: its items a task, from the generated lists
  // (one level makes 4.5 / 5.4 / 6.2 / 7.1 at 10 / 11 / 12 / 13 rows, two make 3.9 / 4.7 / 5.5 / 6.3 each).  A
  // queue that does not fit after all leaves the DFS without work, and the call runs again with a level less
  // (the scratch always holds the tasks).  us with no, one and two levels: 20,011 records of N=16 354 / 288 /
  // 219, of N=17 1640 / 972 / 665.
  int D = choose_split(m, maxt);
  for (; D > 0; D--) {
    const double first = std::max(1.0, 0.8 * maxt - 3.2), next = std::max(1.0, 0.8 * maxt - 4.0);
    if ((double)m * (D == 1 ? first : D == 2 ? next * next : next * next * next) <= (double)P.qcap) break;
  }
  uint64_t hc[4];
  for (;; D--) {
    // the array keeps the previous call's contents: clear what must start at zero
    if (cudaMemsetAsync(c, 0, 32, st) != cudaSuccess) return NQ_ECUDA;
    DfsLaunch L;
    if (D == 0) {
      P.root = (uint4*)(c + used);
      L.m = m;
    } else {
      P.sroot = (uint4*)(c + used);
      L.sroot = P.sroot; L.depth = (uint32_t)D; L.m_dev = P.qn; L.qcap = P.qcap;
    }
    P.ra_words = !ra_in_rd(N, start_min, D);
    if (launch_prepare_split(D, m, P, st) != cudaSuccess) return NQ_ECUDA;
    L.tasks.root = P.root; L.tasks.info = P.info; L.tasks.sched = P.sched; L.tasks.sw = P.sw; L.tasks.wide = false; L.tasks.ra_words = P.ra_words;
    L.cursor = cursor; L.job_totals = totals;
    L.per_task = (unsigned long long*)d_solutions; L.err = err; L.maxt = maxt - D < 1 ? 1 : maxt - D; L.block = 128; L.grid = 0;
    L.chained = true;
    L.big = counts_need_u64(N, m);
    if (launch_dfs(L, st) != cudaSuccess) return NQ_ECUDA;
    if (cudaMemcpyAsync(d_total, totals, 8, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return NQ_ECUDA;
    if (cudaMemcpyAsync(hc, c, 32, cudaMemcpyDeviceToHost, st) != cudaSuccess) return NQ_ECUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return NQ_ECUDA;
    if (D == 0 || hc[3] <= P.qcap) break;
  }
  const uint32_t herr = (uint32_t)hc[2];
  if (herr & DERR_DEPTH) return NQ_ESTACK;
  if (herr & DERR_SHIFT) return NQ_EPRESET;
  if (herr) return NQ_EINVAL;
  return NQ_OK;
}
