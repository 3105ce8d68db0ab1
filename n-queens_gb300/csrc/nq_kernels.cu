// nq_kernels.cu -- sm_103a kernels of the constellation DFS.
//
// prepare_kernel, prepare_split_kernel: one thread per constellation record.
//   It runs the task decision tree of build_soa_for_range
//   (356Py_savesp_narrow.py:1971-2169) and walks the SQ* state machine once
//   (356Py:689-756 does this per thread inside the reference kernel) to write
//   the task's root frame, info word and per-depth schedule, and for a single
//   list the queue of its depth-D frames.
//
// dfs_kernel: persistent, explicit-stack bitboard DFS replacing
//   kernel_dfs_iter_gpu_maxd14..21 (356Py:618-1747) and dfs_iter
//   (356Py:1837-1967).  Every lane runs its own task; a lane whose task is
//   done takes the next one from the warp's pool, which the warp fills from a
//   global queue, and when the queue is empty part of a task of a busy lane
//   of its warp.  Each step every busy lane
//   expands exactly one candidate queen, so lanes stay converged on the same
//   short instruction sequence whatever their task, depth or SQ* variant:
//   the variant lives in the schedule word read from shared memory, not in
//   control flow; the word is laid out so the child row takes two funnel
//   shifts and no field extraction (nq_common.cuh).  The current frame is in
//   registers; saved frames (only those with candidates left, as the
//   reference's packed stack) sit in shared memory, interleaved by lane so
//   every access is conflict-free, above a sentinel frame whose candidates
//   all die, which a finished lane works on until the next check.
//   Bound by shared-memory bandwidth: N=19 takes 8.85 wavefronts a step of
//   32 lanes (a 16-byte frame out, one in, a word), 93 % of that pipe's rate,
//   and 27.0 warp instructions (11.2 on the ALU pipe, 11.4 on FMA) at 72 %
//   issue.
//   Counts are summed per lane in u64 and flushed per job with one atomicAdd
//   per warp (shuffle tree) at exit or per task when the job id changes.
#include <algorithm>
#include <type_traits>

#include "nq_common.cuh"
#include "nq_internal.h"

namespace nq {

constexpr unsigned FULL = 0xFFFFFFFFu;

// DFS steps each lane takes between two checks for finished lanes (flush +
// refill), unrolled.  A lane that runs dry mid-round idles for the rest of the
// round; a check costs two ballots, so checking less often wins until that
// idle time dominates.  At most 30: the sentinel frame holds 31 candidates.
// N=19 / N=17, ms: 30 steps 63.29 / 1.334 (unrolled 10 63.55 / 1.332), 20 63.90 /
// 1.362, 16 64.22 / 1.380, 10 65.12 / 1.434.
constexpr int kStepsPerCheck = 30;
// Searches of at most kShortDepth rows (2 to 40 steps an item) check twice as often, so lanes wait less for their
// next item: us of 256 jobs of N=10..13 replayed 262 -> 258, of the counts N=6..13 300 -> 292.  At 7 rows 64 jobs of
// N=12..15 took 1241 us for 1213; 10 steps a check 1270, 6 steps 1311.  A kernel of its own: a branch between the
// two loops in one kernel took N=19 from 63.4 to 63.9 ms.
constexpr int kShortDepth = 6, kShortSteps = 15;

// A warp takes 32 queue items at a time (one atomic and one coalesced load round for the 32), less towards
// the end of the queue: 1/8 of its even share of what is left, at least 8, so the warps end together.
// Taking the items one by one took 74.1 ms at N=19 and 1.715 at N=17 where the pool took 73.2 and 1.675.  Now
// N=14 / 16 / 17, ms: 0.0247 / 0.261 / 1.334; a share of 1/4 0.0245 / 0.257 / 1.364 (N=19 63.66 against 63.29); at
// least 1 0.0492 / 0.286 / 1.362, at least 16 0.0227 / 0.259 / 1.340 (N=19 63.46).  Short searches (kShortDepth) take
// the whole even share, their items are small enough: 256 jobs of N=9..12, share 1/8 / 1/4 / 1/2 / 1: 66.7 / 61.5 / 56.2
// / 54.6 us, of N=10..14 784 / 778 / 780 / 770; 32 throughout 55.8 and 759, but 64 jobs of N=9..12 37.0 for 33.6.
constexpr float kChunkShare = 8.0f, kShortShare = 1.0f;
constexpr unsigned kMinChunk = 8;
// A frame is given to a lane without work when it is at least this many levels above the terminal depth
// (3 / 5 / 7: N=14 0.0244 / 0.0247 / 0.0262 ms, N=16 0.262 / 0.261 / 0.265, N=17 1.335 / 1.334 / 1.326).
constexpr int kGiveRows = 5;
// What a pool entry needs besides its frame, ready when it is loaded: terminal depth (5 bits), weight (2),
// root count (1), N (5), depth of its first word (5) and what to do with it.
constexpr uint32_t kItemWork = 1u << 18, kItemSpare = 1u << 19;   // search it; more columns than rows are left

template <bool WIDE> using WordT = QueryWord<WIDE>;

// ---------------------------------------------------------------------------
// prepare
// ---------------------------------------------------------------------------
// One record's task: info word, root, and its ops in order, emit(depth, op); returns T or -1.
template <bool WIDE, class Emit>
__device__ __forceinline__ int prepare_task(int N, const uint4 r, int sw, Root& rt, uint32_t& info, unsigned int* err, Emit&& emit) {
  uint32_t status = TS_OK;
  rt = {0, 0, 0, 0};
  uint32_t root_count = 0;
  int T = -1;
  int wexp = 0;
  bool fits = true;
  if (N < 6 || N > kMaxN) {
    status = TS_BADN;
  } else {
    const TaskHead h = decode_record(N, r.x, r.y, r.z, r.w);
    wexp = h.wexp;
    status = h.status;
    if (status == TS_OK) {
      const int lim = sw < kMaxDepth ? sw : kMaxDepth;
      T = walk_schedule(N, h, &rt, &root_count, lim, [&](int d, const Op& o) {
        fits = fits && (WIDE ? wide_fits(o) : compact_fits(o, N));
        emit(d, o);
      });
      if (T == -2) status = (lim < kMaxDepth) ? TS_DEPTH : TS_NOTERM;
      else if (T >= 0 && !fits) status = TS_FORMAT;   // never seen (N=6..21, presets 4-7): fail loudly rather than miscount
    }
  }
  if (status != TS_OK) {
    atomicOr(err, status == TS_BAD_SHIFT ? DERR_SHIFT : status == TS_DEPTH ? DERR_DEPTH
                : status == TS_NOTERM ? DERR_NOTERM : status == TS_FORMAT ? DERR_FORMAT : DERR_BADN);
    T = -1; rt = {0, 0, 0, 0}; root_count = 0;
  }
  info = info_pack((T < 0) ? INFO_NO_DFS : (uint32_t)T, (uint32_t)wexp, root_count, (uint32_t)N, status);
  return T;
}

__device__ __forceinline__ void max_depth_of(unsigned int* tmax, int T) {
  const unsigned v = __reduce_max_sync(FULL, (unsigned)(T < 0 ? 0 : T));
  if ((threadIdx.x & 31u) == 0 && v) atomicMax(tmax, v);
}

// RA of a task's rows as bits of the root's rd: each stands as many places above its own as rows follow.
struct RaInRd {
  unsigned long long bits = 0;
  uint32_t rows = 0;                  // below the root so far
  __device__ __forceinline__ void add(const Op& o) { rows += o.s; bits |= (unsigned long long)o.ra << rows; }
  __device__ __forceinline__ uint32_t at(uint32_t row, unsigned int* err) const {   // as seen from `row` below the root
    const unsigned long long v = bits >> row;
    if (v >> 32) atomicOr(err, DERR_FORMAT);     // not with ra_in_rd's bound: fail loudly rather than miscount
    return (uint32_t)v;
  }
};

template <bool WIDE>
__global__ void __launch_bounds__(256) prepare_kernel(int N, int64_t m, const unsigned* m_dev,
                                                      const uint4* rec, uint4* __restrict__ root,
                                                      uint32_t* __restrict__ info,
                                                      typename WordT<WIDE>::type* __restrict__ sched, int sw, bool ra_words,
                                                      int64_t offset, unsigned int* err, unsigned int* tmax,
                                                      unsigned int* n_out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  chain_next();
  chain_wait();
  if (m_dev) m = *m_dev;
  if (i == 0) *n_out = (unsigned int)m;
  int T = -1;
  if (i < m) {
    const int64_t t = offset + i;
    Root rt;
    uint32_t in;
    RaInRd ra;
    T = prepare_task<WIDE>(N, rec[i], sw, rt, in, err, [&](int d, const Op& o) {
      if constexpr (WIDE) sched[t * sw + d] = make_uint2(device_wide_x(o), o.ra);
      else sched[t * sw + d] = device_compact(o, ra_words);
      ra.add(o);
    });
    if (!WIDE && !ra_words) rt.rd |= ra.at(0, err);
    root[t] = make_uint4(rt.ld, rt.rd, rt.col, T < 0 ? 0u : rt.avail);
    info[t] = in;
  }
  max_depth_of(tmax, T);              // deepest schedule of the launch, for sizing the DFS stack
}

cudaError_t launch_prepare(int N, int64_t m, const unsigned int* m_dev, const uint4* records, const TaskArrays& out,
                           int64_t offset, unsigned int* err, cudaStream_t st, unsigned int* tmax, unsigned int* n_out) {
  if (m <= 0) return cudaSuccess;
  const int B = 256;
  const unsigned G = (unsigned)((m + B - 1) / B);
  if (out.wide)
    return launch_after(prepare_kernel<true>, G, B, 0, st, N, m, m_dev, records, out.root, out.info, (uint2*)out.sched, out.sw,
                        out.ra_words, offset, err, tmax, n_out);
  return launch_after(prepare_kernel<false>, G, B, 0, st, N, m, m_dev, records, out.root, out.info, (uint32_t*)out.sched, out.sw,
                      out.ra_words, offset, err, tmax, n_out);
}

// ---------------------------------------------------------------------------
// Schedule word decoding shared by the split and DFS kernels
// ---------------------------------------------------------------------------
struct Dec { uint32_t s, la, ra, fc; bool term; };
// word of depth k of a task of board N and terminal depth T
__device__ __forceinline__ Dec decode(uint32_t w, uint32_t N, uint32_t k, uint32_t T) {
  const Op o = unpack_compact(w ^ C_NOLOOK, (int)N, k == T);
  return Dec{o.s, o.la, o.ra, o.fc, k == T};
}
__device__ __forceinline__ Dec decode(uint2 w, uint32_t, uint32_t k, uint32_t T) {
  const uint32_t s = w.x & W_S;
  return Dec{s, s ? (w.x >> (32 - s)) : 0u, w.y, ~w.x & W_NOLOOK, k == T};
}

// ---------------------------------------------------------------------------
// prepare + split of a single-N list in one launch: each thread prepares its
// record, counts the task's depth-D frames, takes its warp's slots with one
// atomic and writes them, the words of depths 0..D-1 still in registers.  The
// queue's length stays on the device (the DFS reads it there), so a short list
// needs no read-back between the launches.  Tasks that end above depth D and
// tasks without a DFS are settled here.  D = 0: the tasks themselves are the
// queue.  Bound by latency and the record walk (about 300 instructions a
// record); the three launches it replaces kept 28 ops a record in local memory
// and read tasks back from memory twice.
// ---------------------------------------------------------------------------
template <int K, int D, class W, class F>
__device__ __forceinline__ void frames_at(uint32_t ld, uint32_t rd, uint32_t col, uint32_t avail, const W* w, uint32_t N, uint32_t T, uint32_t& direct, F&& f) {
  if constexpr (K == D) {
    f(make_uint4(ld, rd, col, avail));
  } else {
    const Dec o = decode(w[K], N, (uint32_t)K, T);
    const uint32_t bm = (1u << N) - 1u;
    while (avail) {
      const uint32_t bit = avail & (0u - avail);
      avail ^= bit;
      const uint32_t nld = ((ld | bit) << o.s) | o.la, nrd = ((rd | bit) >> o.s) | o.ra, ncol = col | bit;
      uint32_t nf = bm & ~(nld | nrd | ncol);
      if (o.fc && (bm & ~((nld << 1) | (nrd >> 1) | ncol)) == 0u) nf = 0;
      if (o.term) { direct += nf != 0u ? 1u : 0u; continue; }   // SQd2B: LA bit 0
      if (nf) frames_at<K + 1, D>(nld, nrd, ncol, nf, w, N, T, direct, f);
    }
  }
}

template <int D>
__global__ void __launch_bounds__(256) prepare_split_kernel(const PrepareSplit a) {
  chain_next();
  chain_wait();
  if (a.stamp && blockIdx.x == 0 && threadIdx.x == 0) *a.stamp = device_ns();
  const int64_t m = a.m_dev ? (int64_t)*a.m_dev : a.m;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (D == 0 && t == 0) *a.qn = (unsigned long long)m;
  if ((int64_t)blockIdx.x * blockDim.x >= m) return;
  const unsigned lane = threadIdx.x & 31u;
  Root rt = {0, 0, 0, 0};
  uint32_t in = 0, w[D > 0 ? D : 1] = {0};
  int T = -1;
  RaInRd ra;
  uint32_t rows_d = 0;                           // rows from the root to depth D
  if (t < m) {
    T = prepare_task<false>(a.N, a.rec[t], a.sw, rt, in, a.err, [&](int d, const Op& o) {
      a.sched[t * a.sw + d] = device_compact(o, a.ra_words);
      Op p = o;
      if (d < D) { rows_d += o.s; p.ra = 0; }    // above depth D the words below apply it
#pragma unroll
      for (int k = 0; k < D; k++)
        if (d == k) w[k] = device_compact(o, true);
      ra.add(p);
    });
    a.info[t] = in;
    if (D == 0) {
      if (!a.ra_words) rt.rd |= ra.at(0, a.err);
      a.root[t] = make_uint4(rt.ld, rt.rd, rt.col, T < 0 ? 0u : rt.avail);
      if (a.per_task) a.per_task[t] = 0;      // the DFS adds the task's counts
    }
  }
  if (a.tmax) max_depth_of(a.tmax, T);
  if constexpr (D > 0) {
    uint32_t n = 0, direct = 0;
    if (T >= 0) frames_at<0, D>(rt.ld, rt.rd, rt.col, rt.avail, w, (uint32_t)a.N, (uint32_t)T, direct, [&](uint4) { n++; });
    else if (t < m && info_status(in) == TS_OK) direct = info_root(in);
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, incl, o);
      if ((int)lane >= o) incl += v;
    }
    unsigned long long base = 0;
    if (lane == 31 && incl) base = atomicAdd(a.qn, (unsigned long long)incl);
    base = __shfl_sync(FULL, base, 31) + (incl - n);
    if (n && base + n <= a.qcap) {            // a queue that does not fit is sized by qn and built again
      uint32_t dummy = 0;
      const uint32_t later = a.ra_words ? 0u : ra.at(rows_d, a.err);
      frames_at<0, D>(rt.ld, rt.rd, rt.col, rt.avail, w, (uint32_t)a.N, (uint32_t)T, dummy, [&](uint4 f) {
        a.sroot[base++] = make_uint4(f.x, f.y | later, f.z, (uint32_t)t);
      });
    }
    const unsigned long long dv = (unsigned long long)direct << info_wexp(in);
    if (t < m && a.per_task) a.per_task[t] = dv;
    unsigned long long v = dv;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    if (lane == 0 && v) atomicAdd(a.total, v);
  }
}

cudaError_t launch_prepare_split(int D, int64_t m_max, const PrepareSplit& a, cudaStream_t st) {
  if (m_max <= 0) return cudaSuccess;
  const unsigned B = 256, G = (unsigned)((m_max + B - 1) / B);
  switch (D) {
    case 0: return launch_after(prepare_split_kernel<0>, G, B, 0, st, a);
    case 1: return launch_after(prepare_split_kernel<1>, G, B, 0, st, a);
    case 2: return launch_after(prepare_split_kernel<2>, G, B, 0, st, a);
    case 3: return launch_after(prepare_split_kernel<3>, G, B, 0, st, a);
    default: return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------
// split of a batch's source lists (the records of a board, the frames of a
// query) in one launch each way: list_count_kernel counts every source's
// frames D levels down and gives them slots in its list's queue;
// list_write_kernel writes them for every job, jobs of one board from the same
// list, so each job's items are one range of the batch's queue.  Counts
// settled above that depth are summed per list.  Lists are padded to warps.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int find_range(const unsigned long long* __restrict__ ends, int n, unsigned long long i) {
  int lo = 0, hi = n - 1;              // the first range whose end is above i
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (i < ends[mid]) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// One source's frames: f(frame) for each, the settled count into direct.
template <class W, class F>
__device__ __forceinline__ void source_frames(const BatchList& l, uint32_t r, const ListArgs& a, uint32_t d, uint32_t& task,
                                              uint32_t& in, uint32_t& direct, F&& f) {
  const uint4 s = a.src[l.src0 + r];
  task = l.query ? l.task0 : l.task0 + r;
  in = a.info[task];
  const uint32_t T = info_T(in), N = info_N(in);
  if (T == INFO_NO_DFS || info_status(in) != TS_OK) {
    if (info_status(in) == TS_OK) direct += info_root(in);
    return;
  }
  const W* w = (const W*)a.sched + (size_t)task * a.sw + d;
  switch (l.D) {
    case 0: if (s.w) f(s); break;
    case 1: frames_at<0, 1>(s.x, s.y, s.z, s.w, w, N, T - d, direct, f); break;
    case 2: frames_at<0, 2>(s.x, s.y, s.z, s.w, w, N, T - d, direct, f); break;
    default: frames_at<0, 3>(s.x, s.y, s.z, s.w, w, N, T - d, direct, f); break;
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(256) list_count_kernel(const ListArgs a) {
  using W = typename WordT<WIDE>::type;
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  chain_next();
  chain_wait();
  if ((i & ~31ull) >= a.total) return;
  const int li = find_range(a.ends, a.n, i);
  const BatchList l = a.lists[li];
  const uint32_t r = (uint32_t)(i - (li ? a.ends[li - 1] : 0ull));
  const ListState st = a.state[li];
  uint32_t n = 0, direct = 0, task, in = 0;
  if (r < st.n) source_frames<W>(l, r, a, st.depth, task, in, direct, [&](uint4) { n++; });
  uint32_t incl = n;
  const unsigned lane = threadIdx.x & 31u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(FULL, incl, o);
    if ((int)lane >= o) incl += v;
  }
  unsigned long long base = 0;
  if (lane == 31 && incl) base = atomicAdd(&a.state[li].items, (unsigned long long)incl);
  base = __shfl_sync(FULL, base, 31) + (incl - n);
  a.off[i] = (uint32_t)base;
  unsigned long long v = (unsigned long long)direct << info_wexp(in);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  if (lane == 0 && v) atomicAdd(&a.state[li].settled, v);
}

template <bool WIDE>
__global__ void __launch_bounds__(256) list_write_kernel(const ListArgs a, const BatchJob* __restrict__ jobs,
                                                         uint4* __restrict__ sroot, uint2* __restrict__ sinfo) {
  using W = typename WordT<WIDE>::type;
  const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.total) return;
  const int ji = find_range(a.ends, a.n, i);
  const BatchJob j = jobs[ji];
  const uint32_t r = (uint32_t)(i - (ji ? a.ends[ji - 1] : 0ull));
  const BatchList l = a.lists[j.list];
  const ListState st = a.state[j.list];
  if (r >= st.n) return;
  unsigned long long at = j.base + a.off[j.off0 + r];
  uint32_t task = 0, in, direct = 0;
  source_frames<W>(l, r, a, st.depth, task, in, direct, [&](uint4 f) {
    sroot[at] = f;
    sinfo[at++] = make_uint2(task, (st.depth + l.D) | (j.job << 5));
  });
}

cudaError_t launch_list_count(const ListArgs& a, bool wide, cudaStream_t st) {
  if (a.total == 0) return cudaSuccess;
  const unsigned G = (unsigned)((a.total + 255) / 256);
  return wide ? launch_after(list_count_kernel<true>, G, 256, 0, st, a) : launch_after(list_count_kernel<false>, G, 256, 0, st, a);
}

cudaError_t launch_list_write(const ListArgs& a, const BatchJob* jobs, uint4* sroot, uint2* sinfo, bool wide, cudaStream_t st) {
  if (a.total == 0) return cudaSuccess;
  const unsigned G = (unsigned)((a.total + 255) / 256);
  if (wide) list_write_kernel<true><<<G, 256, 0, st>>>(a, jobs, sroot, sinfo);
  else list_write_kernel<false><<<G, 256, 0, st>>>(a, jobs, sroot, sinfo);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// queue order: largest estimated subtree first.  The reference reorders its
// task list by a hand-tuned cost score before launching (chunkshape148 score
// key and mark-distance risk table, 356Py_savesp_narrow.py:4310-4372 and
// 3646-3748) so long tasks start early instead of forming the tail.  Here the
// estimate is the frame's candidate count plus the free squares of the next
// six rows ignoring later placements, popc(bm & ~((ld << k) | (rd >> k) | col))
// for k = 1..6: at N=16 (split depth 2) its rank correlation with the true
// subtree size is 0.73.  The keys (0..255) are sorted on the device by a
// counting sort: histogram, a descending exclusive scan, and a scatter with
// one atomic per warp and key.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cost_key(const uint4 f, uint32_t bm) {
  uint32_t k = __popc(f.w);
#pragma unroll
  for (int s = 1; s <= 6; s++) k += __popc(bm & ~((f.x << s) | (f.y >> s) | f.z));
  return k < 255u ? k : 255u;
}

__global__ void __launch_bounds__(256) order_hist_kernel(int64_t m, const uint4* __restrict__ sroot,
                                                         const uint4* __restrict__ root, const uint32_t* __restrict__ info,
                                                         uint8_t* __restrict__ keys, unsigned int* hist) {
  __shared__ unsigned int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < m) {
    uint4 f = sroot ? sroot[q] : root[q];
    const uint32_t bm = (1u << info_N(info[sroot ? f.w : (uint32_t)q])) - 1u;
    if (sroot) f.w = bm & ~(f.x | f.y | f.z);
    const uint32_t key = cost_key(f, bm);
    keys[q] = (uint8_t)key;
    atomicAdd(&h[key], 1u);
  }
  __syncthreads();
  if (h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], h[threadIdx.x]);
}

// offs[k] = number of items with a larger key (one block of 256 threads)
__global__ void __launch_bounds__(256) order_scan_kernel(const unsigned int* __restrict__ hist,
                                                         unsigned int* __restrict__ offs) {
  __shared__ unsigned int v[256];
  const int t = threadIdx.x;
  v[t] = hist[255 - t];                // descending key order
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {   // inclusive scan
    const unsigned int x = (t >= o) ? v[t - o] : 0u;
    __syncthreads();
    v[t] += x;
    __syncthreads();
  }
  offs[255 - t] = v[t] - hist[255 - t];
}

__global__ void __launch_bounds__(256) order_scatter_kernel(int64_t m, const uint8_t* __restrict__ keys,
                                                            unsigned int* offs, uint32_t* __restrict__ order) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned lane = threadIdx.x & 31u;
  const bool active = q < m;
  const unsigned live = __ballot_sync(FULL, active);
  if (!active) return;
  const uint32_t key = keys[q];
  const unsigned same = __match_any_sync(live, key);      // lanes of this warp with the same key
  const int leader = __ffs(same) - 1;
  unsigned base = 0;
  if ((int)lane == leader) base = atomicAdd(&offs[key], (unsigned)__popc(same));
  base = __shfl_sync(same, base, leader);
  order[base + __popc(same & ((1u << lane) - 1u))] = (uint32_t)q;
}

cudaError_t launch_order(int64_t m, const uint4* sroot, const TaskArrays& ta, uint8_t* keys,
                         unsigned int* hist_offs, uint32_t* order, cudaStream_t st) {
  if (m <= 0) return cudaSuccess;
  const unsigned G = (unsigned)((m + 255) / 256);
  cudaError_t e = cudaMemsetAsync(hist_offs, 0, 256 * sizeof(unsigned int), st);
  if (e != cudaSuccess) return e;
  order_hist_kernel<<<G, 256, 0, st>>>(m, sroot, ta.root, ta.info, keys, hist_offs);
  order_scan_kernel<<<1, 256, 0, st>>>(hist_offs, hist_offs + 256);
  order_scatter_kernel<<<G, 256, 0, st>>>(m, keys, hist_offs + 256, order);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// DFS
// ---------------------------------------------------------------------------
struct DfsArgs {
  const uint4* root;          // task roots (when sroot == nullptr the queue holds tasks)
  const uint32_t* info;
  const void* sched;
  int sw;
  const uint4* sroot;         // split queue: subtask frames, and ...
  const uint2* sinfo;         // ... {task, depth | job << 5}; or, where this is null, the task in the frames' w and ...
  uint32_t depth;             // ... all of them at this depth (their candidates follow from ld, rd and col)
  int64_t m;                  // queue length, ...
  const unsigned long long* m_dev;   // ... or where it stands on the device (above qcap: the queue did not fit, no work)
  unsigned long long qcap;
  const uint32_t* order;
  unsigned long long* cursor;
  unsigned long long* job_totals;
  uint32_t job_base;
  unsigned long long* per_task;
  unsigned int* err;
  int maxt;
  const uint32_t* ctl;        // copied to host_ctl by the last block to end, where that is set
  unsigned ctl_words;
  unsigned int* blocks_done;
  uint32_t* host_ctl;
  unsigned long long* stamp;
};

__device__ __forceinline__ void flush_job(const DfsArgs& a, unsigned job, unsigned long long v) {
  if (v) atomicAdd(a.job_totals + (job - a.job_base), v);
}

// Shared memory per lane: the sentinel's frame, frames at depths 0..maxt and the base frame's slot, and
// schedule words 0..maxt with the count word behind them.
__host__ __device__ constexpr int stack_slots(int maxt) { return maxt + 3; }
__host__ __device__ constexpr int word_slots(int maxt) { return maxt + 2; }

size_t dfs_smem_bytes(bool wide, int block, int maxt) {
  return (size_t)block * ((size_t)stack_slots(maxt) * sizeof(uint4) + (size_t)word_slots(maxt) * (wide ? 8 : 4));
}

// Shared-memory accesses of the step at 32-bit shared-window addresses.
__device__ __forceinline__ uint32_t lds_word(uint32_t a, uint32_t) {
  uint32_t w;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(a));
  return w;
}
__device__ __forceinline__ uint2 lds_word(uint32_t a, uint2) {
  uint2 w;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w.x), "=r"(w.y) : "r"(a));
  return w;
}

// The sentinel frame under a lane's stack feeds a lane that has run out of work: its word is the count
// word, so each of its 31 candidates dies and is counted, and a check takes the used ones off the lane's
// count.  kStepsPerCheck <= 30 steps therefore never pop below it, and the step tests neither the stack's
// depth nor the lane's activity.
constexpr uint32_t kSentinelAvail = 0xFFFFFFFEu;   // bits 1..31: ld + bit stays odd (ld = 1), so bit 31 of nld is set
static_assert(kStepsPerCheck <= 30, "the sentinel holds 31 candidates, and one has to be left at a check");

enum WordForm { kRaInRd, kRaInWords, kWideWords };   // compact words without and with RA, wide words

// One lane's DFS state and its step.  Every lane runs the same predicated sequence each step: resume a
// saved frame if the current one is exhausted, take the lowest candidate, save the frame with the rest,
// build the child with the depth's schedule word and make it the current frame, without candidates if the
// look-ahead rejects it, so the next step resumes the saved frame.
//  - The frame is stored whether or not candidates are left (the slot above the stack is free) and only the
//    stack pointer moves by the test: the store costs the same wavefronts either way, and the one select
//    left is the child's candidates.  Selecting between parent and child (four selects and a predicate
//    passed into the store): N=19 84.6 ms, this form 75.1.
//  - A solution is a frame in the base row: it has one column left, its word is the count word, and the
//    step adds that word's flag.  Comparing each step's depth with the terminal one and masking the child
//    there (3 instructions more, 1 % fewer steps): N=19 71.8 ms, this form 66.6; N=17 1.63, 1.49.
//  - rest = avail & (avail - 1), bit = avail - rest, instead of bit = avail & -avail: 66.6 -> 65.0.
//  - RA in rd instead of the words (one op): 65.0 -> 63.6.
// '+' and '-' replace '|' and '&~' where the bits are disjoint (a candidate is never in ld or rd, and
// always one of the free columns), so those ops issue on the FMA pipe as well as the ALU pipe.
// Per-task counts are u32 (BIG: u64, where a queue item may count 2^32 solutions).
template <WordForm FORM, bool BIG>
struct Lane {
  // A frame is {ld, rd, fr, avail}: fr holds the columns still free at the frame's
  // row (one fewer per level, so a frame's depth is popc(root fr) - popc(fr) and
  // needs no field of its own) and avail the candidates, a subset of fr.
  uint32_t ld = 0, rd = 0, fr = 0, avail = 0;
  uint32_t sp = 0;      // shared address of the next free frame of this lane's stack
  uint32_t sw0 = 0;     // shared address of the word of the depth where popc(fr) == 0 (word d sits at
                        // sw0 - popc(fr) * row, row = BLOCK words, since popc(fr) = R - d, R = popc(root fr))
  uint32_t ram = 0;     // RA in the words: the bits where RA << s may sit (compact_ra_mask)
  typename std::conditional<BIG, unsigned long long, uint32_t>::type cnt = 0;

  template <int BLOCK>
  __device__ __forceinline__ void step() {
    constexpr bool WIDE = FORM == kWideWords;
    using W = typename WordT<WIDE>::type;
    constexpr uint32_t F = BLOCK * (uint32_t)sizeof(uint4);
    constexpr uint32_t ROW = BLOCK * (uint32_t)sizeof(W);
    // resume: the condition is formed in a predicate register inside the block, so no 0/1 value is
    // materialised for it
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %3, 0;\n\t"
                 "@p sub.u32 %4, %4, %5;\n\t@p ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+r"(ld), "+r"(rd), "+r"(fr), "+r"(avail), "+r"(sp) : "n"(F));
    const uint32_t pf = __popc(fr);                  // R - depth
    const uint32_t rest = avail & (avail - 1u);
    const uint32_t bit = avail - rest;
    const W w = lds_word(sw0 - pf * ROW, W{});
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(sp), "r"(ld), "r"(rd), "r"(fr), "r"(rest) : "memory");
    if (rest != 0u) sp += F;
    // nld = (x << s) | LA in one funnel shift of the word (LA in its top s bits, s in its low 5)
    uint32_t wx, nld, nrd, y = rd + bit;
    if constexpr (WIDE) wx = w.x; else wx = w;
    asm("shf.l.wrap.b32 %0, %1, %2, %1;" : "=r"(nld) : "r"(wx), "r"(ld + bit));
    // RA in the words: nrd = ((y | RA << s) >> s) = (y >> s) | RA, RA << s or-ed in from bits N-1..N; wide
    // words: RA, which may sit anywhere, is or-ed after the right shift
    if constexpr (FORM == kRaInWords) asm("lop3.b32 %0, %1, %2, %3, 0xF8;" : "=r"(y) : "r"(rd + bit), "r"(wx), "r"(ram));   // a | (b & c)
    asm("shf.r.wrap.b32 %0, %1, 0, %2;" : "=r"(nrd) : "r"(y), "r"(wx));
    if constexpr (WIDE) nrd |= w.y;
    const uint32_t free_cols = fr - bit;             // the child row's free columns
    const uint32_t nf = free_cols & ~(nld | nrd);
    const uint32_t ahead = free_cols & ~((nld + nld) | __umulhi(nrd, 0x80000000u));   // nrd >> 1
    const uint32_t keep = ahead | (wx & (WIDE ? W_NOLOOK : C_NOLOOK));
    if (wx & (WIDE ? W_COUNT : C_COUNT)) cnt += 1u;
    ld = nld; rd = nrd; fr = free_cols;
    avail = keep != 0u ? nf : 0u;
  }
};

// Items whose schedule ends with more than one column left (no list of the generators has one): base frames
// count once, whatever candidates they have.  One lane alone, its frames in local memory.
template <WordForm FORM, class W>
__device__ __noinline__ unsigned long long count_base_frames(uint4 f, uint32_t fr, uint32_t N, uint32_t n, const W* words) {
  uint4 st[kMaxDepth];
  unsigned long long c = 0;
  int k = 0;
  st[0] = make_uint4(f.x, f.y, fr, f.w & fr);
  while (k >= 0) {
    uint4& g = st[k];
    if (g.w == 0u) { k--; continue; }
    const uint32_t bit = g.w & (0u - g.w);
    g.w ^= bit;
    const Dec o = decode(words[k], N, (uint32_t)k, n);
    const uint32_t nld = ((g.x | bit) << o.s) | o.la, nrd = ((g.y | bit) >> o.s) | o.ra, free_cols = g.z ^ bit;
    const uint32_t nf = free_cols & ~(nld | nrd);
    if (nf == 0u || (o.fc && (free_cols & ~((nld << 1) | (nrd >> 1))) == 0u)) continue;
    if (o.term) c++;
    else st[++k] = make_uint4(nld, nrd, free_cols, nf);
  }
  return c;
}

__device__ __forceinline__ void sts_frame(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint4 lds_frame(uint32_t a) {
  uint4 f;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(f.x), "=r"(f.y), "=r"(f.z), "=r"(f.w) : "r"(a) : "memory");
  return f;
}
template <WordForm FORM, int BLOCK, bool BIG, int STEPS>
__global__ void __launch_bounds__(BLOCK) dfs_kernel(const DfsArgs a) {
  constexpr bool WIDE = FORM == kWideWords;
  using W = typename WordT<WIDE>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  W* sch = reinterpret_cast<W*>(smem + (size_t)stack_slots(a.maxt) * BLOCK * sizeof(uint4)) + threadIdx.x;  // stride BLOCK
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  const W* gsched = reinterpret_cast<const W*>(a.sched);
  constexpr uint32_t ROW = BLOCK * (uint32_t)sizeof(W);
  constexpr uint32_t F = BLOCK * (uint32_t)sizeof(uint4);
  auto put_word = [&](uint32_t k, W w) { sch[k * BLOCK] = w; };
  auto count_word = [] { W w; if constexpr (WIDE) w = make_uint2(kCountWord, 0u); else w = kCountWord; return w; };
  Lane<FORM, BIG> L;
  const uint32_t sch_sh = (uint32_t)__cvta_generic_to_shared(sch);
  const uint32_t bottom = (uint32_t)__cvta_generic_to_shared(smem) + threadIdx.x * (uint32_t)sizeof(uint4);
  // stack pointer above the sentinel: a lane is idle when no frame but the sentinel is left.  The sentinel
  // is the lane's first slot until a frame above it is given away (below).
  uint32_t top = bottom + F;
  L.sp = top;
  // a base frame has one column (a terminal one two), and where popc(fr) == 1 the word is the count word,
  // for the sentinel too; a lane that never had work reads word 0
  L.sw0 = sch_sh + ROW;
  put_word(0, count_word());
  auto arm = [&]() { sts_frame(top - F, 1u, 0u, 1u, kSentinelAvail); };
  uint32_t wexp = 0, job = a.job_base, task = 0;
  bool have = false, exhausted = false, drained = false;   // exhausted, drained: warp-uniform, as the pool's counters
  chain_wait();
  if (a.stamp && blockIdx.x == 0 && threadIdx.x == 0) *a.stamp = device_ns();
  unsigned long long m = a.m;
  if (a.m_dev) { m = *a.m_dev; if (m > a.qcap) m = 0; }
  // queue items a warp takes first: 32, or its share of a queue smaller than the grid
  const unsigned warps = gridDim.x * (BLOCK / 32);
  const unsigned chunk0 = m >= 32ull * warps ? 32u : ((unsigned)m + warps - 1u) / warps;
  const float share = 1.0f / ((STEPS == kShortSteps ? kShortShare : kChunkShare) * (float)warps);
  unsigned chunk = chunk0, pool_n = 0, pool_at = 0;
  uint4 p_root = make_uint4(0, 0, 0, 0);
  uint32_t p_task = 0, p_meta = 0, p_job = 0;
  unsigned long long acc = 0;
  uint32_t acc_job = a.job_base;

  for (;;) {
    const bool idle = L.avail == 0u && L.sp == top;
    if (__ballot_sync(FULL, idle)) {          // some lane finished: flush, refill, maybe exit
      if (idle) {                             // the steps since it finished have used (and counted) some of its candidates
        L.cnt -= 31u - (uint32_t)__popc(lds_frame(top - F).w);
        arm();
      }
      if (idle && have) {
        const unsigned long long v = (unsigned long long)L.cnt << wexp;
        if (a.per_task && v) atomicAdd(a.per_task + task, v);
        if (job != acc_job) { flush_job(a, acc_job, acc); acc = 0; acc_job = job; }
        acc += v;
        have = false;
      }
      // Refill from the warp's pool of queue items: lane i holds item i of the last chunk taken, loaded and
      // decoded by the whole warp at once, so a lane that needs work costs seven shuffles and its words, not
      // an atomic and two dependent rounds of loads.  (Decoding here, a lane at a time: N=16 307 us, 296 so;
      // serving lanes only by twos or more: N=17 1.380 ms against 1.393, N=19 64.2 against 63.8.)
      bool want = idle && !exhausted;
      for (unsigned need = __ballot_sync(FULL, want); need; need = __ballot_sync(FULL, want)) {
        if (pool_n == 0u) {
          if (drained) { exhausted = true; break; }
          unsigned long long base = 0;
          if (chunk0 < 32u) {                    // the shares cover the queue: no cursor
            base = (unsigned long long)(blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5)) * chunk0;
          } else {
            if (lane == 0) base = atomicAdd(a.cursor, (unsigned long long)chunk);
            base = __shfl_sync(FULL, base, 0);
          }
          const unsigned long long left = base < m ? m - base : 0ull;
          pool_n = left < chunk ? (unsigned)left : chunk;
          pool_at = 0;
          // the next chunk is a share of what is left, so the warps end together; where the first chunks
          // cover the queue there is no next one
          drained = chunk0 < 32u || left <= chunk;
          chunk = min(32u, max(kMinChunk, (unsigned)((float)left * share)));
          if (pool_n == 0u) { exhausted = true; break; }
          if (lane < pool_n) {
            const uint64_t slot = base + lane;
            const uint64_t q = a.order ? (uint64_t)a.order[slot] : slot;
            uint32_t d0 = 0;
            if (a.sinfo) { const uint2 si = a.sinfo[q]; p_task = si.x; d0 = si.y & 31u; p_job = si.y >> 5; p_root = a.sroot[q]; }
            else if (a.sroot) { p_root = a.sroot[q]; p_task = p_root.w; d0 = a.depth; p_root.w = ~(p_root.x | p_root.y); }
            else { p_task = (uint32_t)q; p_root = a.root[q]; }
            // free columns for used ones, R of them; depth d has R - d (one queen per depth), so word d is
            // found from popc(fr) alone
            const uint32_t in = a.info[p_task], T = info_T(in), N = info_N(in), n = T - d0;   // n: terminal depth
            p_root.z = ((1u << N) - 1u) & ~p_root.z;
            p_root.w &= p_root.z;
            const uint32_t R = __popc(p_root.z);
            p_meta = (info_wexp(in) << 5) | (d0 == 0u ? info_root(in) << 7 : 0u) | (N << 8) | (d0 << 13);
            if (T != INFO_NO_DFS && info_status(in) == TS_OK && T >= d0) {
              if ((int)n > a.maxt) atomicOr(a.err, DERR_DEPTH);    // frames at depths 0..n, words 0..n
              else if (n + 2u == R) p_meta |= n | kItemWork;       // fewer free columns than rows: no solution
              else if (n + 2u < R) p_meta |= n | kItemSpare;
            }
          }
        }
        const unsigned give = min((unsigned)__popc(need), pool_n);
        const unsigned rank = __popc(need & lt_mask);
        const int src = (int)(pool_at + rank);
        uint4 r;
        r.x = __shfl_sync(FULL, p_root.x, src); r.y = __shfl_sync(FULL, p_root.y, src);
        r.z = __shfl_sync(FULL, p_root.z, src); r.w = __shfl_sync(FULL, p_root.w, src);
        const uint32_t i_task = __shfl_sync(FULL, p_task, src), meta = __shfl_sync(FULL, p_meta, src);
        const uint32_t i_job = __shfl_sync(FULL, p_job, src);
        pool_at += give; pool_n -= give;
        if (want && rank < give) {
          want = false;
          have = true;
          task = i_task; job = i_job;
          wexp = (meta >> 5) & 3u;
          L.cnt = (meta >> 7) & 1u;
          const uint32_t n = meta & 31u, N = (meta >> 8) & 31u;
          const W* w = gsched + (size_t)task * a.sw + ((meta >> 13) & 31u);
          if (meta & kItemWork) {
            L.ld = r.x; L.rd = r.y; L.fr = r.z; L.avail = r.w;
            L.sw0 = sch_sh + (n + 2u) * ROW;
            if constexpr (FORM == kRaInWords) L.ram = compact_ra_mask((int)N);
            uint32_t k = 0;
#pragma unroll 1
            for (; k + 3u <= n; k += 4) {
              const W w0 = w[k], w1 = w[k + 1], w2 = w[k + 2], w3 = w[k + 3];
              put_word(k, w0); put_word(k + 1, w1); put_word(k + 2, w2); put_word(k + 3, w3);
            }
            for (; k <= n; k++) put_word(k, w[k]);
            put_word(k, count_word());
            arm();
          } else if (meta & kItemSpare) {
            L.cnt += count_base_frames<FORM>(r, r.z, N, n, w);
          }                                    // else no work: the lane stays on its sentinel
        }
      }
      if (exhausted) {
        // The queue is empty: a lane without work takes the bottom saved frame (the largest subtree left) of
        // a busy lane of its warp, or all but one candidate of that lane's current frame.  It reads the
        // giver's schedule words in place: only loading a queue item overwrites words, and none is left.
        // Without this the last items of a warp leave 7 of 32 lanes idle at N=17: 1.475 ms, 1.334 with it; N=16
        // 0.304 / 0.261, N=19 64.4 / 63.3.
        const unsigned starved = __ballot_sync(FULL, !have);
        if (starved) {
          const bool saved = L.sp != top;
          const uint32_t rest = L.avail & (L.avail - 1u);
          const uint32_t gfr = saved ? lds_frame(top).z : L.fr;
          const bool can = have && (saved ? (L.avail != 0u || L.sp != top + F) : rest != 0u) &&
                           __popc(gfr) >= 2 + kGiveRows;
          const unsigned givers = __ballot_sync(FULL, can);
          if (givers) {
            const int n = min(__popc(starved), __popc(givers));
            const bool gives = can && __popc(givers & lt_mask) < n;
            const int srank = __popc(starved & lt_mask);
            const bool takes = !have && srank < n;
            if (gives && !saved) { sts_frame(top, L.ld, L.rd, L.fr, rest); L.avail ^= rest; }
            __syncwarp();
            const int src = takes ? (int)nth_set(givers, (uint32_t)srank) : (int)lane;
            const uint32_t from = __shfl_sync(FULL, top, src), gsw0 = __shfl_sync(FULL, L.sw0, src);
            const uint32_t gram = FORM == kRaInWords ? __shfl_sync(FULL, L.ram, src) : 0u;
            const uint32_t gw = __shfl_sync(FULL, wexp, src), gjob = __shfl_sync(FULL, job, src);
            const uint32_t gtask = __shfl_sync(FULL, task, src);
            if (takes) {
              const uint4 f = lds_frame(from);
              L.ld = f.x; L.rd = f.y; L.fr = f.z; L.avail = f.w;
              L.sw0 = gsw0; L.ram = gram; L.cnt = 0;
              wexp = gw; job = gjob; task = gtask; have = true;
              top = bottom + F; L.sp = top;
              arm();
            }
            __syncwarp();
            if (gives && saved) { top += F; arm(); }   // the sentinel takes the given frame's place
          }
        }
      }
      if (__all_sync(FULL, exhausted && !have)) break;
      asm volatile("" ::: "memory");   // refill stores to the schedule before the steps' loads
    }
#pragma unroll
    for (int s = 0; s < STEPS; ++s) L.template step<BLOCK>();
  }

  const uint32_t j0 = __shfl_sync(FULL, acc_job, 0);
  const bool same = __all_sync(FULL, acc == 0 || acc_job == j0);
  if (same) {
    unsigned long long v = acc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    if (lane == 0) flush_job(a, j0, v);
  } else {
    flush_job(a, acc_job, acc);
  }
  if (a.host_ctl) hand_over(a.ctl, a.ctl_words, a.blocks_done, a.host_ctl, a.stamp ? a.stamp + 1 : nullptr);
}

// The dynamic shared-memory cap of a kernel is one process-wide attribute.
// It is always set to the device's opt-in maximum, never to one launch's
// size: a smaller launch (a per-job run, an occupancy query) must not lower
// the cap under a larger launch captured earlier in a CUDA graph.
template <typename K>
cudaError_t allow_max_dynamic_smem(K kernel) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  return e;
}

template <WordForm FORM, int BLOCK, bool BIG, int STEPS = kStepsPerCheck>
static cudaError_t launch_dfs_t(const DfsLaunch& L, cudaStream_t st) {
  const size_t smem = dfs_smem_bytes(FORM == kWideWords, BLOCK, L.maxt);
  cudaError_t e = allow_max_dynamic_smem(dfs_kernel<FORM, BLOCK, BIG, STEPS>);
  if (e != cudaSuccess) return e;
  int grid = L.grid;
  if (grid <= 0) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, dfs_kernel<FORM, BLOCK, BIG, STEPS>, BLOCK, smem);
    if (e != cudaSuccess) return e;
    if (per <= 0) return cudaErrorInvalidConfiguration;
    grid = sms * per;
    // a short queue takes a warp an item: more blocks than that only start and end
    const int64_t most = L.m_dev ? L.m_bound : L.m;
    if (most > 0) grid = (int)std::min<int64_t>(grid, (most + BLOCK / 32 - 1) / (BLOCK / 32));
  }
  DfsArgs a;
  a.root = L.tasks.root; a.info = L.tasks.info; a.sched = L.tasks.sched; a.sw = L.tasks.sw;
  a.sroot = L.sroot; a.sinfo = L.sinfo; a.depth = L.depth;
  a.m = L.m; a.m_dev = L.m_dev; a.qcap = L.qcap; a.order = L.order; a.cursor = L.cursor; a.job_totals = L.job_totals; a.job_base = L.job_base;
  a.per_task = L.per_task; a.err = L.err; a.maxt = L.maxt;
  a.ctl = L.ctl; a.ctl_words = L.ctl_words; a.blocks_done = L.blocks_done; a.host_ctl = L.host_ctl; a.stamp = L.stamp;
  if (L.chained) return launch_after(dfs_kernel<FORM, BLOCK, BIG, STEPS>, (unsigned)grid, BLOCK, smem, st, a);
  dfs_kernel<FORM, BLOCK, BIG, STEPS><<<grid, BLOCK, smem, st>>>(a);
  return cudaGetLastError();
}


cudaError_t launch_dfs(const DfsLaunch& L, cudaStream_t st) {
  if (L.m <= 0 && !L.m_dev) return cudaSuccess;
  if (L.maxt < 1 || L.maxt > kMaxDepth) return cudaErrorInvalidValue;
#define NQ_DFS_FORM(B, FORM)                                                                \
  return L.big ? launch_dfs_t<FORM, B, true>(L, st)                                         \
       : L.maxt <= kShortDepth ? launch_dfs_t<FORM, B, false, kShortSteps>(L, st) : launch_dfs_t<FORM, B, false>(L, st)
#define NQ_DFS_BLOCK(B)                                   \
  if (L.tasks.wide) NQ_DFS_FORM(B, kWideWords);           \
  if (L.tasks.ra_words) NQ_DFS_FORM(B, kRaInWords);       \
  NQ_DFS_FORM(B, kRaInRd);
  switch (L.block) {
    case 64: { NQ_DFS_BLOCK(64) }
    case 128: { NQ_DFS_BLOCK(128) }
    case 256: { NQ_DFS_BLOCK(256) }
    default: return cudaErrorInvalidValue;
  }
#undef NQ_DFS_BLOCK
#undef NQ_DFS_FORM
}

template <bool WIDE, int BLOCK>
static int occ(int maxt) {
  constexpr WordForm FORM = WIDE ? kWideWords : kRaInWords;      // shared memory bounds it, alike for both compact forms
  const size_t smem = dfs_smem_bytes(WIDE, BLOCK, maxt);
  if (allow_max_dynamic_smem(dfs_kernel<FORM, BLOCK, false, kStepsPerCheck>) != cudaSuccess) return 0;
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, dfs_kernel<FORM, BLOCK, false, kStepsPerCheck>, BLOCK, smem) != cudaSuccess)
    return 0;
  return per;
}

int dfs_blocks_per_sm(bool wide, int block, int maxt) {
  switch (block) {
    case 64: return wide ? occ<true, 64>(maxt) : occ<false, 64>(maxt);
    case 128: return wide ? occ<true, 128>(maxt) : occ<false, 128>(maxt);
    case 256: return wide ? occ<true, 256>(maxt) : occ<false, 256>(maxt);
    default: return 0;
  }
}

// ---------------------------------------------------------------------------
// INT32 ALU throughput probe: 8 independent dependency chains per thread of
// one integer instruction kind (lop3, iadd3, shf or a 1:1:1 mix), used as the
// measured denominator of the DFS kernel's ALU roofline.
// ---------------------------------------------------------------------------
template <int KIND>
__global__ void __launch_bounds__(256) int_peak_kernel(uint32_t* out, int iters, uint32_t seed) {
  uint32_t a[8];
#pragma unroll
  for (int c = 0; c < 8; c++) a[c] = seed * (c + 1) + threadIdx.x * 7919u + blockIdx.x;
  const uint32_t b = seed ^ 0x9e3779b9u, k = (seed >> 3) | 1u;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int u = 0; u < 16; u++) {
#pragma unroll
      for (int c = 0; c < 8; c++) {
        if (KIND == 0 || (KIND == 3 && u % 3 == 0))
          asm volatile("lop3.b32 %0, %0, %1, %2, 0x96;" : "+r"(a[c]) : "r"(b), "r"(k));
        else if (KIND == 1 || (KIND == 3 && u % 3 == 1))
          asm volatile("add.u32 %0, %0, %1;" : "+r"(a[c]) : "r"(b));
        else
          asm volatile("shf.l.wrap.b32 %0, %0, %0, %1;" : "+r"(a[c]) : "r"(k));
      }
    }
  }
  uint32_t x = 0;
#pragma unroll
  for (int c = 0; c < 8; c++) x ^= a[c];
  if (x == 0x12345678u) out[0] = x;   // keeps the chains live
}

cudaError_t int_peak(int kind, int iters, int grid, uint32_t* out, cudaStream_t st) {
  switch (kind) {
    case 0: int_peak_kernel<0><<<grid, 256, 0, st>>>(out, iters, 12345u); break;
    case 1: int_peak_kernel<1><<<grid, 256, 0, st>>>(out, iters, 12345u); break;
    case 2: int_peak_kernel<2><<<grid, 256, 0, st>>>(out, iters, 12345u); break;
    default: int_peak_kernel<3><<<grid, 256, 0, st>>>(out, iters, 12345u); break;
  }
  return cudaGetLastError();
}

}  // namespace nq
