// nq_gen.cu -- task lists built on the device.
//
// gen_kernels: the records of a range of start constellations (the preset-
//   queen expansion of gen_constellations, 14Bit_codon_GPU/
//   356Py_savesp_narrow.py:2759-2835), one launch a queen.
// query_kernel: the queue of one completion query, from its root frame to
//   thousands of frames, in one block; query_level_kernel expands it by
//   another level over the whole GPU.
//
// All of them count a state's children, take the warp's slots with one atomic
// and write them; list order is not kept (a count does not depend on it).
// Bound by launch latency at small boards: a level takes 2-3 us.
#include <cuda_runtime.h>

#include "nq_common.cuh"
#include "nq_internal.h"

namespace nq {
namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;

// First slot of this thread's `n` entries in a list with counter `c` (all lanes of the warp call it).
__device__ __forceinline__ unsigned take_slots(unsigned* c, unsigned n) {
  const unsigned lane = threadIdx.x & 31u;
  unsigned incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(FULL, incl, o);
    if ((int)lane >= o) incl += v;
  }
  unsigned base = 0;
  if (lane == 31 && incl) base = atomicAdd(c, incl);
  return __shfl_sync(FULL, base, 31) + incl - n;
}

// ---------------------------------------------------------------------------
// constellation records.  A state is the record {ld, rd, col, row<<20 | ijkl}
// with its queens in bits 27-30 of the last word; masks keep their low 32 bits,
// which is all a record holds and all the next row's free set reads (columns
// are bits 0..N-1, N <= 27, and rd starts below bit N).  The reference drops
// states it has seen (subconst cache, and the signatures up to preset 5): over
// all N <= 27 and presets 4-6 no state occurs twice (enumerated), and from
// preset 7 on the reference does not look, so nothing is looked up here.
// ---------------------------------------------------------------------------
constexpr unsigned kQueens = 27;

__device__ __forceinline__ uint4 settle(uint32_t ld, uint32_t rd, uint32_t col, int row, int queens, uint32_t ijkl) {
  while (row == getk((int)ijkl) || row == getl((int)ijkl)) { ld <<= 1; rd >>= 1; row++; }   // rows of the side queens
  return make_uint4(ld, rd, col, ((uint32_t)row << 20) | ijkl | ((uint32_t)queens << kQueens));
}

__device__ __forceinline__ uint4 start_state(int N, int sc) {
  const int i = geti(sc), j = getj(sc), k = getk(sc), l = getl(sc);
  const uint32_t L = 1u << (N - 1), Lj = L >> j, Li = L >> i;
  const uint32_t ld = ((i > 0) ? (L >> (i - 1)) : 0u) | (1u << (N - k));
  const uint32_t rd = (L >> (i + 1)) | (1u << (l - 1));
  return settle(ld, rd, 1u | L | Li | Lj, 1, (j == N - 1) ? 3 : 4, (uint32_t)sc);
}

__global__ void __launch_bounds__(128) gen_start_kernel(int N, unsigned n, const int* __restrict__ starts,
                                                        uint4* __restrict__ out, unsigned* gn) {
  const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
  chain_next();
  chain_wait();
  if (q == 0) gn[0] = n;
  if (q >= n) return;
  out[q] = start_state(N, starts[q]);
}

// All start constellations of a board (356Py:2850-2880).  The reference inserts candidates in loop order and
// skips one whose rotation it has inserted: of the candidates that are rotations of each other it inserts the
// first, so each thread takes one candidate and compares it with its three rotations.  The canonical forms
// (jasmin) of what is left are all different.  Both checked against the sequential list for every N of 5..27.
struct Quad { int i, j, k, l; };
__device__ __forceinline__ bool start_candidate(const Quad x, int N) {
  return x.k >= 1 && x.k < (N + 1) / 2 && x.l > x.k && x.l <= N - 2 && x.i > x.k && x.i <= N - 2 && x.i != N - 1 - x.l &&
         x.j >= 1 && x.j <= N - x.k - 2 && x.j != x.i && x.j != x.l;
}
__device__ __forceinline__ int start_rank(const Quad x, int N) {     // place in the loops: the centre column of odd boards first
  const int k = ((N & 1) && x.k == N / 2) ? 0 : x.k;
  return (((k << 5) + x.l) << 10) + (x.i << 5) + (N - x.k - 2 - x.j);
}
__device__ __forceinline__ int rotate90(int x, int N) {
  return ((N - 1 - getk(x)) << 15) + ((N - 1 - getl(x)) << 10) + (getj(x) << 5) + geti(x);
}
__device__ __forceinline__ int jasmin(int x, int N) {                // 356Py:2739-2756
  auto dist = [N](int v) { return min(v, N - 1 - v); };
  int turns = 0, mn = dist(getj(x));
  if (dist(geti(x)) < mn) { turns = 2; mn = dist(geti(x)); }
  if (dist(getk(x)) < mn) { turns = 3; mn = dist(getk(x)); }
  if (dist(getl(x)) < mn) turns = 1;
  for (int a = 0; a < turns; a++) x = rotate90(x, N);
  if (getj(x) < N - 1 - getj(x)) x = ((N - 1 - geti(x)) << 15) + ((N - 1 - getj(x)) << 10) + (getl(x) << 5) + getk(x);
  return x;
}

// Thread q's candidate of a board; true if the reference's loops insert it.
__device__ __forceinline__ bool board_candidate(int q, int N, Quad& x) {
  const int corners = N * N;
  if (q < corners) {                               // a queen in the corner: (0, j, 0, l), j < l
    x = Quad{0, q / N, 0, q % N};
    return x.j >= 1 && x.j < N - 2 && x.l > x.j && x.l <= N - 2;
  }
  q -= corners;
  x.j = q % N; q /= N;
  x.i = q % N; q /= N;
  x.l = q % N; x.k = q / N + 1;
  bool take = start_candidate(x, N);
  if (take) {
    const int rank = start_rank(x, N);
    const Quad r[3] = {{N - 1 - x.k, N - 1 - x.l, x.j, x.i}, {N - 1 - x.j, N - 1 - x.i, N - 1 - x.l, N - 1 - x.k},
                       {x.l, x.k, N - 1 - x.i, N - 1 - x.j}};
#pragma unroll
    for (int t = 0; t < 3; t++) take = take && !(start_candidate(r[t], N) && start_rank(r[t], N) < rank);
  }
  return take;
}

__global__ void __launch_bounds__(128) gen_board_kernel(int N, uint4* __restrict__ out, unsigned cap, unsigned* gn) {
  chain_next();
  chain_wait();
  Quad x;
  const bool take = board_candidate((int)(blockIdx.x * blockDim.x + threadIdx.x), N, x);
  const unsigned at = take_slots(&gn[0], take ? 1u : 0u);
  if (take && at < cap) out[at] = start_state(N, jasmin((x.i << 15) + (x.j << 10) + (x.k << 5) + x.l, N));
}

// The free columns of a state's row, with the side queens' diagonals.
__device__ __forceinline__ uint32_t free_row(const uint4 s, int N, unsigned* err) {
  const int ijkl = (int)(s.w & 0xFFFFFu), sh = N - 1 - ((int)(s.w >> 20) & 31);
  if (sh < 0) { atomicOr(err, DERR_SHIFT); return 0u; }  // the reference raises on a negative shift here
  const uint32_t L = 1u << (N - 1), Lj = L >> getj(ijkl);
  const uint32_t LD = Lj | (L >> getl(ijkl)), RD = Lj | (1u << getk(ijkl));
  return ~(s.x | s.y | s.z | (LD >> sh) | (RD << sh)) & ((1u << N) - 1u);
}
__device__ __forceinline__ uint4 state_child(const uint4 s, uint32_t bit) {
  return settle((s.x | bit) << 1, (s.y | bit) >> 1, s.z | bit, (int)((s.w >> 20) & 31u) + 1, (int)(s.w >> kQueens) + 1, s.w & 0xFFFFFu);
}

// Presets 4 and 5 in one launch: a start constellation is at most kGenFused queens short, and its thread writes its
// records (of a whole board, the corner constellations, which hold a queen less, have a thread a column).  us of a
// count of N=6 / 10 / 13 / 16 with a launch a queen 30.8 / 35.2 / 47.6 / 319, so
// 26.5 / 31.7 / 44.2 / 315.  A third level (preset 6)
// keeps a launch a queen: N=14 70 us and N=16 328 with three in a thread.
template <int DEPTH, class F>
__device__ __forceinline__ void each_record(const uint4 s, int N, int preset, unsigned* err, F&& f) {
  if constexpr (DEPTH > 0) {
    if ((int)(s.w >> kQueens) < preset) {
      for (uint32_t fr = free_row(s, N, err); fr; fr &= fr - 1u) each_record<DEPTH - 1>(state_child(s, fr & (0u - fr)), N, preset, err, f);
      return;
    }
  }
  f(make_uint4(s.x, s.y, s.z, s.w & ((1u << kQueens) - 1u)));
}
__global__ void __launch_bounds__(128) gen_records_kernel(int N, int preset, unsigned n, const int* __restrict__ starts,
                                                          uint4* __restrict__ out, unsigned cap, unsigned* count, unsigned* err) {
  chain_next();
  chain_wait();
  const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
  bool take = q < n;
  int sc = 0, column = -1;               // column: of a corner constellation's fourth queen
  if (starts) {
    if (take) sc = starts[q];
  } else {
    const unsigned corners = (unsigned)(N * N * N);
    column = q < corners ? (int)(q % (unsigned)N) : -1;
    Quad x;
    take = board_candidate(column >= 0 ? (int)(q / (unsigned)N) : (int)(q - corners) + N * N, N, x) && q < n;
    if (take) sc = jasmin((x.i << 15) + (x.j << 10) + (x.k << 5) + x.l, N);
  }
  uint4 s = make_uint4(0, 0, 0, 0);
  unsigned c = 0;
  if (take) {
    s = start_state(N, sc);
    if (column >= 0) {
      const uint32_t bit = 1u << column;
      take = (free_row(s, N, err) & bit) != 0u;
      if (take) s = state_child(s, bit);
    }
  }
  if (take) each_record<kGenFused>(s, N, preset, err, [&](uint4) { c++; });
  unsigned at = take_slots(count, c);
  if (take)
    each_record<kGenFused>(s, N, preset, err, [&](uint4 r) {
      if (at < cap) out[at] = r;
      at++;
    });
}

// One queen more for every state below the preset; the others move on (last: as records).
__global__ void __launch_bounds__(128) gen_level_kernel(int N, int preset, bool last, const uint4* in,
                                                        uint4* __restrict__ out, unsigned cap, unsigned* gn, int level,
                                                        unsigned* err) {
  chain_next();
  chain_wait();
  const unsigned n = min(gn[level], cap);
  for (unsigned q0 = blockIdx.x * blockDim.x; q0 < n; q0 += gridDim.x * blockDim.x) {
    const unsigned q = q0 + threadIdx.x;
    uint4 s = make_uint4(0, 0, 0, 0);
    uint32_t fr = 0;
    bool keep = false;
    if (q < n) {
      s = in[q];
      keep = (int)(s.w >> kQueens) >= preset;
      if (!keep) fr = free_row(s, N, err);
    }
    unsigned at = take_slots(&gn[level + 1], keep ? 1u : (unsigned)__popc(fr));
    const uint32_t mask = last ? (1u << kQueens) - 1u : ~0u;
    if (keep) {
      if (at < cap) out[at] = make_uint4(s.x, s.y, s.z, s.w & mask);
    } else {
      while (fr) {
        const uint32_t bit = fr & (0u - fr);
        fr ^= bit;
        uint4 c = state_child(s, bit);
        c.w &= mask;
        if (at < cap) out[at] = c;
        at++;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// completion queries
// ---------------------------------------------------------------------------
struct QWord { uint32_t s, la, ra, fc; };
__device__ __forceinline__ QWord qword(uint32_t w, uint32_t N) {
  const Op o = unpack_compact(w ^ C_NOLOOK, (int)N, false);
  return QWord{o.s, o.la, o.ra, o.fc};
}
__device__ __forceinline__ QWord qword(uint2 w, uint32_t) {
  const uint32_t s = w.x & W_S;
  return QWord{s, s ? (w.x >> (32 - s)) : 0u, w.y, ~w.x & W_NOLOOK};
}

template <class F>
__device__ __forceinline__ void each_child(const uint4 f, const QWord o, uint32_t bm, F&& fn) {
  for (uint32_t av = f.w; av;) {
    const uint32_t bit = av & (0u - av);
    av ^= bit;
    const uint32_t nl = ((f.x | bit) << o.s) | o.la, nr = ((f.y | bit) >> o.s) | o.ra, nc = f.z | bit;
    const uint32_t nf = bm & ~(nl | nr | nc);
    if (nf && !(o.fc && (bm & ~((nl << 1) | (nr >> 1) | nc)) == 0u)) fn(make_uint4(nl, nr, nc, nf));
  }
}

// The frames of one query, breadth-first from its root until there are `target` of them or they stand at the terminal
// depth.  Returns their number; one block, buffers of `cap` frames, which no level exceeds.
template <class W>
__device__ unsigned expand_query(const uint4 root, uint32_t N, uint32_t T, const W* words, unsigned target, unsigned cap,
                                 uint4* buf0, uint4* buf1, unsigned& depth) {
  __shared__ unsigned cnt;
  const uint32_t bm = (1u << N) - 1u;
  uint4 *in = buf0, *out = buf1;
  if (threadIdx.x == 0) in[0] = root;
  unsigned n = root.w ? 1u : 0u, d = 0;
  __syncthreads();
  while (d < T && n && n < target) {
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    const QWord o = qword(words[d], N);
    for (unsigned q0 = 0; q0 < n; q0 += blockDim.x) {
      const unsigned q = q0 + threadIdx.x;
      const uint4 f = q < n ? in[q] : make_uint4(0, 0, 0, 0);
      unsigned c = 0;
      each_child(f, o, bm, [&](uint4) { c++; });
      unsigned at = take_slots(&cnt, c);
      if (c) each_child(f, o, bm, [&](uint4 g) { out[at++] = g; });
    }
    __syncthreads();
    n = min(cnt, cap);
    uint4* t = in; in = out; out = t;
    d++;
    __syncthreads();
  }
  depth = d;
  if (in != buf0)                       // callers read buf0
    for (unsigned q = threadIdx.x; q < n; q += blockDim.x) buf0[q] = in[q];
  __syncthreads();
  return n;
}

template <bool WIDE>
__global__ void __launch_bounds__(1024) query_kernel(const __grid_constant__ QueryParam p, QueryBuffers b) {
  using W = typename QueryWord<WIDE>::type;
  __shared__ W words[kMaxDepth];
  chain_next();
  if (threadIdx.x <= p.T) {
    const uint2 w = p.words[threadIdx.x];
    if constexpr (WIDE) words[threadIdx.x] = w; else words[threadIdx.x] = w.x;
    ((W*)b.sched)[threadIdx.x] = words[threadIdx.x];
  }
  if (threadIdx.x < QueryCtl::kWords) b.ctl[threadIdx.x] = 0;
  if (threadIdx.x == 0) b.info[0] = info_pack(p.T, 0, 0, p.N, TS_OK);
  __syncthreads();
  unsigned d;
  const unsigned n = expand_query<W>(p.root, p.N, p.T, words, p.target, b.cap[0], b.sroot[0], b.tmp, d);
  for (unsigned q = threadIdx.x; q < n; q += blockDim.x) b.sinfo[0][q] = make_uint2(0u, d);
  if (threadIdx.x == 0) b.ctl[QueryCtl::kQueue] = n;
}

// A batch's queries: task and frames of each.
template <bool WIDE>
__global__ void __launch_bounds__(512) batch_query_kernel(const BatchQuery* __restrict__ qs, uint4* src, uint4* tmp,
                                                          ListState* state, uint32_t* info, void* sched, int sw) {
  using W = typename QueryWord<WIDE>::type;
  __shared__ W words[kMaxDepth];
  chain_next();
  chain_wait();
  const BatchQuery& q = qs[blockIdx.x];
  if (threadIdx.x <= q.p.T) {
    const uint2 w = q.p.words[threadIdx.x];
    if constexpr (WIDE) words[threadIdx.x] = w; else words[threadIdx.x] = w.x;
    ((W*)sched)[(size_t)q.task * sw + threadIdx.x] = words[threadIdx.x];
  }
  __syncthreads();
  unsigned d;
  const unsigned n = expand_query<W>(q.p.root, q.p.N, q.p.T, words, q.p.target, q.cap, src + q.src0, tmp + q.tmp0, d);
  if (threadIdx.x == 0) {
    info[q.task] = info_pack(q.p.T, 0, 0, q.p.N, TS_OK);
    state[q.list].n = n;
    state[q.list].depth = d;
  }
}

// The query's queue by another level (frames at the terminal depth move on).  A level that did not fit its buffer is
// not read: the levels behind it stay empty, so the search does nothing, and the host finds its length.
template <bool WIDE>
__global__ void __launch_bounds__(128) query_level_kernel(uint32_t N, uint32_t T, QueryBuffers b, int level) {
  using W = typename QueryWord<WIDE>::type;
  chain_next();
  chain_wait();
  unsigned n = b.ctl[QueryCtl::kQueue + level];
  if (n > b.cap[level]) n = 0;
  const unsigned cap = b.cap[level + 1];
  const uint4* in = b.sroot[level];
  uint4* __restrict__ out = b.sroot[level + 1];
  uint2* __restrict__ info = b.sinfo[level + 1];
  const uint32_t bm = (1u << N) - 1u;
  for (unsigned q0 = blockIdx.x * blockDim.x; q0 < n; q0 += gridDim.x * blockDim.x) {
    const unsigned q = q0 + threadIdx.x;
    uint4 f = make_uint4(0, 0, 0, 0);
    uint32_t d = 0;
    if (q < n) { f = in[q]; d = b.sinfo[level][q].y; }
    const bool keep = q < n && d >= T;
    const QWord o = keep ? QWord{1, 0, 0, 0} : qword(((const W*)b.sched)[d], N);
    unsigned c = keep ? 1u : 0u;
    if (!keep) each_child(f, o, bm, [&](uint4) { c++; });
    unsigned at = take_slots((unsigned*)&b.ctl[QueryCtl::kQueue + level + 1], c);
    if (at + c > cap) continue;
    if (keep) { out[at] = f; info[at] = make_uint2(0u, d); }
    else if (c) each_child(f, o, bm, [&](uint4 g) { out[at] = g; info[at++] = make_uint2(0u, d + 1u); });
  }
}

}  // namespace

cudaError_t launch_generate(int N, int preset, unsigned n_starts, const int* starts, uint4* buf0, uint4* buf1, unsigned cap,
                            unsigned* gn, unsigned* err, int sms, cudaStream_t st) {
  const int levels = gen_levels(preset);
  uint4* buf[2] = {buf0, buf1};
  const unsigned full = 8u * (unsigned)sms;
  if (starts && n_starts == 0) return cudaSuccess;
  const unsigned board = (unsigned)(N * N * (1 + ((N + 1) / 2 - 1) * N));      // a board's candidates
  if (levels <= kGenFused) {
    const unsigned n = starts ? n_starts : board + (unsigned)(N * N * (N - 1));      // corner ones: a thread a column
    return launch_after(gen_records_kernel, (n + 127) / 128, 128, 0, st, N, preset, n, starts, buf[levels & 1], cap, gn + levels, err);
  }
  if (starts) {
    const cudaError_t e = launch_after(gen_start_kernel, (n_starts + 127) / 128, 128, 0, st, N, n_starts, starts, buf[0], gn);
    if (e != cudaSuccess) return e;
  } else {
    const cudaError_t e = launch_after(gen_board_kernel, (board + 127) / 128, 128, 0, st, N, buf[0], cap, gn);
    if (e != cudaSuccess) return e;
  }
  for (int l = 0; l < levels; l++) {
    const unsigned need = l == 0 ? (n_starts + 127) / 128 : full;
    const cudaError_t e = launch_after(gen_level_kernel, need < full ? need : full, 128, 0, st, N, preset, l + 1 == levels, buf[l & 1],
                                       buf[(l + 1) & 1], cap, gn, l, err);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

cudaError_t launch_query(const QueryParam& p, const QueryBuffers& b, bool wide, int levels, int sms, cudaStream_t st) {
  if (wide) query_kernel<true><<<1, 1024, 0, st>>>(p, b);
  else query_kernel<false><<<1, 1024, 0, st>>>(p, b);
  for (int l = 0; l < levels; l++) {
    const cudaError_t e = wide ? launch_after(query_level_kernel<true>, 4 * sms, 128, 0, st, p.N, p.T, b, l)
                               : launch_after(query_level_kernel<false>, 4 * sms, 128, 0, st, p.N, p.T, b, l);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

cudaError_t launch_batch_queries(int n, const BatchQuery* q, uint4* src, uint4* tmp, ListState* state, const TaskArrays& ta,
                                 cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (ta.wide) return launch_after(batch_query_kernel<true>, n, 512, 0, st, q, src, tmp, state, ta.info, ta.sched, ta.sw);
  return launch_after(batch_query_kernel<false>, n, 512, 0, st, q, src, tmp, state, ta.info, ta.sched, ta.sw);
}

}  // namespace nq
