// nq_unique.cu -- unique and total counts by the symmetry method on sm_103a.
//
// Restates the classic symmetry-elimination search of the reference
// (11Bit_Python/07Py_bit_symmetry.py:65-200; GPU form 10Bit_CUDA/
// 01CUDA_Bit_Symmetry.cu:627-960):
//   * corner solutions: queen at row 0 column 0, row 1 at column bound1
//     (2 <= bound1 <= N-2); rows below bound1 may not use column 1; every
//     solution counts x8 (backTrack1, :152-170);
//   * the rest: row 0 at column bound1 with bound2 = N-1-bound1 and
//     bound1 < bound2; rows above bound1 avoid the side columns, row bound2 is
//     gated on the side columns used so far, the last row must avoid lastmask
//     (backTrack2, :126-151); each solution is classified by its rotations as
//     x2, x4 or x8 or dropped as a non-canonical copy (symmetryops, :65-125).
// Unique = c2 + c4 + c8, total = 2 c2 + 4 c4 + 8 c8.
//
// The first rows of every (part, bound1) start are expanded on the device, a
// row per launch, into the task queue (unique_init_kernel,
// unique_expand_kernel).  unique_kernel is persistent, queue-fed and
// explicit-stack like the constellation DFS (one candidate per lane per step,
// predicated pop/push, the row carried in `down`'s high bits, work shared in a
// warp at the end of the queue), keeping each lane's board (one bit per row)
// in shared memory for the leaf classification.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/nqueens_gb300.h"
#include "nq_common.cuh"
#include "nq_handle.h"
#include "nq_internal.h"

namespace nq {
namespace {

constexpr unsigned FULLM = 0xFFFFFFFFu;
constexpr int kBoardRows = 8;    // rows of the board prefix carried by a task
constexpr int kUniqueSteps = 16;   // steps per lane between checks for finished lanes
constexpr int kReadBackN = 14;     // boards from here on size the stacks to the tasks' rows
constexpr uint32_t kGiveRows = 5;   // rows below a frame worth giving away

// One start configuration (symmetry part and its bounds).
struct UConf {
  uint32_t part;       // 1 corner, 2 no corner
  uint32_t bound1, bound2, endbit, lastmask, sidemask, topbit;
};

// A task: the search state at `row` plus the board rows above it (one byte each, the queen's column), 32 bytes.
struct __align__(16) UTask {
  uint32_t left, down, right, avail;
  uint32_t row, conf;
  uint32_t board[kBoardRows / 4];
};
__device__ __forceinline__ uint32_t board_bit(const UTask& t, uint32_t r) {   // row r's queen as a bit
  return 1u << ((t.board[r >> 2] >> (8u * (r & 3u))) & 31u);
}
__device__ __forceinline__ void board_set(UTask& t, uint32_t r, uint32_t bit) {
  const uint32_t v = (31u - (uint32_t)__clz((int)bit)) << (8u * (r & 3u));
  if (r < 4u) t.board[0] |= v; else t.board[1] |= v;
}

// symmetryops (07Py_bit_symmetry.py:65-125): 2, 4 or 8 for a canonical
// solution, 0 for a rotated copy.  `b(k)` reads board row k.
template <typename B>
__device__ __forceinline__ uint32_t classify(const B& b, int size, const UConf& c) {
  int own, you;
  uint32_t bit, ptn;
  if (b(c.bound2) == 1u) {                        // 90 degrees
    own = 1; ptn = 2;
    while (own <= size - 1) {
      bit = 1; you = size - 1;
      while (b(you) != ptn && b(own) >= bit) { bit <<= 1; you--; }
      if (b(own) > bit) return 0;
      if (b(own) < bit) break;
      own++; ptn <<= 1;
    }
    if (own > size - 1) return 2;
  }
  if (b(size - 1) == c.endbit) {                  // 180 degrees
    own = 1; you = size - 2;
    while (own <= size - 1) {
      bit = 1; ptn = c.topbit;
      while (b(you) != ptn && b(own) >= bit) { bit <<= 1; ptn >>= 1; }
      if (b(own) > bit) return 0;
      if (b(own) < bit) break;
      own++; you--;
    }
    if (own > size - 1) return 4;
  }
  if (b(c.bound1) == c.topbit) {                  // 270 degrees
    own = 1; ptn = c.topbit >> 1;
    while (own <= size - 1) {
      bit = 1; you = 0;
      while (b(you) != ptn && b(own) >= bit) { bit <<= 1; you++; }
      if (b(own) > bit) return 0;
      if (b(own) < bit) break;
      own++; ptn >>= 1;
    }
  }
  return 8;
}

// Row rules of backTrack1/backTrack2 applied to the candidate set of `row`.
__host__ __device__ __forceinline__ uint32_t row_filter(uint32_t bitmap, uint32_t row, uint32_t down, const UConf& c) {
  if (c.part == 1) return row < c.bound1 ? (bitmap & ~2u) : bitmap;
  if (row < c.bound1) return bitmap & ~c.sidemask;
  if (row == c.bound2) {
    const uint32_t ds = down & c.sidemask;
    if (ds == 0u) return 0u;
    if (ds != c.sidemask) return bitmap & c.sidemask;
  }
  return bitmap;
}

// Control block: counts, queue cursor, states after each expanded row.
constexpr int kLevels = kBoardRows - 2;   // expanded rows at most: from row 1, and a task carries the rows above its own
struct UCtl {
  unsigned long long c2, c4, c8;
  unsigned int cursor, pad;
  unsigned int n[kLevels + 1];
};
// The queue is the last level with states in it that its buffer holds (levels alternate between two
// buffers; a level that was large enough, or whose states all died, leaves the next one empty).
__host__ __device__ __forceinline__ int queue_level(const UCtl* c, unsigned cap) {
  int f = 0;
  for (int l = 1; l <= kLevels; l++)
    if (c->n[l] && c->n[l] <= cap) f = l;
  return f;
}

struct UArgs {
  const UTask* tasks[2];
  const UConf* confs;
  int N;
  int maxf;                     // stack frames per lane: N - 2 - (smallest task row)
  unsigned cap;                 // tasks a buffer holds
  UCtl* ctl;
};

// Predicated shared-memory stores (32-bit shared-window addresses), so the push is
// a single predicated instruction, not a branch.
__device__ __forceinline__ void sts_frame_if(uint32_t p, uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.v4.u32 [%1], {%2, %3, %4, %5};\n\t}"
               :: "r"(p), "r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts_word_if(uint32_t p, uint32_t a, uint32_t x) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u32 [%1], %2;\n\t}"
               :: "r"(p), "r"(a), "r"(x) : "memory");
}

__device__ __forceinline__ uint32_t lds_word_u(uint32_t a) {
  uint32_t w;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(a) : "memory");
  return w;
}
__device__ __forceinline__ void lds_frame_u(uint32_t a, uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& w) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a) : "memory");
}

// One lane per task, one candidate per step, all lanes on the same predicated
// sequence: resume a saved frame, take the lowest candidate, record it in the
// board, build the next row with the part's row rules, then count (last row)
// or descend.  The row of a frame rides in `down` bits 27-31 (columns use bits
// 0..N-1, N <= 27), so a saved frame is exactly {left, down, right, avail}.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) unique_kernel(const UArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int N = a.N;
  constexpr uint32_t F = BLOCK * (uint32_t)sizeof(uint4);          // frame stride of one lane's stack
  constexpr uint32_t RB = BLOCK * (uint32_t)sizeof(uint32_t);      // board row stride
  // a lane pushes at most one frame per row from its task's row to N - 3
  uint4* stk = reinterpret_cast<uint4*>(smem) + threadIdx.x;                            // maxf frames, stride BLOCK
  uint32_t* brd = reinterpret_cast<uint32_t*>(smem + (size_t)a.maxf * BLOCK * sizeof(uint4)) + threadIdx.x;  // N rows
  const uint32_t bottom = (uint32_t)__cvta_generic_to_shared(stk);
  uint32_t sbase = bottom;            // moves up when the lane gives its bottom frame away
  const uint32_t bbase = (uint32_t)__cvta_generic_to_shared(brd);
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t mask = (1u << N) - 1u;
  const uint32_t last_row = (uint32_t)N - 1u;
  uint32_t left = 0, down = 0, right = 0, avail = 0, sp = sbase;
  UConf cf = {0, 0, 0, 0, 0, 0, 0};
  uint32_t lowmask = ~0u, b2 = ~0u;      // row rules of the task's part
  // part 1: rows above bound1 avoid column 1; part 2: they avoid the side
  // columns, and row bound2 is gated on the side columns used so far
  auto load_conf = [&](const UConf& c) {
    cf = c;
    lowmask = (cf.part == 1) ? ~2u : ~cf.sidemask;
    b2 = (cf.part == 1) ? ~0u : cf.bound2;
  };
  unsigned long long c2 = 0, c4 = 0, c8 = 0;
  bool exhausted = false;
  const int level = queue_level(a.ctl, a.cap);
  const UTask* __restrict__ tasks = a.tasks[level & 1];
  const unsigned m = a.ctl->n[level];
  // where the queue is smaller than the lanes, each warp takes its share and shares it among its lanes
  const unsigned warps = gridDim.x * (BLOCK / 32);
  const unsigned take = min(32u, (m + warps - 1u) / warps);
  uint32_t conf_ix = 0;
  for (;;) {
    const bool idle = (avail | (sp - sbase)) == 0u;
    if (__ballot_sync(FULLM, idle)) {
      if (idle) sbase = sp = bottom;
      const bool want = idle && !exhausted;
      const unsigned need = __ballot_sync(FULLM, want);
      if (need) {
        const unsigned n_take = min((unsigned)__popc(need), take);
        unsigned base = 0;
        if (lane == 0 && n_take) base = atomicAdd(&a.ctl->cursor, n_take);
        base = __shfl_sync(FULLM, base, 0);
        const unsigned rank = __popc(need & ((1u << lane) - 1u));
        if (want && rank < n_take && base + rank < m) {
          const UTask t = tasks[base + rank];
          conf_ix = t.conf;
          load_conf(a.confs[conf_ix]);
          left = t.left; down = (t.down & mask) | (t.row << 27); right = t.right; avail = t.avail;
          for (uint32_t r = 0; r < t.row && r < (uint32_t)kBoardRows; r++) brd[r * BLOCK] = board_bit(t, r);
        }
        exhausted = take < 32u || base + n_take >= m;   // warp-uniform
      }
      if (exhausted) {
        // The queue is empty: a lane without work takes the bottom saved frame of a busy lane of its warp,
        // or all but one candidate of its current frame, with the rows of the board above it.
        const bool busy = avail != 0u || sp != sbase;
        const unsigned starved = __ballot_sync(FULLM, !busy);
        const bool saved = sp != sbase;
        const uint32_t rest = avail & (avail - 1u);
        const uint32_t gdown = saved ? lds_word_u(sbase + 4u) : down;
        const bool can = busy && (saved ? (avail != 0u || sp != sbase + F) : rest != 0u) &&
                         (gdown >> 27) + kGiveRows <= last_row;
        const unsigned givers = starved ? __ballot_sync(FULLM, can) : 0u;
        if (givers) {
          const unsigned lt = (1u << lane) - 1u;
          const int n = min(__popc(starved), __popc(givers));
          const bool gives = can && __popc(givers & lt) < n;
          const int srank = __popc(starved & lt);
          const bool takes = !busy && srank < n;
          if (gives && !saved) { sts_frame_if(1u, sbase, left, down, right, rest); avail ^= rest; }
          __syncwarp();
          const int src = takes ? (int)nth_set(givers, (uint32_t)srank) : (int)lane;
          const uint32_t from = __shfl_sync(FULLM, sbase, src), fconf = __shfl_sync(FULLM, conf_ix, src);
          const uint32_t fbrd = __shfl_sync(FULLM, bbase, src);
          if (takes) {
            lds_frame_u(from, left, down, right, avail);
            conf_ix = fconf;
            load_conf(a.confs[conf_ix]);
            const uint32_t rows = down >> 27;
            for (uint32_t r = 0; r < rows; r++) brd[r * BLOCK] = lds_word_u(fbrd + r * RB);
          }
          __syncwarp();
          if (gives && saved) sbase += F;
        }
      }
      if (__all_sync(FULLM, exhausted && (avail | (sp - sbase)) == 0u)) break;
      asm volatile("" ::: "memory");   // board stores of the refill before the steps' accesses
    }
    // kUniqueSteps steps between two checks for finished lanes (two ballots each)
#pragma unroll 1
    for (int s = 0; s < kUniqueSteps; ++s) {
      // pop with its condition formed in a predicate register inside the block (no 0/1 value for it)
      asm volatile("{\n\t.reg .pred q;\n\tsetp.eq.u32 q, %3, 0;\n\tsetp.ne.and.u32 q, %4, %5, q;\n\t"
                   "@q sub.u32 %4, %4, %6;\n\t@q ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                   : "+r"(left), "+r"(down), "+r"(right), "+r"(avail), "+r"(sp) : "r"(sbase), "n"(F));
      const uint32_t row = __umulhi(down, 32u);                 // down >> 27
      const bool act = avail != 0u;
      const uint32_t bit = avail & (0u - avail);
      avail -= bit;
      sts_word_if(act ? 1u : 0u, bbase + row * RB, bit);        // board row `row` = the queen taken
      const uint32_t nl = (left + bit) * 2u;
      const uint32_t nd = down + bit;
      const uint32_t nr = __umulhi(right + bit, 0x80000000u);   // (right | bit) >> 1
      const uint32_t nrow = row + 1u;
      const uint32_t nb = mask & ~(nl | nd | nr);
      const bool last = nrow == last_row;
      // row rules of backTrack1/backTrack2 (row_filter) as selects
      uint32_t nbf = nb & ((nrow < cf.bound1) ? lowmask : ~0u);
      const uint32_t ds = nd & cf.sidemask;
      const uint32_t at_b2 = (ds == 0u) ? 0u : ((ds != cf.sidemask) ? (nbf & cf.sidemask) : nbf);
      nbf = (nrow == b2) ? at_b2 : nbf;
      // last row: a solution (part 1: x8) or a board to classify (part 2)
      if (act && last && nb != 0u) {
        if (cf.part == 1) {
          c8++;
        } else if ((nb & cf.lastmask) == 0u) {
          brd[nrow * BLOCK] = nb;
          const uint32_t k = classify([&](int r) { return brd[r * BLOCK]; }, N, cf);
          c2 += (k == 2); c4 += (k == 4); c8 += (k == 8);
        }
      }
      const bool desc = act && !last && nbf != 0u;
      const uint32_t push = (desc && avail != 0u) ? 1u : 0u;
      sts_frame_if(push, sp, left, down, right, avail);
      sp += push ? F : 0u;
      if (desc) { left = nl; down = nd + (1u << 27); right = nr; avail = nbf; }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c2 += __shfl_xor_sync(FULLM, c2, o);
    c4 += __shfl_xor_sync(FULLM, c4, o);
    c8 += __shfl_xor_sync(FULLM, c8, o);
  }
  if (lane == 0) {
    if (c2) atomicAdd(&a.ctl->c2, c2);
    if (c4) atomicAdd(&a.ctl->c4, c4);
    if (c8) atomicAdd(&a.ctl->c8, c8);
  }
}

// ---------------------------------------------------------------------------
// Task queue: every (part, bound1) start of 07Py_bit_symmetry.py NQueens()
// (:171-200), expanded a whole row at a time (tasks of one row are of similar
// size) until there are enough tasks, they reach the last row, or their rows
// no longer fit the board prefix.  Bound by launch latency: about 2 us a row
// at N=12; the same expansion on one host thread and its upload took 0.8 ms at
// N=12, 6 ms at N=14 and 25 ms at N=16.
// ---------------------------------------------------------------------------
__device__ __forceinline__ UConf make_conf(int N, int i) {
  const uint32_t topbit = 1u << (N - 1);
  const int n1 = N - 3;                                 // part 1: bound1 = 2..N-2
  if (i < n1) return UConf{1, (uint32_t)(i + 2), 0, 0, 0, 0, topbit};
  const int k = i - n1;                                 // part 2: bound1 = 1.., bound2 = N-1-bound1
  const uint32_t sidemask = topbit | 1u;
  uint32_t lastmask = sidemask;
  for (int q = 0; q < k; q++) lastmask = (lastmask << 1) | lastmask | (lastmask >> 1);
  return UConf{2, (uint32_t)(k + 1), (uint32_t)(N - 2 - k), topbit >> (k + 1), lastmask, sidemask, topbit};
}

__device__ __forceinline__ uint32_t candidates(const UTask& t, uint32_t mask, const UConf& c) {
  return row_filter(mask & ~(t.left | t.down | t.right), t.row, t.down, c);
}

__global__ void __launch_bounds__(64) unique_init_kernel(int N, int nconf, UConf* confs, UTask* tasks, UCtl* ctl) {
  const int i = threadIdx.x;
  if (i < (int)(sizeof(UCtl) / 4)) reinterpret_cast<unsigned int*>(ctl)[i] = 0;
  __syncthreads();
  if (i >= nconf) return;
  const UConf c = make_conf(N, i);
  confs[i] = c;
  const uint32_t bit = 1u << c.bound1;
  UTask s{};
  s.conf = (uint32_t)i;
  if (c.part == 1) {
    s.left = (2u | bit) << 1; s.down = 1u | bit; s.right = (2u | bit) >> 1; s.row = 2;
    board_set(s, 0, 1u); board_set(s, 1, bit);
  } else {
    s.left = bit << 1; s.down = bit; s.right = bit >> 1; s.row = 1;
    board_set(s, 0, bit);
  }
  s.avail = candidates(s, (1u << N) - 1u, c);
  if (s.avail) tasks[atomicAdd(&ctl->n[0], 1u)] = s;
}

// Level l -> l + 1: one thread per state; its children with candidates left are counted, the warp reserves
// their slots with one atomic, and they are written.  States that must not be expanded move on as they are.
// n[l] <= 2^32: a level below the target (at most 2^21 states) has at most 27 children a state.
__global__ void __launch_bounds__(128) unique_expand_kernel(int N, int level, unsigned target, unsigned cap, const UConf* __restrict__ confs,
                                                            const UTask* __restrict__ in, UTask* __restrict__ out,
                                                            UCtl* ctl) {
  const unsigned n = ctl->n[level];
  if (n >= target) return;
  const uint32_t mask = (1u << N) - 1u;
  const unsigned lane = threadIdx.x & 31u;
  for (unsigned i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
    const unsigned i = i0 + threadIdx.x;
    UTask s{};
    UConf c{};
    bool keep = false;
    unsigned cnt = 0;
    auto each_child = [&](auto&& f) {
      for (uint32_t bm = s.avail; bm;) {
        const uint32_t bit = bm & (0u - bm);
        bm ^= bit;
        UTask t = s;
        t.left = (s.left | bit) << 1; t.down = s.down | bit; t.right = (s.right | bit) >> 1; t.row = s.row + 1;
        t.avail = candidates(t, mask, c);
        if (t.avail) f(t, bit);
      }
    };
    if (i < n) {
      s = in[i];
      c = confs[s.conf];
      keep = (int)s.row + 1 >= N - 1 || s.row + 1 >= (uint32_t)kBoardRows;
      if (keep) cnt = 1;
      else each_child([&](const UTask&, uint32_t) { cnt++; });
    }
    unsigned incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(FULLM, incl, o);
      if ((int)lane >= o) incl += v;
    }
    unsigned base = 0;
    if (lane == 31 && incl) base = atomicAdd(&ctl->n[level + 1], incl);
    base = __shfl_sync(FULLM, base, 31) + incl - cnt;
    if (base + cnt > cap) continue;      // the level does not fit: the queue stays the level before it
    if (keep) out[base] = s;
    else if (cnt) each_child([&](UTask& t, uint32_t bit) {
      board_set(t, s.row, bit);
      out[base++] = t;
    });
  }
}

}  // namespace
}  // namespace nq

using namespace nq;

extern "C" int nq_count_unique(nq_handle* h, int N, uint64_t* unique, uint64_t* total) {
  if (!h) return NQ_EINVAL;
  if (!unique || !total) return h->fail(NQ_EINVAL, "count_unique: null output");
  if (N < 4 || N > kMaxN) return h->fail(NQ_EINVAL, "count_unique: N=%d outside 4..27", N);
  // the handle's device and stream, and buffers the handle keeps between calls
  NQ_CUDA(h, cudaSetDevice(h->device));
  const int dev = h->device, sms = h->sms;
  cudaStream_t st = h->stream;
  const int nconf = (N - 3) + (N - 2) / 2;      // part 1: bound1 2..N-2; part 2: bound1 < N - 1 - bound1
  // Rows are expanded until the queue holds `target` tasks, unless the next row does not fit the buffer.
  // Lanes share work within a warp only, so the warps' sums have to even out: us of a whole count on GB300
  // with a target of 512 / 1024 / 4096 tasks per SM, N=15 303 / 303 / 227, N=16 921 / 936 / 736, N=17 11323 /
  // 4154 / 4204, N=18 56174 / 59898 / 27268 (5 10^5 tasks against 4.9 10^6).
  const unsigned target = (unsigned)sms * (N <= 15 ? 1024u : N <= 17 ? 4096u : 13824u);
  const size_t cap = (size_t)target * 5;
  NQ_CUDA(h, h->utasks.ensure(2 * cap * sizeof(UTask)));
  NQ_CUDA(h, h->uconfs.ensure((size_t)nconf * sizeof(UConf)));
  NQ_CUDA(h, h->uctl.ensure(sizeof(UCtl)));
  UCtl* ctl = (UCtl*)h->uctl.p;
  UConf* confs = (UConf*)h->uconfs.p;
  UTask* buf[2] = {(UTask*)h->utasks.p, (UTask*)h->utasks.p + cap};
  unique_init_kernel<<<1, 64, 0, st>>>(N, nconf, confs, buf[0], ctl);
  const int levels = N <= 9 ? 1 : std::min(kLevels, N - 3);   // N <= 9: a launch costs more than it balances
  for (int l = 0; l < levels; l++)
    unique_expand_kernel<<<l < 2 ? 1 : l == 2 ? sms : 4 * sms, 128, 0, st>>>(N, l, target, (unsigned)cap, confs, buf[l & 1],
                                                                            buf[(l + 1) & 1], ctl);
  NQ_CUDA(h, cudaGetLastError());
  if (int s = h->ensure_pinned(sizeof(UCtl))) return s;
  // Stacks sized to the tasks' rows need the level reached (one read-back); boards whose search takes less
  // than the wait run with the largest stacks.
  int row = 1;
  if (N >= kReadBackN) {
    NQ_CUDA(h, cudaMemcpyAsync(h->h_ctrl, ctl, sizeof(UCtl), cudaMemcpyDeviceToHost, st));
    NQ_CUDA(h, cudaStreamSynchronize(st));
    row = 1 + queue_level((const UCtl*)h->h_ctrl, (unsigned)cap);
  }
  const int maxf = std::max(1, N - 2 - row);
  constexpr int B = 128;
  const size_t smem = (size_t)B * ((size_t)maxf * sizeof(uint4) + (size_t)N * sizeof(uint32_t));
  int optin = 0;   // the cap is process-wide: set it to the device maximum, never to one launch's size
  NQ_CUDA(h, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  NQ_CUDA(h, cudaFuncSetAttribute(unique_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
  int per = 0;
  NQ_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, unique_kernel<B>, B, smem));
  if (per <= 0) return h->fail(NQ_ECUDA, "count_unique: N=%d does not fit on an SM", N);
  UArgs a;
  a.tasks[0] = buf[0]; a.tasks[1] = buf[1]; a.confs = confs; a.N = N; a.maxf = maxf; a.cap = (unsigned)cap; a.ctl = ctl;
  unique_kernel<B><<<sms * per, B, smem, st>>>(a);
  NQ_CUDA(h, cudaGetLastError());
  NQ_CUDA(h, cudaMemcpyAsync(h->h_ctrl, ctl, sizeof(UCtl), cudaMemcpyDeviceToHost, st));
  NQ_CUDA(h, cudaStreamSynchronize(st));
  const UCtl* hc = (const UCtl*)h->h_ctrl;
  *unique = hc->c2 + hc->c4 + hc->c8;
  *total = 2 * hc->c2 + 4 * hc->c4 + 8 * hc->c8;
  return NQ_OK;
}
