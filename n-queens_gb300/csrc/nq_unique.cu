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
// work shared in a warp at the end of the queue), keeping each lane's board
// (one bit per row) in shared memory for the leaf classification.
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
// Steps per lane between checks for finished lanes, a multiple of the steps unrolled.  A whole count at N=18,
// unrolled by 2 / 5 / 10: 18.7 / 18.2 / 18.1 ms; by 30 the loop and the classification in it outgrow the instruction
// cache (a quarter slower), and 20 steps a check are 1 % slower than 30.
constexpr int kUniqueSteps = 30, kUniqueUnroll = 5;
// Boards from here on size the stacks to the tasks' rows (N=14 96 us without the read-back, 111 with; N=15 187
// against 190, and the search grows sixfold a size from there).
constexpr int kReadBackN = 15;
constexpr int kGiveRows = 6;         // rows left in a frame worth giving away

// One start configuration (symmetry part and its bounds).
struct UConf {
  uint32_t part;       // 1 corner, 2 no corner
  uint32_t bound1, bound2, lastmask, sidemask;
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

// symmetryops (07Py_bit_symmetry.py:65-125) on one board, by the warp: 2, 4 or 8 for a canonical solution, 0 for
// a rotated copy.  Lane r holds row r's column `c` (lanes from N on hold nothing).  Row r of the board turned by
// 90, 180 and 270 degrees comes from the row of column r, row N-1-r, and the row of column N-1-r; a rotation
// whose row 0 differs is left out, otherwise the first row that differs decides.  `inv` is 32 words of the warp's
// shared memory for the rows by column.
// Bound by issue: about 60 instructions of the warp a board, on the quarter of the boards that have a rotation
// with their own row 0 (the others count x8 after two loads of their own lane).  One step in 104 stands on such a
// part's last row (N=16), so one warp step in 4 has one: at N=18 a count took 15.0 ms without any
// classification, 21.0 with a lane searching its own board for each column, 23.4 with every board here, and
// 19.6 with the check before.
__device__ __forceinline__ uint32_t classify(uint32_t c, uint32_t lane, uint32_t N, uint32_t* inv) {
  const bool in = lane < N;
  const uint32_t other = in ? N - 1u - lane : lane;
  if (in) inv[c] = lane;
  const uint32_t c180 = N - 1u - __shfl_sync(FULLM, c, (int)other);
  __syncwarp();
  const uint32_t c90 = N - 1u - inv[lane], c270 = inv[other];
  const uint32_t ne90 = __ballot_sync(FULLM, in && c != c90), gt90 = __ballot_sync(FULLM, c > c90);
  const uint32_t ne180 = __ballot_sync(FULLM, in && c != c180), gt180 = __ballot_sync(FULLM, c > c180);
  const uint32_t ne270 = __ballot_sync(FULLM, in && c != c270), gt270 = __ballot_sync(FULLM, c > c270);
  if (ne90 == 0u) return 2;
  if (!(ne90 & 1u) && (gt90 & ne90 & (0u - ne90))) return 0;
  if (ne180 == 0u) return 4;
  if (!(ne180 & 1u) && (gt180 & ne180 & (0u - ne180))) return 0;
  if (!(ne270 & 1u) && (gt270 & ne270 & (0u - ne270))) return 0;
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
  unsigned int cursor, done;    // done: blocks of unique_kernel that have ended
  unsigned int n[kLevels + 1];
};
// Levels alternate between two buffers of cap[0] and cap[1] tasks.
struct UCap { unsigned cap[2]; };
// The queue is the last level with states in it that its buffer holds (a level that was large enough, or whose states
// all died, leaves the next one empty).
__host__ __device__ __forceinline__ int queue_level(const UCtl* c, const UCap& b) {
  int f = 0;
  for (int l = 1; l <= kLevels; l++)
    if (c->n[l] && c->n[l] <= b.cap[l & 1]) f = l;
  return f;
}

struct UArgs {
  const UTask* tasks[2];
  const UConf* confs;
  int N;
  int nconf;
  int maxf;                     // stack frames per lane: the sentinel's and one per row from the smallest task row
  UCap cap;
  UCtl* ctl;
  uint32_t* host;               // pinned: receives the control block
};

// Shared-memory accesses at 32-bit shared-window addresses.
__device__ __forceinline__ void sts_frame_u(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts_word_u(uint32_t a, uint32_t x) {
  asm volatile("st.shared.u32 [%0], %1;" :: "r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ uint32_t lds_word_u(uint32_t a) {
  uint32_t w;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(a) : "memory");
  return w;
}
__device__ __forceinline__ void lds_frame_u(uint32_t a, uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& w) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a) : "memory");
}

// The rules of a configuration's rows as words, read by the columns left (popc(fr)) of a frame: the columns
// its child's row may use, what a frame in the last row counts, and whether the child must have both side
// columns behind it.
constexpr uint32_t U_COUNT = 1u << 27;      // part 1, last row: a solution, x8
constexpr uint32_t U_CLASSIFY = 1u << 28;   // part 2, last row: a board to classify
constexpr uint32_t U_NOLOOK = 1u << 29;     // the child's row is the last one: there is none behind it
constexpr uint32_t U_SIDES = 1u << 31;      // part 2, row bound2 + 1: dead while a side column is free
__host__ __device__ __forceinline__ uint32_t row_word(const UConf& c, int N, int left) {
  if (left == 0) return 0u;                 // the sentinel: every child dies
  if (left == 1) return c.part == 1 ? U_COUNT : U_CLASSIFY;
  const uint32_t child = (uint32_t)(N - left + 1);
  const uint32_t columns = (1u << N) - 1u;
  uint32_t w = columns;
  if (left == 2) w |= U_NOLOOK;
  if (child < c.bound1) w &= c.part == 1 ? ~2u : ~c.sidemask;
  if (c.part != 1) {
    if (child == (uint32_t)N - 1u) w &= ~(c.lastmask & columns);   // lastmask has grown past the board, onto the flags
    // Row bound2 must take the last free side column (backTrack2, :126-151): after it both are behind.  Its
    // own candidates go unfiltered and die one step on: 5 % more steps (N=15 39.7 10^6 against 37.6, N=16 259
    // against 246, before the look-ahead), each about four instructions shorter.
    if (child == c.bound2 + 1u) w |= U_SIDES;
  }
  return w;
}

// One lane per task, one candidate per step, all lanes on the same predicated sequence, as in the
// constellation DFS (nq_kernels.cu): the child always becomes the current frame, the frame is saved with the
// rest of its candidates whether or not there are any, a solution is a frame in the last row, and a sentinel
// frame whose 31 candidates die feeds a lane without work.  Each step also records its queen in the lane's
// board.  A frame is {left, right, free columns, candidates}; its row is N - popc(free columns).
// Bound by issue and latency (N=17: 46 warp instructions a step, a quarter of them the last rows' boards; issue 70 %,
// shared memory 74 % of its wavefronts, ALU 56 %, 24 warps an SM by shared memory).  With the row in `down`'s high
// bits, the rules computed at each step and predicated pushes a count took 27.3 ms at N=18 and 4.2 at N=17; with
// the step as here 21.5 and 3.4; boards classified by the warp 19.6 and 3.08; look-ahead over the row after the
// child (17 % fewer steps for 4 instructions) 18.5 and 2.94; board rows BLOCK words apart, so a step's stores
// meet no bank twice (one word more made the warp's reads of a board meet none instead) 18.2 and 2.90.
constexpr uint32_t kUSentinel = 0xFFFFFFFEu;
static_assert(kUniqueSteps <= 30, "the sentinel holds 31 candidates, and one has to be left at a check");
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) unique_kernel(const UArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int N = a.N;
  constexpr uint32_t F = BLOCK * (uint32_t)sizeof(uint4);          // frame stride of one lane's stack
  constexpr uint32_t RB = BLOCK * (uint32_t)sizeof(uint32_t);      // board row stride
  // maxf frames (the sentinel's, one per row), N + 1 board rows (the last one is the sentinel's), 32 words a
  // warp for classify, the rows' words
  uint32_t* inv = reinterpret_cast<uint32_t*>(smem + (size_t)a.maxf * F + (size_t)(N + 1) * RB) + (threadIdx.x & ~31u);
  uint32_t* table = reinterpret_cast<uint32_t*>(smem + (size_t)a.maxf * F + (size_t)(N + 1) * RB) + BLOCK;
  const uint32_t bottom = (uint32_t)__cvta_generic_to_shared(smem) + threadIdx.x * (uint32_t)sizeof(uint4);
  const uint32_t brd = (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)a.maxf * F + threadIdx.x * 4u;   // row 0
  const uint32_t tab = (uint32_t)__cvta_generic_to_shared(table);
  chain_wait();
  for (int q = threadIdx.x; q < a.nconf * (N + 1); q += BLOCK) table[q] = row_word(a.confs[q / (N + 1)], N, q % (N + 1));
  __syncthreads();
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t mask = (1u << N) - 1u, side = (1u << (N - 1)) | 1u;
  const uint32_t brd_end = brd + (uint32_t)N * RB;
  uint32_t left = 0, right = 0, fr = 0, avail = 0;
  uint32_t top = bottom + F;            // above the sentinel; moves up when the lane gives its bottom frame away
  uint32_t sp = top, conf = 0, words = tab;
  uint32_t brd1 = brd, brd2 = brd, last_col = 0;   // part 2: rows bound1 and bound2 of the board, 1 << bound2
  const uint32_t topbit = 1u << (N - 1);
  auto set_conf = [&](uint32_t k) {
    const uint32_t b1 = a.confs[k].bound1, b2 = a.confs[k].bound2;
    conf = k;
    words = tab + k * (uint32_t)(N + 1) * 4u;
    brd1 = brd + b1 * RB; brd2 = brd + b2 * RB; last_col = 1u << b2;
  };
  uint32_t cnt = 0;
  unsigned long long c8 = 0;
  unsigned long long w2 = 0, w4 = 0, w8 = 0;   // the warp's classified boards, the same in its lanes
  bool exhausted = false;
  auto arm = [&]() { sts_frame_u(top - F, 0u, 0u, 0u, kUSentinel); };
  arm();
  const int level = queue_level(a.ctl, a.cap);
  const UTask* tasks = a.tasks[level & 1];
  const unsigned m = a.ctl->n[level];
  // where the queue is smaller than the lanes, each warp takes its share and shares it among its lanes
  const unsigned warps = gridDim.x * (BLOCK / 32);
  const unsigned take = min(32u, (m + warps - 1u) / warps);
  for (;;) {
    c8 += cnt;
    cnt = 0;
    bool idle = avail == 0u && sp == top;
    if (__ballot_sync(FULLM, idle)) {
      if (idle) { top = bottom + F; sp = top; arm(); }
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
          set_conf(t.conf);
          left = t.left; right = t.right; fr = mask & ~t.down; avail = t.avail;
          for (uint32_t r = 0; r < t.row && r < (uint32_t)kBoardRows; r++) sts_word_u(brd + r * RB, board_bit(t, r));
          idle = false;
        }
        exhausted = take < 32u || base + n_take >= m;   // warp-uniform
      }
      if (exhausted) {
        // The queue is empty: a lane without work takes the bottom saved frame of a busy lane of its warp,
        // or all but one candidate of its current frame, with the rows of the board above it.
        const unsigned starved = __ballot_sync(FULLM, idle);
        const bool saved = sp != top;
        const uint32_t rest = avail & (avail - 1u);
        const uint32_t gfr = saved ? lds_word_u(top + 8u) : fr;
        const bool can = !idle && (saved ? (avail != 0u || sp != top + F) : rest != 0u) && __popc(gfr) >= kGiveRows;
        const unsigned givers = starved ? __ballot_sync(FULLM, can) : 0u;
        if (givers) {
          const unsigned lt = (1u << lane) - 1u;
          const int n = min(__popc(starved), __popc(givers));
          const bool gives = can && __popc(givers & lt) < n;
          const int srank = __popc(starved & lt);
          const bool takes = idle && srank < n;
          if (gives && !saved) { sts_frame_u(top, left, right, fr, rest); avail ^= rest; }
          __syncwarp();
          const int src = takes ? (int)nth_set(givers, (uint32_t)srank) : (int)lane;
          const uint32_t from = __shfl_sync(FULLM, top, src), fconf = __shfl_sync(FULLM, conf, src);
          const uint32_t fbrd = __shfl_sync(FULLM, brd, src);
          if (takes) {
            lds_frame_u(from, left, right, fr, avail);
            set_conf(fconf);
            const uint32_t rows = (uint32_t)(N - __popc(fr));
            for (uint32_t r = 0; r < rows; r++) sts_word_u(brd + r * RB, lds_word_u(fbrd + r * RB));
            idle = false;
          }
          __syncwarp();
          if (gives && saved) { top += F; arm(); }
        }
      }
      if (__all_sync(FULLM, exhausted && idle)) break;
    }
    // kUniqueSteps steps between two checks for finished lanes (two ballots each)
#pragma unroll kUniqueUnroll
    for (int s = 0; s < kUniqueSteps; ++s) {
      asm volatile("{\n\t.reg .pred q;\n\tsetp.eq.u32 q, %3, 0;\n\t"
                   "@q sub.u32 %4, %4, %5;\n\t@q ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
                   : "+r"(left), "+r"(right), "+r"(fr), "+r"(avail), "+r"(sp) : "n"(F));
      const uint32_t pf = __popc(fr);                           // columns, and rows, left
      const uint32_t w = lds_word_u(words + pf * 4u);
      const uint32_t rest = avail & (avail - 1u);
      const uint32_t bit = avail - rest;
      sts_frame_u(sp, left, right, fr, rest);
      if (rest != 0u) sp += F;
      sts_word_u(brd_end - pf * RB, bit);                       // the row's queen
      const uint32_t nl = (left + bit) * 2u;
      const uint32_t nr = __umulhi(right + bit, 0x80000000u);   // (right | bit) >> 1
      const uint32_t free_cols = fr - bit;
      const uint32_t nb = free_cols & ~(nl | nr) & w;
      const uint32_t keep = (free_cols & ~((nl + nl) | __umulhi(nr, 0x80000000u))) | (w & U_NOLOOK);   // look-ahead
      const bool dead = (free_cols & side & (uint32_t)((int32_t)w >> 31)) != 0u;
      if (w & U_COUNT) cnt += 1u;
      if (__any_sync(FULLM, (w & U_CLASSIFY) != 0u)) {
        bool turns = false;               // a rotation has the board's own row 0
        if (w & U_CLASSIFY) {
          turns = lds_word_u(brd2) == 1u || lds_word_u(brd1) == topbit || bit == last_col;
          if (!turns) cnt += 1u;
        }
        unsigned boards = __ballot_sync(FULLM, turns);
        __syncwarp();
        while (boards) {
          const int src = __ffs((int)boards) - 1;
          boards &= boards - 1u;
          const uint32_t from = __shfl_sync(FULLM, brd, src);
          const uint32_t row = lane < (uint32_t)N ? lds_word_u(from + lane * RB) : 1u;
          const uint32_t k = classify((31u - (uint32_t)__clz((int)row)) & 31u, lane, (uint32_t)N, inv);
          w2 += (k == 2); w4 += (k == 4); w8 += (k == 8);
          __syncwarp();
        }
      }
      left = nl; right = nr; fr = free_cols;
      avail = dead || keep == 0u ? 0u : nb;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c8 += __shfl_xor_sync(FULLM, c8, o);
  c8 += w8;
  if (lane == 0) {
    if (w2) atomicAdd(&a.ctl->c2, w2);
    if (w4) atomicAdd(&a.ctl->c4, w4);
    if (c8) atomicAdd(&a.ctl->c8, c8);
  }
  hand_over((const uint32_t*)a.ctl, sizeof(UCtl) / 8, &a.ctl->done, a.host);
}

// ---------------------------------------------------------------------------
// Task queue: every (part, bound1) start of 07Py_bit_symmetry.py NQueens()
// (:171-200), expanded a whole row at a time (tasks of one row are of similar
// size) until there are enough tasks, they reach the last row, or their rows
// no longer fit the board prefix.  Bound by launch latency: about 2 us a row
// at N=12; the same expansion on one host thread and its upload took 0.8 ms at
// N=12, 6 ms at N=14 and 25 ms at N=16.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ UConf make_conf(int N, int i) {
  const uint32_t topbit = 1u << (N - 1);
  const int n1 = N - 3;                                 // part 1: bound1 = 2..N-2
  if (i < n1) return UConf{1, (uint32_t)(i + 2), 0, 0, 0};
  const int k = i - n1;                                 // part 2: bound1 = 1.., bound2 = N-1-bound1
  const uint32_t sidemask = topbit | 1u;
  uint32_t lastmask = sidemask;
  for (int q = 0; q < k; q++) lastmask = (lastmask << 1) | lastmask | (lastmask >> 1);
  return UConf{2, (uint32_t)(k + 1), (uint32_t)(N - 2 - k), lastmask, sidemask};
}

__device__ __forceinline__ uint32_t candidates(const UTask& t, uint32_t mask, const UConf& c) {
  return row_filter(mask & ~(t.left | t.down | t.right), t.row, t.down, c);
}

__global__ void __launch_bounds__(64) unique_init_kernel(int N, int nconf, UConf* confs, UTask* tasks, UCtl* ctl) {
  const int i = threadIdx.x;
  chain_next();
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
// n[l] <= 2^32: a level below the target (at most 2^21 states) has at most 27 children a state.  A level that did not
// fit its buffer is not expanded: the queue stays the level before it.
__global__ void __launch_bounds__(128) unique_expand_kernel(int N, int level, unsigned target, UCap room, const UConf* confs,
                                                            const UTask* in, UTask* __restrict__ out,
                                                            UCtl* ctl) {
  chain_next();
  chain_wait();
  const unsigned n = ctl->n[level];
  if (n >= target || n > room.cap[level & 1]) return;
  const unsigned cap = room.cap[(level + 1) & 1];
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
    if (base + cnt > cap) continue;
    if (keep) out[base] = s;
    else if (cnt) each_child([&](UTask& t, uint32_t bit) {
      board_set(t, s.row, bit);
      out[base++] = t;
    });
  }
}

// States after each level, which sizes the buffers (enumerated; a board whose rows end before holds its states).
uint32_t level_states(int N, int level) {
  static constexpr uint32_t n[kMaxN - 3][kLevels + 1] = {       // N = 4..
      {1, 1, 1, 1, 1, 1, 1},
      {2, 3, 3, 3, 3, 3, 3},
      {4, 7, 7, 5, 5, 5, 5},
      {6, 12, 21, 24, 17, 17, 17},
      {8, 23, 50, 92, 80, 48, 48},
      {9, 35, 97, 243, 358, 308, 174},
      {11, 53, 183, 541, 1107, 1503, 1286},
      {12, 69, 290, 1054, 2903, 5578, 6964},
      {14, 94, 469, 1985, 6608, 16453, 27662},
      {15, 115, 670, 3293, 13070, 41743, 87139},
      {17, 147, 983, 5520, 25294, 95196, 230022},
      {18, 173, 1310, 8349, 43935, 192828, 540547},
      {20, 212, 1797, 12840, 76218, 380680, 1168189},
      {21, 243, 2282, 18161, 121116, 686457, 2272413},
      {23, 289, 2983, 26204, 194112, 1228927, 4388380},
      {24, 325, 3658, 35253, 288698, 2035297, 7724564},
      {26, 378, 4613, 48444, 434896, 3377711, 13757078},
      {27, 419, 5510, 62721, 614466, 5238820, 22456135},
      {29, 479, 6759, 82968, 881352, 8185547, 37537711},
      {30, 525, 7910, 104237, 1195780, 12054968, 57765474},
      {32, 592, 9493, 133760, 1648896, 17937511, 91713177},
      {33, 643, 10930, 164049, 2165344, 25336316, 134614515},
      {35, 717, 12887, 205380, 2891344, 36219683, 204807695},
      {36, 773, 14642, 246981, 3696940, 49438122, 289262952},
  };
  return n[N - 4][level];
}

}  // namespace
}  // namespace nq

using namespace nq;

extern "C" int64_t nq_debug_unique_states(int N, int level) {
  return N < 4 || N > kMaxN || level < 0 || level > kLevels ? NQ_EINVAL : (int64_t)level_states(N, level);
}

extern "C" int nq_debug_unique_words(int N, int conf, uint32_t* words) {
  if (N < 4 || N > kMaxN || conf < 0 || conf >= (N - 3) + (N - 2) / 2 || !words) return NQ_EINVAL;
  for (int left = 0; left <= N; left++) words[left] = row_word(make_conf(N, conf), N, left);
  return NQ_OK;
}

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
  // Lanes share work within a warp only, so the warps' sums have to even out: relative time of a whole count on GB300
  // with a target of 512 / 1024 / 4096 / 13824 tasks per SM, N=15 1.26 / 1.26 / 1 / 1.01 (of 170 us), N=16 1.08 / 1.09 /
  // 1 / 1.01 (540 us), N=17 2.52 / 1 / 1 / 1 (2.90 ms), N=18 1.93 / 1.89 / 1.08 / 1 (18.2 ms).
  const unsigned target = (unsigned)sms * (N <= 17 ? 4096u : 13824u);
  int levels = 0;                               // N <= 9: a launch costs more than it balances
  for (const int most = N <= 9 ? 1 : std::min(kLevels, N - 3);
       levels < most && level_states(N, levels) < target && level_states(N, levels + 1) <= 5ull * target;) levels++;
  UCap room{};
  for (;; levels--) {                           // a level less where the device has no room for it
    room = UCap{};
    for (int l = 0; l <= levels; l++) room.cap[l & 1] = std::max(room.cap[l & 1], level_states(N, l));
    const cudaError_t e = h->utasks.ensure(((size_t)room.cap[0] + room.cap[1]) * sizeof(UTask));
    if (e == cudaErrorMemoryAllocation && levels > 0) { cudaGetLastError(); continue; }
    NQ_CUDA(h, e);
    break;
  }
  NQ_CUDA(h, h->uconfs.ensure((size_t)nconf * sizeof(UConf)));
  NQ_CUDA(h, h->uctl.ensure(sizeof(UCtl)));
  UCtl* ctl = (UCtl*)h->uctl.p;
  UConf* confs = (UConf*)h->uconfs.p;
  UTask* buf[2] = {(UTask*)h->utasks.p, (UTask*)h->utasks.p + room.cap[0]};
  unique_init_kernel<<<1, 64, 0, st>>>(N, nconf, confs, buf[0], ctl);
  for (int l = 0; l < levels; l++)
    NQ_CUDA(h, launch_after(unique_expand_kernel, l < 2 ? 1 : l == 2 ? sms : 4 * sms, 128, 0, st, N, l, target, room, confs,
                            buf[l & 1], buf[(l + 1) & 1], ctl));
  NQ_CUDA(h, cudaGetLastError());
  if (int s = h->ensure_pinned(sizeof(UCtl))) return s;
  // Stacks sized to the tasks' rows need the level reached (one read-back); boards whose search takes less
  // than the wait run with the largest stacks.
  int row = 1;
  if (N >= kReadBackN) {
    NQ_CUDA(h, cudaMemcpyAsync(h->h_ctrl, ctl, sizeof(UCtl), cudaMemcpyDeviceToHost, st));
    NQ_CUDA(h, cudaStreamSynchronize(st));
    row = 1 + queue_level((const UCtl*)h->h_ctrl, room);
  }
  const int maxf = N - row + 1;
  constexpr int B = 128;   // N=18: 64 / 128 / 256 threads 20.3 / 19.6 / 19.9 ms
  const size_t smem = (size_t)B * maxf * sizeof(uint4) + (size_t)(N + 1) * B * sizeof(uint32_t) +
                      (size_t)B * sizeof(uint32_t) + (size_t)nconf * (N + 1) * sizeof(uint32_t);
  int optin = 0;   // the cap is process-wide: set it to the device maximum, never to one launch's size
  NQ_CUDA(h, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  NQ_CUDA(h, cudaFuncSetAttribute(unique_kernel<B>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
  int per = 0;
  NQ_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, unique_kernel<B>, B, smem));
  if (per <= 0) return h->fail(NQ_ECUDA, "count_unique: N=%d does not fit on an SM", N);
  UArgs a;
  a.tasks[0] = buf[0]; a.tasks[1] = buf[1]; a.confs = confs; a.nconf = nconf; a.N = N; a.maxf = maxf; a.cap = room; a.ctl = ctl;
  a.host = (uint32_t*)h->h_ctrl;
  NQ_CUDA(h, launch_after(unique_kernel<B>, sms * per, B, smem, st, a));
  NQ_CUDA(h, cudaStreamSynchronize(st));
  const UCtl* hc = (const UCtl*)h->h_ctrl;
  *unique = hc->c2 + hc->c4 + hc->c8;
  *total = 2 * hc->c2 + 4 * hc->c4 + 8 * hc->c8;
  return NQ_OK;
}
