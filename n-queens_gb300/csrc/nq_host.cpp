// nq_host.cpp -- host-side task builders of the native library.
//
// 1. gen_constellations: start constellations with their x2/x4/x8 classes and
//    their preset-queen expansion (14Bit_codon_GPU/356Py_savesp_narrow.py:
//    2714-2926).  The start-constellation set is built sequentially (the
//    rotation check depends on insertion order, 356Py:2850-2880); the preset
//    expansion of each start constellation is independent and runs on the host
//    threads.  Output order: ascending packed ijkl, then
//    the reference's expansion order within a constellation.
// 2. completion_root: the root frame and per-depth ops of a board with pre-
//    placed queens (no reference counterpart: the reference only counts whole
//    boards).  Rows holding a pre-placed queen are skipped with a multi-row
//    step, and the queens' diagonals are carried in ld/rd from the root or
//    injected when they enter the bitboard, as the reference does for its
//    corner queens (blockK/blockL, 356Py:2586-2589).  The device expands it
//    (nq_gen.cu); build_completion_tasks expands it on the host for the
//    diagnostic nq_debug_completion_tasks.
#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "nq_common.cuh"
#include "nq_host.h"

namespace nq {

// ---------------------------------------------------------------------------
// generator
// ---------------------------------------------------------------------------
namespace {

inline int to_ijkl(int i, int j, int k, int l) { return (i << 15) + (j << 10) + (k << 5) + l; }
inline int rot90h(int x, int N) { return ((N - 1 - getk(x)) << 15) + ((N - 1 - getl(x)) << 10) + (getj(x) << 5) + geti(x); }
inline int canon(int x, int N) {   // jasmin, 356Py:2739-2756
  auto dist = [N](int v) { return std::min(v, N - 1 - v); };
  int arg = 0, mn = dist(getj(x));
  if (dist(geti(x)) < mn) { arg = 2; mn = dist(geti(x)); }
  if (dist(getk(x)) < mn) { arg = 3; mn = dist(getk(x)); }
  if (dist(getl(x)) < mn) { arg = 1; mn = dist(getl(x)); }
  for (int a = 0; a < arg; a++) x = rot90h(x, N);
  if (getj(x) < N - 1 - getj(x)) x = to_ijkl(N - 1 - geti(x), N - 1 - getj(x), getl(x), getk(x));
  return x;
}

// The reference looks every expanded state up (set_pre_queens_cached's subconst cache, 356Py:2773-2784, and
// the signatures up to preset 5, :2820-2824) and drops repeats.  No state occurs twice: enumerated for every
// N of 5..27 and presets 4, 5 and 6 (15.7 M states at N=27), and from preset 7 on the reference does not look.
// So nothing is looked up here; the list is the same, record for record.
struct Expander {
  int N, preset, k, l;
  uint64_t board_mask;
  std::vector<GenRecord>* out;
  uint32_t base;
  int err = 0;

  void expand(uint64_t ld, uint64_t rd, uint64_t col, int row, int queens, uint64_t LD, uint64_t RD) {
    while (row == k || row == l) { ld <<= 1; rd >>= 1; row++; }     // rows of the side queens
    if (queens == preset) {
      out->push_back(GenRecord{ld, rd, col, ((uint32_t)row << 20) | base});
      return;
    }
    const int sh = N - 1 - row;
    if (sh < 0) { err = 1; return; }   // the reference raises on a negative shift here
    uint64_t fr = ~(ld | rd | col | (LD >> sh) | (RD << sh)) & board_mask;
    while (fr) {
      const uint64_t bit = fr & (0 - fr);
      fr &= fr - 1;
      expand((ld | bit) << 1, (rd | bit) >> 1, col | bit, row + 1, queens + 1, LD, RD);
      if (err) return;
    }
  }
};

// Set of packed ijkl values of board N (below N << 15).
struct IjklSet {
  std::vector<uint64_t> w;
  explicit IjklSet(int N) : w((size_t)N << 9, 0) {}
  bool has(int x) const { return (w[(size_t)x >> 6] >> (x & 63)) & 1; }
  void add(int x) { w[(size_t)x >> 6] |= 1ull << (x & 63); }
};

bool rotated_present(const IjklSet& S, int i, int j, int k, int l, int N) {
  const int r1 = ((N - 1 - k) << 15) + ((N - 1 - l) << 10) + (j << 5) + i;
  const int r2 = ((N - 1 - j) << 15) + ((N - 1 - i) << 10) + ((N - 1 - l) << 5) + (N - 1 - k);
  const int r3 = (l << 15) + (k << 10) + ((N - 1 - i) << 5) + (N - 1 - j);
  return S.has(r1) || S.has(r2) || S.has(r3);
}

}  // namespace

int start_constellations(int N, std::vector<int>& starts) {
  starts.clear();
  if (N < 5 || N > kMaxN) return -1;
  const int halfN = (N + 1) / 2, N1 = N - 1, N2 = N - 2;
  // S: the set of start constellations, for the rotation check; C: their canonical
  // forms (jasmin), read out in ascending packed order (4 KB a board row each, so both
  // stay in the cache; byte flags and a sort took 178 us at N=16, these 108)
  IjklSet S(N), C(N);
  auto add = [&](int x) { if (!S.has(x)) { S.add(x); C.add(canon(x, N)); } };
  if (N % 2 == 1) {   // centre column of odd boards (356Py:2857-2867)
    const int c = N / 2;
    for (int l = c + 1; l < N1; l++)
      for (int i = c + 1; i < N1; i++) {
        if (i == N1 - l) continue;
        for (int j = N - c - 2; j > 0; j--)
          if (j != i && j != l && !rotated_present(S, i, j, c, l, N)) add(to_ijkl(i, j, c, l));
      }
  }
  for (int k = 1; k < halfN; k++)   // no queen in a corner (356Py:2869-2878)
    for (int l = k + 1; l < N1; l++)
      for (int i = k + 1; i < N1; i++) {
        if (i == N1 - l) continue;
        for (int j = N - k - 2; j > 0; j--)
          if (j != i && j != l && !rotated_present(S, i, j, k, l, N)) add(to_ijkl(i, j, k, l));
      }
  for (int j = 1; j < N2; j++)      // queen in a corner (356Py:2880)
    for (int l = j + 1; l < N1; l++) add(to_ijkl(0, j, 0, l));
  for (size_t q = 0; q < C.w.size(); q++)
    for (uint64_t b = C.w[q]; b; b &= b - 1) starts.push_back((int)(q << 6) | __builtin_ctzll(b));
  return 0;
}

int expand_starts(int N, int preset, const std::vector<int>& starts, size_t s0, size_t s1,
                  std::vector<GenRecord>& out, int threads) {
  if (N < 5 || N > kMaxN || preset < 1) return -1;
  if (preset < 4) return -2;   // the start constellations already hold 3-4 queens; the reference presets are 4..8
  const int N1 = N - 1;
  s1 = std::min(s1, starts.size());
  if (s0 >= s1) return 0;
  const size_t ns = s1 - s0;
  std::vector<std::vector<GenRecord>> parts(ns);
  std::atomic<size_t> next{0};
  std::atomic<int> err{0};
  auto worker = [&]() {
    Expander e;
    e.N = N; e.preset = preset; e.board_mask = (1ull << N) - 1;
    for (;;) {
      const size_t q = next.fetch_add(1);
      if (q >= ns) break;
      const int sc = starts[s0 + q];
      const int i = geti(sc), j = getj(sc), k = getk(sc), l = getl(sc);
      if (l < 1) { err = 1; break; }
      const uint64_t L = 1ull << N1, Lj = L >> j, Li = L >> i, Ll = L >> l;
      const uint64_t ld = ((i > 0) ? (L >> (i - 1)) : 0) | (1ull << (N - k));
      const uint64_t rd = (L >> (i + 1)) | (1ull << (l - 1));
      const uint64_t col = 1 | L | Li | Lj;
      e.k = k; e.l = l; e.out = &parts[q]; e.base = (uint32_t)to_ijkl(i, j, k, l);
      e.expand(ld, rd, col, 1, (j == N1) ? 3 : 4, Lj | Ll, Lj | (1ull << k));
      if (e.err) { err = 1; break; }
    }
  };
  if (threads <= 0) threads = (int)std::max(1u, std::thread::hardware_concurrency());
  // about 15 ns a record and 60 us a thread: a thread for every 20000 records (about (N - 4)^(preset - 4) a start)
  double est = (double)ns;
  for (int q = 4; q < preset; q++) est *= (double)std::max(1, N - q);
  threads = (int)std::min<double>((double)std::min<size_t>((size_t)threads, std::max<size_t>(1, ns / 8)), std::max(1.0, est / 20000.0));
  if (threads <= 1) worker();
  else {
    std::vector<std::thread> th;
    for (int t = 0; t < threads; t++) th.emplace_back(worker);
    for (auto& t : th) t.join();
  }
  if (err) return -2;
  size_t total = out.size();
  for (auto& p : parts) total += p.size();
  out.reserve(total);
  for (auto& p : parts) out.insert(out.end(), p.begin(), p.end());
  return 0;
}

int gen_constellations(int N, int preset, std::vector<GenRecord>& out, int threads) {
  out.clear();
  if (N < 5 || N > kMaxN || preset < 1) return -1;
  if (preset < 4) return -2;
  std::vector<int> starts;
  if (int s = start_constellations(N, starts)) return s;
  return expand_starts(N, preset, starts, 0, starts.size(), out, threads);
}

uint64_t board_states(int N, int preset) {
  if (N < 6 || N > kMaxN || preset < 4 || preset > 8) return 0;
  static constexpr uint32_t states[kMaxN - 5][5] = {      // N = 6.., preset 4..8
      {16u, 16u, 16u, 16u, 16u},
      {36u, 34u, 34u, 34u, 34u},
      {92u, 134u, 121u, 121u, 121u},
      {184u, 392u, 476u, 453u, 453u},
      {346u, 1007u, 1722u, 1878u, 1837u},
      {580u, 2161u, 5031u, 8100u, 8341u},
      {932u, 4300u, 12943u, 27931u, 40943u},
      {1404u, 7731u, 29043u, 79572u, 155925u},
      {2054u, 13233u, 60127u, 204112u, 512539u},
      {2884u, 21270u, 114209u, 466379u, 1444565u},
      {3964u, 33046u, 205709u, 992487u, 3705028u},
      {5296u, 49207u, 349418u, 1952839u, 8587857u},
      {6962u, 71475u, 571705u, 3653940u, 18656800u},
      {8964u, 100706u, 897071u, 6467354u, 37752890u},
      {11396u, 139232u, 1369061u, 11029570u, 72820769u},
      {14260u, 188147u, 2025282u, 18052162u, 133303405u},
      {17662u, 250485u, 2932689u, 28719035u, 235271863u},
      {21604u, 327606u, 4145833u, 44271796u, 399026853u},
      {26204u, 423338u, 5762269u, 66737631u, 657666813u},
      {31464u, 539335u, 7857828u, 98138478u, 1050644819u},
      {37514u, 680311u, 10568809u, 141731791u, 1640320717u},
      {44356u, 848242u, 13997139u, 200637190u, 2497629355u},
  };
  return states[N - 6][preset - 4];
}

// ---------------------------------------------------------------------------
// completion queries
// ---------------------------------------------------------------------------
int completion_root(int N, int k, const int* rows, const int* cols, uint32_t root[4], Op* ops, int* n_rows) {
  if (N < 1 || N > kMaxN || k < 0 || k > N) return -1;
  int fixed_col[32];
  for (int r = 0; r < N; r++) fixed_col[r] = -1;
  for (int q = 0; q < k; q++) {
    if (rows[q] < 0 || rows[q] >= N || cols[q] < 0 || cols[q] >= N) return -1;
    if (fixed_col[rows[q]] >= 0) return (fixed_col[rows[q]] == cols[q]) ? -1 : 1;
    fixed_col[rows[q]] = cols[q];
  }
  for (int a = 0; a < k; a++)       // attacking pre-placed queens: no completion
    for (int b = a + 1; b < k; b++) {
      const int dr = rows[a] - rows[b], dc = cols[a] - cols[b];
      if (cols[a] == cols[b] || dr == dc || dr == -dc) return 1;
    }
  int F[32], n = 0;
  for (int r = 0; r < N; r++)
    if (fixed_col[r] < 0) F[n++] = r;
  *n_rows = n;
  if (n == 0) return 2;   // every row holds a pre-placed queen and none attack: exactly one placement
  const uint32_t bm = (N >= 32) ? 0xFFFFFFFFu : ((1u << N) - 1u);
  // root frame at row F[0]
  uint32_t ld = 0, rd = 0, col = 0;
  if (n > kMaxDepth) return -1;
  for (int d = 0; d < n; d++) ops[d] = Op{1, 0, 0, 0, 0, 0};
  for (int q = 0; q < k; q++) {
    const int r = rows[q], c = cols[q];
    col |= 1u << c;
    // diagonal c - r + x (ld, moves up one bit per row)
    const int lpos = c - r + F[0];
    if (lpos >= 0) { if (lpos < 32) ld |= 1u << lpos; }
    else {
      const int enter = r - c;   // row where the diagonal reaches bit 0
      for (int d = 0; d + 1 < n; d++)
        if (F[d] < enter && enter <= F[d + 1]) { ops[d].la |= 1u << (F[d + 1] - enter); break; }
    }
    // anti-diagonal c + r - x (rd, moves down one bit per row)
    const int rpos = c + r - F[0];
    if (rpos >= 0 && rpos < 32) rd |= 1u << rpos;
    else if (rpos >= 32) {
      for (int d = 0; d + 1 < n; d++) {
        const int p = c + r - F[d + 1];
        if (p < 32) { if (p >= 0) ops[d].ra |= 1u << p; break; }
      }
    }
  }
  for (int d = 0; d + 1 < n; d++) ops[d].s = (uint32_t)(F[d + 1] - F[d]);
  ops[n - 1].term = 1; ops[n - 1].tall = 1;
  const int T = n - 1;
  extend_lookahead(ops, T);
  for (int d = 0; d < n; d++)
    if (!wide_fits(ops[d])) return -1;
  root[0] = ld; root[1] = rd; root[2] = col; root[3] = bm & ~(ld | rd | col);
  return 0;
}

int build_completion_tasks(int N, int k, const int* rows, const int* cols, int min_tasks, uint32_t job,
                           std::vector<HostTask>& out, int* max_T) {
  uint32_t root[4];
  Op ops[kMaxDepth + 1];
  int n = 0;
  if (const int s = completion_root(N, k, rows, cols, root, ops, &n)) return s;
  const int T = n - 1;
  const uint32_t bm = (1u << N) - 1u;

  // Expand the first levels breadth-first until there are enough tasks.
  struct F4 { uint32_t ld, rd, col, avail; };
  std::vector<F4> cur{F4{root[0], root[1], root[2], root[3]}}, nxt;
  int depth = 0;
  while (depth < T && (int)cur.size() < min_tasks) {
    nxt.clear();
    const Op& o = ops[depth];
    for (const F4& f : cur) {
      uint32_t av = f.avail;
      while (av) {
        const uint32_t bit = av & (0u - av);
        av ^= bit;
        const uint32_t nl = ((f.ld | bit) << o.s) | o.la, nr = ((f.rd | bit) >> o.s) | o.ra, nc = f.col | bit;
        const uint32_t nf = bm & ~(nl | nr | nc);
        if (nf) nxt.push_back(F4{nl, nr, nc, nf});
      }
    }
    cur.swap(nxt);
    depth++;
    if (cur.empty()) break;
  }
  const int Tt = T - depth;
  if (max_T && Tt > *max_T) *max_T = Tt;
  for (const F4& f : cur) {
    if (f.avail == 0) continue;
    HostTask h;
    h.root[0] = f.ld; h.root[1] = f.rd; h.root[2] = f.col; h.root[3] = f.avail;
    h.info = info_pack((uint32_t)Tt, 0, 0, (uint32_t)N, TS_OK);
    h.job = job;
    h.T = Tt;
    for (int d = 0; d <= Tt; d++) { h.sched[2 * d] = pack_wide_x(ops[depth + d]); h.sched[2 * d + 1] = ops[depth + d].ra; }
    out.push_back(h);
  }
  return 0;
}

int64_t start_row_min(const uint32_t* startijkl, int64_t m, int stride_words) {
  int64_t mn = 64;
  for (int64_t i = 0; i < m; i++) {
    const int64_t s = (int64_t)(startijkl[i * stride_words] >> 20);
    if (s < mn) mn = s;
  }
  return mn;
}

}  // namespace nq
