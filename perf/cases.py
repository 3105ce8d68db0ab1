"""The work whose speed this repository answers for: calls a user of the engine makes, with their sizes.

A case is one call (or the calls of one request) through the public entry points, at one size.  The kinds:

  table        whole-board counts of every size up to a limit, one call per board (the loop of the reference's main())
  completions  one completion query: a board with k pre-placed queens, built, counted and released
  request      a batch built, run once and released: what a serving loop does with the requests it has gathered
  replay       a batch whose tasks stay resident, run again through its captured graph
  records      a task list in host memory, per-record solutions back in host memory (the drop-in exec_solutions)
  device       a task list in device memory, per-record solutions left in device memory
  noalloc      the same through the entry point that never allocates
  starts       a range of start constellations of a large board, generated on the host while the GPU counts
               (the unit of a resumable count)
  unique       unique and total counts by the symmetry method, one call per board

Task lists are the engine's own (gen_records), rotated to a seeded offset or cut to a seeded subset, so their values
are those of real lists; queens, job mixes and ranges come from the seed.
"""
import ctypes
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "n-queens_gb300"))

import nqueens  # noqa: E402
from nqueens import CompletionJob, CountJob  # noqa: E402

# Search nodes of a whole board at its default preset (one candidate queen each), and the records of its task list.
NODES = {6: 20, 7: 60, 8: 200, 9: 1000, 10: 4980, 11: 27032, 12: 145880, 13: 787610, 14: 4578224, 15: 27864613,
         16: 182533515, 17: 1247485360, 18: 9087554384, 19: 69276398858, 20: 557537122738, 21: 4.67e12, 22: 4.1e13,
         23: 3.7e14, 24: 3.5e15}
RECORDS = {6: 5, 7: 29, 8: 134, 9: 392, 10: 1007, 11: 2161, 12: 4300, 13: 7731, 14: 13233, 15: 21270, 16: 33046,
           17: 49207, 18: 571705, 19: 897071, 20: 1369061, 21: 2025282, 22: 28.7e6, 23: 44.3e6, 24: 66.7e6}
STARTS = {18: 5728, 19: 7432, 20: 9522, 21: 11997, 22: 14960, 23: 18402, 24: 22462}
NODE_OPS = 12         # integer operations per node: lowest bit, three occupancy updates, next row's free set, test

_lists = {}


def listed():
    return [
        # The reference's own main loop over small boards: nothing but latency, launches and host work.
        {"name": "table_6_13", "kind": "table", "lo": 6, "hi": 13},
        # The smallest interactive query: one board, a few queens, answer in a fraction of a millisecond.
        {"name": "completion_n10_k2", "kind": "completions", "n": 10, "k": 2},
        # An ordinary interactive query (the served stream's middle: N 14..20, k 0..4).
        {"name": "completion_n17_k2", "kind": "completions", "n": 17, "k": 2},
        # A serving loop's batch of small gathered requests: counts and queries mixed, built, run and released.
        {"name": "request_mixed_64", "kind": "request", "jobs": 64, "lo": 9, "hi": 16},
        # Many resident counting jobs replayed as one graph launch (the benchmark's 256-job mix, boards 10..17).
        {"name": "replay_count_256", "kind": "replay", "jobs": 256, "lo": 10, "hi": 17},
        # A small task list through the drop-in call, odd length, per-record results.
        {"name": "records_n14", "kind": "records", "n": 14, "m": 12289},
        # The largest list of preset 5, whole.
        {"name": "records_n17", "kind": "records", "n": 17, "m": 49207},
        # The benchmark's board, whole list resident on the device: the steady state of the search kernel.
        {"name": "device_n19", "kind": "device", "n": 19, "m": 897071},
        # The longest single count a user waits for in one call here.
        {"name": "device_n20", "kind": "device", "n": 20, "m": 1369061},
        # A call that may not allocate, a ragged subset of a mid-size list.
        {"name": "noalloc_n16", "kind": "noalloc", "n": 16, "m": 20011},
        # One step of a resumable count of a large board: preset 7, deep stacks, host generation overlapped.
        {"name": "starts_n22", "kind": "starts", "n": 22, "count": 48},
        # The symmetry-method counter over a table of boards.
        {"name": "unique_12_17", "kind": "unique", "lo": 12, "hi": 17},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["table", "completions", "completions", "request", "replay", "records", "records", "device",
                       "device", "noalloc", "starts", "unique"])
    if kind == "table":
        lo = rng.randint(6, 10)
        return {"kind": kind, "lo": lo, "hi": rng.randint(lo + 3, 16)}
    if kind == "completions":
        n = rng.randint(8, 20)
        return {"kind": kind, "n": n, "k": rng.randint(1 if n < 18 else 2, 5)}
    if kind == "request":
        lo = rng.randint(6, 12)
        return {"kind": kind, "jobs": _log_int(rng, 2, 256), "lo": lo, "hi": rng.randint(lo + 1, 16)}
    if kind == "replay":
        lo = rng.randint(6, 14)
        return {"kind": kind, "jobs": _log_int(rng, 4, 256), "lo": lo, "hi": rng.randint(lo + 1, 17)}
    if kind == "records":
        n = rng.randint(10, 19)
        return {"kind": kind, "n": n, "m": _log_int(rng, 100, RECORDS[n])}
    if kind == "device":
        n = rng.randint(14, 20)
        return {"kind": kind, "n": n, "m": _log_int(rng, RECORDS[n] // 64, RECORDS[n])}
    if kind == "noalloc":
        n = rng.randint(10, 17)
        return {"kind": kind, "n": n, "m": _log_int(rng, 100, RECORDS[n])}
    if kind == "starts":
        n = rng.randint(18, 23)
        return {"kind": kind, "n": n, "count": _log_int(rng, 8, {18: 5000, 19: 5000, 20: 4000, 21: 800, 22: 80, 23: 10}[n])}
    lo = rng.randint(6, 14)
    return {"kind": kind, "lo": lo, "hi": rng.randint(lo + 2, 18)}


def _records(n):
    if n not in _lists:
        _lists[n] = nqueens.gen_records(n)
    return _lists[n]


def _some_records(n, m, rng):
    """m records of the board's list: the list rotated to a seeded offset, or a seeded subset in list order."""
    r = _records(n)
    if m >= len(r):
        return np.roll(r, rng.randrange(1, len(r)))
    at = np.random.default_rng(rng.randrange(1 << 30)).choice(len(r), size=m, replace=False)
    return np.ascontiguousarray(r[np.sort(at)])


def _queens(n, k, rng):
    """k non-attacking queens on an n x n board."""
    while True:
        q = list(zip(rng.sample(range(n), k), (rng.randrange(n) for _ in range(k))))
        if all(a[1] != b[1] and abs(a[0] - b[0]) != abs(a[1] - b[1]) for i, a in enumerate(q) for b in q[:i]):
            return q


def _jobs(case, rng):
    jobs = []
    for _ in range(case["jobs"]):
        n = rng.randint(case["lo"], case["hi"])
        if case["kind"] == "replay" or rng.random() < 0.4:
            jobs.append(CountJob(n))
        else:
            jobs.append(CompletionJob(n, _queens(n, rng.randint(1, 4), rng)))
    return jobs


def prepare(case, seed):
    rng = random.Random(seed * 7919 + 17)
    eng = nqueens.default_engine()
    kind = case["kind"]
    s = {"case": case, "eng": eng}
    if kind in ("table", "unique"):
        s["boards"] = list(range(case["lo"], case["hi"] + 1))
        rng.shuffle(s["boards"])
    elif kind == "completions":
        s["queens"] = _queens(case["n"], case["k"], rng)
    elif kind == "request":
        s["jobs"] = _jobs(case, rng)
    elif kind == "replay":
        s["batch"] = eng.batch(_jobs(case, rng))
    elif kind == "records":
        s["records"] = _some_records(case["n"], case["m"], rng)
    elif kind in ("device", "noalloc"):
        r = _some_records(case["n"], case["m"], rng)
        s["m"], s["start_min"] = len(r), int((r["startijkl"] >> 20).min())
        s["records"] = torch.from_numpy(r.view(np.int32).copy()).cuda()
        s["solutions"] = torch.zeros(len(r), dtype=torch.int64, device="cuda")
        s["total"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
    elif kind == "starts":
        # the middle of the list, where the units' sizes are close to their mean
        s["first"] = rng.randrange(STARTS[case["n"]] // 4, 3 * STARTS[case["n"]] // 4 + 1)
        s["first"] = min(s["first"], STARTS[case["n"]] - case["count"])
    return s


def run(s):
    case, eng = s["case"], s["eng"]
    kind = case["kind"]
    if kind == "table":
        return [eng.count(n).total for n in s["boards"]]
    if kind == "unique":
        r = [eng.count_unique(n) for n in s["boards"]]
        return [[x.unique, x.total] for x in r]
    if kind == "completions":
        return eng.count_completions(case["n"], s["queens"])
    if kind == "request":
        b = eng.batch(s["jobs"])
        try:
            return b.run(use_graph=False)
        finally:
            b.close()
    if kind == "replay":
        return s["batch"].run(use_graph=True)
    if kind == "records":
        total, solutions = eng.exec_records(case["n"], s["records"], want_solutions=True)
        return {"total": total, "solutions": solutions}
    if kind == "device":
        eng.exec_device(case["n"], s["records"].data_ptr(), s["m"], s["start_min"], s["total"].data_ptr(),
                        s["solutions"].data_ptr())
        eng.sync()
        return {"total": s["total"], "solutions": s["solutions"]}
    if kind == "noalloc":
        status = nqueens.lib().nq_exec_solutions_noalloc(
            case["n"], ctypes.c_void_p(s["records"].data_ptr()), s["m"], s["start_min"],
            ctypes.c_void_p(s["solutions"].data_ptr()), ctypes.c_void_p(s["total"].data_ptr()), None)
        if status != 0:
            raise RuntimeError("noalloc: status %d" % status)
        return {"total": s["total"], "solutions": s["solutions"]}
    return eng.count_starts(case["n"], s["first"], case["count"])


def work(case):
    """Integer operations of the search (12 a node, nodes by board and share of its task list) and the bytes of its
    inputs and outputs.  A completion query's nodes are the whole board's (8 x the symmetric search) over n per queen."""
    kind = case["kind"]
    if kind in ("table", "unique"):
        boards = range(case["lo"], case["hi"] + 1)
        return {"bytes": 16.0 * len(boards), "flops": NODE_OPS * sum(float(NODES[n]) for n in boards)}
    if kind == "completions":
        return {"bytes": 8.0 + 2 * case["k"], "flops": NODE_OPS * 8.0 * NODES[case["n"]] / case["n"] ** case["k"]}
    if kind in ("request", "replay"):
        boards = range(case["lo"], case["hi"] + 1)
        count = sum(float(NODES[n]) for n in boards) / len(boards)
        query = sum(8.0 * NODES[n] / n ** k for n in boards for k in (1, 2, 3, 4)) / (4.0 * len(boards))
        share = 1.0 if kind == "replay" else 0.4
        return {"bytes": 40.0 * case["jobs"], "flops": NODE_OPS * case["jobs"] * (share * count + (1 - share) * query)}
    if kind == "starts":
        return {"bytes": 16.0 * RECORDS[case["n"]] * case["count"] / STARTS[case["n"]],
                "flops": NODE_OPS * NODES[case["n"]] * case["count"] / STARTS[case["n"]]}
    m = min(case["m"], RECORDS[case["n"]])
    return {"bytes": 24.0 * m, "flops": NODE_OPS * NODES[case["n"]] * m / float(RECORDS[case["n"]])}


def _count_rows(n, queens):
    """Completions of the board, row by row over whole arrays of partial boards in 64-bit integers."""
    fixed = dict(queens)
    state = np.zeros((1, 3), np.int64)                 # columns, rising and falling diagonals (from row 0)
    for r, c in queens:
        state[0] |= np.array([1 << c, 1 << (r + c), 1 << (r - c + n)], np.int64)
    for r in range(n):
        if r in fixed:
            continue
        parts = []
        for c in range(n):
            q = np.array([1 << c, 1 << (r + c), 1 << (r - c + n)], np.int64)
            ok = ((state & q) == 0).all(axis=1)
            parts.append(state[ok] | q)
        state = np.concatenate(parts)
    return len(state)


def exact(case, seed):
    """A completion query's count by a plain breadth-first search over numpy arrays, on boards where that is quick."""
    if case["kind"] != "completions" or case["n"] > 12:
        return None
    return _count_rows(case["n"], prepare_queens(case, seed))


def prepare_queens(case, seed):
    return _queens(case["n"], case["k"], random.Random(seed * 7919 + 17))
