"""The counts that programs ask this framework for, as timed cases.

Each case goes through the package's public entry points and returns what the
entry point returns (partial counts, per-unit counts, node counts).  Kinds:

  range    LunnonPlan.count_range: a range of one map's prefix states, host
           buffers, persistent kernel (what `gpu_folding` and `gpu_folding_v2`
           run; a job split over several processes counts a range each)
  states   LunnonPlan.count_states_device: one thread per prefix state, on
           prefix states that are on the GPU already
  batch    LunnonBatch.run: many uneven maps in one recorded launch
  chunk    SymPlan.solve: consecutive cases of an n x n square, the unit that
           sweeps and volunteers hand out (`sym_fold n threads max start`)
  cases    count_cases_batched_device: per-case counts of cases on the GPU
  depth    count_cases_device: how many cells-deep continuations each case
           has, one thread per case (the lookahead that scores cases)
  costs    SymPlan.block_costs: that score per block of a case range, from
           which cost-weighted chunks are cut
  unit     solve_cases: one volunteer work unit (the WASM kernel's contract)
  serve    a request server: opened, given square chunks and whole maps at
           once, drained, closed
"""
from __future__ import annotations

import functools
import random

import numpy as np
import torch

import map_folding_gb300 as mf
from map_folding_gb300.serving import Server
from map_folding_gb300.workloads import uneven_instances


def listed():
    return [
        # The smallest call: a few dozen prefix states of a 3x4 map; launch,
        # copies and host work are all there is.
        {"name": "range_3x4", "kind": "range", "dims": "3x4", "depth": 9, "states": 41},
        # A 1-D strip: no row above, every leaf held by the one before it.
        {"name": "range_1x16", "kind": "range", "dims": "1x16", "depth": 10, "states": 701},
        # The 5x5 map at the depth gpu_folding is quoted at.
        {"name": "range_5x5", "kind": "range", "dims": "5x5", "depth": 15, "states": 12000},
        # Half of the 6x6 map at depth 18: the largest map of the tables.
        {"name": "range_6x6", "kind": "range", "dims": "6x6", "depth": 18, "states": 56001},
        # The plain kernel on the 5x5 map's states, per-state counts.
        {"name": "states_5x5", "kind": "states", "dims": "5x5", "depth": 15, "states": 8191},
        # 64 maps of uneven shape in one launch.
        {"name": "batch_64", "kind": "batch", "maps": 64},
        # A 7x7 chunk: 5,000 of the full count's 433,131 cases.
        {"name": "chunk_7x7", "kind": "chunk", "n": 7, "expanded": 24, "cases": 5000},
        # 8x8 at the sweep's depth: a slice of a 50,000-case chunk.
        {"name": "chunk_8x8", "kind": "chunk", "n": 8, "expanded": 36, "cases": 2000},
        # 9x9: 128-bit masks.
        {"name": "chunk_9x9", "kind": "chunk", "n": 9, "expanded": 48, "cases": 300},
        # Per-case counts of cases drawn from the whole 7x7 list, on the GPU.
        {"name": "cases_7x7", "kind": "cases", "n": 7, "expanded": 24, "cases": 3001},
        # Lookahead scores of an 8x8 case range, per block of 1,000.
        {"name": "costs_8x8", "kind": "costs", "n": 8, "expanded": 36, "cases": 100000, "depth": 6,
         "block": 1000},
        # A volunteer's unit: 64 prefixes of 14 cells, counted to 28.
        {"name": "unit_7x7", "kind": "unit", "n": 7, "expanded": 14, "cases": 64, "stop": 28},
    ]


def draw(rng: random.Random):
    def spread(lo, hi):
        return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))

    kind = rng.choice(["range", "range", "states", "batch", "chunk", "chunk", "chunk", "cases",
                       "depth", "costs", "unit", "serve"])
    if kind == "range":
        dims, depth, most = rng.choice([
            ("2x5", 7, 25), ("3x3", 7, 50), ("3x4", 9, 130), ("2x8", 11, 600), ("4x4", 11, 800),
            ("1x12", 8, 130), ("1x18", 11, 3000), ("2x2x4", 11, 170), ("4x5", 13, 5000),
            ("5x5", 14, 7000), ("5x6", 16, 20000), ("6x5", 15, 12000), ("6x6", 18, 56000)])
        return {"kind": kind, "dims": dims, "depth": depth, "states": spread(max(8, most // 16), most)}
    if kind == "states":
        dims, depth, most = rng.choice([("4x5", 13, 5000), ("5x5", 15, 12000), ("2x2x5", 15, 1600)])
        return {"kind": kind, "dims": dims, "depth": depth, "states": spread(most // 16, most)}
    if kind == "batch":
        return {"kind": kind, "maps": spread(4, 96)}
    if kind == "chunk":
        n, expanded, most = rng.choice([(6, 16, 1200), (7, 24, 5000), (7, 28, 20000),
                                        (7, 37, 100000), (8, 36, 2000), (8, 40, 10000),
                                        (9, 48, 300), (9, 52, 2000)])
        return {"kind": kind, "n": n, "expanded": expanded, "cases": spread(max(1, most // 64), most)}
    if kind == "cases":
        n, expanded, most = rng.choice([(6, 16, 1225), (7, 24, 3000), (8, 36, 1000)])
        return {"kind": kind, "n": n, "expanded": expanded, "cases": spread(most // 16, most)}
    if kind == "depth":
        n, expanded, most = rng.choice([(7, 24, 100000), (8, 24, 100000)])
        return {"kind": kind, "n": n, "expanded": expanded, "cases": spread(256, most),
                "stop": expanded + rng.randint(3, 6)}
    if kind == "costs":
        return {"kind": kind, "n": 8, "expanded": 36, "cases": spread(3000, 100000),
                "depth": rng.randint(3, 6), "block": rng.choice([100, 1000])}
    if kind == "unit":
        n, expanded = rng.choice([(6, 16), (7, 14)])
        return {"kind": kind, "n": n, "expanded": expanded, "cases": spread(8, 256),
                "stop": min(n * n, expanded + rng.randint(9, 14))}
    return {"kind": "serve", "n": 6, "requests": spread(2, 12), "cases": spread(40, 1000)}


def _dims(case):
    return tuple(int(d) for d in case["dims"].split("x"))


@functools.lru_cache(maxsize=None)
def _sym_plan(n, expanded):
    """A program that counts chunks keeps its plan for all of them."""
    return mf.SymPlan(n, expanded)


def _some_cases(plan, count, rng):
    """`count` cases from all over the plan's list: 16 runs of neighbours."""
    runs = min(16, count)
    got = []
    for k in range(runs):
        m = count // runs + (k < count % runs)
        m = min(m, plan.total_cases)
        got.append(plan.cases(int(rng.integers(0, plan.total_cases - m + 1)), m)[0])
    return np.concatenate(got)[:count]


def prepare(case, seed):
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("range", "states"):
        plan = mf.LunnonPlan(_dims(case))
        depth = case["depth"]
        total = plan.count_prefixes(depth)
        count = min(case["states"], max(1, total * 9 // 10))
        s |= {"plan": plan, "depth": depth, "count": count,
              "first": int(rng.integers(0, total - count + 1))}
        if kind == "states":
            pick = np.sort(rng.choice(total, count, replace=False))
            s["states"] = torch.from_numpy(np.ascontiguousarray(plan.collect(depth)[pick])).cuda()
    elif kind == "batch":
        s["batch"] = mf.LunnonBatch(uneven_instances(seed, case["maps"]))
    elif kind in ("chunk", "costs"):
        plan = _sym_plan(case["n"], case["expanded"])
        count = min(case["cases"], plan.total_cases)
        s |= {"plan": plan, "count": count,
              "first": int(rng.integers(0, plan.total_cases - count + 1))}
        if kind == "costs":
            s |= {"depth": case["depth"], "block": case["block"]}
    elif kind == "serve":
        plan = _sym_plan(case["n"], 0)
        maps = [d for d in uneven_instances(seed, 8 * case["requests"]) if np.prod(d) <= 25]
        s |= {"n": case["n"], "count": case["cases"], "requests": case["requests"], "maps": maps,
              "starts": rng.integers(0, plan.total_cases - case["cases"] + 1, case["requests"])}
    else:
        plan = _sym_plan(case["n"], case["expanded"])
        count = min(case["cases"], plan.total_cases)
        cycles = _some_cases(plan, count, rng)
        s |= {"n": case["n"], "start": plan.start_i, "stop": case.get("stop", case["n"] ** 2),
              "count": count}
        if kind == "unit":
            s["buffer"] = mf.pack_case_buffer(cycles, [1 + k % 16 for k in range(count)], case["n"])
        else:
            s["cycles"] = torch.from_numpy(cycles).cuda()
    return s


def _words(value):
    """A count of up to 128 bits as four 32-bit words, low word first."""
    return [(value >> (32 * k)) & 0xFFFFFFFF for k in range(4)]


def run(s):
    kind = s["kind"]
    if kind == "range":
        total, states, st = s["plan"].count_range(s["depth"], s["first"], s["count"])
        return {"count": _words(total), "states": states, "nodes": int(st.nodes)}
    if kind == "states":
        per_state = torch.empty(s["count"], dtype=torch.int64, device="cuda")
        total = torch.zeros(1, dtype=torch.int64, device="cuda")
        s["plan"].count_states_device(s["depth"] + 1, s["states"].data_ptr(), s["count"],
                                      per_state.data_ptr(), total.data_ptr(),
                                      stream=torch.cuda.current_stream().cuda_stream)
        return {"per_state": per_state, "total": total}
    if kind == "batch":
        counts, st = s["batch"].run()
        return {"counts": np.array(counts, np.int64), "nodes": int(st.nodes)}
    if kind == "chunk":
        answer, st = s["plan"].solve(s["count"], s["first"])
        return {"answer": _words(answer), "nodes": int(st.nodes)}
    if kind == "costs":
        return {"costs": s["plan"].block_costs(s["first"], s["count"], s["depth"], s["block"])}
    if kind == "unit":
        count, nodes, status = mf.solve_cases(s["n"], s["start"], s["stop"], s["buffer"], s["count"])
        return {"count": _words(count), "nodes": nodes, "status": status}
    if kind == "serve":
        with Server() as server:
            ids = []
            for k in range(s["requests"]):
                ids.append(server.submit_sym(s["n"], 0, int(s["starts"][k]), s["count"]))
                if s["maps"]:
                    ids.append(server.submit_lunnon(s["maps"][k % len(s["maps"])]))
            answers = [server.wait(rid) for rid in ids]
        return {"answers": [w for a, _ in answers for w in _words(a)][:4 * 15],
                "nodes": sum(int(info.nodes) for _, info in answers)}
    stream = torch.cuda.current_stream().cuda_stream
    counts = torch.empty(s["count"], dtype=torch.int64, device="cuda")
    if kind == "depth":
        mf.count_cases_device(s["n"], s["start"], s["stop"], s["cycles"].data_ptr(), s["count"],
                              counts.data_ptr(), stream=stream)
        return {"counts": counts}
    nodes = torch.zeros(1, dtype=torch.int64, device="cuda")
    if "workspace" not in s:
        s["workspace"] = torch.empty(mf.sym_workspace_bytes(), dtype=torch.uint8, device="cuda")
    mf.count_cases_batched_device(s["n"], s["start"], s["stop"], s["cycles"].data_ptr(), s["count"],
                                  counts.data_ptr(), s["workspace"].data_ptr(),
                                  s["workspace"].numel(), nodes.data_ptr(), stream=stream)
    return {"counts": counts, "nodes": nodes}


#: Search nodes below one unit (a case or a prefix state), on average over
#: strided samples: what a search that enumerates has to visit.
_NODES = {("chunk", 6): 5.7e5, ("chunk", 7): 1.3e6, ("chunk", 8): 3e6, ("chunk", 9): 6e6}


def work(case):
    kind = case["kind"]
    if kind in ("range", "states"):
        leaves = int(np.prod(_dims(case)))
        below = 2.2 ** (leaves - case["depth"] - 1) if leaves < 30 else 1e5
        return {"bytes": case["states"] * (leaves + 1 + (8 if kind == "states" else 0)) + 16,
                "flops": case["states"] * below}
    if kind == "batch":
        return {"bytes": case["maps"] * 8 * 1024, "flops": case["maps"] * 2e7}
    n, cases = case["n"], case["cases"]
    record = n * n + 8
    if kind in ("chunk", "cases"):
        shallower = case["expanded"] - {6: 16, 7: 24, 8: 36, 9: 48}[n]
        below = max(10.0, _NODES[("chunk", n)] / 1.7 ** shallower)
        return {"bytes": cases * record, "flops": cases * below}
    if kind == "serve":
        return {"bytes": case["requests"] * cases * record,
                "flops": case["requests"] * cases * _NODES[("chunk", 6)]}
    steps = case["depth"] if kind == "costs" else case["stop"] - case["expanded"]
    return {"bytes": cases * record, "flops": cases * 1.7 ** steps}


def _lunnon_reference(dims, depth, first, count):
    """Lunnon's search in plain Python: the count below prefix states
    [first, first + count) at `depth` leaves, and the insertions made."""
    n, radix = int(np.prod(dims)), [1]
    for d in dims:
        radix.append(radix[-1] * d)
    coord = [[(m - 1) // radix[i] % d if m else 0 for m in range(n + 1)] for i, d in enumerate(dims)]

    def step(i, leaf, m):
        if m == 0:
            return 0
        if (coord[i][leaf] - coord[i][m]) % 2 == 0:
            return m if coord[i][m] == 0 else m - radix[i]
        return m if coord[i][m] == dims[i] - 1 or m + radix[i] > leaf else m + radix[i]

    below = [0] * (n + 1)

    def gaps(leaf):
        hits, order, held = {}, [], 0
        for i in range(len(dims)):
            m = step(i, leaf, leaf)
            if m == leaf:
                continue
            held += 1
            while m != leaf:
                if m not in hits:
                    hits[m] = 0
                    order.append(m)
                hits[m] += 1
                m = step(i, leaf, below[m])
        return [m for m in order if hits[m] == held] if held else list(range(leaf))

    seen = total = nodes = 0

    def search(leaf, counting):
        nonlocal seen, total, nodes
        if leaf >= 2 and below[0] != 1:
            return
        if leaf == depth + 1 and not counting:
            seen += 1
            if not first < seen <= first + count:
                return
            counting = True
        if leaf > n:
            total += n
            return
        for m in reversed(gaps(leaf)):
            nodes += counting
            below[leaf] = below[m]
            below[m] = leaf
            search(leaf + 1, counting)
            below[m] = below[leaf]

    search(1, False)
    return total, nodes


def exact(case, seed):
    """The small ranges, from a plain search; counts are whole numbers, so the
    larger cases are held to equality alone."""
    if case["kind"] != "range" or int(np.prod(_dims(case))) > 12:
        return None
    s = prepare(case, seed)
    total, nodes = _lunnon_reference(_dims(case), s["depth"], s["first"], s["count"])
    return {"count": _words(total), "states": s["count"], "nodes": nodes}
