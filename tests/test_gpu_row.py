"""The last row counted on masks (tail.cuh) against the list walk: per-case
counts and node counts of the batched kernel equal the oracle's for every board
size and for cases that end before, at and inside the last row; cases that no
folding gives (permutations whose arcs cross, lists of several cycles) equal
the plain kernel, which walks."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batched(engine, torch, n, start, cycles):
    d = torch.from_numpy(np.ascontiguousarray(cycles)).cuda()
    counts = torch.zeros(len(cycles), dtype=torch.int64, device="cuda")
    nodes = torch.zeros(1, dtype=torch.int64, device="cuda")
    ws = torch.empty(engine.sym_workspace_bytes(), dtype=torch.uint8, device="cuda")
    engine.count_cases_batched_device(n, start, n * n, d.data_ptr(), len(cycles), counts.data_ptr(),
                                      ws.data_ptr(), ws.numel(), nodes.data_ptr())
    torch.cuda.synchronize()
    return counts.cpu().numpy().view(np.uint64), int(nodes.item())


def _plain(engine, torch, n, start, cycles):
    d = torch.from_numpy(np.ascontiguousarray(cycles)).cuda()
    counts = torch.zeros(len(cycles), dtype=torch.int64, device="cuda")
    nodes = torch.zeros(1, dtype=torch.int64, device="cuda")
    engine.count_cases_device(n, start, n * n, d.data_ptr(), len(cycles), counts.data_ptr(),
                              nodes.data_ptr())
    torch.cuda.synchronize()
    return counts.cpu().numpy().view(np.uint64), int(nodes.item())


def _descend(orc, n, cycle, i, stop, rng):
    """`cycle` of i cells grown to `stop` cells at random, going back a few
    cells from a dead end."""
    edges = orc.sym_edges(n).astype(int)
    path = [cycle.copy()]
    while i + len(path) - 1 < stop:
        c, at = path[-1], i + len(path) - 1
        good = set(range(at))
        for e in edges:
            other = e[at]
            if other >= at:
                continue
            allowed, j = {other}, int(c[other])
            while j != other:
                j = int(e[j]) if e[j] < at else j
                allowed.add(j)
                j = int(c[j])
            good &= allowed
        if not good:
            del path[max(1, len(path) - 6):]
            continue
        j = int(rng.choice(sorted(good)))
        c = c.copy()
        c[at] = c[j]
        c[j] = at
        path.append(c)
    return path[-1]


# Cells placed relative to the row's first cell: above it, at it, inside it.
# (Far above, a 7x7 or 8x8 case would take the oracle hours.)
OFFSETS = {5: (-10, -1, 0, 1, 3), 6: (-9, -1, 0, 1, 2, 4), 7: (-7, -1, 0, 1, 2, 5),
           8: (-3, -1, 0, 1, 2, 3, 6)}


@pytest.mark.parametrize("n,offset", [(n, o) for n, os_ in OFFSETS.items() for o in os_])
def test_cases_around_the_row_match_oracle(engine, cuda, orc, n, offset):
    start = n * n - n + offset
    rng = np.random.default_rng([n, offset + 20])
    root = np.zeros(64, np.uint8)
    root[:3] = (1, 2, 0)
    cases = np.array([_descend(orc, n, root, 3, start, rng) for _ in range(70)])  # > two warps
    got, nodes = _batched(engine, cuda, n, start, cases)
    _, want, w = orc.sym_count_cases(n, start, cases, None, threads=os.cpu_count() or 4)
    assert (got == want).all()
    assert nodes == w.nodes


@pytest.mark.parametrize("n", [5, 6, 7])
def test_cases_that_are_no_foldings(engine, cuda, n):
    """Any permutation of the placed cells is counted as get_good walks it."""
    rng = np.random.default_rng(n)
    start = n * n - n - 2
    cases = np.zeros((64, 64), np.uint8)
    for k in range(64):
        p = rng.permutation(start)
        if k % 2:  # one cycle in random order, its arcs crossing
            cases[k, p] = np.roll(p, 1)
        else:      # several cycles
            cases[k, :start] = p
    got, nodes = _batched(engine, cuda, n, start, cases)
    want, want_nodes = _plain(engine, cuda, n, start, cases)
    assert (got == want).all()
    assert nodes == want_nodes


@pytest.mark.parametrize("n,start", [(5, 21), (7, 44), (8, 58)])
@pytest.mark.parametrize("num", [1, 31, 1519, 1521, 12000, 48641])
def test_many_shallow_units(engine, cuda, orc, n, start, num):
    """Units that end a few cells further, at the numbers where their spreading
    over the warps changes."""
    rng = np.random.default_rng([n, start])
    root = np.zeros(64, np.uint8)
    root[:3] = (1, 2, 0)
    some = np.array([_descend(orc, n, root, 3, start, rng) for _ in range(37)])
    got, nodes = _batched(engine, cuda, n, start, some[np.arange(num) % 37])
    want, want_nodes = _plain(engine, cuda, n, start, some[np.arange(num) % 37])
    assert (got == want).all()
    assert nodes == want_nodes
    _, first, _ = orc.sym_count_cases(n, start, some, None, threads=4)
    assert (got[:37] == first[:num]).all()


@pytest.mark.parametrize("n,start", [(5, 19), (7, 43)])
@pytest.mark.parametrize("levels", [1, 3, 4, 6])
@pytest.mark.parametrize("num", [1, 33, 1521, 20000])
def test_plain_units_of_a_few_levels(engine, cuda, orc, n, start, levels, num):
    """Where the plain kernel begins to share, and how it spreads such units."""
    rng = np.random.default_rng([n, start, levels])
    root = np.zeros(64, np.uint8)
    root[:3] = (1, 2, 0)
    some = np.array([_descend(orc, n, root, 3, start, rng) for _ in range(37)])
    want = np.array([orc.sym_count_to(n, c, start, start + levels)[0] for c in some], np.uint64)
    d = cuda.from_numpy(np.ascontiguousarray(some[np.arange(num) % 37])).cuda()
    counts = cuda.full((num,), 7, dtype=cuda.int64, device="cuda")
    engine.count_cases_device(n, start, start + levels, d.data_ptr(), num, counts.data_ptr())
    cuda.cuda.synchronize()
    assert (counts.cpu().numpy().view(np.uint64) == want[np.arange(num) % 37]).all()
