"""Rows that the row count meets less often: maps whose rows are longer than the
six leaves counted (they begin inside the row), in the batched kernel and in the
request server, whose rows go up to eight; searches that begin above, at and
inside the row; nodes as well as counts, against the oracle.  Server nodes of
square chunks equal the batched kernel's; 8x8 cases that are no foldings are
counted as the oracle walks them."""
import os

import numpy as np
import pytest

from test_gpu_row import _batched, _descend

pytestmark = pytest.mark.gpu

MAPS = [((7, 2), 4), ((7, 2), 7), ((7, 2), 9), ((7, 3), 11), ((7, 3), 15), ((8, 2), 6), ((8, 2), 9),
        ((8, 2), 12), ((9, 2), 8), ((10, 2), 9), ((10, 2), 15), ((6, 3), 10), ((4, 5), 12)]


def _oracle(orc, dims, depth):
    a, b, _ = orc.lunnon_collect(dims, depth)
    total, _, w = orc.lunnon_resume_many(dims, depth + 1, a, b, threads=os.cpu_count() or 4)
    return total, w.nodes


@pytest.mark.parametrize("dims,depth", MAPS)
def test_long_rows_batched(engine, cuda, orc, dims, depth):
    plan = engine.LunnonPlan(dims)
    total, _, st = plan.count_range(depth)
    plan.close()
    assert (total, int(st.nodes)) == _oracle(orc, dims, depth)


def test_long_rows_served(engine, cuda, orc):
    from map_folding_gb300.serving import Server

    with Server() as server:
        ids = [server.submit_lunnon(dims, depth) for dims, depth in MAPS]
        chunk = server.submit_sym(6, 16, 100, 300)
        got = [server.wait(rid) for rid in ids]
        answer, info = server.wait(chunk)
    for (dims, depth), (total, i) in zip(MAPS, got):
        assert (total, int(i.nodes)) == _oracle(orc, dims, depth), (dims, depth)
    plan = engine.SymPlan(6, 16)
    want, st = plan.solve(300, 100)
    plan.close()
    assert (answer, int(info.nodes)) == (want, int(st.nodes))


@pytest.mark.parametrize("offset", [-1, 0])
def test_8x8_cases_that_are_no_foldings(engine, cuda, orc, offset):
    """Foldings with two neighbours swapped (arcs that cross) or cut into two
    cycles; other lists of so many cells have searches of hours."""
    rng = np.random.default_rng(80 + offset)
    start = 56 + offset
    root = np.zeros(64, np.uint8)
    root[:3] = (1, 2, 0)
    cases = np.array([_descend(orc, 8, root, 3, start, rng) for _ in range(64)])
    for k, c in enumerate(cases):
        a = int(rng.integers(0, start))
        if k % 3 == 0:
            b, d = int(c[a]), int(c[c[a]])
            c[a], c[d], c[b] = d, b, c[d]
        elif k % 3 == 1:
            b = int(rng.integers(0, start))
            c[a], c[b] = c[b], c[a]
    got, nodes = _batched(engine, cuda, 8, start, cases)
    _, want, w = orc.sym_count_cases(8, start, cases, None, threads=os.cpu_count() or 4)
    assert (got == want).all()
    assert nodes == w.nodes
