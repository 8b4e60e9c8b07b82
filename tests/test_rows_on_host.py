"""The persistent kernels' device code on the CPU (tests/host), one block, each
lane running by itself between warp-wide operations, in random order: counts
and node counts equal the oracle's whatever the order."""
import ctypes
import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "map_folding_gb300" / "csrc"


def _cut(text, begin, end):
    at = text.index(begin)
    return text[at:text.index(end, at)]


def _build(d, change=lambda name, text: text):
    """The kernels' device code as a host library; change(file, text) may edit it."""
    src = d / "pkg" / "csrc"
    src.mkdir(parents=True)
    shutil.copytree(HERE.parent / "include", d / "include")
    for f in (*CSRC.glob("*.cuh"), *CSRC.glob("*.hpp"), *CSRC.glob("*.inl")):
        text = f.read_text()
        text = re.sub(r'asm\("shl\.b(\d+).*"r"\((\w)\)\);', r"r = \2 < \1 ? decltype(r)(1) << \2 : 0;", text)
        (src / f.name).write_text(change(f.name, text))
    loop = _cut((CSRC / "dfs_kernels.cu").read_text(), "// Lunnon: levels to go",
                "template <int TPB, int LEVELS, int TMAX>\n__global__")
    (src / "persistent.inc").write_text(
        '#include "dfs_core.cuh"\n#include "tail.cuh"\nnamespace mf {\nnamespace {\n' + loop + "}\n}\n")
    wide = (CSRC / "wide_kernels.cu").read_text()
    wide = wide[:wide.index("__global__ void wide_ring_init")]
    wide = wide.replace("extern __shared__ __align__(16) uint8_t smem[];", "uint8_t *smem = host::shared;")
    (src / "wide.inc").write_text(wide + "}\n}\n")
    lib = d / "rows.so"
    shutil.copy(CSRC / "host.cpp", src / "host.cpp")  # the 9x9 edge pages
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-U_FORTIFY_SOURCE", "-w",
                    "-I", str(HERE / "host"), "-I", str(src), str(HERE / "host" / "rows.cpp"),
                    str(src / "host.cpp"), "-o", str(lib), "-pthread"], check=True)
    return ctypes.CDLL(str(lib))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("rows"))


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def _out(num):
    return np.zeros(num, np.uint64), np.zeros(1, np.uint64), np.zeros(1, np.uint64)


def _sym(host, edges, n, start, cases, seed, rows=True):
    """(counts, nodes, sum of the counts when the first warp left)"""
    cases = np.ascontiguousarray(cases)
    counts, nodes, left = _out(len(cases))
    assert host.host_sym(_ptr(edges), n, start, _ptr(cases), ctypes.c_uint64(len(cases)), int(rows),
                         seed, _ptr(counts), _ptr(nodes), _ptr(left)) == 0
    return counts, int(nodes[0]), int(left[0])


def _wide(host, edges, start, cases, seed, rows=True):
    cases = np.ascontiguousarray(cases)
    counts, nodes, left = _out(len(cases))
    assert host.host_wide(_ptr(edges), start, _ptr(cases), ctypes.c_uint64(len(cases)), int(rows),
                          seed, _ptr(counts), _ptr(nodes), _ptr(left)) == 0
    return counts, int(nodes[0]), int(left[0])


def _lunnon(host, maps, seed, rows=True):
    """maps: (dims, depth, b lists) each; (counts per map, nodes, left)."""
    meta, inst, states, owner = bytearray(), [], [], []
    for k, (dims, depth, b) in enumerate(maps):
        n = int(np.prod(dims))
        row = dims[0] if len(dims) == 2 and dims[0] >= 3 and dims[1] >= 2 and rows else 0
        inst.append((len(meta), n, len(dims), depth + 1, row))
        meta += _neighbours(dims).tobytes()
        meta += bytes(-len(meta) % 16)
        rec = np.zeros((len(b), 80), np.uint8)
        rec[:, :n + 1] = b
        states.append(rec)
        owner += [k] * len(b)
    offset = len(meta)
    meta += np.array(inst, "<u4,<i2,<i2,<i2,<i2").tobytes()
    meta += bytes(-len(meta) % 16)
    meta = np.frombuffer(bytes(meta), np.uint8)
    states, owner = np.concatenate(states), np.array(owner, np.uint32)
    counts, nodes, left = _out(len(maps))
    assert host.host_lunnon(_ptr(meta), len(meta), offset, _ptr(states), _ptr(owner), 80,
                            ctypes.c_uint64(len(states)), ctypes.c_uint64(len(maps)), int(rows), seed,
                            _ptr(counts), _ptr(nodes), _ptr(left)) == 0
    return counts, int(nodes[0]), int(left[0])


def _neighbours(dims):
    """next[i][l][m]: the leaf reached from m in dimension i, leaves 1..l placed."""
    n = int(np.prod(dims))
    out = np.zeros((len(dims), n + 1, n + 1), np.uint8)
    step = 1
    for i, d in enumerate(dims):
        c = [0] + [(m - 1) // step % d for m in range(1, n + 1)]
        for l in range(1, n + 1):
            for m in range(1, l + 1):
                if (c[l] - c[m]) % 2 == 0:
                    out[i, l, m] = m if c[m] == 0 else m - step
                else:
                    out[i, l, m] = m if c[m] == d - 1 or m + step > l else m + step
        step *= d
    return out


def _gaps(edges, c, at):
    """Positions after which cell `at` may follow, by walking the pages."""
    good = set(range(at))
    for e in edges:
        other = int(e[at])
        if other >= at:
            continue
        allowed, j = {other}, int(c[other])
        while j != other:
            j = int(e[j]) if e[j] < at else j
            allowed.add(j)
            j = int(c[j])
        good &= allowed
    return good


def _descend(edges, start, rng, back=8):
    """A list of `start` cells grown at random, going back from dead ends."""
    c = np.zeros(edges.shape[1], np.uint8)
    c[:3] = (1, 2, 0)
    path = [c]
    while 2 + len(path) < start:
        c, at = path[-1], 2 + len(path)
        good = sorted(_gaps(edges, c, at))
        if not good:
            del path[max(1, len(path) - back):]
            continue
        j = int(rng.choice(good))
        c = c.copy()
        c[at] = c[j]
        c[j] = at
        path.append(c)
    return path[-1]


def _search(edges, c, at, last):
    """(completions, nodes) below a list of `at` cells."""
    good = _gaps(edges, c, at)
    if at == last:
        return len(good), 1
    leaves, nodes = 0, 1
    for j in good:
        c[at] = c[j]
        c[j] = at
        a, b = _search(edges, c, at + 1, last)
        leaves += a
        nodes += b
        c[j] = c[at]
    return leaves, nodes


def _sym_cases(orc, n, start, count, seed):
    rng = np.random.default_rng([n, start, seed])
    edges = orc.sym_edges(n)
    return edges, np.array([_descend(edges, start, rng) for _ in range(count)])


@pytest.mark.parametrize("n,start,count", [(5, 16, 3), (5, 20, 70), (5, 22, 70), (6, 29, 70), (6, 30, 40),
                                           (7, 42, 40), (7, 44, 40), (8, 56, 33)])
@pytest.mark.parametrize("seed", [1, 2])
def test_square_rows(host, orc, n, start, count, seed):
    edges, cases = _sym_cases(orc, n, start, count, seed)
    got, nodes, _ = _sym(host, edges, n, start, cases, seed)
    _, want, w = orc.sym_count_cases(n, start, cases, None, threads=4)
    assert (got == want).all()
    assert nodes == w.nodes


# Rows of a side's length, longer than the six leaves counted, of a map's.
MAPS = [((3, 4), 5), ((5, 3), 6), ((5, 4), 12), ((6, 3), 8), ((7, 2), 5), ((7, 3), 11), ((8, 2), 6),
        ((9, 2), 8), ((10, 2), 11), ((7, 2), 9), ((8, 2), 13), ((2, 2, 3), 5), ((1, 9), 4)]


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("some", [[k] for k in range(len(MAPS))] + [list(range(0, len(MAPS), 2))])
def test_map_rows(host, orc, some, seed):
    rng = np.random.default_rng(seed)
    maps, want, nodes = [], [], 0
    for dims, depth in [MAPS[k] for k in some]:
        a, b, _ = orc.lunnon_collect(dims, depth)
        pick = np.sort(rng.permutation(len(a))[:40])
        total, _, w = orc.lunnon_resume_many(dims, depth + 1, a[pick], b[pick])
        maps.append((dims, depth, b[pick]))
        want.append(total)
        nodes += w.nodes
    got, got_nodes, _ = _lunnon(host, maps, seed)
    assert list(got) == want
    assert got_nodes == nodes


def _edges9(host):
    edges = np.zeros((4, 96), np.uint8)
    host.host_edges(9, _ptr(edges))
    return edges


@pytest.mark.parametrize("start", [70, 72, 74, 78])
def test_9x9_rows(host, start):
    edges = _edges9(host)
    rng = np.random.default_rng(start)
    cases = np.array([_descend(edges, start, rng, back=30) for _ in range(36)])
    want = [_search(edges, c.astype(int), start, 80) for c in cases]
    for rows in (True, False):
        got, nodes, _ = _wide(host, edges, start, cases, 1, rows)
        assert list(got) == [l for l, _ in want]
        assert nodes == sum(k for _, k in want)


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("kind", ["square", "map", "strip", "9x9"])
def test_warps_stay_until_shared_pieces_are_done(host, orc, kind, seed):
    """No warp goes home while a piece shared within another still runs: all is
    counted when the first one leaves."""
    if kind == "square":
        edges, cases = _sym_cases(orc, 5, 13, 1, seed)
        got, _, left = _sym(host, edges, 5, 13, cases, seed)
    elif kind == "9x9":
        edges, rng = _edges9(host), np.random.default_rng(seed)
        cases = np.array([_descend(edges, 56, rng, back=30)])
        got, _, left = _wide(host, edges, 56, cases, seed)
    else:
        dims, depth = {"map": ((5, 4), 9), "strip": ((1, 14), 5)}[kind]
        _, b, _ = orc.lunnon_collect(dims, depth)
        got, _, left = _lunnon(host, [(dims, depth, b[seed:seed + 1])], seed)
    assert left == got.sum()


def test_long_counts_go_on_in_64_bits(tmp_path, orc):
    """Where a row count's 32-bit sums might not do they are taken over in time;
    here as soon as anything has been counted, on rows of eight and nine."""
    def at_once(name, text):
        if name != "tail.cuh":
            return text
        assert text.count("kTailNodes = 1 << 21;") == 1
        return text.replace("kTailNodes = 1 << 21;", "kTailNodes = 1;")

    host = _build(tmp_path, at_once)
    test_square_rows(host, orc, 8, 54, 40, 1)
    test_square_rows(host, orc, 8, 57, 40, 2)
    test_9x9_rows(host, 70)
    test_9x9_rows(host, 74)


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("strips", [1, 6, 30])
def test_rows_beside_maps_without(host, orc, strips, seed):
    """Few and many lanes of a warp on maps that have no row: the others' rows are
    counted without them, a few roots by list."""
    maps, want, nodes = [], [], 0
    for dims, depth, most in (((1, 13), 5, strips), ((5, 4), 10, 40), ((2, 2, 3), 4, strips), ((7, 2), 6, 30)):
        a, b, _ = orc.lunnon_collect(dims, depth)
        total, _, w = orc.lunnon_resume_many(dims, depth + 1, a[:most], b[:most])
        maps.append((dims, depth, b[:most]))
        want.append(total)
        nodes += w.nodes
    got, got_nodes, left = _lunnon(host, maps, seed)
    assert list(got) == want and got_nodes == nodes
    assert left == got.sum()
