"""GAF lines written by a warp each, at the edges of its 32-wide steps: runs of edit ops that end
on, before and after a step's edge, run lengths of one to five digits, paths of 1 to 70 entries
with named and unnamed nodes of either strand, in one batch and alone."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_gaf_device_gpu import gaf_call  # noqa: E402

pytestmark = pytest.mark.gpu

CODE = "=XID"


@pytest.fixture(scope="module")
def aligner():
    from graphaligner_gb300 import graph as gg
    from graphaligner_gb300.align import Aligner, preset
    from graphaligner_gb300.extend import DeviceGraph, Extender
    rng = np.random.default_rng(3)
    names = [str(k + 1) if k % 3 == 0 else ("n" * (1 + k % 40) + str(k)) for k in range(70)]
    seqs = ["".join("ACGT"[c] for c in rng.integers(0, 4, 25_000 if k == 0 else 40)) for k in range(70)]
    gfa = "".join(f"S\t{n}\t{s}\n" for n, s in zip(names, seqs)) + "".join(f"L\t{a}\t+\t{b}\t+\t0M\n" for a, b in zip(names, names[1:]))
    g = gg.build_from_gfa(gfa)
    yield g, Aligner(Extender(DeviceGraph(g), arena_bytes=64 << 20), g, preset("vg"))


def label(g, bignode):
    i = {int(x): k for k, x in enumerate(g.lookup_ids)}[bignode]
    return g.names[i] or str(bignode // 2)


def line_of(ops, node, first_offset=0):
    """Items of one node whose edit ops are `ops` (the first is a match or mismatch)."""
    items, off, seq = [], first_offset, 0
    for k, op in enumerate(ops):
        if k:
            if op == "D":
                off += 1
            elif op == "I":
                seq += 1
            else:
                off += 1
                seq += 1
        items.append((node, off, seq, 0, ord("C") if op == "X" else ord("A"), ord("A"), 0))
    return items


def cigar(ops):
    out, k = "", 0
    while k < len(ops):
        j = k
        while j < len(ops) and ops[j] == ops[k]:
            j += 1
        out += f"{j - k}{ops[k]}"
        k = j
    return out


RUNS = [[1], [31], [32], [33], [64], [1, 1, 1], [31, 1], [31, 2, 31], [32, 32], [33, 31, 1], [9, 10, 99, 100, 101], [999, 1, 1000], [9999, 10_000],
        [1] * 200, [2, 1] * 60]


def test_cigar_runs(cuda_lib, aligner):
    g, a = aligner
    node = int(g.lookup_ids[np.argmax(g.original_size)])
    items, lines, want, lens = [], [], [], []
    for r, runs in enumerate(RUNS):
        ops = "".join(CODE[k % 4] * n for k, n in enumerate(runs))
        it = line_of(ops, node)
        lines.append((len(items), len(it), r, 1234, 60))
        items += it
        lens.append(it[-1][2] + 1)
        want.append(cigar(ops))
    names = ["read" * (k % 20) + str(k) for k in range(len(RUNS))]
    body, ends, failed = gaf_call(a, lines, items, names, lens)
    out = body.split("\n")
    assert failed == [0] * len(RUNS) and ends[-1] == len(body)
    for k in range(len(RUNS)):
        f = out[k].split("\t")
        assert f[0] == names[k] and f[1] == str(lens[k]) and f[-1] == "cg:Z:" + want[k], k
        n = len(line_of("".join(CODE[q % 4] * c for q, c in enumerate(RUNS[k])), node))
        assert f[10] == str(n) and f[13] == "AS:f:12.34"
        alone, _, _ = gaf_call(a, [(0, lines[k][1], 0, 1234, 60)], items[lines[k][0]:lines[k][0] + lines[k][1]], [names[k]], [lens[k]])
        assert alone == out[k] + "\n"


@pytest.mark.parametrize("entries", [1, 2, 31, 32, 33, 64, 65, 70])
def test_node_paths(cuda_lib, aligner, entries):
    g, a = aligner
    ids = sorted(int(x) for x in g.lookup_ids)
    rng = np.random.default_rng(entries)
    path = [ids[int(k)] for k in rng.integers(0, len(ids), entries)]
    path = [p for k, p in enumerate(path) if k == 0 or p != path[k - 1]]
    items = []
    for k, p in enumerate(path):
        items.append((p, 0, k, 1, ord("A"), ord("A"), 0))
    body, _, failed = gaf_call(a, [(0, len(items), 0, -100, 0)], items, ["r"], [len(items)])
    assert failed == [0]
    f = body.rstrip("\n").split("\t")
    assert f[5] == "".join(("<" if p % 2 else ">") + label(g, p) for p in path)
    assert f[-1] == f"cg:Z:{len(items)}=" and not any(x.startswith("AS:f") for x in f)
