"""k-mer lookups of reads by segments (seed_kernel.cu), against iterateKmers' rules
(MinimizerSeeder.cpp:59-102) restated here over the index's own arrays: homopolymers and non-ACGT
bases across the segments' and steps' edges, reads shorter than a k-mer and of several rounds."""
import numpy as np
import pytest

from graphaligner_gb300 import graph as gg
from graphaligner_gb300.align import Aligner, preset
from graphaligner_gb300.extend import DeviceGraph, Extender

pytestmark = pytest.mark.gpu

CODE = {c: k for k, c in enumerate("ACGT")} | {c: k for k, c in enumerate("acgt")}


def lookups(seq: str, k: int, w: int):
    """(position, k-mer) of every k-mer the reference looks up."""
    window = w - k + 1
    out, run, kmer, last = [], 0, 0, None
    for p, c in enumerate(seq):
        if c not in CODE:
            run = 0
            continue
        kmer = ((kmer << 2) | CODE[c]) & ((1 << (2 * k)) - 1)
        run += 1
        if run < k:
            continue
        if run == k or kmer != last[1] or p < window or p - last[0] >= window:
            last = (p, kmer)
            out.append(last)
    return out


@pytest.fixture(scope="module")
def workload():
    rng = np.random.default_rng(4)
    rand = lambda n: "".join("ACGT"[c] for c in rng.integers(0, 4, n))  # noqa: E731
    nodes = [rand(90) + b * 40 + rand(60) for b in "ACGT"] + [rand(200) for _ in range(40)]
    gfa = "".join(f"S\t{i + 1}\t{s}\n" for i, s in enumerate(nodes)) + "".join(f"L\t{i + 1}\t+\t{i + 2}\t+\t0M\n" for i in range(len(nodes) - 1))
    g = gg.build_from_gfa(gfa)
    reads = ["A", rand(14), nodes[5][:15], nodes[5][:20], "N" * 40]
    for run in (15, 16, 20, 21, 22, 31, 32, 33, 100, 127, 128, 129, 160, 255, 300, 1024, 1200):
        for lead in (0, 1, 97, 127):
            b = "ACGT"[run % 4]
            reads.append((nodes[6] + nodes[7])[:lead] + b * run + nodes[0][:150] + "N" + nodes[8])
    for n in (126, 127, 128, 129, 1023, 1024, 1025, 3000):
        r = "".join(nodes)[:n]
        reads.append(r)
        at = rng.integers(0, n, 6)
        reads.append("".join("Nn-RacgA"[int(rng.integers(0, 8))] if p in at else c for p, c in enumerate(r)))
    return g, [r.encode() for r in reads]


@pytest.mark.parametrize("k,w", [(15, 20), (15, 15), (19, 30), (31, 31), (31, 94), (5, 40)])
def test_lookups_match_the_rules(cuda_lib, workload, k, w):
    g, reads = workload
    p = preset("vg")
    p.minimizer_length, p.minimizer_window, p.minimizer_discard_fraction, p.minimizer_density = k, w, 0.0, 1e6
    a = Aligner(Extender(DeviceGraph(g), arena_bytes=64 << 20), g, p)
    info, keys, start, pos = a.index(arrays=True)
    place = {int(x): i for i, x in enumerate(keys)}
    for i, (read, seeds) in enumerate(zip(reads, a.seeds(reads))):
        want = []
        for at, kmer in lookups(read.decode(), k, w):
            j = place.get(kmer)
            if j is None or int(start[j + 1] - start[j]) >= info["max_count"]:
                continue
            want += [(at, int(x) >> 6, int(x) & 63) for x in pos[int(start[j]):int(start[j + 1])]]
        assert sorted((s[2], s[5], s[6]) for s in seeds) == sorted(want), f"read {i}"
