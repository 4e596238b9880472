"""k-mer lookups of reads with runs of one base that reach over many of the kernel's rounds of 1,024
positions: the same lookups as the rules give, in time linear in the run's length."""
import os
import sys
import time

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from test_seed_lookup_gpu import lookups  # noqa: E402

from graphaligner_gb300 import graph as gg  # noqa: E402
from graphaligner_gb300.align import Aligner, preset  # noqa: E402
from graphaligner_gb300.extend import DeviceGraph, Extender  # noqa: E402

pytestmark = pytest.mark.gpu


def aligner(k, w):
    rng = np.random.default_rng(12)
    rand = lambda n: "".join("ACGT"[c] for c in rng.integers(0, 4, n))  # noqa: E731
    nodes = [rand(90) + b * 40 + rand(60) for b in "ACGT"] + [rand(200) for _ in range(8)]
    gfa = "".join(f"S\t{i + 1}\t{s}\n" for i, s in enumerate(nodes)) + "".join(f"L\t{i + 1}\t+\t{i + 2}\t+\t0M\n" for i in range(len(nodes) - 1))
    g = gg.build_from_gfa(gfa)
    p = preset("vg")
    p.minimizer_length, p.minimizer_window, p.minimizer_discard_fraction, p.minimizer_density = k, w, 0.0, 1e6
    return nodes, Aligner(Extender(DeviceGraph(g), arena_bytes=64 << 20), g, p)


@pytest.mark.parametrize("k,w", [(15, 20), (31, 94), (5, 40)])
def test_runs_over_many_rounds(cuda_lib, k, w):
    nodes, a = aligner(k, w)
    fill = "".join(nodes[4:])
    reads = []
    for lead in (0, 1, 127, 900, 1023, 1024, 1025):
        for run in (1024, 2047, 2048, 2049, 5000, 9217):
            b = "ACGT"[(lead + run) % 4]
            # one run, and two that meet with nothing, an N or a base of the other case between them
            reads.append(fill[:lead] + b * run + nodes[0])
            reads.append(fill[:lead] + b * run + ("N", b.lower(), "")[run % 3] + b * 1500 + nodes[1])
    info, keys, start, pos = a.index(arrays=True)
    place = {int(x): i for i, x in enumerate(keys)}
    for i, (read, seeds) in enumerate(zip(reads, a.seeds([r.encode() for r in reads]))):
        want = []
        for at, kmer in lookups(read, k, w):
            j = place.get(kmer)
            if j is None or int(start[j + 1] - start[j]) >= info["max_count"]:
                continue
            want += [(at, int(x) >> 6, int(x) & 63) for x in pos[int(start[j]):int(start[j + 1])]]
        assert sorted((s[2], s[5], s[6]) for s in seeds) == sorted(want), f"read {i}"


def test_time_is_linear_in_the_run(cuda_lib):
    # no k-mer of the run is looked up often or found often: a window of many bases, and an index whose
    # longest run is 40
    _, a = aligner(31, 94)

    def best_ms(n):
        read = [b"A" * n]
        a.seeds(read)
        times = []
        for _ in range(3):
            t = time.perf_counter()
            a.seeds(read)
            times.append((time.perf_counter() - t) * 1e3)
        return min(times)
    # eight times the length: 8 times the time at most where it is linear, up to 64 where every segment
    # walks back to the run's beginning; halfway between them on a scale of factors
    assert best_ms(1 << 20) < 8 * 8 ** 0.5 * best_ms(1 << 17)
