"""X-scores below the 32-bit range (an X-drop cutoff near it, a high error cost and a long mismatching
tail): the tail's slices do not come back as good ones, so the extension ends where a cutoff that is
reached in range ends it too, which is the oracle's answer.  (Where single columns of a slice lie on
both sides of the range the reference's own int arithmetic overflows: such reads are not among these.)"""
import random

import numpy as np
import pytest

from graphaligner_gb300 import graph as gg
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, pack_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def workload():
    rng = random.Random(5)
    segs = ["".join(rng.choice("ACGT") for _ in range(rng.randint(50, 150))) for _ in range(30)]
    gfa = "".join(f"S\t{i + 1}\t{s}\n" for i, s in enumerate(segs)) + "".join(f"L\t{i + 1}\t+\t{(i + 1) % 30 + 1}\t+\t0M\n" for i in range(30))
    path = "".join(segs)
    reads = [(path[1:1 + n] + "".join(rng.choice("ACGT") for _ in range(tail))).encode()
             for n, tail in ((300, 1000), (300, 70_000), (1000, 90_000), (64, 100_000), (500, 120_000))]
    return gg.build_from_gfa(gfa), reads


@pytest.mark.parametrize("cost,which", [(10_000, [0, 1, 2, 3, 4]), (50_000, [0, 1, 3, 4]), (65_535, [0, 1, 2, 3])])
def test_tails_out_of_range(cuda_lib, oracle_lib, workload, cost, which):
    g, reads = workload
    batch = pack_batch(g, [reads[k] for k in which], [2] * len(which), [0] * len(which))
    ext = Extender(DeviceGraph(g), arena_bytes=256 << 20)
    got = ext.run(ExtendParams(bandwidth=10, xdrop=2**31 - 1, xscore_error_cost=cost), batch)
    want = oracle_lib.extend(g, ExtendParams(bandwidth=10, xdrop=2**30, xscore_error_cost=cost), batch, threads=4)
    assert np.all(want.status == 0)
    assert np.array_equal(got.status, want.status) and np.array_equal(got.score, want.score)
    for i in range(batch.num):
        assert np.array_equal(got.items(i), want.items(i)), f"trace {i}"
    ext.close()
