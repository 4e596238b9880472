"""The seed-start column of the multiseed DP (a row per lane, twice): reads that end at every kind of row
of their last slice, at several X-score error costs, trace for trace against the oracle."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from golden_sets import load_graph  # noqa: E402
from test_multiseed_gpu import multiseed_seeds, read_fasta  # noqa: E402
from test_read_pipeline_host import harness  # noqa: E402,F401  (the host read-level harness)

pytestmark = pytest.mark.gpu

ENDS = [1, 2, 31, 32, 33, 34, 63, 64]


# below 100 some rows score two more than the row before, which a column cannot hold: the oracle
# asserts in every such read, the GPU's fill only where a check meets the row
TWO_A_ROW = pytest.param(99, marks=pytest.mark.xfail(strict=True, reason="the oracle asserts in reads whose statuses here are OK"))


@pytest.mark.parametrize("cost", [1, TWO_A_ROW, 100, 101, 333, 1700])
def test_seed_columns_at_read_ends(cuda_lib, oracle_lib, harness, tmp_path, cost):  # noqa: F811
    from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, MultiseedBatch
    g = load_graph("vg50k")
    _, seqs = read_fasta("vg50k_reads")
    seeds = multiseed_seeds(harness[0], "vg50k", "vg50k_reads", False, tmp_path)
    cut, kept = [], []
    for i, (s, sd) in enumerate(zip(seqs, seeds)):
        if not sd:
            continue
        # the read ends in the slice of its second seed (or of its only one)
        last = sorted(x[0] for x in sd)[min(1, len(sd) - 1)]
        end = min(len(s), 64 * last + ENDS[i % len(ENDS)])
        cut.append(s[:end])
        kept.append([x for x in sd if 64 * x[0] < end])
    batch = MultiseedBatch.pack(cut, kept, max_traces=256, items_per_bp=64)
    p = ExtendParams(bandwidth=10, xscore_error_cost=cost)
    gpu = Extender(DeviceGraph(g)).multiseed(p, batch)
    cpu = oracle_lib.multiseed(g, p, batch, threads=8)
    assert np.array_equal(gpu.status, cpu.status)
    assert np.array_equal(gpu.num_traces, cpu.num_traces)
    for i in range(batch.num):
        for (gs, gi), (cs, ci) in zip(gpu.traces(i), cpu.traces(i)):
            assert gs == cs and np.array_equal(gi, ci), f"read {i}"
