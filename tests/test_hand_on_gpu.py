"""Extensions that all outgrow the small tables, around the most that one call hands on to the second
fill (8,192; the ones above it start again in the next layout), and batches on both sides of the line
up to which a graph that is mostly cycles starts with the medium tables."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from golden_sets import MAX_CELLS, digest, load_digests, load_graph, load_requests  # noqa: E402
from test_extension_degrees_gpu import bubbles  # noqa: E402

from graphaligner_gb300 import graph as gg  # noqa: E402
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, pack_batch  # noqa: E402

pytestmark = pytest.mark.gpu

HANDED_ON = 8192
# kernels of a pass: the fill, the second fill where it runs, the traceback, the count of statuses
FIRST_PASS, NEXT_PASS = 4, 3


@pytest.mark.parametrize("count", [8191, 8192, 8193, 9000])
def test_more_than_a_call_hands_on(cuda_lib, oracle_lib, count):
    rng = np.random.default_rng(40)
    gfa, path = bubbles(40, 4, rng)          # 40 branches: more nodes than the small tables' 32
    g = gg.build_from_gfa(gfa)
    reads = ["".join("ACGT"[int(rng.integers(0, 4))] if rng.random() < 0.04 else c for c in path[3:]).encode() for _ in range(7)]
    params = ExtendParams(bandwidth=10)
    want = oracle_lib.extend(g, params, pack_batch(g, reads, [2] * 7, [2] * 7), threads=2)
    of = np.arange(count) % 7
    ext = Extender(DeviceGraph(g), arena_bytes=1 << 30)
    got = ext.run(params, pack_batch(g, [reads[k] for k in of], [2] * count, [2] * count))
    assert np.array_equal(got.status, want.status[of]) and np.array_equal(got.score, want.score[of])
    assert np.array_equal(got.cell_steps, want.cell_steps[of])
    for i in range(count):
        assert np.array_equal(got.items(i), want.items(int(of[i]))), f"trace {i}"
    assert ext.last_layout_counts() == [count, count, 0]
    assert ext.last_launches() == FIRST_PASS + (NEXT_PASS if count > HANDED_ON else 0)
    ext.close()


@pytest.mark.parametrize("over", [0, 1])
def test_batch_sizes_at_the_medium_tables_line(cuda_lib, over):
    import torch
    # four times the warps with medium tables that are on the GPU at once, five on an SM
    count = 4 * 5 * torch.cuda.get_device_properties(0).multi_processor_count + over
    g = load_graph("dbg100k")
    seqs, nodes, offs = load_requests("dbg100k")
    of = np.arange(count) % len(seqs)
    expected = load_digests("dbg100k", 10)
    ext = Extender(DeviceGraph(g))
    res = ext.run(ExtendParams(bandwidth=10, max_cells_per_slice=MAX_CELLS["dbg100k"]), pack_batch(g, [seqs[k] for k in of], nodes[of], offs[of]))
    bad = [i for i in range(count) if digest(res, i) != expected[of[i]]]
    assert not bad, f"{len(bad)} extensions differ, first {bad[:5]}"
    counts = ext.last_layout_counts()
    assert counts[0] == count and (counts[1] > 0) == bool(over)      # handed on by the small tables
    ext.close()
