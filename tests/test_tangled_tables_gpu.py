"""Which tables the fill starts with on a graph with shared component numbers: the medium ones where at
least half of the nodes share theirs and the batch is not too large for them, else the small ones,
whose overflow is handed on.  Both sides of both lines against the oracle and the golden digests."""
import dataclasses

import numpy as np
import pytest

from graphaligner_gb300 import datagen as dg
from graphaligner_gb300 import graph as gg
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, pack_batch

from golden_sets import MAX_CELLS, digest, load_digests, load_graph, load_requests

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def workload():
    vg = dg.make_variation_graph(15_000, 40, 0.6, 20, seed=22)
    g = gg.build_from_gfa(vg.to_gfa())
    nl = np.zeros(len(vg.node_seqs) + 1, dtype=np.int64)
    nl[1:] = [len(s) for s in vg.node_seqs]
    reads = dg.sample_reads(vg, 12, 9, dg.uniform_length(1, 1500), dg.uniform_error(0.02, 0.2))
    return g, dg.seed_extensions(reads, nl, 11, 3)


@pytest.mark.parametrize("share", ["two", "under half", "half"])
def test_shared_component_numbers(cuda_lib, oracle_lib, workload, share):
    g, ext = workload
    n = g.num_nodes
    assert len(np.unique(g.component)) == n
    pairs = {"two": 1, "under half": (n - 1) // 4, "half": (n + 3) // 4}[share]
    # the numbers in order, the first `pairs` pairs of neighbours sharing one
    rank = np.argsort(np.argsort(g.component)).astype(np.int64)
    g = dataclasses.replace(g, component=np.where(rank < 2 * pairs, rank // 2 * 2, rank).astype(np.uint32))
    batch = pack_batch(g, ext.seqs, ext.bignode, ext.offset)
    x = Extender(DeviceGraph(g), arena_bytes=256 << 20)
    for params in (ExtendParams(bandwidth=10), ExtendParams(bandwidth=35, max_cells_per_slice=3000)):
        got = x.run(params, batch)
        want = oracle_lib.extend(g, params, batch, threads=2)
        assert np.array_equal(got.status, want.status) and np.array_equal(got.score, want.score)
        assert np.array_equal(got.cell_steps, want.cell_steps)
        for i in range(batch.num):
            assert np.array_equal(got.items(i), want.items(i)), f"trace {i}"
    x.close()


@pytest.mark.parametrize("count", [1, 7, 1000, 6000])
def test_batch_sizes_on_a_tangled_graph(cuda_lib, count):
    g = load_graph("dbg100k")
    seqs, nodes, offs = load_requests("dbg100k")
    of = np.arange(count) % len(seqs)
    batch = pack_batch(g, [seqs[k] for k in of], nodes[of], offs[of])
    expected = load_digests("dbg100k", 10)
    x = Extender(DeviceGraph(g))
    res = x.run(ExtendParams(bandwidth=10, max_cells_per_slice=MAX_CELLS["dbg100k"]), batch)
    bad = [i for i in range(count) if digest(res, i) != expected[of[i]]]
    assert not bad, f"{len(bad)} extensions differ, first {bad[:5]}"
    counts = x.last_layout_counts()
    assert counts[0] == count
    if count == 6000:
        assert counts[1] > 0        # handed on by the small tables
    x.close()
