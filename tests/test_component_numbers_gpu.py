"""The component queue with and without shared component numbers, against the oracle on the same
arrays: numbers of their own (no heap), shared by pairs and by all (the reference's heap), and of
their own but spread widely (taken for shared)."""
import dataclasses

import numpy as np
import pytest

from graphaligner_gb300 import datagen as dg
from graphaligner_gb300 import graph as gg
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, pack_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def workload():
    vg = dg.make_variation_graph(15_000, 40, 0.6, 20, seed=21)
    g = gg.build_from_gfa(vg.to_gfa())
    nl = np.zeros(len(vg.node_seqs) + 1, dtype=np.int64)
    nl[1:] = [len(s) for s in vg.node_seqs]
    reads = dg.sample_reads(vg, 16, 8, dg.uniform_length(100, 2500), dg.uniform_error(0.02, 0.2))
    ext = dg.seed_extensions(reads, nl, 11, 3)
    return g, ext


@pytest.mark.parametrize("name,of", [("own", lambda c: c), ("pairs", lambda c: c // 2), ("one", lambda c: c * 0), ("spread", lambda c: c * 40 + 7)])
def test_component_numbers(cuda_lib, oracle_lib, workload, name, of):
    g, ext = workload
    assert len(np.unique(g.component)) == g.num_nodes
    g = dataclasses.replace(g, component=of(g.component.astype(np.int64)).astype(np.uint32))
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
