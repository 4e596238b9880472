"""X-score error costs around where the fill's 32-bit X-scores end (cost 2^16), below the
value of a match (100) and zero, against the oracle: the slices' best X-scores decide the X-drop
stop and where each trace starts."""
import numpy as np
import pytest

from graphaligner_gb300 import datagen as dg
from graphaligner_gb300 import graph as gg
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, pack_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def workload():
    vg = dg.make_variation_graph(20_000, 60, 0.6, 20, seed=9)
    g = gg.build_from_gfa(vg.to_gfa())
    nl = np.zeros(len(vg.node_seqs) + 1, dtype=np.int64)
    nl[1:] = [len(s) for s in vg.node_seqs]
    reads = dg.sample_reads(vg, 24, 8, dg.uniform_length(50, 3000), dg.uniform_error(0.02, 0.25))
    ext = dg.seed_extensions(reads, nl, 11, 3)
    batch = pack_batch(g, ext.seqs, ext.bignode, ext.offset)
    x = Extender(DeviceGraph(g), arena_bytes=256 << 20)
    yield g, batch, x
    x.close()


@pytest.mark.parametrize("cost", [1, 99, 100, 101, 295, 1000, 65_535, 65_536, 100_000])
@pytest.mark.parametrize("bandwidth,xdrop", [(10, 14705), (40, 2000)])
def test_cost_matches_the_oracle(cuda_lib, oracle_lib, workload, cost, bandwidth, xdrop):
    g, batch, x = workload
    params = ExtendParams(bandwidth=bandwidth, xdrop=xdrop, xscore_error_cost=cost)
    got = x.run(params, batch)
    want = oracle_lib.extend(g, params, batch, threads=2)
    assert np.array_equal(got.status, want.status) and np.array_equal(got.score, want.score)
    assert np.array_equal(got.cell_steps, want.cell_steps)
    for i in range(batch.num):
        assert np.array_equal(got.items(i), want.items(i)), f"trace {i}"
