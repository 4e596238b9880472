"""A graph with nodes whose neighbour arrays are inconsistent is uploaded as it is, and extensions that
do not come near those nodes run: the node records made at the upload read nothing outside the
arrays."""
import dataclasses
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from golden_sets import compare, golden_case, load_digests  # noqa: E402

from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams  # noqa: E402

pytestmark = pytest.mark.gpu


def test_nodes_out_of_reach(cuda_lib):
    g, batch = golden_case("vg50k")
    n, extra = g.num_nodes, 3

    def more(a, values):
        return np.concatenate([a, np.array(values, dtype=np.uint64).astype(a.dtype)])
    far = [n + 10**6, 2**32 - 2, 2**30 - 1, n + extra]
    # the first one's offsets pass the end of the neighbours, the second one's begin behind it, the third
    # one's neighbours are no nodes
    bad = dataclasses.replace(
        g, num_nodes=n + extra, node_length=more(g.node_length, [64, 1, 33]), linearizable=more(g.linearizable, [0] * extra),
        component=more(g.component, int(g.component.max()) + 1 + np.arange(extra)), seq_ambiguous=more(g.seq_ambiguous, [1, 0, 0, 0] * extra),
        in_offsets=more(g.in_offsets, [2**32 - 16, len(g.in_neighbors), len(g.in_neighbors) + 4]), in_neighbors=more(g.in_neighbors, far),
        out_offsets=more(g.out_offsets, [2**32 - 16, len(g.out_neighbors), len(g.out_neighbors) + 4]), out_neighbors=more(g.out_neighbors, far))
    ext = Extender(DeviceGraph(bad), arena_bytes=256 << 20)
    assert not compare(ext.run(ExtendParams(bandwidth=10), batch), load_digests("vg50k", 10))
    ext.close()
