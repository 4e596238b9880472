"""The column store holds what finds room (at most four times the arena): with less room than the
batch's columns take, some node-slices are recomputed by the traceback, and the results are the
same.  Against the reference's vectors, in every table layout."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from golden_sets import MAX_CELLS, compare, golden_case, load_digests  # noqa: E402

from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,bandwidth,layout", [("vg50k", 10, 0), ("vg50k", 10, 1), ("dbg100k", 5, 0), ("dbg100k", 5, 2)])
@pytest.mark.parametrize("room", [1.05, 1.5, 3.0, 20.0])
def test_part_of_the_columns_kept(cuda_lib, name, bandwidth, layout, room):
    g, batch = golden_case(name)
    params = ExtendParams(bandwidth=bandwidth, max_cells_per_slice=MAX_CELLS.get(name, 2**64 - 1))
    dgraph = DeviceGraph(g)
    ext = Extender(dgraph)
    ext.run(params, batch)
    tables = ext.last_arena_bytes()
    ext.close()
    ext = Extender(dgraph, arena_bytes=int(tables * room) + batch.num * (4 << 10))
    ext.set_launch_shape(warps_per_block=4, blocks_per_sm=0, first_layout=layout, chunk_kib=4)
    for _ in range(2):
        res = ext.run(params, batch)
        bad = compare(res, load_digests(name, bandwidth))
        assert not bad, f"{len(bad)} extensions differ, first {bad[:5]}"
    ext.close()
    assert np.all(res.trace_len[res.status == 0] > 0)
