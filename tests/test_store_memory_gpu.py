"""The column store only saves time: a call whose buffers find no memory while the store holds some
gets that memory and gives the same results without a store."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from golden_sets import compare, digest, golden_case, load_digests, load_graph, load_reads, load_requests  # noqa: E402
from test_multiseed_gpu import multiseed_seeds  # noqa: E402
from test_read_pipeline_host import harness  # noqa: E402,F401  (the host read-level harness)

from graphaligner_gb300.align import Aligner, preset  # noqa: E402
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, MultiseedBatch, pack_batch  # noqa: E402

pytestmark = pytest.mark.gpu

MB = 1 << 20
ARENA = 64 * MB
STORE = 4 * ARENA            # the most that the store takes


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


class OtherUser:
    """Device memory that the process holds for something else."""

    def __init__(self):
        self.blocks = []

    def leave(self, size):
        """Takes memory until about `size` bytes are free."""
        import torch
        step = (free_bytes() - size) // (2 * MB) * (2 * MB)
        if step > 0:
            self.blocks.append(torch.empty(step, dtype=torch.uint8, device="cuda"))

    def close(self):
        import torch
        self.blocks.clear()
        torch.cuda.empty_cache()


@pytest.fixture
def other():
    o = OtherUser()
    yield o
    o.close()


def filling_batch(g):
    """A batch whose columns fill the store."""
    seqs, nodes, offs = load_requests("vg50k")
    reps = -(-STORE // (16 * 3) // sum(map(len, seqs)))
    of = np.tile(np.arange(len(seqs)), reps + 1)
    return of, pack_batch(g, [seqs[k] for k in of], nodes[of], offs[of])


def load_kernels(dgraph, params, batch):
    """What the first call of a process takes on the device besides an extender's buffers."""
    ext = Extender(dgraph, arena_bytes=ARENA)
    ext.run(params, batch)
    ext.close()


def starve(other, ext, batch, params):
    """Runs the batch with room for the whole store, then leaves 200 MB; the bytes a buffer has to ask
    for so that it fits with the store's memory only."""
    other.leave(2 * STORE + 512 * MB + batch.total_items * 8 + 64 * batch.num)
    before = free_bytes()
    ext.run(params, batch)
    assert before - free_bytes() >= STORE
    other.leave(200 * MB)
    return free_bytes() + batch.total_items * 8 + STORE // 2


def test_host_batch(cuda_lib, other):
    g, one = golden_case("vg50k")
    expected = load_digests("vg50k", 10)
    params = ExtendParams(bandwidth=10)
    dgraph = DeviceGraph(g)
    load_kernels(dgraph, params, one)
    ext = Extender(dgraph, arena_bytes=ARENA)
    of, many = filling_batch(g)
    need = starve(other, ext, many, params)
    roomy = one.subset(np.arange(4))
    roomy.trace_capacity[3] = need // 8
    res = ext.run(params, roomy)
    assert [digest(res, i) for i in range(4)] == expected[:4]
    # the next batch has a store again, as large as half of what is free
    assert not compare(ext.run(params, one), expected)
    ext.close()


def test_multiseed_batch(cuda_lib, other, harness, tmp_path):  # noqa: F811
    g = load_graph("vg50k")
    _, seqs = load_reads("vg50k")
    seeds = multiseed_seeds(harness[0], "vg50k", "vg50k_reads", False, tmp_path)
    params = ExtendParams(bandwidth=10)
    dgraph = DeviceGraph(g)
    load_kernels(dgraph, params, golden_case("vg50k")[1])
    batch = MultiseedBatch.pack(seqs[:6], seeds[:6], max_traces=256, items_per_bp=64)
    ext = Extender(dgraph, arena_bytes=ARENA)
    want = ext.multiseed(params, batch)
    ext.close()
    ext = Extender(dgraph, arena_bytes=ARENA)
    need = starve(other, ext, filling_batch(g)[1], params)
    batch.trace_capacity[5] = need // 8
    got = ext.multiseed(params, batch)
    assert np.array_equal(got.status, want.status) and np.array_equal(got.num_traces, want.num_traces)
    for i in range(batch.num):
        for (gs, gi), (ws, wi) in zip(got.traces(i), want.traces(i)):
            assert gs == ws and np.array_equal(gi, wi)
    ext.close()


def test_seeding(cuda_lib, other):
    g, one = golden_case("vg50k")
    params = ExtendParams(bandwidth=10)
    dgraph = DeviceGraph(g)
    load_kernels(dgraph, params, one)
    ext = Extender(dgraph, arena_bytes=ARENA)
    a = Aligner(ext, g, preset("vg"))
    _, seqs = load_reads("vg50k")
    want = a.seeds(seqs[:3])
    need = starve(other, ext, filling_batch(g)[1], params)
    # a match slot of 16 bytes a read base, and the base itself
    reads = list(seqs[:3]) + [b"N" * (need // 17 // 64)] * 64
    got = a.seeds(reads)
    assert list(got[:3]) == list(want) and not any(len(x) for x in got[3:])
    a.close()
    ext.close()


def test_bounded_store_stays(cuda_lib, other):
    """Where free memory bounds the store, a little more of it does not make the store move."""
    g, one = golden_case("vg50k")
    params = ExtendParams(bandwidth=10)
    dgraph = DeviceGraph(g)
    load_kernels(dgraph, params, one)
    ext = Extender(dgraph, arena_bytes=ARENA)
    batch = filling_batch(g)[1]
    spare = OtherUser()
    other.leave(STORE + batch.total_items * 8 + 32 * MB)
    spare.leave(free_bytes() - 32 * MB)
    before = free_bytes()
    ext.run(params, batch)
    held = before - free_bytes()
    assert held > batch.total_items * 8 + 64 * MB        # a store, and not the whole one
    assert held < batch.total_items * 8 + STORE
    left = free_bytes()
    spare.close()
    freed = free_bytes() - left
    assert freed >= 32 * MB
    ext.run(params, batch)
    assert free_bytes() == left + freed
    ext.close()


@pytest.mark.parametrize("limit", [0, 1, 4096 * 16, 40 * MB])
def test_store_limit(cuda_lib, limit):
    """A store of at most the caller's bound, from the start or once it is larger, and the same results."""
    g, one = golden_case("vg50k")
    expected = load_digests("vg50k", 10)
    params = ExtendParams(bandwidth=10)
    dgraph = DeviceGraph(g)
    load_kernels(dgraph, params, one)
    slack = 4 * MB               # allocations are whole pages, and the store ends some units early

    def grown_by(ext, calls):
        before = free_bytes()
        for _ in range(calls):
            assert not compare(ext.run(params, one), expected)
        return before - free_bytes()
    ext = Extender(dgraph, arena_bytes=ARENA)
    ext.set_store_limit(0)
    staging = grown_by(ext, 1)
    ext.close()
    ext = Extender(dgraph, arena_bytes=ARENA)
    ext.set_store_limit(limit)
    assert abs(grown_by(ext, 2) - staging - limit) <= slack
    ext.close()
    ext = Extender(dgraph, arena_bytes=ARENA)
    full = grown_by(ext, 1) - staging
    assert full > 40 * MB + slack
    before = free_bytes()
    ext.set_store_limit(limit)
    assert abs(free_bytes() - before - full) <= slack
    assert abs(grown_by(ext, 2) - limit) <= slack
    ext.close()
