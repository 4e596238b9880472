"""Extensions through nodes of many neighbours, against the oracle: the node record holds the
first two in- and three out-neighbours and degrees up to 4094, the rest come from the arrays;
bands of more than 32 nodes leave the shared-memory tables."""
import numpy as np
import pytest

from graphaligner_gb300 import graph as gg
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams, pack_batch

pytestmark = pytest.mark.gpu


def bubbles(branches: int, sites: int, rng):
    """A chain of 40-90 bp segments with a bubble of `branches` branches of 1-3 bp between them."""
    def seq(n):
        return "".join("ACGT"[k] for k in rng.integers(0, 4, n))
    lines, path, prev, node = [], "", [], 0
    for s in range(sites + 1):
        node += 1
        body = seq(int(rng.integers(40, 91)))
        lines.append(f"S\t{node}\t{body}")
        lines += [f"L\t{p}\t+\t{node}\t+\t0M" for p in prev]
        path += body
        if s == sites:
            break
        backbone, prev = node, []
        for b in range(branches):
            node += 1
            allele = seq(int(rng.integers(1, 4)))
            lines += [f"S\t{node}\t{allele}", f"L\t{backbone}\t+\t{node}\t+\t0M"]
            prev.append(node)
            if b == branches - 1:
                path += allele
    return "\n".join(lines) + "\n", path


@pytest.mark.parametrize("branches,sites", [(1, 8), (2, 8), (3, 8), (4, 8), (7, 6), (31, 4), (33, 4), (40, 4), (4094, 1), (4097, 1)])
def test_many_neighbours_match_the_oracle(cuda_lib, oracle_lib, branches, sites):
    rng = np.random.default_rng(branches)
    gfa, path = bubbles(branches, sites, rng)
    g = gg.build_from_gfa(gfa)
    reads = []
    for err in (0.0, 0.03, 0.10):
        r = [("ACGT"[int(rng.integers(0, 4))] if rng.random() < err else c) for c in path[3:]]
        reads.append("".join(r).encode())
    first = 2                                # bigraph node of segment 1, forward
    batch = pack_batch(g, reads + [reads[0][:1], reads[0][:64], reads[0][:65]], [first] * 6, [2] * 6)
    params = ExtendParams(bandwidth=10)
    ext = Extender(DeviceGraph(g), arena_bytes=256 << 20)
    got = ext.run(params, batch)
    want = oracle_lib.extend(g, params, batch, threads=2)
    assert np.array_equal(got.status, want.status) and np.array_equal(got.score, want.score)
    assert np.array_equal(got.cell_steps, want.cell_steps)
    for i in range(batch.num):
        assert np.array_equal(got.items(i), want.items(i)), f"trace {i}"
    ext.close()
