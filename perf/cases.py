"""The work that a user of this framework has it do, as cases that can be timed.

Graphs and read lengths are those of the benchmark's and the tests' configurations: a
50 kbp variation graph (a bubble every ~200 bp), a 5 Mbp one (a variant every ~100 bp)
and the k=63 de Bruijn graph of a 1 Mbp genome with repeats and tandem arrays.  A case
names one call on one graph and the reads it takes; reads are windows of the graph's
sequence on a random strand with 60 % substitutions, 20 % insertions and 20 % deletions.

``prepare`` keeps what a program keeps between calls (the graph on the device, the
extender, the aligner with its index) and makes the case's own inputs from the seed.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from graphaligner_gb300 import _abi
from graphaligner_gb300 import datagen as dg
from graphaligner_gb300 import graph as gg
from graphaligner_gb300._lib import check, lib
from graphaligner_gb300.align import Aligner, preset
from graphaligner_gb300.extend import BatchResult, DeviceGraph, Extender, ExtendParams, PackedBatch

SEED_LENGTH = 15
GRAPH_BP = {"vg50k": 50_000, "vg5m": 5_000_000, "dbg1m": 1_150_000}


def _case(name, call, graph, reads, shortest, longest, error_low, error_high, mean=0, sigma=0.0, bandwidth=10, tangle=0):
    """sigma 0: lengths uniform in [shortest, longest]; else log-normal with this mean, clipped.
    tangle 0: no limit on the cells of a slice."""
    c = {"call": call, "graph": graph, "reads": reads, "shortest": shortest, "longest": longest, "error_low": error_low,
         "error_high": error_high, "mean": mean, "sigma": sigma, "bandwidth": bandwidth, "tangle": tangle}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one seed of one read: both extensions in one host-buffer call (an interactive caller, a server's quiet hour)
        _case("extend_one", "host", "vg5m", 1, 10_000, 10_000, 0.10, 0.10),
        # a few short reads or anchors: a handful of slices each, where launches and copies count
        _case("extend_short", "host", "vg5m", 32, 150, 600, 0.005, 0.02),
        # one round of a read-level seed loop: some hundred reads' extensions through pinned host buffers
        _case("extend_round", "host", "vg5m", 256, 1_000, 50_000, 0.05, 0.15, mean=10_000, sigma=0.6),
        # the batched workload of the benchmark at half its reads: resident in device memory
        _case("extend_batch", "device", "vg5m", 25_000, 1_000, 50_000, 0.05, 0.15, mean=10_000, sigma=0.6),
        # ultra-long reads: few extensions, many slices each
        _case("extend_long", "device", "vg5m", 48, 50_000, 100_000, 0.05, 0.15),
        # accurate long reads
        _case("extend_accurate", "device", "vg5m", 2_000, 1_000, 30_000, 0.002, 0.02, mean=15_000, sigma=0.3),
        # a cyclic, tangled graph with the dbg preset's bandwidth and tangle effort
        _case("extend_tangled", "device", "dbg1m", 500, 20_000, 20_000, 0.12, 0.12, bandwidth=5, tangle=10_000),
        # whole reads to GAF: seeding, seed loop, selection, lines
        _case("align_vg", "align", "vg50k", 200, 5_000, 15_000, 0.10, 0.10),
        # one read at a time, as a request handler calls it
        _case("align_one", "align", "vg5m", 1, 10_000, 10_000, 0.10, 0.10),
        _case("align_tangled", "align", "dbg1m", 100, 20_000, 20_000, 0.12, 0.12, bandwidth=5, tangle=10_000),
        # the multiseed DP: every seed of a read in one full-read pass
        _case("multiseed_tangled", "multiseed", "dbg1m", 40, 20_000, 20_000, 0.12, 0.12, bandwidth=5, tangle=10_000),
        # a program's start: the minimizer index of its graph
        _case("index_vg", "index", "vg5m", 1, 1_000, 1_000, 0.10, 0.10),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    call = rng.choice(["host", "host", "device", "device", "device", "align", "align", "multiseed", "index"])
    if call == "index":
        # the graph decides an index's work; the window of the read that follows makes cases distinct
        n = log_int(500, 5_000)
        return _case("", call, rng.choice(["vg5m", "dbg1m"]), 1, n, n, 0.10, 0.10)
    dbg = rng.random() < 0.25
    graph = "dbg1m" if dbg else rng.choice(["vg50k", "vg5m", "vg5m"])
    mean = log_int(300, 20_000)
    low = round(rng.uniform(0.002, 0.10), 4)
    high = round(rng.uniform(low, 0.15), 4)
    most = {"host": 600, "device": 6_000, "align": 200, "multiseed": 60}[call]
    reads = log_int(1, max(2, min(most, 60_000_000 // mean)))
    if dbg:
        reads = min(reads, max(1, {"host": 300, "device": 600, "align": 100, "multiseed": 40}[call] * 20_000 // max(mean, 5_000)))
    if call in ("align", "multiseed"):
        return _case("", call, graph, reads, max(100, mean // 4), min(30_000, mean * 3), low, high, mean, round(rng.uniform(0.2, 0.7), 2),
                     5 if dbg else 10, 10_000 if dbg else 0)
    return _case("", call, graph, reads, max(70, mean // 8), min(40_000, mean * 4), low, high, mean, round(rng.uniform(0.2, 0.7), 2),
                 rng.choice([5, 5, 10]) if dbg else rng.choice([5, 10, 10, 17]), 10_000 if dbg else 0)


# ---- graphs, with the place of every base of a walk through them ----

class _Source:
    def __init__(self, name):
        dev = torch.device("cuda")
        if name == "dbg1m":
            genome = dg.mid_dbg_genome(0)
            dbg = dg.compact_dbg(genome, 63, with_positions=True)
            self.graph = gg.build_from_gfa(dbg.gfa)
            walks = [(genome, dbg.pos_bignode, dbg.pos_offset)]
        else:
            vg = dg.small_vg(0) if name == "vg50k" else dg.batch_vg(0)
            self.graph = gg.build_from_gfa(vg.to_gfa())
            walks = []
            for h in range(2):
                hap = dg.sample_haplotype(vg, 11 + h)
                walks.append((hap.seq, hap.node * 2, hap.offset))
        g = self.graph
        codes = np.searchsorted(np.frombuffer(b"ACGT", dtype=np.uint8), np.concatenate([w[0] for w in walks])).astype(np.uint8)
        self.code = torch.from_numpy(codes).to(dev)
        self.node = torch.from_numpy(np.concatenate([w[1] for w in walks]).astype(np.int64)).to(dev)
        self.offset = torch.from_numpy(np.concatenate([w[2] for w in walks]).astype(np.int64)).to(dev)
        lens = np.array([len(w[0]) for w in walks], dtype=np.int64)
        self.walk_len = torch.from_numpy(lens).to(dev)
        self.walk_base = torch.from_numpy(np.cumsum(lens) - lens).to(dev)
        # split node of (bigraph node, offset): pieces sorted by (bigraph node, offset of the piece)
        ids = g.node_ids.astype(np.int64)
        key = (ids << 32) | g.node_offset.astype(np.int64)
        order = np.argsort(key, kind="stable")
        self.piece_key = torch.from_numpy(key[order]).to(dev)
        self.piece_node = torch.from_numpy(order.astype(np.int64)).to(dev)
        self.piece_start = torch.from_numpy(g.node_offset.astype(np.int64)).to(dev)
        size = np.zeros(int(g.lookup_ids.max()) + 2, dtype=np.int64)
        size[g.lookup_ids] = g.original_size
        self.size = torch.from_numpy(size).to(dev)
        self.device_graph = DeviceGraph(g)
        self.extender = Extender(self.device_graph)
        self.aligners = {}

    def split(self, bignode, offset):
        k = torch.searchsorted(self.piece_key, (bignode << 32) | offset, right=True) - 1
        node = self.piece_node[k]
        return node, offset - self.piece_start[node]

    def aligner(self, params_of, key):
        if key not in self.aligners:
            self.aligners[key] = Aligner(Extender(self.device_graph), self.graph, params_of())
        return self.aligners[key]


_SOURCES = {}


def _source(name):
    if name not in _SOURCES:
        _SOURCES[name] = _Source(name)
    return _SOURCES[name]


# ---- reads ----

def _starts(lens):
    return torch.cumsum(lens, 0) - lens


def _lengths(case):
    """The reads' lengths, the same for every seed, so that the outputs' shapes are."""
    rng = np.random.default_rng(7)
    n = case["reads"]
    if case["sigma"] > 0:
        mu = math.log(case["mean"]) - case["sigma"] ** 2 / 2
        return np.clip(rng.lognormal(mu, case["sigma"], n), case["shortest"], case["longest"]).astype(np.int64)
    return rng.integers(case["shortest"], case["longest"] + 1, n)


def _reads(src, case, seed):
    """Base codes of all reads end to end, each base's place in the source's walks (-1: edited), the
    reads' lengths and strands."""
    dev = src.code.device
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    n = case["reads"]

    def uniform(count):
        return torch.rand(count, generator=gen, device=dev)
    want = torch.from_numpy(_lengths(case)).to(dev)
    walk = (uniform(n) * len(src.walk_len)).long().clamp(max=len(src.walk_len) - 1)
    # a window a little longer than the read, cut to its length after the edits
    lens = torch.minimum(want + want // 16 + 64, src.walk_len[walk] - 1)
    start = src.walk_base[walk] + (uniform(n).double() * (src.walk_len[walk] - lens)).long()
    reverse = uniform(n) < 0.5
    error = case["error_low"] + uniform(n) * (case["error_high"] - case["error_low"])
    total = int(lens.sum())
    read = torch.repeat_interleave(torch.arange(n, device=dev), lens)
    pos = torch.arange(total, device=dev) - _starts(lens)[read]
    place = torch.where(reverse[read], start[read] + lens[read] - 1 - pos, start[read] + pos)
    truth = src.code[place]
    truth = torch.where(reverse[read], 3 - truth, truth)
    edited = uniform(total) < error[read]
    kind = uniform(total)
    sub = edited & (kind < 0.6)
    ins = edited & (kind >= 0.6) & (kind < 0.8)
    keep = ~(edited & (kind >= 0.8))
    base = torch.where(sub, (truth + 1 + (uniform(total) * 3).to(torch.uint8).clamp(max=2)) % 4, truth)
    count = keep.long() + ins.long()
    at = torch.cumsum(count, 0) - count
    out = torch.zeros(int(count.sum()), dtype=torch.uint8, device=dev)
    out_place = torch.full(out.shape, -1, dtype=torch.int64, device=dev)
    out[at[ins]] = (uniform(int(ins.sum())) * 4).to(torch.uint8).clamp(max=3)
    to = (at + ins.long())[keep]
    out[to] = base[keep]
    out_place[to] = torch.where(sub, torch.full_like(place, -1), place)[keep]
    made = torch.zeros(n, dtype=torch.int64, device=dev).scatter_add_(0, read, count)
    out_read = torch.repeat_interleave(torch.arange(n, device=dev), made)
    use = torch.arange(len(out), device=dev) - _starts(made)[out_read] < want[out_read]
    return out[use], out_place[use], torch.minimum(made, want), reverse, uniform(n)


def _extensions(src, case, seed):
    """Both extensions of one exact seed of each read, as device tensors in the batch layout."""
    code, place, lens, reverse, where = _reads(src, case, seed)
    dev = code.device
    n, total = len(lens), len(code)
    begin = _starts(lens)
    end = begin + lens
    i = torch.arange(total, device=dev)
    exact = place >= 0
    step = torch.ones(total, dtype=torch.bool, device=dev)
    step[1:] = exact[1:] & exact[:-1] & ((place[1:] - place[:-1]).abs() == 1)
    step[begin[lens > 0]] = False
    last_break = torch.cummax(torch.where(step, torch.full_like(i, -1), i), 0).values
    valid = exact & (i - last_break + 1 >= SEED_LENGTH)
    following = torch.cummin(torch.where(valid, i, torch.full_like(i, total)).flip(0), 0).values.flip(0)
    q = following[(begin + (where.double() * lens).long()).clamp(max=total - 1)]
    q = torch.where(q < end, q, following[begin.clamp(max=total - 1)])
    has = q < end
    q, begin, end, reverse = q[has], begin[has], end[has], reverse[has]
    at = place[q]
    node, off = src.node[at], src.offset[at]
    size = src.size[node]
    fw_node = torch.where(reverse, node ^ 1, node)
    fw_off = torch.where(reverse, size - 1 - off, off)
    # per read: the backward extension (reverse complement of what precedes the seed's last base), then the forward one
    ext_len = torch.stack([q - begin, end - 1 - q], 1).reshape(-1)
    ext_node = torch.stack([fw_node ^ 1, fw_node], 1).reshape(-1)
    ext_off = torch.stack([size - 1 - fw_off, fw_off], 1).reshape(-1)
    ext_from = torch.stack([q - 1, q + 1], 1).reshape(-1)
    back = (torch.arange(len(ext_len), device=dev) % 2) == 0
    some = ext_len > 0
    ext_len, ext_node, ext_off, ext_from, back = ext_len[some], ext_node[some], ext_off[some], ext_from[some], back[some]
    e = torch.repeat_interleave(torch.arange(len(ext_len), device=dev), ext_len)
    p = torch.arange(len(e), device=dev) - _starts(ext_len)[e]
    c = code[torch.where(back[e], ext_from[e] - p, ext_from[e] + p)]
    c = torch.where(back[e], 3 - c, c)
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=dev)
    split, split_off = src.split(ext_node, ext_off)
    room = ext_len + ext_len // 4 + 512
    return {"seq": letters[c.long()], "seq_offset": _starts(ext_len), "seq_len": ext_len.int(), "start_node": split.int(),
            "start_offset": split_off.int(), "trace_offset": _starts(room), "trace_capacity": room.int()}


_UNSIGNED = {torch.int32: np.uint32, torch.int64: np.uint64, torch.uint8: np.uint8}


def _pinned(t):
    """A pinned host copy as a numpy array of the C ABI's (unsigned) type."""
    return t.cpu().pin_memory().numpy().view(_UNSIGNED[t.dtype])


def _params(case):
    p = ExtendParams(bandwidth=case["bandwidth"])
    if case["tangle"]:
        p.max_cells_per_slice = case["tangle"]
    return p


def _text_room(case):
    """Room for a call's GAF text, zeros after its end."""
    return np.zeros(int(_lengths(case).sum()) * 16 + 4096 * case["reads"], dtype=np.uint8)


def _text(state, gaf):
    data = np.frombuffer(gaf.encode(), dtype=np.uint8)
    if len(data) > len(state["text"]):
        return data
    state["text"][:len(data)] = data
    return state["text"]


def prepare(case, seed):
    src = _source(case["graph"])
    call = case["call"]
    if call == "index":
        which = "dbg" if case["graph"] == "dbg1m" else "vg"
        codes, _, _, _, _ = _reads(src, case, seed)
        read = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=codes.device)[codes.long()].cpu().numpy().tobytes()
        return {"call": call, "src": src, "params": preset(which), "read": read, "text": _text_room(case)}
    if call in ("align", "multiseed"):
        code, _, lens, _, _ = _reads(src, case, seed)
        blob = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=code.device)[code.long()].cpu().numpy().tobytes()
        ends = np.cumsum(lens.cpu().numpy())
        seqs = [blob[int(e - n):int(e)] for e, n in zip(ends, lens.cpu().numpy())]
        which = "dbg" if case["graph"] == "dbg1m" else "vg"
        multi = call == "multiseed"
        aligner = src.aligner(lambda: preset(which, bandwidth=case["bandwidth"], tangle_effort=case["tangle"] or None, multiseed=multi),
                              (which, case["bandwidth"], case["tangle"], multi))
        return {"call": call, "aligner": aligner, "names": [f"read{i}" for i in range(len(seqs))], "seqs": seqs, "text": _text_room(case)}
    t = _extensions(src, case, seed)
    n = len(t["seq_len"])
    # the outputs' room is the same for every seed: two extensions a read, and their trace items
    most = 2 * case["reads"]
    lens = _lengths(case)
    items = int((lens + lens // 4 + 1024).sum())
    state = {"call": call, "src": src, "params": _params(case), "num": n}
    if call == "host":
        batch = PackedBatch(*(_pinned(t[k]) for k in ("seq", "seq_offset", "seq_len", "start_node", "start_offset", "trace_offset", "trace_capacity")))

        def room(count, dtype, view):
            return torch.zeros(count, dtype=dtype).pin_memory().numpy().view(view)
        out = BatchResult(room(most, torch.int32, np.int32), room(most, torch.int32, np.int32), room(most, torch.int32, np.uint32),
                          room(items, torch.int64, np.uint64), batch.trace_offset, room(most, torch.int64, np.uint64))
        return dict(state, batch=batch, out=out, flat=np.zeros(items, dtype=np.uint64))
    dev = t["seq"].device
    r = {"status": torch.zeros(most, dtype=torch.int32, device=dev), "score": torch.zeros(most, dtype=torch.int32, device=dev),
         "trace_len": torch.zeros(most, dtype=torch.int32, device=dev), "trace_items": torch.zeros(items, dtype=torch.int64, device=dev),
         "cell_steps": torch.zeros(most, dtype=torch.int64, device=dev)}
    c_of = {torch.uint8: ctypes.c_uint8, torch.int32: ctypes.c_uint32, torch.int64: ctypes.c_uint64}

    def p(x, c=None):
        return ctypes.cast(ctypes.c_void_p(x.data_ptr()), ctypes.POINTER(c or c_of[x.dtype]))
    batch = _abi.BatchDesc(n, p(t["seq"]), p(t["seq_offset"]), p(t["seq_len"]), p(t["start_node"]), p(t["start_offset"]),
                           p(t["trace_offset"]), p(t["trace_capacity"]))
    res = _abi.Results(p(r["status"], ctypes.c_int32), p(r["score"], ctypes.c_int32), p(r["trace_len"]), p(r["trace_items"]), p(r["cell_steps"]))
    return dict(state, batch=batch, res=res, tensors=t, out=r)


def run(state):
    call = state["call"]
    if call == "device":
        p = state["params"].c()
        check(lib().ga_extend_batch_device(state["src"].extender.handle, ctypes.byref(p), ctypes.byref(state["batch"]),
                                           ctypes.byref(state["res"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["out"]
    if call == "host":
        r = state["src"].extender.run(state["params"], state["batch"], state["out"])
        items = [r.items(i) for i in range(state["num"])]
        if items:
            # the traces end to end, as a caller takes them out of their rooms
            np.concatenate(items, out=state["flat"][:sum(len(x) for x in items)])
        return {"status": r.status, "score": r.score, "trace_len": r.trace_len.view(np.int32), "cell_steps": r.cell_steps.view(np.int64),
                "items": state["flat"].view(np.int64)}
    if call == "index":
        src = state["src"]
        aligner = Aligner(src.extender, src.graph, state["params"])
        info, keys, start, pos = aligner.index(arrays=True)
        gaf = aligner.align(["read"], [state["read"]])
        aligner.close()
        return {"max_count": info["max_count"], "keys": keys.view(np.int64), "start": start.view(np.int64), "pos": pos.view(np.int64),
                "gaf": _text(state, gaf)}
    gaf = state["aligner"].align(state["names"], state["seqs"])
    return {"gaf": _text(state, gaf), "read_bp": state["aligner"].read_bp(len(state["seqs"])).view(np.int64)}


def _mean_length(case):
    return case["mean"] if case["sigma"] > 0 else (case["shortest"] + case["longest"]) / 2


def work(case):
    """Bytes: the reads in and the trace items (8 B each) or GAF text (about 2 B per read bp) out, and
    the graph's sequence for an index, with 16 B per occurrence and 24 B per k-mer out.
    Operations: the column steps of the 64-row DP, about 2 per read bp at 40 integer operations
    (20 on 64-bit words)."""
    bp = case["reads"] * _mean_length(case)
    if case["call"] == "index":
        return {"bytes": GRAPH_BP[case["graph"]] * 2 * (0.25 + 0.2 * 40), "flops": GRAPH_BP[case["graph"]] * 2 * 10}
    per_bp = 1 + 2 if case["call"] in ("align", "multiseed") else 1 + 8
    return {"bytes": bp * per_bp, "flops": bp * 2 * 40}


def exact(case, seed):
    """Every output is whole numbers or bytes."""
    return None
