// Batched seed extension on GB300: one warp per extension.
//
// Persistent kernels run back to back.  In the fill kernel a warp owns one
// extension at a time and runs the banded Myers DP over the graph with the
// component-ordered frontier and X-drop, writing each committed slice into the
// batch's DP-table arena and, while there is room, each column into the column
// store; a second fill goes on with the extensions that outgrew the first one's
// tables; the traceback kernel then gives each warp one filled extension to walk
// back.  The DP of one extension is a sequential chain: each
// 64-row slice depends on the whole band of the previous one, and inside a slice
// nodes are computed one at a time in frontier order, the admission test using the
// running minimum.  So a warp runs that control flow warp-uniformly (every lane
// holds the same scalars, branches never diverge) and spreads over its lanes the
// work that is parallel inside it:
//   - the match masks of a slice (lane k reads rows k and k + 32; ballots),
//   - the match mask of every column of a node, before its column loop,
//   - per node: the horizontal deltas of every column, its X-score (lane k:
//     columns k and k + 32), the minimum and its first column (reduce + ballot) and
//     the bottom-row deltas (ballots), so the column loop itself only runs the
//     Myers recurrence on VP and VN,
//   - cellwise merges of columns and the changed-minimum test (row scores by
//     popcount, then a shuffle, ballots and a reduction),
//   - the small tables' node table, a slot per lane (ballots); the larger tables'
//     lookups, 32 probes of the open-addressing table per step,
//   - committing a slice to the DP table (coalesced copies),
//   - the traceback's end-cell choice (slices and columns across lanes), its band
//     lookups (ballot over the slice's node ids), and its walk inside a node and
//     slice: whole runs of one direction at a time, found in the columns' bits.
// The fill's frontier tables come in three sizes (see FillTables): the small ones
// in lane registers and shared memory, the medium ones in shared memory, the large
// ones in global memory.  A node's recorded columns are in shared memory always.
// Fill and traceback are separate kernels so that the warps of an SM share one
// phase's code.  With the traceback run by the fill's warps right after it, 50,000
// extensions (250 Mbp) took 95 ms instead of 51: the two phases' code does not fit
// the instruction caches.
//
// Times below that go from one figure to another are of the change that made the form, with the
// code around it as it was then.  As it stands, that batch takes 48.0 ms in these kernels
// (fill and traceback), one seed of a 10 kbp read 2.67 ms, 1,000 tangled extensions of 20 kbp
// reads 28.2 ms.
// Cold paths (crossing rules, end-cell choice, sequential fallbacks) are out of line.
//
// Warps take extensions from a device counter over a longest-first order.
//
// Reference correspondence (GraphAligner src/):
//   fill_extension   getReverseTraceFromSeed / getXdropSlices  (GraphAlignerBitvectorBanded.h:59-76, 580-725)
//   fill_slice       calculateSlice                            (GraphAlignerBitvectorBanded.h:255-511)
//   node_calc<Fill>  calculateNodeInner                        (GraphAlignerBitvectorCommon.h:1113-1478)
//   trace_extension  getReverseTraceFromTableExactEndPos / getReverseTraceFromTable
//                                                              (GraphAlignerBitvectorCommon.h:496-758)
//   bt_corner etc.   pickBacktraceInside/HorizontalCrossing/VerticalCrossing/Corner (:770-1054)
#include <cuda_runtime.h>
#include <stdint.h>
#include "extend.cuh"
#include "../../include/graphaligner_gb300.h"

namespace gadev
{

static constexpr unsigned kFull = 0xffffffffu;

// a pending incoming column of a node (ComponentPriorityQueue::extras entry)
struct Extra
{
    u64 VP, VN;
    i32 end;
    i32 before;         // the score above the column's first row
    uint16_t next;
    uint16_t skip;      // bit 0 EdgeWithPriority::skipFirst, bit 1 ::forceCalculation
};

static constexpr uint16_t kNil = 0xffff;

// node-table slot value: where the node sits in the slice's band and its queue state
struct NodeVal
{
    int16_t band;       // index in the slice's band, -1 until the node is first popped
    uint16_t active;    // node has a heap entry (ComponentPriorityQueue::active)
    uint16_t head;      // pending incoming columns, FIFO
    uint16_t tail;
};

// A fill warp's place in the arena and in the column store, in shared memory: it is asked for
// once a slice and once a node, and its registers are missed in between
struct ArenaCursor
{
    u64 pos;
    u64 end;
    u64 used;           // bytes handed out to this warp since the launch began
    u32 unit;           // this warp's units of the column store
    u32 unitEnd;
    u32 storeFull;
};

// A warp's recorded columns of one node-slice, in shared memory in every kernel: the fills' dynamic
// shared memory starts with a FillWarp per warp of the block.
struct __align__(16) NodeCols
{
    // what the column loop writes
    struct __align__(16) V { u64 VP, VN; } v[64];
    // what is worked out from them across the lanes
    struct __align__(16) X
    {
        u64 rows;       // the fill: horizontal -1 deltas of the step (the X-score's candidate mask);
                        // the traceback's recomputation: the rows with an open diagonal step
        i32 end;        // score of the last row
        u32 pad;
    } x[64];
    u64 base[4];        // the slice's match masks, one per base
    u64 eqcol[64 + 2];  // match mask of each column with its horizontal -1 input; [64] is read ahead of the last column

    __device__ __forceinline__ WS column(u32 k) const { return ws_make(v[k].VP, v[k].VN, x[k].end); }
    __device__ __forceinline__ i32 value(u32 k, u32 row) const { return ws_value(column(k), (int)row); }
};
struct __align__(16) FillWarp
{
    NodeCols cols;
    ArenaCursor arena;
};
extern __shared__ __align__(16) uint8_t dsmem[];

__device__ __forceinline__ FillWarp& fill_warp() { return ((FillWarp*)dsmem)[threadIdx.x >> 5]; }
__device__ __forceinline__ NodeCols& fill_cols() { return fill_warp().cols; }

__device__ __forceinline__ u32 hash_node(u32 node)
{
    u32 h = node * 0x9E3779B1u;
    return h ^ (h >> 15);
}

// A node's record put together from the graph's arrays (a graph without records).
__device__ __noinline__ void gather_record(const DevGraph& g, u32 node, NodeRec& r)
{
    const u32 in = g.inOff[node], inN = g.inOff[node + 1] - in;
    const u32 out = g.outOff[node], outN = g.outOff[node + 1] - out;
    // a record is made of every node, whether an extension comes near it or not: what an inconsistent
    // graph's arrays say about a node is not followed outside them
    const u32 inEnd = g.inOff[g.N], outEnd = g.outOff[g.N];
    r.seq[0] = node < g.firstAmbiguous ? g.seq2[(u64)node * 2] : 0;
    r.seq[1] = node < g.firstAmbiguous ? g.seq2[(u64)node * 2 + 1] : 0;
    r.comp = g.comp[node];
    r.meta = g.len[node] | (g.lin[node] ? kRecLinearizable : 0) | ((inN < kRecDegree ? inN : kRecDegree) << 8)
        | ((outN < kRecDegree ? outN : kRecDegree) << 20);
    r.inOff = in;
    r.outOff = out;
    for (u32 k = 0; k < kRecIn; k++) r.inNb[k] = k < inN && in < inEnd && k < inEnd - in ? g.inNb[in + k] : 0xffffffffu;
    for (u32 k = 0; k < kRecOut; k++)
    {
        r.outNb[k] = k < outN && out < outEnd && k < outEnd - out ? g.outNb[out + k] : 0xffffffffu;
        r.outComp[k] = r.outNb[k] < g.N ? g.comp[r.outNb[k]] : 0;
    }
}

__global__ void node_records_kernel(DevGraph g, NodeRec* rec)
{
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < g.N; i += gridDim.x * blockDim.x) gather_record(g, i, rec[i]);
}

__device__ __forceinline__ NodeRec node_record(const DevGraph& g, u32 node)
{
    NodeRec r;
    if (g.rec)
    {
        const uint4* src = (const uint4*)(g.rec + node);
        uint4* dst = (uint4*)&r;
#pragma unroll
        for (u32 k = 0; k < 4; k++) dst[k] = __ldg(src + k);
    }
    else
    {
        NodeRec x;          // its address is taken, r stays in registers
        gather_record(g, node, x);
        r = x;
    }
    return r;
}

// What a node's computation needs of its record; the out-neighbours are asked for afterwards,
// so that they do not take registers meanwhile
struct NodeHead
{
    u64 seq[2];
    u32 meta;
    u32 inNb;              // the first in-neighbour
};

// One warp's tables in global memory.  A node-table key is (generation << 32) | node; a slot whose
// generation is not the slice's is empty, so tables are never cleared between slices.
struct WSpace
{
    Item* band[2];
    u64* key[2];
    NodeVal* val[2];
    HeapItem* heap;
    Extra* extras;
    u32* columns;       // [band] where each band node's columns are in the column store
    i32* nodeMax;       // multiseed DP: [band] each band node's best exact-end-position X-score
};

__host__ __device__ inline u64 align16(u64 x) { return (x + 15) & ~15ULL; }

__host__ __device__ inline u64 wspace_bytes(const Caps& c, bool multi = false)
{
    u64 b = (multi ? 2 : 1) * align16((u64)c.band * 4);
    b += 2 * align16((u64)c.band * sizeof(Item));
    b += 2 * align16((u64)c.hash * 8);
    b += 2 * align16((u64)c.hash * sizeof(NodeVal));
    b += align16((u64)c.heap * sizeof(HeapItem));
    b += align16((u64)c.extras * sizeof(Extra));
    return align16(b);
}

__device__ __forceinline__ WSpace wspace_at(uint8_t* base, const Caps& c)
{
    WSpace w;
    u64 off = 0;
    w.band[0] = (Item*)(base + off); off += align16((u64)c.band * sizeof(Item));
    w.band[1] = (Item*)(base + off); off += align16((u64)c.band * sizeof(Item));
    w.key[0] = (u64*)(base + off); off += align16((u64)c.hash * 8);
    w.key[1] = (u64*)(base + off); off += align16((u64)c.hash * 8);
    w.val[0] = (NodeVal*)(base + off); off += align16((u64)c.hash * sizeof(NodeVal));
    w.val[1] = (NodeVal*)(base + off); off += align16((u64)c.hash * sizeof(NodeVal));
    w.heap = (HeapItem*)(base + off); off += align16((u64)c.heap * sizeof(HeapItem));
    w.extras = (Extra*)(base + off); off += align16((u64)c.extras * sizeof(Extra));
    w.columns = (u32*)(base + off); off += align16((u64)c.band * 4);
    w.nodeMax = (i32*)(base + off);    // inside the stride only when it was sized for the multiseed DP
    return w;
}

// Node-table lookup with 32 linear probes per step (lane k probes the k-th slot of the
// step); the first slot in probe order that is the node's or empty ends the probe.
// Returns the node's slot or -1.  Every lane gets the same answer.
__device__ __forceinline__ int tbl_find(const u64* key, u32 cap, u32 gen, u32 node, u32 lane)
{
    const u32 h = hash_node(node);
    const u64 want = ((u64)gen << 32) | node;
    #pragma unroll 1
    for (u32 base = 0; base < cap; base += 32)
    {
        const u32 slot = (h + base + lane) & (cap - 1);
        const u64 k = key[slot];
        const u32 hit = __ballot_sync(kFull, k == want);
        const u32 stop = hit | __ballot_sync(kFull, (u32)(k >> 32) != gen);
        if (stop)
        {
            const u32 first = __ffs((int)stop) - 1;
            return ((hit >> first) & 1) ? (int)((h + base + first) & (cap - 1)) : -1;
        }
    }
    return -1;
}

// the node's slot, claimed (band -1, inactive, no pending columns) if it has none;
// -1 when the table would pass half full
__device__ __forceinline__ int tbl_get_or_add(u64* key, NodeVal* val, u32 cap, u32 gen, u32 node, u32& used, u32 lane)
{
    const u32 h = hash_node(node);
    const u64 want = ((u64)gen << 32) | node;
    #pragma unroll 1
    for (u32 base = 0; base < cap; base += 32)
    {
        const u32 slot = (h + base + lane) & (cap - 1);
        const u64 k = key[slot];
        const u32 hit = __ballot_sync(kFull, k == want);
        const u32 stop = hit | __ballot_sync(kFull, (u32)(k >> 32) != gen);
        if (stop)
        {
            const u32 first = __ffs((int)stop) - 1;
            const u32 s = (h + base + first) & (cap - 1);
            if ((hit >> first) & 1) return (int)s;
            if (2 * (used + 1) > cap) return -1;
            used++;
            key[s] = want;
            NodeVal v;
            v.band = -1;
            v.active = 0;
            v.head = kNil;
            v.tail = kNil;
            val[s] = v;
            return (int)s;
        }
    }
    return -1;
}

// ---- the two forms of the fill's frontier tables ----
//
// Both give a slice a node table (slot: the node's place in the band, whether it is queued, its
// pending columns in order), the band of this slice and the one before, the heap of the
// component queue and the pool of pending columns.  next() starts a slice: the current band
// becomes the previous one.

struct SmallSpace
{
    Item band[2][kSmallBand];
    NodeRec rec[32];       // records of the slots' nodes
    HeapItem heap[kSmallHeap];
    Extra extras[kSmallExtras];
};

__device__ __forceinline__ SmallSpace& small_space()
{
    return ((SmallSpace*)(dsmem + (blockDim.x >> 5) * sizeof(FillWarp)))[threadIdx.x >> 5];
}

// The tables of a warp whose bands hold at most 32 nodes: slot k of the node table is lane k's
// registers, a lookup one ballot, and the nodes' records are copied into shared memory while
// they wait in the queue.  With a hash table and the records' fields read from global memory
// the pops and inserts took 17k of the fill's 45k cycles per slice of an extension alone.
//
// Unique: no two nodes of the graph share a component number, as in a variation graph.  The
// component queue then has one order whatever its heap looks like, the component numbers', so the
// queued slots are not in a heap at all and the next one is found by a minimum over the lanes.
// (Where numbers are shared, equal scores come off in the order the heap's layout gives.)
// With the heap instead, 50,000 extensions (250 Mbp) take 48.9 ms instead of 48.0, one seed of a
// 10 kbp read 2.72 instead of 2.67.  The lane tables and records against a hash table and the
// graph's arrays: 102.9 -> 92.7 ms, one seed 8 % less, 1,000 tangled extensions 14 % less.
template <bool Unique>
struct SmallTables
{
    static constexpr bool kSmall = true;
    static constexpr uint16_t kNoExtra = 0xff;
    static constexpr u32 kFresh = 0x00ffffffu;     // bits 0-7 band, 8-15 first and 16-23 last pending column (0xff: none), 24 queued
    static constexpr u32 kQueued = 1u << 24;
    static constexpr u32 kLinear = 1u << 25;       // the node is linearizable
    u32 lane;
    u32 id, val, comp;     // this lane's slot
    u32 bandSlot;          // the slot of band entry `lane`
    u32 columns;           // where the columns of band entry `lane` are
    u32 prevId, prevComp;  // the previous band's entry `lane`
    bool prevLinear;
    u32 used, heapN, poolN, count, prevCount, side;

    __device__ __forceinline__ SmallTables(const FillArgs&, u64, u32 lane_) : lane(lane_), id(0), val(0), comp(0), bandSlot(0), columns(0), prevId(0), prevComp(0),
        prevLinear(false), used(0), heapN(0), poolN(0), count(0), prevCount(0), side(0) {}
    __device__ __forceinline__ Item* band() const { return small_space().band[side]; }
    __device__ __forceinline__ const Item* prev_band() const { return small_space().band[side ^ 1]; }
    __device__ __forceinline__ HeapItem* heap() const { return small_space().heap; }
    __device__ __forceinline__ Extra* extras() const { return small_space().extras; }
    __device__ __forceinline__ i32* node_max() const { return nullptr; }
    __device__ __forceinline__ void restart() { count = 0; }
    __device__ __forceinline__ void next()
    {
        // a record that was asked for and not used may still be on its way to its slot
        asm volatile("cp.async.wait_all;" ::: "memory");
        prevId = __shfl_sync(kFull, id, (int)bandSlot);
        prevComp = __shfl_sync(kFull, comp, (int)bandSlot);
        prevLinear = (__shfl_sync(kFull, val, (int)bandSlot) & kLinear) != 0;
        prevCount = count;
        side ^= 1;
        used = heapN = poolN = count = 0;
    }
    // band index of node in the previous slice, or -1
    __device__ __forceinline__ int prev_of(u32 node) const
    {
        return __ffs((int)__ballot_sync(kFull, lane < prevCount && prevId == node)) - 1;
    }
    __device__ __forceinline__ int add(const DevGraph& g, u32 node, u32 component)
    {
        if (used >= 32) return -1;
        const u32 slot = used++;
        if (lane == slot)
        {
            id = node;
            comp = component;
            val = kFresh;
        }
        NodeRec& r = small_space().rec[slot];
        if (g.rec)
        {
            if (lane < 4)
            {
                const u32 to = (u32)__cvta_generic_to_shared((uint4*)&r + lane);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" :: "r"(to), "l"((const uint4*)(g.rec + node) + lane) : "memory");
            }
        }
        else gather_record(g, node, r);
        return (int)slot;
    }
    __device__ __forceinline__ int slot_of(const DevGraph& g, u32 node, u32 component)
    {
        const u32 hit = __ballot_sync(kFull, lane < used && id == node);
        return hit ? __ffs((int)hit) - 1 : add(g, node, component);
    }
    // one more pending column of `slot`; false when a table is full
    __device__ __forceinline__ bool queue(int slot, u32 node, u32 component, i32 score, const Extra& x)
    {
        u32 v = __shfl_sync(kFull, val, slot);
        if (!(v & kQueued))
        {
            if (heapN >= kSmallHeap) return false;
            if (Unique) heapN++;
            else
            {
                HeapItem h;
                h.component = component; h.score = score; h.node = node; h.slot = (u32)slot;
                heap_push(heap(), heapN, h);
            }
            v = (v & (kLinear | 0xffu)) | 0xffff00u | kQueued;
        }
        if (poolN >= kSmallExtras) return false;
        const u32 e = poolN++;
        extras()[e] = x;
        const u32 last = (v >> 16) & 0xff;
        if (last == 0xff) v = (v & ~0xff00u) | (e << 8);
        else extras()[last].next = (uint16_t)e;
        v = (v & ~0xff0000u) | (e << 16);
        if (lane == (u32)slot) val = v;
        return true;
    }
    // the queue's first node, and its slot
    __device__ __forceinline__ u32 top(u32& slot) const
    {
        if (!Unique)
        {
            slot = heap()[0].slot;
            return heap()[0].node;
        }
        const u32 key = lane < used && (val & kQueued) ? comp : 0xffffffffu;
        const u32 least = __reduce_min_sync(kFull, key);
        slot = (u32)__ffs((int)__ballot_sync(kFull, key == least && lane < used && (val & kQueued))) - 1;
        return __shfl_sync(kFull, id, (int)slot);
    }
    // takes the node off the queue; its first pending column
    __device__ __forceinline__ uint16_t take(u32 slot, int& bandIndex)
    {
        if (Unique) heapN--;
        else heap_pop(heap(), heapN);
        const u32 v = __shfl_sync(kFull, val, (int)slot);
        if (lane == slot) val = (v & (kLinear | 0xffu)) | 0xffff00u;
        bandIndex = (v & 0xff) == 0xff ? -1 : (int)(v & 0xff);
        return (uint16_t)((v >> 8) & 0xff);
    }
    // the node's band entry; -1 when the band is full
    __device__ __forceinline__ int enter(u32 slot)
    {
        if (count >= kSmallBand) return -1;
        if (lane == slot) val = (val & ~0xffu) | count;
        if (lane == count) bandSlot = slot;
        return (int)count++;
    }
    __device__ __forceinline__ u32 columns_of(u32 at) const { return __shfl_sync(kFull, columns, (int)at); }
    __device__ __forceinline__ void set_columns(u32 at, u32 where) { if (lane == at) columns = where; }
    // of the band entry this lane commits (entry `lane`, the only one)
    __device__ __forceinline__ u32 lane_columns(u32) const { return columns; }
    __device__ __forceinline__ int band_of(u32 slot) const
    {
        const u32 b = __shfl_sync(kFull, val, (int)slot) & 0xff;
        return b == 0xff ? -1 : (int)b;
    }
    __device__ __forceinline__ NodeHead head(const DevGraph&, u32 slot, u32)
    {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        const NodeRec& r = small_space().rec[slot];
        const NodeHead h { { r.seq[0], r.seq[1] }, r.meta, r.inNb[0] };
        if ((h.meta & kRecLinearizable) && lane == slot) val |= kLinear;
        return h;
    }
    // the record, for its out-neighbours
    __device__ __forceinline__ const NodeRec* record(const DevGraph&, u32 slot, u32, NodeRec&) const { return &small_space().rec[slot]; }
    __device__ __forceinline__ u32 prev_component(const DevGraph&, u32 k, u32) const { return __shfl_sync(kFull, prevComp, (int)k); }
    __device__ __forceinline__ bool prev_linear(const DevGraph&, u32 k, u32) const { return __shfl_sync(kFull, (int)prevLinear, (int)k) != 0; }
};

// Larger tables, a hash table with generation stamps: in global memory, or (Shared) in the block's
// shared memory for the extensions that outgrow the tables above.
template <bool Shared>
struct HashTables
{
    static constexpr bool kSmall = false;
    static constexpr uint16_t kNoExtra = kNil;
    WSpace w;
    Caps caps;
    u32 lane;
    u32 gen, prevGen;
    u32 used, heapN, poolN, count, prevCount, side;

    __device__ __forceinline__ static uint8_t* place(const FillArgs& a, u64 gwarp)
    {
        if (Shared) return dsmem + (blockDim.x >> 5) * sizeof(FillWarp) + (u64)(threadIdx.x >> 5) * a.workspaceStride;
        return a.workspace + gwarp * a.workspaceStride;
    }
    __device__ __forceinline__ HashTables(const FillArgs& a, u64 gwarp, u32 lane_) : w(wspace_at(place(a, gwarp), a.caps)),
        caps(a.caps), lane(lane_), gen(0), prevGen(0), used(0), heapN(0), poolN(0), count(0), prevCount(0), side(0)
    {
        clear();
    }
    // generation 0 marks every node-table slot empty
    __device__ __forceinline__ void clear()
    {
        __syncwarp();
#pragma unroll 1
        for (u32 k = lane; k < caps.hash; k += 32)
        {
            w.key[0][k] = 0;
            w.key[1][k] = 0;
        }
        __syncwarp();
    }
    __device__ __forceinline__ Item* band() const { return w.band[side]; }
    __device__ __forceinline__ const Item* prev_band() const { return w.band[side ^ 1]; }
    __device__ __forceinline__ HeapItem* heap() const { return w.heap; }
    __device__ __forceinline__ Extra* extras() const { return w.extras; }
    __device__ __forceinline__ i32* node_max() const { return w.nodeMax; }
    __device__ __forceinline__ void restart()
    {
        count = 0;
        if (gen > 0xF0000000u)
        {
            // generation stamps are about to wrap: clear this warp's tables
            clear();
            gen = 0;
        }
    }
    __device__ __forceinline__ void next()
    {
        prevGen = gen++;
        prevCount = count;
        side ^= 1;
        used = heapN = poolN = count = 0;
    }
    __device__ __forceinline__ int prev_of(u32 node) const
    {
        const int s = tbl_find(w.key[side ^ 1], caps.hash, prevGen, node, lane);
        return s < 0 ? -1 : (int)w.val[side ^ 1][s].band;
    }
    __device__ __forceinline__ int add(const DevGraph& g, u32 node, u32 component) { return slot_of(g, node, component); }
    __device__ __forceinline__ int slot_of(const DevGraph&, u32 node, u32)
    {
        return tbl_get_or_add(w.key[side], w.val[side], caps.hash, gen, node, used, lane);
    }
    __device__ __forceinline__ bool queue(int slot, u32 node, u32 component, i32 score, const Extra& x)
    {
        NodeVal& s = w.val[side][slot];
        if (!s.active)
        {
            if (heapN >= caps.heap) return false;
            HeapItem h;
            h.component = component; h.score = score; h.node = node; h.slot = (u32)slot;
            heap_push(w.heap, heapN, h);
            s.active = 1;
            s.head = kNil;
            s.tail = kNil;
        }
        if (poolN >= caps.extras) return false;
        const uint16_t e = (uint16_t)poolN++;
        w.extras[e] = x;
        if (s.head == kNil) s.head = e;
        else w.extras[s.tail].next = e;
        s.tail = e;
        return true;
    }
    __device__ __forceinline__ u32 top(u32& slot) const
    {
        slot = w.heap[0].slot;
        return w.heap[0].node;
    }
    __device__ __forceinline__ uint16_t take(u32 slot, int& bandIndex)
    {
        heap_pop(w.heap, heapN);
        NodeVal& s = w.val[side][slot];
        const uint16_t head = s.head;
        bandIndex = s.band;
        s.active = 0;
        s.head = kNil;
        s.tail = kNil;
        return head;
    }
    __device__ __forceinline__ int enter(u32 slot)
    {
        if (count >= caps.band || count >= 32767) return -1;
        w.val[side][slot].band = (int16_t)count;
        return (int)count++;
    }
    __device__ __forceinline__ u32 columns_of(u32 at) const { return w.columns[at]; }
    __device__ __forceinline__ void set_columns(u32 at, u32 where) { w.columns[at] = where; }
    __device__ __forceinline__ u32 lane_columns(u32 at) const { return w.columns[at]; }
    __device__ __forceinline__ int band_of(u32 slot) const { return w.val[side][slot].band; }
    __device__ __forceinline__ NodeHead head(const DevGraph& g, u32, u32 node)
    {
        const NodeRec r = node_record(g, node);
        return NodeHead { { r.seq[0], r.seq[1] }, r.meta, r.inNb[0] };
    }
    __device__ __forceinline__ const NodeRec* record(const DevGraph& g, u32, u32 node, NodeRec& room) const
    {
        if (g.rec) return g.rec + node;
        gather_record(g, node, room);
        return &room;
    }
    __device__ __forceinline__ u32 prev_component(const DevGraph& g, u32, u32 node) const { return g.comp[node]; }
    __device__ __forceinline__ bool prev_linear(const DevGraph& g, u32, u32 node) const { return g.lin[node] != 0; }
};

using LargeTables = HashTables<false>;
using MediumTables = HashTables<true>;

// ---- the traceback's shared memory ----

// A copy of one committed slice whose band has at most kCachedBand nodes
static constexpr u32 kCachedBand = 12;

struct __align__(16) SliceSlot
{
    SliceRec rec;
    Item items[kCachedBand];
    u32 slice;             // the slice, 0xffffffff = none
    u32 pad[3];
};

// One warp's.  The walk works on one slice and the one before it while the next one is on its
// way, so three slots (by the slice's number) hold them; the columns of a slice's whole band are
// copied from the column store while the walk is in the slice after it.
static constexpr u32 kKeptUnits = 128;

struct __align__(16) TraceWarp
{
    union
    {
        NodeCols cols;                         // a node-slice recomputed
        ColumnUnit kept[2][kKeptUnits];        // or the columns of two slices (odd and even)
    };
    ColumnUnit columns[64];                    // the recomputed node-slice in the column store's form
    u64 ring[64];                              // trace items not yet written out
    SliceSlot slots[3];
};

__device__ __forceinline__ TraceWarp& trace_warp() { return ((TraceWarp*)dsmem)[threadIdx.x >> 5]; }
__device__ __forceinline__ NodeCols& trace_cols() { return trace_warp().cols; }

// 16 bytes from global to shared memory, not waited for
__device__ __forceinline__ void copy_ahead(void* to, const void* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((u32)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void copies_done()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// IUPAC membership of every byte value (bit0 A, bit1 C, bit2 G, bit3 T; 0 = '-',
// -1 = not a sequence character), filled from iupac_mask on the host at load time and
// copied into shared memory by every block (lanes index it by data: the constant
// cache would serialise distinct addresses of a warp, shared memory serves them at once)
__constant__ int8_t c_iupac[256];
__shared__ int8_t s_iupac[256];

// all threads of the block must call this before any other work
__device__ __forceinline__ void load_iupac_table()
{
    for (u32 k = threadIdx.x; k < 256; k += blockDim.x) s_iupac[k] = c_iupac[k];
    __syncthreads();
}

// The read's bytes at rows lane and lane + 32 of the slice at j, -1 past the read's end
struct RowBytes
{
    int lo, hi;
};

__device__ __forceinline__ RowBytes row_bytes(const uint8_t* seq, u32 len, int64_t j, u32 lane)
{
    RowBytes r;
    r.lo = j + lane < (int64_t)len ? seq[j + lane] : -1;
    r.hi = j + lane + 32 < (int64_t)len ? seq[j + lane + 32] : -1;
    return r;
}

// Match masks of 64 rows (getEqVector, Common.h:279-318): the masks come from ballots.  False
// when a row holds a non-sequence byte, or a gap inside a full 64-row window (the reference
// asserts).  eq: NodeCols::base.
__device__ __forceinline__ bool eq_of_rows(const RowBytes& r, u64* eq)
{
    const bool full = __ballot_sync(kFull, r.hi < 0) == 0;
    int m0 = 0, m1 = 0;
    bool bad = false;
    if (r.lo >= 0)
    {
        m0 = s_iupac[r.lo];
        bad |= m0 < 0 || (m0 == 0 && full);
    }
    if (r.hi >= 0)
    {
        m1 = s_iupac[r.hi];
        bad |= m1 < 0 || (m1 == 0 && full);
    }
    const u64 e0 = (u64)__ballot_sync(kFull, m0 & 1) | ((u64)__ballot_sync(kFull, m1 & 1) << 32);
    const u64 e1 = (u64)__ballot_sync(kFull, m0 & 2) | ((u64)__ballot_sync(kFull, m1 & 2) << 32);
    const u64 e2 = (u64)__ballot_sync(kFull, m0 & 4) | ((u64)__ballot_sync(kFull, m1 & 4) << 32);
    const u64 e3 = (u64)__ballot_sync(kFull, m0 & 8) | ((u64)__ballot_sync(kFull, m1 & 8) << 32);
    __syncwarp();
    eq[0] = e0;
    eq[1] = e1;
    eq[2] = e2;
    eq[3] = e3;
    const bool ok = __ballot_sync(kFull, bad) == 0;
    __syncwarp();
    return ok;
}

// graph character of node n at pos (AlignmentGraph::NodeSequences) as an IUPAC mask
__device__ __forceinline__ int node_char_mask(const DevGraph& g, u32 n, u32 pos)
{
    if (n < g.firstAmbiguous)
    {
        u64 chunk = g.seq2[(u64)n * 2 + (pos >> 5)];
        return 1 << ((chunk >> ((pos & 31) * 2)) & 3);
    }
    const u64* a = g.seqAmb + (u64)(n - g.firstAmbiguous) * 4;
    return (int)((a[0] >> pos) & 1) | (int)(((a[1] >> pos) & 1) << 1) | (int)(((a[2] >> pos) & 1) << 2) | (int)(((a[3] >> pos) & 1) << 3);
}

// GraphAlignerCommon::characterMatch on a read byte and a graph position
__device__ __forceinline__ bool char_match(const DevGraph& g, uint8_t c, u32 n, u32 pos, bool& bad)
{
    int a = s_iupac[c];
    if (a < 0) { bad = true; return false; }
    int b = node_char_mask(g, n, pos);
    // identical characters always match; for distinct ones the IUPAC sets must overlap
    return (a & b) != 0;
}

// ---------------------------------------------------------------- warp column algebra
//
// A column's scores at rows lane and lane + 32 are two prefix popcounts away from its
// row-above score.  With them the cellwise operations take one shuffle, ballot or
// reduction step instead of the bit walks of WordSlice::differenceMasksBitTwiddle
// (WordSlice.h:566-664), whose trip counts depend on the data.  They return exactly what
// ws_merge (mergeTwoSlices: the cellwise minimum) and ws_changed_min
// (changedMinScoreLocalMinima: the least score among rows, and the row above, where the
// column improved on the old one) return for valid columns.  Scores beyond +-2^29 take
// the sequential forms, so no sum here can wrap.

static constexpr i32 kWarpScoreLimit = 1 << 29;

__device__ __forceinline__ bool score_ok(i32 v) { return v > -kWarpScoreLimit && v < kWarpScoreLimit; }

// scores of rows lane and lane + 32 (WordSlice::getValue)
__device__ __forceinline__ void ws_rows(const WS& w, i32 before, u32 lane, i32& v0, i32& v1)
{
    const u32 upto = (2u << lane) - 1u;
    const u32 vpl = (u32)w.VP, vnl = (u32)w.VN;
    const i32 low = popc32(vpl) - popc32(vnl);
    v0 = before + popc32(vpl & upto) - popc32(vnl & upto);
    v1 = before + low + popc32((u32)(w.VP >> 32) & upto) - popc32((u32)(w.VN >> 32) & upto);
}

// a column from its row-above score and its scores at rows lane and lane + 32
__device__ __forceinline__ WS ws_from_rows(i32 before, i32 m0, i32 m1, u32 lane)
{
    i32 p0 = __shfl_up_sync(kFull, m0, 1);
    i32 p1 = __shfl_up_sync(kFull, m1, 1);
    const i32 m31 = __shfl_sync(kFull, m0, 31);
    if (lane == 0)
    {
        p0 = before;
        p1 = m31;
    }
    const i32 d0 = m0 - p0, d1 = m1 - p1;
    WS r;
    r.VP = (u64)__ballot_sync(kFull, d0 == 1) | ((u64)__ballot_sync(kFull, d1 == 1) << 32);
    r.VN = (u64)__ballot_sync(kFull, d0 == -1) | ((u64)__ballot_sync(kFull, d1 == -1) << 32);
    r.end = __shfl_sync(kFull, m1, 31);
    return r;
}

__device__ __noinline__ WS merge_seq(WS a, WS b) { return ws_merge(a, b); }
__device__ __noinline__ i32 changed_min_seq(WS w, WS old) { return ws_changed_min(w, old); }

// mergeTwoSlices (WordSlice.h:502-541) across the lanes; ba and bb: ws_before of a and b
__device__ __forceinline__ WS merge_w(const WS& a, i32 ba, const WS& b, i32 bb, u32 lane)
{
    if (!(score_ok(ba) && score_ok(bb) && score_ok(a.end) && score_ok(b.end))) return merge_seq(a, b);
    i32 a0, a1, b0, b1;
    ws_rows(a, ba, lane, a0, a1);
    ws_rows(b, bb, lane, b0, b1);
    return ws_from_rows(imin(ba, bb), imin(a0, b0), imin(a1, b1), lane);
}
__device__ __forceinline__ WS merge_w(const WS& a, const WS& b, u32 lane) { return merge_w(a, ws_before(a), b, ws_before(b), lane); }

// changedMinScoreLocalMinima (WordSlice.h:438-472) across the lanes; old may be the
// never-computed column (0, 0, INT32_MAX), whose every score is INT32_MAX.  bw: ws_before(w)
__device__ __forceinline__ i32 changed_min_w(const WS& w, i32 bw, const WS& old, u32 lane)
{
    const i32 bo = ws_before(old);
    const bool oldUnset = old.VP == 0 && old.VN == 0 && old.end == kIntMax;
    if (!(score_ok(bw) && score_ok(w.end) && (oldUnset || (score_ok(bo) && score_ok(old.end))))) return changed_min_seq(w, old);
    i32 w0, w1, o0, o1;
    ws_rows(w, bw, lane, w0, w1);
    // a node's first column in the slice improves every row
    if (oldUnset) return imin(bw, __reduce_min_sync(kFull, imin(w0, w1)));
    ws_rows(old, bo, lane, o0, o1);
    i32 best = bw < bo ? bw : kIntMax;
    if (w0 < o0) best = imin(best, w0);
    if (w1 < o1) best = imin(best, w1);
    return __reduce_min_sync(kFull, best);
}

struct NodeCalc
{
    i32 minScore;
    u32 minScoreNode;
    u32 minScoreOffset;
    i32 maxX;
    u32 maxXNode;
    u32 cells;
};

struct PrevInfo
{
    bool exists;
    i32 sEnd;
    u64 HP, HN;
};

// An upper bound of ws_max_xscore(w, seqOffset, cost, 64, mask): every candidate row m scores
// 100 (m + 1) - cost s(m) with s(m) >= -popc(VN), plus 100 seqOffset - cost before.
__device__ __forceinline__ int64_t xscore_bound(const WS& w, i32 seqOffset, i32 cost)
{
    const i32 vn = popc64(w.VN);
    const i32 before = w.end - (popc64(w.VP) - vn);
    return 6400 + (int64_t)cost * vn + (int64_t)seqOffset * 100 - (int64_t)cost * before;
}

// ws_max_xscore(w, seqOffset, cost, 64, rows) less 100 seqOffset - cost ref, for a column whose
// scores are near ref (64 columns from one that ends within 4096 of it) and 0 <= cost < kCostLimit,
// so that no term wraps; or
// something not above `beat` if the column's best is not above it.
//
// Rows 0 and 63 always count.  The other candidates are the rows of `rows` just below a run of
// +1 deltas, (VP >> 1) & ~VP.  A candidate in the lower half is at most 3200 plus cost times the
// -1 deltas there, one in the upper half at most 6400 less cost times the lower half's sum plus
// cost times the upper half's -1 deltas; the candidates of a half that cannot beat `beat` are
// dropped.  Both halves' candidates are walked at once, so a warp goes round as often as the
// lane with most in one half, in 32 bits: with 64-bit bounds and one candidate a round the
// X-scores were 17 % of the fill (50,000 extensions 56.4 -> 55.2 ms, 1,000 tangled ones 45.6 ->
// 42.7 ms).
static constexpr i32 kCostLimit = 1 << 16;
static constexpr int64_t kOriginLimit = -(1LL << 30);     // with the greatest terms (4,160 kCostLimit) still within 32 bits
__device__ __forceinline__ bool near(i32 a, i32 b) { return (u32)a - (u32)b + 4096u <= 8192u; }

__device__ __forceinline__ i32 column_xscore(const WS& w, i32 ref, i32 cost, u64 rows, i32 beat)
{
    const u32 vpl = (u32)w.VP, vnl = (u32)w.VN, vph = (u32)(w.VP >> 32), vnh = (u32)(w.VN >> 32);
    const i32 nl = popc32(vnl), nh = popc32(vnh);
    const i32 low = popc32(vpl) - nl;
    const i32 all = low + popc32(vph) - nh;
    const i32 base = cost * (ref - w.end + all);
    i32 best = base + imax(100 - cost * ((i32)(vpl & 1) - (i32)(vnl & 1)), 6400 - cost * all);
    u32 candl = __funnelshift_r(vpl, vph, 1) & ~vpl & (u32)rows & ~1u;
    u32 candh = (vph >> 1) & ~vph & (u32)(rows >> 32);
    const i32 above = base - cost * low;
    if (base + 3200 + cost * nl <= beat) candl = 0;
    if (above + 6400 + cost * nh <= beat) candh = 0;
    #pragma unroll 1
    while (candl | candh)
    {
        if (candl)
        {
            const u32 upto = candl ^ (candl - 1);
            best = imax(best, base + 100 * popc32(upto) - cost * (popc32(vpl & upto) - popc32(vnl & upto)));
            candl &= ~upto;
        }
        if (candh)
        {
            const u32 upto = candh ^ (candh - 1);
            best = imax(best, above + 3200 + 100 * popc32(upto) - cost * (popc32(vph & upto) - popc32(vnh & upto)));
            candh &= ~upto;
        }
    }
    return best;
}

// Below this read offset no term of the X-score can wrap around in 32 bits, so the bound
// above also bounds the reference's (wrapping) arithmetic.
static constexpr i32 kXBoundOffsetLimit = 10000000;

// The part of calculateNodeInner (Common.h:1209-1300) that runs when the node already
// has a column in this slice: merge the new first column into it.  leave: the reference leaves
// the node early (nothing changed).  Out of line: a node is computed again within a slice only
// inside cyclic components.  (Out of line functions take and return values: a variable handed
// over by reference stays in local memory wherever it is used, and the walk's and the fill's own
// variables are read all the time.)
struct Merged
{
    WS ws;
    bool leave;
};

__device__ __noinline__ Merged merge_existing(WS ws, const Item& slice, bool hasSkipless, bool singleInEdge, u32 lane)
{
    WS s = ws_make(slice.sVP, slice.sVN, slice.sEnd);
    if (hasSkipless && singleInEdge)
    {
        if (ws.end > s.end) return Merged { ws, true };
        if (ws.end < s.end) return Merged { ws, false };
        u64 newBigger = (ws.VP & ~s.VP) | (s.VN & ~ws.VN);
        u64 oldBigger = (s.VP & ~ws.VP) | (ws.VN & ~s.VN);
        if (newBigger > oldBigger) return Merged { ws, false };
        if (oldBigger > newBigger) return Merged { ws, true };
        if (newBigger == 0 && oldBigger == 0) return Merged { ws, true };
        WS t = merge_w(ws, s, lane);
        return Merged { ws_eq(t, s) ? ws : t, ws_eq(t, s) };
    }
    WS t = merge_w(ws, s, lane);
    // the reference compares test.VP against the stored VN here (Common.h:1282)
    if (t.end == s.end && t.VP == s.VP && t.VP == s.VN) return Merged { ws, true };
    return Merged { t, false };
}

// The horizontal input along the slice's first row when the column enters below the
// previous slice's last row (Common.h:1310-1343): fixedHP/HN and, for a seed start, the
// columns whose first row is forced.  ok = false where the reference asserts.  Out of line:
// rarely taken.
struct FixedRow
{
    u64 HP, HN, force;
    bool ok;
};

__device__ __noinline__ FixedRow fix_horizontal(i32 scoreBefore, i32 scoreComparison, u64 fixedHP, u64 fixedHN)
{
    #pragma unroll 1
    for (int off = 1; off < 64; off++)
    {
        i32 next = scoreComparison + (i32)((fixedHP >> off) & 1) - (i32)((fixedHN >> off) & 1);
        u64 mask = 1ULL << off;
        if (scoreBefore > next) return FixedRow { fixedHP, fixedHN, 0, false };
        if (scoreBefore < next)
        {
            fixedHP |= mask;
            fixedHN &= ~mask;
        }
        else
        {
            fixedHP &= ~mask;
            fixedHN &= ~mask;
        }
        scoreBefore++;
        scoreComparison = next;
        if (scoreBefore >= scoreComparison) break;
    }
    return FixedRow { fixedHP, fixedHN, 0, true };
}

// The same when the node is a seed start of the multiseed DP (Common.h:1314-1362): the row
// above follows the lower of the previous slice's last row and the seed start's score
// before the slice, and every column of the first row takes its delta from that.
__device__ __noinline__ FixedRow fix_horizontal_extra(i32 scoreBefore, i32 scoreComparison, i32 extraBefore, u32 nodeLength, u64 fixedHP, u64 fixedHN)
{
    u64 forceMask = 0;
    scoreBefore = imin(scoreBefore, extraBefore);
    if (scoreBefore < scoreComparison) forceMask |= 1;
    i32 adjust = imin(scoreBefore, scoreComparison);
    #pragma unroll 1
    for (u32 off = 1; off < 64 && off < nodeLength; off++)
    {
        const i32 next = scoreComparison + (i32)((fixedHP >> off) & 1) - (i32)((fixedHN >> off) & 1);
        if (scoreBefore < extraBefore) scoreBefore += 1;
        const u64 mask = 1ULL << off;
        if (scoreBefore < next) forceMask |= mask;
        const i32 na = imin(next, scoreBefore);
        if (na < adjust - 1 || na > adjust + 1) return FixedRow { fixedHP, fixedHN, forceMask, false };
        if (na == adjust - 1)
        {
            fixedHN |= mask;
            fixedHP &= ~mask;
        }
        else if (na == adjust)
        {
            fixedHP &= ~mask;
            fixedHN &= ~mask;
        }
        else
        {
            fixedHP |= mask;
            fixedHN &= ~mask;
        }
        adjust = na;
        scoreComparison = next;
    }
    return FixedRow { fixedHP, fixedHN, forceMask, true };
}

// The columns 1.. of a seed start of the multiseed DP: its column `extra` joins every column.  hp, hn and
// fm: the horizontal inputs and the forced columns, bit 0: column 1.  Out of line: 1 node in 300 is one,
// and inside node_calc this loop made the other columns' 83 cycles a column instead of 36.
template <bool Fill>
__device__ __noinline__ WS seeded_columns(WS ws, WS extra, u64 hp, u64 hn, u64 fm, u32 columns, u32 lane)
{
    NodeCols& nc = Fill ? fill_cols() : trace_cols();
    #pragma unroll 1
    for (u32 pos = 1; pos < columns; pos++)
    {
        u64 Ph, Mh;
        WS nw = myers_step(nc.eqcol[pos], ws, hp & 1, hn & 1, Ph, Mh);
        if (fm & 1)
        {
            nw.VP &= kAllOnes ^ 1;
            nw.VN |= 1;
        }
        hp >>= 1;
        hn >>= 1;
        fm >>= 1;
        ws = merge_w(nw, extra, lane);
        nc.v[pos] = { ws.VP, ws.VN };
        nc.x[pos] = { Mh, ws.end, 0 };
    }
    return ws;
}

// calculateNodeInner (Common.h:1113-1478).  nodeLength, c0, c1: the node's length and 2-bit
// sequence.  flags: the band entry's, 0 for a node that has none yet.  singleInPrevBand: the
// node's only in-neighbour is in the previous band.  endColumn: the node's last column in this
// slice.  kept: the node-slice's units in the column store, or null.  Multi = false: the single-seed path, whose extra
// slice is always the fake one.  Multi = true: the multiseed DP, where `extra` (non-null for
// a node that is a seed start in this slice) is merged into every column and an incoming
// column that starts a seed forces the computation (EdgeWithPriority::forceCalculation).
// Fill = true: the slice fill (early leave allowed, calculateNodeClipPrecise).
// Fill = false: recalcNodeWordslice (no early leave); columns 0..lastColumn land in cols.
// The column loop runs the Myers recurrence warp-uniformly and records every column; the
// per-column minimum, X-score and horizontal output bits are then taken across the lanes.
//
// What bounds the loop is its chain: a warp alone waits about 4 cycles for each instruction
// that needs the last one, and a full SM has no issue slots left.  So a column does only the
// recurrence, on 32-bit halves: the horizontal -1 input is already in the column's match mask
// (where it is set the row's bits of VP and VN do not depend on the mask), the +1 input enters
// through the funnel shift that moves Ph down a row, the next mask is loaded a column ahead, and
// only VP and VN are recorded: afterwards lanes k and k + 32 run columns k and k + 32's step once
// more from the columns before them, which gives Ph and Mh, hence the last-row scores, for 64
// columns in the instructions of two.  The reference forces the
// first row's delta to -1 where the row above the slice is cheaper than the band above
// (forceMask); there the input is +1 and the column before it has that delta already, so the
// recurrence gives it by itself (the first column's merges keep it: the cheaper row above wins
// the minimum in both rows).  Only a seed start's columns need the force.
// Against 64-bit steps with inputs, force and deltas shifted out of words per column and the
// records behind generic pointers: 50,000 extensions (250 Mbp) 115.6 -> 102.9 ms, one seed of a
// 10 kbp read 13 % less.
template <bool Fill, bool Multi = false>
__device__ __forceinline__ NodeCalc node_calc(const DevGraph& g, i32 cost, u32 i, u32 nodeLength, u64 c0, u64 c1, Item& slice, u32 flags,
    const PrevInfo& prev, const Extra* pool, uint16_t head, uint16_t nil, const WS* singleIncoming, bool singleInPrevBand,
    i32 seqOffset, WS& endColumn, ColumnUnit* kept, u32& steps, int& err, u32 lane, i32 sliceMaxX = kIntMin, u32 lastColumn = 63, const WS* extra = nullptr)
{
    NodeCols& nc = Fill ? fill_cols() : trace_cols();
    u64* const eqcol = nc.eqcol;
    const bool hasExtra = Multi && extra != nullptr;
    bool forceCalculation = false;
    const bool boundOk = seqOffset < kXBoundOffsetLimit;
    NodeCalc result;
    result.minScore = kIntMax;
    result.minScoreNode = 0xffffffffu;
    result.minScoreOffset = 0xffffffffu;
    result.maxX = kIntMin;
    result.maxXNode = 0xffffffffu;
    result.cells = 0;
    const bool amb = i >= g.firstAmbiguous;
    u64 a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    if (amb)
    {
        const u64* a = g.seqAmb + (u64)(i - g.firstAmbiguous) * 4;
        a0 = a[0]; a1 = a[1]; a2 = a[2]; a3 = a[3];
    }
    auto mask_at = [&](u32 pos) -> u64
    {
        if (!amb) return nc.base[((pos < 32 ? c0 : c1) >> ((pos & 31) * 2)) & 3];
        return eq_amb(EqV4 { nc.base[0], nc.base[1], nc.base[2], nc.base[3] }, (u32)(((a0 >> pos) & 1) | (((a1 >> pos) & 1) << 1) | (((a2 >> pos) & 1) << 2) | (((a3 >> pos) & 1) << 3)));
    };
    const u64 eq0 = mask_at(0);

    WS ws = ws_make(0, 0, 0);
    i32 wsBefore = 0;           // ws_before(ws), carried along: a column's popcounts are a dozen instructions
    bool hasWs = false;
    bool hasSkipless = false;
    if (singleIncoming)
    {
        result.cells = 1;
        ws = *singleIncoming;
        wsBefore = ws_before(ws);
        hasWs = true;
    }
    else
    {
        #pragma unroll 1
        for (uint16_t e = head; e != nil;)
        {
            const Extra inc = pool[e];
            e = inc.next;
            WS incWs = ws_make(inc.VP, inc.VN, inc.end);
            result.cells++;
            if (Multi && (inc.skip & 2)) forceCalculation = true;
            if (inc.skip & 1)
            {
                ws = hasWs ? merge_w(ws, wsBefore, incWs, inc.before, lane) : incWs;
                wsBefore = hasWs ? imin(wsBefore, inc.before) : inc.before;
                hasWs = true;
                continue;
            }
            hasSkipless = true;
            i32 compareHin = prev.exists ? prev.sEnd : kIntMax;
            if (hasExtra) compareHin = imin(compareHin, ws_before(*extra));
            const i32 incBefore = inc.before;
            u64 hinP = 0, hinN = 0;
            if (compareHin < incBefore) hinN = 1;
            else if (compareHin > incBefore) hinP = 1;
            u64 Ph, Mh;
            WS nw = myers_step(eq0, incWs, hinP, hinN, Ph, Mh);
            steps++;
            // (as popcounts give it, the forced first row included)
            i32 nwBefore = incBefore + (i32)hinP - (i32)hinN;
            if (!prev.exists || nwBefore < prev.sEnd)
            {
                nwBefore += 1 - (i32)(nw.VN & 1) + (i32)(nw.VP & 1);
                nw.VP &= kAllOnes ^ 1;
                nw.VN |= 1;
            }
            ws = hasWs ? merge_w(ws, wsBefore, nw, nwBefore, lane) : nw;
            wsBefore = hasWs ? imin(wsBefore, nwBefore) : nwBefore;
            hasWs = true;
        }
    }
    if (!hasWs) { err = GA_ASSERT; return result; }
    // column 0 as the incoming columns make it: the node's first minimum candidate and,
    // with every row a candidate, its first X-score
    const WS ws0 = ws;
    result.minScore = ws.end;
    result.minScoreNode = i;
    result.minScoreOffset = 0;
    result.maxXNode = i;
    // the seed start's column joins after the first minimum and before the first X-score
    if (hasExtra)
    {
        ws = merge_w(ws, *extra, lane);
        wsBefore = ws_before(ws);
    }
    const WS wsX = ws;
    // (the recomputation starts from the stored first column, whose merge with itself changes nothing)
    bool leave = false;
    if (Fill && !forceCalculation && (flags & kExists) != 0)
    {
        const Merged m = merge_existing(ws, slice, hasSkipless, singleInPrevBand, lane);
        ws = m.ws;
        wsBefore = ws_before(ws);
        leave = m.leave;
    }
    if (leave)
    {
        endColumn = ws_make(slice.eVP, slice.eVN, slice.eEnd);
        if (!boundOk || xscore_bound(wsX, seqOffset, cost) > (int64_t)sliceMaxX)
            result.maxX = ws_max_xscore(wsX, seqOffset, cost, 64, kAllOnes);
        return result;
    }
    if (prev.exists && wsBefore > prev.sEnd)
    {
        ws = merge_w(ws, wsBefore, ws_source(prev.sEnd), prev.sEnd, lane);
        wsBefore = prev.sEnd;
    }
    u64 forceMask = 0;
    u64 fixedHP = prev.HP;
    u64 fixedHN = prev.HN;
    if (prev.exists)
    {
        i32 scoreBefore = wsBefore;
        i32 scoreComparison = prev.sEnd;
        if (scoreBefore > scoreComparison) { err = GA_ASSERT; return result; }
        if (hasExtra || scoreBefore < scoreComparison)
        {
            const FixedRow r = hasExtra ? fix_horizontal_extra(scoreBefore, scoreComparison, ws_before(*extra), nodeLength, fixedHP, fixedHN)
                : fix_horizontal(scoreBefore, scoreComparison, fixedHP, fixedHN);
            if (!r.ok) { err = GA_ASSERT; return result; }
            fixedHP = r.HP;
            fixedHN = r.HN;
            forceMask = r.force;
        }
    }
    else
    {
        forceMask = kAllOnes;
    }
    slice.sVP = ws.VP;
    slice.sVN = ws.VN;
    slice.sEnd = ws.end;
    slice.node = i | kExists | (flags & kSeedStart);
    const u64 forceEq = prev.exists ? kAllOnes : (kAllOnes ^ 1);
    // the traceback's recomputation stops at the column it needs last
    const u32 columns = Fill ? nodeLength : (lastColumn + 1 < nodeLength ? lastColumn + 1 : nodeLength);
    const i32 startEnd = ws.end;
    // the match mask of every column (lane k: columns k and k + 32), with the horizontal -1 input
    __syncwarp();
    #pragma unroll 1
    for (u32 pos = lane; pos < columns; pos += 32)
    {
        const u64 e = mask_at(pos);
        eqcol[pos] = pos == 0 ? e : (e & forceEq) | ((fixedHN >> pos) & 1);
    }
    nc.v[0] = { ws.VP, ws.VN };     // column 0 after the merges
    __syncwarp();
    if (!hasExtra)
    {
        u32 vpl = (u32)ws.VP, vph = (u32)(ws.VP >> 32), vnl = (u32)ws.VN, vnh = (u32)(ws.VN >> 32);
        u32 pos = 1;
        u64 eq = eqcol[1];
        #pragma unroll 1
        for (u32 half = 0; half < 2; half++)
        {
            // the horizontal inputs of columns 1..32, then 33..63, the next one in the top bit
            u32 hp = __brev((u32)(fixedHP >> (half ? 33 : 1)));
            u32 hn = __brev((u32)(fixedHN >> (half ? 33 : 1)));
            const u32 stop = half ? columns : (columns < 33 ? columns : 33);
            #pragma unroll 2
            for (; pos < stop; pos++)
            {
                const u32 eql = (u32)eq, eqh = (u32)(eq >> 32);
                eq = eqcol[pos + 1];
                const u64 sum = (((u64)(eqh & vph) << 32) | (eql & vpl)) + (((u64)vph << 32) | vpl);
                const u32 xhl = ((u32)sum ^ vpl) | eql, xhh = ((u32)(sum >> 32) ^ vph) | eqh;
                const u32 pl = vnl | ~(xhl | vpl), ph = vnh | ~(xhh | vph);
                const u32 ml = vpl & xhl, mh = vph & xhh;
                const u32 spl = __funnelshift_l(hp, pl, 1), sph = __funnelshift_l(pl, ph, 1);
                const u32 sml = __funnelshift_l(hn, ml, 1), smh = __funnelshift_l(ml, mh, 1);
                hp <<= 1;
                hn <<= 1;
                const u32 xvl = eql | vnl, xvh = eqh | vnh;
                vpl = sml | ~(xvl | spl);
                vph = smh | ~(xvh | sph);
                vnl = spl & xvl;
                vnh = sph & xvh;
                nc.v[pos] = { ((u64)vph << 32) | vpl, ((u64)vnh << 32) | vnl };
            }
        }
        ws.VP = ((u64)vph << 32) | vpl;
        ws.VN = ((u64)vnh << 32) | vnl;
    }
    else
    {
        ws = seeded_columns<Fill>(ws, *extra, fixedHP >> 1, fixedHN >> 1, forceMask >> 1, columns, lane);
    }
    __syncwarp();
    steps += columns - 1;
    result.cells = columns;
    // lane k: columns k and k + 32
    NodeCols::V col[2];
    u64 rows[2] = { kAllOnes, kAllOnes };
    i32 ends[2] = { startEnd, startEnd };
    u64 outHP, outHN;
    {
        bool plus[2] = { false, false }, minus[2] = { false, false };
        bool topPlus[2] = { false, false }, topMinus[2] = { false, false };
#pragma unroll
        for (u32 h = 0; h < 2; h++)
        {
            const u32 pos = lane + 32 * h;
            col[h] = { 0, 0 };
            if (pos >= columns) continue;
            col[h] = nc.v[pos];
            if (pos == 0) continue;
            const NodeCols::V before = nc.v[pos - 1];
            const u64 eq = eqcol[pos];
            const u64 Xh = (((eq & before.VP) + before.VP) ^ before.VP) | eq;
            const u64 Ph = before.VN | ~(Xh | before.VP);
            const u64 Mh = before.VP & Xh;
            rows[h] = Fill ? Mh : diagonal_rows(eq, Xh, before.VN);
            if (Fill && kept)
            {
                kept[pos] = { col[h].VP, diagonal_rows(eq, Xh, before.VN) };
                topPlus[h] = Ph & 1;
                topMinus[h] = Mh & 1;
            }
            plus[h] = (Ph >> 63) != 0;
            minus[h] = (Mh >> 63) != 0;
            if (hasExtra)
            {
                // the merged columns' deltas are not the step's
                const NodeCols::X x = nc.x[pos];
                const i32 last = pos == 1 ? startEnd : nc.x[pos - 1].end;
                if (Fill) rows[h] = x.rows;
                ends[h] = x.end;
                plus[h] = x.end == wadd(last, 1);
                minus[h] = x.end == wsub(last, 1);
            }
        }
        outHP = (u64)__ballot_sync(kFull, plus[0]) | ((u64)__ballot_sync(kFull, plus[1]) << 32);
        outHN = (u64)__ballot_sync(kFull, minus[0]) | ((u64)__ballot_sync(kFull, minus[1]) << 32);
        if (!hasExtra)
        {
            const u32 upto = (2u << lane) - 1u;
            const i32 low = popc32((u32)outHP) - popc32((u32)outHN);
            ends[0] = startEnd + popc32((u32)outHP & upto) - popc32((u32)outHN & upto);
            ends[1] = startEnd + low + popc32((u32)(outHP >> 32) & upto) - popc32((u32)(outHN >> 32) & upto);
            ws.end = startEnd + popc64(outHP) - popc64(outHN);
        }
        if (Fill && kept)
        {
            const u64 tp = (u64)__ballot_sync(kFull, topPlus[0]) | ((u64)__ballot_sync(kFull, topPlus[1]) << 32);
            const u64 tm = (u64)__ballot_sync(kFull, topMinus[0]) | ((u64)__ballot_sync(kFull, topMinus[1]) << 32);
            if (lane == 0) kept[0] = { tp, tm };
        }
        if (!Fill)
        {
#pragma unroll
            for (u32 h = 0; h < 2; h++)
                if (lane + 32 * h < columns) nc.x[lane + 32 * h] = { rows[h], ends[h], 0 };
            __syncwarp();
        }
    }
    if (Fill)
    {
        // Across the lanes: the first column of least score and the greatest X-score.
        // A column whose X-score bound is at most the slice's best so far cannot change the
        // slice's choice (it keeps the first node of strictly greatest X-score), so its exact
        // X-score is skipped; every column above that bound is scored exactly.
        u32 loKey = 0xffffffffu, hiKey = 0xffffffffu;
        i32 lmax = kIntMin;
        // scores and X-scores are counted from the node's first column
        const int64_t origin = (int64_t)seqOffset * 100 - (int64_t)cost * startEnd;
        // (far below zero a column's X-score leaves the 32 bits: each column is then bounded in 64 bits before
        // it is scored, and one that is out of their range does not come back as a great one)
        const bool small = boundOk && cost >= 0 && cost < kCostLimit && score_ok(startEnd) && near(ws0.end, startEnd) && near(wsX.end, startEnd)
            && origin > kOriginLimit;
        const int64_t toBeat = (int64_t)sliceMaxX - origin;
        const i32 beat = toBeat < -kWarpScoreLimit ? -kWarpScoreLimit : toBeat > kWarpScoreLimit ? kWarpScoreLimit : (i32)toBeat;
#pragma unroll
        for (u32 h = 0; h < 2; h++)
        {
            const u32 pos = lane + 32 * h;
            if (pos < columns)
            {
                // column 0 counts as it enters the node, every row a candidate; its X-score is
                // taken after the seed start's column joins it
                const bool first = pos == 0;
                const u32 key = (u32)(first ? ws0.end : ends[h]) ^ 0x80000000u;   // signed order as unsigned
                if (h == 0) loKey = key; else hiKey = key;
                const WS cw = first ? wsX : ws_make(col[h].VP, col[h].VN, ends[h]);
                if (small) lmax = imax(lmax, column_xscore(cw, startEnd, cost, rows[h], beat));
                else if (!boundOk || xscore_bound(cw, seqOffset, cost) > (int64_t)sliceMaxX)
                    lmax = imax(lmax, ws_max_xscore(cw, seqOffset, cost, 64, rows[h]));
            }
        }
        const u32 gkey = __reduce_min_sync(kFull, loKey < hiKey ? loKey : hiKey);
        const i32 gmax = __reduce_max_sync(kFull, lmax);
        const u32 onLo = __ballot_sync(kFull, loKey == gkey);
        const u32 onHi = __ballot_sync(kFull, hiKey == gkey);
        // column 0 always takes part, so the key is a real score
        result.minScore = (i32)(gkey ^ 0x80000000u);
        result.minScoreOffset = onLo ? (u32)(__ffs((int)onLo) - 1) : (u32)(32 + __ffs((int)onHi) - 1);
        result.maxX = small ? (i32)((u32)gmax + (u32)origin) : gmax;
        slice.HP = outHP;
        slice.HN = outHN;
    }
    slice.eVP = ws.VP;
    slice.eVN = ws.VN;
    slice.eEnd = ws.end;
    endColumn = ws;
    return result;
}

// ---------------------------------------------------------------- arena

// (the cursor is every lane's: each one has read it before any of them moves it)
// `columns` units of the column store, or kNoColumns
__device__ __forceinline__ u32 store_alloc(const FillArgs& a, ArenaCursor& c, u32 columns, u32 lane)
{
    u32 at = c.unit;
    const u32 end = c.unitEnd;
    if (end - at < columns)
    {
        if (c.storeFull) return kNoColumns;
        unsigned long long p = 0;
        if (lane == 0) p = atomicAdd(a.arenaCursor + 2, (unsigned long long)kStoreChunk);
        p = __shfl_sync(kFull, p, 0);
        if (p + kStoreChunk > a.storeUnits)
        {
            c.storeFull = 1;
            __syncwarp();
            return kNoColumns;
        }
        at = (u32)p;
        c.unitEnd = (u32)p + kStoreChunk;
    }
    __syncwarp();
    c.unit = at + columns;
    __syncwarp();
    return at;
}

// bytes from the warp's current chunk, else a new chunk (one atomic per chunk)
__device__ __forceinline__ bool arena_alloc(const FillArgs& a, ArenaCursor& c, u64 bytes, u64& out, u32 lane)
{
    bytes = align16(bytes);
    u64 at = c.pos;
    const u64 end = c.end, used = c.used;
    if (at + bytes > end)
    {
        const u64 grab = bytes > a.chunkBytes ? bytes : a.chunkBytes;
        unsigned long long p = 0;
        if (lane == 0) p = atomicAdd(a.arenaCursor, (unsigned long long)grab);
        p = __shfl_sync(kFull, p, 0);
        if (p + grab > a.arenaBytes) return false;
        at = p;
        c.end = p + grab;
    }
    __syncwarp();
    out = at;
    c.pos = at + bytes;
    c.used = used + bytes;
    __syncwarp();
    return true;
}

__device__ __forceinline__ u64 rec_ids_bytes(u32 count) { return align16((u64)count * 4); }

// slots of a committed band's index: none up to kHashedBand nodes, else the power of two at
// least twice the band (the index is at most half full)
__device__ __forceinline__ u32 band_hash_size(u32 count)
{
    if (count <= kHashedBand) return 0;
    u32 h = 256;
    while (h < 2 * count) h <<= 1;
    return h;
}

// write one slice of the tables (record, band in first-pop order, node ids and, for the multiseed DP, each
// node's best X-score and a large band's index) into the arena, lanes copying
template <class Tables>
__device__ __forceinline__ bool commit_slice(const FillArgs& a, ArenaCursor& c, u64* dir, u32 index, const Tables& t, i32 minScore, i32 quit,
    i32 maxX, u32 maxXNode, bool notValid, u32 lane, const i32* nodeMax = nullptr)
{
    const Item* band = t.band();
    const u32 count = t.count;
    const u64 idBytes = rec_ids_bytes(count);
    u64 off;
    const u64 maxBytes = nodeMax ? rec_ids_bytes(count) : 0;
    const u32 hashSize = nodeMax ? band_hash_size(count) : 0;
    const u64 hashOff = sizeof(SliceRec) + idBytes + (u64)count * sizeof(Item) + maxBytes;
    if (!arena_alloc(a, c, hashOff + (u64)hashSize * 4, off, lane)) return false;
    uint8_t* base = a.arena + off;
    if (lane == 0)
    {
        SliceRec r;
        r.minScore = minScore;
        r.quit = quit;
        r.maxX = maxX;
        r.maxXNode = maxXNode;
        r.count = count;
        r.notValid = notValid ? 1u : 0u;
        r.hashSize = hashSize;
        r.hashOff = hashSize ? (u32)hashOff : 0;
        *(SliceRec*)base = r;
        dir[index] = off;
    }
    uint4* const items = (uint4*)(base + sizeof(SliceRec));
    u32* const ids = (u32*)(items + count * 4);
    #pragma unroll 1
    for (u32 k = lane; k < count * 4; k += 32)
    {
        if ((k & 3) != 3) items[k] = ((const uint4*)band)[k];
    }
    #pragma unroll 1
    for (u32 k = lane; k < count; k += 32)
    {
        // the last quarter of an entry, with the place of the node's columns
        uint4 v = ((const uint4*)(band + k))[3];
        v.z = t.lane_columns(k);
        items[k * 4 + 3] = v;
        ids[k] = v.w & kNodeMask;
    }
    if (nodeMax)
    {
        i32* m = (i32*)(base + sizeof(SliceRec) + idBytes + (u64)count * sizeof(Item));
        #pragma unroll 1
        for (u32 k = lane; k < count; k += 32) m[k] = nodeMax[k];
    }
    if (hashSize)
    {
        // every slot empty, then each entry claims the first empty slot from its node's hash
        u32* slots = (u32*)(base + hashOff);
        #pragma unroll 1
        for (u32 k = lane; k < hashSize; k += 32) slots[k] = kEmptySlot;
        __syncwarp();
        #pragma unroll 1
        for (u32 k = lane; k < count; k += 32)
        {
            u32 h = hash_node(band[k].node & kNodeMask) & (hashSize - 1);
            #pragma unroll 1
            while (atomicCAS(&slots[h], kEmptySlot, k) != kEmptySlot) h = (h + 1) & (hashSize - 1);
        }
        __syncwarp();
    }
    return true;
}

// the band entries of committed slice r, and their node ids
__device__ __forceinline__ const Item* rec_items(const SliceRec* r) { return (const Item*)((const uint8_t*)r + sizeof(SliceRec)); }
__device__ __forceinline__ const u32* rec_ids(const SliceRec* r) { return (const u32*)(rec_items(r) + r->count); }

// position of node's entry in committed slice r (whose node ids are `ids`) through its band
// index: 32 slots per probe step, the first slot in probe order that is empty or the node's
// ends it.  Out of line: most bands are small, and the lookups are inlined in many places.
__device__ __noinline__ int rec_index_hashed(const SliceRec* r, const u32* ids, u32 node, u32 lane)
{
    const u32 hashSize = r->hashSize;
    const u32* slots = (const u32*)((const uint8_t*)r + r->hashOff);
    const u32 h = hash_node(node);
#pragma unroll 1
    for (u32 step = 0; step < hashSize; step += 32)
    {
        const u32 e = __ldcg(&slots[(h + step + lane) & (hashSize - 1)]);
        const bool empty = e == kEmptySlot;
        const bool hit = !empty && ids[e] == node;
        const u32 stop = __ballot_sync(kFull, empty || hit);
        if (stop) return __shfl_sync(kFull, hit ? (int)e : -1, __ffs((int)stop) - 1);
    }
    return -1;
}

// position of node's entry in committed slice r (whose node ids are `ids`), or -1; every lane
// gets the answer.  Hashed (the multiseed DP's tables): through the band index where the slice
// has one.  Else a ballot over the ids: the extension's tables have no index, and their lookups
// keep the short form.
template <bool Hashed>
__device__ __forceinline__ int rec_index(const SliceRec* r, const u32* ids, u32 node, u32 lane)
{
    if (Hashed && r->hashSize) return rec_index_hashed(r, ids, node, lane);
    const u32 n = r->count;
#pragma unroll 1
    for (u32 base = 0; base < n; base += 32)
    {
        const u32 k = base + lane;
        const u32 hit = __ballot_sync(kFull, k < n && ids[k] == node);
        if (hit) return (int)(base + __ffs((int)hit) - 1);
    }
    return -1;
}

// the multiseed DP's per-node best X-scores of a committed slice
__device__ __forceinline__ const i32* rec_node_max(const SliceRec* r)
{
    return (const i32*)((const uint8_t*)r + sizeof(SliceRec) + rec_ids_bytes(r->count) + (u64)r->count * sizeof(Item));
}

// ---------------------------------------------------------------- fill

struct SliceResult
{
    i32 minScore;
    u32 minScoreNode;
    i32 maxX;
    u32 maxXNode;
    u64 cells;
};

// getSeedSlice (Common.h:320-353): the column of starting an alignment at each row of the slice
// at j, each row scored as the X-score's error cost of the read before it (rows past the read's
// end one more each).  A row's score needs a 64-bit division, so lane k takes rows k and k + 32: row
// by row in every lane it was 19k of the multiseed fill's 123k cycles per slice.
__device__ __noinline__ WS seed_ws(int64_t j, u32 seqLen, i32 cost, u32 lane)
{
    auto score = [&](u32 before) { return (i32)(((j + before) * 100 + cost / 2) / cost); };
    const u32 inRead = j + 64 <= (int64_t)seqLen ? 64 : (u32)((int64_t)seqLen - j);     // a slice has one row at least
    const i32 lo = score(lane + 1), hi = score(lane + 33);
    const i32 start = j > 0 ? score(0) : 0;
    const i32 upLo = __shfl_up_sync(kFull, lo, 1), upHi = __shfl_up_sync(kFull, hi, 1), mid = __shfl_sync(kFull, lo, 31);
    const i32 beforeLo = lane == 0 ? start : upLo, beforeHi = lane == 0 ? mid : upHi;
    const u32 bitsLo = __ballot_sync(kFull, lane >= inRead || lo == wadd(beforeLo, 1));
    const u32 bitsHi = __ballot_sync(kFull, lane + 32 >= inRead || hi == wadd(beforeHi, 1));
    const u32 last = inRead - 1;
    const i32 endLo = __shfl_sync(kFull, lo, (int)(last & 31)), endHi = __shfl_sync(kFull, hi, (int)(last & 31));
    return ws_make((((u64)bitsHi << 32) | bitsLo) & ~1ULL, 1, wadd(last < 32 ? endLo : endHi, (i32)(64 - inRead)));
}

// The seeds the multiseed DP starts in one slice, with the slice's seed-start column.
struct SliceSeeds
{
    const u32* nodes;
    u32 count;
    WS ws;
};

// calculateSlice (GraphAlignerBitvectorBanded.h:255-511), component-queue branch.  Multi:
// the multiseed DP's slice, whose seeds enter the band first (addSeedHitToScoresAndQueue,
// :228-253) and whose nodes keep their best exact-end-position X-score in the tables' node_max.
// rows: the slice's read bytes on entry, the next slice's on return (loaded while this one runs).
template <class Tables, bool Multi = false>
__device__ __forceinline__ SliceResult fill_slice(const FillArgs& a, Tables& t, ArenaCursor& arena, const uint8_t* seq, u32 seqLen, RowBytes& rows,
    int64_t j, i32 prevQuit, i32 prevMin, u32& steps, int& err, u32 lane, const SliceSeeds* seeds = nullptr)
{
    if (Multi)
    {
        if (prevMin == kIntMax - (i32)a.bandwidth - 1)
        {
            prevMin = ws_before(seeds->ws);
            prevQuit = wadd(prevMin, (i32)a.bandwidth);
        }
        if (prevMin > seeds->ws.end)
        {
            prevMin = seeds->ws.end;
            prevQuit = wadd(seeds->ws.end, (i32)a.bandwidth);
        }
    }
    const DevGraph& g = a.g;
    const int bw = (int)a.bandwidth;
    t.next();
    Item* const band = t.band();
    const Item* const prevBand = t.prev_band();
    i32* const nodeMax = t.node_max();
    const uint16_t nil = Tables::kNoExtra;
    SliceResult res;
    res.minScore = kIntMax - bw - 1;
    res.minScoreNode = 0xffffffffu;
    res.maxX = kIntMin;
    res.maxXNode = 0;
    res.cells = 0;
    if (!eq_of_rows(rows, fill_cols().base)) { err = GA_ASSERT; return res; }
    rows = row_bytes(seq, seqLen, j + 64, lane);

    auto insert = [&](int slot, u32 node, u32 component, i32 score, const WS& c, i32 before, bool skip, bool force) -> bool
    {
        if (slot < 0) return false;
        Extra x;
        x.VP = c.VP; x.VN = c.VN; x.end = c.end; x.before = before; x.next = nil; x.skip = (skip ? 1 : 0) | (force ? 2 : 0);
        return t.queue(slot, node, component, score, x);
    };

    // the previous band's nodes that are within its quit score, 32 entries at a time
    #pragma unroll 1
    for (u32 from = 0; from < t.prevCount; from += 32)
    {
        i32 minScore = kIntMax, sEnd = 0;
        u32 id = 0;
        if (from + lane < t.prevCount)
        {
            const Item& it = prevBand[from + lane];
            minScore = it.minScore;
            sEnd = it.sEnd;
            id = it.node & kNodeMask;
        }
        const u32 have = t.prevCount - from < 32 ? (1u << (t.prevCount - from)) - 1u : kFull;
        u32 admitted = __ballot_sync(kFull, minScore <= prevQuit) & have;
        if (j == 0 && admitted != have) { err = GA_ASSERT; return res; }
        #pragma unroll 1
        while (admitted)
        {
            const u32 k = (u32)__ffs((int)admitted) - 1;
            admitted &= admitted - 1;
            const u32 node = __shfl_sync(kFull, id, (int)k);
            if (j != 0 && t.prev_linear(g, from + k, node))
            {
                const int pb = t.prev_of(g.inNb[g.inOff[node]]);
                if (pb >= 0)
                {
                    const Item& pn = prevBand[pb];
                    if (pn.eEnd < prevQuit && pn.minScore < prevQuit) continue;
                }
            }
            const u32 component = t.prev_component(g, from + k, node);
            const i32 above = __shfl_sync(kFull, sEnd, (int)k);
            // the band's nodes are distinct and the table is still empty of them
            if (!insert(t.add(g, node, component), node, component, __shfl_sync(kFull, minScore, (int)k), ws_source(above), above, true, false))
            {
                err = GA_CAPACITY;
                return res;
            }
        }
    }
    if (!Multi && t.heapN == 0) { err = GA_ASSERT; return res; }
    if (Multi && ws_before(seeds->ws) < wadd(prevQuit, 64))
    {
        // the seed starts: in the band before any node of the queue, computed first among equals
        #pragma unroll 1
        for (u32 k = 0; k < seeds->count; k++)
        {
            const u32 node = seeds->nodes[k];
            const u32 component = g.comp[node];
            const int slot = t.slot_of(g, node, component);
            if (slot < 0) { err = GA_CAPACITY; return res; }
            if (t.band_of((u32)slot) >= 0) { err = GA_ASSERT; return res; }
            const int at = t.enter((u32)slot);
            if (at < 0) { err = GA_CAPACITY; return res; }
            Item ni;
            ni.sVP = seeds->ws.VP; ni.sVN = seeds->ws.VN; ni.sEnd = seeds->ws.end;
            ni.eVP = seeds->ws.VP; ni.eVN = seeds->ws.VN; ni.eEnd = seeds->ws.end;
            ni.HP = 0; ni.HN = 0;
            ni.minScore = seeds->ws.end;
            ni.node = node | kExists | kSeedStart;
            band[at] = ni;
            nodeMax[at] = 0;
            t.set_columns((u32)at, kNoColumns);     // a seed start's columns are merged, their steps are not bits
            if (!insert(slot, node, component, ws_value(seeds->ws, 0), seeds->ws, ws_before(seeds->ws), true, true)) { err = GA_CAPACITY; return res; }
        }
    }
    i32 curMin = res.minScore;
    const i32 seqOffset = (i32)j;
    #pragma unroll 1
    while (t.heapN > 0)
    {
        u32 slot;
        const u32 i = t.top(slot);
        const NodeHead rec = t.head(g, slot, i);
        int at;
        const uint16_t head = t.take(slot, at);
        const bool fresh = at < 0;
        if (fresh)
        {
            at = t.enter(slot);
            if (at < 0) { err = GA_CAPACITY; return res; }
            if (Multi) nodeMax[at] = 0;
            t.set_columns((u32)at, store_alloc(a, arena, rec_len(rec.meta), lane));
        }
        const u32 columnsAt = t.columns_of((u32)at);
        Item& thisNode = band[at];
        const u32 flags = fresh ? 0 : thisNode.node & (kExists | kSeedStart);
        WS oldEnd = (flags & kExists) ? ws_make(thisNode.eVP, thisNode.eVN, thisNode.eEnd) : ws_make(0, 0, kIntMax);
        const WS* extra = (Multi && (flags & kSeedStart)) ? &seeds->ws : nullptr;
        if (Multi && extra) oldEnd = merge_w(oldEnd, *extra, lane);
        PrevInfo prev;
        const int pb = t.prev_of(i);
        prev.exists = pb >= 0;
        prev.sEnd = 0;
        prev.HP = kAllOnes;
        prev.HN = 0;
        if (pb >= 0)
        {
            const Item& pi = prevBand[pb];
            prev.sEnd = pi.sEnd;
            prev.HP = pi.HP;
            prev.HN = pi.HN;
        }
        // asked for only when a node is computed again
        const bool singleInPrev = (flags & kExists) && rec_in_degree(rec.meta) == 1 && t.prev_of(rec.inNb) >= 0;
        // a column whose X-score bound is at most both the slice's and the node's best so far
        // changes neither, so the node computation may skip its exact X-score
        const i32 skipBelow = Multi ? imin(res.maxX, nodeMax[at]) : res.maxX;
        WS newEnd;
        const NodeCalc nc = node_calc<true, Multi>(g, a.cost, i, rec_len(rec.meta), rec.seq[0], rec.seq[1], thisNode, flags, prev, t.extras(), head,
            nil, nullptr, singleInPrev, seqOffset, newEnd, columnsAt == kNoColumns ? nullptr : a.store + columnsAt, steps, err, lane, skipBelow, 63, extra);
        if (err) return res;
        if (Multi) nodeMax[at] = imax(nc.maxX, nodeMax[at]);
        if (nc.minScore > wadd(wadd(seqOffset, bw), 128)) { err = GA_ASSERT; return res; }
        curMin = imin(curMin, nc.minScore);
        if (fresh || nc.minScore < thisNode.minScore) thisNode.minScore = nc.minScore;
        if (!ws_eq(newEnd, oldEnd))
        {
            const i32 newEndBefore = ws_before(newEnd);
            const i32 newEndMin = changed_min_w(newEnd, newEndBefore, oldEnd, lane);
            if (newEndMin == kIntMax) { err = GA_ASSERT; return res; }
            if (newEndMin <= wadd(curMin, bw))
            {
                NodeRec room;
                const NodeRec* r = t.record(g, slot, i, room);
                u32 degree = rec_out_degree(rec.meta);
                if (degree >= kRecDegree) degree = g.outOff[i + 1] - r->outOff;
                #pragma unroll 1
                for (u32 e = 0; e < degree; e++)
                {
                    u32 target, component;
                    if (e < kRecOut)
                    {
                        target = r->outNb[e];
                        component = r->outComp[e];
                    }
                    else
                    {
                        target = g.outNb[r->outOff + e];
                        component = g.comp[target];
                    }
                    if (!insert(t.slot_of(g, target, component), target, component, newEndMin, newEnd, newEndBefore, false, false))
                    {
                        err = GA_CAPACITY;
                        return res;
                    }
                }
            }
        }
        if (nc.minScore < res.minScore)
        {
            res.minScore = nc.minScore;
            res.minScoreNode = nc.minScoreNode;
        }
        if (nc.maxX > res.maxX)
        {
            res.maxX = nc.maxX;
            res.maxXNode = nc.maxXNode;
        }
        if (res.minScore != curMin || nc.cells == 0) { err = GA_ASSERT; return res; }
        res.cells += nc.cells;
        if (res.cells > a.maxCells) break;
    }
    if (res.minScoreNode == 0xffffffffu && !(Multi && seeds->count == 0)) err = GA_ASSERT;
    return res;
}

// Writes down an extension for the medium tables, if there is room.  Out of line: rare, and the
// fill's registers are full.
__device__ __noinline__ void hand_on(ResumeRec* resume, u32 cap, u32* count, const Item* prevBand, u32 prevCount, FillState f, u32 ext, u32 lane)
{
    u32 k = 0;
    if (lane == 0) k = atomicAdd(count, 1u);
    k = __shfl_sync(kFull, k, 0);
    if (k >= cap) return;
    ResumeRec& rec = resume[k];
    #pragma unroll 1
    for (u32 q = lane; q < prevCount * 4; q += 32) ((uint4*)rec.band)[q] = ((const uint4*)prevBand)[q];
    if (lane == 0)
    {
        rec.state = f;
        rec.ext = ext;
        rec.count = prevCount;
    }
}

// The slices of an extension from f.slice on.  With the small tables, an extension that outgrows
// them at a slice is handed on to the medium ones while there is room for it.
template <class Tables>
__device__ __forceinline__ ExtState fill_slices(const FillArgs& a, Tables& t, ArenaCursor& arena, u32 ext, FillState& f, u32 lane)
{
    const uint8_t* seq = a.seq + a.seqOff[ext];
    const u32 seqLen = a.seqLen[ext];
    const u32 numSlices = (seqLen + 63) / 64;
    u64* dir = (u64*)(a.arena + f.dir);
    int err = 0;
    RowBytes rows = row_bytes(seq, seqLen, (int64_t)f.slice * 64, lane);
    #pragma unroll 1
    for (; f.slice < numSlices; f.slice++)
    {
        const int64_t j = (int64_t)f.slice * 64;
        u32 steps = 0;
        SliceResult r = fill_slice(a, t, arena, seq, seqLen, rows, j, f.lastQuit, f.lastMin, steps, err, lane);
        if (Tables::kSmall && err == GA_CAPACITY && a.resume)
        {
            hand_on(a.resume, a.resumeCap, a.resumeCount, t.prev_band(), t.prevCount, f, ext, lane);
        }
        f.steps += steps;
        if (err) break;
        if (r.maxX > f.bestX) f.bestX = r.maxX;
        const bool notValid = r.cells >= a.maxCells;
        if ((int64_t)r.maxX < (int64_t)f.bestX - (int64_t)a.xdrop) break;
        if (r.minScore < f.lastMin) { err = GA_ASSERT; break; }
        const i32 quit = wadd(r.minScore, (i32)a.bandwidth);
        if (!commit_slice(a, arena, dir, f.committed, t, r.minScore, quit, r.maxX, r.maxXNode, notValid, lane))
        {
            err = GA_CAPACITY;
            break;
        }
        f.committed++;
        f.lastMin = r.minScore;
        f.lastQuit = quit;
    }
    ExtState st;
    st.dir = f.dir;
    st.committed = f.committed;
    st.status = err ? err : f.committed <= 1 ? GA_TRACE_FAILED : GA_OK;
    st.steps = f.steps;
    st.aux = 0;
    return st;
}

template <class Tables>
__device__ __forceinline__ ExtState fill_extension(const FillArgs& a, Tables& t, ArenaCursor& arena, u32 ext, u32 lane)
{
    const DevGraph& g = a.g;
    ExtState st;
    st.dir = 0;
    st.committed = 0;
    st.status = GA_OK;
    st.steps = 0;
    st.aux = 0;
    const u32 seqLen = a.seqLen[ext];
    const u32 startNode = a.startNode[ext];
    const u32 startOff = a.startOffset[ext];
    const u32 numSlices = (seqLen + 63) / 64;
    if (startNode >= g.N || startOff >= g.len[startNode])
    {
        st.status = GA_BAD_REQUEST;
        return st;
    }
    u64 dirOff;
    if (!arena_alloc(a, arena, (u64)(numSlices + 1) * 8, dirOff, lane))
    {
        st.status = GA_CAPACITY;
        return st;
    }
    u64* dir = (u64*)(a.arena + dirOff);
    st.dir = dirOff;
    // start slice (getInitialSliceExactPosition, Common.h:1551-1587): one node, scores = distance from the offset
    t.restart();
    t.next();
    {
        Item it;
        u32 L = g.len[startNode];
        it.sVP = 0; it.sVN = 0; it.sEnd = (i32)startOff;
        it.eVP = 0; it.eVN = 0; it.eEnd = (i32)L - 1 - (i32)startOff;
        it.minScore = 0;
        it.node = startNode | kExists;
        // -1 along columns 1..startOff, +1 after them
        const u64 upToL = (L == 64 ? kAllOnes : (1ULL << L) - 1) & ~1ULL;
        it.HN = upToL & (startOff == 63 ? kAllOnes : (2ULL << startOff) - 1);
        it.HP = upToL & ~it.HN;
        const int slot = t.add(g, startNode, g.comp[startNode]);
        const int at = t.enter((u32)slot);
        t.band()[at] = it;
        t.set_columns((u32)at, kNoColumns);
        if (!commit_slice(a, arena, dir, 0, t, 0, 1, 0, startNode, false, lane))
        {
            st.status = GA_CAPACITY;
            return st;
        }
    }
    FillState f;
    f.dir = dirOff;
    f.steps = 0;
    f.slice = 0;
    f.committed = 1;
    f.bestX = 0;
    f.lastMin = 0;
    f.lastQuit = 1;
    return fill_slices(a, t, arena, ext, f, lane);
}

// GraphAlignerBitvectorBanded::getMultiseedSlices (GraphAlignerBitvectorBanded.h:727-822): every
// slice of read r from the empty initial slice, each slice's seeds started in it.  Each slice's
// best X-score also goes to a per-read array (st.aux) that the traceback lowers as it finds
// traces.
__device__ ExtState fill_multiseed(const FillArgs& a, LargeTables& t, ArenaCursor& arena, u32 r, u32 lane)
{
    ExtState st;
    st.dir = 0;
    st.committed = 0;
    st.status = GA_OK;
    st.steps = 0;
    st.aux = 0;
    const uint8_t* seq = a.seq + a.seqOff[r];
    const u32 seqLen = a.seqLen[r];
    const u32 numSlices = (seqLen + 63) / 64;
    const i32 bw = (i32)a.bandwidth;
    u64 dirOff, auxOff;
    if (!arena_alloc(a, arena, (u64)(numSlices + 1) * 8, dirOff, lane) || !arena_alloc(a, arena, (u64)(numSlices + 1) * 4, auxOff, lane))
    {
        st.status = GA_CAPACITY;
        return st;
    }
    u64* dir = (u64*)(a.arena + dirOff);
    i32* sliceMax = (i32*)(a.arena + auxOff);
    st.dir = dirOff;
    st.aux = auxOff;
    // getInitialEmptySlice (Common.h:1541-1549): no nodes, minimum 0, bandwidth 1
    t.restart();
    t.next();
    if (!commit_slice(a, arena, dir, 0, t, 0, 1, kIntMin, 0xffffffffu, false, lane, t.node_max()))
    {
        st.status = GA_CAPACITY;
        return st;
    }
    if (lane == 0) sliceMax[0] = kIntMin;
    u32 committed = 1;
    i32 lastMin = 0;
    i32 lastQuit = 1;
    u64 k = a.seedOff[r];
    const u64 kEnd = a.seedOff[r + 1];
    int err = 0;
    RowBytes rows = row_bytes(seq, seqLen, 0, lane);
    #pragma unroll 1
    for (u32 s = 0; s < numSlices; s++)
    {
        const int64_t j = (int64_t)s * 64;
        u64 next = k;
        while (next < kEnd && a.seedSlice[next] == s) next++;
        SliceSeeds seeds;
        seeds.nodes = a.seedNode + k;
        seeds.count = (u32)(next - k);
        seeds.ws = seed_ws(j, seqLen, a.cost, lane);
        k = next;
        u32 steps = 0;
        SliceResult res = fill_slice<LargeTables, true>(a, t, arena, seq, seqLen, rows, j, lastQuit, lastMin, steps, err, lane, &seeds);
        st.steps += steps;
        if (err) break;
        // fillDPSlice's checks of a slice that started seeds (GraphAlignerBitvectorBanded.h:543-549)
        if (seeds.count > 0)
        {
            const double lim = ((double)j + 64) * (double)a.cost;
            if (res.minScore > (i32)j + 64 || res.maxX == kIntMin || (double)res.maxX < -lim || (double)res.maxX > lim) { err = GA_ASSERT; break; }
        }
        if (!(res.minScore >= lastMin || res.minScore >= ws_value(seeds.ws, 0) || lastMin == kIntMax - bw - 1)) { err = GA_ASSERT; break; }
        const bool notValid = res.cells >= a.maxCells;
        const i32 quit = wadd(res.minScore, bw);
        if (!commit_slice(a, arena, dir, committed, t, res.minScore, quit, res.maxX, res.maxXNode, notValid, lane, t.node_max()))
        {
            err = GA_CAPACITY;
            break;
        }
        if (lane == 0) sliceMax[committed] = res.maxX;
        committed++;
        lastMin = res.minScore;
        lastQuit = quit;
    }
    if (!err && k != kEnd) err = GA_ASSERT;
    st.committed = committed;
    if (err) st.status = err;
    __syncwarp();
    return st;
}

// ---------------------------------------------------------------- traceback

// The record of slice s; a slice of at most kCachedBand nodes is first copied into its slot
// (lanes copy 16 bytes each)
__device__ __noinline__ const SliceRec* load_slice(const uint8_t* arena, const u64* dir, u32 s, u32 lane)
{
    const SliceRec* r = (const SliceRec*)(arena + dir[s]);
    const u32 n = r->count;
    if (n > kCachedBand) return r;
    SliceSlot& sl = trace_warp().slots[s % 3];
    __syncwarp();
#pragma unroll 1
    for (u32 k = lane; k < 2 + n * 4; k += 32) ((uint4*)&sl)[k] = ((const uint4*)r)[k];
    sl.slice = s;
    __syncwarp();
    return &sl.rec;
}

struct Table
{
    const uint8_t* arena;
    const u64* dir;
    u32 lane;
    __device__ __forceinline__ void init()
    {
        for (u32 k = 0; k < 3; k++) trace_warp().slots[k].slice = 0xffffffffu;
        __syncwarp();
    }
    // the slice's record: its shared copy (made on first use when the band is small), else
    // the arena's
    __device__ __forceinline__ const SliceRec* rec(u32 s)
    {
        SliceSlot& sl = trace_warp().slots[s % 3];
        if (sl.slice == s) return &sl.rec;
        return load_slice(arena, dir, s, lane);
    }
    // the band entry of node in slice s, or nullptr (Hashed: the multiseed DP's tables)
    template <bool Hashed = false>
    __device__ __forceinline__ const Item* find(u32 s, u32 node)
    {
        const SliceRec* r = rec(s);
        const SliceSlot& sl = trace_warp().slots[s % 3];
        if (sl.slice == s)
        {
            const u32 hit = __ballot_sync(kFull, lane < r->count && (sl.items[lane < kCachedBand ? lane : 0].node & kNodeMask) == node);
            return hit ? &sl.items[__ffs((int)hit) - 1] : nullptr;
        }
        const int k = rec_index<Hashed>(r, rec_ids(r), node, lane);
        return k < 0 ? nullptr : rec_items(r) + k;
    }
};

struct TPos
{
    u32 node;
    u32 off;
    i32 seq;          // below GA_MAX_SEQ_LEN; -1 = the row above the read
};

__device__ __forceinline__ bool tpos_eq(const TPos& a, const TPos& b) { return a.node == b.node && a.off == b.off && a.seq == b.seq; }

struct TStep
{
    TPos pos;
    bool sw;
};

// What a step takes off an item's upper word: a column (bits 32-37) or a row (bits 39-63).  Runs
// of steps of one kind lie inside one node, so the lower word, the node, stays.
static constexpr u32 kColumnStep = 1u, kRowStep = 1u << 7;

// Trace items go out one per lane, a run of steps of one kind at once, and into a 64-entry ring in
// shared memory that the circularity check reads.
// counting (MayCount only, the multiseed traceback): nothing goes out, the items are only
// counted.
template <bool MayCount>
struct TraceOutT
{
    u64* items;
    u64* ring;
    u32 cap;
    u32 n;
    u32 lane;
    TPos back;
    bool overflow;
    bool counting = false;
    // `count` (1..64) items, each `step` less in the upper word than the one before
    __device__ __forceinline__ void emit(u32 node, u32 upper, u32 step, u32 count)
    {
#pragma unroll 1
        for (u32 from = 0; from < count; from += 32)
        {
            const u32 k = from + lane;
            if (k < count)
            {
                const u64 x = ((u64)(upper - k * step) << 32) | node;
                ring[(n + k) & 63] = x;
                if (!(MayCount && counting)) items[n + k] = x;
            }
        }
        n += count;
        __syncwarp();
    }
    __device__ __forceinline__ static u32 upper_word(const TPos& p, bool sw)
    {
        return (p.off & 63) | (sw ? 1u << 6 : 0) | ((u32)(p.seq + 1) << 7);
    }
    __device__ __forceinline__ void push(const TPos& p, bool sw)
    {
        if (n >= cap) { overflow = true; return; }
        emit(p.node, upper_word(p, sw), 0, 1);
        back = p;
    }
    // `count` (1..64) steps of the same kind from `p`, which is the first item; every item stays
    // inside the read's rows
    __device__ __forceinline__ void push_run(TPos p, int dOff, int dSeq, u32 count)
    {
        if (count > cap - n) { overflow = true; count = cap - n; }
        if (count == 0) return;
        emit(p.node, upper_word(p, false), (dOff ? kColumnStep : 0) + (dSeq ? kRowStep : 0), count);
        p.off += (u32)(dOff * (int)(count - 1));
        p.seq += dSeq * (int)(count - 1);
        back = p;
    }
};
using TraceOut = TraceOutT<false>;

__device__ __forceinline__ u32 mod64(i32 seq) { return (u32)seq & 63; }

// checkBacktraceCircularity (Common.h:760-768): the newest item must not repeat an
// earlier item of the same read position.  Items still in the ring are read there, older
// ones from the written output (a counting walk checks the ring only).
__device__ __noinline__ bool trace_circular(const u64* items, const u64* ring, u32 n, bool ringOnly = false)
{
    if (n < 2) return false;
    const u64 keyMask = ~(1ULL << 38);
    const u64 last = ring[(n - 1) & 63];
#pragma unroll 1
    for (int k = (int)n - 2; k >= 0; k--)
    {
        if (ringOnly && (u32)k + 63 < n) return false;
        const u64 x = (u32)k + 63 >= n ? ring[k & 63] : items[k];
        if ((x & keyMask) == (last & keyMask)) return true;
        if ((x >> 39) != (last >> 39)) return false;
    }
    return false;
}

// The extraSlice of a node-slice: the multiseed DP's seed-start column (getSeedSlice) where the
// node is a seed start, else the fake column (0, 0, INT32_MAX), all of whose scores are INT32_MAX.
__device__ __forceinline__ WS fake_ws() { return ws_make(0, 0, kIntMax); }
// the extraSlice's score at a row and before the slice: the seed-start column's (Multi) or
// the fake column's, INT32_MAX, which no cell reaches
template <bool Multi> __device__ __forceinline__ i32 xval(const WS& e, int row) { return Multi ? ws_value(e, row) : kIntMax; }
template <bool Multi> __device__ __forceinline__ i32 xbefore(const WS& e) { return Multi ? ws_before(e) : kIntMax; }



// pickBacktraceCorner (Common.h:936-1054).  Out of line, like the other crossing rules:
// the walk inside a node-slice is the hot path.  t is a copy (its record cache is a hint).
template <bool Multi>
__device__ __noinline__ TStep bt_corner(const DevGraph& g, const uint8_t* seq, Table t, u32 cs, u32 node, i32 j, int& err, WS extra)
{
    const SliceRec* cr = t.rec(cs);
    const SliceRec* pr = t.rec(cs - 1);
    const Item* self = t.template find<Multi>(cs, node);
    TStep out; out.pos.node = 0; out.pos.off = 0; out.pos.seq = 0; out.sw = false;
    if (!self) { err = GA_ASSERT; return out; }
    i32 scoreHere = ws_value(ws_make(self->sVP, self->sVN, self->sEnd), 0);
    const Item* prevSelf = t.template find<Multi>(cs - 1, node);
    if (cr->notValid || scoreHere > cr->quit)
    {
        if (scoreHere == xval<Multi>(extra, 0)) { out.pos = TPos { node, 0, j }; return out; }
        i32 smallest = scoreHere + 1;
        TPos sp = TPos { 0xffffffffu, 0xffffffffu, -2 };
        bool change = false;
        if (prevSelf)
        {
            smallest = prevSelf->sEnd;
            sp = TPos { node, 0, j - 1 };
            change = false;
        }
        #pragma unroll 1
        for (u32 e = g.inOff[node]; e < g.inOff[node + 1]; e++)
        {
            u32 nb = g.inNb[e];
            const Item* pn = t.template find<Multi>(cs - 1, nb);
            if (pn && pn->eEnd <= smallest)
            {
                smallest = pn->eEnd;
                sp = TPos { nb, g.len[nb] - 1, j - 1 };
                change = true;
            }
            const Item* cn = t.template find<Multi>(cs, nb);
            if (cn && nb != node)
            {
                i32 v = ws_value(ws_make(cn->eVP, cn->eVN, cn->eEnd), 0);
                if (v < smallest)
                {
                    smallest = v;
                    sp = TPos { nb, g.len[nb] - 1, j };
                    change = true;
                }
            }
        }
        if (sp.node == 0xffffffffu) { err = GA_ASSERT; return out; }
        out.pos = sp; out.sw = change;
        return out;
    }
    bool bad = false;
    bool eq = char_match(g, seq[j], node, 0, bad);
    if (bad) { err = GA_ASSERT; return out; }
    TPos bestInvalid = TPos { 0xffffffffu, 0xffffffffu, -2 };
    i32 bestInvalidScore = scoreHere + 1;
    bool bestInvalidSw = false;
    if (prevSelf)
    {
        i32 ps = prevSelf->sEnd;
        if (ps < scoreHere - 1) { err = GA_ASSERT; return out; }
        if (ps == scoreHere - 1) { out.pos = TPos { node, 0, j - 1 }; return out; }
        if (pr->notValid || ps > pr->quit)
        {
            if (ps < bestInvalidScore)
            {
                bestInvalidScore = ps;
                bestInvalid = TPos { node, 0, j - 1 };
                bestInvalidSw = false;
            }
        }
    }
    #pragma unroll 1
    for (u32 e = g.inOff[node]; e < g.inOff[node + 1]; e++)
    {
        u32 nb = g.inNb[e];
        const Item* cn = t.template find<Multi>(cs, nb);
        if (cn)
        {
            i32 v = ws_value(ws_make(cn->eVP, cn->eVN, cn->eEnd), 0);
            if (v < scoreHere - 1) { err = GA_ASSERT; return out; }
            if (v == scoreHere - 1) { out.pos = TPos { nb, g.len[nb] - 1, j }; out.sw = true; return out; }
        }
        const Item* pn = t.template find<Multi>(cs - 1, nb);
        if (pn)
        {
            i32 corner = pn->eEnd;
            if (pr->notValid || corner > pr->quit)
            {
                if (corner < bestInvalidScore)
                {
                    bestInvalidScore = corner;
                    bestInvalid = TPos { nb, g.len[nb] - 1, j - 1 };
                    bestInvalidSw = true;
                }
            }
            else
            {
                if (corner < scoreHere - (eq ? 0 : 1)) { err = GA_ASSERT; return out; }
                if (corner == scoreHere - (eq ? 0 : 1)) { out.pos = TPos { nb, g.len[nb] - 1, j - 1 }; out.sw = true; return out; }
            }
        }
    }
    if (eq && scoreHere == xbefore<Multi>(extra)) { out.pos = TPos { node, 0, j }; return out; }
    if (scoreHere == xval<Multi>(extra, 0)) { out.pos = TPos { node, 0, j }; return out; }
    if (bestInvalidScore < scoreHere + 1) { out.pos = bestInvalid; out.sw = bestInvalidSw; return out; }
    err = GA_ASSERT;
    return out;
}

// The match masks of slice s into the warp's columns
__device__ __forceinline__ bool slice_masks(const uint8_t* seq, u32 seqLen, u32 s, u32 lane)
{
    return eq_of_rows(row_bytes(seq, seqLen, ((int64_t)s - 1) * 64, lane), trace_cols().base);
}

// recalcNodeWordslice (Common.h:1078-1102), after slice_masks: the columns 0..lastColumn of one node-slice
// into cols (the traceback only moves left inside a node, so it never needs the columns
// after the one it enters at).  When every column is recomputed the last one must equal
// the stored end column, as the reference asserts.  Returns 0 or the error status.
template <bool Multi = false>
__device__ __noinline__ int recalc(const DevGraph& g, i32 cost, Table t, u32 s, u32 node, u32 lane, u32 lastColumn,
    WS extra = fake_ws())
{
    const Item* it = t.template find<Multi>(s, node);
    if (!it) return GA_ASSERT;
    PrevInfo prev;
    const Item* pi = t.template find<Multi>(s - 1, node);
    if (pi) { prev.exists = true; prev.sEnd = pi->sEnd; prev.HP = pi->HP; prev.HN = pi->HN; }
    else { prev.exists = false; prev.sEnd = 0; prev.HP = kAllOnes; prev.HN = 0; }
    Item copy;
    WS start = ws_make(it->sVP, it->sVN, it->sEnd);
    WS last;
    u32 steps = 0;
    int err = 0;
    int64_t j = ((int64_t)s - 1) * 64;
    const NodeRec rec = node_record(g, node);
    const u32 L = rec_len(rec.meta);
    node_calc<false, Multi>(g, cost, node, L, rec.seq[0], rec.seq[1], copy, it->node, prev, nullptr, kNil, kNil, &start, false, (i32)j, last,
        nullptr, steps, err, lane, kIntMin, lastColumn, (Multi && extra.end != kIntMax) ? &extra : nullptr);
    if (err) return err;
    const NodeCols& nc = trace_cols();
    if (!ws_eq(nc.column(0), start)) return GA_ASSERT;
    if (lastColumn + 1 >= L && !ws_eq(nc.column(L - 1), ws_make(it->eVP, it->eVN, it->eEnd))) return GA_ASSERT;
    return 0;
}

// pickBacktraceVerticalCrossing (Common.h:886-934), the step out of (p.node, p.off > 0, row 0)
// into the previous slice; pself is the node's entry there, here the cell's score, eq whether its
// characters match
template <bool Multi>
__device__ __forceinline__ TStep vertical_step(const SliceRec* cr, const SliceRec* pr, const Item* pself, TPos p, i32 here, bool eq, int& err, const WS& extra)
{
    TStep second;
    second.pos = p;
    second.sw = false;
    // the previous slice's last row at column p.off - 1: its first column plus the deltas of columns 1..p.off-1
    const u64 upto = p.off >= 2 ? ((kAllOnes >> (64 - (p.off - 1))) << 1) : 0;
    i32 diag = pself->sEnd + popc64(pself->HP & upto) - popc64(pself->HN & upto);
    i32 up = diag + (i32)((pself->HP >> p.off) & 1) - (i32)((pself->HN >> p.off) & 1);
    if (pr->notValid || cr->notValid || here > cr->quit || diag > pr->quit || up > pr->quit)
    {
        if (here == xval<Multi>(extra, 0)) second = TStep { p, false };
        else if (diag < up) second = TStep { TPos { p.node, p.off - 1, p.seq - 1 }, false };
        else second = TStep { TPos { p.node, p.off, p.seq - 1 }, false };
        return second;
    }
    if (up < here - 1 || diag < here - (eq ? 0 : 1)) { err = GA_ASSERT; return second; }
    if (up == here - 1) return TStep { TPos { p.node, p.off, p.seq - 1 }, false };
    if (diag == here - (eq ? 0 : 1)) return TStep { TPos { p.node, p.off - 1, p.seq - 1 }, false };
    if (here != xval<Multi>(extra, 0)) err = GA_ASSERT;
    return second;
}

// pickBacktraceHorizontalCrossing (Common.h:817-884) at a cell whose score the tangle-effort
// cap left invalid: the least of what the in-neighbours and the cell above offer
template <bool Multi>
__device__ __noinline__ TStep horizontal_step_invalid(const DevGraph& g, Table t, u32 curSlice, u32 curNode, const Item* self, TPos p, u32 off,
    int& err, WS extra)
{
    TStep second;
    second.pos = p;
    second.sw = false;
    WS sws = ws_make(self->sVP, self->sVN, self->sEnd);
    i32 here = ws_value(sws, (int)off);
    i32 smallest = ws_value(sws, (int)off - 1);
    TPos sp = TPos { curNode, 0, p.seq - 1 };
    bool change = false;
    #pragma unroll 1
    for (u32 e = g.inOff[curNode]; e < g.inOff[curNode + 1]; e++)
    {
        u32 nb = g.inNb[e];
        const Item* cn = t.template find<Multi>(curSlice, nb);
        if (cn)
        {
            WS nws = ws_make(cn->eVP, cn->eVN, cn->eEnd);
            if (ws_value(nws, (int)off - 1) <= smallest)
            {
                smallest = ws_value(nws, (int)off - 1);
                sp = TPos { nb, g.len[nb] - 1, p.seq - 1 };
                change = true;
            }
            if (ws_value(nws, (int)off) < smallest && nb != curNode)
            {
                smallest = ws_value(nws, (int)off);
                sp = TPos { nb, g.len[nb] - 1, p.seq };
                change = true;
            }
        }
    }
    if (tpos_eq(sp, p) && here != xval<Multi>(extra, (int)off)) { err = GA_ASSERT; return second; }
    return TStep { sp, change };
}

struct EndCell
{
    u32 node;
    u32 nodeOffset;
    u32 bvOffset;
    i32 score;
    i32 j;
    int err;
};

// getReverseTraceFromTableExactEndPos (Common.h:496-562): the first slice of greatest
// X-score (lanes stride over the slices), then across the lanes (lane k: columns k and
// k + 32 of its best node) the cell of greatest row among those scoring the slice's
// X-score, the first column on ties.  The node's columns are left in cols.
__device__ __noinline__ EndCell end_cell(const DevGraph& g, i32 cost, const uint8_t* arena, Table t, u32 committed, const uint8_t* seq,
    u32 seqLen, u32 lane)
{
    const NodeCols& nc = trace_cols();
    EndCell ec;
    ec.err = 0;
    ec.nodeOffset = 0xffffffffu;
    ec.bvOffset = 0xffffffffu;
    i32 bx = kIntMin;
    u32 bs = 0xffffffffu;
    #pragma unroll 1
    for (u32 s = 1 + lane; s < committed; s += 32)
    {
        const i32 mx = ((const SliceRec*)(arena + t.dir[s]))->maxX;
        if (mx > bx) { bx = mx; bs = s; }
    }
    const i32 gbx = __reduce_max_sync(kFull, bx);
    const u32 best = __reduce_min_sync(kFull, bx == gbx ? bs : 0xffffffffu);
    const SliceRec* br = t.rec(best);
    ec.node = br->maxXNode;
    ec.score = br->maxX;
    ec.j = ((i32)best - 1) * 64;
    const i32 j = ec.j;
    if (!slice_masks(seq, seqLen, best, lane)) { ec.err = GA_ASSERT; return ec; }
    ec.err = recalc(g, cost, t, best, ec.node, lane, 63);
    if (ec.err) return ec;
    const int cells = (i32)seqLen - j < 64 ? (i32)seqLen - j : 64;
    const u32 L = g.len[ec.node];
    bool bad = false;
    int candOff = -1;
    u32 candCol = 0xffffffffu;
    #pragma unroll 1
    for (u32 h = 0; h < 2; h++)
    {
        const u32 i = lane + 32 * h;
        if (i >= L || bad) continue;
        const WS cw = nc.column(i);
        i32 mx = ws_max_xscore(cw, (i32)j, cost, cells, kAllOnes);
        if (mx > ec.score) { bad = true; continue; }
        if (mx == ec.score)
        {
            #pragma unroll 1
            for (int off = 63; off >= 0; off--)
            {
                if (j + off >= (i32)seqLen) continue;
                i32 here = ws_xscore(cw, (i32)j, off, cost);
                if (here > ec.score) { bad = true; break; }
                if (here == ec.score && off > candOff)
                {
                    candOff = off;
                    candCol = i;
                }
            }
        }
    }
    if (__ballot_sync(kFull, bad)) { ec.err = GA_ASSERT; return ec; }
    const int gOff = __reduce_max_sync(kFull, candOff);
    const u32 gCol = __reduce_min_sync(kFull, candOff == gOff ? candCol : 0xffffffffu);
    if (gOff < 0 || j + gOff >= (i32)seqLen) { ec.err = GA_ASSERT; return ec; }
    ec.nodeOffset = gCol;
    ec.bvOffset = (u32)gOff;
    return ec;
}

// the start node's row above the read (Common.h:721-756): walks left along the start
// slice while the score falls by one, then into an in-neighbour at offset 0
__device__ __noinline__ int row_above(const DevGraph& g, Table t, TraceOut& to)
{
    if (to.back.seq != -1) return GA_ASSERT;
    const Item* it = t.find(0, to.back.node);
    if (!it) return GA_ASSERT;
    const u32 L = g.len[to.back.node];
    // before[k] = score of column k in the row above the read
    const u64 hp = it->HP, hn = it->HN;
    const i32 s0 = it->sEnd;
    auto before = [&](u32 k) -> i32
    {
        const u64 upto = k >= 1 ? ((kAllOnes >> (64 - k)) << 1) : 0;   // columns 1..k
        return s0 + popc64(hp & upto) - popc64(hn & upto);
    };
    if (before(L - 1) != it->eEnd) return GA_ASSERT;
    #pragma unroll 1
    while (!to.overflow)
    {
        TPos q = to.back;
        i32 bq = before(q.off);
        if (!(bq != 0 && q.off > 0 && before(q.off - 1) == bq - 1)) break;
        to.push(TPos { q.node, q.off - 1, q.seq }, false);
    }
    TPos q = to.back;
    if (!to.overflow && q.off == 0 && before(0) != 0)
    {
        #pragma unroll 1
        for (u32 e = g.inOff[q.node]; e < g.inOff[q.node + 1]; e++)
        {
            u32 nb = g.inNb[e];
            const Item* ni = t.find(0, nb);
            if (ni && ws_before(ws_make(ni->eVP, ni->eVN, ni->eEnd)) == before(0) - 1)
            {
                to.push(TPos { nb, g.len[nb] - 1, q.seq }, true);
                break;
            }
        }
    }
    return 0;
}

// Columns 0..off of node-slice (s, node), recomputed into the warp's columns (NodeCols) and, in
// the column store's form, into `out`.  Returns 0 or the error status.  Out of line: only what
// found no room in the column store, and the multiseed DP's seed starts, come here.
template <bool Multi>
__device__ __noinline__ int recompute(const DevGraph& g, i32 cost, Table t, const uint8_t* seq, u32 seqLen, u32 s, u32 node, u32 off, WS extra, u32 lane)
{
    ColumnUnit* const out = trace_warp().columns;
    if (!slice_masks(seq, seqLen, s, lane)) return GA_ASSERT;
    const int err = recalc<Multi>(g, cost, t, s, node, lane, off, extra);
    if (err) return err;
    const NodeCols& nc = trace_cols();
    i32 v[2];
#pragma unroll
    for (u32 h = 0; h < 2; h++) v[h] = lane + 32 * h <= off ? nc.value(lane + 32 * h, 0) : 0;
    i32 p0 = __shfl_up_sync(kFull, v[0], 1);
    i32 p1 = __shfl_up_sync(kFull, v[1], 1);
    const i32 v31 = __shfl_sync(kFull, v[0], 31);
    if (lane == 0)
    {
        p0 = v[0];
        p1 = v31;
    }
    const i32 d0 = lane <= off ? wsub(v[0], p0) : 0, d1 = lane + 32 <= off ? wsub(v[1], p1) : 0;
    const u64 plus = (u64)__ballot_sync(kFull, d0 == 1) | ((u64)__ballot_sync(kFull, d1 == 1) << 32);
    const u64 minus = (u64)__ballot_sync(kFull, d0 == -1) | ((u64)__ballot_sync(kFull, d1 == -1) << 32);
    __syncwarp();
#pragma unroll
    for (u32 h = 0; h < 2; h++)
    {
        const u32 pos = lane + 32 * h;
        if (pos > 0 && pos <= off) out[pos] = { nc.v[pos].VP, nc.x[pos].rows };
    }
    if (lane == 0) out[0] = { plus, minus };
    __syncwarp();
    return 0;
}

// bits 1..off
__device__ __forceinline__ u64 columns_upto(u32 off) { return (off == 63 ? kAllOnes : (2ULL << off) - 1) & ~1ULL; }

// getReverseTraceFromTable's walk (Common.h:571-720) from `start`, whose score is startScore,
// up to the row above the read or, in the multiseed DP (Multi), to a seed start.  resultScore:
// the trace's OnewayTrace::score.  Returns 0 or the error status.
//
// The walk is a chain of dependent lookups, so it is bound by how long each takes: with a
// slice's record, entries and columns, the node's record, its neighbours' lengths and the read's
// bytes each loaded where they were needed, a warp waited six cycles for every instruction.  They
// are all on their way beforehand: when the walk enters slice s, the band's columns in s - 1 and
// the record and entries of s - 2 are copied to shared memory (in pieces of fixed sizes, larger
// bands are read in place), the read's rows of s - 1 loaded; when it enters a node, lanes 0-15 and
// 16-31 load the records of its first two in-neighbours, a word each.  Columns that are not kept
// are recomputed; the crossings whose slices' scores are all valid are done in place, the ones at
// a tangle's cut-off go through the general rules out of line.
// Ahead of time against on demand: one seed of a 10 kbp read 3.12 -> 2.80 ms, 50,000 extensions
// (250 Mbp) 61.5 -> 58.5 ms, the multiseed DP of 40 tangled reads 107 -> 92 ms.
template <bool Multi>
__device__ __forceinline__ int trace_walk(const DevGraph& g, i32 cost, const uint8_t* seq, u32 seqLen, u32 committed, Table& t, TraceOutT<Multi>& to,
    const ColumnUnit* store, TPos start, i32 startScore, i32& resultScore, u32 lane)
{
    int err = 0;
    const NodeCols& nc = trace_cols();
    // steps a walk may take (a trace that needs 2^32 has no room anywhere)
    const u32 guardCap = (Multi && to.counting) ? 1u << 26 : to.cap;
    const u32 guardMax = guardCap < (1u << 29) ? guardCap * 4 + 1024 : 0xffffffffu;
    resultScore = startScore;
    to.push(start, false);
    // the extraSlice of the current node-slice and its score at a row
    WS extra = fake_ws();
    auto xv = [&](u32 row) -> i32 { return Multi ? ws_value(extra, (int)row) : kIntMax; };
    u32 curSlice = 0;
    u32 curNode = 0xffffffffu;
    u32 colsUpTo = 0;             // columns 0..colsUpTo of (curSlice, curNode) are at `columns`
    const ColumnUnit* columns = nullptr;
    const Item* self = nullptr;
    i32 lastScore = kIntMax - 1;  // score of the last cell the walk looked at, where it can end
    u32 guard = 0;
    // the current slice and the one before it
    const SliceRec* recCur = nullptr;
    const SliceRec* recPrev = nullptr;
    u32 idCur = 0xffffffffu, idPrev = 0xffffffffu;     // their bands' node ids where they have a slot (lane k: entry k)
    bool slotCur = false, slotPrev = false;
    RowBytes rows { -1, -1 }, rowsNext { -1, -1 };
    u32 rowsSlice = 0, ahead = 0xffffffffu;            // the slice of rowsNext, the slice on its way to a slot
    u64 dirNext = 0;                                   // where slice dirSlice lies
    u32 dirSlice = 0xffffffffu;
    u32 keptCur = kNoColumns, keptNext = kNoColumns, keptSlice = 0;    // first unit of the copied columns of the current slice and of keptSlice
    // the current node's record (lane k: word k & 15) and its first two in-neighbours'
    u32 word = 0, nbWord = 0;
    u32 meta = 0, inOff = 0, inNb0 = 0xffffffffu, inNb1 = 0xffffffffu;

    auto corner = [&]() -> TStep
    {
        int e = 0;
        const TStep step = bt_corner<Multi>(g, seq, t, curSlice, curNode, ((i32)curSlice - 1) * 64, e, extra);
        if (e) err = e;
        return step;
    };
    auto find_cur = [&](u32 node) -> const Item*
    {
        if (!slotCur) return t.template find<Multi>(curSlice, node);
        const u32 hit = __ballot_sync(kFull, idCur == node);
        return hit ? &trace_warp().slots[curSlice % 3].items[__ffs((int)hit) - 1] : nullptr;
    };
    auto find_prev = [&](u32 node) -> const Item*
    {
        if (!slotPrev) return t.template find<Multi>(curSlice - 1, node);
        const u32 hit = __ballot_sync(kFull, idPrev == node);
        return hit ? &trace_warp().slots[(curSlice - 1) % 3].items[__ffs((int)hit) - 1] : nullptr;
    };
    // a slice's band in the lanes; false when it has no slot
    auto band_ids = [&](u32 s, const SliceRec* r, u32& id) -> bool
    {
        const SliceSlot& sl = trace_warp().slots[s % 3];
        id = 0xffffffffu;
        if (sl.slice != s) return false;
        if (lane < r->count) id = sl.items[lane].node & kNodeMask;
        return true;
    };
    // whether the read's character at `row` of the current slice matches column `off` of the node
    auto matches = [&](u32 off, u32 row) -> bool
    {
        const u32 byte = row < 32 ? (u32)__shfl_sync(kFull, rows.lo, (int)row) : (u32)__shfl_sync(kFull, rows.hi, (int)row - 32);
        const u32 base = (__shfl_sync(kFull, word, (int)(off >> 4)) >> ((off & 15) * 2)) & 3;
        const u32 mask = curNode < g.firstAmbiguous ? 1u << base : (u32)node_char_mask(g, curNode, off);
        return ((u32)s_iupac[byte & 0xff] & mask) != 0;
    };
    // pickBacktraceHorizontalCrossing (Common.h:817-884), the step out of (p.node, offset 0,
    // row off > 0) into an in-neighbour
    auto horizontal = [&](const TPos& p, u32 off) -> TStep
    {
        const i32 here = ws_value(ws_make(self->sVP, self->sVN, self->sEnd), (int)off);
        if (recCur->notValid || here > recCur->quit)
        {
            int x = 0;
            const TStep step = horizontal_step_invalid<Multi>(g, t, curSlice, curNode, self, p, off, x, extra);
            if (x) err = x;
            return step;
        }
        const i32 diagonal = here - (matches(0, off) ? 0 : 1);
        u32 degree = rec_in_degree(meta);
        if (degree >= kRecDegree) degree = g.inOff[curNode + 1] - inOff;
        #pragma unroll 1
        for (u32 e = 0; e < degree; e++)
        {
            const u32 nb = e == 0 ? inNb0 : e == 1 ? inNb1 : g.inNb[inOff + e];
            const Item* cn = find_cur(nb);
            if (!cn) continue;
            const u64 vp = cn->eVP, vn = cn->eVN;
            const i32 v0 = ws_value(ws_make(vp, vn, cn->eEnd), (int)off);
            const i32 v1 = v0 - (i32)((vp >> off) & 1) + (i32)((vn >> off) & 1);
            if (v0 < here - 1 || v1 < diagonal) { err = GA_ASSERT; return TStep { p, false }; }
            if (v0 != here - 1 && v1 != diagonal) continue;
            const u32 last = (e < 2 && g.rec ? rec_len(__shfl_sync(kFull, nbWord, (int)(16 * e + 5))) : g.len[nb]) - 1;
            return TStep { TPos { nb, last, v0 == here - 1 ? p.seq : p.seq - 1 }, true };
        }
        if (here != xval<Multi>(extra, (int)off)) err = GA_ASSERT;
        return TStep { p, false };
    };

    #pragma unroll 1
    while (!err && !to.overflow && to.back.seq != -1)
    {
        if (++guard > guardMax) { err = GA_CAPACITY; break; }
        const TPos b = to.back;
        const u32 newSlice = ((u32)b.seq >> 6) + 1;
        if (newSlice >= committed) { err = GA_ASSERT; break; }
        // a self-loop can re-enter the same node-slice further right than it was computed
        if (newSlice != curSlice || b.node != curNode || b.off > colsUpTo)
        {
            if (newSlice != curSlice)
            {
                TraceWarp& tw = trace_warp();
                copies_done();
                if (ahead != 0xffffffffu)
                {
                    SliceSlot& sl = tw.slots[ahead % 3];
                    sl.slice = sl.rec.count <= kCachedBand ? ahead : 0xffffffffu;
                    ahead = 0xffffffffu;
                    __syncwarp();
                }
                curSlice = newSlice;
                keptCur = keptSlice == curSlice ? keptNext : kNoColumns;
                keptNext = kNoColumns;
                recCur = t.rec(curSlice);
                recPrev = t.rec(curSlice - 1);
                slotCur = band_ids(curSlice, recCur, idCur);
                slotPrev = band_ids(curSlice - 1, recPrev, idPrev);
                rows = rowsSlice == curSlice ? rowsNext : row_bytes(seq, seqLen, ((int64_t)curSlice - 1) * 64, lane);
                if (curSlice >= 2)
                {
                    rowsNext = row_bytes(seq, seqLen, ((int64_t)curSlice - 2) * 64, lane);
                    rowsSlice = curSlice - 1;
                    const u32 first = slotPrev && recPrev->count ? (u32)tw.slots[(curSlice - 1) % 3].items[0].minScore : kNoColumns;
                    if (first != kNoColumns)
                    {
                        keptNext = first;
                        keptSlice = curSlice - 1;
                        ColumnUnit* to16 = tw.kept[keptSlice & 1];
#pragma unroll
                        for (u32 k = 0; k < kKeptUnits; k += 32) copy_ahead(to16 + k + lane, store + first + k + lane);
                    }
                    ahead = curSlice - 2;
                    SliceSlot& sl = tw.slots[ahead % 3];
                    sl.slice = 0xffffffffu;
                    const uint4* from = (const uint4*)(t.arena + (dirSlice == ahead ? dirNext : t.dir[ahead]));
                    if (ahead > 0)
                    {
                        dirSlice = ahead - 1;
                        dirNext = t.dir[dirSlice];
                    }
                    #pragma unroll 1
                    for (u32 k = lane; k < 2 + 4 * kCachedBand; k += 32) copy_ahead((uint4*)&sl + k, from + k);
                }
            }
            if (b.node != curNode)
            {
                curNode = b.node;
                if (g.rec && curNode == inNb0) word = __shfl_sync(kFull, nbWord, (int)(lane & 15));
                else if (g.rec && curNode == inNb1) word = __shfl_sync(kFull, nbWord, (int)(16 + (lane & 15)));
                else if (g.rec) word = __ldg((const u32*)(g.rec + curNode) + (lane & 15));
                else
                {
                    NodeRec x;
                    gather_record(g, curNode, x);
                    word = ((const u32*)&x)[lane & 15];
                }
                meta = __shfl_sync(kFull, word, 5);
                inOff = __shfl_sync(kFull, word, 6);
                inNb0 = __shfl_sync(kFull, word, 8);
                inNb1 = __shfl_sync(kFull, word, 9);
                const u32 nb = lane < 16 ? inNb0 : inNb1;
                if (g.rec && nb < g.N) nbWord = __ldg((const u32*)(g.rec + nb) + (lane & 15));
            }
            self = find_cur(curNode);
            if (!self) { err = GA_ASSERT; break; }
            if (Multi) extra = (self->node & kSeedStart) ? seed_ws(((int64_t)curSlice - 1) * 64, seqLen, cost, lane) : fake_ws();
            const u32 at = (u32)self->minScore;
            if (at != kNoColumns)
            {
                columns = keptCur != kNoColumns && at - keptCur <= kKeptUnits - rec_len(meta) ? trace_warp().kept[curSlice & 1] + (at - keptCur)
                    : store + at;
                colsUpTo = 63;
            }
            else
            {
                // the recomputed columns lie where the kept ones are copied to
                copies_done();
                keptCur = keptNext = kNoColumns;
                err = recompute<Multi>(g, cost, t, seq, seqLen, curSlice, curNode, b.off, extra, lane);
                if (err) break;
                columns = trace_warp().columns;
                colsUpTo = b.off;
            }
        }
        const bool seeded = Multi && extra.end != kIntMax;
        const i32 sj = ((i32)curSlice - 1) * 64;
        if (b.off >= rec_len(meta)) { err = GA_ASSERT; break; }
        const u32 row = mod64(b.seq);
        // the walk ends above the read, so from row 0 or up column 0 to it, or at a seed start
        if (seeded) lastScore = nc.value(b.off, row);
        if (row == 0)
        {
            const i32 first = ws_value(ws_make(self->sVP, self->sVN, self->sEnd), 0);
            const ColumnUnit top = columns[0];
            if (!seeded) lastScore = first + popc64(top.x & columns_upto(b.off)) - popc64(top.y & columns_upto(b.off));
            if (b.off == 0)
            {
                TStep bt = corner();
                if (err) break;
                if (seeded && tpos_eq(bt.pos, b) && !bt.sw && nc.value(bt.pos.off, mod64(bt.pos.seq)) == xv(mod64(bt.pos.seq))) break;
                if (seeded && tpos_eq(bt.pos, b) && !bt.sw && nc.value(bt.pos.off, mod64(bt.pos.seq)) == ws_before(extra)) break;
                to.push(bt.pos, bt.sw);
                if (!to.overflow && trace_circular(to.items, to.ring, to.n, Multi && to.counting)) { err = GA_ASSERT; break; }
                continue;
            }
            const Item* pself = find_prev(curNode);
            if (!pself)
            {
                to.push_run(TPos { curNode, b.off - 1, b.seq }, -1, 0, b.off);
                continue;
            }
            // pickBacktraceVerticalCrossing (Common.h:886-934)
            // step left along row 0 while the score falls by one per column: the run ends at the
            // highest column at or below b.off without a +1 delta (column 0 has none)
            TPos p = b;
            p.off = 63 - (u32)__clzll((long long)(~top.x & (columns_upto(b.off) | 1)));
            TStep second;
            if (p.off == 0) second = corner();
            else
            {
                const i32 here = seeded ? nc.value(p.off, 0) : first + popc64(top.x & columns_upto(p.off)) - popc64(top.y & columns_upto(p.off));
                second = vertical_step<Multi>(recCur, recPrev, pself, p, here, matches(p.off, 0), err, extra);
            }
            if (err) break;
            if (seeded && second.pos.seq == b.seq && nc.value(second.pos.off, mod64(second.pos.seq)) == xv(mod64(second.pos.seq))) break;
            if (p.off != b.off) to.push_run(TPos { p.node, b.off - 1, p.seq }, -1, 0, b.off - p.off);
            if (tpos_eq(second.pos, to.back)) { err = GA_ASSERT; break; }
            to.push(second.pos, second.sw);
            continue;
        }
        if (b.off == 0)
        {
            // pickBacktraceHorizontalCrossing (Common.h:817-884)
            // step up column 0 while its score falls by one per row (the start column's VP
            // bits): the run ends at the highest row at or below this one whose bit is clear
            // (row 0 always ends it)
            TPos p = b;
            const u64 stops = (~self->sVP | 1ULL) & (row == 63 ? kAllOnes : ((2ULL << row) - 1));
            const u32 off = 63 - (u32)__clzll((long long)stops);
            p.seq -= (i32)(row - off);
            if (!seeded && off == 0) lastScore = ws_value(ws_make(self->sVP, self->sVN, self->sEnd), (int)row);
            TStep second = off == 0 ? corner() : horizontal(p, off);
            if (err) break;
            if (seeded && second.pos.node == b.node && !second.sw && nc.value(second.pos.off, mod64(second.pos.seq)) == xv(mod64(second.pos.seq))) break;
            if (p.seq != b.seq) to.push_run(TPos { p.node, p.off, b.seq - 1 }, 0, -1, (u32)(b.seq - p.seq));
            if (tpos_eq(second.pos, to.back)) { err = GA_ASSERT; break; }
            to.push(second.pos, second.sw);
            if (!to.overflow && trace_circular(to.items, to.ring, to.n, Multi && to.counting)) { err = GA_ASSERT; break; }
            continue;
        }
        // pickBacktraceInside (Common.h:770-815): up while the column's delta is +1, else
        // diagonally where that step is open, else left.  Inside a node-slice the steps are
        // bits of its columns, so a run of diagonal steps is found in one ballot, lane k testing
        // the cell k steps down the diagonal, and a run of up steps is a leading-one count.
        // Cell by cell (two scores carried, every lane the same) this walk took 21.9k of the
        // traceback's 58.8k cycles per 64-row slice of an extension alone.
        if (!seeded)
        {
            u32 hori = b.off;
            u32 vert = row;
            #pragma unroll 1
            while (hori > 0 && vert > 0 && !to.overflow)
            {
                const u32 most = hori < vert ? hori : vert;
                ColumnUnit c { 0, 0 };
                if (lane < most) c = columns[hori - lane];
                const u64 bit = 1ULL << ((vert - lane) & 63);
                const u32 run = (u32)__ffs((int)~__ballot_sync(kFull, (c.y & ~c.x & bit) != 0));
                if (run != 1)
                {
                    // __ffs(0) = 0: all 32 lanes' steps are diagonal
                    const u32 count = run ? run - 1 : 32;
                    to.push_run(TPos { b.node, hori - 1, sj + (i32)vert - 1 }, -1, -1, count);
                    hori -= count;
                    vert -= count;
                    continue;
                }
                const u64 vp = __shfl_sync(kFull, c.x, 0);
                if ((vp >> vert) & 1)
                {
                    const u32 count = up_run(vp, vert);
                    to.push_run(TPos { b.node, hori, sj + (i32)vert - 1 }, 0, -1, count);
                    vert -= count;
                    continue;
                }
                hori--;
                to.push(TPos { b.node, hori, sj + (i32)vert }, false);
            }
            continue;
        }
        // A seed start's columns are merged with its seed column, so their steps are not the
        // recurrence's bits: cell by cell, the four neighbouring scores carried incrementally.
        // A vertical step moves up one row in both columns (score(r-1) = score(r) - VP_r +
        // VN_r); a diagonal or horizontal step makes the left column current and loads the next
        // one.  The read/graph match of a cell is bit `row` of the column's match mask (the
        // fill's Eq), which is GraphAlignerCommon::characterMatch for every read and graph
        // character.
        {
            u32 hori = b.off;
            u32 vert = row;
            // the recomputation left each column's match mask (the fill's Eq) in eqcol
            const u64* eqcol = nc.eqcol;
            if (hori > 0 && vert > 0)
            {
                WS colH = nc.column(hori);
                WS colL = nc.column(hori - 1);
                i32 here = ws_value(colH, (int)vert);
                i32 left = ws_value(colL, (int)vert);
                u64 eqH = eqcol[hori];
                #pragma unroll 1
                while (true)
                {
                    const i32 vs = here - (i32)((colH.VP >> vert) & 1) + (i32)((colH.VN >> vert) & 1);
                    const i32 ds = left - (i32)((colL.VP >> vert) & 1) + (i32)((colL.VN >> vert) & 1);
                    const bool eq = (eqH >> vert) & 1;
                    if (vs == here - 1)
                    {
                        vert--;
                        to.push(TPos { b.node, hori, sj + (i32)vert }, false);
                        here = vs;
                        left = ds;
                    }
                    else if (ds == here - (eq ? 0 : 1))
                    {
                        hori--;
                        vert--;
                        to.push(TPos { b.node, hori, sj + (i32)vert }, false);
                        here = ds;
                        colH = colL;
                        if (hori > 0)
                        {
                            colL = nc.column(hori - 1);
                            left = ws_value(colL, (int)vert);
                            eqH = eqcol[hori];
                        }
                    }
                    else if (left == here - 1)
                    {
                        hori--;
                        to.push(TPos { b.node, hori, sj + (i32)vert }, false);
                        here = left;
                        colH = colL;
                        if (hori > 0)
                        {
                            colL = nc.column(hori - 1);
                            left = ws_value(colL, (int)vert);
                            eqH = eqcol[hori];
                        }
                    }
                    else
                    {
                        if (here != xv(vert)) err = GA_ASSERT;
                        break;
                    }
                    if (to.overflow || hori == 0 || vert == 0) break;
                }
            }
            if (err || to.overflow) break;
            if (nc.value(to.back.off, mod64(to.back.seq)) == xv(mod64(to.back.seq))) break;
        }
    }
    // the next trace writes where copies may still be on their way
    copies_done();
    if (!err && !to.overflow)
    {
        if (resultScore < lastScore) err = GA_ASSERT;
        resultScore -= lastScore;
    }
    return err;
}

__device__ void trace_extension(const TraceArgs& a, u32 ext, const ExtState& st, u32 lane)
{
    const DevGraph& g = a.g;
    u64* out = a.traceItems + a.traceOffset[ext];
    const u32 cap = a.traceCap[ext];
    if (lane == 0 && a.cellSteps) a.cellSteps[ext] = st.steps;
    if (st.status != GA_OK)
    {
        if (lane == 0)
        {
            a.status[ext] = st.status;
            a.score[ext] = 0;
            a.traceLen[ext] = 0;
        }
        return;
    }
    const uint8_t* seq = a.seq + a.seqOff[ext];
    const u32 seqLen = a.seqLen[ext];
    Table t;
    t.arena = a.arena;
    t.dir = (const u64*)(a.arena + st.dir);
    t.lane = lane;
    t.init();
    const NodeCols& nc = trace_cols();
    TraceOut to;
    to.items = out;
    to.ring = trace_warp().ring;
    to.cap = cap;
    to.n = 0;
    to.lane = lane;
    to.overflow = false;
    int err = 0;
    i32 resultScore = 0;
    const EndCell ec = end_cell(g, a.cost, a.arena, t, st.committed, seq, seqLen, lane);
    err = ec.err;
    if (!err)
    {
        // getReverseTraceFromTable (Common.h:571-758)
        TPos start = TPos { ec.node, ec.nodeOffset, ec.j + (i32)ec.bvOffset };
        i32 startScore = nc.value(ec.nodeOffset, ec.bvOffset);
        err = trace_walk<false>(g, a.cost, seq, seqLen, st.committed, t, to, a.store, start, startScore, resultScore, lane);
        if (!err && !to.overflow)
        {
            TraceOut end = to;
            err = row_above(g, t, end);
            to = end;
        }
    }
    int status = err ? err : (to.overflow ? GA_CAPACITY : GA_OK);
    if (lane == 0)
    {
        a.status[ext] = status;
        a.score[ext] = status == GA_OK ? resultScore : 0;
        a.traceLen[ext] = status == GA_OK ? to.n : 0;
    }
}

// The multiseed DP's best X-score of node in committed slice s (read from the arena); false
// when the node is not in the slice's band
__device__ __forceinline__ bool slice_node_max(const uint8_t* arena, const u64* dir, u32 s, u32 node, u32 lane, i32& out)
{
    const SliceRec* r = (const SliceRec*)(arena + dir[s]);
    const int k = rec_index<true>(r, rec_ids(r), node, lane);
    if (k < 0) return false;
    out = rec_node_max(r)[k];
    return true;
}

// getLocalMaximaTracesFromTable's (Common.h:355-494) local-maximum test of `node` in committed
// slice cs, whose best X-score there is `score`: not below its own in the slices above and
// below, nor below its in-neighbours' in this slice and the one above or its out-neighbours'
// in this slice and the one below.
__device__ bool ms_local_max(const DevGraph& g, const uint8_t* arena, const u64* dir, u32 cs, u32 last, u32 node, i32 score, u32 lane)
{
    i32 other;
    if (slice_node_max(arena, dir, cs - 1, node, lane, other) && other > score) return false;
    if (cs < last && slice_node_max(arena, dir, cs + 1, node, lane, other) && other >= score) return false;
#pragma unroll 1
    for (u32 e = g.inOff[node]; e < g.inOff[node + 1]; e++)
    {
        const u32 nb = g.inNb[e];
        if (slice_node_max(arena, dir, cs, nb, lane, other) && other > score) return false;
        if (slice_node_max(arena, dir, cs - 1, nb, lane, other) && other > score) return false;
    }
#pragma unroll 1
    for (u32 e = g.outOff[node]; e < g.outOff[node + 1]; e++)
    {
        const u32 nb = g.outNb[e];
        if (slice_node_max(arena, dir, cs, nb, lane, other) && other > score) return false;
        if (cs < last && slice_node_max(arena, dir, cs + 1, nb, lane, other) && other > score) return false;
    }
    return true;
}

// The candidates of read r in getLocalMaximaTracesFromTable's order (slices from the last,
// band order within a slice): band nodes whose best X-score is positive, reaches the
// multimap fraction of the slice's best as the fill left it and is a local maximum.  The
// slice bests only rise as traces are taken, so the traces the read keeps are among these.
// Of these, the ones in part `part` of the read's slices (kCandParts equal runs, the last slices
// first): write = false counts them, write = true fills their place in the read's run of the list.
// A warp to a read, 40 reads of 313 slices took 8.9 ms each time.
__device__ void ms_candidates(const MultiTraceArgs& a, u32 r, const ExtState& st, u32 part, bool write, u32 lane)
{
    u32 c = 0;
    const u64 base = write ? a.candBegin[r] + a.candPart[(u64)r * kCandParts + part] : 0;
    if (st.status == GA_OK)
    {
        const u64* dir = (const u64*)(a.arena + st.dir);
        const i32* sliceMax = (const i32*)(a.arena + st.aux);
        const u32 last = st.committed - 1;
        const u32 run = (last + kCandParts - 1) / kCandParts;
        const u32 from = part * run < last ? last - part * run : 0, to = (part + 1) * run < last ? last - (part + 1) * run : 0;
#pragma unroll 1
        for (u32 cs = from; cs > to; cs--)
        {
            const SliceRec* cr = (const SliceRec*)(a.arena + dir[cs]);
            if (cr->maxX <= 0) continue;
            const u32 n = cr->count;
            const u32* ids = rec_ids(cr);
            const Item* items = rec_items(cr);
            const i32* nodeMax = rec_node_max(cr);
            const double threshold = (double)sliceMax[cs] * a.multimapScoreFraction;
#pragma unroll 1
            for (u32 b = 0; b < n; b += 32)
            {
                const u32 k = b + lane;
                bool pass = false;
                if (k < n)
                {
                    const i32 score = nodeMax[k];
                    pass = (items[k].node & kExists) && score > 0 && !((double)score < threshold);
                }
                u32 m = __ballot_sync(kFull, pass);
#pragma unroll 1
                while (m)
                {
                    const u32 kk = b + __ffs((int)m) - 1;
                    m &= m - 1;
                    const u32 node = ids[kk];
                    const i32 score = nodeMax[kk];
                    if (!ms_local_max(a.g, a.arena, dir, cs, last, node, score, lane)) continue;
                    if (write && lane == 0 && base + c < a.candCap)
                    {
                        MsCand x {};
                        x.read = r;
                        x.slice = cs;
                        x.index = kk;
                        x.score = score;
                        x.slot = kNoSlot;
                        a.cands[base + c] = x;
                    }
                    c++;
                }
            }
        }
    }
    if (!write && lane == 0) a.candPart[(u64)r * kCandParts + part] = c;
    __syncwarp();
}

// The first cell of a candidate's trace (getLocalMaximaTracesFromTable): among the node's
// columns, recomputed with its seed start, the cell of greatest row that scores the node's
// best X-score (the first column on ties); a cell above it is GA_ASSERT.
__device__ int ms_start_cell(const MultiTraceArgs& a, Table& t, const uint8_t* seq, u32 seqLen, const MsCand& c,
    TPos& start, i32& startScore, u32 lane)
{
    const DevGraph& g = a.g;
    const SliceRec* cr = (const SliceRec*)(a.arena + t.dir[c.slice]);
    const Item* items = rec_items(cr);
    const u32 node = items[c.index].node & kNodeMask;
    const i32 j = ((i32)c.slice - 1) * 64;
    if (!slice_masks(seq, seqLen, c.slice, lane)) return GA_ASSERT;
    const WS extra = (items[c.index].node & kSeedStart) ? seed_ws(j, seqLen, a.cost, lane) : fake_ws();
    int err = recalc<true>(g, a.cost, t, c.slice, node, lane, 63, extra);
    if (err) return err;
    const NodeCols& nc = trace_cols();
    const i32 score = c.score;
    const int cells = (i32)seqLen - j < 64 ? (i32)seqLen - j : 64;
    const u32 L = g.len[node];
    bool bad = false;
    int candOff = -1;
    u32 candCol = 0xffffffffu;
#pragma unroll 1
    for (u32 h = 0; h < 2; h++)
    {
        const u32 i = lane + 32 * h;
        if (i >= L || bad) continue;
        const WS cw = nc.column(i);
        const i32 mx = ws_max_xscore(cw, (i32)j, a.cost, cells, kAllOnes);
        if (mx > score) { bad = true; continue; }
        if (mx != score) continue;
#pragma unroll 1
        for (int off = 63; off >= 0; off--)
        {
            if (j + off >= (i32)seqLen) continue;
            const i32 here = ws_xscore(cw, (i32)j, off, a.cost);
            if (here > score) { bad = true; break; }
            if (here == score && off > candOff)
            {
                candOff = off;
                candCol = i;
            }
        }
    }
    if (__ballot_sync(kFull, bad)) return GA_ASSERT;
    const int gOff = __reduce_max_sync(kFull, candOff);
    const u32 gCol = __reduce_min_sync(kFull, candOff == gOff ? candCol : 0xffffffffu);
    if (gOff < 0 || j + gOff >= (i32)seqLen) return GA_ASSERT;
    start = TPos { node, gCol, j + gOff };
    startScore = nc.value(gCol, gOff);
    return 0;
}

// One candidate's trace (getReverseTraceFromTable to a seed start).  write = false: finds the
// first cell and walks the trace only counting its items, recording its length, score, read
// span and last cell.  write = true (a kept trace of a read whose traces all fit and, with
// exact room, that removeDuplicateTraces kept): walks it again into the read's output at
// the place the read's selection (or the host, with exact room) gave it.
__device__ void ms_trace_cand(const MultiTraceArgs& a, MsCand* cp, bool write, u32 lane)
{
    const MsCand c = *cp;
    const u32 r = c.read;
    if (write)
    {
        // the read's status can change under other warps (a kept trace of it that failed)
        int readStatus = 0;
        if (lane == 0) readStatus = a.status[r];
        readStatus = __shfl_sync(kFull, readStatus, 0);
        if (c.slot == kNoSlot || readStatus != GA_OK) return;
    }
    const ExtState st = a.states[r];
    const uint8_t* seq = a.seq + a.seqOff[r];
    const u32 seqLen = a.seqLen[r];
    Table t;
    t.arena = a.arena;
    t.dir = (const u64*)(a.arena + st.dir);
    t.lane = lane;
    t.init();
    TPos start;
    i32 startScore = 0;
    int err = 0;
    if (write)
    {
        start = TPos { c.startNode, c.startOff, (i32)c.startSeq };
        startScore = c.startScore;
    }
    else
    {
        err = ms_start_cell(a, t, seq, seqLen, c, start, startScore, lane);
    }
    const bool exact = a.traceBase != nullptr;
    // exact room: the kept trace's place after the duplicates went, or none
    const u64 kept = exact && write ? a.traceBase[r] + c.slot : 0;
    const u32 outSlot = exact && write ? a.keptSlot[kept] : 0;
    if (exact && write && outSlot == kNoSlot) return;
    TraceOutT<true> to;
    to.items = write ? a.traceItems + (exact ? a.keptItem[kept] : a.traceOffset[r] + c.outOff) : nullptr;
    to.ring = trace_warp().ring;
    to.lane = lane;
    to.counting = !write;
    to.cap = write ? c.len : 0xffffffffu;
    to.n = 0;
    to.overflow = false;
    to.back = start;
    i32 traceScore = 0;
    if (!err)
    {
        err = trace_walk<true>(a.g, a.cost, seq, seqLen, st.committed, t, to, a.store, start, startScore, traceScore, lane);
            // a walk past its step guard or its counted length is broken, not short of room
        if (err == GA_CAPACITY || (!err && to.overflow)) err = GA_ASSERT;
        if (!err && (to.back.seq < 0 || start.seq < to.back.seq)) err = GA_ASSERT;
    }
    if (lane == 0)
    {
        if (!write)
        {
            cp->startNode = start.node;
            cp->startOff = start.off;
            cp->startSeq = start.seq;
            cp->startScore = startScore;
            cp->err = err;
            cp->traceScore = traceScore;
            cp->len = err ? 0 : to.n;
            cp->traceStart = to.back.seq;
            cp->lastNode = to.back.node;
            cp->lastOff = to.back.off;
            cp->state = kTraced;
        }
        else if (err || to.n != c.len || traceScore != c.traceScore)
        {
            // the walk differs from its count only where the written trace's full circularity
            // check (the counting walk checks the ring) stops it
            a.status[r] = err ? err : GA_ASSERT;
            a.numTraces[r] = 0;
        }
        else
        {
            const u64 slot = exact ? outSlot : (u64)r * a.maxTraces + c.slot;
            a.traceScore[slot] = traceScore;
            a.traceStart[slot] = exact ? a.itemBias + a.keptItem[kept] : c.outOff;
            a.traceLen[slot] = to.n;
        }
    }
    __syncwarp();
}

// getLocalMaximaTracesFromTable's selection for read r, one round: its candidates in order
// from the cursor.  A candidate below the multimap fraction of its slice's best (as raised so
// far) is passed over for good, the slice bests only rise.  One that reaches it is kept once
// its trace has been walked, and raises the best of the slices its trace spans beyond its
// first 5 %; the first one whose walk is still to come stops the round.  Then the read queues
// that walk and up to window - 1 more of the candidates after it that the slice bests do not
// yet rule out.  Kept traces get their place in the read's output while they fit its room
// (max_traces, trace_capacity); past that they are only counted, and the read reports the
// room it needs.  With exact room (a.traceBase) every kept trace gets its place, and the read
// reports the items they take.  A kept trace that failed fails the read.
__device__ void ms_resolve(const MultiTraceArgs& a, u32 r, const ExtState& st, u32 lane)
{
    MsSel* sp = a.sel + r;
    if (sp->done) return;
    if (st.status != GA_OK)
    {
        if (lane == 0)
        {
            if (a.cellSteps) a.cellSteps[r] = st.steps;
            a.status[r] = st.status;
            a.numTraces[r] = 0;
            sp->done = 1;
        }
        __syncwarp();
        return;
    }
    MsSel sel = *sp;
    i32* sliceMax = (i32*)(a.arena + st.aux);
    const bool exact = a.traceBase != nullptr;
    const u64 cap = exact ? ~0ULL : a.traceCap[r];
    const u32 maxTraces = exact ? 0xffffffffu : a.maxTraces;
    const u64 begin = a.candBegin[r];
    const u32 count = a.candCount[r];
    int err = 0;
    u32 i = sel.cursor;
#pragma unroll 1
    for (; i < count; i++)
    {
        MsCand* cp = a.cands + begin + i;
        const u32 cs = cp->slice;
        const i32 score = cp->score;
        if ((double)score < (double)sliceMax[cs] * a.multimapScoreFraction) continue;
        if (cp->state != kTraced) break;
        if (cp->err)
        {
            err = cp->err;
            break;
        }
        const u32 len = cp->len;
        if (!sel.full && (sel.nt >= maxTraces || len > cap - sel.used)) sel.full = 1;
        if (!sel.full)
        {
            if (lane == 0)
            {
                cp->slot = sel.nt;
                cp->outOff = sel.used;
            }
            sel.used += len;
            sel.nt++;
        }
        sel.items += len;
        sel.traces++;
        const int64_t traceEnd = cp->startSeq, traceStart = cp->traceStart;
        const u32 startSlice = (u32)(((double)(traceEnd - traceStart) * 0.05 + (double)traceStart + 64 - 1) / 64 + 1);
        __syncwarp();
#pragma unroll 1
        for (u32 k = startSlice + lane; k < cs; k += 32) sliceMax[k] = imax(sliceMax[k], score);
        __syncwarp();
    }
    sel.cursor = i;
    if (err || i == count)
    {
        if (lane == 0)
        {
            const bool room = !sel.full;
            if (a.cellSteps) a.cellSteps[r] = st.steps;
            a.status[r] = err ? err : (room ? GA_OK : kMsRoom);
            a.numTraces[r] = (err || !room) ? 0 : sel.nt;
            // with exact room: the items the read's traces take
            if (a.itemsNeeded) a.itemsNeeded[r] = err ? 0 : (exact ? sel.used : (!room ? sel.items : 0));
            if (a.tracesNeeded) a.tracesNeeded[r] = (!err && !room) ? sel.traces : 0;
            sel.done = 1;
            *sp = sel;
        }
        __syncwarp();
        return;
    }
    // the walk the read waits for, and a few after it that may be kept too
    u32 queued = 0;
#pragma unroll 1
    for (u32 j = i; j < count && queued < a.window; j++)
    {
        MsCand* cp = a.cands + begin + j;
        if (cp->state != kUntraced) continue;
        if ((double)cp->score < (double)sliceMax[cp->slice] * a.multimapScoreFraction) continue;
        if (lane == 0)
        {
            cp->state = kQueued;
            a.work[atomicAdd(a.workCount, 1u)] = (u32)(begin + j);
        }
        queued++;
    }
    if (lane == 0) *sp = sel;
    __syncwarp();
}

// The next extension for this warp from the work counter, or false when none is left;
// with a filter only extensions whose previous status is GA_CAPACITY are taken.
__device__ __forceinline__ bool next_extension(u32* counter, u32 num, const u32* order, const i32* prevStatus, u32 lane, u32& ext)
{
#pragma unroll 1
    while (true)
    {
        u32 k = 0;
        if (lane == 0) k = atomicAdd(counter, 1u);
        k = __shfl_sync(kFull, k, 0);
        if (k >= num) return false;
        ext = order ? order[k] : k;
        if (!prevStatus || prevStatus[ext] == GA_CAPACITY) return true;
    }
}

// The fill: a warp takes the next extension of the longest-first order, fills its DP table
// into the arena and records where it is, then takes the next.
template <class Tables>
__device__ __forceinline__ void fill_extensions(const FillArgs& fa, u32* counter)
{
    load_iupac_table();
    const u32 lane = threadIdx.x & 31;
    Tables t(fa, (u64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane);
    ArenaCursor& arena = fill_warp().arena;
    arena = { 0, 0, 0, 0, 0, fa.store == nullptr ? 1u : 0u };
    __syncwarp();
    u32 ext;
#pragma unroll 1
    while (next_extension(counter, fa.num, fa.order, fa.prevStatus, lane, ext))
    {
        __syncwarp();
        const ExtState st = fill_extension(fa, t, arena, ext, lane);
        if (lane == 0) fa.states[ext] = st;
    }
    if (lane == 0 && arena.used) atomicAdd(fa.arenaCursor + 1, (unsigned long long)arena.used);
}

__global__ void __launch_bounds__(128, 4) fill_kernel(const __grid_constant__ FillArgs fa, u32* counter) { fill_extensions<SmallTables<true>>(fa, counter); }
// the same for graphs that share component numbers
__global__ void __launch_bounds__(128, 4) fill_shared_kernel(const __grid_constant__ FillArgs fa, u32* counter) { fill_extensions<SmallTables<false>>(fa, counter); }

// The extensions that the fill above handed on, each from the slice it stopped at.
__global__ void __launch_bounds__(128, 1) fill_medium_kernel(const __grid_constant__ FillArgs fa, u32* counter)
{
    load_iupac_table();
    const u32 lane = threadIdx.x & 31;
    const u32 handed = fa.resumeCount[0] < fa.resumeCap ? fa.resumeCount[0] : fa.resumeCap;
    if (handed == 0) return;
    MediumTables t(fa, 0, lane);
    ArenaCursor& arena = fill_warp().arena;
    arena = { 0, 0, 0, 0, 0, fa.store == nullptr ? 1u : 0u };
    __syncwarp();
    u32 k;
#pragma unroll 1
    while (next_extension(counter, handed, nullptr, nullptr, lane, k))
    {
        __syncwarp();
        const ResumeRec& r = fa.resume[k];
        t.restart();
        t.next();
        #pragma unroll 1
        for (u32 e = 0; e < r.count; e++)
        {
            const u32 node = r.band[e].node & kNodeMask;
            const int at = t.enter((u32)t.slot_of(fa.g, node, 0));
            t.band()[at] = r.band[e];
        }
        __syncwarp();
        FillState f = r.state;
        const ExtState st = fill_slices(fa, t, arena, r.ext, f, lane);
        if (lane == 0) fa.states[r.ext] = st;
    }
    if (lane == 0 && arena.used) atomicAdd(fa.arenaCursor + 1, (unsigned long long)arena.used);
}
// the extensions of a graph that is mostly cycles, with the medium tables from the start
__global__ void __launch_bounds__(32, 6) fill_tangled_kernel(const __grid_constant__ FillArgs fa, u32* counter) { fill_extensions<MediumTables>(fa, counter); }
__global__ void __launch_bounds__(128, 4) fill_large_kernel(const __grid_constant__ FillArgs fa, u32* counter) { fill_extensions<LargeTables>(fa, counter); }

// The traceback: a warp takes the next filled extension and walks its table back.  Four blocks of
// 128 registers a thread on an SM: with six of 80 the walk's state spills, and 50,000 extensions
// (250 Mbp) take 52.9 ms instead of 48.0, with five of 96 49.5.  Its
// shared memory holds the recomputed columns, the match masks and the trace staging.
__global__ void __launch_bounds__(128, 4) trace_kernel(const __grid_constant__ TraceArgs ta, u32* counter)
{
    load_iupac_table();
    const u32 lane = threadIdx.x & 31;
    u32 ext;
#pragma unroll 1
    while (next_extension(counter, ta.num, ta.order, ta.prevStatus, lane, ext))
    {
        __syncwarp();
        trace_extension(ta, ext, ta.states[ext], lane);
    }
}


// The multiseed DP's fill: a warp takes the next read and fills its whole DP table; its
// frontier tables and per-node X-scores live in the global workspace.  A batch has few reads and waits
// for its longest one's chain, so a block is one warp, with all the registers it can use: 40 tangled reads
// of 20 kbp 57.8 -> 53.7 ms with the two functions taken out of line (seed_ws, seeded_columns), 20.5 -> 17.3
// on a variation graph; 1,000 reads take as long as with four blocks of four warps on an SM.
__global__ void __launch_bounds__(32, 8) fill_multiseed_kernel(const __grid_constant__ FillArgs fa, u32* counter)
{
    load_iupac_table();
    const u32 lane = threadIdx.x & 31;
    LargeTables t(fa, (u64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane);
    ArenaCursor& arena = fill_warp().arena;
    arena = { 0, 0, 0, 0, 0, fa.store == nullptr ? 1u : 0u };
    __syncwarp();
    u32 r;
#pragma unroll 1
    while (next_extension(counter, fa.num, fa.order, fa.prevStatus, lane, r))
    {
        __syncwarp();
        const ExtState st = fill_multiseed(fa, t, arena, r, lane);
        if (lane == 0) fa.states[r] = st;
    }
    if (lane == 0 && arena.used) atomicAdd(fa.arenaCursor + 1, (unsigned long long)arena.used);
}

// The candidates of the multiseed traceback (write = false: counted, write = true: listed), a
// warp per part of a read.
__global__ void __launch_bounds__(128, 6) ms_candidates_kernel(const __grid_constant__ MultiTraceArgs ta, u32* counter, int write)
{
    const u32 lane = threadIdx.x & 31;
#pragma unroll 1
    while (true)
    {
        u32 k = 0;
        if (lane == 0) k = atomicAdd(counter, 1u);
        k = __shfl_sync(kFull, k, 0);
        if (k >= ta.num * kCandParts) break;
        const u32 r = ta.order[k / kCandParts];
        if (ta.prevStatus && ta.prevStatus[r] != GA_CAPACITY) continue;
        ms_candidates(ta, r, ta.states[r], k % kCandParts, write != 0, lane);
    }
}

// Each read's run of the candidate list and its parts' places in it, a warp per read (lane k:
// part k).
__global__ void ms_reserve_kernel(const __grid_constant__ MultiTraceArgs ta)
{
    static_assert(kCandParts == 32, "a part per lane");
    const u32 lane = threadIdx.x & 31;
    const u32 k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (k >= ta.num) return;
    const u32 r = ta.order[k];
    if (ta.prevStatus && ta.prevStatus[r] != GA_CAPACITY) return;
    const u32 own = ta.candPart[(u64)r * kCandParts + lane];
    u32 sum = own;
#pragma unroll
    for (u32 d = 1; d < 32; d <<= 1)
    {
        const u32 up = __shfl_up_sync(kFull, sum, d);
        if (lane >= d) sum += up;
    }
    ta.candPart[(u64)r * kCandParts + lane] = sum - own;
    if (lane == 31)
    {
        ta.candCount[r] = sum;
        ta.candBegin[r] = sum ? atomicAdd(ta.candTotal, (unsigned long long)sum) : 0;
    }
}

// Exact room: each kept trace of a read that finished GA_OK, summarised for the host's
// removeDuplicateTraces, a thread per candidate.
__global__ void ms_keys_kernel(MultiTraceArgs ta)
{
    const u64 total = *ta.candTotal < ta.candCap ? *ta.candTotal : ta.candCap;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (u64)gridDim.x * blockDim.x)
    {
        const MsCand& c = ta.cands[i];
        if (c.slot == kNoSlot || ta.status[c.read] != GA_OK) continue;
        MsKey k;
        k.first = c.startSeq;
        k.last = c.traceStart;
        k.lastNode = c.lastNode;
        k.lastOff = c.lastOff;
        k.score = c.traceScore;
        k.len = c.len;
        ta.keys[ta.traceBase[c.read] + c.slot] = k;
    }
}

__global__ void __launch_bounds__(128, 6) ms_resolve_kernel(const __grid_constant__ MultiTraceArgs ta, u32* counter)
{
    const u32 lane = threadIdx.x & 31;
    u32 r;
#pragma unroll 1
    while (next_extension(counter, ta.num, ta.order, ta.prevStatus, lane, r))
    {
        __syncwarp();
        ms_resolve(ta, r, ta.states[r], lane);
    }
}

// The candidates' traces, a warp per candidate (write = false: the round's queued walks,
// counted; write = true: the kept ones written).  A read's traces spread over as many warps
// as it has walks in the round.
__global__ void __launch_bounds__(128, 4) ms_trace_kernel(const __grid_constant__ MultiTraceArgs ta, u32* counter, int write)
{
    load_iupac_table();
    const u32 lane = threadIdx.x & 31;
    const u64 total = write ? (*ta.candTotal < ta.candCap ? *ta.candTotal : ta.candCap) : *ta.workCount;
#pragma unroll 1
    while (true)
    {
        u32 i = 0;
        if (lane == 0) i = atomicAdd(counter, 1u);
        i = __shfl_sync(kFull, i, 0);
        if (i >= total) break;
        __syncwarp();
        ms_trace_cand(ta, ta.cands + (write ? i : ta.work[i]), write != 0, lane);
    }
}
}

// dynamic shared memory of a block of the fill kernels and of the traceback kernels
static size_t fill_smem(int warpsPerBlock, gadev::FillTables tables)
{
    const size_t own = tables == gadev::FillTables::Small ? sizeof(gadev::SmallSpace)
        : tables == gadev::FillTables::Medium ? (size_t)gadev::wspace_bytes(gadev::medium_caps()) : 0;
    return (sizeof(gadev::FillWarp) + own) * warpsPerBlock;
}
static auto fill_function(gadev::FillTables tables, bool unique)
{
    return tables == gadev::FillTables::Small ? (unique ? gadev::fill_kernel : gadev::fill_shared_kernel) : tables == gadev::FillTables::Medium ? gadev::fill_tangled_kernel
        : gadev::fill_large_kernel;
}
static size_t trace_smem(int warpsPerBlock) { return sizeof(gadev::TraceWarp) * warpsPerBlock; }

uint64_t ga_warp_tables_bytes(const gadev::Caps& c) { return gadev::wspace_bytes(c); }
uint64_t ga_multiseed_tables_bytes(const gadev::Caps& c) { return gadev::wspace_bytes(c, true); }

static bool set_smem(const void* kernel, size_t smem)
{
    return smem <= 48 * 1024 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
}

int ga_fill_blocks_per_sm(int warpsPerBlock, gadev::FillTables tables, bool unique)
{
    const size_t smem = fill_smem(warpsPerBlock, tables);
    const auto kernel = fill_function(tables, unique);
    if (!set_smem((const void*)kernel, smem)) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, warpsPerBlock * 32, smem) != cudaSuccess) return 0;
    return n;
}

int ga_trace_blocks_per_sm(int warpsPerBlock)
{
    const size_t smem = trace_smem(warpsPerBlock);
    if (!set_smem((const void*)gadev::trace_kernel, smem)) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gadev::trace_kernel, warpsPerBlock * 32, smem) != cudaSuccess) return 0;
    return n;
}

int ga_launch_extend(const gadev::FillArgs& fa, const gadev::TraceArgs& ta, uint32_t* counters, int fillBlocks, int mediumBlocks,
    int traceBlocks, int warpsPerBlock, void* stream)
{
    const int fillWarps = fa.tables == gadev::FillTables::Medium ? 1 : warpsPerBlock;
    const size_t fillSmem = fill_smem(fillWarps, fa.tables);
    const auto fill = fill_function(fa.tables, fa.g.uniqueComponents != 0);
    const size_t traceSmem = trace_smem(warpsPerBlock);
    if (!set_smem((const void*)fill, fillSmem) || !set_smem((const void*)gadev::trace_kernel, traceSmem)) return -1;
    fill<<<fillBlocks, fillWarps * 32, fillSmem, (cudaStream_t)stream>>>(fa, counters);
    if (cudaGetLastError() != cudaSuccess) return -1;
    if (fa.resume)
    {
        gadev::FillArgs fm = fa;
        fm.tables = gadev::FillTables::Medium;
        fm.caps = gadev::medium_caps();
        fm.workspaceStride = gadev::wspace_bytes(fm.caps);
        const size_t smem = fill_smem(1, gadev::FillTables::Medium);
        if (!set_smem((const void*)gadev::fill_medium_kernel, smem)) return -1;
        gadev::fill_medium_kernel<<<mediumBlocks, 32, smem, (cudaStream_t)stream>>>(fm, counters + 3);
        if (cudaGetLastError() != cudaSuccess) return -1;
    }
    gadev::trace_kernel<<<traceBlocks, warpsPerBlock * 32, traceSmem, (cudaStream_t)stream>>>(ta, counters + 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_launch_multiseed_fill(const gadev::FillArgs& fa, const gadev::MultiTraceArgs& ta, uint32_t* counters, int fillBlocks, int partBlocks,
    int warpsPerBlock, void* stream)
{
    if (!fa.workspace) return -1;
    const size_t fillSmem = fill_smem(1, gadev::FillTables::Global);
    if (!set_smem((const void*)gadev::fill_multiseed_kernel, fillSmem)) return -1;
    gadev::fill_multiseed_kernel<<<fillBlocks, 32, fillSmem, (cudaStream_t)stream>>>(fa, counters);
    if (cudaGetLastError() != cudaSuccess) return -1;
    gadev::ms_candidates_kernel<<<partBlocks, warpsPerBlock * 32, 0, (cudaStream_t)stream>>>(ta, counters + 1, 0);
    if (cudaGetLastError() != cudaSuccess) return -1;
    gadev::ms_reserve_kernel<<<(ta.num + 3) / 4, 128, 0, (cudaStream_t)stream>>>(ta);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_launch_multiseed_list(const gadev::MultiTraceArgs& ta, uint32_t* counters, int partBlocks, int warpsPerBlock, void* stream)
{
    gadev::ms_candidates_kernel<<<partBlocks, warpsPerBlock * 32, 0, (cudaStream_t)stream>>>(ta, counters + 3, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_launch_multiseed_keys(const gadev::MultiTraceArgs& ta, void* stream)
{
    gadev::ms_keys_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(ta);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_launch_multiseed_resolve(const gadev::MultiTraceArgs& ta, uint32_t* counters, int readBlocks, int warpsPerBlock, void* stream)
{
    gadev::ms_resolve_kernel<<<readBlocks, warpsPerBlock * 32, 0, (cudaStream_t)stream>>>(ta, counters + 4);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_launch_multiseed_walk(const gadev::MultiTraceArgs& ta, uint32_t* counters, int candBlocks, int warpsPerBlock, void* stream)
{
    const size_t traceSmem = trace_smem(warpsPerBlock);
    if (!set_smem((const void*)gadev::ms_trace_kernel, traceSmem)) return -1;
    gadev::ms_trace_kernel<<<candBlocks, warpsPerBlock * 32, traceSmem, (cudaStream_t)stream>>>(ta, counters + 5, 0);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_launch_multiseed_write(const gadev::MultiTraceArgs& ta, uint32_t* counters, int candBlocks, int warpsPerBlock, void* stream)
{
    const size_t traceSmem = trace_smem(warpsPerBlock);
    if (!set_smem((const void*)gadev::ms_trace_kernel, traceSmem)) return -1;
    gadev::ms_trace_kernel<<<candBlocks, warpsPerBlock * 32, traceSmem, (cudaStream_t)stream>>>(ta, counters + 6, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_build_node_records(const gadev::DevGraph& g, gadev::NodeRec* rec, void* stream)
{
    cudaGetLastError();      // an upload fails by its own errors only, not by one that the process has left
    gadev::node_records_kernel<<<(g.N + 255) / 256, 256, 0, (cudaStream_t)stream>>>(g, rec);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ga_upload_tables()
{
    int8_t t[256];
    for (int i = 0; i < 256; i++) t[i] = (int8_t)gadev::iupac_mask((unsigned char)i);
    return cudaMemcpyToSymbol(gadev::c_iupac, t, sizeof(t)) == cudaSuccess ? 0 : -1;
}
