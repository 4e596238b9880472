// Shared declarations of the batched seed-extension kernels (fill, then traceback; one warp per extension).
#pragma once
#include <stdint.h>
#include "wordslice.cuh"

namespace gadev
{

// What the DP needs of one node, in one 64-byte record: read field by field from the arrays
// below, a node's computation waited for five loads in a row (offsets, then neighbours, then
// their components), about 600 cycles each from L2 for a warp alone.
struct __align__(16) NodeRec
{
    u64 seq[2];            // 2-bit sequence; not set for an ambiguous node
    u32 comp;
    u32 meta;              // bits 0-6 length, 7 linearizable, 8-19 in-degree, 20-31 out-degree (each 4095 at most)
    u32 inOff;
    u32 outOff;
    u32 inNb[2];           // the first neighbours, the others are read from the arrays
    u32 outNb[3];
    u32 outComp[3];        // components of outNb
};
static constexpr u32 kRecIn = 2, kRecOut = 3, kRecDegree = 4095;
static constexpr u32 kRecLinearizable = 0x80;
GA_HD u32 rec_len(u32 meta) { return meta & 0x7f; }
GA_HD u32 rec_in_degree(u32 meta) { return (meta >> 8) & kRecDegree; }
GA_HD u32 rec_out_degree(u32 meta) { return meta >> 20; }

// AlignmentGraph fields the DP reads (AlignmentGraph.h:121-139), device copies.
struct DevGraph
{
    const NodeRec* rec;    // [N], or null: the records are put together from the arrays as they are needed
    u32 uniqueComponents;  // no two nodes share a component number (0: they may)
    u32 N;
    u32 firstAmbiguous;
    const u32* len;
    const u64* seq2;       // [firstAmbiguous][2] 2-bit chunks of 32 bp
    const u64* seqAmb;     // [N - firstAmbiguous][4] A,C,G,T masks
    const u32* inOff;
    const u32* inNb;
    const u32* outOff;
    const u32* outNb;
    const uint8_t* lin;
    const u32* comp;
};

// One band entry: the state of a <= 64 bp node for one 64-row slice
// (NodeSliceMapItemStruct, NodeSlice.h:15-47).  64 bytes.
struct __align__(16) Item
{
    u64 sVP, sVN;          // first column
    u64 eVP, eVN;          // last column
    u64 HP, HN;            // horizontal deltas along the slice's last row
    i32 sEnd, eEnd;
    i32 minScore;          // in a committed slice: where the node's columns are (u32, kNoColumns: not kept)
    u32 node;              // bit 31: the node has been computed ("exists"); bit 30: it is a
                           // seed start in this slice (multiseed DP, DPSlice::seedstartNodes)
};
static constexpr u32 kExists = 0x80000000u;
static constexpr u32 kSeedStart = 0x40000000u;
static constexpr u32 kNodeMask = 0x3fffffffu;

// The column store: what the traceback needs of a node-slice's columns, kept by the fill in
// 16-byte units while there is room.  Unit 0 holds the +1 and -1 deltas along the slice's first
// row (bit c: column c against column c - 1), unit c > 0 column c's VP and its rows with an open
// diagonal step.  About 37 bytes per read base at bandwidth 10, written once and about half of it
// read, where memory bandwidth is otherwise idle (below 1 % of the copy peak).  Without the store
// the traceback recomputes the columns, with the lookups, loads and masks that takes: 50,000
// extensions (250 Mbp) take 74.3 ms instead of 48.0, one seed of a 10 kbp read 3.59 instead of
// 2.67, 1,000 tangled extensions 29.1 instead of 28.2.
struct __align__(16) ColumnUnit
{
    u64 x, y;
};
static constexpr u32 kNoColumns = 0xffffffffu;
static constexpr u32 kStoreChunk = 2048;   // units a warp takes at once

// The traceback copies slices and their columns ahead in pieces of fixed sizes, which may reach
// past the last one: so much is readable behind the arena (bytes) and the store (units).
static constexpr u32 kArenaPad = 1024;
static constexpr u32 kStorePad = 128;

// A committed DP slice in the arena: this 32-byte record, then count Items in first-pop order
// (the multiseed DP's seed starts first), then their node ids (u32, padded to 16 bytes), then
// for the multiseed DP each node's best exact-end-position
// X-score (count i32, DPSlice::nodeMaxExactEndposScore) and, for a band of more than
// kHashedBand nodes, an open-addressing index of the band (hashSize u32 slots, each an
// entry's position or kEmptySlot, linear probing from the node's hash).  The traceback finds
// a node's entry through the index where there is one, else by a warp ballot over the ids.
static constexpr u32 kHashedBand = 64;
static constexpr u32 kEmptySlot = 0xffffffffu;
struct __align__(16) SliceRec
{
    i32 minScore;
    i32 quit;              // minScore + bandwidth (the slice's band quit score)
    i32 maxX;              // maxExactEndposScore
    u32 maxXNode;          // maxExactEndposNode
    u32 count;
    u32 notValid;          // scoresNotValid: the tangle-effort cap was hit
    u32 hashSize;          // slots of the band index (a power of two), 0 = none
    u32 hashOff;           // byte offset of the band index from the record
};

// Per-extension state passed from the fill to the traceback.
struct ExtState
{
    u64 dir;               // arena offset of the slice directory (u64 record offsets)
    u32 committed;         // slices in the table, including the start slice
    i32 status;
    u64 steps;             // Myers column steps in the fill
    u64 aux;               // multiseed DP: arena offset of the per-slice best X-scores (i32 [committed])
};

// The fill's tables in shared memory: band entries and node-table slots of a slice, heap
// entries, pending incoming columns of a slice.  A slot belongs to a lane, so 32 is the most.
static constexpr u32 kSmallBand = 32, kSmallHeap = 32, kSmallExtras = 64;

// Capacities of one warp's frontier tables in global memory.
struct Caps
{
    u32 band;              // band entries per slice
    u32 hash;              // node-table slots per slice (power of two, >= 32)
    u32 heap;              // heap entries
    u32 extras;            // pending incoming columns per slice
};

// How far an extension's fill has come: its next slice and what the slices before it left.
struct FillState
{
    u64 dir;               // as in ExtState
    u64 steps;
    u32 slice;
    u32 committed;
    i32 bestX;
    i32 lastMin;
    i32 lastQuit;
};

// An extension that outgrew the small tables at a slice, with the band of the slice before it: the
// medium tables go on from there.  Started again with the tables in global memory, after a pass of
// their own, the 233 of 1,000 tangled extensions that this happens to took the call from 39.0 ms to
// 45.8; started again with the medium ones 41.7.
struct __align__(16) ResumeRec
{
    Item band[kSmallBand];
    FillState state;
    u32 ext;
    u32 count;             // band entries
};

// Where a warp's frontier tables are: in lane registers and shared memory (kSmall*), in shared
// memory with medium_caps(), or in global memory with FillArgs::caps.
enum class FillTables { Small, Medium, Global };

// 35 KB a warp, 38 with its recorded columns, five warps on an SM: for the few extensions that
// outgrow the small tables, and from the start for graphs that are mostly cycles
// (ga_graph::tangled).  There one extension in four to twenty outgrows the small tables, and those,
// which go on only when all others have ended, are what the call waits for.  With 64 band entries,
// ten warps on an SM and the rest handed on, 1,000 extensions of tangled 20 kbp reads took 30.2 ms
// instead of 28.7.
//
// The small tables let sixteen warps on an SM, and their nodes cost a tenth less, so all other graphs
// keep them.  The line for the graphs that are mostly cycles is kMediumWaves times the warps that are
// on the GPU at once (152 SMs: 3,040 extensions), a bound of what is lost where a graph's numbers
// are shared but its reads meet no tangles, at the price of the tangled batches between it and
// the crossing.  Milliseconds with the medium tables / with the small ones:
//   extensions                                1,000       3,000       4,800      10,000
//   tangled graph, 20 kbp reads at 12 %   28.5/36.1   31.1/43.2   36.4/41.4   66.2/61.8
//   tangled graph, accurate 1 kbp reads     3.0/4.5     3.7/5.9     3.4/5.4     4.3/6.5
//   variation graph with its numbers
//     shared in pairs, 10 kbp at 10 %       4.1/3.5     7.3/5.1    10.7/5.9   22.1/11.0
//   the same, accurate 1 kbp reads         0.52/0.49   0.92/0.72   1.38/0.92   2.75/1.66
static constexpr u32 kMediumWaves = 4;
inline Caps medium_caps()
{
    Caps c;
    c.band = 128; c.hash = 256; c.heap = 128; c.extras = 256;
    return c;
}

struct FillArgs
{
    DevGraph g;
    u32 bandwidth;
    i32 xdrop;
    u64 maxCells;
    i32 cost;
    u32 num;
    const u32* order;      // processing order (longest first); nullptr = index order
    const uint8_t* seq;
    const u64* seqOff;
    const u32* seqLen;
    const u32* startNode;
    const u32* startOffset;
    uint8_t* arena;        // DP tables of the batch, handed out in chunks
    u64 arenaBytes;        // kArenaPad more are readable behind them
    unsigned long long* arenaCursor;   // [0] bytes handed out in chunks, [1] bytes the tables took, [2] units of the column store
                                       // handed out (all start at 0)
    ColumnUnit* store;     // the column store, or null
    u64 storeUnits;        // below kNoColumns
    u64 chunkBytes;        // arena bytes a warp takes at once
    FillTables tables;
    ResumeRec* resume;     // small tables: [resumeCap] the extensions handed on to the medium tables, or null
    u32 resumeCap;
    u32* resumeCount;      // starts at 0
    uint8_t* workspace;    // global tables: where they are
    u64 workspaceStride;   // medium and global tables: bytes of one warp's
    Caps caps;             // and their capacities
    const i32* prevStatus; // when non-null, only extensions whose previous status is GA_CAPACITY run
    ExtState* states;      // [num] where each extension's table is, for the traceback
    // multiseed DP (nullptr otherwise): read i's seeds are [seedOff[i], seedOff[i+1]),
    // slice index and split node each, in slice order
    const u64* seedOff;
    const u32* seedSlice;
    const u32* seedNode;
};

struct TraceArgs
{
    DevGraph g;
    i32 cost;
    u32 num;
    const u32* order;      // the fill's processing order; nullptr = index order
    const i32* prevStatus; // the fill's filter
    const ExtState* states;
    const uint8_t* seq;
    const u64* seqOff;
    const u32* seqLen;
    const uint8_t* arena;
    const ColumnUnit* store;
    const u64* traceOffset;
    const u32* traceCap;
    i32* status;
    i32* score;
    u32* traceLen;
    u64* traceItems;
    u64* cellSteps;
};

// One local maximum of a multiseed read's table that may start a trace: a node whose best
// X-score in a slice beats its neighbours' and reaches the multimap fraction of the slice's
// best before any trace raised it.  The traces from the candidates are independent, so one
// warp traces each; the read's own pass keeps them in getLocalMaximaTracesFromTable's order
// against the raised slice bests, in rounds: a candidate is traced only once the traces kept
// before it have not ruled it out (or as one of a few traced ahead of the read's next one).
struct MsCand
{
    u32 read;
    u32 slice;
    u32 index;             // the node's position in the slice's band
    i32 score;             // its best X-score in the slice
    u32 startNode;         // the trace's first cell
    u32 startOff;
    int64_t startSeq;
    i32 startScore;
    i32 err;               // 0 or the status the trace failed with
    i32 traceScore;
    u32 len;               // trace items
    int64_t traceStart;    // read position of the trace's last item
    u64 outOff;            // kept traces: items from the read's trace_offset
    u32 slot;              // kept traces: the trace's index in the read, else kNoSlot
    u32 state;             // kUntraced, kQueued (for this round's walks) or kTraced
    u32 lastNode;          // the trace's last item (its start in the read)
    u32 lastOff;
};

// What removeDuplicateTraces looks at in a kept trace: the read positions of its first and
// last items, its last item's cell, its score (and its length, for the room it takes).
struct MsKey
{
    int64_t first;
    int64_t last;
    u32 lastNode;
    u32 lastOff;
    i32 score;
    u32 len;
};
static constexpr u32 kNoSlot = 0xffffffffu;
static constexpr u32 kUntraced = 0, kQueued = 1, kTraced = 2;

// A multiseed read's selection so far: its candidates before `cursor` are decided.
struct MsSel
{
    u64 used;              // items of the kept traces that have their place
    u64 items;             // items of all kept traces
    u32 nt;                // kept traces that have their place
    u32 traces;            // kept traces
    u32 cursor;
    u32 full;              // the kept traces have outgrown the read's room
    u32 done;
    u32 pad;
};
// the status of a multiseed read whose traces outgrew its room (reported as GA_CAPACITY with
// the room it needs; the batch does not run it again as it does a read whose tables ran out)
static constexpr i32 kMsRoom = 100;

static constexpr u32 kCandParts = 32;

// The multiseed DP's traceback outputs (ga_multiseed_results).
struct MultiTraceArgs
{
    DevGraph g;
    i32 cost;
    u32 num;
    const u32* order;
    const i32* prevStatus;
    const ExtState* states;
    const uint8_t* seq;
    const u64* seqOff;
    const u32* seqLen;
    const uint8_t* arena;
    const ColumnUnit* store;
    const u64* traceOffset;
    const u64* traceCap;
    u32 maxTraces;
    double multimapScoreFraction;
    i32* status;
    u32* numTraces;
    i32* traceScore;
    u64* traceStart;
    u32* traceLen;
    u64* traceItems;
    u64* cellSteps;
    u64* itemsNeeded;      // [num] or null: when the traces outgrow the read's room, the room they need
                           // (with exact room: the items of the kept traces)
    u32* tracesNeeded;
    // exact room (traceBase non-null): read i's kept traces are traceBase[i] + slot in the
    // kept list, whose summaries go to keys; after removeDuplicateTraces kept trace k is
    // written as trace keptSlot[k] (kNoSlot: a duplicate) with its items from keptItem[k], its
    // start counted from itemBias; traceOffset, traceCap and maxTraces are not used
    const u64* traceBase;
    MsKey* keys;
    const u32* keptSlot;
    const u64* keptItem;
    u64 itemBias;
    MsSel* sel;            // [num] each read's selection
    u32* work;             // this round's candidates to walk (indices into cands)
    u32* workCount;
    u32 window;            // candidates a read may have walked in this round
    MsCand* cands;         // [candCap] the batch's candidates, each read's together and in order
    u64 candCap;
    u64* candBegin;        // [num] read i's candidates are [candBegin[i], candBegin[i] + candCount[i])
    u32* candCount;
    u32* candPart;         // [num][kCandParts] candidates of each part of a read's slices, then where they start in its run
    unsigned long long* candTotal;   // candidates of the batch
};

}

// bytes of one warp's frontier tables in global memory for these capacities (the multiseed DP's add each band
// node's best X-score)
uint64_t ga_warp_tables_bytes(const gadev::Caps& caps);
uint64_t ga_multiseed_tables_bytes(const gadev::Caps& caps);
// resident blocks of 32 * warpsPerBlock threads per SM of the fill kernel (shared: tables in
// shared memory) and of the traceback kernel
int ga_fill_blocks_per_sm(int warpsPerBlock, gadev::FillTables tables, bool unique);
int ga_trace_blocks_per_sm(int warpsPerBlock);
// launches the fill kernel, with fa.resume the medium tables' (mediumBlocks blocks of one warp),
// and then the traceback kernel on `stream`, blocks of warpsPerBlock warps, one extension per warp
// at a time; counters[0], [1] and [3] must be zero
int ga_launch_extend(const gadev::FillArgs& fa, const gadev::TraceArgs& ta, uint32_t* counters, int fillBlocks, int mediumBlocks,
    int traceBlocks, int warpsPerBlock, void* stream);
// the multiseed DP in steps, each on `stream`, its frontier tables always in the global workspace; blocks
// of warpsPerBlock warps but for the fill, whose fillBlocks are of one:
// - fill: the fill and the count of each read's trace candidates (counters[0], [1] and
//   ta.candTotal zero);
// - list: once ta.cands has room for *ta.candTotal, the candidates listed (counters[3] zero,
//   ta.sel zeroed);
// - rounds, until a resolve queues nothing: resolve (each read decides its candidates in
//   order as far as their walks are known, then queues the next ta.window walks; counters[4]
//   and *ta.workCount zero) and walk (the queued candidates' traces counted; counters[5] zero);
// - write: the kept traces written (counters[6] zero).
// counters[2] is left to the caller.
int ga_launch_multiseed_fill(const gadev::FillArgs& fa, const gadev::MultiTraceArgs& ta, uint32_t* counters, int fillBlocks, int partBlocks,
    int warpsPerBlock, void* stream);
int ga_launch_multiseed_list(const gadev::MultiTraceArgs& ta, uint32_t* counters, int partBlocks, int warpsPerBlock, void* stream);
int ga_launch_multiseed_resolve(const gadev::MultiTraceArgs& ta, uint32_t* counters, int readBlocks, int warpsPerBlock, void* stream);
int ga_launch_multiseed_walk(const gadev::MultiTraceArgs& ta, uint32_t* counters, int candBlocks, int warpsPerBlock, void* stream);
int ga_launch_multiseed_write(const gadev::MultiTraceArgs& ta, uint32_t* counters, int candBlocks, int warpsPerBlock, void* stream);
// exact room: each kept trace's summary into ta.keys
int ga_launch_multiseed_keys(const gadev::MultiTraceArgs& ta, void* stream);
int ga_upload_tables();
// fills rec[0..N) from the graph's arrays
int ga_build_node_records(const gadev::DevGraph& g, gadev::NodeRec* rec, void* stream);
void ga_set_last_error(const char* message);
