// C ABI of the GB300 seed-extension path (declared in include/graphaligner_gb300.h).
//
// Handles own their device memory.  ga_extend_batch copies a host batch in,
// runs the fill and traceback kernels (and again with larger frontier tables for
// the few extensions that outgrew the first pass's), and copies the results out.  No CPU fallback exists:
// every extension is computed by the kernels or reported with its status.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>
#include "extend.cuh"
#include "launch_grid.h"
#include "trace_dedupe.h"
#include "../../include/graphaligner_gb300.h"

namespace
{
thread_local std::string g_lastError;
thread_local cudaError_t g_lastCuda = cudaSuccess;     // of the last call that GA_CUDA refused

int fail(int code, const std::string& msg)
{
    g_lastError = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* what)
{
    g_lastCuda = e;
    cudaGetLastError();      // reported here: the next launch's check must not find it again
    return fail(GA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define GA_CUDA(call) do { cudaError_t _e = (call); if (_e != cudaSuccess) return cuda_fail(_e, #call); } while (0)

template <typename T>
struct DevBuf
{
    T* ptr = nullptr;
    size_t count = 0;
    cudaError_t reserve(size_t n)
    {
        if (n <= count) return cudaSuccess;
        // 1.5x headroom: growing frees the old buffer, and cudaFree synchronises the device
        const size_t grow = std::max(n, count * 3 / 2);
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        count = 0;
        cudaError_t e = cudaMalloc((void**)&ptr, std::max<size_t>(grow, 1) * sizeof(T));
        if (e == cudaSuccess) count = grow;
        return e;
    }
    void release()
    {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        count = 0;
    }
};

// pinned host memory that grows keeping its first `keep` elements
template <typename T>
struct HostPinned
{
    T* ptr = nullptr;
    size_t count = 0;
    bool reserve(size_t n, size_t keep)
    {
        if (n <= count) return true;
        const size_t grow = std::max(n, count * 3 / 2);
        T* q = nullptr;
        if (cudaHostAlloc((void**)&q, grow * sizeof(T), cudaHostAllocDefault) != cudaSuccess)
        {
            cudaGetLastError();
            return false;
        }
        if (keep) memcpy(q, ptr, keep * sizeof(T));
        if (ptr) cudaFreeHost(ptr);
        ptr = q;
        count = grow;
        return true;
    }
    void release()
    {
        if (ptr) cudaFreeHost(ptr);
        ptr = nullptr;
        count = 0;
    }
};

// ga_multiseed_batch_exact's results, kept until the extender's next call
struct MsExactOut
{
    std::vector<int32_t> status;
    std::vector<uint32_t> numTraces;
    std::vector<uint64_t> traceFirst, cellSteps;
    HostPinned<int32_t> score;
    HostPinned<uint64_t> start, item;
    HostPinned<uint32_t> len;
    uint64_t traces = 0, items = 0;
    bool grow(uint64_t t, uint64_t i)
    {
        return score.reserve(std::max<uint64_t>(t, 1), traces) && start.reserve(std::max<uint64_t>(t, 1), traces)
            && len.reserve(std::max<uint64_t>(t, 1), traces) && item.reserve(std::max<uint64_t>(i, 1), items);
    }
    void publish(ga_multiseed_output* o) const
    {
        o->status = status.data();
        o->num_traces = numTraces.data();
        o->trace_first = traceFirst.data();
        o->trace_score = score.ptr;
        o->trace_start = start.ptr;
        o->trace_len = len.ptr;
        o->trace_items = item.ptr;
        o->cell_steps = cellSteps.data();
        o->total_traces = traces;
        o->total_items = items;
    }
    ~MsExactOut()
    {
        score.release(); start.release(); item.release(); len.release();
    }
};

__global__ void count_status_kernel(const int32_t* status, uint32_t n, int32_t value, uint32_t* out)
{
    uint32_t local = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (status[i] == value) local++;
    if (local) atomicAdd(out, local);
}
}

struct ga_graph
{
    int device = 0;
    uint32_t N = 0;
    gadev::DevGraph d {};
    bool tangled = false;     // at least half of the nodes share their component number
    std::vector<void*> allocations;
};

struct ga_extender
{
    ga_graph* graph = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[6] {};                 // kernel start/end, D2H start, H2D start/end, D2H end
    // the trace items of a host-buffer batch go back in chunks on these streams, so that
    // several copy engines share the (largest) device-to-host copy
    static constexpr int kCopyStreams = 4;
    cudaStream_t copy[kCopyStreams] {};
    cudaEvent_t copyDone[kCopyStreams] {};
    int sms = 0;
    ga_launch_shape shape {};             // warps per block, blocks per SM, first table layout, arena chunk
    uint8_t* workspace = nullptr;         // frontier tables of the global-memory layouts
    uint64_t workspaceBytes = 0;
    uint8_t* arena = nullptr;
    uint64_t arenaBytes = 0;
    uint32_t* counters = nullptr;          // [0] work counter, [2] status count; the multiseed DP: work counters [1], [3]-[6], candidate total (u64) [8]-[9]
    unsigned long long* arenaCursor = nullptr;   // [0] overflow cursor, [1] bytes taken, [2] column store units taken
    gadev::ColumnUnit* store = nullptr;    // the column store, grown to the largest batch within its bound
    uint64_t storeUnits = 0;
    uint64_t storeLimit = 0;               // the store's bound in bytes
    bool storeWithheld = false;            // this call goes without a column store
    float lastFillMs = 0;
    float lastTraceMs = 0;
    float lastH2DMs = 0;                    // host-buffer copies of the last ga_extend_batch
    float lastD2HMs = 0;
    uint64_t lastArenaBytes = 0;
    uint32_t lastLaunches = 0;
    uint32_t lastRounds[3] {};              // extensions run in each layout by the last call
    std::vector<uint32_t> orderHost;      // processing order of the last host batch
    // host-batch staging
    DevBuf<uint8_t> seq;
    DevBuf<uint64_t> seqOff, traceOff, traceItems, cellSteps;
    DevBuf<uint32_t> seqLen, startNode, startOffset, traceCap, traceLen, order;
    DevBuf<int32_t> status, score, prevStatus;
    DevBuf<gadev::ExtState> states;        // where the fill left each extension's table
    DevBuf<gadev::ResumeRec> resume;       // extensions handed on from the small tables to the medium ones
    // multiseed DP staging
    DevBuf<uint64_t> msSeedOff, msTraceCap, msTraceStart, msItemsNeeded;
    DevBuf<uint32_t> msSeedSlice, msSeedNode, msNumTraces, msTraceLen, msTracesNeeded;
    DevBuf<int32_t> msTraceScore;
    DevBuf<uint64_t> msCandBegin, msTraceBase, msKeptItem;
    DevBuf<uint32_t> msCandCount, msCandPart, msWork, msKeptSlot;
    DevBuf<gadev::MsKey> msKeys;
    DevBuf<gadev::MsCand> msCands;
    DevBuf<gadev::MsSel> msSel;
    MsExactOut msOut;                      // ga_multiseed_batch_exact's results
    uint64_t lastCandidates = 0, lastKept = 0, lastWalks = 0;
    uint32_t lastResolveRounds = 0;
};

extern "C" const char* ga_last_error(void) { return g_lastError.c_str(); }

void ga_set_last_error(const char* message) { g_lastError = message; }
extern "C" const char* ga_version(void) { return "graphaligner_gb300 0.1 (sm_103a)"; }

// How many of the n nodes share their component number with another, or n + 1 where the numbers are
// spread too widely to tell cheaply
static uint64_t shared_components(const uint32_t* component, uint32_t n)
{
    uint32_t most = 0;
    for (uint32_t i = 0; i < n; i++) most = std::max(most, component[i]);
    if (most >= 16ull * n + 1024 || most == 0xffffffffu) return (uint64_t)n + 1;
    std::vector<uint64_t> seen((size_t)most / 64 + 1, 0), again(seen.size(), 0);
    bool any = false;
    for (uint32_t i = 0; i < n; i++)
    {
        uint64_t& word = seen[component[i] / 64];
        const uint64_t bit = 1ull << (component[i] % 64);
        again[component[i] / 64] |= word & bit;
        any |= (word & bit) != 0;
        word |= bit;
    }
    uint64_t shared = 0;
    if (any)
        for (uint32_t i = 0; i < n; i++) shared += (again[component[i] / 64] >> (component[i] % 64)) & 1;
    return shared;
}

extern "C" int ga_graph_upload(const ga_graph_desc* desc, int device, ga_graph_t* out)
{
    if (!desc || !out) return fail(GA_ERR_ARGUMENT, "null argument");
    if (desc->num_nodes == 0 || desc->first_ambiguous > desc->num_nodes) return fail(GA_ERR_ARGUMENT, "bad node counts");
    // a band entry keeps two flags above the node index
    if (desc->num_nodes > gadev::kNodeMask) return fail(GA_ERR_ARGUMENT, "more than 2^30 - 1 split nodes");
    const uint32_t N = desc->num_nodes;
    for (uint32_t i = 0; i < N; i++)
        if (desc->node_length[i] == 0 || desc->node_length[i] > 64) return fail(GA_ERR_ARGUMENT, "node length outside 1..64");
    GA_CUDA(cudaSetDevice(device));
    if (ga_upload_tables() != 0) return fail(GA_ERR_CUDA, "constant tables");
    ga_graph* g = new ga_graph();
    g->device = device;
    g->N = N;
    auto up = [&](const void* src, size_t bytes, void** dst) -> cudaError_t
    {
        *dst = nullptr;
        cudaError_t e = cudaMalloc(dst, std::max<size_t>(bytes, 16));
        if (e != cudaSuccess) return e;
        g->allocations.push_back(*dst);
        if (bytes) e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
        return e;
    };
    const uint32_t nIn = desc->in_offsets[N];
    const uint32_t nOut = desc->out_offsets[N];
    void *len, *seq2, *seqAmb, *inOff, *inNb, *outOff, *outNb, *lin, *comp;
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = up(desc->node_length, (size_t)N * 4, &len);
    if (e == cudaSuccess) e = up(desc->seq2bit, (size_t)desc->first_ambiguous * 16, &seq2);
    if (e == cudaSuccess) e = up(desc->seq_ambiguous, (size_t)(N - desc->first_ambiguous) * 32, &seqAmb);
    if (e == cudaSuccess) e = up(desc->in_offsets, (size_t)(N + 1) * 4, &inOff);
    if (e == cudaSuccess) e = up(desc->in_neighbors, (size_t)nIn * 4, &inNb);
    if (e == cudaSuccess) e = up(desc->out_offsets, (size_t)(N + 1) * 4, &outOff);
    if (e == cudaSuccess) e = up(desc->out_neighbors, (size_t)nOut * 4, &outNb);
    if (e == cudaSuccess) e = up(desc->linearizable, (size_t)N, &lin);
    if (e == cudaSuccess) e = up(desc->component, (size_t)N * 4, &comp);
    if (e != cudaSuccess)
    {
        for (void* p : g->allocations) cudaFree(p);
        delete g;
        return cuda_fail(e, "graph upload");
    }
    g->d.N = N;
    const uint64_t shared = shared_components(desc->component, N);
    g->d.uniqueComponents = shared == 0;
    g->tangled = shared <= N && 2 * shared >= N;
    g->d.firstAmbiguous = desc->first_ambiguous;
    g->d.len = (const uint32_t*)len;
    g->d.seq2 = (const uint64_t*)seq2;
    g->d.seqAmb = (const uint64_t*)seqAmb;
    g->d.inOff = (const uint32_t*)inOff;
    g->d.inNb = (const uint32_t*)inNb;
    g->d.outOff = (const uint32_t*)outOff;
    g->d.outNb = (const uint32_t*)outNb;
    g->d.lin = (const uint8_t*)lin;
    g->d.comp = (const uint32_t*)comp;
    // the nodes' records; without room for them the kernels gather each from the arrays
    void* rec = nullptr;
    if (cudaMalloc(&rec, (size_t)N * sizeof(gadev::NodeRec)) == cudaSuccess)
    {
        g->allocations.push_back(rec);
        if (ga_build_node_records(g->d, (gadev::NodeRec*)rec, nullptr) != 0 || (e = cudaStreamSynchronize(nullptr)) != cudaSuccess)
        {
            for (void* p : g->allocations) cudaFree(p);
            delete g;
            return fail(GA_ERR_CUDA, "node records");
        }
        g->d.rec = (const gadev::NodeRec*)rec;
    }
    else cudaGetLastError();
    *out = g;
    return GA_OK;
}

extern "C" int ga_graph_free(ga_graph_t g)
{
    if (!g) return GA_OK;
    cudaSetDevice(g->device);
    for (void* p : g->allocations) cudaFree(p);
    delete g;
    return GA_OK;
}

// Default launch shape (results never depend on it): blocks of 4 warps, as many blocks per
// SM as registers and shared memory allow, the frontier tables in shared memory first, and
// 64 KiB arena chunks (the DP tables of a few extensions of a few kbp).
static ga_launch_shape default_shape()
{
    ga_launch_shape sh;
    sh.warps_per_block = 4;
    sh.blocks_per_sm = 0;
    sh.first_layout = 0;
    sh.chunk_kib = 64;
    return sh;
}

static bool shape_ok(const ga_launch_shape& sh)
{
    return sh.warps_per_block >= 1 && sh.warps_per_block <= 4 && sh.first_layout <= 2 && sh.chunk_kib >= 1 && sh.chunk_kib <= (1u << 20);
}

// Frontier-table capacities of the three layouts: small tables in shared memory (a variation
// graph's bands hold a handful of nodes), then larger ones in global memory for the
// extensions that outgrew them (tangled de Bruijn graphs).
static gadev::Caps layout_caps(int layout)
{
    gadev::Caps c;
    if (layout == 0) { c.band = gadev::kSmallBand; c.hash = 0; c.heap = gadev::kSmallHeap; c.extras = gadev::kSmallExtras; }
    else if (layout == 1) { c.band = 512; c.hash = 1024; c.heap = 512; c.extras = 1024; }
    else { c.band = 16384; c.hash = 65536; c.heap = 16384; c.extras = 32768; }
    return c;
}

// Extensions that one call hands on from the small tables to the medium ones (2 KB each); more
// start again in the next layout
static constexpr uint32_t kResumeCap = 8192;

static const char* kShapeError = "launch shape: warps_per_block within 1..4, first_layout within 0..2, chunk_kib within 1..2^20";

extern "C" int ga_extender_create(ga_graph_t graph, uint64_t arena_bytes, ga_extender_t* out)
{
    if (!graph || !out) return fail(GA_ERR_ARGUMENT, "null argument");
    GA_CUDA(cudaSetDevice(graph->device));
    ga_extender* x = new ga_extender();
    x->graph = graph;
    cudaDeviceProp prop;
    GA_CUDA(cudaGetDeviceProperties(&prop, graph->device));
    x->sms = prop.multiProcessorCount;
    x->shape = default_shape();
    // the global-memory layouts' tables: room for a few thousand warps of the medium layout
    x->workspaceBytes = 256ULL << 20;
    GA_CUDA(cudaStreamCreateWithFlags(&x->stream, cudaStreamNonBlocking));
    for (int k = 0; k < ga_extender::kCopyStreams; k++)
    {
        GA_CUDA(cudaStreamCreateWithFlags(&x->copy[k], cudaStreamNonBlocking));
        GA_CUDA(cudaEventCreateWithFlags(&x->copyDone[k], cudaEventDisableTiming));
    }
    for (auto& e : x->ev) GA_CUDA(cudaEventCreate(&e));
    cudaError_t e = cudaMalloc((void**)&x->workspace, x->workspaceBytes);
    if (e != cudaSuccess) { delete x; return cuda_fail(e, "workspace"); }
    if (arena_bytes == 0) arena_bytes = 4ULL << 30;
    x->arenaBytes = arena_bytes;
    x->storeLimit = arena_bytes * 4;
    e = cudaMalloc((void**)&x->arena, x->arenaBytes + gadev::kArenaPad);
    if (e != cudaSuccess) { cudaFree(x->workspace); delete x; return cuda_fail(e, "arena"); }
    GA_CUDA(cudaMalloc((void**)&x->counters, 16 * sizeof(uint32_t)));
    GA_CUDA(cudaMalloc((void**)&x->arenaCursor, 3 * sizeof(unsigned long long)));
    *out = x;
    return GA_OK;
}

extern "C" int ga_extender_create_like(ga_extender_t x, ga_extender_t* out)
{
    if (!x || !out) return fail(GA_ERR_ARGUMENT, "null argument");
    int rc = ga_extender_create(x->graph, x->arenaBytes, out);
    if (rc != GA_OK) return rc;
    (*out)->shape = x->shape;
    (*out)->storeLimit = x->storeLimit;
    return GA_OK;
}

extern "C" int ga_extender_free(ga_extender_t x)
{
    if (!x) return GA_OK;
    cudaSetDevice(x->graph->device);
    cudaStreamSynchronize(x->stream);
    cudaFree(x->workspace);
    cudaFree(x->arena);
    cudaFree(x->counters);
    cudaFree(x->arenaCursor);
    cudaFree(x->store);
    x->seq.release(); x->seqOff.release(); x->traceOff.release(); x->traceItems.release(); x->cellSteps.release();
    x->seqLen.release(); x->startNode.release(); x->startOffset.release(); x->traceCap.release(); x->traceLen.release();
    x->order.release(); x->status.release(); x->score.release(); x->prevStatus.release(); x->states.release(); x->resume.release();
    x->msSeedOff.release(); x->msTraceCap.release(); x->msTraceStart.release(); x->msItemsNeeded.release();
    x->msSeedSlice.release(); x->msSeedNode.release(); x->msNumTraces.release(); x->msTraceLen.release(); x->msTracesNeeded.release();
    x->msTraceScore.release(); x->msCandBegin.release(); x->msCandCount.release(); x->msCandPart.release(); x->msCands.release();
    x->msTraceBase.release(); x->msKeptItem.release(); x->msWork.release(); x->msSel.release();
    x->msKeptSlot.release(); x->msKeys.release();
    for (auto& e : x->ev) cudaEventDestroy(e);
    cudaStreamDestroy(x->stream);
    for (int k = 0; k < ga_extender::kCopyStreams; k++)
    {
        if (x->copy[k]) cudaStreamDestroy(x->copy[k]);
        if (x->copyDone[k]) cudaEventDestroy(x->copyDone[k]);
    }
    delete x;
    return GA_OK;
}

static void release_store(ga_extender* x)
{
    cudaFree(x->store);
    x->store = nullptr;
    x->storeUnits = 0;
}

bool ga_extender_give_back_store(ga_extender_t x)
{
    if (!x || !x->store) return false;
    release_store(x);
    return true;
}

// Runs a call that may find no memory for its buffers while the column store, which only saves
// time, holds some: the store is then given back and the call made again without one.
template <class Call>
static int with_store_given_back(ga_extender* x, Call call)
{
    g_lastCuda = cudaSuccess;
    int rc = call();
    if (rc != GA_ERR_CUDA || g_lastCuda != cudaErrorMemoryAllocation || !ga_extender_give_back_store(x)) return rc;
    x->storeWithheld = true;
    rc = call();
    x->storeWithheld = false;
    return rc;
}

// Room in the column store for a batch of readBp bases: a band of bandwidth 10 computes 2.4
// columns per base on the variation graphs (5.5 on the tangled ones), 3 and a chunk for every
// warp are asked for.  The store holds at most its limit (four times the arena unless the caller
// sets another) and half of the memory that is free when it grows; what finds no room in it is
// recomputed by the traceback.
static void reserve_store(ga_extender* x, uint64_t readBp, uint64_t warps)
{
    if (x->storeWithheld) return;
    const uint64_t unit = sizeof(gadev::ColumnUnit);
    uint64_t want = readBp * 3 + warps * gadev::kStoreChunk;
    // (what is allocated ends kStorePad units behind the store)
    const uint64_t limit = x->storeLimit / unit;
    const uint64_t bound = std::min<uint64_t>(limit - std::min<uint64_t>(limit, gadev::kStorePad), (uint64_t)gadev::kNoColumns - 1);
    want = std::min(want, bound);
    if (want <= x->storeUnits) return;
    size_t freeBytes = 0, totalBytes = 0;
    if (cudaMemGetInfo(&freeBytes, &totalBytes) != cudaSuccess) return;
    const uint64_t most = std::min<uint64_t>((freeBytes / unit + x->storeUnits) / 2, bound);
    want = std::min(most, std::max(want, x->storeUnits * 3 / 2));
    // where free memory is the bound it moves with every other allocation of the process: a store that
    // would gain less than a quarter stays as it is (growing it frees it first, which waits for the device)
    if (want <= x->storeUnits || (want == most && want < x->storeUnits + x->storeUnits / 4)) return;
    release_store(x);
    if (cudaMalloc((void**)&x->store, (want + gadev::kStorePad) * unit) == cudaSuccess) x->storeUnits = want;
    else
    {
        x->store = nullptr;
        cudaGetLastError();
    }
}

// Runs one batch whose buffers are all on the device, readBp bases in all.  order: processing order
// (longest first).  Extensions that outgrow a layout's tables (GA_CAPACITY) run again
// in the next, larger layout; only those run.
static int run_device(ga_extender* x, const ga_extend_params* p, const ga_extend_batch_desc* b, ga_extend_results* r,
    const uint32_t* order, int32_t* prevStatus, uint64_t readBp, cudaStream_t stream)
{
    gadev::FillArgs fa {};
    fa.g = x->graph->d;
    fa.bandwidth = p->bandwidth;
    fa.xdrop = p->xdrop;
    fa.maxCells = p->max_cells_per_slice;
    fa.cost = p->xscore_error_cost;
    fa.num = b->num;
    fa.order = order;
    fa.seq = b->seq;
    fa.seqOff = b->seq_offset;
    fa.seqLen = b->seq_len;
    fa.startNode = b->start_node;
    fa.startOffset = b->start_offset;
    fa.arena = x->arena;
    fa.arenaBytes = x->arenaBytes;
    fa.arenaCursor = x->arenaCursor;

    gadev::TraceArgs ta {};
    ta.g = x->graph->d;
    ta.cost = p->xscore_error_cost;
    ta.seq = b->seq;
    ta.seqOff = b->seq_offset;
    ta.seqLen = b->seq_len;
    ta.arena = x->arena;
    ta.traceOffset = b->trace_offset;
    ta.traceCap = b->trace_capacity;
    ta.status = r->status;
    ta.score = r->score;
    ta.traceLen = r->trace_len;
    ta.traceItems = r->trace_items;
    ta.cellSteps = r->cell_steps;

    const uint32_t n = b->num;
    GA_CUDA(x->states.reserve(n));
    fa.states = x->states.ptr;
    const uint32_t resumeCap = std::min<uint32_t>(n, kResumeCap);
    GA_CUDA(x->resume.reserve(resumeCap));
    ta.num = n;
    ta.order = order;
    ta.states = x->states.ptr;
    x->lastFillMs = 0;
    x->lastTraceMs = 0;
    x->lastLaunches = 0;
    for (int k = 0; k < 3; k++) x->lastRounds[k] = 0;
    const ga_launch_shape& sh = x->shape;
    const int wpb = (int)sh.warps_per_block;
    fa.chunkBytes = (uint64_t)sh.chunk_kib << 10;
    uint32_t pending = n;                    // extensions the next round runs
    reserve_store(x, readBp, std::min<uint64_t>(n, (uint64_t)x->sms * 16));
    fa.store = x->store;
    fa.storeUnits = x->storeUnits;
    ta.store = x->store;
    for (int layout = (int)sh.first_layout; layout < 3; layout++)
    {
        const bool shared = layout == 0;
        const int mediumPerSm = shared ? ga_fill_blocks_per_sm(1, gadev::FillTables::Medium, false) : 0;
        // (the line is explained at medium_caps)
        const bool medium = x->graph->tangled && mediumPerSm > 0 && pending <= (uint64_t)gadev::kMediumWaves * x->sms * mediumPerSm;
        const gadev::FillTables tables = medium ? gadev::FillTables::Medium : shared ? gadev::FillTables::Small : gadev::FillTables::Global;
        const int fillWarps = medium ? 1 : wpb;
        const gadev::Caps caps = medium ? gadev::medium_caps() : layout_caps(layout);
        const uint64_t stride = ga_warp_tables_bytes(caps);
        const int fillPerSm = ga_fill_blocks_per_sm(fillWarps, tables, x->graph->d.uniqueComponents != 0);
        const int tracePerSm = ga_trace_blocks_per_sm(wpb);
        if (fillPerSm <= 0 || tracePerSm <= 0) return fail(GA_ERR_CUDA, "the extension kernels do not fit an SM with this launch shape");
        gadev::LaunchGrid grid = gadev::launch_grid(sh, x->sms, fillPerSm, fillWarps, mediumPerSm, tracePerSm, pending, resumeCap);
        if (!shared) grid.fill = std::max<uint64_t>(1, std::min<uint64_t>(grid.fill, x->workspaceBytes / stride / wpb));
        if (layout > (int)sh.first_layout)
        {
            // only extensions that ran out of a capacity in the previous round run again
            GA_CUDA(cudaMemcpyAsync(prevStatus, r->status, (size_t)n * 4, cudaMemcpyDeviceToDevice, stream));
        }
        fa.caps = caps;
        fa.tables = tables;
        fa.workspace = shared ? nullptr : x->workspace;
        fa.workspaceStride = stride;
        fa.resume = mediumPerSm > 0 && !medium ? x->resume.ptr : nullptr;
        fa.resumeCap = resumeCap;
        fa.resumeCount = x->counters + 4;
        fa.prevStatus = layout > (int)sh.first_layout ? prevStatus : nullptr;
        ta.prevStatus = fa.prevStatus;
        GA_CUDA(cudaMemsetAsync(x->counters, 0, 16 * sizeof(uint32_t), stream));
        GA_CUDA(cudaMemsetAsync(x->arenaCursor, 0, 3 * sizeof(unsigned long long), stream));
        GA_CUDA(cudaEventRecord(x->ev[0], stream));
        if (ga_launch_extend(fa, ta, x->counters, (int)grid.fill, (int)grid.medium, (int)grid.trace, wpb, stream) != 0)
            return fail(GA_ERR_CUDA, std::string("extension kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
        x->lastLaunches += fa.resume ? 3 : 2;
        x->lastRounds[layout] += pending;
        GA_CUDA(cudaEventRecord(x->ev[1], stream));
        count_status_kernel<<<64, 256, 0, stream>>>(r->status, n, GA_CAPACITY, x->counters + 2);
        GA_CUDA(cudaGetLastError());
        x->lastLaunches += 1;
        uint32_t counts[3] = {0, 0, 0};          // capacity failures, -, extensions handed on
        unsigned long long used[2] = {0, 0};
        GA_CUDA(cudaMemcpyAsync(counts, x->counters + 2, 12, cudaMemcpyDeviceToHost, stream));
        GA_CUDA(cudaMemcpyAsync(used, x->arenaCursor, 16, cudaMemcpyDeviceToHost, stream));
        GA_CUDA(cudaStreamSynchronize(stream));
        const uint32_t capFails = counts[0];
        if (layout == 0) x->lastRounds[1] += std::min(counts[2], resumeCap);
        if (layout == (int)sh.first_layout) x->lastArenaBytes = used[1];
        float ms = 0;
        GA_CUDA(cudaEventElapsedTime(&ms, x->ev[0], x->ev[1]));
        x->lastFillMs += ms;
        pending = capFails;
        if (capFails == 0) break;
    }
    return GA_OK;
}

// The packed trace item holds seqPos + 1 in 25 bits.
static_assert(GA_MAX_SEQ_LEN == (1u << 25) - 1, "read position field of the trace item");

static int check_lengths(const uint32_t* len, uint32_t n)
{
    for (uint32_t i = 0; i < n; i++)
        if (len[i] > GA_MAX_SEQ_LEN)
            return fail(GA_ERR_ARGUMENT, "extension " + std::to_string(i) + ": sequence longer than GA_MAX_SEQ_LEN (33,554,431 bp)");
    return GA_OK;
}

static uint64_t sum_lengths(const uint32_t* len, uint32_t n) { return std::accumulate(len, len + n, (uint64_t)0); }

static std::vector<uint32_t> longest_first(const uint32_t* len, uint32_t n)
{
    std::vector<uint32_t> order(n);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [len](uint32_t a, uint32_t b) { return len[a] > len[b]; });
    return order;
}

// Copies a host batch into the extender's device buffers and points db/dr at them.
// items: trace items the batch spans.
static int stage_host_batch(ga_extender* x, const ga_extend_batch_desc* b, ga_extend_batch_desc* db,
    ga_extend_results* dr, uint64_t* itemsOut)
{
    const uint32_t n = b->num;
    int rc = check_lengths(b->seq_len, n);
    if (rc != GA_OK) return rc;
    uint64_t seqBytes = 0, items = 0;
    for (uint32_t i = 0; i < n; i++)
    {
        seqBytes = std::max<uint64_t>(seqBytes, b->seq_offset[i] + b->seq_len[i]);
        items = std::max<uint64_t>(items, b->trace_offset[i] + b->trace_capacity[i]);
    }
    std::vector<uint32_t>& order = x->orderHost;   // kept until the next batch: the copy below is asynchronous
    order = longest_first(b->seq_len, n);
    GA_CUDA(x->seq.reserve(seqBytes));
    GA_CUDA(x->seqOff.reserve(n));
    GA_CUDA(x->seqLen.reserve(n));
    GA_CUDA(x->startNode.reserve(n));
    GA_CUDA(x->startOffset.reserve(n));
    GA_CUDA(x->traceOff.reserve(n));
    GA_CUDA(x->traceCap.reserve(n));
    GA_CUDA(x->order.reserve(n));
    GA_CUDA(x->status.reserve(n));
    GA_CUDA(x->prevStatus.reserve(n));
    GA_CUDA(x->score.reserve(n));
    GA_CUDA(x->traceLen.reserve(n));
    GA_CUDA(x->cellSteps.reserve(n));
    GA_CUDA(x->traceItems.reserve(std::max<uint64_t>(items, 1)));
    cudaStream_t s = x->stream;
    GA_CUDA(cudaEventRecord(x->ev[3], s));
    GA_CUDA(cudaMemcpyAsync(x->seq.ptr, b->seq, seqBytes, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->seqOff.ptr, b->seq_offset, n * 8ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->seqLen.ptr, b->seq_len, n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->startNode.ptr, b->start_node, n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->startOffset.ptr, b->start_offset, n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->traceOff.ptr, b->trace_offset, n * 8ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->traceCap.ptr, b->trace_capacity, n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->order.ptr, order.data(), n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaEventRecord(x->ev[4], s));
    *db = *b;
    db->seq = x->seq.ptr;
    db->seq_offset = x->seqOff.ptr;
    db->seq_len = x->seqLen.ptr;
    db->start_node = x->startNode.ptr;
    db->start_offset = x->startOffset.ptr;
    db->trace_offset = x->traceOff.ptr;
    db->trace_capacity = x->traceCap.ptr;
    dr->status = x->status.ptr;
    dr->score = x->score.ptr;
    dr->trace_len = x->traceLen.ptr;
    dr->trace_items = x->traceItems.ptr;
    dr->cell_steps = x->cellSteps.ptr;
    *itemsOut = items;
    return GA_OK;
}

static int extend_host_batch(ga_extender* x, const ga_extend_params* p, const ga_extend_batch_desc* b, ga_extend_results* r)
{
    GA_CUDA(cudaSetDevice(x->graph->device));
    x->lastH2DMs = x->lastD2HMs = 0;
    const uint32_t n = b->num;
    if (n == 0) return GA_OK;
    ga_extend_batch_desc db;
    ga_extend_results dr;
    uint64_t items = 0;
    int rc = stage_host_batch(x, b, &db, &dr, &items);
    if (rc != GA_OK) return rc;
    cudaStream_t s = x->stream;
    rc = run_device(x, p, &db, &dr, x->order.ptr, x->prevStatus.ptr, sum_lengths(b->seq_len, n), s);
    if (rc != GA_OK) return rc;
    GA_CUDA(cudaMemcpyAsync(r->status, dr.status, n * 4ULL, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaMemcpyAsync(r->score, dr.score, n * 4ULL, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaMemcpyAsync(r->trace_len, dr.trace_len, n * 4ULL, cudaMemcpyDeviceToHost, s));
    if (r->cell_steps) GA_CUDA(cudaMemcpyAsync(r->cell_steps, dr.cell_steps, n * 8ULL, cudaMemcpyDeviceToHost, s));
    // trace items: chunks on the copy streams, each after the kernels
    GA_CUDA(cudaEventRecord(x->ev[2], s));
    const uint64_t chunk = (items + ga_extender::kCopyStreams - 1) / ga_extender::kCopyStreams;
    for (int k = 0; k < ga_extender::kCopyStreams; k++)
    {
        const uint64_t from = std::min<uint64_t>(items, (uint64_t)k * chunk);
        const uint64_t to = std::min<uint64_t>(items, from + chunk);
        GA_CUDA(cudaStreamWaitEvent(x->copy[k], x->ev[2], 0));
        if (to > from) GA_CUDA(cudaMemcpyAsync(r->trace_items + from, dr.trace_items + from, (to - from) * 8ULL, cudaMemcpyDeviceToHost, x->copy[k]));
        GA_CUDA(cudaEventRecord(x->copyDone[k], x->copy[k]));
        GA_CUDA(cudaStreamWaitEvent(s, x->copyDone[k], 0));
    }
    GA_CUDA(cudaEventRecord(x->ev[5], s));
    GA_CUDA(cudaStreamSynchronize(s));
    GA_CUDA(cudaEventElapsedTime(&x->lastH2DMs, x->ev[3], x->ev[4]));
    GA_CUDA(cudaEventElapsedTime(&x->lastD2HMs, x->ev[2], x->ev[5]));
    return GA_OK;
}

extern "C" int ga_extend_batch(ga_extender_t x, const ga_extend_params* p, const ga_extend_batch_desc* b, ga_extend_results* r)
{
    if (!x || !p || !b || !r) return fail(GA_ERR_ARGUMENT, "null argument");
    return with_store_given_back(x, [&] { return extend_host_batch(x, p, b, r); });
}

// ---- multiseed DP ----

// The multiseed batch with the caller's room (r) or, with ex, exact room in the extender's
// own buffers: each pass's finished reads get their room once their traces are counted.
static int multiseed_run(ga_extender_t x, const ga_extend_params* p, const ga_multiseed_batch_desc* b, ga_multiseed_results* r,
    ga_multiseed_output* ex)
{
    if (!x || !p || !b || (!r && !ex)) return fail(GA_ERR_ARGUMENT, "null argument");
    const bool exact = ex != nullptr;
    const uint32_t n = b->num;
    if (exact)
    {
        MsExactOut& o = x->msOut;
        o.status.assign(n, 0);
        o.numTraces.assign(n, 0);
        o.traceFirst.assign(n, 0);
        o.cellSteps.assign(n, 0);
        o.traces = 0;
        o.items = 0;
        o.publish(ex);
    }
    if (n == 0) return GA_OK;
    if (!b->seq || !b->seq_offset || !b->seq_len || !b->seed_offset)
        return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: a required array is NULL");
    if (!exact && (!b->trace_offset || !b->trace_capacity || !r->status || !r->num_traces || !r->trace_score || !r->trace_start || !r->trace_len
        || !r->trace_items))
        return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: a required array is NULL");
    if (!exact && b->max_traces == 0) return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: max_traces must be at least 1");
    int rc = check_lengths(b->seq_len, n);
    if (rc != GA_OK) return rc;
    // seeds: in the graph, within their read, in slice order
    const uint64_t seedBase = b->seed_offset[0];
    const uint64_t seedEnd = b->seed_offset[n];
    if (seedEnd > seedBase && (!b->seed_slice || !b->seed_node)) return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: seeds without seed arrays");
    for (uint32_t i = 0; i < n; i++)
    {
        if (b->seed_offset[i + 1] < b->seed_offset[i]) return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: seed_offset decreases at read " + std::to_string(i));
        const uint32_t slices = (b->seq_len[i] + 63) / 64;
        for (uint64_t k = b->seed_offset[i]; k < b->seed_offset[i + 1]; k++)
        {
            if (b->seed_node[k] >= x->graph->N || b->seed_slice[k] >= slices || (k > b->seed_offset[i] && b->seed_slice[k] < b->seed_slice[k - 1]))
                return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: read " + std::to_string(i) + " seed " + std::to_string(k - b->seed_offset[i])
                    + " is outside the graph or the read, or out of slice order");
        }
    }
    GA_CUDA(cudaSetDevice(x->graph->device));
    uint64_t seqBytes = 0, items = 0;
    for (uint32_t i = 0; i < n; i++)
    {
        seqBytes = std::max<uint64_t>(seqBytes, b->seq_offset[i] + b->seq_len[i]);
        if (!exact) items = std::max<uint64_t>(items, b->trace_offset[i] + b->trace_capacity[i]);
    }
    const uint64_t seeds = seedEnd;     // seed arrays are indexed from 0 as given
    const uint64_t tables = exact ? 0 : (uint64_t)n * b->max_traces;
    std::vector<uint32_t>& order = x->orderHost;
    order = longest_first(b->seq_len, n);
    GA_CUDA(x->seq.reserve(std::max<uint64_t>(seqBytes, 1)));
    GA_CUDA(x->seqOff.reserve(n));
    GA_CUDA(x->seqLen.reserve(n));
    GA_CUDA(x->msSeedOff.reserve(n + 1));
    GA_CUDA(x->msSeedSlice.reserve(std::max<uint64_t>(seeds, 1)));
    GA_CUDA(x->msSeedNode.reserve(std::max<uint64_t>(seeds, 1)));
    GA_CUDA(x->traceOff.reserve(n));
    GA_CUDA(x->msTraceCap.reserve(n));
    GA_CUDA(x->order.reserve(n));
    GA_CUDA(x->status.reserve(n));
    GA_CUDA(x->prevStatus.reserve(n));
    GA_CUDA(x->msNumTraces.reserve(n));
    GA_CUDA(x->msItemsNeeded.reserve(n));
    GA_CUDA(x->msTracesNeeded.reserve(n));
    GA_CUDA(x->cellSteps.reserve(n));
    GA_CUDA(x->msTraceScore.reserve(std::max<uint64_t>(tables, 1)));
    GA_CUDA(x->msTraceStart.reserve(std::max<uint64_t>(tables, 1)));
    GA_CUDA(x->msTraceLen.reserve(std::max<uint64_t>(tables, 1)));
    GA_CUDA(x->traceItems.reserve(std::max<uint64_t>(items, 1)));
    if (exact)
    {
        GA_CUDA(x->msTraceBase.reserve(n));
    }
    GA_CUDA(x->states.reserve(n));
    GA_CUDA(x->msCandBegin.reserve(n));
    GA_CUDA(x->msCandCount.reserve(n));
    GA_CUDA(x->msCandPart.reserve((size_t)n * gadev::kCandParts));
    GA_CUDA(x->msSel.reserve(n));
    cudaStream_t s = x->stream;
    GA_CUDA(cudaMemcpyAsync(x->seq.ptr, b->seq, seqBytes, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->seqOff.ptr, b->seq_offset, n * 8ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->seqLen.ptr, b->seq_len, n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemcpyAsync(x->msSeedOff.ptr, b->seed_offset, (n + 1) * 8ULL, cudaMemcpyHostToDevice, s));
    if (seeds)
    {
        GA_CUDA(cudaMemcpyAsync(x->msSeedSlice.ptr, b->seed_slice, seeds * 4, cudaMemcpyHostToDevice, s));
        GA_CUDA(cudaMemcpyAsync(x->msSeedNode.ptr, b->seed_node, seeds * 4, cudaMemcpyHostToDevice, s));
    }
    if (!exact)
    {
        GA_CUDA(cudaMemcpyAsync(x->traceOff.ptr, b->trace_offset, n * 8ULL, cudaMemcpyHostToDevice, s));
        GA_CUDA(cudaMemcpyAsync(x->msTraceCap.ptr, b->trace_capacity, n * 8ULL, cudaMemcpyHostToDevice, s));
    }
    GA_CUDA(cudaMemcpyAsync(x->order.ptr, order.data(), n * 4ULL, cudaMemcpyHostToDevice, s));
    GA_CUDA(cudaMemsetAsync(x->msItemsNeeded.ptr, 0, n * 8ULL, s));
    GA_CUDA(cudaMemsetAsync(x->msTracesNeeded.ptr, 0, n * 4ULL, s));

    gadev::FillArgs fa {};
    fa.g = x->graph->d;
    fa.bandwidth = p->bandwidth;
    fa.xdrop = p->xdrop;
    fa.maxCells = p->max_cells_per_slice;
    fa.cost = p->xscore_error_cost;
    fa.num = n;
    fa.order = x->order.ptr;
    fa.seq = x->seq.ptr;
    fa.seqOff = x->seqOff.ptr;
    fa.seqLen = x->seqLen.ptr;
    fa.arena = x->arena;
    fa.arenaBytes = x->arenaBytes;
    fa.arenaCursor = x->arenaCursor;
    fa.states = x->states.ptr;
    fa.seedOff = x->msSeedOff.ptr;
    fa.seedSlice = x->msSeedSlice.ptr;
    fa.seedNode = x->msSeedNode.ptr;
    fa.chunkBytes = (uint64_t)x->shape.chunk_kib << 10;
    reserve_store(x, 2 * sum_lengths(b->seq_len, n), std::min<uint64_t>(n, (uint64_t)x->sms * 16));
    fa.store = x->store;
    fa.storeUnits = x->storeUnits;
    gadev::MultiTraceArgs ta {};
    ta.store = x->store;
    ta.g = x->graph->d;
    ta.cost = p->xscore_error_cost;
    ta.num = n;
    ta.order = x->order.ptr;
    ta.states = x->states.ptr;
    ta.seq = x->seq.ptr;
    ta.seqOff = x->seqOff.ptr;
    ta.seqLen = x->seqLen.ptr;
    ta.arena = x->arena;
    ta.traceOffset = exact ? nullptr : x->traceOff.ptr;
    ta.traceCap = exact ? nullptr : x->msTraceCap.ptr;
    ta.maxTraces = exact ? 0 : b->max_traces;
    ta.traceBase = exact ? x->msTraceBase.ptr : nullptr;
    ta.itemBias = 0;
    ta.multimapScoreFraction = b->multimap_score_fraction;
    ta.status = x->status.ptr;
    ta.numTraces = x->msNumTraces.ptr;
    ta.traceScore = x->msTraceScore.ptr;
    ta.traceStart = x->msTraceStart.ptr;
    ta.traceLen = x->msTraceLen.ptr;
    ta.traceItems = x->traceItems.ptr;
    ta.cellSteps = x->cellSteps.ptr;
    ta.itemsNeeded = x->msItemsNeeded.ptr;
    ta.tracesNeeded = x->msTracesNeeded.ptr;
    ta.candBegin = x->msCandBegin.ptr;
    ta.candCount = x->msCandCount.ptr;
    ta.candPart = x->msCandPart.ptr;
    ta.candTotal = (unsigned long long*)(x->counters + 8);

    x->lastFillMs = 0;
    x->lastLaunches = 0;
    x->lastCandidates = 0;
    x->lastKept = 0;
    x->lastWalks = 0;
    x->lastResolveRounds = 0;
    for (int k = 0; k < 3; k++) x->lastRounds[k] = 0;
    const int wpb = 4;
    uint32_t pending = n;
    // The frontier tables are in the global workspace: the multiseed band holds every seed
    // start of a slice besides the alignments' own nodes.  A read that runs out of room (its
    // tables, or the arena the batch shares) runs again in the next pass, which starts a fresh
    // arena; passes go on while they finish reads, then once more with the large tables.  A
    // read whose traces outgrow its output room (kMsRoom) is not run again: it reports the
    // room it needs.  Between the fill and the traceback the host sizes the candidate list.
    int layout = 1;
    std::vector<uint8_t> finished(exact ? n : 0, 0);
    std::vector<uint64_t> traceBase(exact ? n : 0, 0);
    for (int pass = 0; pass < 32; pass++)
    {
        const gadev::Caps caps = layout_caps(layout);
        const uint64_t stride = ga_multiseed_tables_bytes(caps);
        const uint64_t pendingBlocks = std::max<uint64_t>(1, ((uint64_t)pending + wpb - 1) / wpb);
        uint64_t fillBlocks = std::min<uint64_t>((uint64_t)x->sms * 16, std::max<uint64_t>(1, pending));
        fillBlocks = std::max<uint64_t>(1, std::min<uint64_t>(fillBlocks, x->workspaceBytes / stride));
        const uint64_t readBlocks = std::min<uint64_t>((uint64_t)x->sms * 6, pendingBlocks);
        const uint64_t partBlocks = std::min<uint64_t>((uint64_t)x->sms * 6, ((uint64_t)pending * gadev::kCandParts + wpb - 1) / wpb);
        if (pass > 0) GA_CUDA(cudaMemcpyAsync(x->prevStatus.ptr, x->status.ptr, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));
        fa.caps = caps;
        fa.workspace = x->workspace;
        fa.workspaceStride = stride;
        fa.prevStatus = pass > 0 ? x->prevStatus.ptr : nullptr;
        ta.prevStatus = fa.prevStatus;
        GA_CUDA(cudaMemsetAsync(x->counters, 0, 16 * sizeof(uint32_t), s));
        GA_CUDA(cudaMemsetAsync(x->arenaCursor, 0, 3 * sizeof(unsigned long long), s));
        GA_CUDA(cudaEventRecord(x->ev[0], s));
        if (ga_launch_multiseed_fill(fa, ta, x->counters, (int)fillBlocks, (int)partBlocks, wpb, s) != 0)
            return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
        unsigned long long candTotal = 0;
        GA_CUDA(cudaMemcpyAsync(&candTotal, ta.candTotal, 8, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaStreamSynchronize(s));
        GA_CUDA(x->msCands.reserve(std::max<uint64_t>(candTotal, 1)));
        ta.cands = x->msCands.ptr;
        ta.candCap = x->msCands.count;
        x->lastCandidates += candTotal;
        if (candTotal > 0xffffffffULL) return fail(GA_ERR_ARGUMENT, "ga_multiseed_batch: more than 2^32 - 1 trace candidates in one batch");
        GA_CUDA(x->msWork.reserve(std::max<uint64_t>(candTotal, 1)));
        ta.work = x->msWork.ptr;
        ta.workCount = x->counters + 7;
        ta.sel = x->msSel.ptr;
        const uint64_t candBlocks = std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)x->sms * 6, (candTotal + wpb - 1) / wpb));
        GA_CUDA(cudaMemsetAsync(x->msSel.ptr, 0, n * sizeof(gadev::MsSel), s));
        if (ga_launch_multiseed_list(ta, x->counters, (int)partBlocks, wpb, s) != 0)
            return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
        x->lastLaunches += 4;
        // rounds: each read decides its candidates as far as their walks are known and queues
        // the next walks, twice as many each round, up to 1024, and at least as many as there are
        // warps for: a round takes as long as its longest walk, so walks that may turn out not to be
        // needed cost nothing on warps that would be idle (40 reads: 7 rounds of 5 ms without)
        const uint32_t idle = std::min<uint32_t>(1024, std::max<uint32_t>(1, (uint32_t)x->sms * 16 / pending));
        for (uint32_t round = 0;; round++)
        {
            GA_CUDA(cudaMemsetAsync(x->counters + 4, 0, 4 * sizeof(uint32_t), s));
            ta.window = std::max(idle, round < 10 ? 1u << round : 1024u);
            if (ga_launch_multiseed_resolve(ta, x->counters, (int)readBlocks, wpb, s) != 0)
                return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
            uint32_t walks = 0;
            GA_CUDA(cudaMemcpyAsync(&walks, ta.workCount, 4, cudaMemcpyDeviceToHost, s));
            GA_CUDA(cudaStreamSynchronize(s));
            x->lastLaunches += 1;
            if (walks == 0) break;
            x->lastWalks += walks;
            x->lastResolveRounds++;
            const uint64_t walkBlocks = std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)x->sms * 6, ((uint64_t)walks + wpb - 1) / wpb));
            if (ga_launch_multiseed_walk(ta, x->counters, (int)walkBlocks, wpb, s) != 0)
                return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
            x->lastLaunches += 1;
        }
        if (exact)
        {
            // The reads this pass finished list their kept traces; the host removes the
            // duplicates (removeDuplicateTraces, as getMultiseedTraces does), and the survivors
            // get trace and item runs after the earlier passes' (this pass's tables are gone
            // once the next one starts).  Only the survivors are written and copied back.
            // (only the reads this pass finished take their status and kept count from the
            // device: the others keep what their own pass gave them)
            MsExactOut& o = x->msOut;
            std::vector<int32_t> passStatus(n);
            std::vector<uint32_t> passKeptCount(n);
            GA_CUDA(cudaMemcpyAsync(passStatus.data(), x->status.ptr, n * 4ULL, cudaMemcpyDeviceToHost, s));
            GA_CUDA(cudaMemcpyAsync(passKeptCount.data(), x->msNumTraces.ptr, n * 4ULL, cudaMemcpyDeviceToHost, s));
            GA_CUDA(cudaStreamSynchronize(s));
            std::vector<uint32_t> passReads;
            uint64_t passKept = 0;
            for (uint32_t i = 0; i < n; i++)
            {
                if (finished[i] || passStatus[i] == GA_CAPACITY) continue;
                finished[i] = 1;
                o.status[i] = passStatus[i];
                o.numTraces[i] = passKeptCount[i];
                if (o.status[i] != GA_OK) continue;
                traceBase[i] = passKept;
                passKept += o.numTraces[i];
                passReads.push_back(i);
            }
            x->lastKept += passKept;
            GA_CUDA(x->msKeys.reserve(std::max<uint64_t>(passKept, 1)));
            GA_CUDA(x->msKeptSlot.reserve(std::max<uint64_t>(passKept, 1)));
            GA_CUDA(x->msKeptItem.reserve(std::max<uint64_t>(passKept, 1)));
            GA_CUDA(cudaMemcpyAsync(x->msTraceBase.ptr, traceBase.data(), n * 8ULL, cudaMemcpyHostToDevice, s));
            ta.keys = x->msKeys.ptr;
            ta.keptSlot = x->msKeptSlot.ptr;
            ta.keptItem = x->msKeptItem.ptr;
            std::vector<gadev::MsKey> keys(passKept);
            if (passKept)
            {
                if (ga_launch_multiseed_keys(ta, s) != 0)
                    return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
                x->lastLaunches += 1;
                GA_CUDA(cudaMemcpyAsync(keys.data(), x->msKeys.ptr, passKept * sizeof(gadev::MsKey), cudaMemcpyDeviceToHost, s));
                GA_CUDA(cudaStreamSynchronize(s));
            }
            std::vector<uint32_t> keptSlot(passKept, gadev::kNoSlot);
            std::vector<uint64_t> keptItem(passKept, 0);
            uint64_t passTraces = 0, passItems = 0;
            std::vector<gahost::DedupeKey> dk;
            for (uint32_t i : passReads)
            {
                const uint64_t base = traceBase[i];
                dk.resize(o.numTraces[i]);
                for (uint32_t t = 0; t < o.numTraces[i]; t++)
                {
                    const gadev::MsKey& k = keys[base + t];
                    const uint64_t start = (uint64_t)k.lastNode | ((uint64_t)(k.lastOff & 63) << 32) | ((uint64_t)(k.last + 1) << 39);
                    dk[t] = gahost::DedupeKey { gahost::dedupeScore((size_t)k.first, (size_t)k.last, k.score, p->xscore_error_cost), t, start };
                }
                const std::vector<uint32_t> order = gahost::dedupeOrder(dk);
                o.traceFirst[i] = o.traces + passTraces;
                o.numTraces[i] = (uint32_t)order.size();
                for (uint32_t t : order)
                {
                    keptSlot[base + t] = (uint32_t)passTraces++;
                    keptItem[base + t] = passItems;
                    passItems += keys[base + t].len;
                }
            }
            if (passKept)
            {
                GA_CUDA(cudaMemcpyAsync(x->msKeptSlot.ptr, keptSlot.data(), passKept * 4, cudaMemcpyHostToDevice, s));
                GA_CUDA(cudaMemcpyAsync(x->msKeptItem.ptr, keptItem.data(), passKept * 8, cudaMemcpyHostToDevice, s));
            }
            GA_CUDA(x->msTraceScore.reserve(std::max<uint64_t>(passTraces, 1)));
            GA_CUDA(x->msTraceStart.reserve(std::max<uint64_t>(passTraces, 1)));
            GA_CUDA(x->msTraceLen.reserve(std::max<uint64_t>(passTraces, 1)));
            GA_CUDA(x->traceItems.reserve(std::max<uint64_t>(passItems, 1)));
            ta.traceScore = x->msTraceScore.ptr;
            ta.traceStart = x->msTraceStart.ptr;
            ta.traceLen = x->msTraceLen.ptr;
            ta.traceItems = x->traceItems.ptr;
            ta.itemBias = o.items;
            if (ga_launch_multiseed_write(ta, x->counters, (int)candBlocks, wpb, s) != 0)
                return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
            if (!o.grow(o.traces + passTraces, o.items + passItems))
                return fail(GA_ERR_CUDA, "ga_multiseed_batch_exact: pinned host memory for the traces");
            if (passTraces)
            {
                GA_CUDA(cudaMemcpyAsync(o.score.ptr + o.traces, x->msTraceScore.ptr, passTraces * 4, cudaMemcpyDeviceToHost, s));
                GA_CUDA(cudaMemcpyAsync(o.start.ptr + o.traces, x->msTraceStart.ptr, passTraces * 8, cudaMemcpyDeviceToHost, s));
                GA_CUDA(cudaMemcpyAsync(o.len.ptr + o.traces, x->msTraceLen.ptr, passTraces * 4, cudaMemcpyDeviceToHost, s));
            }
            if (passItems) GA_CUDA(cudaMemcpyAsync(o.item.ptr + o.items, x->traceItems.ptr, passItems * 8, cudaMemcpyDeviceToHost, s));
            o.traces += passTraces;
            o.items += passItems;
        }
        else
        {
            if (ga_launch_multiseed_write(ta, x->counters, (int)candBlocks, wpb, s) != 0)
                return fail(GA_ERR_CUDA, std::string("multiseed kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
        }
        x->lastLaunches += 1;
        x->lastRounds[layout] += pending;
        GA_CUDA(cudaEventRecord(x->ev[1], s));
        count_status_kernel<<<64, 256, 0, s>>>(x->status.ptr, n, GA_CAPACITY, x->counters + 2);
        GA_CUDA(cudaGetLastError());
        x->lastLaunches += 1;
        uint32_t capFails = 0;
        unsigned long long used[2] = {0, 0};
        GA_CUDA(cudaMemcpyAsync(&capFails, x->counters + 2, 4, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaMemcpyAsync(used, x->arenaCursor, 16, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaStreamSynchronize(s));
        if (pass == 0) x->lastArenaBytes = used[1];
        float ms = 0;
        GA_CUDA(cudaEventElapsedTime(&ms, x->ev[0], x->ev[1]));
        x->lastFillMs += ms;
        const bool progress = capFails < pending;
        pending = capFails;
        if (capFails == 0) break;
        if (!progress)
        {
            if (layout == 2) break;
            layout = 2;
        }
    }
    if (exact)
    {
        // a kept trace whose written walk failed fails its read after the counts were taken
        MsExactOut& o = x->msOut;
        GA_CUDA(cudaMemcpyAsync(o.status.data(), x->status.ptr, n * 4ULL, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaMemcpyAsync(o.cellSteps.data(), x->cellSteps.ptr, n * 8ULL, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaStreamSynchronize(s));
        for (uint32_t i = 0; i < n; i++)
            if (o.status[i] != GA_OK) o.numTraces[i] = 0;
        o.publish(ex);
        return GA_OK;
    }
    GA_CUDA(cudaMemcpyAsync(r->status, x->status.ptr, n * 4ULL, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaMemcpyAsync(r->num_traces, x->msNumTraces.ptr, n * 4ULL, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaMemcpyAsync(r->trace_score, x->msTraceScore.ptr, tables * 4, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaMemcpyAsync(r->trace_start, x->msTraceStart.ptr, tables * 8, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaMemcpyAsync(r->trace_len, x->msTraceLen.ptr, tables * 4, cudaMemcpyDeviceToHost, s));
    if (r->cell_steps) GA_CUDA(cudaMemcpyAsync(r->cell_steps, x->cellSteps.ptr, n * 8ULL, cudaMemcpyDeviceToHost, s));
    if (r->items_needed) GA_CUDA(cudaMemcpyAsync(r->items_needed, x->msItemsNeeded.ptr, n * 8ULL, cudaMemcpyDeviceToHost, s));
    if (r->traces_needed) GA_CUDA(cudaMemcpyAsync(r->traces_needed, x->msTracesNeeded.ptr, n * 4ULL, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaStreamSynchronize(s));
    for (uint32_t i = 0; i < n; i++)
    {
        if (r->status[i] == gadev::kMsRoom) r->status[i] = GA_CAPACITY;
        if (r->status[i] == GA_OK) x->lastKept += r->num_traces[i];
    }
    // Trace items: a read's traces lie back to back from its trace_offset, and only those come
    // back (the room is usually far larger), in runs that take in gaps of up to 256 KiB.
    const uint64_t kGap = 32768;
    uint64_t runFrom = 0, runTo = 0;
    bool open = false;
    for (uint32_t i = 0; i < n; i++)
    {
        if (r->status[i] != GA_OK) continue;
        uint64_t used = 0;
        for (uint32_t t = 0; t < r->num_traces[i]; t++) used += r->trace_len[(uint64_t)i * b->max_traces + t];
        if (used == 0) continue;
        const uint64_t from = b->trace_offset[i], to = from + used;
        if (open && from >= runTo && from - runTo <= kGap)
        {
            runTo = to;
            continue;
        }
        if (open) GA_CUDA(cudaMemcpyAsync(r->trace_items + runFrom, x->traceItems.ptr + runFrom, (runTo - runFrom) * 8, cudaMemcpyDeviceToHost, s));
        runFrom = from;
        runTo = to;
        open = true;
    }
    if (open) GA_CUDA(cudaMemcpyAsync(r->trace_items + runFrom, x->traceItems.ptr + runFrom, (runTo - runFrom) * 8, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaStreamSynchronize(s));
    return GA_OK;
}

extern "C" int ga_multiseed_batch(ga_extender_t x, const ga_extend_params* p, const ga_multiseed_batch_desc* b, ga_multiseed_results* r)
{
    if (!x || !r) return fail(GA_ERR_ARGUMENT, "null argument");
    return with_store_given_back(x, [&] { return multiseed_run(x, p, b, r, nullptr); });
}

extern "C" int ga_multiseed_batch_exact(ga_extender_t x, const ga_extend_params* p, const ga_multiseed_batch_desc* b, ga_multiseed_output* out)
{
    if (!x || !out) return fail(GA_ERR_ARGUMENT, "null argument");
    return with_store_given_back(x, [&] { return multiseed_run(x, p, b, nullptr, out); });
}

static int autotune(ga_extender* x, const ga_extend_params* p, const ga_extend_batch_desc* b, const ga_launch_shape* shapes, uint32_t count,
    uint32_t repeats, float* ms_out)
{
    GA_CUDA(cudaSetDevice(x->graph->device));
    x->lastH2DMs = x->lastD2HMs = 0;
    const uint32_t n = b->num;
    if (n == 0) return GA_OK;
    repeats = std::max<uint32_t>(repeats, 1);
    ga_extend_batch_desc db;
    ga_extend_results dr;
    uint64_t items = 0;
    int rc = stage_host_batch(x, b, &db, &dr, &items);
    if (rc != GA_OK) return rc;
    cudaStream_t s = x->stream;
    std::vector<int32_t> refStatus(n), refScore(n), status(n), score(n);
    uint32_t best = 0;
    float bestMs = 0;
    for (uint32_t i = 0; i < count; i++)
    {
        x->shape = shapes[i];
        std::vector<float> ms;
        for (uint32_t rep = 0; rep < repeats; rep++)
        {
            rc = run_device(x, p, &db, &dr, x->order.ptr, x->prevStatus.ptr, sum_lengths(b->seq_len, n), s);
            if (rc != GA_OK) return rc;
            ms.push_back(x->lastFillMs);
        }
        std::sort(ms.begin(), ms.end());
        const float median = ms[ms.size() / 2];
        if (ms_out) ms_out[i] = median;
        if (i == 0 || median < bestMs) { best = i; bestMs = median; }
        int32_t* st = i == 0 ? refStatus.data() : status.data();
        int32_t* sc = i == 0 ? refScore.data() : score.data();
        GA_CUDA(cudaMemcpyAsync(st, dr.status, n * 4ULL, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaMemcpyAsync(sc, dr.score, n * 4ULL, cudaMemcpyDeviceToHost, s));
        GA_CUDA(cudaStreamSynchronize(s));
        if (i > 0 && (status != refStatus || score != refScore))
        {
            x->shape = shapes[0];
            return fail(GA_ERR_STATE, "launch shape " + std::to_string(i) + " changed results");
        }
    }
    x->shape = shapes[best];
    return GA_OK;
}

extern "C" int ga_extender_autotune(ga_extender_t x, const ga_extend_params* p, const ga_extend_batch_desc* b,
    const ga_launch_shape* shapes, uint32_t count, uint32_t repeats, float* ms_out)
{
    if (!x || !p || !b || !shapes) return fail(GA_ERR_ARGUMENT, "null argument");
    if (count == 0) return fail(GA_ERR_ARGUMENT, "no launch shapes");
    for (uint32_t i = 0; i < count; i++)
        if (!shape_ok(shapes[i])) return fail(GA_ERR_ARGUMENT, kShapeError);
    return with_store_given_back(x, [&] { return autotune(x, p, b, shapes, count, repeats, ms_out); });
}

static int extend_device_batch(ga_extender* x, const ga_extend_params* p, const ga_extend_batch_desc* b, ga_extend_results* r, void* stream)
{
    GA_CUDA(cudaSetDevice(x->graph->device));
    x->lastH2DMs = x->lastD2HMs = 0;
    const uint32_t n = b->num;
    if (n == 0) return GA_OK;
    // the processing order needs the lengths; read them back once (4 bytes per extension)
    std::vector<uint32_t> len(n);
    cudaStream_t s = stream ? (cudaStream_t)stream : x->stream;
    GA_CUDA(cudaMemcpyAsync(len.data(), b->seq_len, n * 4ULL, cudaMemcpyDeviceToHost, s));
    GA_CUDA(cudaStreamSynchronize(s));
    int rc = check_lengths(len.data(), n);
    if (rc != GA_OK) return rc;
    std::vector<uint32_t> order = longest_first(len.data(), n);
    GA_CUDA(x->order.reserve(n));
    GA_CUDA(x->prevStatus.reserve(n));
    GA_CUDA(cudaMemcpyAsync(x->order.ptr, order.data(), n * 4ULL, cudaMemcpyHostToDevice, s));
    return run_device(x, p, b, r, x->order.ptr, x->prevStatus.ptr, sum_lengths(len.data(), n), s);
}

extern "C" int ga_extend_batch_device(ga_extender_t x, const ga_extend_params* p, const ga_extend_batch_desc* b,
    ga_extend_results* r, void* stream)
{
    if (!x || !p || !b || !r) return fail(GA_ERR_ARGUMENT, "null argument");
    return with_store_given_back(x, [&] { return extend_device_batch(x, p, b, r, stream); });
}

extern "C" int ga_extender_last_kernel_ms(ga_extender_t x, float* ms)
{
    if (!x || !ms) return fail(GA_ERR_ARGUMENT, "null argument");
    *ms = x->lastFillMs + x->lastTraceMs;
    return GA_OK;
}

extern "C" int ga_extender_last_times(ga_extender_t x, float* fill_ms, float* trace_ms)
{
    if (!x || !fill_ms || !trace_ms) return fail(GA_ERR_ARGUMENT, "null argument");
    *fill_ms = x->lastFillMs;
    *trace_ms = x->lastTraceMs;   // the traceback runs inside the same kernel as the fill
    return GA_OK;
}

extern "C" int ga_extender_last_copy_ms(ga_extender_t x, float* h2d_ms, float* d2h_ms)
{
    if (!x || !h2d_ms || !d2h_ms) return fail(GA_ERR_ARGUMENT, "null argument");
    *h2d_ms = x->lastH2DMs;
    *d2h_ms = x->lastD2HMs;
    return GA_OK;
}

extern "C" int ga_extender_last_launches(ga_extender_t x, uint32_t* launches)
{
    if (!x || !launches) return fail(GA_ERR_ARGUMENT, "null argument");
    *launches = x->lastLaunches;
    return GA_OK;
}

extern "C" int ga_extender_set_launch_shape(ga_extender_t x, const ga_launch_shape* shape)
{
    if (!x || !shape) return fail(GA_ERR_ARGUMENT, "null argument");
    if (!shape_ok(*shape)) return fail(GA_ERR_ARGUMENT, kShapeError);
    x->shape = *shape;
    return GA_OK;
}

extern "C" int ga_extender_set_store_limit(ga_extender_t x, uint64_t max_bytes)
{
    if (!x) return fail(GA_ERR_ARGUMENT, "null argument");
    GA_CUDA(cudaSetDevice(x->graph->device));
    x->storeLimit = max_bytes;
    if (x->store && (x->storeUnits + gadev::kStorePad) * sizeof(gadev::ColumnUnit) > max_bytes) release_store(x);
    return GA_OK;
}

extern "C" int ga_extender_get_launch_shape(ga_extender_t x, ga_launch_shape* shape)
{
    if (!x || !shape) return fail(GA_ERR_ARGUMENT, "null argument");
    *shape = x->shape;
    return GA_OK;
}

extern "C" int ga_extender_last_arena_bytes(ga_extender_t x, uint64_t* bytes)
{
    if (!x || !bytes) return fail(GA_ERR_ARGUMENT, "null argument");
    *bytes = x->lastArenaBytes;
    return GA_OK;
}

extern "C" int ga_extender_last_layout_counts(ga_extender_t x, uint32_t counts[3])
{
    if (!x || !counts) return fail(GA_ERR_ARGUMENT, "null argument");
    for (int k = 0; k < 3; k++) counts[k] = x->lastRounds[k];
    return GA_OK;
}

extern "C" int ga_extender_last_multiseed_counts(ga_extender_t x, uint64_t* candidates, uint64_t* walks, uint64_t* traces, uint32_t* rounds)
{
    if (!x || !candidates || !walks || !traces || !rounds) return fail(GA_ERR_ARGUMENT, "null argument");
    *candidates = x->lastCandidates;
    *walks = x->lastWalks;
    *traces = x->lastKept;
    *rounds = x->lastResolveRounds;
    return GA_OK;
}

namespace
{
// Independent chains of 32-bit xor + add (LOP3 + IADD3 in SASS), the operation mix of
// the Myers column step, to measure the integer-ALU issue rate of this GPU.
__global__ void int_peak_kernel(uint32_t* out, int iters, uint32_t seed)
{
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t a0 = t ^ seed, a1 = t + 1, a2 = t + 2, a3 = t + 3, a4 = t + 4, a5 = t + 5, a6 = t + 6, a7 = t + 7;
    const uint32_t k1 = seed | 1, k2 = seed * 3 + 7;
    for (int i = 0; i < iters; i++)
    {
#pragma unroll
        for (int u = 0; u < 8; u++)
        {
            a0 = (a0 ^ k1) + k2; a1 = (a1 ^ k2) + k1; a2 = (a2 ^ k1) + k2; a3 = (a3 ^ k2) + k1;
            a4 = (a4 ^ k1) + k2; a5 = (a5 ^ k2) + k1; a6 = (a6 ^ k1) + k2; a7 = (a7 ^ k2) + k1;
        }
    }
    uint32_t r = a0 ^ a1 ^ a2 ^ a3 ^ a4 ^ a5 ^ a6 ^ a7;
    if (r == 0x12345678u) out[t] = r;
}
}

extern "C" int ga_measure_int32_peak(int device, double* ops_per_second)
{
    if (!ops_per_second) return fail(GA_ERR_ARGUMENT, "null argument");
    GA_CUDA(cudaSetDevice(device));
    cudaDeviceProp prop;
    GA_CUDA(cudaGetDeviceProperties(&prop, device));
    const int block = 256;
    const int grid = prop.multiProcessorCount * 8;
    const int iters = 4096;
    uint32_t* out = nullptr;
    GA_CUDA(cudaMalloc((void**)&out, (size_t)grid * block * 4));
    cudaEvent_t e0, e1;
    GA_CUDA(cudaEventCreate(&e0));
    GA_CUDA(cudaEventCreate(&e1));
    int_peak_kernel<<<grid, block>>>(out, 64, 1u);
    GA_CUDA(cudaDeviceSynchronize());
    float best = 1e30f;
    for (int rep = 0; rep < 5; rep++)
    {
        GA_CUDA(cudaEventRecord(e0));
        int_peak_kernel<<<grid, block>>>(out, iters, (uint32_t)rep + 3);
        GA_CUDA(cudaEventRecord(e1));
        GA_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        GA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        best = std::min(best, ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    const double ops = (double)grid * block * iters * 8.0 * 8.0 * 2.0;
    *ops_per_second = ops / (best * 1e-3);
    return GA_OK;
}

extern "C" int ga_host_alloc(uint64_t bytes, void** out)
{
    if (!out) return fail(GA_ERR_ARGUMENT, "null argument");
    GA_CUDA(cudaHostAlloc(out, std::max<uint64_t>(bytes, 16), cudaHostAllocDefault));
    return GA_OK;
}

extern "C" int ga_host_free(void* p)
{
    if (p) GA_CUDA(cudaFreeHost(p));
    return GA_OK;
}
