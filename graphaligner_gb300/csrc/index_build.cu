// Minimizer index of the graph built on the GPU (MinimizerSeeder::initMinimizers and
// initMaxCount with one bucket, MinimizerSeeder.cpp:104-189, 299-491, 557-575).
//
// It produces the arrays of the host build in seeding.cpp, element for element:
//   1. one thread per bigraph node (AlignmentGraph::nodeLookup order), or for a node of kLongNode
//      bases and more one thread per base, walks the node's
//      sequence over its pieces and reports its window minimizers (iterateMinimizersReal,
//      ties in hash reported together, restarts after non-ACGT characters) from the end
//      of the last piece entered from another bigraph node on (MinimizerSeeder.cpp:323-340),
//      as (k-mer, (split node << 6) | offset).  A counting pass, an exclusive scan and a
//      writing pass lay the occurrences out in node order;
//   2. a stable LSD radix sort by k-mer (8-bit digits) keeps each k-mer's occurrences in
//      insertion order;
//   3. the distinct k-mers and their first occurrences come from a scan of "new k-mer"
//      flags, and each k-mer's occurrences are written in reverse insertion order, as the
//      reference's counting sort leaves them;
//   4. initMaxCount's quantile of the occurrence counts (every k-mer but the last) is read
//      off a device histogram;
//   5. the open-addressing lookup table (seed_table.h) is filled on the device by
//      compare-and-swap claims.
#include <cuda_runtime.h>
#include <algorithm>
#include <stdint.h>
#include <string>
#include <vector>
#include "index_build.h"
#include "index_walk.cuh"

namespace gadev
{

// Nodes of at least this many bases are not walked by one thread but by a thread per base
// (minimizers_at), in chunks of kChunk bases a block.  A thread's walk takes 1.4 us a base (its
// window lies in local memory), so the unitigs of a de Bruijn graph, up to 100 kbp long, set the
// time of the whole build: 143 ms on the graph of a 1 Mbp genome, 2.0 ms by bases.  The nodes of
// a variation graph are shorter and many, where a block for each would be mostly idle.
static constexpr uint32_t kLongNode = 256;
static constexpr uint32_t kChunk = 256;
static constexpr uint32_t kHalo = 128;      // bases before a chunk that its windows reach: w + 3 <= 31 + 63 + 3

__global__ void count_minimizers_kernel(IndexGraph g, uint32_t k, uint32_t w, uint32_t* counts, uint32_t* error)
{
    const uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= g.numLookup || g.originalSize[li] >= kLongNode) return;
    bool bad = false;
    counts[li] = node_minimizers(g, li, k, w, nullptr, nullptr, bad);
    if (bad) atomicOr(error, 1u);
}

__global__ void write_minimizers_kernel(IndexGraph g, uint32_t k, uint32_t w, const uint32_t* first, uint64_t* kmers, uint64_t* positions,
    uint32_t* order, uint32_t* error)
{
    const uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= g.numLookup || g.originalSize[li] >= kLongNode) return;
    const uint32_t from = first[li];
    bool bad = false;
    const uint32_t n = node_minimizers(g, li, k, w, kmers + from, positions + from, bad);
    if (bad) atomicOr(error, 1u);
    for (uint32_t i = 0; i < n; i++) order[from + i] = from + i;
}

// chunks[li] = the chunks of node li if it is long, else 0
__global__ void count_chunks_kernel(IndexGraph g, uint32_t* chunks)
{
    const uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li < g.numLookup) chunks[li] = g.originalSize[li] >= kLongNode ? (g.originalSize[li] + kChunk - 1) / kChunk : 0;
}

// the node of each chunk
__global__ void chunk_nodes_kernel(IndexGraph g, const uint32_t* firstChunk, uint32_t* chunkNode)
{
    const uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= g.numLookup) return;
    for (uint32_t c = firstChunk[li]; c < firstChunk[li + 1]; c++) chunkNode[c] = li;
}

// A block per chunk: its share of the node's pieces checked (they tile the node in order) and of
// the search for the last piece entered from another bigraph node (minStart, zeroed before).
__global__ void long_nodes_kernel(IndexGraph g, const uint32_t* firstChunk, const uint32_t* chunkNode, uint32_t* minStart, uint32_t* error)
{
    const uint32_t li = chunkNode[blockIdx.x];
    const uint32_t part = blockIdx.x - firstChunk[li], parts = firstChunk[li + 1] - firstChunk[li];
    const uint32_t from = g.lookupOff[li], to = g.lookupOff[li + 1];
    bool bad = from == to;
    uint32_t start = 0;
    for (uint32_t e = from + part * blockDim.x + threadIdx.x; e < to; e += parts * blockDim.x)
    {
        const uint32_t piece = g.lookupNodes[e];
        if (piece >= g.N)
        {
            bad = true;
            continue;
        }
        const uint32_t end = g.nodeOffset[piece] + g.len[piece];
        const uint32_t next = e + 1 < to ? g.lookupNodes[e + 1] : 0;
        if (e + 1 < to ? (next >= g.N || g.nodeOffset[next] != end) : end != g.originalSize[li]) bad = true;
        if (e == from && g.nodeOffset[piece] != 0) bad = true;
        for (uint32_t p = g.inOff[piece]; p < g.inOff[piece + 1]; p++)
            if (g.nodeIds[g.inNb[p]] != g.nodeIds[piece] && g.nodeOffset[piece] > start) start = g.nodeOffset[piece];
    }
    if (bad) atomicOr(error, 1u);
    if (start) atomicMax(&minStart[li], start);
}

// The minimizers of one chunk of a long node, a thread per base: counted (kmers == nullptr), or
// written behind the chunks before it.  The bases of the chunk and of the windows that reach into
// it are laid out in shared memory first, then the k-mers' hashes.
__global__ void __launch_bounds__(kChunk) long_minimizers_kernel(IndexGraph g, uint32_t k, uint32_t w, const uint32_t* firstChunk, const uint32_t* chunkNode,
    const uint32_t* minStart, const uint32_t* error, uint32_t* chunkCount, uint32_t* nodeCount, const uint32_t* first, uint64_t* kmers, uint64_t* positions,
    uint32_t* order)
{
    constexpr uint32_t kBases = kChunk + kHalo;
    __shared__ int8_t code[kBases];
    __shared__ uint32_t pieceOf[kBases];
    __shared__ uint64_t kmerAt[kBases], hashOf[kBases];
    __shared__ uint32_t warpSum[kChunk / 32];
    if (*error) return;                 // pieces that do not tile their node
    const uint32_t li = chunkNode[blockIdx.x];
    const uint32_t size = g.originalSize[li];
    const uint32_t chunkStart = (blockIdx.x - firstChunk[li]) * kChunk;
    const uint32_t base = chunkStart > kHalo ? chunkStart - kHalo : 0;     // node offset of the first base laid out
    const uint32_t end = chunkStart + kChunk < size ? chunkStart + kChunk : size;
    // the last piece that starts at or before `base`
    uint32_t lo = g.lookupOff[li], hi = g.lookupOff[li + 1];
    while (hi - lo > 1)
    {
        const uint32_t mid = (lo + hi) / 2;
        if (g.nodeOffset[g.lookupNodes[mid]] <= base) lo = mid;
        else hi = mid;
    }
    for (uint32_t e = lo + threadIdx.x; e < g.lookupOff[li + 1]; e += kChunk)
    {
        const uint32_t piece = g.lookupNodes[e];
        const uint32_t at = g.nodeOffset[piece];
        if (at >= end) break;
        const uint32_t stop = at + g.len[piece] < end ? at + g.len[piece] : end;
        for (uint32_t p = at < base ? base : at; p < stop; p++)
        {
            code[p - base] = (int8_t)piece_code(g, piece, p - at);
            pieceOf[p - base] = piece;
        }
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < end - base; q += kChunk)
    {
        uint64_t kmer = 0;
        for (uint32_t i = q + 1 < k ? 0 : q + 1 - k; i <= q; i++) kmer = (kmer << 2) | (uint64_t)(code[i] & 3);
        kmerAt[q] = kmer;
        hashOf[q] = kmer_hash(kmer);
    }
    __syncthreads();
    const uint32_t P = chunkStart + threadIdx.x;
    uint32_t run = 0;
    if (P < end)
        while (run < w + 3 && run <= P - base && code[P - base - run] >= 0) run++;
    const uint32_t from = minStart[li];
    auto hashAt = [&](uint32_t p) { return hashOf[p - base]; };
    uint32_t n = 0;
    minimizers_at(P, run, k, w, hashAt, [&](uint32_t p) { if (p >= from) n++; });
    // this thread's place among the chunk's minimizers
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = n;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1)
    {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
    }
    if (lane == 31) warpSum[warp] = incl;
    __syncthreads();
    uint32_t before = incl - n, all = 0;
    for (uint32_t q = 0; q < kChunk / 32; q++)
    {
        if (q < warp) before += warpSum[q];
        all += warpSum[q];
    }
    if (!kmers)
    {
        if (threadIdx.x == 0)
        {
            chunkCount[blockIdx.x] = all;
            if (all) atomicAdd(&nodeCount[li], all);
        }
        return;
    }
    // chunkCount is scanned by now
    uint32_t to = first[li] + chunkCount[blockIdx.x] - chunkCount[firstChunk[li]] + before;
    minimizers_at(P, run, k, w, hashAt, [&](uint32_t p)
    {
        if (p < from) return;
        const uint32_t piece = pieceOf[p - base];
        kmers[to] = kmerAt[p - base];
        positions[to] = ((uint64_t)piece << 6) + (p - g.nodeOffset[piece]);
        order[to] = to;
        to++;
    });
}

// ---------------------------------------------------------------- exclusive scan (u32)

static constexpr uint32_t kScanBlock = 1024;   // elements per block: 256 threads x 4

// scans each block's 1024 elements in place and writes the block's total
__global__ void scan_blocks_kernel(uint32_t* data, uint32_t n, uint32_t* blockSums)
{
    __shared__ uint32_t warpTotals[8];
    const uint32_t base = blockIdx.x * kScanBlock + threadIdx.x * 4;
    uint32_t v[4];
    uint32_t local = 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        v[q] = base + q < n ? data[base + q] : 0;
        local += v[q];
    }
    // inclusive scan of the per-thread totals within the warp, then across the warps
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = local;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1)
    {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) warpTotals[warp] = incl;
    __syncthreads();
    uint32_t warpBase = 0;
    for (uint32_t q = 0; q < warp; q++) warpBase += warpTotals[q];
    uint32_t running = warpBase + incl - local;
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        if (base + q < n) data[base + q] = running;
        running += v[q];
    }
    if (threadIdx.x == 255) blockSums[blockIdx.x] = running;
}

__global__ void add_block_offsets_kernel(uint32_t* data, uint32_t n, const uint32_t* offsets)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) data[i] += offsets[i / kScanBlock];
}

// exclusive scan of n values in place; scratch holds the block sums of every level
static cudaError_t exclusive_scan(uint32_t* data, uint32_t n, cudaStream_t s, std::vector<uint32_t*>& scratch)
{
    if (n == 0) return cudaSuccess;
    const uint32_t blocks = (n + kScanBlock - 1) / kScanBlock;
    uint32_t* sums = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&sums, (size_t)blocks * 4, s);
    if (e != cudaSuccess) return e;
    scratch.push_back(sums);
    scan_blocks_kernel<<<blocks, 256, 0, s>>>(data, n, sums);
    if (blocks > 1)
    {
        e = exclusive_scan(sums, blocks, s, scratch);
        if (e != cudaSuccess) return e;
        add_block_offsets_kernel<<<(n + 255) / 256, 256, 0, s>>>(data, n, sums);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------- stable LSD radix sort

static constexpr uint32_t kSortThreads = 256;
static constexpr uint32_t kSortRounds = 16;
static constexpr uint32_t kSortTile = kSortThreads * kSortRounds;   // 4096 items per block

// digit histogram of each block's tile, digit-major: hist[d * blocks + b]
__global__ void sort_histogram_kernel(const uint64_t* key, uint32_t n, uint32_t shift, uint32_t* hist)
{
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * kSortTile;
    for (uint32_t r = 0; r < kSortRounds; r++)
    {
        const uint32_t i = base + r * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(key[i] >> shift) & 255], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// scatters each block's tile to its digits' places, keeping the input order within a digit:
// items are taken 256 at a time in order, and an item's place among its round's items of
// the same digit is the number of them before it (match within the warp, then the earlier
// warps' counts)
__global__ void sort_scatter_kernel(const uint64_t* key, const uint32_t* val, uint32_t n, uint32_t shift, const uint32_t* offsets,
    uint64_t* keyOut, uint32_t* valOut)
{
    __shared__ uint32_t running[256];
    __shared__ uint32_t warpCount[kSortThreads / 32][256];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    running[threadIdx.x] = offsets[threadIdx.x * gridDim.x + blockIdx.x];
    const uint32_t base = blockIdx.x * kSortTile;
    for (uint32_t r = 0; r < kSortRounds; r++)
    {
        for (uint32_t q = 0; q < kSortThreads / 32; q++) warpCount[q][threadIdx.x] = 0;
        __syncthreads();
        const uint32_t i = base + r * kSortThreads + threadIdx.x;
        const bool live = i < n;
        const uint64_t kk = live ? key[i] : 0;
        const uint32_t d = live ? (uint32_t)((kk >> shift) & 255) : 256 + lane;   // dead items match nothing live
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t rankInWarp = __popc(peers & ((1u << lane) - 1));
        if (live && rankInWarp == 0) warpCount[warp][d] = __popc(peers);
        __syncthreads();
        if (live)
        {
            uint32_t before = 0;
            for (uint32_t q = 0; q < warp; q++) before += warpCount[q][d];
            const uint32_t to = running[d] + before + rankInWarp;
            keyOut[to] = kk;
            valOut[to] = val[i];
        }
        __syncthreads();
        uint32_t total = 0;
        for (uint32_t q = 0; q < kSortThreads / 32; q++) total += warpCount[q][threadIdx.x];
        running[threadIdx.x] += total;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- groups, table

__global__ void new_kmer_flags_kernel(const uint64_t* kmers, uint32_t n, uint32_t* flags)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flags[i] = (i == 0 || kmers[i] != kmers[i - 1]) ? 1u : 0u;
}

// rank = exclusive scan of the flags: distinct k-mer r starts at the i whose flag is set
__global__ void group_starts_kernel(const uint64_t* kmers, const uint32_t* rank, uint32_t n, uint64_t* keys, uint64_t* startPos)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0 || kmers[i] != kmers[i - 1])
    {
        keys[rank[i]] = kmers[i];
        startPos[rank[i]] = i;
    }
}

// occurrence j of a group [from, to) goes to from + (to - 1 - j): reverse insertion order
__global__ void reverse_groups_kernel(const uint64_t* kmers, const uint32_t* rank, const uint32_t* order, const uint64_t* positions,
    const uint64_t* startPos, uint32_t n, uint64_t* out)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t r = rank[j] - ((j == 0 || kmers[j] != kmers[j - 1]) ? 0u : 1u);
    const uint64_t from = startPos[r], to = startPos[r + 1];
    out[from + (to - 1 - j)] = positions[order[j]];
}

// histogram of the occurrence counts of every k-mer id but the last (counts at or above
// `cap` go to the last bin).  Nearly all counts are 1 or 2, so the small ones are gathered in
// shared memory first: one atomic for each k-mer on those two bins took 1.4 ms of a 4.3 ms build.
static constexpr uint32_t kHistShared = 64, kHistThreads = 256;

__global__ void __launch_bounds__(kHistThreads) count_histogram_kernel(const uint64_t* startPos, uint32_t numCounts, uint32_t cap, uint32_t* hist)
{
    __shared__ uint32_t low[kHistShared];
    if (threadIdx.x < kHistShared) low[threadIdx.x] = 0;
    __syncthreads();
    uint32_t ones = 0;
    for (uint32_t r = blockIdx.x * kHistThreads + threadIdx.x; r < numCounts; r += gridDim.x * kHistThreads)
    {
        const uint64_t c = startPos[r + 1] - startPos[r];
        if (c == 1) ones++;
        else if (c < kHistShared && c < cap) atomicAdd(&low[c], 1u);
        else atomicAdd(&hist[c < cap ? c : cap], 1u);
    }
    ones = __reduce_add_sync(0xffffffffu, ones);
    if ((threadIdx.x & 31) == 0 && ones) atomicAdd(&low[1], ones);
    __syncthreads();
    if (threadIdx.x < kHistShared && low[threadIdx.x]) atomicAdd(&hist[threadIdx.x < cap ? threadIdx.x : cap], low[threadIdx.x]);
}

__global__ void fill_table_kernel(const uint64_t* keys, const uint64_t* startPos, uint32_t numKeys, SeedSlot* slots, uint64_t capacity)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= numKeys) return;
    const uint64_t key = keys[r];
    uint64_t h = seed_slot_hash(key) & (capacity - 1);
    // every slot a key's probe passes was claimed before it looks, so lookups find it
    // whatever order the claims come in
    for (uint64_t probe = 0; probe < capacity; probe++)
    {
        const unsigned long long prev = atomicCAS((unsigned long long*)&slots[h].key, (unsigned long long)kEmptyKmer, (unsigned long long)key);
        if (prev == kEmptyKmer)
        {
            slots[h].start = (uint32_t)startPos[r];
            slots[h].count = (uint32_t)(startPos[r + 1] - startPos[r]);
            return;
        }
        h = (h + 1) & (capacity - 1);
    }
}

}

namespace
{
template <typename T>
cudaError_t up(const std::vector<T>& v, T** out, cudaStream_t s, std::vector<void*>& keep)
{
    *out = nullptr;
    cudaError_t e = cudaMallocAsync((void**)out, std::max<size_t>(v.size(), 1) * sizeof(T), s);
    if (e != cudaSuccess) return e;
    keep.push_back(*out);
    return v.empty() ? cudaSuccess : cudaMemcpyAsync(*out, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}
}

int ga_build_index_gpu(const gahost::HostGraph& hg, size_t k, size_t w, double keepLeastFrequentFraction, gahost::MinimizerIndex& idx,
    gadev::SeedSlot** slotsOut, uint64_t* capacityOut, std::string& error)
{
    using namespace gadev;
    idx.k = k;
    idx.w = w;
    idx.maxCount = 0;
    *slotsOut = nullptr;
    *capacityOut = 0;
    if (w < k || w - k + 1 > kMaxRealWindow || k == 0 || k > 31)
    {
        error = "minimizer length 1..31 and a window of at most 64 minimizer positions";
        return -1;
    }
    if (hg.bpSize >= ((size_t)1 << 31))
    {
        error = "graphs of 2^31 bp or more are not indexed on the GPU";
        return -1;
    }
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
    {
        error = "index build: stream";
        return -2;
    }
    std::vector<void*> keep;           // device buffers freed at the end
    std::vector<uint32_t*> scanScratch;
    auto release = [&]()
    {
        for (void* p : keep) cudaFreeAsync(p, s);
        for (uint32_t* p : scanScratch) cudaFreeAsync(p, s);
        keep.clear();
        scanScratch.clear();
        cudaStreamSynchronize(s);
        cudaStreamDestroy(s);
    };
    auto fail = [&](const char* what, cudaError_t e) -> int
    {
        error = std::string("index build: ") + what + (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : std::string());
        release();
        cudaGetLastError();      // reported here: the next launch's check must not find it again
        return e != cudaSuccess ? -2 : -1;
    };
#define IDX_CUDA(call, what) do { cudaError_t _e = (call); if (_e != cudaSuccess) return fail(what, _e); } while (0)
    IndexGraph g {};
    g.N = hg.N;
    g.firstAmbiguous = hg.firstAmbiguous;
    g.numLookup = (uint32_t)hg.lookupIds.size();
    uint32_t *len, *inOff, *inNb, *nodeOffset, *lookupOff, *lookupNodes, *originalSize;
    uint64_t *seq2, *seqAmb;
    int32_t* nodeIds;
    IDX_CUDA(up(hg.len, &len, s, keep), "graph upload");
    IDX_CUDA(up(hg.seq2, &seq2, s, keep), "graph upload");
    IDX_CUDA(up(hg.seqAmb, &seqAmb, s, keep), "graph upload");
    IDX_CUDA(up(hg.inOff, &inOff, s, keep), "graph upload");
    IDX_CUDA(up(hg.inNb, &inNb, s, keep), "graph upload");
    IDX_CUDA(up(hg.nodeIds, &nodeIds, s, keep), "graph upload");
    IDX_CUDA(up(hg.nodeOffset, &nodeOffset, s, keep), "graph upload");
    IDX_CUDA(up(hg.lookupOff, &lookupOff, s, keep), "graph upload");
    IDX_CUDA(up(hg.lookupNodes, &lookupNodes, s, keep), "graph upload");
    IDX_CUDA(up(hg.originalSize, &originalSize, s, keep), "graph upload");
    g.len = len; g.seq2 = seq2; g.seqAmb = seqAmb; g.inOff = inOff; g.inNb = inNb; g.nodeIds = nodeIds;
    g.nodeOffset = nodeOffset; g.lookupOff = lookupOff; g.lookupNodes = lookupNodes; g.originalSize = originalSize;

    // 1. minimizers per bigraph node: count, scan, write
    const uint32_t numLookup = g.numLookup;
    uint32_t *first = nullptr, *errorFlag = nullptr;
    IDX_CUDA(cudaMallocAsync((void**)&first, ((size_t)numLookup + 1) * 4, s), "counts");
    keep.push_back(first);
    IDX_CUDA(cudaMallocAsync((void**)&errorFlag, 4, s), "flag");
    keep.push_back(errorFlag);
    IDX_CUDA(cudaMemsetAsync(errorFlag, 0, 4, s), "flag");
    IDX_CUDA(cudaMemsetAsync(first + numLookup, 0, 4, s), "counts");
    // the long nodes' chunks
    uint32_t *firstChunk, *minStart, *chunkNode = nullptr, *chunkCount = nullptr;
    IDX_CUDA(cudaMallocAsync((void**)&firstChunk, ((size_t)numLookup + 1) * 4, s), "chunks"); keep.push_back(firstChunk);
    IDX_CUDA(cudaMallocAsync((void**)&minStart, std::max<size_t>(numLookup, 1) * 4, s), "chunks"); keep.push_back(minStart);
    IDX_CUDA(cudaMemsetAsync(firstChunk + numLookup, 0, 4, s), "chunks");
    IDX_CUDA(cudaMemsetAsync(first, 0, (size_t)numLookup * 4, s), "counts");
    IDX_CUDA(cudaMemsetAsync(minStart, 0, (size_t)numLookup * 4, s), "chunks");
    const uint32_t nodeBlocks = (numLookup + 127) / 128;
    if (numLookup) count_chunks_kernel<<<nodeBlocks, 128, 0, s>>>(g, firstChunk);
    IDX_CUDA(cudaGetLastError(), "chunks");
    IDX_CUDA(exclusive_scan(firstChunk, numLookup + 1, s, scanScratch), "chunk scan");
    uint32_t chunks = 0;
    IDX_CUDA(cudaMemcpyAsync(&chunks, firstChunk + numLookup, 4, cudaMemcpyDeviceToHost, s), "chunks");
    if (numLookup) count_minimizers_kernel<<<nodeBlocks, 128, 0, s>>>(g, (uint32_t)k, (uint32_t)w, first, errorFlag);
    IDX_CUDA(cudaGetLastError(), "minimizer count");
    IDX_CUDA(cudaStreamSynchronize(s), "chunks");
    if (chunks)
    {
        IDX_CUDA(cudaMallocAsync((void**)&chunkNode, (size_t)chunks * 4, s), "chunks"); keep.push_back(chunkNode);
        IDX_CUDA(cudaMallocAsync((void**)&chunkCount, (size_t)chunks * 4, s), "chunks"); keep.push_back(chunkCount);
        chunk_nodes_kernel<<<nodeBlocks, 128, 0, s>>>(g, firstChunk, chunkNode);
        long_nodes_kernel<<<chunks, 128, 0, s>>>(g, firstChunk, chunkNode, minStart, errorFlag);
        long_minimizers_kernel<<<chunks, kChunk, 0, s>>>(g, (uint32_t)k, (uint32_t)w, firstChunk, chunkNode, minStart, errorFlag, chunkCount, first, nullptr,
            nullptr, nullptr, nullptr);
        IDX_CUDA(cudaGetLastError(), "minimizer count");
        IDX_CUDA(exclusive_scan(chunkCount, chunks, s, scanScratch), "chunk scan");
    }
    // counts in [0, numLookup), 0 at numLookup: the exclusive scan leaves the total there
    IDX_CUDA(exclusive_scan(first, numLookup + 1, s, scanScratch), "scan");
    uint32_t total = 0, bad = 0;
    IDX_CUDA(cudaMemcpyAsync(&total, first + numLookup, 4, cudaMemcpyDeviceToHost, s), "total");
    IDX_CUDA(cudaMemcpyAsync(&bad, errorFlag, 4, cudaMemcpyDeviceToHost, s), "flag");
    IDX_CUDA(cudaStreamSynchronize(s), "minimizer count");
    if (bad) return fail("the pieces of a bigraph node do not tile it in order", cudaSuccess);
    const uint32_t n = total;
    uint64_t *kmers, *positions, *kmers2;
    uint32_t *order, *order2;
    const size_t cells = std::max<size_t>(n, 1);
    IDX_CUDA(cudaMallocAsync((void**)&kmers, cells * 8, s), "occurrences"); keep.push_back(kmers);
    IDX_CUDA(cudaMallocAsync((void**)&positions, cells * 8, s), "occurrences"); keep.push_back(positions);
    IDX_CUDA(cudaMallocAsync((void**)&kmers2, cells * 8, s), "occurrences"); keep.push_back(kmers2);
    IDX_CUDA(cudaMallocAsync((void**)&order, cells * 4, s), "occurrences"); keep.push_back(order);
    IDX_CUDA(cudaMallocAsync((void**)&order2, cells * 4, s), "occurrences"); keep.push_back(order2);
    if (numLookup) write_minimizers_kernel<<<(numLookup + 127) / 128, 128, 0, s>>>(g, (uint32_t)k, (uint32_t)w, first, kmers, positions, order, errorFlag);
    if (chunks)
        long_minimizers_kernel<<<chunks, kChunk, 0, s>>>(g, (uint32_t)k, (uint32_t)w, firstChunk, chunkNode, minStart, errorFlag, chunkCount, nullptr, first,
            kmers, positions, order);
    IDX_CUDA(cudaGetLastError(), "minimizer write");

    // 2. stable LSD radix sort of (k-mer, occurrence) by the k-mer's 2k bits
    const uint32_t sortBlocks = std::max<uint32_t>(1, (n + kSortTile - 1) / kSortTile);
    uint32_t* hist;
    IDX_CUDA(cudaMallocAsync((void**)&hist, (size_t)sortBlocks * 256 * 4, s), "sort"); keep.push_back(hist);
    for (uint32_t shift = 0; shift < 2 * k && n > 0; shift += 8)
    {
        sort_histogram_kernel<<<sortBlocks, kSortThreads, 0, s>>>(kmers, n, shift, hist);
        IDX_CUDA(cudaGetLastError(), "sort histogram");
        IDX_CUDA(exclusive_scan(hist, sortBlocks * 256, s, scanScratch), "sort scan");
        sort_scatter_kernel<<<sortBlocks, kSortThreads, 0, s>>>(kmers, order, n, shift, hist, kmers2, order2);
        IDX_CUDA(cudaGetLastError(), "sort scatter");
        std::swap(kmers, kmers2);
        std::swap(order, order2);
    }

    // 3. distinct k-mers, their first occurrences, occurrences in reverse insertion order
    uint32_t* rank;
    IDX_CUDA(cudaMallocAsync((void**)&rank, (cells + 1) * 4, s), "groups"); keep.push_back(rank);
    IDX_CUDA(cudaMemsetAsync(rank + n, 0, 4, s), "groups");
    if (n) new_kmer_flags_kernel<<<(n + 255) / 256, 256, 0, s>>>(kmers, n, rank);
    IDX_CUDA(exclusive_scan(rank, n + 1, s, scanScratch), "group scan");
    uint32_t numKeys = 0;
    IDX_CUDA(cudaMemcpyAsync(&numKeys, rank + n, 4, cudaMemcpyDeviceToHost, s), "groups");
    IDX_CUDA(cudaStreamSynchronize(s), "groups");
    uint64_t *keys, *startPos, *posOut;
    IDX_CUDA(cudaMallocAsync((void**)&keys, std::max<size_t>(numKeys, 1) * 8, s), "groups"); keep.push_back(keys);
    IDX_CUDA(cudaMallocAsync((void**)&startPos, ((size_t)numKeys + 1) * 8, s), "groups"); keep.push_back(startPos);
    IDX_CUDA(cudaMallocAsync((void**)&posOut, cells * 8, s), "groups"); keep.push_back(posOut);
    const uint64_t total64 = n;
    IDX_CUDA(cudaMemcpyAsync(startPos + numKeys, &total64, 8, cudaMemcpyHostToDevice, s), "groups");
    if (n)
    {
        group_starts_kernel<<<(n + 255) / 256, 256, 0, s>>>(kmers, rank, n, keys, startPos);
        reverse_groups_kernel<<<(n + 255) / 256, 256, 0, s>>>(kmers, rank, order, positions, startPos, n, posOut);
    }
    IDX_CUDA(cudaGetLastError(), "groups");

    // 4. initMaxCount: the count at the keep fraction of the sorted counts of every id but the
    // last, plus one (MinimizerSeeder.cpp:557-575)
    const uint32_t kCap = 1u << 16;
    uint32_t* countHist;
    IDX_CUDA(cudaMallocAsync((void**)&countHist, ((size_t)kCap + 1) * 4, s), "max count"); keep.push_back(countHist);
    IDX_CUDA(cudaMemsetAsync(countHist, 0, ((size_t)kCap + 1) * 4, s), "max count");
    const uint32_t numCounts = numKeys >= 2 ? numKeys - 1 : 0;
    if (numCounts) count_histogram_kernel<<<std::min<uint32_t>((numCounts + kHistThreads - 1) / kHistThreads, 608), kHistThreads, 0, s>>>(startPos, numCounts, kCap, countHist);
    IDX_CUDA(cudaGetLastError(), "max count");

    // host copies: the selection step reads positions; keys and start positions are kept with them
    idx.keys.resize(numKeys);
    idx.startPos.resize((size_t)numKeys + 1);
    idx.positions.resize(n);
    std::vector<uint32_t> countHistHost(kCap + 1);
    if (numKeys) IDX_CUDA(cudaMemcpyAsync(idx.keys.data(), keys, (size_t)numKeys * 8, cudaMemcpyDeviceToHost, s), "copy back");
    IDX_CUDA(cudaMemcpyAsync(idx.startPos.data(), startPos, ((size_t)numKeys + 1) * 8, cudaMemcpyDeviceToHost, s), "copy back");
    if (n) IDX_CUDA(cudaMemcpyAsync(idx.positions.data(), posOut, (size_t)n * 8, cudaMemcpyDeviceToHost, s), "copy back");
    IDX_CUDA(cudaMemcpyAsync(countHistHost.data(), countHist, ((size_t)kCap + 1) * 4, cudaMemcpyDeviceToHost, s), "copy back");

    // 5. the lookup table, on the device
    uint64_t capacity = 16;
    while (capacity < 2 * (uint64_t)numKeys) capacity <<= 1;
    SeedSlot* slots = nullptr;
    IDX_CUDA(cudaMalloc((void**)&slots, capacity * sizeof(SeedSlot)), "table");
    cudaError_t e = cudaMemsetAsync(slots, 0xff, capacity * sizeof(SeedSlot), s);   // every key kEmptyKmer
    if (e == cudaSuccess && numKeys) fill_table_kernel<<<(numKeys + 255) / 256, 256, 0, s>>>(keys, startPos, numKeys, slots, capacity);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
    {
        cudaFree(slots);
        return fail("table", e);
    }
    if (numCounts)
    {
        size_t index = (size_t)(numCounts * keepLeastFrequentFraction);
        if (index == numCounts) index = numCounts - 1;
        size_t seen = 0;
        bool done = false;
        for (uint32_t c = 0; c < kCap && !done; c++)
        {
            seen += countHistHost[c];
            if (seen > index)
            {
                idx.maxCount = c + 1;
                done = true;
            }
        }
        if (!done)
        {
            // the quantile lies among counts of 2^16 or more: sort those counts on the host
            std::vector<uint64_t> big;
            for (uint32_t r = 0; r < numCounts; r++)
                if (idx.startPos[r + 1] - idx.startPos[r] >= kCap) big.push_back(idx.startPos[r + 1] - idx.startPos[r]);
            std::sort(big.begin(), big.end());
            idx.maxCount = big[index - seen] + 1;
        }
    }
    release();
    *slotsOut = slots;
    *capacityOut = capacity;
    return 0;
#undef IDX_CUDA
}
