// Minimizer index lookup on the GPU (MinimizerSeeder::getSeeds, MinimizerSeeder.cpp:521-537).
//
// A block walks one read, each warp a segment, 32 positions per step (lane j: position base + j):
//   - the bases come in as one coalesced 32-byte load;
//   - the k-mer ending at each position is built by a shuffle-doubling pack of the
//     2-bit codes (five steps) on top of the previous step's last k-mer;
//   - a position holds a k-mer when the last non-ACGT character lies at least k
//     positions back (a ballot finds the last one at or before each lane);
//   - iterateKmers (MinimizerSeeder.cpp:59-102) looks a k-mer up when it is the first
//     after a restart, differs from the last one looked up, or that one is at least
//     w-k+1 positions back (unsigned, so every position below w-k+1 qualifies).  The last
//     one looked up always holds the previous position's k-mer, so a k-mer that differs
//     from its predecessor is looked up; only in a step that holds a repeat of its
//     predecessor (a homopolymer longer than k) are the positions resolved in order;
//   - the lookups probe the index hash table resident in HBM independently, and the
//     matches with count < maxCount are compacted by ballot and prefix popcount and
//     written in read order, the order the host's selection (a std::sort by count,
//     MinimizerSeeder.cpp:493-519) needs.
#include <cuda_runtime.h>
#include <stdint.h>
#include "seed_kernel.cuh"

namespace gadev
{

static constexpr unsigned kAllLanes = 0xffffffffu;

__device__ __forceinline__ int base_code(uint8_t c)
{
    switch (c)
    {
        case 'a': case 'A': return 0;
        case 'c': case 'C': return 1;
        case 'g': case 'G': return 2;
        case 't': case 'T': return 3;
    }
    return -1;
}

// A block per read, kWarps segments of 32 kSteps positions at a time.  A warp knows what it needs of
// the positions before its segment from the 32 bases there (and, inside a homopolymer longer than a
// k-mer, from where that began); the segments' matches are placed by a sum over the warps.  The
// probes of a segment's steps go on together.  About 310 instructions a step of 32 positions, one
// step after the other by a single warp, took 0.49 ms for a 10 kbp read (the lookups of one, copies
// included, 0.46 -> 0.11 ms; of 200 reads 1.06 -> 0.40 ms; of 100 reads of 20 kbp 1.26 -> 0.42 ms).
constexpr int kSteps = 4, kWarps = 8;

// Where the run of base code c that ends before `at` began.  It is looked for back to `round`, the start of
// the segments that are walked together (32 divides at - round); a run that is older than that began
// at `carried`, which the round before left.  So a read takes time linear in its length: with every
// segment of a homopolymer walking back to its beginning, the lookups of a run of 131 kbp took 32 ms
// and twice the length four times as long; now 2.1 ms, and 16 ms for 1 Mbp.
__device__ __noinline__ int64_t run_start(const uint8_t* s, int64_t at, int c, int64_t round, int64_t carried, uint32_t lane)
{
#pragma unroll 1
    for (int64_t end = at; end > round; end -= 32)
    {
        const uint32_t other = __ballot_sync(kAllLanes, base_code(s[end - 1 - lane]) != c);
        if (other) return end - (__ffs((int)other) - 1);
    }
    return round > 0 && base_code(s[round - 1]) == c ? carried : round;
}

// The last position before `at` that was looked up, when the k-mer ending at `at` repeats the one
// before it: a run of one base that began at `first`, so that its first k-mer was looked up, then
// every realWindow-th (and every one below realWindow).
__device__ __forceinline__ int64_t lookup_before(int64_t at, int64_t first, int64_t k, int64_t realWindow)
{
    int64_t last = first + k - 1;
    if (last < realWindow - 1) last = at - 1 < realWindow - 1 ? at - 1 : realWindow - 1;
    return last + (at - 1 - last) / realWindow * realWindow;
}

__global__ void __launch_bounds__(32 * kWarps) seed_lookup_kernel(SeedTable t, uint32_t k, uint32_t w, uint32_t numReads,
    const uint8_t* seq, const uint64_t* seqOff, const uint32_t* seqLen, const uint64_t* outOff, SeedMatch* out, uint32_t* outCount)
{
    __shared__ uint32_t found[2][kWarps];
    __shared__ int64_t runBefore[2];        // where the run of one base that ends before the round began
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t r = blockIdx.x;
    const uint8_t* s = seq + seqOff[r];
    const int64_t len = seqLen[r];
    SeedMatch* o = out + outOff[r];
    const uint64_t mask = ~(0xFFFFFFFFFFFFFFFFULL << (k * 2));
    const int64_t realWindow = (int64_t)w - (int64_t)k + 1;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t n = 0;
    uint32_t turn = 0;
    // codes up to this lane's packed, 2 bits each
    auto pack = [&](int c) -> uint64_t
    {
        uint64_t packed = c < 0 ? 0 : (uint64_t)c;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1)
        {
            const uint64_t t2 = __shfl_up_sync(kAllLanes, packed, d);
            if (lane >= d) packed = (t2 << (2 * d)) | packed;
        }
        return packed;
    };
#pragma unroll 1
    for (int64_t round = 0; round < len; round += 32 * kSteps * kWarps, turn ^= 1)
    {
        const int64_t from = round + 32 * kSteps * (int64_t)warp;
        uint32_t hits[kSteps];
        SeedSlot slot[kSteps];
        uint32_t own = 0;
#pragma unroll
        for (int q = 0; q < kSteps; q++) hits[q] = 0;
        if (from < len)
        {
            int code[kSteps];
#pragma unroll
            for (int q = 0; q < kSteps; q++)
            {
                const int64_t p = from + 32 * q + lane;
                code[q] = p < len ? base_code(s[p]) : -1;
            }
            uint64_t prevKmer = 0;          // k-mer (2-bit packing) of the position before this step
            int64_t lastInvalid = -1;       // last non-ACGT position before this step (-1: the read start)
            int64_t lastPos = 0;            // position of the last k-mer looked up
            if (from > 0)
            {
                const int c = base_code(s[from - 32 + lane]);
                const uint32_t inv = __ballot_sync(kAllLanes, c < 0);
                prevKmer = __shfl_sync(kAllLanes, pack(c), 31) & mask;
                // no position further back matters to a k-mer of at most 31
                lastInvalid = inv ? from - 1 - __clz((int)inv) : from - 64;
            }
            uint64_t kmers[kSteps], slotAt[kSteps];
            bool open[kSteps], hit[kSteps];
#pragma unroll
            for (int q = 0; q < kSteps; q++)
            {
                const int64_t base = from + 32 * q;
                const int64_t p = base + lane;
                const int c = code[q];
                // last non-ACGT position at or before p (positions past the end count as non-ACGT)
                const uint32_t inv = __ballot_sync(kAllLanes, c < 0);
                const uint32_t invUpTo = inv & (below | (1u << lane));
                const int64_t li = invUpTo ? base + (31 - __clz((int)invUpTo)) : lastInvalid;
                // codes base..p packed, then the k-mer ending at p
                const uint64_t kmer = ((lane < 31 ? prevKmer << (2 * (lane + 1)) : 0) | pack(c)) & mask;
                const bool valid = p < len && p - li >= (int64_t)k;
                const bool first = valid && p - li == (int64_t)k;
                uint64_t kPrev = __shfl_up_sync(kAllLanes, kmer, 1);
                if (lane == 0) kPrev = prevKmer;
                const bool repeat = valid && !first && kmer == kPrev;
                uint32_t look = __ballot_sync(kAllLanes, valid && !repeat);
                const uint32_t repeats = __ballot_sync(kAllLanes, repeat);
                if (repeats)
                {
                    // positions in order: a repeat is looked up when the last lookup lies w-k+1 back
                    // (or the position is below w-k+1)
                    if (q == 0 && (repeats & 1) && from > 0)
                        lastPos = lookup_before(from, run_start(s, from, __shfl_sync(kAllLanes, c, 0), round, round ? runBefore[turn] : 0, lane), k, realWindow);
                    look = 0;
                    const uint32_t validMask = __ballot_sync(kAllLanes, valid);
#pragma unroll 1
                    for (uint32_t j = 0; j < 32; j++)
                    {
                        if (!((validMask >> j) & 1)) continue;
                        const int64_t pj = base + j;
                        if (!((repeats >> j) & 1) || pj < realWindow || pj - lastPos >= realWindow)
                        {
                            look |= 1u << j;
                            lastPos = pj;
                        }
                    }
                }
                else if (look)
                {
                    lastPos = base + (31 - __clz((int)look));
                }
                kmers[q] = kmer;
                open[q] = (look >> lane) & 1;
                hit[q] = false;
                slotAt[q] = seed_slot_hash(kmer) & (t.capacity - 1);
                if (open[q]) slot[q] = t.slots[slotAt[q]];
                prevKmer = __shfl_sync(kAllLanes, kmer, 31);
                lastInvalid = __shfl_sync(kAllLanes, li, 31);
            }
#pragma unroll 1
            for (uint64_t probes = 0; probes < t.capacity; probes++)
            {
                bool any = false;
#pragma unroll
                for (int q = 0; q < kSteps; q++)
                {
                    if (!open[q]) continue;
                    hit[q] = slot[q].key == kmers[q];
                    open[q] = !hit[q] && slot[q].key != kEmptyKmer;
                    if (!open[q]) continue;
                    any = true;
                    slotAt[q] = (slotAt[q] + 1) & (t.capacity - 1);
                    slot[q] = t.slots[slotAt[q]];
                }
                if (!__any_sync(kAllLanes, any)) break;
            }
#pragma unroll
            for (int q = 0; q < kSteps; q++)
            {
                hits[q] = __ballot_sync(kAllLanes, hit[q] && slot[q].count < t.maxCount);
                own += __popc(hits[q]);
            }
        }
        const int64_t next = round + 32 * kSteps * kWarps;
        if (warp == kWarps - 1 && next < len)
        {
            const int64_t began = run_start(s, next, base_code(s[next - 1]), round, round ? runBefore[turn] : 0, lane);
            if (lane == 0) runBefore[turn ^ 1] = began;
        }
        // the segments' matches one behind the other (two rows: a warp may be a round ahead)
        if (lane == 0) found[turn][warp] = own;
        __syncthreads();
        uint32_t to = n;
#pragma unroll
        for (uint32_t q = 0; q < kWarps; q++)
        {
            if (q < warp) to += found[turn][q];
            n += found[turn][q];
        }
#pragma unroll
        for (int q = 0; q < kSteps; q++)
        {
            if ((hits[q] >> lane) & 1)
                o[to + __popc(hits[q] & below)] = SeedMatch { (uint64_t)(from + 32 * q + lane), slot[q].start, slot[q].count };
            to += __popc(hits[q]);
        }
    }
    if (threadIdx.x == 0) outCount[r] = n;
}

}

void ga_launch_seed_lookup(const gadev::SeedTable& t, uint32_t k, uint32_t w, uint32_t numReads, const uint8_t* seq,
    const uint64_t* seqOff, const uint32_t* seqLen, const uint64_t* outOff, gadev::SeedMatch* out, uint32_t* outCount, void* stream)
{
    if (numReads == 0) return;
    gadev::seed_lookup_kernel<<<numReads, 32 * gadev::kWarps, 0, (cudaStream_t)stream>>>(t, k, w, numReads, seq, seqOff, seqLen, outOff, out, outCount);
}
