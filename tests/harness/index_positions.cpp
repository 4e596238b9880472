// Checks minimizers_at (a long node's minimizers base by base) against node_minimizers (the walk)
// on random nodes: low-complexity sequences full of equal hashes, non-ACGT bases, k from 3 to 31
// and windows of 1 to 64 k-mers.
#include <cstdio>
#include <random>
#include <string>
#include <vector>
#include "../../graphaligner_gb300/csrc/index_walk.cuh"
using namespace gadev;

int main()
{
    std::mt19937_64 rng(99);
    for (int round = 0; round < 4000; round++)
    {
        const uint32_t k = 3 + (uint32_t)(rng() % 29), w = k + (uint32_t)(rng() % (round % 3 ? 12 : 64));
        const uint32_t size = 1 + (uint32_t)(rng() % 700);
        // codes: a short unit repeated, random bases or a mix; now and then a non-ACGT base
        std::vector<int> code(size);
        const uint32_t unit = 1 + (uint32_t)(rng() % 7);
        for (uint32_t p = 0; p < size; p++)
            code[p] = (p >= unit && rng() % 16 < (uint64_t)(round % 17)) ? code[p - unit] : (int)(rng() % (round % 2 ? 2 : 4));
        for (uint32_t q = 0; q < (uint32_t)(rng() % 4); q++) code[rng() % size] = -1;
        // pieces of up to 64 bases, all stored as masks
        const uint32_t pieces = (size + 63) / 64;
        std::vector<uint32_t> len(pieces), inOff(pieces + 1, 0), inNb(1, 0), nodeOffset(pieces), lookupNodes(pieces);
        std::vector<int32_t> ids(pieces, 2);
        std::vector<uint64_t> amb(pieces * 4, 0), seq2(2, 0);
        for (uint32_t i = 0; i < pieces; i++)
        {
            len[i] = size - i * 64 < 64 ? size - i * 64 : 64;
            nodeOffset[i] = i * 64;
            lookupNodes[i] = i;
            for (uint32_t p = 0; p < len[i]; p++)
                for (int c = 0; c < 4; c++)
                    if (code[i * 64 + p] == c || code[i * 64 + p] < 0) amb[i * 4 + c] |= 1ULL << p;
        }
        const uint32_t lookupOff[2] = { 0, pieces }, originalSize[1] = { size };
        IndexGraph g { pieces, 0, len.data(), seq2.data(), amb.data(), inOff.data(), inNb.data(), ids.data(), nodeOffset.data(), lookupOff,
            lookupNodes.data(), originalSize, 1 };
        std::vector<uint64_t> kmers(size * 2 + 2), positions(size * 2 + 2);
        bool bad = false;
        const uint32_t n = node_minimizers(g, 0, k, w, kmers.data(), positions.data(), bad);
        if (bad) { printf("bad node\n"); return 1; }
        std::vector<uint64_t> kmer(size, 0), hash(size, 0), gotKmer, gotPos;
        for (uint32_t p = 0; p < size; p++)
        {
            for (uint32_t i = p + 1 < k ? 0 : p + 1 - k; i <= p; i++) kmer[p] = (kmer[p] << 2) | (uint64_t)(code[i] & 3);
            hash[p] = kmer_hash(kmer[p]);
        }
        uint32_t run = 0;
        for (uint32_t p = 0; p < size; p++)
        {
            run = code[p] < 0 ? 0 : run + 1;
            minimizers_at(p, run < w + 3 ? run : w + 3, k, w, [&](uint32_t q) { return hash[q]; }, [&](uint32_t q)
            {
                gotKmer.push_back(kmer[q]);
                gotPos.push_back(((uint64_t)(q / 64) << 6) + q % 64);
            });
        }
        kmers.resize(n);
        positions.resize(n);
        if (kmers != gotKmer || positions != gotPos) { printf("round %d: k %u w %u size %u: %zu reports, not %u\n", round, k, w, size, gotPos.size(), n); return 1; }
    }
    printf("ok\n");
    return 0;
}
