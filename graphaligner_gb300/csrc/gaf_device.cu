// GAF lines and alignment selection on the GPU (GraphAlignerGAFAlignment::traceToAlignment,
// GraphAlignerGAFAlignment.h:37-200; AlignmentSelection::SelectAlignments,
// AlignmentSelection.cpp:31-95).
//
// The host's cores walk each selected alignment's trace once (gaf::classify_line: one edit-op
// byte per trace item, the node-path entries, the counts), between seed-loop rounds; the ops,
// entries and line records go down in chunks, one warp per line measures its line, the host
// places the lines, and one warp per line writes it (names, numbers, the doubles, the
// CIGAR's runs).  The node names,
// the bigraph-id lookup and the node sizes stay resident from the aligner's creation.
// Selection runs one thread per read over its alignments' spans and X-scores.
#include <cuda_runtime.h>
#include <chrono>
#include <cmath>
#include <cstring>
#include "aligner.h"
#include "extend.cuh"

namespace
{

constexpr unsigned kFull = 0xffffffffu;

// sum of v over the lanes below this one, and over all of them
__device__ __forceinline__ uint32_t lanes_before(uint32_t v, uint32_t lane, uint32_t& all)
{
    uint32_t sum = v;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1)
    {
        const uint32_t up = __shfl_up_sync(kFull, sum, d);
        if (lane >= d) sum += up;
    }
    all = __shfl_sync(kFull, sum, 31);
    return sum - v;
}

__device__ __forceinline__ uint32_t digits(uint32_t v)
{
    uint32_t n = 1;
    while (v >= 10)
    {
        v /= 10;
        n++;
    }
    return n;
}

// A line's numbers, each written by its own lane with the tabs and tags around it
constexpr uint32_t kFields = 13, kHeadFields = 3, kFieldBytes = 48;
struct LineFields
{
    char text[kFields][kFieldBytes];
};

__device__ int field_text(const gaf::LineMeta& m, uint32_t field, char* out)
{
    int n = 0;
    auto putS = [&](const char* p) { while (*p) out[n++] = *p++; };
    const double total = (double)(m.matches + m.edits);
    switch (field)
    {
        case 9: putS("\tNM:i:"); break;
        case 10: if (m.xscore100 == -100) return 0; putS("\tAS:f:"); break;
        case 11: putS("\tdv:f:"); break;
        case 12: putS("\tid:f:"); break;
        default: putS("\t");
    }
    if (field == 8) n += gaf::fmt_i64(m.mapq, out + n);
    else if (field < 10)
    {
        const uint64_t v = field == 0 ? m.readLen : field == 1 ? m.readStart : field == 2 ? m.readEnd : field == 3 ? m.nodePathLen
            : field == 4 ? m.nodePathStart : field == 5 ? m.nodePathEnd : field == 6 ? m.matches : field == 7 ? m.count : m.edits;
        n += gaf::fmt_u64(v, out + n);
    }
    else
    {
        const double v = field == 10 ? (double)m.xscore100 / 100.0 : field == 11 ? 1.0 - ((double)m.matches / total) : (double)m.matches / total;
        n += gaf::fmt_g(v, out + n);
    }
    if (field == 2) putS("\t+\t");
    if (field == 12) putS("\tcg:Z:");
    return n;
}

// gaf::write_line (no newline) by a warp: each number by its own lane, then 32 node-path entries
// and 32 edit ops at a time, each lane's text placed by a sum over the lanes before it.  Write =
// false: only the length.
//
// A thread a line walked its ops one byte after the other, about 15 cycles each: a 10 kbp read's
// line took 3.8 ms to measure and 5.7 ms to write, whatever the number of lines.
template <bool Write>
__device__ uint64_t warp_line(const gaf::Names& nm, const gaf::LineMeta& m, const uint8_t* ops, const int32_t* entries, char* out, LineFields& fields,
    uint32_t lane)
{
    uint32_t len = 0;
    if (lane < kFields) len = (uint32_t)field_text(m, lane, fields.text[lane]);
    __syncwarp();
    uint32_t all;
    const uint32_t before = lanes_before(len, lane, all);
    const uint32_t head = __shfl_sync(kFull, before, kHeadFields);
    const uint64_t nameFrom = nm.readNameOff[m.read];
    const uint64_t nameLen = nm.readNameOff[m.read + 1] - nameFrom;
    uint64_t n = nameLen;
    if (Write)
    {
        for (uint64_t k = lane; k < nameLen; k += 32) out[k] = (char)nm.readNames[nameFrom + k];
        if (lane < kHeadFields)
            for (uint32_t k = 0; k < len; k++) out[n + before + k] = fields.text[lane][k];
    }
    n += head;
    // the node path
    for (uint32_t base = 0; base < m.entries; base += 32)
    {
        uint32_t size = 0;
        int32_t bignode = 0;
        uint64_t from = 0;
        uint32_t nameSize = 0;
        char number[24];
        if (base + lane < m.entries)
        {
            bignode = entries[m.entry + base + lane];
            const uint32_t li = gaf::lookup_id(nm, bignode);
            from = nm.nodeNameOff[li];
            nameSize = (uint32_t)(nm.nodeNameOff[li + 1] - from);
            size = 1 + (nameSize ? nameSize : (uint32_t)gaf::fmt_i64(bignode / 2, number));
        }
        uint32_t sum;
        const uint32_t at = lanes_before(size, lane, sum);
        if (Write && size)
        {
            char* o = out + n + at;
            o[0] = (bignode % 2 == 1) ? '<' : '>';
            for (uint32_t k = 0; k + 1 < size; k++) o[1 + k] = nameSize ? (char)nm.nodeNames[from + k] : number[k];
        }
        n += sum;
    }
    if (Write && lane >= kHeadFields && lane < kFields)
        for (uint32_t k = 0; k < len; k++) out[n + (before - head) + k] = fields.text[lane][k];
    n += all - head;
    // the CIGAR: a run of one edit op ends before the lane whose op differs from the one before
    // it, and at the line's last item
    const uint8_t* o = ops + m.op;
    uint32_t start = 0;         // where the run that is open began
    uint32_t last = 0;          // the op before this step's first
    for (uint32_t base = 0; base <= m.count; base += 32)
    {
        const uint32_t pos = base + lane;
        const uint32_t op = pos < m.count ? o[pos] : 0xff;
        uint32_t prev = __shfl_up_sync(kFull, op, 1);
        if (lane == 0) prev = last;
        const bool ends = pos > 0 && pos <= m.count && (pos == m.count || op != prev);
        const uint32_t marks = __ballot_sync(kFull, ends);
        last = __shfl_sync(kFull, op, 31);
        if (!marks) continue;
        const uint32_t below = marks & ((1u << lane) - 1u);
        const uint32_t run = pos - (below ? base + 31 - (uint32_t)__clz((int)below) : start);
        uint32_t sum;
        const uint32_t size = ends ? digits(run) + 1 : 0;
        const uint32_t at = lanes_before(size, lane, sum);
        if (Write && ends)
        {
            char* to = out + n + at;
            uint32_t v = run;
            for (uint32_t k = size - 1; k > 0; k--)
            {
                to[k - 1] = (char)('0' + v % 10);
                v /= 10;
            }
            to[size - 1] = prev == gaf::OpMatch ? '=' : prev == gaf::OpMismatch ? 'X' : prev == gaf::OpMatchOrMismatch ? 'M' : prev == gaf::OpInsertion ? 'I' : 'D';
        }
        n += sum;
        start = base + 31 - (uint32_t)__clz((int)marks);
    }
    return n;
}

constexpr uint32_t kLineWarps = 4;

__global__ void __launch_bounds__(32 * kLineWarps) gaf_measure_kernel(gaf::Names nm, const gaf::LineMeta* lines, const uint8_t* ops,
    const int32_t* entries, uint32_t n, int64_t* len)
{
    __shared__ LineFields fields[kLineWarps];
    const uint32_t k = blockIdx.x * kLineWarps + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (k >= n) return;
    const gaf::LineMeta m = lines[k];
    const uint64_t v = warp_line<false>(nm, m, ops, entries, nullptr, fields[threadIdx.x / 32], lane);
    if (lane == 0) len[k] = (int64_t)v;
}

__global__ void __launch_bounds__(32 * kLineWarps) gaf_write_kernel(gaf::Names nm, const gaf::LineMeta* lines, const uint8_t* ops,
    const int32_t* entries, uint32_t n, const uint64_t* start, char* text)
{
    __shared__ LineFields fields[kLineWarps];
    const uint32_t k = blockIdx.x * kLineWarps + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (k >= n) return;
    const gaf::LineMeta m = lines[k];
    char* out = text + start[k];
    const uint64_t len = warp_line<true>(nm, m, ops, entries, out, fields[threadIdx.x / 32], lane);
    if (lane == 0) out[len] = '\n';
}

__global__ void select_kernel(const uint64_t* first, const uint64_t* start, const uint64_t* end, const double* score, uint32_t n,
    int minAlignmentScore, double fraction, char* keep)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const uint64_t a = first[r];
    gaf::select_read((uint32_t)(first[r + 1] - a), start + a, end + a, score + a, minAlignmentScore, fraction, keep + a);
}

double ms_since(std::chrono::steady_clock::time_point t)
{
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count();
}

gaf::Names device_names(const GafDevice& d)
{
    gaf::Names nm {};
    nm.nodeNames = d.nodeNames.p;
    nm.nodeNameOff = d.nodeNameOff.p;
    nm.originalSize = d.originalSize.p;
    nm.ids = gaf::IdView { d.host.ids.key.empty() ? nullptr : d.idKey.p, d.idVal.p, d.host.ids.val.size(), d.host.ids.base };
    return nm;
}

template <typename T>
bool upload(DevGrow<T>& dst, const std::vector<T>& src, cudaStream_t s)
{
    return dst.reserve(std::max<size_t>(src.size(), 1))
        && (src.empty() || cudaMemcpyAsync(dst.p, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice, s) == cudaSuccess);
}

// edit ops of at most this many trace items go down at once
constexpr uint64_t kChunkOps = 1ULL << 27;

// Writes the classified lines of reads on the device in chunks and appends them, each with its
// newline, to text; readEnd[i] = where read i's text ends.  False on a CUDA error.
bool write_reads(GafDevice& d, const std::vector<const std::string*>& names, const std::vector<const gahost::ClassifiedLines*>& reads,
    std::string& text, std::vector<uint64_t>& readEnd)
{
    const size_t n = reads.size();
    text.clear();
    readEnd.assign(n, 0);
    cudaStream_t s = d.stream;
    size_t from = 0;
    while (from < n)
    {
        size_t to = from;
        uint64_t ops = 0;
        while (to < n && (to == from || ops + reads[to]->ops.size() <= kChunkOps)) ops += reads[to++]->ops.size();
        const size_t m = to - from;
        // where each read's lines, ops, entries and name go in the chunk
        std::vector<uint64_t> lineAt(m + 1, 0), opAt(m + 1, 0), entryAt(m + 1, 0);
        uint64_t nameBytes = 0;
        for (size_t k = 0; k < m; k++)
        {
            const auto& c = *reads[from + k];
            lineAt[k + 1] = lineAt[k] + c.lines.size();
            opAt[k + 1] = opAt[k] + c.ops.size();
            entryAt[k + 1] = entryAt[k] + c.entries.size();
            nameBytes += names[from + k]->size();
        }
        const uint64_t lines = lineAt[m], entries = entryAt[m];
        if (!d.hOps.reserve(std::max<uint64_t>(ops, 1)) || !d.hMeta.reserve(std::max<uint64_t>(lines, 1)) || !d.hEntries.reserve(std::max<uint64_t>(entries, 1))
            || !d.hNames.reserve(std::max<uint64_t>(nameBytes, 1)) || !d.hNameOff.reserve(m + 1) || !d.hLen.reserve(std::max<uint64_t>(lines, 1))
            || !d.hStart.reserve(std::max<uint64_t>(lines, 1)))
            return false;
        uint64_t at = 0;
        for (size_t k = 0; k < m; k++)
        {
            d.hNameOff[k] = at;
            at += names[from + k]->size();
        }
        d.hNameOff[m] = at;
        gahost::parallelFor(m, [&](size_t k)
        {
            const auto& c = *reads[from + k];
            memcpy(d.hNames.p + d.hNameOff[k], names[from + k]->data(), names[from + k]->size());
            if (!c.ops.empty()) memcpy(d.hOps.p + opAt[k], c.ops.data(), c.ops.size());
            if (!c.entries.empty()) memcpy(d.hEntries.p + entryAt[k], c.entries.data(), c.entries.size() * 4);
            for (size_t q = 0; q < c.lines.size(); q++)
            {
                gaf::LineMeta meta = c.lines[q];
                meta.op += opAt[k];
                meta.entry += entryAt[k];
                meta.read = (uint32_t)k;
                d.hMeta[lineAt[k] + q] = meta;
            }
        });
        if (!d.ops.reserve(std::max<uint64_t>(ops, 1)) || !d.meta.reserve(std::max<uint64_t>(lines, 1)) || !d.entries.reserve(std::max<uint64_t>(entries, 1))
            || !d.names.reserve(std::max<uint64_t>(nameBytes, 1)) || !d.nameOff.reserve(m + 1) || !d.len.reserve(std::max<uint64_t>(lines, 1))
            || !d.start.reserve(std::max<uint64_t>(lines, 1)))
            return false;
        if ((ops && cudaMemcpyAsync(d.ops.p, d.hOps.p, ops, cudaMemcpyHostToDevice, s) != cudaSuccess)
            || (lines && cudaMemcpyAsync(d.meta.p, d.hMeta.p, lines * sizeof(gaf::LineMeta), cudaMemcpyHostToDevice, s) != cudaSuccess)
            || (entries && cudaMemcpyAsync(d.entries.p, d.hEntries.p, entries * 4, cudaMemcpyHostToDevice, s) != cudaSuccess)
            || (nameBytes && cudaMemcpyAsync(d.names.p, d.hNames.p, nameBytes, cudaMemcpyHostToDevice, s) != cudaSuccess)
            || cudaMemcpyAsync(d.nameOff.p, d.hNameOff.p, (m + 1) * 8, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return false;
        gaf::Names nm = device_names(d);
        nm.readNames = d.names.p;
        nm.readNameOff = d.nameOff.p;
        nm.readLen = nullptr;
        const uint32_t blocks = (uint32_t)((lines + kLineWarps - 1) / kLineWarps);
        if (lines)
        {
            gaf_measure_kernel<<<blocks, 32 * kLineWarps, 0, s>>>(nm, d.meta.p, d.ops.p, d.entries.p, (uint32_t)lines, d.len.p);
            if (cudaGetLastError() != cudaSuccess) return false;
            if (cudaMemcpyAsync(d.hLen.p, d.len.p, lines * 8, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
                return false;
        }
        uint64_t total = 0;
        const uint64_t base = text.size();
        for (size_t k = 0; k < m; k++)
        {
            for (uint64_t q = lineAt[k]; q < lineAt[k + 1]; q++)
            {
                d.hStart[q] = total;
                total += (uint64_t)d.hLen[q] + 1;
            }
            readEnd[from + k] = base + total;
        }
        if (lines)
        {
            if (!d.text.reserve(std::max<uint64_t>(total, 1))) return false;
            if (cudaMemcpyAsync(d.start.p, d.hStart.p, lines * 8, cudaMemcpyHostToDevice, s) != cudaSuccess) return false;
            gaf_write_kernel<<<blocks, 32 * kLineWarps, 0, s>>>(nm, d.meta.p, d.ops.p, d.entries.p, (uint32_t)lines, d.start.p, d.text.p);
            if (cudaGetLastError() != cudaSuccess) return false;
            text.resize(base + total);
            if (cudaMemcpyAsync(&text[base], d.text.p, total, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
                return false;
        }
        from = to;
    }
    return true;
}

}

int ga_gaf_device_init(GafDevice& d, const gahost::HostGraph& g)
{
    cudaGetDevice(&d.device);
    if (!d.stream && cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking) != cudaSuccess) return GA_ERR_CUDA;
    gaf::build_names(g.lookupIds, g.names, g.originalSize, d.host);
    cudaStream_t s = d.stream;
    if (!upload(d.nodeNames, d.host.nodeNames, s) || !upload(d.nodeNameOff, d.host.nodeNameOff, s) || !upload(d.originalSize, d.host.originalSize, s)
        || !upload(d.idKey, d.host.ids.key, s) || !upload(d.idVal, d.host.ids.val, s) || cudaStreamSynchronize(s) != cudaSuccess)
        return GA_ERR_CUDA;
    return GA_OK;
}

bool ga_gaf_device_write(void* ctx, const std::vector<const std::string*>& names, const std::vector<const gahost::ClassifiedLines*>& reads,
    std::string& text, std::vector<uint64_t>& readEnd)
{
    GafDevice& d = *(GafDevice*)ctx;
    const auto t0 = std::chrono::steady_clock::now();
    const bool ok = write_reads(d, names, reads, text, readEnd);
    if (!ok) ga_set_last_error("GAF lines on the device failed");
    d.ms += ms_since(t0);
    return ok;
}

bool ga_gaf_device_select(void* ctx, const std::vector<uint64_t>& first, const std::vector<uint64_t>& start, const std::vector<uint64_t>& end,
    const std::vector<double>& xscore, int minAlignmentScore, double fractionCutoff, std::vector<char>& keep)
{
    GafDevice& d = *(GafDevice*)ctx;
    const auto t0 = std::chrono::steady_clock::now();
    const uint32_t reads = (uint32_t)(first.size() - 1);
    const uint64_t m = start.size();
    cudaStream_t s = d.stream;
    bool ok = d.hSel.reserve(first.size() + 2 * m) && d.hScore.reserve(std::max<uint64_t>(m, 1)) && d.hKeep.reserve(std::max<uint64_t>(m, 1))
        && d.sel.reserve(first.size() + 2 * m) && d.score.reserve(std::max<uint64_t>(m, 1)) && d.keep.reserve(std::max<uint64_t>(m, 1));
    if (ok)
    {
        memcpy(d.hSel.p, first.data(), first.size() * 8);
        memcpy(d.hSel.p + first.size(), start.data(), m * 8);
        memcpy(d.hSel.p + first.size() + m, end.data(), m * 8);
        memcpy(d.hScore.p, xscore.data(), m * 8);
        ok = cudaMemcpyAsync(d.sel.p, d.hSel.p, (first.size() + 2 * m) * 8, cudaMemcpyHostToDevice, s) == cudaSuccess
            && cudaMemcpyAsync(d.score.p, d.hScore.p, m * 8, cudaMemcpyHostToDevice, s) == cudaSuccess;
    }
    if (ok)
    {
        select_kernel<<<(reads + 127) / 128, 128, 0, s>>>(d.sel.p, d.sel.p + first.size(), d.sel.p + first.size() + m, d.score.p, reads,
            minAlignmentScore, fractionCutoff, d.keep.p);
        ok = cudaGetLastError() == cudaSuccess && cudaMemcpyAsync(d.hKeep.p, d.keep.p, m, cudaMemcpyDeviceToHost, s) == cudaSuccess
            && cudaStreamSynchronize(s) == cudaSuccess;
    }
    if (ok) memcpy(keep.data(), d.hKeep.p, m);
    else ga_set_last_error("alignment selection on the device failed");
    d.ms += ms_since(t0);
    return ok;
}

// ---- C ABI ----

extern "C" int ga_aligner_format_gaf(ga_aligner_t a, uint32_t num_lines, const ga_gaf_line* lines, uint64_t num_items, const ga_gaf_item* items,
    uint32_t num_reads, const char* const* read_names, const uint32_t* read_lens, uint8_t cigar_match_mismatch, const char** text, uint64_t* bytes,
    const uint64_t** line_ends, const uint8_t** failed)
{
    static_assert(sizeof(ga_gaf_item) == sizeof(gaf::Item) && sizeof(ga_gaf_line) == sizeof(gaf::Line), "GAF record layouts");
    if (!a || !text || !bytes || !line_ends || !failed || (num_lines && !lines) || (num_items && !items) || (num_reads && (!read_names || !read_lens)))
        return GA_ERR_ARGUMENT;
    GafDevice& d = a->gafDev;
    for (uint32_t k = 0; k < num_lines; k++)
    {
        const ga_gaf_line& l = lines[k];
        if (l.read >= num_reads || l.first_item + l.item_count > num_items || l.item_count == 0)
        {
            ga_set_last_error(("ga_aligner_format_gaf: line " + std::to_string(k) + " names a read or items it was not given").c_str());
            return GA_ERR_ARGUMENT;
        }
    }
    // each line is walked on the host's cores, then the good ones are written on the device
    const gaf::NamesHost& nh = d.host;
    auto sizeOf = [&nh](int32_t bignode) -> uint64_t
    {
        const uint32_t i = nh.ids.find(bignode);
        return i == gaf::kNoId ? 0 : nh.originalSize[i];
    };
    std::vector<gahost::ClassifiedLines> cls(num_lines);
    std::vector<std::string> names(num_lines);
    d.lastFailed.assign(num_lines, 0);
    gahost::parallelFor(num_lines, [&](size_t k)
    {
        const ga_gaf_line& l = lines[k];
        const gaf::Item* it = (const gaf::Item*)items + l.first_item;
        gahost::ClassifiedLines& c = cls[k];
        c.lines.resize(1);
        c.ops.resize(l.item_count);
        c.entries.resize(l.item_count);
        gaf::LineMeta& m = c.lines[0];
        if (!gaf::classify_line([it](uint32_t q) { return it[q]; }, l.item_count, read_lens[l.read], cigar_match_mismatch != 0, sizeOf, m,
                c.ops.data(), c.entries.data()))
        {
            d.lastFailed[k] = 1;
            c = gahost::ClassifiedLines {};
            return;
        }
        m.op = 0;
        m.entry = 0;
        m.xscore100 = l.xscore100;
        m.mapq = l.mapq;
        c.entries.resize(m.entries);
        names[k] = read_names[l.read] ? read_names[l.read] : "";
    });
    std::vector<const std::string*> np;
    std::vector<const gahost::ClassifiedLines*> rp;
    for (uint32_t k = 0; k < num_lines; k++)
    {
        if (d.lastFailed[k]) continue;
        np.push_back(&names[k]);
        rp.push_back(&cls[k]);
    }
    std::string body;
    std::vector<uint64_t> ends;
    if (!write_reads(d, np, rp, body, ends))
    {
        ga_set_last_error("ga_aligner_format_gaf: device formatting failed");
        return GA_ERR_CUDA;
    }
    // the text in line order, a failed line as a lone newline
    d.lastText.clear();
    d.lastEnds.assign(num_lines, 0);
    size_t g = 0;
    uint64_t prev = 0;
    for (uint32_t k = 0; k < num_lines; k++)
    {
        if (d.lastFailed[k]) d.lastText += '\n';
        else
        {
            d.lastText.append(body, prev, ends[g] - prev);
            prev = ends[g++];
        }
        d.lastEnds[k] = d.lastText.size();
    }
    *text = d.lastText.data();
    *bytes = d.lastText.size();
    *line_ends = d.lastEnds.data();
    *failed = d.lastFailed.data();
    return GA_OK;
}

extern "C" int ga_aligner_select_alignments(ga_aligner_t a, uint32_t num_reads, const uint64_t* first, const uint64_t* starts,
    const uint64_t* ends, const double* xscores, int32_t min_alignment_score, double multimap_score_fraction, uint8_t* keep)
{
    if (!a || !first || !keep || (num_reads && (!starts || !ends || !xscores))) return GA_ERR_ARGUMENT;
    std::vector<uint64_t> f(first, first + num_reads + 1);
    for (uint32_t r = 0; r < num_reads; r++)
        if (f[r + 1] < f[r]) return GA_ERR_ARGUMENT;
    const uint64_t m = f[num_reads] - f[0];
    for (auto& x : f) x -= first[0];
    std::vector<uint64_t> s(starts + first[0], starts + first[0] + m), e(ends + first[0], ends + first[0] + m);
    std::vector<double> x(xscores + first[0], xscores + first[0] + m);
    std::vector<char> k(m, 0);
    if (m && !ga_gaf_device_select(&a->gafDev, f, s, e, x, min_alignment_score, multimap_score_fraction, k)) return GA_ERR_CUDA;
    for (uint64_t i = 0; i < m; i++) keep[first[0] + i] = (uint8_t)k[i];
    return GA_OK;
}
