// parquet.cu -- Parquet column chunks decoded on the device, with a runtime
// key filter evaluated on their encoded pages.
//
// Reference: the engine's Parquet reader decodes row groups on the host
// (crates/krishiv-io/src/parquet/decode.rs, through the parquet crate) and
// evaluates pushed predicates on a chunk's dictionary entries, once per entry
// (parquet/dict_probe.rs: `all_dictionary`, `passes`), so that a predicate on
// a dictionary-encoded column costs one test per entry and a lookup per row;
// a row group none of whose entries passes is skipped (`any_entry_in`).
// Here the chunk's bytes cross to HBM as the file stores them and:
//  - the host walks the page headers (Thrift compact protocol: parquet.thrift
//    PageHeader, DataPageHeader, DataPageHeaderV2, DictionaryPageHeader) and
//    lays every page out at a 16-byte aligned place of a staging buffer;
//  - stage_kernel (one CTA per page) copies each page's raw bytes there and
//    snappy_kernel decompresses Snappy (the raw format Parquet uses), one CTA
//    per fragment of a page (runs of about 64 KiB of output that the host
//    finds by walking the tags), its elements and its back-references followed
//    by pointer doubling in shared memory; a large page of many short elements
//    is decoded by the whole device (the big_*_kernels);
//  - dict_filter_kernel tests every dictionary entry against the key filter
//    (one byte per entry);
//  - page_decode_kernel (one CTA per data page, tiles of 1024 rows) decodes
//    the definition levels and the dictionary indices (RLE / bit-packed
//    hybrid: the levels' runs listed by pointer doubling, the indices' by one
//    thread, every thread decoding its rows from the lists), ranks the tile's non-NULL rows with a block scan,
//    and writes the Arrow column, its validity and the filter's bit per row
//    (a dictionary entry's answer, or the member test of a PLAIN value);
//  - BYTE_ARRAY columns: ba_walk_kernel walks the PLAIN values of the
//    dictionary page and of PLAIN data pages into a (start, length) table,
//    page_decode_kernel writes each row's reference into it, and the string
//    gather of the join's payloads makes the UTF-8 / binary column.
// Flat columns only (max repetition level 0, max definition level 0 or 1);
// physical types INT32, INT64, DOUBLE and BYTE_ARRAY; PLAIN, PLAIN_DICTIONARY and
// RLE_DICTIONARY values; UNCOMPRESSED and SNAPPY chunks; data pages v1 and
// v2. Anything else returns KRV_UNSUPPORTED; bytes that do not decode return
// KRV_INVALID_ARGUMENT. Kernels read only inside their page's bytes.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "krv_filter.cuh"
#include "ops.h"

namespace krv {

namespace {

// parquet.thrift enums
constexpr int kPageData = 0, kPageIndex = 1, kPageDict = 2, kPageDataV2 = 3;
constexpr int kEncPlain = 0, kEncPlainDict = 2, kEncRle = 3, kEncRleDict = 8;
constexpr int kTile = 1024;        // rows per tile of page_decode_kernel
constexpr int kDecodeThreads = 256;
constexpr int kStageThreads = 256;
constexpr uint32_t ST_CORRUPT = 1u << 8;  // a page's bytes do not decode

// ---- host: the page headers ---------------------------------------------------------
struct Thrift {
    const uint8_t *p, *end;
    int depth = 0;
    [[noreturn]] static void corrupt(const char *what) {
        fail(KRV_INVALID_ARGUMENT, std::string("corrupt Parquet page header: ") + what);
    }
    uint8_t byte() {
        if (p >= end) corrupt("truncated");
        return *p++;
    }
    uint64_t varint() {
        uint64_t v = 0;
        for (int s = 0; s < 64; s += 7) {
            const uint8_t b = byte();
            v |= (uint64_t)(b & 0x7F) << s;
            if (!(b & 0x80)) return v;
        }
        corrupt("varint longer than 10 bytes");
    }
    int64_t zigzag() {
        const uint64_t v = varint();
        return (int64_t)(v >> 1) ^ -(int64_t)(v & 1);
    }
    void skip_bytes(uint64_t n) {
        if (n > (uint64_t)(end - p)) corrupt("truncated");
        p += n;
    }
    void skip(int type) {
        switch (type) {
        case 1: case 2: return;  // a struct field's bool lives in its type nibble
        case 3: skip_bytes(1); return;
        case 4: case 5: case 6: varint(); return;
        case 7: skip_bytes(8); return;
        case 8: skip_bytes(varint()); return;
        case 9: case 10: {  // list, set
            const uint8_t h = byte();
            uint64_t n = h >> 4;
            const int et = h & 15;
            if (n == 15) n = varint();
            for (uint64_t i = 0; i < n; i++) skip_elem(et);
            return;
        }
        case 11: {  // map
            const uint64_t n = varint();
            if (n == 0) return;
            const uint8_t kv = byte();
            for (uint64_t i = 0; i < n; i++) {
                skip_elem(kv >> 4);
                skip_elem(kv & 15);
            }
            return;
        }
        case 12: skip_struct(); return;
        default: corrupt("unknown field type");
        }
    }
    void skip_elem(int type) {
        if (type == 1 || type == 2) skip_bytes(1);  // bools inside containers are one byte
        else skip(type);
    }
    // Calls f(field id, type) for every field of a struct; f reads or skips it.
    template <class F> void fields(F &&f) {
        if (++depth > 32) corrupt("nested too deep");
        int16_t last = 0;
        for (;;) {
            const uint8_t h = byte();
            if (h == 0) break;
            const int type = h & 15, delta = h >> 4;
            const int16_t id = delta ? (int16_t)(last + delta) : (int16_t)zigzag();
            last = id;
            f(id, type);
        }
        depth--;
    }
    void skip_struct() {
        fields([&](int, int t) { skip(t); });
    }
    int32_t i32(int type) {
        if (type != 5) corrupt("expected an i32");
        const int64_t v = zigzag();
        if (v < INT32_MIN || v > INT32_MAX) corrupt("i32 out of range");
        return (int32_t)v;
    }
};

struct PageHdr {
    int type = -1;
    int32_t usize = -1, csize = -1;
    int32_t nvalues = -1, encoding = -1, def_encoding = kEncRle;
    int32_t def_len = 0, rep_len = 0;
    bool compressed = true;  // v2: is_compressed
};

PageHdr parse_page_header(Thrift &t) {
    PageHdr h;
    t.fields([&](int id, int type) {
        switch (id) {
        case 1: h.type = t.i32(type); break;
        case 2: h.usize = t.i32(type); break;
        case 3: h.csize = t.i32(type); break;
        case 5:  // DataPageHeader
            if (type != 12) Thrift::corrupt("data_page_header");
            t.fields([&](int f, int ft) {
                if (f == 1) h.nvalues = t.i32(ft);
                else if (f == 2) h.encoding = t.i32(ft);
                else if (f == 3) h.def_encoding = t.i32(ft);
                else t.skip(ft);
            });
            break;
        case 7:  // DictionaryPageHeader
            if (type != 12) Thrift::corrupt("dictionary_page_header");
            t.fields([&](int f, int ft) {
                if (f == 1) h.nvalues = t.i32(ft);
                else if (f == 2) h.encoding = t.i32(ft);
                else t.skip(ft);
            });
            break;
        case 8:  // DataPageHeaderV2
            if (type != 12) Thrift::corrupt("data_page_header_v2");
            t.fields([&](int f, int ft) {
                if (f == 1) h.nvalues = t.i32(ft);
                else if (f == 4) h.encoding = t.i32(ft);
                else if (f == 5) h.def_len = t.i32(ft);
                else if (f == 6) h.rep_len = t.i32(ft);
                else if (f == 7) h.compressed = ft == 1;  // bool: 1 true, 2 false
                else t.skip(ft);
            });
            break;
        default: t.skip(type);
        }
    });
    return h;
}

// ---- device descriptors ---------------------------------------------------------------
struct StageDev {
    int64_t src, dst;   // page payload in the chunk; its staged place
    int32_t csize, usize;
    int32_t raw;        // leading bytes copied as they are (v2 levels)
    int32_t snappy;     // the rest is Snappy-compressed
};
// A run of a Snappy stream's elements that decodes alone: its first element
// in the chunk, its first output byte in the staging buffer, their lengths.
struct FragDev {
    int64_t src, dst;
    int32_t slen, dlen;
};
struct PageDev {
    int64_t staged;     // offset of the staged (uncompressed) page
    int64_t row0;       // the page's first row in the chunk
    int32_t usize;
    int32_t nvalues;
    int32_t v2;         // levels without a length prefix (data page v2)
    int32_t dict;       // values are dictionary indices
    int32_t def_len;    // v2: bytes of the definition levels
    int32_t pad;
};
// OUT_REF (BYTE_ARRAY): each row's value is written as a reference, its
// dictionary entry or dict_n + (its page's first row) + (its rank among the
// page's non-NULL values), into the (start, length) table the walk filled;
// -1 for NULL. The string column is then gathered by those references.
enum OutKind : int32_t { OUT_SAME = 0, OUT_I32_TO_I64 = 1, OUT_TO_DEC128 = 2, OUT_REF = 3 };
struct DecodeArgs {
    const PageDev *pages;
    const uint8_t *staged;
    int32_t max_def;
    int32_t pwidth;     // bytes per PLAIN value: 4 or 8
    int32_t out_kind;
    int32_t is_int;     // the values are integers (the filter tests them)
    void *out;
    uint32_t *valid;    // null when the column is required
    const uint8_t *dict;
    int64_t dict_n;
    const uint8_t *dict_pass;  // the filter's answer per dictionary entry (null without a filter)
    int32_t has_filter;
    int32_t pad;
    KeyFilterDev f;
    uint32_t *pass;     // the filter's bit per row
    unsigned long long *counts;  // [0] rows passing the filter
    uint32_t *status;
    long long *ref;      // OUT_REF: each row's value reference
    const int32_t *walked;  // OUT_REF: the values the walk found in each PLAIN page
};
// A BYTE_ARRAY page whose values are walked: PLAIN values, each a 4-byte
// little-endian length and its bytes, one after another.
struct WalkDev {
    int64_t staged;     // the staged page
    int64_t base;       // its first value's slot in the (start, length) table
    int32_t usize;
    int32_t kind;       // 0 dictionary page, 1 data page v1, 2 data page v2
    int32_t def_len;    // v2: bytes of the definition levels
    int32_t limit;      // the values it may hold
    int32_t page;       // the data page's index (walked[page]); -1 for the dictionary
    int32_t pad;
};

// ---- stage: copy or Snappy-decompress each page ------------------------------------------
// Copies n bytes (any alignment) with `threads` threads, thread t taking
// bytes t, t + threads, ...: every thread issues kCopyDepth loads before its
// stores, so that many bytes are in flight per thread instead of one
// load-to-store round trip per byte. src and dst do not overlap.
constexpr int kCopyDepth = 16;
__device__ __forceinline__ void copy_bytes(uint8_t *dst, const uint8_t *src, int64_t n, int t, int threads) {
    for (int64_t i0 = 0; i0 < n; i0 += (int64_t)threads * kCopyDepth) {
        uint8_t v[kCopyDepth];
#pragma unroll
        for (int u = 0; u < kCopyDepth; u++) {
            const int64_t i = i0 + (int64_t)u * threads + t;
            v[u] = i < n ? src[i] : 0;
        }
#pragma unroll
        for (int u = 0; u < kCopyDepth; u++) {
            const int64_t i = i0 + (int64_t)u * threads + t;
            if (i < n) dst[i] = v[u];
        }
    }
}

// Snappy (raw format): a varint of the uncompressed length, then elements:
// literals (tag & 3 == 0) and back-references with 1-, 2- or 4-byte offsets.
// The elements are a chain (each starts where the last ended) and their bytes
// another (a back-reference may copy what the element before it wrote: the
// zero bytes of a page of small integers refer from value to value through
// the whole page). Both chains are followed by pointer doubling, a batch of
// the stream at a time, one CTA per fragment:
//  1. kSnappyWin stream bytes go to shared memory and every position is
//     parsed as if an element began there: its end is a link;
//  2. the links are squared until the whole chain from the batch's first
//     element is marked (log2 of its elements rounds), and the marked
//     positions are compacted and their lengths scanned into output places;
//  3. every output byte of the batch (at most kSnappyOut) gets its source: a
//     stream byte, an output byte before the batch, or one of the batch;
//  4. sources inside the batch are replaced by their own sources until none is
//     left (again log2 of the longest chain rounds), and the bytes written.
// A literal that does not fit the window is copied by the whole CTA. Bound by
// the rounds' barriers and shared-memory accesses. Measured on B200: a
// dictionary page of 100,000 int64 keys (13 fragments of 64 KiB) 4.0 ms with
// one warp per fragment taking the elements one after another, 0.24 ms
// now.
constexpr int kSnappyThreads = 1024;
constexpr int kSnappyWin = 4096;   // stream bytes per batch
constexpr int kSnappyOut = 16384;  // output bytes per batch
constexpr int kSnappyElems = kSnappyWin / 2;  // the shortest element takes two bytes
constexpr int kSnappyPer = kSnappyWin / kSnappyThreads;
constexpr int kSnappyLong = 32;    // elements from here on are spread over a warp
struct SnappySmem {
    int src[kSnappyOut];             // per output byte: >= 0 a byte of the batch; -1 - i stream byte i of the
                                     // window; kSnappyPrior - i output byte i before the batch
    uint16_t link[2][kSnappyWin + 8];
    uint16_t el_pos[kSnappyElems], el_out[kSnappyElems];
    uint16_t longs[kSnappyElems];
    uint8_t win[kSnappyWin + 8];
    uint8_t mark[kSnappyWin + 8];
    unsigned warp_sum[2][kSnappyThreads / 32];
    int end, nel, nout, nlong, bad;
};
constexpr int kSnappyPrior = -8192;
static_assert(kSnappyPrior < -kSnappyWin && kSnappyPer == 4, "source codes do not meet; marks are read four at a time");

// The element at window byte i: stream bytes of its tag and length (`head`),
// output bytes (`len`), the back-reference's offset (0: a literal). False when
// the window's n bytes do not hold its head.
__device__ __forceinline__ bool snappy_element(const uint8_t *w, int i, int n, int &head, int64_t &len, int64_t &off) {
    const uint8_t tag = w[i];
    const int kind = tag & 3;
    off = 0;
    if (kind == 0) {
        len = tag >> 2;
        const int nb = len >= 60 ? (int)len - 59 : 0;
        head = 1 + nb;
        if (i + head > n) return false;
        if (nb) {
            len = 0;
            for (int k = 0; k < nb; k++) len |= (int64_t)w[i + 1 + k] << (8 * k);
        }
        len += 1;
        return true;
    }
    head = kind == 1 ? 2 : kind == 2 ? 3 : 5;
    if (i + head > n) return false;
    if (kind == 1) {
        len = 4 + ((tag >> 2) & 7);
        off = ((int64_t)(tag >> 5) << 8) | w[i + 1];
    } else {
        len = 1 + (tag >> 2);
        for (int k = 0; k + 1 < head; k++) off |= (int64_t)w[i + 1 + k] << (8 * k);
    }
    if (off == 0) off = -1;  // never a valid offset
    return true;
}

// The elements of one fragment: stream bytes [0, slen) to output bytes
// [0, dlen); a back-reference reaching before the fragment is corrupt. The
// same answer on every thread.
__device__ bool snappy_fragment(SnappySmem &S, const uint8_t *src, int64_t slen, uint8_t *dst, int64_t dlen) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int64_t ip = 0, op = 0;
    while (ip < slen) {
        const int n = (int)min((int64_t)kSnappyWin, slen - ip);
#pragma unroll
        for (int k = 0; k < kSnappyPer; k++) {
            const int i = k * kSnappyThreads + t;
            if (i < n) S.win[i] = src[ip + i];
            S.mark[i] = i == 0;
        }
        if (t == 0) {
            S.link[0][n] = S.link[1][n] = (uint16_t)n;
            S.end = n;
            S.nel = S.nout = S.nlong = S.bad = 0;
        }
        __syncthreads();
        // 1. every position's element (this thread's are neighbours: 4t ..)
        int elen[kSnappyPer];
        unsigned stop = 0;
#pragma unroll
        for (int k = 0; k < kSnappyPer; k++) {
            const int i = t * kSnappyPer + k;
            elen[k] = 0;
            if (i >= n) continue;
            int head;
            int64_t len, off;
            int next = n;
            if (!snappy_element(S.win, i, n, head, len, off) || (off == 0 && i + head + len > n)) {
                stop |= 1u << k;  // it ends the chain of this batch
            } else {
                elen[k] = (int)len;
                next = i + head + (off == 0 ? (int)len : 0);
            }
            S.link[0][i] = (uint16_t)next;
        }
        __syncthreads();
        // 2. the chain from position 0
        int cur = 0;
        for (int round = 0; round < 12; round++) {  // 2^11 elements at most
            const bool last = S.link[cur][0] == n;
#pragma unroll
            for (int k = 0; k < kSnappyPer; k++) {
                const int i = t * kSnappyPer + k;
                if (i >= n) continue;
                const int j = S.link[cur][i];
                if (S.mark[i] && j < n) S.mark[j] = 1;
                S.link[cur ^ 1][i] = S.link[cur][j];
            }
            __syncthreads();
            if (last) break;
            cur ^= 1;
        }
        const unsigned marks = reinterpret_cast<const unsigned *>(S.mark)[t];
        unsigned cnt = 0, bytes = 0;
#pragma unroll
        for (int k = 0; k < kSnappyPer; k++)
            if (t * kSnappyPer + k < n && ((marks >> (8 * k)) & 1u)) {
                cnt++;
                bytes += (unsigned)elen[k];
            }
        unsigned ci = cnt, bi = bytes;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned y = __shfl_up_sync(0xFFFFFFFFu, ci, d), z = __shfl_up_sync(0xFFFFFFFFu, bi, d);
            if (lane >= d) ci += y, bi += z;
        }
        if (lane == 31) S.warp_sum[0][warp] = ci, S.warp_sum[1][warp] = bi;
        __syncthreads();
        unsigned cw = S.warp_sum[0][lane], bw = S.warp_sum[1][lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned y = __shfl_up_sync(0xFFFFFFFFu, cw, d), z = __shfl_up_sync(0xFFFFFFFFu, bw, d);
            if (lane >= d) cw += y, bw += z;
        }
        unsigned at = (warp ? __shfl_sync(0xFFFFFFFFu, cw, (warp + 31) & 31) : 0u) + ci - cnt;
        unsigned o = (warp ? __shfl_sync(0xFFFFFFFFu, bw, (warp + 31) & 31) : 0u) + bi - bytes;
#pragma unroll
        for (int k = 0; k < kSnappyPer; k++) {
            const int i = t * kSnappyPer + k;
            if (i >= n || !((marks >> (8 * k)) & 1u)) continue;
            if (((stop >> k) & 1u) || o + elen[k] > (unsigned)kSnappyOut) {
                atomicMin(&S.end, i);  // the next batch begins at the first element not taken
            } else {
                S.el_pos[at] = (uint16_t)i;
                S.el_out[at] = (uint16_t)o;
                atomicMax(&S.nel, (int)at + 1);
                atomicMax(&S.nout, (int)(o + elen[k]));
            }
            at++;
            o += (unsigned)elen[k];
        }
        __syncthreads();
        const int nel = S.nel, nout = S.nout, end = S.end;
        if (nel == 0) {
            // a literal past the window, or bytes that end inside an element
            int head;
            int64_t len, off;
            const bool ok = snappy_element(S.win, 0, n, head, len, off) && off == 0 && ip + head + len <= slen &&
                            op + len <= dlen;
            if (!ok) return false;
            copy_bytes(dst + op, src + ip + head, len, t, kSnappyThreads);
            ip += head + len;
            op += len;
            __syncthreads();
            continue;
        }
        if (op + nout > dlen) return false;
        // 3. every output byte's source
        for (int e = t; e < nel; e += kSnappyThreads) {
            int head;
            int64_t len, off;
            const int i = S.el_pos[e], o0 = S.el_out[e];
            snappy_element(S.win, i, n, head, len, off);
            if (off != 0 && (off < 0 || off > op + o0)) {
                S.bad = 1;
                continue;
            }
            if (len >= kSnappyLong) {
                S.longs[atomicAdd(&S.nlong, 1)] = (uint16_t)e;
                continue;
            }
            for (int k = 0; k < (int)len; k++) {
                const int64_t from = (int64_t)o0 + k - off;
                S.src[o0 + k] = off == 0 ? -1 - (i + head + k) : from >= 0 ? (int)from : kSnappyPrior - (int)(op + from);
            }
        }
        __syncthreads();
        if (S.bad) return false;
        for (int q = warp; q < S.nlong; q += kSnappyThreads / 32) {
            int head;
            int64_t len, off;
            const int e = S.longs[q], i = S.el_pos[e], o0 = S.el_out[e];
            snappy_element(S.win, i, n, head, len, off);
            for (int k = lane; k < (int)len; k += 32) {
                const int64_t from = (int64_t)o0 + k - off;
                S.src[o0 + k] = off == 0 ? -1 - (i + head + k) : from >= 0 ? (int)from : kSnappyPrior - (int)(op + from);
            }
        }
        __syncthreads();
        // 4. sources of sources. A source only ever moves down its chain, so
        // reading one that another thread has just moved is as good.
        bool more = true;
        while (__syncthreads_or(more)) {
            more = false;
            for (int j = t; j < nout; j += kSnappyThreads) {
                const int v = *reinterpret_cast<volatile int *>(&S.src[j]);
                if (v < 0) continue;
                const int w = *reinterpret_cast<volatile int *>(&S.src[v]);
                *reinterpret_cast<volatile int *>(&S.src[j]) = w;
                more = more || w >= 0;
            }
        }
        for (int j = t; j < nout; j += kSnappyThreads) {
            const int v = S.src[j];
            dst[op + j] = v > kSnappyPrior ? S.win[-1 - v] : dst[kSnappyPrior - v];
        }
        ip += end;
        op += nout;
        __syncthreads();  // the output is read by the next batch, the shared memory rewritten
    }
    return op == dlen;
}

// A large page of many short elements (a dictionary of small integers: 200,000
// of them) is one long chain whose fragments nobody knows yet; walking its
// tags takes a host core 5 ns an element. Such a page is decoded by the whole
// device instead, the same two chains in pieces:
//  - big_link_kernel, a CTA per window of kSnappyWin stream bytes, finds for
//    every position of the window where the chain that begins there leaves it
//    and how many bytes it writes until then (links doubled with their sums);
//  - big_chase_kernel (one CTA) follows the page's chain from window to window
//    and notes each window's first element and its output place;
//  - big_source_kernel marks each window's elements from there, writes the
//    literals and every back-reference byte's source (an output place);
//  - big_jump_kernel, a CTA per kSnappyOut output bytes, replaces sources
//    inside its piece by their own sources until none is left, and
//    big_copy_kernel follows the rest (one hop per piece) to a literal's byte.
// A page that does not parse writes nothing and is reported. Measured on B200,
// 100,000 int64 keys: 0.09 ms for all five, against 0.24 ms for 13 fragments
// in one kernel and 0.6 ms of host time to find them.
struct BigPage {
    int64_t src, dst;    // the stream after its length (in the chunk), its staged output
    int32_t slen, dlen;
    int32_t win0, nwin;  // its windows in the window tables
    int64_t exit0;       // its first stream byte in the exit table
    int64_t from0;       // its first output byte in the source table
    int32_t tile0, ntile;  // its pieces of kSnappyOut output bytes
};
struct BigExit {
    uint32_t bytes;  // output bytes until the chain leaves the window
    uint32_t next;   // where it does, in the page's stream; kBigBad: an element does not end in it
};
constexpr uint32_t kBigBad = 0xFFFFFFFFu;
struct BigEntry {
    int32_t ip, op;  // the window's first element and its output place (ip -1: the chain passes the window by)
};
constexpr int kBigThreads = 1024;
constexpr int kBigHead = 8;  // bytes kept past a window: an element's tag and length

// The page's bytes from `at` on in shared memory: a window and the head of an
// element that begins at its end. How many of them there are.
__device__ __forceinline__ int big_load(const uint8_t *src, int64_t slen, int64_t at, uint8_t *win) {
    const int n = (int)min((int64_t)kSnappyWin + kBigHead, slen - at);
    for (int i = threadIdx.x; i < n; i += kBigThreads) win[i] = src[at + i];
    return n;
}

struct BigLinkSmem {
    uint32_t sum[2][kSnappyWin];   // the chain's bytes until its link
    uint16_t link[2][kSnappyWin];  // its position 1, 2, 4, ... elements on; kSnappyWin: it left the window
    uint16_t tail[2][kSnappyWin];  // its last position in the window until there
    uint8_t win[kSnappyWin + kBigHead];
};

__global__ void __launch_bounds__(kBigThreads) big_link_kernel(const BigPage *pages, const int32_t *win_page,
                                                               const uint8_t *chunk, BigExit *exits) {
    extern __shared__ __align__(16) uint8_t link_smem[];
    BigLinkSmem &L = *reinterpret_cast<BigLinkSmem *>(link_smem);
    uint8_t *s_win = L.win;
    uint16_t(*s_link)[kSnappyWin] = L.link, (*s_tail)[kSnappyWin] = L.tail;
    uint32_t(*s_sum)[kSnappyWin] = L.sum;
    __shared__ int s_more;
    const BigPage P = pages[win_page[blockIdx.x]];
    const int64_t at = (int64_t)(blockIdx.x - P.win0) * kSnappyWin;
    const uint8_t *src = chunk + P.src;
    const int n = big_load(src, P.slen, at, s_win);
    const int m = min(n, kSnappyWin);
    __syncthreads();
    constexpr int kPer = kSnappyWin / kBigThreads;
    uint32_t leave[kPer];  // where the element at this thread's positions ends, when past the window
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int i = k * kBigThreads + threadIdx.x;
        leave[k] = kBigBad;
        if (i >= m) continue;
        int head;
        int64_t len, off;
        uint32_t sum = 0;
        int next = kSnappyWin;
        if (snappy_element(s_win, i, n, head, len, off)) {
            const int64_t end = at + i + head + (off == 0 ? len : 0);
            if (end <= P.slen && len <= P.dlen) {
                sum = (uint32_t)len;
                if (end < at + m) next = (int)(end - at);
                else leave[k] = (uint32_t)end;
            }
        }
        s_link[0][i] = (uint16_t)next;
        s_sum[0][i] = sum;
        s_tail[0][i] = (uint16_t)i;
    }
    int cur = 0;
    for (int round = 0; round < 13; round++) {
        if (threadIdx.x == 0) s_more = 0;
        __syncthreads();
        bool more = false;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const int i = k * kBigThreads + threadIdx.x;
            if (i >= m) continue;
            int j = s_link[cur][i], tail = s_tail[cur][i];
            uint32_t sum = s_sum[cur][i];
            if (j < kSnappyWin) {
                sum += s_sum[cur][j];  // at most 64 x 2048 bytes and one literal of at most dlen (2^24)
                tail = s_tail[cur][j];
                j = s_link[cur][j];
                more = true;
            }
            s_link[cur ^ 1][i] = (uint16_t)j;
            s_sum[cur ^ 1][i] = sum;
            s_tail[cur ^ 1][i] = (uint16_t)tail;
        }
        if (more) s_more = 1;
        __syncthreads();
        cur ^= 1;
        const bool go = s_more != 0;
        __syncthreads();
        if (!go) break;
    }
    // the last element's own end closes the chain: through shared memory, its
    // thread is another
    uint32_t *s_leave = s_sum[cur ^ 1];
#pragma unroll
    for (int k = 0; k < kPer; k++) s_leave[k * kBigThreads + threadIdx.x] = leave[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int i = k * kBigThreads + threadIdx.x;
        if (i < m) exits[P.exit0 + at + i] = BigExit{s_sum[cur][i], s_leave[s_tail[cur][i]]};
    }
}

// One CTA per page. A chain usually enters a window at one of its first
// bytes: those exits are read into shared memory first.
constexpr int kChaseAhead = 16;
constexpr int kChaseWins = 256;
__global__ void __launch_bounds__(256) big_chase_kernel(const BigPage *pages, const BigExit *exits, BigEntry *entries,
                                                        uint32_t *status) {
    __shared__ BigExit s_exit[kChaseWins * kChaseAhead];
    __shared__ int s_ip, s_op;
    const BigPage P = pages[blockIdx.x];
    if (threadIdx.x == 0) s_ip = s_op = 0;
    for (int w0 = 0; w0 < P.nwin; w0 += kChaseWins) {
        const int nw = min(kChaseWins, P.nwin - w0);
        for (int i = threadIdx.x; i < nw * kChaseAhead; i += blockDim.x) {
            const int64_t pos = (int64_t)(w0 + i / kChaseAhead) * kSnappyWin + i % kChaseAhead;
            if (pos < P.slen) s_exit[i] = exits[P.exit0 + pos];
        }
        for (int i = threadIdx.x; i < nw; i += blockDim.x) entries[P.win0 + w0 + i] = BigEntry{-1, 0};
        __syncthreads();
        if (threadIdx.x == 0) {
            int64_t ip = s_ip, op = s_op;
            while (ip >= 0 && ip < P.slen && ip / kSnappyWin < w0 + nw) {
                const int w = (int)(ip / kSnappyWin), r = (int)(ip % kSnappyWin);
                const BigExit e = r < kChaseAhead ? s_exit[(w - w0) * kChaseAhead + r] : exits[P.exit0 + ip];
                entries[P.win0 + w] = BigEntry{(int32_t)ip, (int32_t)op};
                op += e.bytes;
                ip = e.next == kBigBad || op > P.dlen ? -1 : (int64_t)e.next;  // every exit lies past its window
            }
            s_ip = (int)ip;
            s_op = (int)op;
        }
        __syncthreads();
    }
    __syncthreads();
    if (s_ip == P.slen && s_op == P.dlen) return;
    // the stream does not decode to its length: nothing of it is written
    for (int i = threadIdx.x; i < P.nwin; i += blockDim.x) entries[P.win0 + i] = BigEntry{-1, 0};
    if (threadIdx.x == 0) atomicOr(status, ST_CORRUPT);
}

__global__ void __launch_bounds__(kBigThreads) big_source_kernel(const BigPage *pages, const int32_t *win_page,
                                                                 const uint8_t *chunk, const BigEntry *entries,
                                                                 uint8_t *staged, int32_t *from, uint32_t *status) {
    __shared__ uint8_t s_win[kSnappyWin + kBigHead];
    __shared__ __align__(4) uint8_t s_mark[kSnappyWin];
    __shared__ uint16_t s_link[2][kSnappyWin + 8];
    __shared__ uint16_t s_long[kSnappyElems];
    __shared__ int s_long_op[kSnappyElems];
    __shared__ unsigned s_warp[kBigThreads / 32];
    __shared__ int s_nlong;
    const BigPage P = pages[win_page[blockIdx.x]];
    const BigEntry E = entries[blockIdx.x];
    if (E.ip < 0) return;  // the same for the whole CTA
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int64_t at = (int64_t)(blockIdx.x - P.win0) * kSnappyWin;
    const uint8_t *src = chunk + P.src;
    uint8_t *dst = staged + P.dst;
    const int n = big_load(src, P.slen, at, s_win);
    const int m = min(n, kSnappyWin);
    const int first = (int)(E.ip - at);
    __syncthreads();
    constexpr int kPer = kSnappyWin / kBigThreads;
    static_assert(kPer == 4, "marks are read four at a time");
    int elen[kPer];
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int i = t * kPer + k;
        elen[k] = 0;
        if (i >= m) continue;
        int head;
        int64_t len, off;
        int next = m;
        if (snappy_element(s_win, i, n, head, len, off)) {
            elen[k] = (int)min(len, (int64_t)P.dlen + 1);
            const int64_t end = i + head + (off == 0 ? len : 0);
            if (end < m) next = (int)end;
        }
        s_link[0][i] = (uint16_t)next;
        s_mark[i] = i == first;
    }
    if (t == 0) {
        s_link[0][m] = s_link[1][m] = (uint16_t)m;
        s_nlong = 0;
    }
    __syncthreads();
    int cur = 0;
    for (int round = 0; round < 12; round++) {
        const bool last = s_link[cur][first] == m;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const int i = t * kPer + k;
            if (i >= m) continue;
            const int j = s_link[cur][i];
            if (s_mark[i] && j < m) s_mark[j] = 1;
            s_link[cur ^ 1][i] = s_link[cur][j];
        }
        __syncthreads();
        if (last) break;
        cur ^= 1;
    }
    unsigned bytes = 0, marks = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++)
        if (t * kPer + k < m && s_mark[t * kPer + k]) {
            marks |= 1u << k;
            bytes += (unsigned)elen[k];
        }
    unsigned bi = bytes;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, bi, d);
        if (lane >= d) bi += y;
    }
    if (lane == 31) s_warp[warp] = bi;
    __syncthreads();
    unsigned before = 0;
    for (int w = 0; w < warp; w++) before += s_warp[w];
    int64_t op = (int64_t)E.op + before + (bi - bytes);
    int32_t *out_from = from + P.from0;
    bool bad = false;
    // short elements by their thread, longer ones by a warp each
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        if (!((marks >> k) & 1u)) continue;
        const int i = t * kPer + k;
        int head;
        int64_t len, off;
        snappy_element(s_win, i, n, head, len, off);
        // the chain was followed to the page's end before: it stays inside
        if (off != 0 && (off < 0 || off > op)) bad = true;
        else if (op + len > P.dlen || at + i + head + (off == 0 ? len : 0) > P.slen) bad = true;
        else if (len >= kSnappyLong) {
            const int q = atomicAdd(&s_nlong, 1);
            s_long[q] = (uint16_t)i;
            s_long_op[q] = (int)op;
        } else if (off == 0) {
            for (int b = 0; b < (int)len; b++) {
                dst[op + b] = i + head + b < n ? s_win[i + head + b] : src[at + i + head + b];
                out_from[op + b] = -1;
            }
        } else {
            for (int b = 0; b < (int)len; b++) out_from[op + b] = (int)(op + b - off);
        }
        op += elen[k];
    }
    if (bad) atomicOr(status, ST_CORRUPT);
    __syncthreads();
    for (int q = warp; q < s_nlong; q += kBigThreads / 32) {
        int head;
        int64_t len, off;
        const int i = s_long[q], o = s_long_op[q];
        snappy_element(s_win, i, n, head, len, off);
        for (int64_t b = lane; b < len; b += 32) {
            if (off == 0) dst[o + b] = src[at + i + head + b];
            out_from[o + b] = off == 0 ? -1 : (int)(o + b - off);
        }
    }
}

// Pieces of kSnappyOut output bytes: sources inside the piece followed to a
// byte that is not a back-reference or lies before the piece.
__global__ void __launch_bounds__(kBigThreads) big_jump_kernel(const BigPage *pages, const int32_t *tile_page, int32_t *from) {
    extern __shared__ int s_from[];
    const BigPage P = pages[tile_page[blockIdx.x]];
    const int o0 = (blockIdx.x - P.tile0) * kSnappyOut, n = min(kSnappyOut, P.dlen - o0);
    int32_t *mine = from + P.from0 + o0;
    for (int j = threadIdx.x; j < n; j += kBigThreads) s_from[j] = mine[j];
    bool more = true;
    while (__syncthreads_or(more)) {
        more = false;
        for (int j = threadIdx.x; j < n; j += kBigThreads) {
            const int v = *reinterpret_cast<volatile int *>(s_from + j);
            if (v < o0) continue;  // no back-reference, or one that leaves the piece
            const int w = *reinterpret_cast<volatile int *>(s_from + (v - o0));
            if (w < 0) continue;   // its source is a literal's byte
            *reinterpret_cast<volatile int *>(s_from + j) = w;
            more = more || w >= o0;
        }
    }
    for (int j = threadIdx.x; j < n; j += kBigThreads) mine[j] = s_from[j];
}

__global__ void __launch_bounds__(256) big_copy_kernel(const BigPage *pages, const int32_t *tile_page,
                                                       const int32_t *from, uint8_t *staged) {
    const BigPage P = pages[tile_page[blockIdx.x]];
    const int o0 = (blockIdx.x - P.tile0) * kSnappyOut, n = min(kSnappyOut, P.dlen - o0);
    const int32_t *page_from = from + P.from0;
    uint8_t *dst = staged + P.dst;
    for (int j = (int)(blockIdx.y * blockDim.x + threadIdx.x); j < n; j += (int)(gridDim.y * blockDim.x)) {
        int v = page_from[o0 + j];
        if (v < 0) continue;  // a literal's byte is in place
        for (int w; (w = page_from[v]) >= 0;) v = w;  // sources only lie before: this ends
        dst[o0 + j] = dst[v];
    }
}

// Copies each page's leading raw bytes (all of an uncompressed page, a v2
// page's levels) to its staged place, one CTA per page.
__global__ void __launch_bounds__(kStageThreads) stage_kernel(const StageDev *pages, const uint8_t *chunk,
                                                              uint8_t *staged) {
    const StageDev P = pages[blockIdx.x];
    const uint8_t *src = chunk + P.src;
    uint8_t *dst = staged + P.dst;
    const int64_t raw = P.snappy ? P.raw : P.usize;  // uncompressed: the whole page is copied
    if (((uintptr_t)src & 15) == 0) {  // dst is 16-byte aligned: whole 16-byte words where src is too
        const int64_t words = raw / 16;
        for (int64_t i = threadIdx.x; i < words; i += blockDim.x)
            reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
        for (int64_t i = words * 16 + threadIdx.x; i < raw; i += blockDim.x) dst[i] = src[i];
    } else {
        copy_bytes(dst, src, raw, threadIdx.x, blockDim.x);
    }
}

// Decompresses the Snappy fragments, one CTA each.
__global__ void __launch_bounds__(kSnappyThreads) snappy_kernel(const FragDev *frags, const uint8_t *chunk,
                                                                uint8_t *staged, uint32_t *status) {
    extern __shared__ __align__(16) uint8_t snappy_smem[];
    const FragDev F = frags[blockIdx.x];
    const bool ok = snappy_fragment(*reinterpret_cast<SnappySmem *>(snappy_smem), chunk + F.src, F.slen, staged + F.dst, F.dlen);
    if (!ok && threadIdx.x == 0) atomicOr(status, ST_CORRUPT);
}

// ---- the filter over the dictionary entries ------------------------------------------------
__device__ __forceinline__ int64_t load_int(const uint8_t *p, int width) {
    if (width == 4) {
        uint32_t v;
        memcpy(&v, p, 4);
        return (int64_t)(int32_t)v;
    }
    uint64_t v;
    memcpy(&v, p, 8);
    return (int64_t)v;
}

__global__ void dict_filter_kernel(KeyFilterDev f, const uint8_t *dict, int64_t n, int width, uint8_t *pass,
                                   unsigned long long *npass) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const bool p = filter_pass(f, load_int(dict + i * width, width));
        pass[i] = p;
        if (p) atomicAdd(npass, 1ull);
    }
}

// ---- the data pages -------------------------------------------------------------------------
// RLE / bit-packed hybrid (Parquet Encodings.md): runs, each a ULEB128 header;
// header & 1 == 0: an RLE run of header >> 1 copies of one value stored in
// ceil(bit_width / 8) bytes; else (header >> 1) groups of 8 bit-packed values.
// Offsets are bytes from the staged page's start (pages are at most 256 MiB).
struct Hybrid {
    int32_t p, end;     // the stream's next byte and its end
    int32_t bw;
    int32_t kind;       // 0 RLE, 1 bit-packed
    int64_t left;       // values left in the current run
    uint32_t value;     // RLE: the value
    int32_t base;       // bit-packed: the run's first byte
    int32_t bytes;      // bit-packed: the run's bytes
    int32_t bit;        // bit-packed: bit of the next value within the run
};
struct Run {
    int32_t first;      // the run's first value within the tile's list
    uint32_t value;     // RLE: the value
    int32_t base;       // bit-packed: the run's first byte; -1 for an RLE run
    int32_t bytes;
    int32_t bit;        // bit of the run's first listed value
};

__device__ bool next_run(Hybrid &h, const uint8_t *page) {
    for (int guard = 0; guard < 1 << 20; guard++) {
        uint64_t hdr = 0;
        for (int s = 0;; s += 7) {
            if (h.p >= h.end || s > 35) return false;
            const uint8_t b = page[h.p++];
            hdr |= (uint64_t)(b & 0x7F) << s;
            if (!(b & 0x80)) break;
        }
        if (!(hdr & 1)) {
            h.kind = 0;
            h.left = (int64_t)(hdr >> 1);
            const int nb = (h.bw + 7) / 8;
            if (h.end - h.p < nb) return false;
            uint32_t v = 0;
            for (int i = 0; i < nb; i++) v |= (uint32_t)page[h.p + i] << (8 * i);
            h.p += nb;
            if (h.bw < 32 && (v >> h.bw)) return false;
            h.value = v;
        } else {
            h.kind = 1;
            const int64_t groups = (int64_t)(hdr >> 1);
            const int64_t bytes = groups * h.bw;
            if (bytes > (int64_t)(h.end - h.p)) return false;
            h.left = groups * 8;
            h.base = h.p;
            h.bytes = (int32_t)bytes;
            h.bit = 0;
            h.p += (int32_t)bytes;
        }
        if (h.left > 0) return true;
    }
    return false;
}

// Lists the runs covering the next `need` values (thread 0 only).
__device__ bool emit_runs(Hybrid &stream, const uint8_t *page, int need, Run *runs, int &nruns) {
    Hybrid h = stream;  // in registers: the list is one thread's chain
    int at = 0, count = 0;
    while (at < need) {
        if (h.left == 0 && !next_run(h, page)) return false;
        const int take = (int)(h.left < (int64_t)(need - at) ? h.left : (int64_t)(need - at));
        Run r;
        r.first = at;
        r.value = h.value;
        r.base = h.kind ? h.base : -1;
        r.bytes = h.bytes;
        r.bit = h.bit;
        runs[count++] = r;
        if (h.kind == 1) h.bit += take * h.bw;
        h.left -= take;
        at += take;
    }
    stream = h;
    nruns = count;
    return true;
}

// The run that holds value j (0-based within the tile's list).
__device__ __forceinline__ int run_of(const Run *runs, int nruns, int j) {
    int lo = 0, hi = nruns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (runs[mid].first <= j) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
// Value j of the dictionary indices: the two aligned words that hold its at
// most 32 bits and the bit offset (the staging buffer has room past its last
// page; a run's values lie inside the run's bytes).
__device__ __forceinline__ uint32_t run_value(const Run *runs, int nruns, int j, int bw, const uint8_t *page) {
    const Run &r = runs[run_of(runs, nruns, j)];
    if (r.base < 0) return r.value;
    const uint64_t bit = (uint64_t)r.bit + (uint64_t)(j - r.first) * (unsigned)bw;
    const uint64_t at = (uint64_t)(uintptr_t)(page + r.base) + (bit >> 3);
    const uint32_t *w = reinterpret_cast<const uint32_t *>((uintptr_t)(at & ~3ull));
    const unsigned sh = (unsigned)(at & 3) * 8 + (unsigned)(bit & 7);  // at most 31
    const uint32_t lo = w[0], hi = sh + bw > 32 ? w[1] : 0u;
    const uint32_t v = __funnelshift_r(lo, hi, sh);
    return bw == 32 ? v : v & ((1u << bw) - 1u);
}
// The definition levels (0 or 1) of a page, kLevelWin stream bytes at a time.
// Their runs are a chain (20,000 rows with 2% NULLs have about 800 runs, and
// one thread takes 0.3 us a run), so it is followed as the Snappy elements
// are: every byte of the window is parsed as if a run began there, the links
// are doubled until the window's runs are marked, and the marked ones listed
// with a scan of their rows. `bits` of an RLE run is its level, of a
// bit-packed run the place of its first level in the page's bits. Measured on
// B200, 100 pages of 20,000 rows: page_decode_kernel 311 -> 165 us.
constexpr int kLevelWin = 1024;
constexpr int kLevelPer = kLevelWin / kDecodeThreads;
struct LevelRun {
    int32_t first;   // its first row in the page
    uint32_t bits;
};
constexpr uint32_t kLevelRle = 0xFFFFFFFEu;  // + the level (a page has at most 2^28 bytes)
struct Levels {
    LevelRun run[kLevelWin];
    uint16_t link[2][kLevelWin + 1];
    __align__(4) uint8_t mark[kLevelWin];
    uint8_t win[kLevelWin + 8];
    unsigned warp_sum[2][kDecodeThreads / 32];
    int32_t p, end;    // the stream's next byte and its end
    int32_t next;      // where the window's chain goes on
    int32_t nruns;
    int32_t row1;      // the first row that the listed runs do not cover
};
// The run at byte i of the window's n bytes (stream bytes p ..): its stream
// bytes, levels and code. False when it is no run that ends in the stream.
__device__ __forceinline__ bool level_run(const Levels &L, int i, int n, int &size, int64_t &rows, uint32_t &bits) {
    uint64_t hdr = 0;
    int k = 0;
    for (int s = 0;; s += 7) {
        if (i + k >= n || s > 35) return false;
        const uint8_t b = L.win[i + k++];
        hdr |= (uint64_t)(b & 0x7F) << s;
        if (!(b & 0x80)) break;
    }
    rows = (int64_t)(hdr >> 1);
    if (!(hdr & 1)) {
        if (i + k >= n || L.win[i + k] > 1) return false;
        bits = kLevelRle + L.win[i + k];
        size = k + 1;
        return true;
    }
    const int64_t at = (int64_t)L.p + i + k;
    if (rows > L.end - at) return false;
    bits = (uint32_t)at * 8u;
    size = k + (int)rows;
    rows *= 8;
    return true;
}
// Lists the runs from the stream's next byte on that begin in a window, the
// first of them at page row `row0`; `most` rows are enough. All threads; false
// when the stream has no run there.
__device__ bool list_levels(Levels &L, const uint8_t *page, int row0, int most) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) L.p = L.next;
    __syncthreads();
    const int n = min(kLevelWin + 8, L.end - L.p), m = min(kLevelWin, n);
    if (n <= 0) return false;
    for (int i = t; i < n; i += kDecodeThreads) L.win[i] = page[L.p + i];
    __syncthreads();
    uint32_t bits[kLevelPer];
    int rows[kLevelPer], size[kLevelPer];
    unsigned good = 0;
#pragma unroll
    for (int k = 0; k < kLevelPer; k++) {
        const int i = t * kLevelPer + k;
        L.mark[i] = i == 0;
        bits[k] = 0;
        rows[k] = size[k] = 0;
        if (i >= m) continue;
        int64_t r;
        int next = m;
        if (level_run(L, i, n, size[k], r, bits[k])) {
            good |= 1u << k;
            rows[k] = (int)min(r, (int64_t)most);
            next = min(i + size[k], m);
        }
        L.link[0][i] = (uint16_t)next;
    }
    if (t == 0) {
        L.link[0][m] = L.link[1][m] = (uint16_t)m;
        L.nruns = 0;
        L.row1 = row0;
    }
    __syncthreads();
    int cur = 0;
    for (int round = 0; round < 12; round++) {  // at most 2^10 runs (a run of no rows takes one byte)
        const bool last = L.link[cur][0] == m;
#pragma unroll
        for (int k = 0; k < kLevelPer; k++) {
            const int i = t * kLevelPer + k;
            if (i >= m) continue;
            const int j = L.link[cur][i];
            if (L.mark[i] && j < m) L.mark[j] = 1;
            L.link[cur ^ 1][i] = L.link[cur][j];
        }
        __syncthreads();
        if (last) break;
        cur ^= 1;
    }
    static_assert(kLevelPer == 4, "marks are read four at a time");
    const unsigned marks = reinterpret_cast<const unsigned *>(L.mark)[t];
    // rows are counted up to `most` (below 2^31: two capped counts add up in 32 bits)
    unsigned cnt = 0, sum = 0;
#pragma unroll
    for (int k = 0; k < kLevelPer; k++)
        if (((marks >> (8 * k)) & 1u) && ((good >> k) & 1u)) {
            cnt++;
            sum = min(sum + (unsigned)rows[k], (unsigned)most);
        }
    unsigned ci = cnt, si = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, ci, d), z = __shfl_up_sync(0xFFFFFFFFu, si, d);
        if (lane >= d) ci += y, si = min(si + z, (unsigned)most);
    }
    if (lane == 31) L.warp_sum[0][warp] = ci, L.warp_sum[1][warp] = si;
    // exclusive within the warp, from the lane before
    unsigned at = __shfl_up_sync(0xFFFFFFFFu, ci, 1), row = __shfl_up_sync(0xFFFFFFFFu, si, 1);
    if (lane == 0) at = row = 0;
    __syncthreads();
    for (int w = 0; w < warp; w++) {
        at += L.warp_sum[0][w];
        row = min(row + L.warp_sum[1][w], (unsigned)most);
    }
    // The listed runs are those up to the first that reaches `most` rows (the
    // capped sums of later ones say nothing); the chain goes on after the last.
#pragma unroll
    for (int k = 0; k < kLevelPer; k++) {
        const int i = t * kLevelPer + k;
        if (!((marks >> (8 * k)) & 1u) || !((good >> k) & 1u)) continue;
        if (row < (unsigned)most) {
            L.run[at] = LevelRun{row0 + (int)row, bits[k]};
            atomicMax(&L.nruns, (int)at + 1);
            atomicMax(&L.row1, row0 + (int)min(row + (unsigned)rows[k], (unsigned)most));
            atomicMax(&L.next, L.p + i + size[k]);
        }
        at++;
        row = min(row + (unsigned)rows[k], (unsigned)most);
    }
    __syncthreads();
    return L.nruns > 0;
}
// The levels of page rows j .. j + 8 (those below n), a bit each.
__device__ __forceinline__ unsigned eight_levels(const Levels &L, int j, int n, const uint8_t *page) {
    const LevelRun *runs = L.run;
    const int nruns = L.nruns;
    int lo = 0, hi = nruns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (runs[mid].first <= j) lo = mid;
        else hi = mid - 1;
    }
    unsigned out = 0;
    const int j1 = min(j + 8, n);
    for (int row = j; row < j1; lo++) {
        const LevelRun r = runs[lo];
        const int end = min(lo + 1 < nruns ? runs[lo + 1].first : n, j1);
        const unsigned mask = (1u << (end - row)) - 1u;
        unsigned v = r.bits & 1u ? mask : 0u;
        if (r.bits < kLevelRle) {
            const uint32_t bit = r.bits + (uint32_t)(row - r.first);
            const int32_t byte = (int32_t)(bit >> 3);
            const unsigned sh = bit & 7;
            v = page[byte] >> sh;
            if ((int)sh + end - row > 8) v |= (unsigned)page[byte + 1] << (8 - sh);
            v &= mask;
        }
        out |= v << (row - j);
        row = end;
    }
    return out;
}

__device__ __forceinline__ void bitmap_or(uint32_t *words, int64_t row, unsigned bits32) {
    // bits32: 32 consecutive rows starting at `row`
    if (!bits32) return;
    const int64_t w = row >> 5;
    const int s = (int)(row & 31);
    atomicOr(words + w, bits32 << s);
    if (s) {
        const unsigned hi = bits32 >> (32 - s);
        if (hi) atomicOr(words + w + 1, hi);
    }
}

// The PLAIN BYTE_ARRAY values of a dictionary page or a data page, one warp
// (lane 0) per page: each value's start in the staging buffer and its length
// into the table, every length checked against the page.
__global__ void __launch_bounds__(32) ba_walk_kernel(const WalkDev *items, const uint8_t *staged, int max_def,
                                                     long long *starts, int32_t *lens, int32_t *walked,
                                                     uint32_t *status) {
    if (threadIdx.x != 0) return;
    const WalkDev W = items[blockIdx.x];
    const uint8_t *page = staged + W.staged;
    auto le32 = [&](int64_t at) {
        return (uint32_t)page[at] | ((uint32_t)page[at + 1] << 8) | ((uint32_t)page[at + 2] << 16) |
               ((uint32_t)page[at + 3] << 24);
    };
    int64_t pos = 0;
    const int64_t end = W.usize;
    if (W.kind == 1 && max_def > 0) {  // v1: the levels' 4-byte length, then the levels
        if (end < 4 || (int64_t)le32(0) > end - 4) {
            atomicOr(status, ST_CORRUPT);
            return;
        }
        pos = 4 + (int64_t)le32(0);
    } else if (W.kind == 2) {
        pos = W.def_len;
    }
    int32_t n = 0;
    while (pos < end && n < W.limit) {
        if (end - pos < 4) break;
        const int64_t len = le32(pos);
        if (len > end - pos - 4) break;
        starts[W.base + n] = (long long)(W.staged + pos + 4);
        lens[W.base + n] = (int32_t)len;
        pos += 4 + len;
        n++;
    }
    if (W.page >= 0) walked[W.page] = n;
    if (pos != end || (W.page < 0 && n != W.limit)) atomicOr(status, ST_CORRUPT);
}

__global__ void __launch_bounds__(kDecodeThreads) page_decode_kernel(DecodeArgs A) {
    constexpr int U = kTile / kDecodeThreads;
    __shared__ Hybrid s_idx;
    __shared__ Levels s_def;  // the definition levels' runs
    __shared__ Run s_runs[kTile];  // a tile's runs of indices
    __shared__ uint8_t s_bits[kTile / 8];
    __shared__ int s_ni, s_ok;
    __shared__ int s_warp[kDecodeThreads / 32];
    __shared__ const uint8_t *s_values;
    __shared__ int64_t s_values_len;
    const PageDev P = A.pages[blockIdx.x];
    const uint8_t *page = A.staged + P.staged;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_ok = 1;
        const uint8_t *p = page, *end = page + P.usize;
        if (A.max_def > 0) {
            int64_t len;
            if (P.v2) {
                len = P.def_len;
            } else {
                if (end - p < 4) s_ok = 0;
                len = s_ok ? (int64_t)((uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) |
                                       ((uint32_t)p[3] << 24))
                           : 0;
                p += s_ok ? 4 : 0;
            }
            if (len < 0 || len > end - p) s_ok = 0;
            if (s_ok) {
                s_def.next = (int32_t)(p - page);
                s_def.end = (int32_t)(p - page + len);
                s_def.row1 = 0;
                p += len;
            }
        } else if (P.v2) {
            p += P.def_len;  // no levels are stored for a required column (def_len 0)
        }
        if (s_ok && P.dict) {
            if (p >= end) {
                // no index bytes: only an all-NULL page may have none (a run is never asked for)
                s_idx = Hybrid{P.usize, P.usize, 0, 0, 0, 0, 0, 0, 0};
            } else {
                const int bw = *p++;
                if (bw > 32) s_ok = 0;
                s_idx = Hybrid{(int32_t)(p - page), P.usize, bw, 0, 0, 0, 0, 0, 0};
            }
        }
        s_values = p;
        s_values_len = end - p;
    }
    __syncthreads();
    if (!s_ok) {
        if (tid == 0) atomicOr(A.status, ST_CORRUPT);
        return;
    }
    const bool aligned = ((uintptr_t)s_values & (uintptr_t)(A.pwidth - 1)) == 0;
    int64_t nn_base = 0;  // non-NULL values before this tile
    unsigned npass = 0;   // rows of this thread's words that pass the filter
    // Tiles of kTile rows; one ends where the listed level runs do.
    for (int t0 = 0, n; t0 < P.nvalues; t0 += n) {
        n = min(kTile, P.nvalues - t0);
        if (A.max_def > 0) {
            // the same on every thread: list_levels ends with a barrier
            bool ok = true;
            while (ok && s_def.row1 <= t0) ok = list_levels(s_def, page, t0, P.nvalues - t0);
            if (!ok) {
                if (tid == 0) atomicOr(A.status, ST_CORRUPT);
                break;
            }
            n = min(n, s_def.row1 - t0);
            if (tid * 8 < n) s_bits[tid] = (uint8_t)eight_levels(s_def, t0 + tid * 8, t0 + n, page);
            __syncthreads();
        }
        bool v[U];
        int cnt = 0;
        static_assert(U == 4, "a thread takes half a byte of levels");
        const unsigned mine = A.max_def > 0 ? s_bits[tid >> 1] >> (4 * (tid & 1)) : 0xFu;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = tid * U + u;  // consecutive rows per thread: ranks by a scan of counts
            v[u] = i < n && ((mine >> u) & 1u);
            cnt += v[u];
        }
        // block exclusive scan of cnt
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int wbase = 0, total = 0;
        for (int w = 0; w < kDecodeThreads / 32; w++) {
            if (w < warp) wbase += s_warp[w];
            total += s_warp[w];
        }
        int rank = wbase + incl - cnt;
        if (tid == 0 && P.dict && total > 0 && !emit_runs(s_idx, page, total, s_runs, s_ni)) s_ok = 0;
        __syncthreads();
        if (!s_ok) break;
        // The rows' dependent reads (index, entry, the filter's answer) in steps
        // over all U rows, so that each step's reads are in flight together.
        unsigned vbits = 0, pbits = 0;
        const int64_t row = P.row0 + t0 + tid * U;
        uint32_t idx[U];
        int64_t rk[U];  // the row's rank among the page's non-NULL rows
#pragma unroll
        for (int u = 0; u < U; u++) {
            rk[u] = nn_base + rank;
            rank += v[u];
            idx[u] = v[u] && P.dict ? run_value(s_runs, s_ni, (int)(rk[u] - nn_base), s_idx.bw, page) : 0u;
        }
        bool bad = false;
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!v[u]) continue;
            if (P.dict ? (int64_t)idx[u] >= A.dict_n
                       : A.out_kind == OUT_REF ? rk[u] >= A.walked[blockIdx.x] : (rk[u] + 1) * A.pwidth > s_values_len) {
                bad = true;
                v[u] = false;
            }
        }
        if (bad) atomicOr(A.status, ST_CORRUPT);
        if (A.out_kind == OUT_REF) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if (tid * U + u < n)
                    A.ref[row + u] = !v[u] ? -1ll : P.dict ? (long long)idx[u] : (long long)(A.dict_n + P.row0 + rk[u]);
        } else {
            uint64_t raw[U];
            bool pass[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                raw[u] = 0;
                pass[u] = A.f.nulls_pass != 0;
                if (!v[u]) continue;
                const uint8_t *src = P.dict ? A.dict + (int64_t)idx[u] * A.pwidth : s_values + rk[u] * A.pwidth;
                if (A.pwidth == 4) {
                    uint32_t w;
                    if (P.dict || aligned) w = *reinterpret_cast<const uint32_t *>(src);
                    else memcpy(&w, src, 4);
                    raw[u] = w;
                } else {
                    uint64_t w;
                    if (P.dict || aligned) w = *reinterpret_cast<const uint64_t *>(src);
                    else memcpy(&w, src, 8);
                    raw[u] = w;
                }
                if (A.has_filter && P.dict && A.dict_pass) pass[u] = A.dict_pass[idx[u]] != 0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (tid * U + u >= n) continue;
                const int64_t ival = A.pwidth == 4 ? (int64_t)(int32_t)raw[u] : (int64_t)raw[u];
                if (v[u]) {
                    vbits |= 1u << u;
                    if (A.has_filter && !(P.dict && A.dict_pass)) pass[u] = filter_pass(A.f, ival);
                }
                if (A.has_filter && pass[u]) pbits |= 1u << u;
                if (A.out_kind == OUT_SAME) {
                    if (A.pwidth == 4) static_cast<uint32_t *>(A.out)[row + u] = (uint32_t)raw[u];
                    else static_cast<uint64_t *>(A.out)[row + u] = raw[u];
                } else if (A.out_kind == OUT_I32_TO_I64) {
                    static_cast<int64_t *>(A.out)[row + u] = v[u] ? ival : 0;
                } else {
                    static_cast<int64_t *>(A.out)[2 * (row + u)] = v[u] ? ival : 0;
                    static_cast<int64_t *>(A.out)[2 * (row + u) + 1] = v[u] && ival < 0 ? -1 : 0;
                }
            }
        }
        // U consecutive rows per thread: 8 threads hold 32 consecutive rows
        static_assert(U == 4, "bitmap packing assumes 4 rows per thread");
        const int sub = lane & 7;
        unsigned vw = vbits << (4 * sub), pw = pbits << (4 * sub);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            vw |= __shfl_xor_sync(0xFFFFFFFFu, vw, o);
            pw |= __shfl_xor_sync(0xFFFFFFFFu, pw, o);
        }
        if (sub == 0) {
            if (A.valid) bitmap_or(A.valid, row, vw);
            if (A.has_filter) {
                bitmap_or(A.pass, row, pw);
                npass += __popc(pw);
            }
        }
        nn_base += total;
        __syncthreads();
    }
    if (!s_ok && tid == 0) atomicOr(A.status, ST_CORRUPT);
    if (A.has_filter) {  // one update of the chunk's count per warp and page
        npass = __reduce_add_sync(0xFFFFFFFFu, npass);
        if (lane == 0 && npass) atomicAdd(A.counts, (unsigned long long)npass);
    }
}

}  // namespace

// ---- the operator ----------------------------------------------------------------------------
namespace {
// The fragments of one page's Snappy stream. A page's elements are a chain
// (each starts where the last ended), so one CTA decoding a large page is
// slow; but a Snappy compressor codes its input in independent blocks of
// 64 KiB (Google's snappy::Compress), so the stream splits into runs of
// elements whose back-references stay inside the run. The host walks the
// tags (skipping literal bytes), starts a fragment at the first element
// boundary after each 64 KiB of output, and merges a fragment back into the
// one before whenever a back-reference reaches behind its start, so every
// fragment decodes alone whatever compressor wrote the stream. The host
// copies no data: the CTAs decompress every byte. A stream that does not
// parse stays one fragment, whose CTA reports it. A page that turns out to
// have many short elements (more than kWalkElements) and fits kBigBytes goes
// to the big-page kernels instead (true is returned, `big` filled): on those
// the walk costs the host more than the kernels take.
constexpr int64_t kFragBytes = 65536;
constexpr int64_t kBigBytes = 16 << 20;
constexpr int kWalkElements = 4096;
bool plan_fragments(const uint8_t *chunk, const StageDev &s, std::vector<FragDev> &out, bool allow_big, BigPage &big) {
    const uint8_t *p = chunk + s.src + s.raw;
    const int64_t slen = (int64_t)s.csize - s.raw, dlen = (int64_t)s.usize - s.raw;
    if (slen == 0) {
        if (dlen != 0) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page: an empty Snappy stream");
        return false;
    }
    int64_t ip = 0;
    uint64_t n = 0;
    for (int sh = 0;; sh += 7) {
        if (ip >= slen || sh > 28) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page: the Snappy length");
        const uint8_t b = p[ip++];
        n |= (uint64_t)(b & 0x7F) << sh;
        if (!(b & 0x80)) break;
    }
    if ((int64_t)n != dlen) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page: the Snappy length");
    std::vector<std::pair<int64_t, int64_t>> starts{{ip, 0}};  // (stream, output) offsets of each fragment
    if (dlen > 2 * kFragBytes) {
        int64_t op = 0;
        const int64_t ip0 = ip;
        for (int64_t elements = 0; ip < slen; elements++) {
            if (elements == kWalkElements && allow_big && dlen <= kBigBytes && slen <= kBigBytes) {
                big = BigPage{};
                big.src = s.src + s.raw + ip0;
                big.dst = s.dst + s.raw;
                big.slen = (int32_t)(slen - ip0);
                big.dlen = (int32_t)dlen;
                big.nwin = (int32_t)ceil_div(big.slen, kSnappyWin);
                big.ntile = (int32_t)ceil_div(big.dlen, kSnappyOut);
                return true;
            }
            const uint8_t tag = p[ip++];
            int64_t len, off = 0;
            const int kind = tag & 3;
            if (kind == 0) {
                len = tag >> 2;
                if (len >= 60) {
                    const int nb = (int)len - 59;
                    if (ip + nb > slen) break;
                    len = 0;
                    for (int i = 0; i < nb; i++) len |= (int64_t)p[ip + i] << (8 * i);
                    ip += nb;
                }
                len += 1;
                if (ip + len > slen) break;
                ip += len;
            } else {
                const int nb = kind == 1 ? 1 : kind == 2 ? 2 : 4;
                if (ip + nb > slen) break;
                if (kind == 1) {
                    len = 4 + ((tag >> 2) & 7);
                    off = ((int64_t)(tag >> 5) << 8) | p[ip];
                } else {
                    len = 1 + (tag >> 2);
                    for (int i = 0; i < nb; i++) off |= (int64_t)p[ip + i] << (8 * i);
                }
                ip += nb;
                if (off <= 0 || off > op) break;
                while (starts.size() > 1 && op - off < starts.back().second) starts.pop_back();
            }
            op += len;
            if (op > dlen) break;
            if (op - starts.back().second >= kFragBytes && ip < slen) starts.push_back({ip, op});
        }
    }
    for (size_t k = 0; k < starts.size(); k++) {
        const int64_t ip0 = starts[k].first, op0 = starts[k].second;
        const int64_t ip1 = k + 1 < starts.size() ? starts[k + 1].first : slen;
        const int64_t op1 = k + 1 < starts.size() ? starts[k + 1].second : dlen;
        out.push_back(FragDev{s.src + s.raw + ip0, s.dst + s.raw + op0, (int32_t)(ip1 - ip0), (int32_t)(op1 - op0)});
    }
    return false;
}

// The pages that the big-page kernels decode, and their tables.
struct BigPlan {
    std::vector<BigPage> pages;
    std::vector<int32_t> win_page, tile_page;
    int64_t exits = 0, from = 0;
    DBuf dpages, dwin, dtile, dexit, dentry, dfrom;

    void add(BigPage p) {
        p.win0 = (int32_t)win_page.size();
        p.tile0 = (int32_t)tile_page.size();
        p.exit0 = exits;
        p.from0 = from;
        win_page.insert(win_page.end(), (size_t)p.nwin, (int32_t)pages.size());
        tile_page.insert(tile_page.end(), (size_t)p.ntile, (int32_t)pages.size());
        exits += p.slen;
        from += p.dlen;
        pages.push_back(p);
    }
    void alloc(Runtime *rt) {
        dpages = DBuf(rt, pages.size() * sizeof(BigPage));
        dwin = DBuf(rt, win_page.size() * 4);
        dtile = DBuf(rt, tile_page.size() * 4);
        dexit = DBuf(rt, (size_t)exits * sizeof(BigExit));
        dentry = DBuf(rt, win_page.size() * sizeof(BigEntry));
        dfrom = DBuf(rt, (size_t)from * 4);
        KRV_CUDA(cudaMemcpyAsync(dpages.get(), pages.data(), pages.size() * sizeof(BigPage), cudaMemcpyHostToDevice, rt->stream));
        KRV_CUDA(cudaMemcpyAsync(dwin.get(), win_page.data(), win_page.size() * 4, cudaMemcpyHostToDevice, rt->stream));
        KRV_CUDA(cudaMemcpyAsync(dtile.get(), tile_page.data(), tile_page.size() * 4, cudaMemcpyHostToDevice, rt->stream));
        KRV_CUDA(cudaMemsetAsync(dfrom.get(), 0xFF, (size_t)from * 4, rt->stream));
    }
    void launch(Runtime *rt, const uint8_t *chunk, uint8_t *staged) {
        const BigPage *P = dpages.as<BigPage>();
        const unsigned nwin = (unsigned)win_page.size(), ntile = (unsigned)tile_page.size();
        KRV_CUDA(cudaFuncSetAttribute(big_link_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BigLinkSmem)));
        big_link_kernel<<<nwin, kBigThreads, sizeof(BigLinkSmem), rt->stream>>>(P, dwin.as<int32_t>(), chunk, dexit.as<BigExit>());
        big_chase_kernel<<<(unsigned)pages.size(), 256, 0, rt->stream>>>(P, dexit.as<BigExit>(), dentry.as<BigEntry>(),
                                                                        status_word(rt));
        big_source_kernel<<<nwin, kBigThreads, 0, rt->stream>>>(P, dwin.as<int32_t>(), chunk, dentry.as<BigEntry>(), staged,
                                                                dfrom.as<int32_t>(), status_word(rt));
        KRV_CUDA(cudaFuncSetAttribute(big_jump_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSnappyOut * 4));
        big_jump_kernel<<<ntile, kBigThreads, kSnappyOut * 4, rt->stream>>>(P, dtile.as<int32_t>(), dfrom.as<int32_t>());
        big_copy_kernel<<<dim3(ntile, 8), 256, 0, rt->stream>>>(P, dtile.as<int32_t>(), dfrom.as<int32_t>(), staged);
        rt->launches += 5;
        check_launch("big-page Snappy kernels");
    }
};
}  // namespace

// `device_tables`: large pages of short elements may take the big-page kernels;
// left true when some did.
static ParquetChunk decode_chunk(Runtime *rt, const uint8_t *chunk, int64_t bytes, const krv_parquet_column &col,
                                 const KeyFilterImpl *filter, bool &device_tables) {
    const bool allow_big = device_tables;
    device_tables = false;
    if (!chunk && bytes > 0) fail(KRV_INVALID_ARGUMENT, "chunk is NULL");
    if (bytes < 0) fail(KRV_INVALID_ARGUMENT, "chunk_bytes < 0");
    if (col.num_values < 0) fail(KRV_INVALID_ARGUMENT, "num_values < 0");
    if (col.max_def_level < 0 || col.max_def_level > 1)
        fail(KRV_UNSUPPORTED, "the GPU Parquet decoder takes flat columns (max definition level 0 or 1)");
    if (col.codec != KRV_PQ_UNCOMPRESSED && col.codec != KRV_PQ_SNAPPY)
        fail(KRV_UNSUPPORTED, "Parquet codec " + std::to_string(col.codec) + " on the GPU decoder (UNCOMPRESSED, SNAPPY)");
    int pwidth = 0;  // 0: BYTE_ARRAY (a 4-byte length before each value)
    if (col.physical_type == KRV_PQ_INT32) pwidth = 4;
    else if (col.physical_type == KRV_PQ_INT64 || col.physical_type == KRV_PQ_DOUBLE) pwidth = 8;
    else if (col.physical_type != KRV_PQ_BYTE_ARRAY)
        fail(KRV_UNSUPPORTED, "Parquet physical type " + std::to_string(col.physical_type) + " on the GPU decoder");
    const bool var = col.physical_type == KRV_PQ_BYTE_ARRAY;
    if (!col.format) fail(KRV_INVALID_ARGUMENT, "format is NULL");
    const DType out_t = parse_format(col.format);
    int out_kind = -1;
    if (col.physical_type == KRV_PQ_INT32) {
        if (out_t.id == Type::I32 || out_t.id == Type::Date32) out_kind = OUT_SAME;
        else if (out_t.id == Type::I64 || out_t.id == Type::Dec64) out_kind = OUT_I32_TO_I64;
        else if (out_t.id == Type::Dec128) out_kind = OUT_TO_DEC128;
    } else if (col.physical_type == KRV_PQ_INT64) {
        if (out_t.id == Type::I64 || out_t.id == Type::Dec64) out_kind = OUT_SAME;
        else if (out_t.id == Type::Dec128) out_kind = OUT_TO_DEC128;
    } else if (col.physical_type == KRV_PQ_DOUBLE) {
        if (out_t.id == Type::F64) out_kind = OUT_SAME;
    } else if (out_t.id == Type::Utf8 || out_t.id == Type::Binary) {
        out_kind = OUT_REF;
    }
    if (out_kind < 0) fail(KRV_UNSUPPORTED, std::string("Parquet column decoded as ") + col.format);
    const bool is_int = col.physical_type == KRV_PQ_INT32 || col.physical_type == KRV_PQ_INT64;
    if (filter && !is_int) fail(KRV_UNSUPPORTED, "key filters test integer columns");

    // The page headers, on the host.
    std::vector<StageDev> stages;
    std::vector<PageDev> pages;
    int64_t staged_bytes = 0, rows = 0;
    int dict_stage = -1;
    int64_t dict_n = 0;
    bool all_dict = true;  // every data page is dictionary encoded (dict_probe.rs `all_dictionary`)
    Thrift t{chunk, chunk + bytes};
    while (t.p < t.end && rows < col.num_values) {
        const PageHdr h = parse_page_header(t);
        const int64_t at = t.p - chunk;
        if (h.csize < 0 || h.usize < 0 || h.csize > t.end - t.p)
            fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page header: page sizes");
        if (h.usize > (1 << 28)) fail(KRV_UNSUPPORTED, "Parquet pages of more than 256 MiB on the GPU decoder");
        t.p += h.csize;
        if (h.type == kPageIndex) continue;
        if (h.type != kPageData && h.type != kPageDataV2 && h.type != kPageDict)
            fail(KRV_UNSUPPORTED, "Parquet page type " + std::to_string(h.type));
        if (h.nvalues < 0) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page header: num_values");
        StageDev s{};
        s.src = at;
        s.dst = staged_bytes;
        s.csize = h.csize;
        s.usize = h.usize;
        s.snappy = col.codec == KRV_PQ_SNAPPY && (h.type != kPageDataV2 || h.compressed);
        if (h.type == kPageDataV2) {
            if (h.rep_len != 0) fail(KRV_UNSUPPORTED, "repeated Parquet columns on the GPU decoder");
            if (h.def_len < 0 || h.def_len > h.csize || h.def_len > h.usize)
                fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page header: level lengths");
            if (col.max_def_level == 0 && h.def_len != 0)
                fail(KRV_INVALID_ARGUMENT, "definition levels in a required column");
            s.raw = h.def_len;
        }
        if (!s.snappy && h.csize != h.usize) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page: sizes of an uncompressed page differ");
        if (h.type == kPageDict) {
            if (dict_stage >= 0 || !pages.empty()) fail(KRV_INVALID_ARGUMENT, "a dictionary page after the first page");
            if (h.encoding != kEncPlain && h.encoding != kEncPlainDict)
                fail(KRV_UNSUPPORTED, "Parquet dictionary encoding " + std::to_string(h.encoding));
            if ((int64_t)h.nvalues * (var ? 4 : pwidth) > h.usize) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet dictionary page");
            dict_stage = (int)stages.size();
            dict_n = h.nvalues;
        } else {
            PageDev p{};
            p.staged = staged_bytes;
            p.row0 = rows;
            p.usize = h.usize;
            p.nvalues = h.nvalues;
            p.v2 = h.type == kPageDataV2;
            p.def_len = h.def_len;
            if (h.encoding == kEncPlainDict || h.encoding == kEncRleDict) {
                if (dict_stage < 0) fail(KRV_INVALID_ARGUMENT, "a dictionary-encoded Parquet page without a dictionary");
                p.dict = 1;
            } else if (h.encoding != kEncPlain) {
                fail(KRV_UNSUPPORTED, "Parquet encoding " + std::to_string(h.encoding) + " on the GPU decoder");
            } else {
                all_dict = false;
            }
            if (!p.v2 && col.max_def_level > 0 && h.def_encoding != kEncRle)
                fail(KRV_UNSUPPORTED, "Parquet definition level encoding " + std::to_string(h.def_encoding));
            pages.push_back(p);
            rows += h.nvalues;
        }
        stages.push_back(s);
        staged_bytes += ((int64_t)h.usize + 15) / 16 * 16;
    }
    if (rows != col.num_values)
        fail(KRV_INVALID_ARGUMENT, "the chunk's data pages hold " + std::to_string(rows) + " values, not " +
                                       std::to_string(col.num_values));

    ParquetChunk r;
    r.info.rows = rows;
    r.info.pages = (int64_t)pages.size();
    r.info.dictionary_entries = dict_n;
    r.info.dictionary_passing = -1;
    r.info.passing_rows = -1;
    const std::string name = col.name ? col.name : "";
    DevCol out = var ? DevCol{} : make_col(rt, out_t, rows, col.max_def_level > 0, name);
    r.batch.rows = rows;
    DevCol pass;
    if (filter) {
        // bit-packed, written as 32-bit words: room for the last word
        pass.type = DType{Type::Bool, 0, 0};
        pass.length = rows;
        pass.nullable = false;
        pass.name = "pass";
        pass.hold_data = std::make_shared<DBuf>(rt, (size_t)ceil_div(rows, 32) * 4 + 8);
        pass.data = pass.hold_data->get();
        KRV_CUDA(cudaMemsetAsync(pass.hold_data->get(), 0, pass.hold_data->bytes(), rt->stream));
    }
    if (out.valid) KRV_CUDA(cudaMemsetAsync(const_cast<uint8_t *>(out.valid), 0, out.hold_valid->bytes(), rt->stream));
    if (rows > 0) {
        DBuf dchunk(rt, (size_t)bytes);
        KRV_CUDA(cudaMemcpyAsync(dchunk.get(), chunk, (size_t)bytes, cudaMemcpyHostToDevice, rt->stream));
        DBuf staged(rt, (size_t)staged_bytes + 16);  // indices are read in whole words, past the last page too
        DBuf dstages(rt, stages.size() * sizeof(StageDev));
        DBuf dpages(rt, std::max<size_t>(pages.size(), 1) * sizeof(PageDev));
        DBuf counts(rt, 16);
        std::vector<FragDev> frags;
        BigPlan big;
        BigPage bp;
        for (const StageDev &st : stages)
            if (st.snappy && plan_fragments(chunk, st, frags, allow_big, bp)) big.add(bp);
        if (!big.pages.empty()) {
            try {
                big.alloc(rt);
            } catch (const Error &e) {
                if (e.code != KRV_NEED_MEMORY) throw;
                // no room for the tables (8 B a stream byte, 4 B an output byte): walk those pages after all
                big = BigPlan{};
                frags.clear();
                for (const StageDev &st : stages)
                    if (st.snappy) plan_fragments(chunk, st, frags, false, bp);
            }
        }
        device_tables = !big.pages.empty();
        DBuf dfrags(rt, std::max<size_t>(frags.size(), 1) * sizeof(FragDev));
        if (!frags.empty())
            KRV_CUDA(cudaMemcpyAsync(dfrags.get(), frags.data(), frags.size() * sizeof(FragDev), cudaMemcpyHostToDevice,
                                     rt->stream));
        KRV_CUDA(cudaMemcpyAsync(dstages.get(), stages.data(), stages.size() * sizeof(StageDev), cudaMemcpyHostToDevice,
                                 rt->stream));
        KRV_CUDA(cudaMemcpyAsync(dpages.get(), pages.data(), pages.size() * sizeof(PageDev), cudaMemcpyHostToDevice,
                                 rt->stream));
        KRV_CUDA(cudaMemsetAsync(counts.get(), 0, 16, rt->stream));
        clear_status(rt);
        stage_kernel<<<(unsigned)stages.size(), kStageThreads, 0, rt->stream>>>(
            dstages.as<StageDev>(), dchunk.as<uint8_t>(), staged.as<uint8_t>());
        rt->launches++;
        check_launch("stage_kernel");
        if (col.codec == KRV_PQ_SNAPPY) {
            static bool smem_set[64] = {};  // the kernel's attribute, set once per device
            int dev = 0;
            KRV_CUDA(cudaGetDevice(&dev));
            if (dev < 0 || dev >= 64 || !smem_set[dev]) {
                KRV_CUDA(cudaFuncSetAttribute(snappy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)sizeof(SnappySmem)));
                if (dev >= 0 && dev < 64) smem_set[dev] = true;
            }
            if (!frags.empty()) {
                snappy_kernel<<<(unsigned)frags.size(), kSnappyThreads, sizeof(SnappySmem), rt->stream>>>(
                    dfrags.as<FragDev>(), dchunk.as<uint8_t>(), staged.as<uint8_t>(), status_word(rt));
                rt->launches++;
                check_launch("snappy_kernel");
            }
            if (!big.pages.empty()) big.launch(rt, dchunk.as<uint8_t>(), staged.as<uint8_t>());
        }
        DecodeArgs A{};
        A.pages = dpages.as<PageDev>();
        A.staged = staged.as<uint8_t>();
        A.max_def = col.max_def_level;
        A.pwidth = pwidth;
        A.out_kind = out_kind;
        A.is_int = is_int;
        A.out = const_cast<void *>(out.data);
        A.valid = out.valid ? reinterpret_cast<uint32_t *>(const_cast<uint8_t *>(out.valid)) : nullptr;
        A.status = status_word(rt);
        A.counts = counts.as<unsigned long long>();
        DBuf dict_pass;
        if (dict_stage >= 0) {
            A.dict = staged.as<uint8_t>() + stages[dict_stage].dst;
            A.dict_n = dict_n;
        }
        if (filter) {
            A.has_filter = 1;
            A.f = key_filter_dev(*filter);
            A.pass = reinterpret_cast<uint32_t *>(const_cast<void *>(pass.data));
            if (dict_stage >= 0 && dict_n > 0) {
                dict_pass = DBuf(rt, (size_t)dict_n);
                dict_filter_kernel<<<grid_for(rt, dict_n, 256, 4), 256, 0, rt->stream>>>(
                    A.f, A.dict, dict_n, pwidth, dict_pass.as<uint8_t>(), counts.as<unsigned long long>() + 1);
                rt->launches++;
                check_launch("dict_filter_kernel");
                A.dict_pass = dict_pass.as<uint8_t>();
            }
        } else {
            A.f.nulls_pass = 1;
        }
        // BYTE_ARRAY: the (start, length) table of the dictionary's entries,
        // then of every PLAIN page's values at the page's first row; each
        // row's reference into it.
        DBuf vstarts, vlens, walked, refs, dwalk;
        if (var) {
            const int64_t slots = dict_n + rows;
            vstarts = DBuf(rt, (size_t)std::max<int64_t>(slots, 1) * 8);
            vlens = DBuf(rt, (size_t)std::max<int64_t>(slots, 1) * 4);
            walked = DBuf(rt, std::max<size_t>(pages.size(), 1) * 4);
            refs = DBuf(rt, (size_t)rows * 8);
            KRV_CUDA(cudaMemsetAsync(walked.get(), 0, walked.bytes(), rt->stream));
            std::vector<WalkDev> items;
            if (dict_stage >= 0 && dict_n > 0)
                items.push_back(WalkDev{stages[dict_stage].dst, 0, stages[dict_stage].usize, 0, 0, (int32_t)dict_n, -1, 0});
            for (size_t i = 0; i < pages.size(); i++)
                if (!pages[i].dict)
                    items.push_back(WalkDev{pages[i].staged, dict_n + pages[i].row0, pages[i].usize, pages[i].v2 ? 2 : 1,
                                            pages[i].def_len, pages[i].nvalues, (int32_t)i, 0});
            if (!items.empty()) {
                dwalk = DBuf(rt, items.size() * sizeof(WalkDev));
                KRV_CUDA(cudaMemcpyAsync(dwalk.get(), items.data(), items.size() * sizeof(WalkDev),
                                         cudaMemcpyHostToDevice, rt->stream));
                ba_walk_kernel<<<(unsigned)items.size(), 32, 0, rt->stream>>>(
                    dwalk.as<WalkDev>(), staged.as<uint8_t>(), col.max_def_level, vstarts.as<long long>(),
                    vlens.as<int32_t>(), walked.as<int32_t>(), status_word(rt));
                rt->launches++;
                check_launch("ba_walk_kernel");
            }
            A.ref = refs.as<long long>();
            A.walked = walked.as<int32_t>();
            A.valid = nullptr;  // the gather writes the validity
        }
        if (!pages.empty()) {
            page_decode_kernel<<<(unsigned)pages.size(), kDecodeThreads, 0, rt->stream>>>(A);
            rt->launches++;
            check_launch("page_decode_kernel");
        }
        unsigned long long c[2];
        read_device(rt, counts.get(), 16, c);
        const uint32_t st = take_status(rt);
        if (st & ST_CORRUPT) fail(KRV_INVALID_ARGUMENT, "corrupt Parquet page: its bytes do not decode");
        if (st) fail(KRV_CUDA_ERROR, "Parquet decode status " + std::to_string(st));
        if (var) {
            const VarSrc src{nullptr, vstarts.as<long long>(), vlens.as<int32_t>(), staged.as<uint8_t>(), nullptr, 0};
            out = var_gather(rt, src, refs.as<long long>(), rows, out_t, col.max_def_level > 0, name);
        }
        if (filter) {
            r.info.passing_rows = (int64_t)c[0];
            // the dictionary decides for the chunk only when every data page uses it
            if (dict_stage >= 0 && all_dict) r.info.dictionary_passing = (int64_t)c[1];
        }
    } else {
        if (filter) r.info.passing_rows = 0;
        if (var) out = var_gather(rt, VarSrc{}, nullptr, 0, out_t, col.max_def_level > 0, name);
    }
    r.batch.cols.push_back(out);
    if (filter) r.batch.cols.push_back(pass);
    return r;
}

ParquetChunk decode_parquet_chunk(Runtime *rt, const uint8_t *chunk, int64_t bytes, const krv_parquet_column &col,
                                  const KeyFilterImpl *filter) {
    bool tables = true;
    try {
        return decode_chunk(rt, chunk, bytes, col, filter, tables);
    } catch (const Error &e) {
        // The big-page kernels' tables are a convenience: a chunk that does not
        // fit beside them is decoded without.
        if (e.code != KRV_NEED_MEMORY || !tables) throw;
    }
    tables = false;
    return decode_chunk(rt, chunk, bytes, col, filter, tables);
}

}  // namespace krv
