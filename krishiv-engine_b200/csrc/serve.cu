// serve.cu -- a request server for join + grouped aggregate queries:
//   SELECT t.g, SUM(p.x), COUNT(*) FROM probe p JOIN table t ON p.k = t.k GROUP BY t.g
// over build tables kept resident on the device, with requests admitted by an
// HBM budget and run in ticks.
//
// Batched mode. A tick is one CUDA graph of three or four kernels over
// descriptors uploaded before it in one copy: clear the accumulators of newly
// admitted requests; a probe + aggregate launch over a device work queue of
// (request, row range) items from every running request, CTAs taking items off
// an atomic cursor (a second launch when requests have some thousand groups);
// and compaction of the groups of the requests that end in the tick. A tick
// takes at most `tick_rows` probe rows, so a large request spans several
// ticks while requests that arrive meanwhile join the next one and finish
// early (continuous batching). Two ticks may be queued at once: the host
// forms and uploads the next while the device runs the current one.
// Aggregation runs in shared memory for requests with few groups (per-CTA
// 96-bit partial sums merged once per item) and in global memory otherwise.
// An online autotuner tries the candidate kernel shapes (block size, item
// rows, shared-memory group limit) on the first ticks and keeps the fastest.
//
// Plain mode runs each request through the operators one launch at a time:
// HashJoin probe (materialized (x, g) pairs), then HashAggregate.
//
// Reference semantics: HashJoin inner join (crates/krishiv-exec/src/join/
// mod.rs:1014) and HashAggregate SUM(int64) -> int64 with ANSI overflow,
// COUNT(*) (crates/krishiv-exec/src/aggregate/sink.rs:181); the operator
// protocol's NeedMemory for admission (crates/krishiv-exec/src/operator.rs:
// 314-330).
#include <algorithm>
#include <chrono>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "krv_device.cuh"
#include "limbs.h"
#include "ops.h"

namespace krv {

namespace {

constexpr uint32_t kNoRow = 0xFFFFFFFFu;
constexpr int kMaxTickRequests = 512;
constexpr int kMaxTickItems = 16384;
constexpr int kTickRowsPerThread = 4;  // in flight together
// Shared-memory aggregation: 16 bytes per group (see SmemGroups). The lookups
// of a step are thousands of scattered reads, each holding a line of L1 while it
// is on its way, and L1 is what shared memory leaves: so most requests run in
// CTAs that leave three quarters of it (32 KB in each of two CTAs of 512
// threads, or 16 KB in four of 256), and those with more groups, up to
// kMidGroups, in a launch of their own with one CTA of 512 threads per SM.
// Measured on B200, a tick of 38.5M rows of 24 requests with 10 to 68,000
// groups: 0.41 ms; 0.68 with 7168 groups in each of two CTAs for all, 0.58 with
// at most 2048 groups in shared memory, 0.45 with up to 12288 in the second
// launch.
constexpr int kSmemGroupBytes = 16;
constexpr int tick_smem_groups(int threads) { return threads == 256 ? 1024 : 2048; }
constexpr int kMidThreads = 512;
constexpr int kMidGroups = 7168;
// Requests of up to this many groups aggregate there however few rows an item
// has, or (the autotuner's other choice, 0) only where the rows pay for it, as
// all others do.
constexpr int kSmemGroupsAlways = 2048;
constexpr int kSmemRowsPerGroup = 4;
constexpr unsigned long long kGroupEmpty = 0x8000000000000000ull;

// How a resident table answers key -> group id:
//  - kDirect: unique keys over a span of at most 4 x rows: gid at key - lo;
//  - kRecords: unique keys: (key, gid) records at the join table's slot
//    positions, probed in the same order, one 16-byte read per step;
//  - kChains: duplicate keys: the join table's slots and newest-first chains.
enum Layout : int32_t { kDirect = 0, kRecords = 1, kChains = 2 };

struct Record {
    long long key;
    int32_t gid;   // -1: empty slot
    int32_t pad;
};

struct TableView {
    const unsigned long long *slots;
    uint64_t mask;
    const uint32_t *next;
    uint64_t seed;
    const long long *keys;
    const int32_t *gid;
    const Record *rec;       // kRecords
    const int32_t *direct;   // kDirect
    long long lo;            // kDirect: smallest key
    unsigned long long span; // kDirect: largest key - lo
    int32_t layout;
    int32_t pad;
};

// One running request, as the tick kernels see it.
struct ReqDev {
    const long long *k;
    const uint8_t *kvalid;
    int64_t kvoff;
    const long long *x;
    TableView t;
    unsigned long long *lo;  // per group: SUM (lo, hi) and COUNT(*)
    long long *hi;
    unsigned long long *cnt;
    const long long *gkeys;  // group value of each dense group id
    long long *out_g, *out_sum, *out_cnt;
    int32_t ngroups;
    int32_t use_smem;
    int32_t split;   // SUM = hi * 2^32 + lo (at most 2^32 rows join); else 128 bits
    int32_t copies;  // log2 of the copies of each group in shared memory
};
struct Item {
    int32_t req;
    int32_t pad;
    int64_t row0;
    int64_t rows;
};
struct TickHeader {
    unsigned long long cursor[2];  // of the two launches' work queues
    int32_t n_items[2], items_at[2];  // the items follow the tick's requests: index (in Items) from TickDev::items
    int32_t n_init, n_final;
};
struct Report {
    unsigned long long groups;
    unsigned int overflow;
    unsigned int pad;
};

// Device descriptor area of one tick slot.
struct TickDev {
    TickHeader *hdr;
    ReqDev *reqs;
    Item *items;
    int32_t *init;   // requests whose accumulators start at zero in this tick
    int32_t *final;  // requests that end in this tick
    Report *report;  // one per entry of `final`
};

// The lookups of U rows (`has`: those with a key), their first reads in flight
// together: from clamped addresses, without a branch before them.
template <int U>
__device__ __forceinline__ void table_heads(const TableView &t, const long long (&k)[U], unsigned has, uint32_t (&row)[U]) {
    uint32_t tag[U];
    uint64_t pos[U];
    unsigned long long first[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint64_t g = finalize(hash_word((uint64_t)k[u]), t.seed);
        tag[u] = slot_tag(g);
        pos[u] = g & t.mask;
        first[u] = __ldg(t.slots + pos[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        row[u] = kNoRow;
        if (!((has >> u) & 1u)) continue;
        unsigned long long s = first[u];
        for (uint64_t p = 0; p <= t.mask && s != 0; p++) {
            if (slot_matches(s, tag[u])) {
                const uint32_t o = slot_row(s);
                if (__ldg(t.keys + o) == k[u]) {
                    row[u] = o;
                    break;
                }
            }
            pos[u] = (pos[u] + 1) & t.mask;
            s = __ldg(t.slots + pos[u]);
        }
    }
}

template <int U>
__device__ __forceinline__ void record_gids(const TableView &t, const long long (&k)[U], unsigned has, int (&g)[U]) {
    uint64_t pos[U];
    longlong2 first[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        pos[u] = finalize(hash_word((uint64_t)k[u]), t.seed) & t.mask;
        first[u] = __ldg(reinterpret_cast<const longlong2 *>(t.rec + pos[u]));
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        g[u] = -1;
        if (!((has >> u) & 1u)) continue;
        longlong2 r = first[u];
        for (uint64_t p = 0; p <= t.mask; p++) {
            const int gid = (int)(int32_t)(r.y & 0xFFFFFFFFll);
            if (gid < 0) break;
            if (r.x == k[u]) {
                g[u] = gid;
                break;
            }
            pos[u] = (pos[u] + 1) & t.mask;
            r = __ldg(reinterpret_cast<const longlong2 *>(t.rec + pos[u]));
        }
    }
}

template <int U>
__device__ __forceinline__ void direct_gids(const TableView &t, const long long (&k)[U], unsigned has, int (&g)[U]) {
#pragma unroll
    for (int u = 0; u < U; u++) {
        const unsigned long long off = (unsigned long long)(k[u] - t.lo);
        g[u] = __ldg(t.direct + (off <= t.span ? off : 0ull));
    }
#pragma unroll
    for (int u = 0; u < U; u++)
        if (!((has >> u) & 1u) || (unsigned long long)(k[u] - t.lo) > t.span) g[u] = -1;
}

// Fills the records of a table with unique keys from its join slots.
__global__ void records_kernel(const unsigned long long *slots, uint64_t n, const long long *keys,
                               const int32_t *gid, Record *rec) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long s = slots[i];
        Record r{0, -1, 0};
        if (s) {
            const uint32_t row = slot_row(s);
            r.key = keys[row];
            r.gid = gid[row];
        }
        rec[i] = r;
    }
}

__global__ void direct_kernel(const long long *keys, const int32_t *gid, int64_t n, long long lo, int32_t *direct) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        direct[(unsigned long long)(keys[i] - lo)] = gid[i];
}

// The groups of the requests listed in `list`, a chunk of kChunkGroups at a
// time, spread over all CTAs: f(index into the list, request, first group).
// (A loop over the requests waited for each one's descriptor in turn: 24
// requests took 14 us to clear and 46 us to compact, now 3 and 10.)
constexpr int kChunkThreads = 256;
constexpr int kChunkGroups = 4 * kChunkThreads;
template <class F> __device__ __forceinline__ void for_chunks(const TickDev &d, const int32_t *list, int n, F f) {
    __shared__ int s_first[kMaxTickRequests + 1];  // each request's first chunk
    __shared__ int s_warp[kChunkThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int before = 0;
    for (int i0 = 0; i0 < n; i0 += kChunkThreads) {
        const int i = i0 + threadIdx.x;
        const int c = i < n ? (d.reqs[list[i]].ngroups + kChunkGroups - 1) / kChunkGroups : 0;
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int mine = before;
        for (int w = 0; w < kChunkThreads / 32; w++) {
            if (w < warp) mine += s_warp[w];
            before += s_warp[w];
        }
        if (i < n) s_first[i] = mine + incl - c;
        __syncthreads();
    }
    for (int c = blockIdx.x; c < before; c += gridDim.x) {
        int lo = 0, hi = n - 1;  // the last request whose first chunk is at most c and that has one
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (s_first[mid] <= c) lo = mid;
            else hi = mid - 1;
        }
        f(lo, d.reqs[list[lo]], (c - s_first[lo]) * kChunkGroups);
    }
}

__global__ void __launch_bounds__(kChunkThreads) tick_init_kernel(TickDev d) {
    const TickHeader h = *d.hdr;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < h.n_final; i += gridDim.x * blockDim.x) d.report[i] = Report{0, 0, 0};
    for_chunks(d, d.init, h.n_init, [&](int, const ReqDev &r, int g0) {
        for (int gi = g0 + threadIdx.x; gi < min(g0 + kChunkGroups, r.ngroups); gi += kChunkThreads) {
            r.lo[gi] = 0;
            r.hi[gi] = 0;
            r.cnt[gi] = 0;
        }
    });
}

// ---- the groups' accumulators --------------------------------------------------
// In device memory: SUM of a request whose joined rows cannot pass 2^32 is
// kept as the sums of its values' low 32 bits and of their high parts, which
// two atomics add without waiting for what they add to (the high part of a
// small value is 0: none); otherwise as 128 bits, where the low word's old
// value tells the carry.
struct GroupSums {
    unsigned long long *lo, *hi, *cnt;
    bool split;
    __device__ __forceinline__ void add(int g, long long x) const {
        if (split) {
            atomicAdd(lo + g, (unsigned long long)(uint32_t)x);
            if (x >> 32) atomicAdd(hi + g, (unsigned long long)(x >> 32));
        } else {
            atomic_add_i128_from_i64(lo + g, reinterpret_cast<long long *>(hi) + g, x);
        }
        atomicAdd(cnt + g, 1ull);
    }
};
// In shared memory: four 32-bit words per group and copy, word planes apart
// (64-bit shared atomics are compare-and-swap loops, 32-bit ones are not): the
// count, then SUM in 96 bits with its carries. Few groups have up to 32 copies,
// one per lane, so that the lanes of a warp do not queue on one word.
template <int CAP> struct SmemGroups {
    uint32_t *w;
    // `many`: more than 2^32 rows may join (duplicate build keys): what the
    // count and the sum carry past their words goes straight to device memory,
    // where such a request's sums have 128 bits.
    __device__ __forceinline__ void add(int g, int copies, int copy, bool many, const GroupSums &G, long long x) const {
        const int e = (g << copies) + copy;
        if (!many) atomicAdd(w + e, 1u);
        else if (atomicAdd(w + e, 1u) == 0xFFFFFFFFu) atomicAdd(G.cnt + g, 1ull << 32);
        uint32_t *sum = w + CAP + e;
        const int over = sum96_add([=](int p, uint32_t v) { return atomicAdd(sum + p * CAP, v); }, x);
        if (many && over) atomicAdd(G.hi + g, (unsigned long long)((long long)over * (1ll << 32)));
    }
    __device__ __forceinline__ void clear(const ReqDev &R, int threads) const {
        const int n = R.ngroups << R.copies;
        for (int e = threadIdx.x; e < n; e += threads) {
#pragma unroll
            for (int p = 0; p < 4; p++) w[p * CAP + e] = 0;
        }
    }
    // Adds the groups up and into device memory.
    __device__ __forceinline__ void merge(const ReqDev &R, int threads) const {
        for (int g = threadIdx.x; g < R.ngroups; g += threads) {
            unsigned long long count = 0;
            __int128 sum = 0;
            for (int q = 0; q < (1 << R.copies); q++) {
                const int e = (g << R.copies) + ((q + g) & ((1 << R.copies) - 1));
                count += w[e];
                sum += (__int128)(((unsigned long long)w[2 * CAP + e] << 32) | w[CAP + e]) +
                       ((__int128)(long long)(int32_t)w[3 * CAP + e] << 64);
            }
            if (count) atomicAdd(R.cnt + g, count);
            if (!sum) continue;
            if (R.split) {
                atomicAdd(R.lo + g, (unsigned long long)(uint32_t)sum);
                atomicAdd(reinterpret_cast<unsigned long long *>(R.hi) + g, (unsigned long long)(long long)(sum >> 32));
            } else {
                atomic_add_i128(R.lo + g, R.hi + g, (int64_t)sum, (int64_t)(sum >> 64));
            }
        }
    }
};

// One item's rows: U a thread and step, their loads in flight
// together and the next step's keys and values loaded ahead. What a row needs of
// its request is in registers, and no load stands behind a branch, where it
// would be waited for by itself. Bound by the scattered lookups: the tick above
// takes 0.15 ms without them, and 0.63 ms took it before (64-bit shared atomics,
// the request's fields read again for every row, items of 32,768 rows).
template <int THREADS, int U, int LAYOUT, bool SMEM, class S>
__device__ __forceinline__ void item_rows(const ReqDev &R, const Item &it, const S &sums) {
    const TableView T = R.t;
    const GroupSums G{R.lo, reinterpret_cast<unsigned long long *>(R.hi), R.cnt, R.split != 0};
    const int copies = R.copies, copy = (int)lane_id() & ((1 << copies) - 1);
    const int64_t end = it.row0 + it.rows;
    const long long *keys = R.k, *values = R.x;
    const uint8_t *kvalid = R.kvalid;
    const int64_t kvoff = R.kvoff;
    auto add = [&](int g, long long x) {
        if (SMEM) sums.add(g, copies, copy, LAYOUT == kChains, G, x);
        else G.add(g, x);
    };
    long long k1[U], x1[U];  // the next step's rows
    unsigned has1 = 0;
    auto load = [&](int64_t base) {
        has1 = 0;
#pragma unroll
        for (int u = 0; u < U; u++) {  // past the end: the last row again
            const int64_t r = min(base + (int64_t)u * THREADS + threadIdx.x, end - 1);
            k1[u] = __ldcs(keys + r);
            x1[u] = __ldcs(values + r);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t r = base + (int64_t)u * THREADS + threadIdx.x;
            if (r < end && (!kvalid || bit_get(kvalid, kvoff, r))) has1 |= 1u << u;
        }
    };
    load(it.row0);
    for (int64_t base = it.row0; base < end; base += (int64_t)THREADS * U) {
        long long k[U], x[U];
        const unsigned has = has1;
#pragma unroll
        for (int u = 0; u < U; u++) {
            k[u] = k1[u];
            x[u] = x1[u];
        }
        load(base + (int64_t)THREADS * U);
        if constexpr (LAYOUT == kChains) {
            uint32_t row[U];
            table_heads<U>(T, k, has, row);
#pragma unroll
            for (int u = 0; u < U; u++)  // every build row with this key (duplicates chain newest-first)
                for (uint32_t b = row[u]; b != kNoRow; b = __ldg(T.next + b)) add(__ldg(T.gid + b), x[u]);
        } else {
            int g[U];
            if constexpr (LAYOUT == kDirect) direct_gids<U>(T, k, has, g);
            else record_gids<U>(T, k, has, g);
#pragma unroll
            for (int u = 0; u < U; u++)
                if (g[u] >= 0) add(g[u], x[u]);
        }
    }
}

// QUEUE 0: the requests of few groups (in shared memory) or very many (in
// device memory); 1: those between.
template <int THREADS, int QUEUE>
__global__ void __launch_bounds__(THREADS, QUEUE ? 1 : 1024 / THREADS) tick_probe_kernel(TickDev d) {
    constexpr int U = kTickRowsPerThread;
    extern __shared__ __align__(16) uint8_t smem[];
    const SmemGroups<QUEUE ? kMidGroups : tick_smem_groups(THREADS)> S{reinterpret_cast<uint32_t *>(smem)};
    __shared__ int s_item;
    const int n_items = d.hdr->n_items[QUEUE];
    const Item *items = d.items + d.hdr->items_at[QUEUE];
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(&d.hdr->cursor[QUEUE], 1ull);
        __syncthreads();
        const int item = s_item;
        if (item >= n_items) break;
        const Item it = items[n_items - 1 - item];
        const ReqDev &R = d.reqs[it.req];
        const bool sm = QUEUE || R.use_smem != 0;
        if (sm) S.clear(R, THREADS);
        __syncthreads();
        if (sm) {
            if (R.t.layout == kDirect) item_rows<THREADS, U, kDirect, true>(R, it, S);
            else if (R.t.layout == kRecords) item_rows<THREADS, U, kRecords, true>(R, it, S);
            else item_rows<THREADS, U, kChains, true>(R, it, S);
        } else if constexpr (QUEUE == 0) {
            if (R.t.layout == kDirect) item_rows<THREADS, U, kDirect, false>(R, it, S);
            else if (R.t.layout == kRecords) item_rows<THREADS, U, kRecords, false>(R, it, S);
            else item_rows<THREADS, U, kChains, false>(R, it, S);
        }
        __syncthreads();  // and s_item has been read by all
        if (sm) {
            S.merge(R, THREADS);
            __syncthreads();
        }
    }
}

// The groups of each request that ends in this tick, compacted.
__global__ void __launch_bounds__(kChunkThreads) tick_final_kernel(TickDev d) {
    const TickHeader h = *d.hdr;
    constexpr int U = kChunkGroups / kChunkThreads;
    __shared__ unsigned s_warp[kChunkThreads / 32];
    __shared__ unsigned long long s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for_chunks(d, d.final, h.n_final, [&](int i, const ReqDev &r, int g0) {
        unsigned long long cnt[U];
        int mine = 0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int gi = g0 + u * kChunkThreads + threadIdx.x;
            cnt[u] = gi < r.ngroups ? r.cnt[gi] : 0;
            mine += cnt[u] != 0;
        }
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_warp[warp] = (unsigned)incl;
        __syncthreads();
        unsigned at = 0, total = 0;
        for (int w = 0; w < kChunkThreads / 32; w++) {
            if (w < warp) at += s_warp[w];
            total += s_warp[w];
        }
        if (threadIdx.x == 0) s_base = total ? atomicAdd(&d.report[i].groups, (unsigned long long)total) : 0ull;
        __syncthreads();
        unsigned long long pos = s_base + at + (unsigned)(incl - mine);
        bool over = false;
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!cnt[u]) continue;
            const int gi = g0 + u * kChunkThreads + threadIdx.x;
            unsigned long long l = r.lo[gi];
            long long hh = r.hi[gi];
            if (r.split) {
                const __int128 sum = (__int128)hh * ((__int128)1 << 32) + (__int128)l;
                l = (unsigned long long)sum;
                hh = (long long)(sum >> 64);
            }
            over = over || !((hh == 0 && !(l >> 63)) || (hh == -1 && (l >> 63)));
            r.out_g[pos] = r.gkeys[gi];
            r.out_sum[pos] = (long long)l;
            r.out_cnt[pos] = (long long)cnt[u];
            pos++;
        }
        if (over) atomicOr(&d.report[i].overflow, 1u);
        __syncthreads();  // s_warp and s_base are written by the next chunk
    });
}

// ---- the group directory of a resident table ------------------------------------
// Dense ids for the distinct group values of a build table, with no waits:
// keys are claimed by compare-and-swap, ids handed to occupied slots, then
// every row reads its id.
__global__ void gdir_insert_kernel(const long long *g, int64_t n, unsigned long long *keys, uint64_t mask,
                                   unsigned int *has_marker) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long v = (unsigned long long)g[i];
        if (v == kGroupEmpty) {
            *has_marker = 1;
            continue;
        }
        uint64_t p = finalize(hash_word(v), 0x6772) & mask;
        for (uint64_t t = 0; t <= mask; t++) {
            unsigned long long cur = keys[p];
            if (cur == kGroupEmpty) cur = atomicCAS(&keys[p], kGroupEmpty, v);
            if (cur == kGroupEmpty || cur == v) break;
            p = (p + 1) & mask;
        }
    }
}

__global__ void gdir_assign_kernel(const unsigned long long *keys, uint64_t slots, const unsigned int *has_marker,
                                   int32_t *slot_gid, long long *gkeys, unsigned long long *count) {
    const int64_t span = ((int64_t)slots + 1 + 31) / 32 * 32;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < span; i += (int64_t)gridDim.x * blockDim.x) {
        const bool used = i < (int64_t)slots ? keys[i] != kGroupEmpty : (i == (int64_t)slots && *has_marker != 0);
        const unsigned long long id = warp_alloc(count, used, 0xFFFFFFFFu);
        if (!used) continue;
        slot_gid[i] = (int32_t)id;
        gkeys[id] = i < (int64_t)slots ? (long long)keys[i] : (long long)kGroupEmpty;
    }
}

__global__ void gdir_lookup_kernel(const long long *g, int64_t n, const unsigned long long *keys, uint64_t mask,
                                   const int32_t *slot_gid, int32_t *gid) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long v = (unsigned long long)g[i];
        int32_t id = -1;
        if (v == kGroupEmpty) {
            id = slot_gid[mask + 1];
        } else {
            uint64_t p = finalize(hash_word(v), 0x6772) & mask;
            for (uint64_t t = 0; t <= mask; t++) {
                if (keys[p] == v) {
                    id = slot_gid[p];
                    break;
                }
                p = (p + 1) & mask;
            }
        }
        gid[i] = id;
    }
}

uint64_t pow2_at_least(uint64_t v) {
    uint64_t p = 1;
    while (p < v) p <<= 1;
    return p;
}

}  // namespace

// ---- resident tables --------------------------------------------------------------
struct ResidentTable {
    std::unique_ptr<HashJoin> join;  // inner join on key; arena (key, group)
    DBuf gid;                        // dense group id per build row
    DBuf gkeys;                      // group value per dense id
    DBuf rec;                        // kRecords: (key, gid) per join slot
    DBuf direct;                     // kDirect: gid per key - lo
    int32_t layout = kChains;
    long long lo = 0;
    unsigned long long span = 0;
    int64_t rows = 0;
    int64_t ngroups = 0;
};

// ---- the server -------------------------------------------------------------------------
class Server {
  public:
    Server(Runtime *rt, const krv_server_options &o) : rt_(rt), opt_(o) {
        if (opt_.mode != KRV_SERVE_BATCHED && opt_.mode != KRV_SERVE_PLAIN)
            fail(KRV_INVALID_ARGUMENT, "server mode must be KRV_SERVE_BATCHED or KRV_SERVE_PLAIN");
        if (opt_.tick_rows <= 0) opt_.tick_rows = 64ll << 20;
        if (opt_.max_tick_requests <= 0 || opt_.max_tick_requests > kMaxTickRequests)
            opt_.max_tick_requests = kMaxTickRequests;
        DeviceGuard g(rt_);
        for (int s = 0; s < 2; s++) {
            Slot &sl = slots_[s];
            sl.bytes = layout(nullptr);
            sl.dev = DBuf(rt_, sl.bytes);
            KRV_CUDA(cudaHostAlloc(&sl.host, sl.bytes, cudaHostAllocDefault));
            KRV_CUDA(cudaHostAlloc(&sl.report_host, sizeof(Report) * kMaxTickRequests, cudaHostAllocDefault));
            KRV_CUDA(cudaEventCreateWithFlags(&sl.start, cudaEventDefault));
            KRV_CUDA(cudaEventCreateWithFlags(&sl.done, cudaEventDefault));
        }
        build_candidates();
    }
    ~Server() {
        DeviceGuard g(rt_);
        cudaStreamSynchronize(rt_->stream);
        for (auto &kv : graphs_) cudaGraphExecDestroy(kv.second);
        for (auto &sl : slots_) {
            cudaFreeHost(sl.host);
            cudaFreeHost(sl.report_host);
            cudaEventDestroy(sl.start);
            cudaEventDestroy(sl.done);
        }
    }

    int64_t add_table(const DevBatch &b, int key_col, int group_col) {
        DeviceGuard g(rt_);
        const int nc = (int)b.cols.size();
        if (key_col < 0 || key_col >= nc || group_col < 0 || group_col >= nc)
            fail(KRV_INVALID_ARGUMENT, "table column out of range");
        const DevCol &kc = b.cols[key_col], &gc = b.cols[group_col];
        if (kc.type.id != Type::I64 || gc.type.id != Type::I64)
            fail(KRV_UNSUPPORTED, "server tables are (int64 key, int64 group)");
        if (gc.valid) fail(KRV_UNSUPPORTED, "server table groups without NULLs");
        if (b.rows >= (int64_t)0x7FFFFFFF) fail(KRV_UNSUPPORTED, "server tables below 2^31 rows");
        auto t = std::make_shared<ResidentTable>();
        krv_join_spec js;
        krv_join_spec_init(&js);
        js.join_type = KRV_JOIN_INNER;
        js.n_keys = 1;
        js.probe_keys[0] = 0;
        js.build_keys[0] = 0;
        js.runtime_filter = 0;
        js.build_rows_hint = b.rows;
        t->join.reset(new HashJoin(rt_, js));
        DevBatch kb;
        kb.rows = b.rows;
        kb.cols = {kc, gc};
        t->join->build_push(kb);
        t->join->build_finish();
        t->rows = b.rows;
        // group directory
        const int64_t n = b.rows;
        const DevCol &ag = t->join->arena().cols[1];
        const uint64_t cap = pow2_at_least((uint64_t)std::max<int64_t>(2 * n, 16));
        DBuf keys(rt_, cap * 8), slot_gid(rt_, (cap + 1) * 4), marker(rt_, 8), count(rt_, 8);
        fill_empty(keys.as<unsigned long long>(), cap);
        KRV_CUDA(cudaMemsetAsync(marker.get(), 0, 8, rt_->stream));
        KRV_CUDA(cudaMemsetAsync(count.get(), 0, 8, rt_->stream));
        t->gid = DBuf(rt_, (size_t)std::max<int64_t>(n, 1) * 4);
        if (n > 0) {
            gdir_insert_kernel<<<grid_for(rt_, n, 256, 8), 256, 0, rt_->stream>>>(
                static_cast<const long long *>(ag.data), n, keys.as<unsigned long long>(), cap - 1,
                marker.as<unsigned int>());
            rt_->launches++;
            check_launch("gdir_insert_kernel");
        }
        t->gkeys = DBuf(rt_, (size_t)std::max<int64_t>(n, 1) * 8);
        gdir_assign_kernel<<<grid_for(rt_, (int64_t)cap + 1, 256, 8), 256, 0, rt_->stream>>>(
            keys.as<unsigned long long>(), cap, marker.as<unsigned int>(), slot_gid.as<int32_t>(),
            t->gkeys.as<long long>(), count.as<unsigned long long>());
        rt_->launches++;
        check_launch("gdir_assign_kernel");
        if (n > 0) {
            gdir_lookup_kernel<<<grid_for(rt_, n, 256, 8), 256, 0, rt_->stream>>>(
                static_cast<const long long *>(ag.data), n, keys.as<unsigned long long>(), cap - 1,
                slot_gid.as<int32_t>(), t->gid.as<int32_t>());
            rt_->launches++;
            check_launch("gdir_lookup_kernel");
        }
        t->ngroups = (int64_t)read_scalar<unsigned long long>(rt_, count.get());
        choose_layout(*t);
        const int64_t id = next_table_++;
        tables_[id] = t;
        return id;
    }

    // Unique non-NULL keys get a one-read lookup: a direct array when the keys
    // are dense (span at most 4 x rows), else records at the slot positions.
    void choose_layout(ResidentTable &t) {
        HashJoin &j = *t.join;
        const int64_t rows = t.rows;
        const auto c = j.counters();
        t.layout = kChains;
        if (rows <= 0 || j.indexed_rows() != rows || c.build_keys != rows) return;
        const __int128 span = (__int128)j.key_hi() - (__int128)j.key_lo();
        const long long *keys = static_cast<const long long *>(j.arena().cols[0].data);
        if (span >= 0 && span < (__int128)4 * rows && span < ((__int128)1 << 31)) {
            t.lo = j.key_lo();
            t.span = (unsigned long long)span;
            t.direct = DBuf(rt_, ((size_t)span + 1) * 4);
            KRV_CUDA(cudaMemsetAsync(t.direct.get(), 0xFF, ((size_t)span + 1) * 4, rt_->stream));
            direct_kernel<<<grid_for(rt_, rows, 256, 8), 256, 0, rt_->stream>>>(keys, t.gid.as<int32_t>(), rows, t.lo,
                                                                               t.direct.as<int32_t>());
            rt_->launches++;
            check_launch("direct_kernel");
            t.layout = kDirect;
            return;
        }
        const auto tv = j.table_dev();
        const uint64_t n = tv.mask + 1;
        t.rec = DBuf(rt_, n * sizeof(Record));
        records_kernel<<<grid_for(rt_, (int64_t)n, 256, 8), 256, 0, rt_->stream>>>(tv.slots, n, keys,
                                                                                  t.gid.as<int32_t>(), t.rec.as<Record>());
        rt_->launches++;
        check_launch("records_kernel");
        t.layout = kRecords;
    }

    void drop_table(int64_t id) {
        auto it = tables_.find(id);
        if (it == tables_.end()) fail(KRV_INVALID_ARGUMENT, "no table " + std::to_string(id));
        for (auto &r : reqs_)
            if (r.second->table == it->second) fail(KRV_INVALID_ARGUMENT, "table has requests in flight");
        tables_.erase(it);
    }

    int64_t submit(int64_t table, const DevBatch &b, int key_col, int value_col) {
        auto it = tables_.find(table);
        if (it == tables_.end()) fail(KRV_INVALID_ARGUMENT, "no table " + std::to_string(table));
        const int nc = (int)b.cols.size();
        if (key_col < 0 || key_col >= nc || value_col < 0 || value_col >= nc)
            fail(KRV_INVALID_ARGUMENT, "request column out of range");
        if (b.cols[key_col].type.id != Type::I64 || b.cols[value_col].type.id != Type::I64)
            fail(KRV_UNSUPPORTED, "requests are (int64 key, int64 value)");
        if (b.cols[value_col].valid) fail(KRV_UNSUPPORTED, "request values without NULLs");
        auto r = std::make_shared<Req>();
        r->id = next_req_++;
        r->table = it->second;
        r->batch = b;
        r->k = b.cols[key_col];
        r->x = b.cols[value_col];
        r->rows = b.rows;
        r->bytes = (size_t)std::max<int64_t>(it->second->ngroups, 1) * 48;
        if (opt_.hbm_budget_bytes > 0 && (int64_t)r->bytes > opt_.hbm_budget_bytes)
            fail(KRV_NEED_MEMORY, "request state is larger than the server's HBM budget");
        reqs_[r->id] = r;
        pending_.push_back(r);
        return r->id;
    }

    // Retires finished ticks, then forms and launches the next work.
    // Returns the number of requests still queued or running.
    int64_t step(bool wait) {
        DeviceGuard g(rt_);
        if (opt_.mode == KRV_SERVE_PLAIN) {
            if (!pending_.empty()) {
                auto r = pending_.front();
                run_plain(*r);
                pending_.pop_front();
            }
            return (int64_t)pending_.size();
        }
        retire(false);
        if (inflight_.size() < 2 && (!pending_.empty() || !active_.empty())) launch_tick();
        if (wait && !inflight_.empty()) retire(true);
        return (int64_t)(pending_.size() + active_.size() + waiting_final_count());
    }

    // The next finished request: its id and status, and its result columns
    // (group, SUM, COUNT) when it succeeded. False when none has finished.
    bool poll(int64_t &id, krv_status &status, DevBatch &out) {
        if (done_.empty()) return false;
        auto r = done_.front();
        done_.pop_front();
        id = r->id;
        status = r->status;
        out = r->result;
        reqs_.erase(r->id);
        return true;
    }

    krv_server_stats stats() const {
        krv_server_stats s{};
        s.ticks = ticks_;
        s.requests_done = requests_done_;
        s.rows_probed = rows_probed_;
        s.pending = (int64_t)pending_.size();
        s.running = (int64_t)active_.size();
        s.budget_in_use = budget_used_;
        s.tuned = tuned_ ? 1 : 0;
        const Cand &c = cands_[best_];
        s.threads = c.threads;
        s.item_rows = c.item_rows;
        s.smem_groups = c.smem_groups;
        return s;
    }

  private:
    struct Req {
        int64_t id;
        std::shared_ptr<ResidentTable> table;
        DevBatch batch;
        DevCol k, x;
        int64_t rows = 0, next_row = 0;
        size_t bytes = 0;
        DBuf acc, out;  // accumulators (lo, hi, cnt) and output columns
        bool admitted = false;
        bool inited = false;  // accumulators cleared by a tick
        int last_tick = -1;  // tick that processes its last rows
        krv_status status = KRV_OK;
        DevBatch result;
    };
    struct Slot {
        DBuf dev;
        void *host = nullptr;
        Report *report_host = nullptr;
        size_t bytes = 0;
        cudaEvent_t start = nullptr, done = nullptr;
    };
    struct Tick {
        int slot;
        int64_t id;
        int cand;
        int64_t rows;
        std::vector<std::shared_ptr<Req>> finals;
    };
    struct Cand {
        int threads;
        int64_t item_rows;
        int smem_groups;
        double rows_per_ms_sum = 0;
        int runs = 0;
    };

    // Descriptor layout of a slot; fills `d` with device pointers when given.
    size_t layout(TickDev *d, uint8_t *base = nullptr) const {
        size_t off = 0;
        auto take = [&](size_t bytes) {
            const size_t o = off;
            off = (off + bytes + 255) / 256 * 256;
            return base + o;
        };
        // what a tick uses lies together, so that one copy uploads it
        uint8_t *hdr = take(sizeof(TickHeader));
        uint8_t *init = take(sizeof(int32_t) * kMaxTickRequests);
        uint8_t *fin = take(sizeof(int32_t) * kMaxTickRequests);
        uint8_t *reqs = take(sizeof(ReqDev) * kMaxTickRequests + sizeof(Item) * (kMaxTickItems + 1));
        uint8_t *items = reqs;
        uint8_t *rep = take(sizeof(Report) * kMaxTickRequests);
        if (d) {
            d->hdr = reinterpret_cast<TickHeader *>(hdr);
            d->reqs = reinterpret_cast<ReqDev *>(reqs);
            d->items = reinterpret_cast<Item *>(items);
            d->init = reinterpret_cast<int32_t *>(init);
            d->final = reinterpret_cast<int32_t *>(fin);
            d->report = reinterpret_cast<Report *>(rep);
        }
        return off;
    }

    void fill_empty(unsigned long long *p, uint64_t n);

    void build_candidates() {
        const int threads[2] = {256, 512};
        const int64_t items[2] = {32 << 10, 128 << 10};
        const int smem[2] = {0, kSmemGroupsAlways};
        for (int a : threads)
            for (int64_t b : items)
                for (int c : smem) cands_.push_back(Cand{a, b, c});
        // Fixed shape (no tuning): 512 threads, 128 Ki-row items, shared memory
        // aggregation of few groups always.
        best_ = (int)cands_.size() - 1;
        tuned_ = !opt_.autotune;
    }

    int choose_cand() {
        if (tuned_) return best_;
        for (int i = 0; i < (int)cands_.size(); i++)
            if (cands_[i].runs < 2) return i;
        int b = 0;
        for (int i = 1; i < (int)cands_.size(); i++)
            if (cands_[i].rows_per_ms_sum / cands_[i].runs > cands_[b].rows_per_ms_sum / cands_[b].runs) b = i;
        best_ = b;
        tuned_ = true;
        return best_;
    }

    int64_t waiting_final_count() const {
        int64_t n = 0;
        for (const Tick &t : inflight_) n += (int64_t)t.finals.size();
        return n;
    }

    void admit() {
        while (!pending_.empty() && (int)active_.size() < opt_.max_tick_requests) {
            auto r = pending_.front();
            if (opt_.hbm_budget_bytes > 0 && budget_used_ + (int64_t)r->bytes > opt_.hbm_budget_bytes) break;
            const size_t ng = (size_t)std::max<int64_t>(r->table->ngroups, 1);
            DBuf acc, out;
            try {
                acc = DBuf(rt_, ng * 24);
                out = DBuf(rt_, ng * 24);
            } catch (const Error &e) {
                // the request waits on; those that run may free memory for it
                if (e.code != KRV_NEED_MEMORY || (active_.empty() && inflight_.empty())) throw;
                return;
            }
            pending_.pop_front();
            r->acc = std::move(acc);
            r->out = std::move(out);
            r->admitted = true;
            budget_used_ += (int64_t)r->bytes;
            active_.push_back(r);
        }
    }

    // Where `rows` rows of a request aggregate: in shared memory, by the first
    // launch (0) or the second (1), or in device memory (-1).
    static int smem_of(const Req &r, const Cand &c, int64_t rows) {
        const int64_t ng = r.table->ngroups;
        const bool pays = kSmemRowsPerGroup * ng <= std::min(rows, c.item_rows);
        if (ng <= tick_smem_groups(c.threads) && (ng <= c.smem_groups || pays)) return 0;
        return ng <= kMidGroups && pays ? 1 : -1;
    }

    ReqDev req_dev(const Req &r, const Cand &c, int smem) const {
        const ResidentTable &t = *r.table;
        const auto tv = t.join->table_dev();
        const size_t ng = (size_t)std::max<int64_t>(t.ngroups, 1);
        ReqDev d{};
        d.k = static_cast<const long long *>(r.k.data);
        d.kvalid = r.k.valid;
        d.kvoff = r.k.valid_off;
        d.x = static_cast<const long long *>(r.x.data);
        d.t = TableView{tv.slots, tv.mask, tv.next, tv.seed, static_cast<const long long *>(t.join->arena().cols[0].data),
                        t.gid.as<int32_t>(), t.rec.as<Record>(), t.direct.as<int32_t>(), t.lo, t.span, t.layout, 0};
        d.lo = r.acc.as<unsigned long long>();
        d.hi = reinterpret_cast<long long *>(d.lo + ng);
        d.cnt = d.lo + 2 * ng;
        d.gkeys = t.gkeys.as<long long>();
        d.out_g = r.out.as<long long>();
        d.out_sum = d.out_g + ng;
        d.out_cnt = d.out_g + 2 * ng;
        d.ngroups = (int32_t)t.ngroups;
        d.use_smem = smem >= 0 ? 1 : 0;
        d.copies = 0;
        const int64_t cap = smem > 0 ? kMidGroups : tick_smem_groups(c.threads);
        while (d.copies < 5 && (t.ngroups << (d.copies + 1)) <= cap) d.copies++;
        d.split = t.layout != kChains && r.rows < (1ll << 32) ? 1 : 0;
        return d;
    }

    void launch_tick() {
        admit();
        if (active_.empty()) return;
        const int s = (int)(tick_seq_ & 1);
        Slot &sl = slots_[s];
        // The staging area and report of this slot belong to the tick two back:
        // it must have been retired (in order) before the slot is reused.
        while (std::any_of(inflight_.begin(), inflight_.end(), [&](const Tick &t) { return t.slot == s; }))
            retire(true);
        const int ci = choose_cand();
        const Cand &c = cands_[ci];
        TickDev hd;
        layout(&hd, static_cast<uint8_t *>(sl.host));
        // Shortest remaining first: small requests finish in the tick they join.
        std::vector<std::shared_ptr<Req>> order(active_.begin(), active_.end());
        std::stable_sort(order.begin(), order.end(), [](const std::shared_ptr<Req> &a, const std::shared_ptr<Req> &b) {
            return a->rows - a->next_row < b->rows - b->next_row;
        });
        int nreq = 0, nitems = 0, ninit = 0, nfinal = 0;
        int64_t budget = opt_.tick_rows, rows = 0;
        items_[0].clear();
        items_[1].clear();
        // Items of about an eighth of a CTA's share of the tick, at least one
        // step of the kernel.
        int64_t due = 0;
        for (const auto &r : order) due += r->rows - r->next_row;
        due = std::min(due, budget);
        const int64_t step = (int64_t)c.threads * kTickRowsPerThread;
        const int64_t share = std::max(step, ceil_div(due, (int64_t)8 * rt_->sm_count * (1024 / c.threads)));
        Tick tick{s, tick_seq_, ci, 0, {}};
        std::vector<std::shared_ptr<Req>> keep;
        for (auto &r : order) {
            const int64_t left = r->rows - r->next_row;
            int64_t take = std::min(left, budget);
            int64_t item_rows = std::min(c.item_rows, share);
            const int smem = smem_of(*r, c, take);
            // Groups in shared memory: an item's rows pay for their clearing and
            // merging, and the second launch's CTAs get as many items each.
            // Groups in device memory: an SM's atomics are the limit, so all SMs
            // get some of the rows.
            if (smem >= 0) item_rows = std::min(c.item_rows, std::max(item_rows, kSmemRowsPerGroup * r->table->ngroups));
            else item_rows = std::min(item_rows, std::max(step, ceil_div(take, kMaxTickItems / 8)));
            if (smem == 1) {
                const int64_t turns = ceil_div(take, item_rows * rt_->sm_count);
                item_rows = std::max((int64_t)kMidThreads * kTickRowsPerThread, ceil_div(take, turns * rt_->sm_count));
            }
            const int64_t need_items = (take + item_rows - 1) / item_rows;
            if (nitems + need_items > kMaxTickItems) take = (int64_t)(kMaxTickItems - nitems) * item_rows;
            if (take <= 0 && left > 0) continue;
            const int idx = nreq++;
            hd.reqs[idx] = req_dev(*r, c, smem);
            if (!r->inited) {
                hd.init[ninit++] = idx;
                r->inited = true;
            }
            for (int64_t o = 0; o < take; o += item_rows)
                items_[smem == 1].push_back(Item{idx, 0, r->next_row + o, std::min(item_rows, take - o)});
            nitems = (int)(items_[0].size() + items_[1].size());
            r->next_row += take;
            budget -= take;
            rows += take;
            if (r->next_row == r->rows) {
                hd.final[nfinal++] = idx;
                tick.finals.push_back(r);
            }
            if (nreq == kMaxTickRequests) break;
        }
        if (nreq == 0) return;
        for (auto &r : tick.finals) active_.erase(std::find(active_.begin(), active_.end(), r));
        hd.hdr->n_init = ninit;
        hd.hdr->n_final = nfinal;
        // The items of the largest requests, last in the list, are taken first
        // (the device takes them from its end): the end of a tick is short items.
        int at = (int)ceil_div((int64_t)(sizeof(ReqDev) * nreq), (int64_t)sizeof(Item));
        for (int q = 0; q < 2; q++) {
            hd.hdr->cursor[q] = 0;
            hd.hdr->n_items[q] = (int)items_[q].size();
            hd.hdr->items_at[q] = at;
            if (!items_[q].empty()) std::memcpy(hd.items + at, items_[q].data(), sizeof(Item) * items_[q].size());
            at += (int)items_[q].size();
        }
        tick.rows = rows;
        // Upload the used parts of the descriptors, then run the tick's graph.
        TickDev dd;
        layout(&dd, static_cast<uint8_t *>(sl.dev.get()));
        const size_t used = (size_t)((uint8_t *)(hd.items + at) - (uint8_t *)hd.hdr);
        KRV_CUDA(cudaMemcpyAsync(dd.hdr, hd.hdr, used, cudaMemcpyHostToDevice, rt_->stream));
        KRV_CUDA(cudaEventRecord(sl.start, rt_->stream));
        KRV_CUDA(cudaGraphLaunch(graph_for(s, c.threads, !items_[1].empty(), dd, sl), rt_->stream));
        rt_->launches += items_[1].empty() ? 3 : 4;
        KRV_CUDA(cudaEventRecord(sl.done, rt_->stream));
        tick_seq_++;
        ticks_++;
        rows_probed_ += rows;
        inflight_.push_back(std::move(tick));
    }

    cudaGraphExec_t graph_for(int s, int threads, bool mid, const TickDev &dd, Slot &sl) {
        const int key = s * 4096 + threads * 2 + (mid ? 1 : 0);
        auto it = graphs_.find(key);
        if (it != graphs_.end()) return it->second;
        // The shape of the tick: the kernels read their counts from the
        // descriptors, so one graph serves every tick of this slot and shape.
        const int grid = rt_->sm_count * (threads == 256 ? 4 : 2);
        const size_t smem = (size_t)tick_smem_groups(threads) * kSmemGroupBytes;
        const size_t mid_smem = (size_t)kMidGroups * kSmemGroupBytes;
        const auto probe = threads == 256 ? tick_probe_kernel<256, 0> : tick_probe_kernel<512, 0>;
        const auto mid_probe = tick_probe_kernel<kMidThreads, 1>;
        KRV_CUDA(cudaFuncSetAttribute(probe, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        KRV_CUDA(cudaFuncSetAttribute(mid_probe, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mid_smem));
        cudaStream_t cs;
        KRV_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            tick_init_kernel<<<rt_->sm_count * 2, kChunkThreads, 0, cs>>>(dd);
            if (mid) mid_probe<<<rt_->sm_count, kMidThreads, mid_smem, cs>>>(dd);
            probe<<<grid, threads, smem, cs>>>(dd);
            tick_final_kernel<<<rt_->sm_count * 2, kChunkThreads, 0, cs>>>(dd);
            cudaMemcpyAsync(sl.report_host, dd.report, sizeof(Report) * kMaxTickRequests, cudaMemcpyDeviceToHost, cs);
            e = cudaStreamEndCapture(cs, &graph);
        }
        cudaStreamDestroy(cs);
        if (e != cudaSuccess) fail(KRV_CUDA_ERROR, std::string("tick graph capture: ") + cudaGetErrorString(e));
        cudaGraphExec_t exec = nullptr;
        e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) fail(KRV_CUDA_ERROR, std::string("tick graph instantiate: ") + cudaGetErrorString(e));
        graphs_[key] = exec;
        return exec;
    }

    void retire(bool block) {
        while (!inflight_.empty()) {
            Tick &t = inflight_.front();
            Slot &sl = slots_[t.slot];
            if (block) {
                KRV_CUDA(cudaEventSynchronize(sl.done));
                block = false;  // wait for the oldest only
            } else {
                const cudaError_t q = cudaEventQuery(sl.done);
                if (q == cudaErrorNotReady) return;
                if (q != cudaSuccess) fail(KRV_CUDA_ERROR, std::string("tick: ") + cudaGetErrorString(q));
            }
            float ms = 0.f;
            if (cudaEventElapsedTime(&ms, sl.start, sl.done) == cudaSuccess && ms > 0.f && !tuned_ && t.rows > 0) {
                Cand &c = cands_[t.cand];
                c.rows_per_ms_sum += (double)t.rows / ms;
                c.runs++;
            }
            for (size_t i = 0; i < t.finals.size(); i++) finish_req(*t.finals[i], sl.report_host[i]);
            inflight_.pop_front();
        }
    }

    void finish_req(Req &r, const Report &rep) {
        budget_used_ -= (int64_t)r.bytes;
        r.acc.reset();
        if (rep.overflow && opt_.ansi) {
            r.status = KRV_ARITHMETIC_OVERFLOW;
            r.out.reset();
        } else {
            r.result = result_batch(r, (int64_t)rep.groups);
        }
        r.batch = DevBatch{};
        r.k = DevCol{};
        r.x = DevCol{};
        done_.push_back(reqs_.at(r.id));
        requests_done_++;
    }

    DevBatch result_batch(Req &r, int64_t groups) {
        auto hold = std::make_shared<DBuf>(std::move(r.out));
        const size_t ng = (size_t)std::max<int64_t>(r.table->ngroups, 1);
        DevBatch b;
        b.rows = groups;
        const char *names[3] = {"g", "sum", "count"};
        for (int c = 0; c < 3; c++) {
            DevCol col;
            col.type = DType{Type::I64, 0, 0};
            col.length = groups;
            col.nullable = false;
            col.name = names[c];
            col.hold_data = hold;
            col.data = hold->as<long long>() + c * ng;
            b.cols.push_back(col);
        }
        return b;
    }

    void run_plain(Req &r) {
        // (k, x) JOIN table -> (x, g), then GROUP BY g: SUM(x), COUNT(*)
        DevBatch in;
        in.rows = r.rows;
        in.cols = {r.k, r.x};
        krv_join_spec js = r.table->join->spec();
        js.probe_keys[0] = 0;
        js.n_probe_out = 1;
        js.probe_out[0] = 1;
        js.n_build_out = 1;
        js.build_out[0] = 1;
        HashJoin &j = *r.table->join;
        const krv_join_spec saved = j.spec();
        j.set_probe_shape(js);
        DevBatch pairs;
        try {
            pairs = j.probe(in);
        } catch (...) {
            j.set_probe_shape(saved);
            throw;
        }
        j.set_probe_shape(saved);
        krv_agg_spec as;
        krv_agg_spec_init(&as);
        as.n_group_by = 1;
        as.group_by[0] = 1;
        as.n_aggregates = 2;
        as.aggregates[0] = krv_agg_expr{KRV_AGG_SUM, 0, KRV_AGG_INPUT_RAW, -1, 0, 0, 0, 0};
        as.aggregates[1] = krv_agg_expr{KRV_AGG_COUNT_STAR, 0, KRV_AGG_INPUT_RAW, -1, 0, 0, 0, 0};
        as.ansi = opt_.ansi;
        as.expected_groups = std::max<int64_t>(r.table->ngroups, 1);
        std::unique_ptr<HashAggregate, void (*)(HashAggregate *)> a(make_aggregate(rt_, as), agg_destroy);
        try {
            if (pairs.rows > 0) agg_push(a.get(), pairs);
            agg_finish(a.get());
            DevBatch res = agg_result(a.get());
            if (res.cols.size() != 3) {
                // no joined row reached the aggregate: an empty result of the same shape
                res = DevBatch{};
                for (int c = 0; c < 3; c++) res.cols.push_back(make_col(rt_, DType{Type::I64, 0, 0}, 0, false, ""));
            }
            res.cols[0].name = "g";
            res.cols[1].name = "sum";
            res.cols[2].name = "count";
            r.result = res;
        } catch (const Error &e) {
            if (e.code != KRV_ARITHMETIC_OVERFLOW) throw;
            r.status = KRV_ARITHMETIC_OVERFLOW;
        }
        rows_probed_ += r.rows;
        r.batch = DevBatch{};
        done_.push_back(reqs_.at(r.id));
        requests_done_++;
    }

    Runtime *rt_;
    krv_server_options opt_;
    Slot slots_[2];
    std::map<int, cudaGraphExec_t> graphs_;
    std::vector<Cand> cands_;
    int best_ = 0;
    bool tuned_ = false;
    std::map<int64_t, std::shared_ptr<ResidentTable>> tables_;
    std::map<int64_t, std::shared_ptr<Req>> reqs_;
    std::deque<std::shared_ptr<Req>> pending_, done_;
    std::vector<std::shared_ptr<Req>> active_;
    std::vector<Item> items_[2];  // of the tick being formed, by launch
    std::deque<Tick> inflight_;
    int64_t next_table_ = 1, next_req_ = 1, tick_seq_ = 0;
    int64_t ticks_ = 0, requests_done_ = 0, rows_probed_ = 0, budget_used_ = 0;
};

namespace {
__global__ void fill_u64_kernel(unsigned long long *p, uint64_t n, unsigned long long v) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = v;
}
}  // namespace

void Server::fill_empty(unsigned long long *p, uint64_t n) {
    fill_u64_kernel<<<grid_for(rt_, (int64_t)n, 256, 8), 256, 0, rt_->stream>>>(p, n, kGroupEmpty);
    rt_->launches++;
    check_launch("fill_u64_kernel");
}

Server *make_server(Runtime *rt, const krv_server_options &o) { return new Server(rt, o); }
int64_t server_add_table(Server *s, const DevBatch &b, int key_col, int group_col) {
    return s->add_table(b, key_col, group_col);
}
void server_drop_table(Server *s, int64_t id) { s->drop_table(id); }
int64_t server_submit(Server *s, int64_t table, const DevBatch &b, int key_col, int value_col) {
    return s->submit(table, b, key_col, value_col);
}
int64_t server_step(Server *s, bool wait) { return s->step(wait); }
bool server_poll(Server *s, int64_t &id, krv_status &status, DevBatch &out) { return s->poll(id, status, out); }
krv_server_stats server_stats(const Server *s) { return s->stats(); }
void server_destroy(Server *s) { delete s; }

}  // namespace krv
