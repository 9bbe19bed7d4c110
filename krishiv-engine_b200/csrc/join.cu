// join.cu -- the hash join operator: build arena, open-addressing table over
// the engine's key hash, a probe in two kernels (the lookup counts every tile's
// output rows, the emission writes them with the payload gather fused in), and
// the right/full join tails.
//
// Reference: crates/krishiv-exec/src/join/ (HashJoin, join/mod.rs:1014;
// BuildSink, join/build.rs; ProbeOp, join/probe.rs; JoinIndex,
// crates/krishiv-exec/src/rows/index.rs).
//
// Table layout (one per join): `slots` is a power-of-two array of u64, each a
// chained bit, 31 tag bits of g = fin(h ^ seed) and row + 1 (krv_device.cuh),
// 0 = empty, probed linearly from g & mask; `next` chains the build rows of
// one key newest-first (the reference's salted directory keeps a 16-bit salt
// and row + 1 the same way, rows/index.rs:1-32, 211-283). A probe reads a
// build row's key only when the tag matches, and its chain link only when the
// slot says that the key has more rows.
#include <algorithm>
#include <string>
#include <type_traits>

#include "krv_device.cuh"
#include "ops.h"

namespace krv {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ bool key_valid(const KeyColDev &c, int64_t i) {
    return bit_get(c.valid, c.voff, i);
}

__device__ __forceinline__ void key_words(const KeyColDev &c, int64_t i, uint64_t &w0, uint64_t &w1) {
    if (c.width == 4) {
        w0 = static_cast<const uint32_t *>(c.data)[i];
        w1 = 0;
    } else if (c.width == 8) {
        w0 = static_cast<const uint64_t *>(c.data)[i];
        if (c.is_float) w0 = normalize_f64_bits(w0);
        w1 = 0;
    } else {
        const uint64_t *p = static_cast<const uint64_t *>(c.data) + 2 * i;
        w0 = p[0];
        w1 = p[1];
    }
}

// Every `=` key valid (join/keys.rs:17-19: a NULL `=` key never matches).
__device__ __forceinline__ bool matchable(const KeysDev &k, int64_t i) {
    for (int c = 0; c < k.n; c++)
        if (!((k.null_safe >> c) & 1u) && !key_valid(k.c[c], i)) return false;
    return true;
}

// The seedless row hash h (rows/layout.rs:487-555): NULL under a validity bit
// (null-safe key) mixes NULL_HASH, a value mixes its 8-byte words.
__device__ __forceinline__ uint64_t row_hash(const KeysDev &k, int64_t i) {
    uint64_t h = 0;  // fold(SEEDLESS = 0, MIX)
    for (int c = 0; c < k.n; c++) {
        if (!key_valid(k.c[c], i)) {
            if ((k.null_safe >> c) & 1u) h = mix(h, kNullHash);
            continue;
        }
        uint64_t w0, w1;
        key_words(k.c[c], i, w0, w1);
        h = mix(h, w0);
        if (k.c[c].width == 16) h = mix(h, w1);
    }
    return fold(h, kFinish);
}

__device__ __forceinline__ bool keys_eq(const KeysDev &a, int64_t i, const KeysDev &b, int64_t j) {
    for (int c = 0; c < a.n; c++) {
        const bool va = key_valid(a.c[c], i), vb = key_valid(b.c[c], j);
        if (va != vb) return false;
        if (!va) continue;
        uint64_t a0, a1, b0, b1;
        key_words(a.c[c], i, a0, a1);
        key_words(b.c[c], j, b0, b1);
        if (a0 != b0 || a1 != b1) return false;
    }
    return true;
}

// FAST: one non-float int64 key column.
template <bool FAST>
__device__ __forceinline__ uint64_t hash_of(const KeysDev &k, int64_t i) {
    if (FAST) return hash_word(static_cast<const uint64_t *>(k.c[0].data)[i]);
    return row_hash(k, i);
}
template <bool FAST>
__device__ __forceinline__ bool eq_of(const KeysDev &a, int64_t i, const KeysDev &b, int64_t j) {
    if (FAST)
        return static_cast<const int64_t *>(a.c[0].data)[i] == static_cast<const int64_t *>(b.c[0].data)[j];
    return keys_eq(a, i, b, j);
}

// The table's insertion: kBuildRows rows per thread side by side, so that
// their slot reads, compare-and-swaps and key compares (each a round trip to
// L2) are in flight together.
// ctr (zeroed): [0] distinct keys, [1] a NULL `=` key seen, [2] / [3] the
// largest ~order(k) / order(k) of an int64 key (FAST), [4] indexed rows,
// [5] status bits. The counts are reduced per CTA and the grid is a few CTAs
// per SM: with one update per warp and counter, all on one cache line, the
// updates took most of the kernel. Two rows per thread suit one int64 key
// (four measured 10% slower), one row any other key (more code per row; two
// rows measured 50% slower). krv_join_build_finish on B200, before -> after:
// 1M unique keys 150 -> 89 us, 3M keys with duplicates 225 -> 130 us, 2M
// (int64, int32) keys 140 -> 118 us.
constexpr int kBuildThreads = 256;
constexpr int kBuildRowsFast = 2, kBuildRowsAny = 1;
constexpr unsigned long long kOrderBit = 1ull << 63;  // int64 order as unsigned order
template <bool FAST>
__global__ void __launch_bounds__(kBuildThreads) build_kernel(KeysDev keys, int64_t n, unsigned long long *slots,
                                                              uint64_t mask, uint32_t *next, uint64_t seed,
                                                              unsigned long long *ctr) {
    constexpr int U = FAST ? kBuildRowsFast : kBuildRowsAny, kWarps = kBuildThreads / 32;
    __shared__ unsigned long long s_red[4][kWarps];
    unsigned long long heads = 0, rows = 0, lo = 0, hi = 0;
    bool nulls = false, full = false;
    const int64_t step = (int64_t)gridDim.x * kBuildThreads * U;
    for (int64_t b0 = (int64_t)blockIdx.x * kBuildThreads * U; b0 < n; b0 += step) {
        const int64_t i0 = b0 + threadIdx.x;
        bool act[U];
        uint32_t tag[U], nx[U];
        uint64_t pos[U];
        unsigned long long s[U], entry[U];
        bool more = false;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t i = i0 + u * kBuildThreads;
            act[u] = i < n && matchable(keys, i);
            nulls = nulls || (i < n && !act[u]);
            nx[u] = kNone;
            tag[u] = 0;
            pos[u] = 0;
            entry[u] = 0;
            if (!act[u]) continue;
            more = true;
            rows++;
            if (FAST) {
                const unsigned long long k = static_cast<const unsigned long long *>(keys.c[0].data)[i] ^ kOrderBit;
                lo = ~k > lo ? ~k : lo;
                hi = k > hi ? k : hi;
            }
            const uint64_t g = finalize(hash_of<FAST>(keys, i), seed);
            tag[u] = slot_tag(g);
            pos[u] = g & mask;
            entry[u] = ((unsigned long long)tag[u] << 32) | (unsigned long long)(i + 1);
        }
#pragma unroll
        for (int u = 0; u < U; u++) s[u] = act[u] ? __ldcg(slots + pos[u]) : 0ull;
        // every row is at a slot it has read: claim it when empty, else join
        // its chain when the key is the row's, else go on to the next slot
        for (uint64_t probes = 0; more; probes++) {
            if (probes > 2 * mask + 2) {
                full = true;  // more rows than slots: cannot happen below a load of 0.9
                break;
            }
            unsigned long long old[U];
#pragma unroll
            for (int u = 0; u < U; u++) old[u] = act[u] && s[u] == 0 ? atomicCAS(slots + pos[u], 0ull, entry[u]) : 1ull;
            bool eq[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (act[u] && s[u] == 0) {
                    if (old[u] == 0) {
                        heads++;
                        act[u] = false;
                    }
                    s[u] = old[u];
                }
                eq[u] = act[u] && slot_matches(s[u], tag[u]) &&
                        eq_of<FAST>(keys, i0 + u * kBuildThreads, keys, slot_row(s[u]));
            }
            more = false;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (!act[u]) continue;
                if (eq[u]) {
                    // Same key: this row becomes the head, the old head its next.
                    nx[u] = slot_row(atomicExch(slots + pos[u], entry[u] | kSlotChained));
                    act[u] = false;
                    continue;
                }
                pos[u] = (pos[u] + 1) & mask;
                s[u] = __ldcg(slots + pos[u]);
                more = true;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * kBuildThreads < n) next[i0 + u * kBuildThreads] = nx[u];
    }
    for (int d = 16; d > 0; d >>= 1) {
        heads += __shfl_xor_sync(kFull, heads, d);
        rows += __shfl_xor_sync(kFull, rows, d);
        lo = max(lo, __shfl_xor_sync(kFull, lo, d));
        hi = max(hi, __shfl_xor_sync(kFull, hi, d));
    }
    if ((threadIdx.x & 31) == 0) {
        s_red[0][threadIdx.x >> 5] = heads;
        s_red[1][threadIdx.x >> 5] = rows;
        s_red[2][threadIdx.x >> 5] = lo;
        s_red[3][threadIdx.x >> 5] = hi;
    }
    const bool any_null = __syncthreads_or(nulls), any_full = __syncthreads_or(full);
    if (threadIdx.x) return;
    for (int w = 1; w < kWarps; w++) {
        heads += s_red[0][w];
        rows += s_red[1][w];
        lo = max(lo, s_red[2][w]);
        hi = max(hi, s_red[3][w]);
    }
    if (heads) atomicAdd(ctr, heads);
    if (rows) atomicAdd(ctr + 4, rows);
    if (FAST && rows) {
        atomicMax(ctr + 2, lo);
        atomicMax(ctr + 3, hi);
    }
    if (any_null) ctr[1] = 1;  // a NULL `=` key in the build (null-aware anti join)
    if (any_full) ctr[5] = ST_CAPACITY;
}

template <bool FAST>
__device__ __forceinline__ uint32_t lookup(const KeysDev &pk, int64_t i, const KeysDev &bk,
                                           const unsigned long long *slots, uint64_t mask, uint64_t seed) {
    const uint64_t g = finalize(hash_of<FAST>(pk, i), seed);
    const uint32_t tag = slot_tag(g);
    uint64_t pos = g & mask;
    for (uint64_t probes = 0; probes <= mask; probes++) {
        const unsigned long long s = __ldg(slots + pos);
        if (s == 0) return kNone;
        if (slot_matches(s, tag)) {
            const uint32_t o = slot_row(s);
            if (eq_of<FAST>(pk, i, bk, o)) return o;
        }
        pos = (pos + 1) & mask;
    }
    return kNone;
}

// ---- residual filter (JoinSpec::filter, join/probe.rs:425-436) -------------------
__device__ __forceinline__ bool filter_operand(const FilterOpDev &o, int64_t p, uint32_t b, long long &iv, double &fv) {
    if (o.side == 2) {
        iv = o.ci;
        fv = o.is_float ? o.cf : (double)o.ci;
        return true;
    }
    const int64_t r = o.side == 0 ? p : (int64_t)b;
    if (!bit_get(o.valid, o.voff, r)) return false;
    if (o.width == 4) {
        iv = static_cast<const int *>(o.data)[r];
        fv = (double)iv;
    } else if (o.is_float) {
        fv = static_cast<const double *>(o.data)[r];
        iv = 0;
    } else {
        iv = static_cast<const long long *>(o.data)[r];
        fv = (double)iv;
    }
    return true;
}
template <class T>
__device__ __forceinline__ bool compare(int op, T a, T b) {
    switch (op) {
    case KRV_CMP_EQ: return a == b;
    case KRV_CMP_NE: return a != b;
    case KRV_CMP_LT: return a < b;
    case KRV_CMP_LE: return a <= b;
    case KRV_CMP_GT: return a > b;
    default: return a >= b;
    }
}
__device__ bool filter_true(const FilterDev &F, int64_t p, uint32_t b) {
    for (int t = 0; t < F.n; t++) {
        const FilterTermDev &T = F.t[t];
        long long li, ri;
        double lf, rf;
        if (!filter_operand(T.l, p, b, li, lf) || !filter_operand(T.r, p, b, ri, rf)) return false;
        const bool ok = T.as_float ? compare(T.op, f64_order_key(lf), f64_order_key(rf)) : compare(T.op, li, ri);
        if (!ok) return false;
    }
    return true;
}
// The first build row of the chain from `cur` (newest first) whose pair
// with probe row p passes the filter.
__device__ __forceinline__ uint32_t first_true(const FilterDev &F, int64_t p, uint32_t cur, const uint32_t *next) {
    while (cur != kNone && !filter_true(F, p, cur)) cur = next[cur];
    return cur;
}

struct OutColDev {
    const void *src;
    const uint8_t *src_valid;
    int64_t src_voff;
    void *dst;
    uint32_t *dst_valid;  // zeroed bitmap words, or null (non-nullable output)
    int32_t width;
    int32_t side;         // 0 probe row, 1 build row, 2 constant NULL; 3 / 4 the probe / build row
                          // index itself (int64, -1 for a NULL side): the rows string columns are gathered from
};
struct OutDev {
    OutColDev c[2 * KRV_MAX_OUT_COLUMNS];
    int32_t n;
};

__device__ __forceinline__ void copy_value(void *dst, const void *src, int64_t di, int64_t si, int w) {
    switch (w) {
    case 1: static_cast<uint8_t *>(dst)[di] = static_cast<const uint8_t *>(src)[si]; break;
    case 4: static_cast<uint32_t *>(dst)[di] = static_cast<const uint32_t *>(src)[si]; break;
    case 8: static_cast<uint64_t *>(dst)[di] = static_cast<const uint64_t *>(src)[si]; break;
    default:
        static_cast<uint4 *>(dst)[di] = static_cast<const uint4 *>(src)[si];
        break;
    }
}
__device__ __forceinline__ void zero_value(void *dst, int64_t di, int w) {
    switch (w) {
    case 1: static_cast<uint8_t *>(dst)[di] = 0; break;
    case 4: static_cast<uint32_t *>(dst)[di] = 0; break;
    case 8: static_cast<uint64_t *>(dst)[di] = 0; break;
    default: static_cast<uint4 *>(dst)[di] = make_uint4(0, 0, 0, 0); break;
    }
}

// Writes one round of a warp's output rows: lane `want` writes row `pos`
// from probe row `prow` and build row `brow` (kNone: NULL build side; a
// negative prow: NULL probe side). Validity bits of the round are combined in
// rank order and OR-ed in with at most two atomics per column.
__device__ __forceinline__ void emit_round(const OutDev &out, bool want, unsigned long long pos,
                                           unsigned long long first, int64_t prow, uint32_t brow,
                                           unsigned long long cap) {
    const unsigned ballot = __ballot_sync(kFull, want);
    const unsigned rank = __popc(ballot & lanemask_lt());
    for (int k = 0; k < out.n; k++) {
        const OutColDev &c = out.c[k];
        bool v = false;
        if (want && pos < cap) {
            if (c.side == 3) {
                static_cast<long long *>(c.dst)[pos] = prow >= 0 ? prow : -1;
            } else if (c.side == 4) {
                static_cast<long long *>(c.dst)[pos] = brow != kNone ? (long long)brow : -1;
            } else if (c.side == 0 && prow >= 0) {
                copy_value(c.dst, c.src, (int64_t)pos, prow, c.width);
                v = bit_get(c.src_valid, c.src_voff, prow);
            } else if (c.side == 1 && brow != kNone) {
                copy_value(c.dst, c.src, (int64_t)pos, brow, c.width);
                v = bit_get(c.src_valid, c.src_voff, brow);
            } else {
                zero_value(c.dst, (int64_t)pos, c.width);
            }
        }
        if (c.dst_valid) {
            const unsigned m = __reduce_or_sync(kFull, (want && v) ? (1u << rank) : 0u);
            if (lane_id() == 0 && m) {
                const unsigned long long w = first >> 5;
                const unsigned sh = (unsigned)(first & 31);
                const unsigned long long capw = (cap + 31) >> 5;
                if (w < capw) atomicOr(c.dst_valid + w, m << sh);
                if (sh && w + 1 < capw && (m >> (32 - sh))) atomicOr(c.dst_valid + w + 1, m >> (32 - sh));
            }
        }
    }
}

// ---- the probe ---------------------------------------------------------------------
// Every probe that emits rows (inner, left / right / full outer, semi, anti;
// join/probe.rs:266-502) takes two kernels and one host read between them:
//  1. lookup_kernel finds each probe row's first build row (its head) and its
//     number of output rows, writes both (4 or 8 B per row) and the sum of
//     every tile of kTileRows rows; tile_scan_kernel turns the sums into every
//     tile's first output row and tells the host the total;
//  2. emit_kernel, into output columns of exactly that size, stages each
//     tile's (probe row, build row) pairs in shared memory in output order
//     and writes them column by column: neighbouring threads write neighbouring
//     output rows, so stores are coalesced, and a warp owns whole validity
//     words. Tiles of more than kWindow output rows are emit_long_kernel's,
//     launched when the scan has seen one.
// The lookup is bound by the latency of its dependent random reads (slot,
// build key, chain link), so it keeps few registers and many warps, with no
// barrier or atomic between the reads; the emission is bound by the build
// payload's random reads and the output's stores. One kernel for both
// measured slower: it holds the registers of both phases and its warps wait at
// the output reservation. On B200, the probe call, before (one output
// reservation per warp and step, all on one counter) -> after: left outer of
// 24M rows with 3M build rows of sparse keys, duplicates and NULLs 6.1 -> 0.99
// ms (lookup 0.46, emission 0.46); semi join of 16M rows on (int64, int32)
// 0.60 -> 0.43 ms; inner join of 10M rows over 1M dense keys 0.16 -> 0.15 ms.
//
// How a row finds its build rows:
//  - kDirect: unique, dense int64 keys (`=`): an index of key - lo;
//  - kUnique: no duplicate build keys: the slot's row is the only match;
//  - kChains: the slot's row and its chain;
//  - kRowsOnly: semi and anti joins: whether there is a match.
enum Look : int { kDirect, kUnique, kChains, kRowsOnly };
constexpr int kProbeThreads = 256;
constexpr int kTileRows = 1024;
constexpr int kRowsPerThread = 2;  // lookup: probe rows in flight per thread
constexpr int kLookupBlocks = 6;   // resident lookup CTAs per SM
constexpr int kEmitRows = kTileRows / kProbeThreads;
constexpr int kEmitBlocks = 8;  // resident emission CTAs per SM
constexpr int kWindow = 2048;  // staged pairs
struct DirectDev {
    const uint32_t *row;  // build row of key lo + i, kNone where no row has it
    long long lo;
    unsigned long long span;  // hi - lo
};
struct ProbeDev {
    KeysDev pk, bk;
    int64_t n;
    const unsigned long long *slots;
    uint64_t mask;
    const uint32_t *next;
    uint64_t seed;
    DirectDev dir;
    uint8_t *marks;             // build rows that matched (null: not wanted)
    int pad;                    // unmatched probe rows are emitted with a NULL build side
    int single_match;
    int kind;                   // kRowsOnly: 0 semi, 1 anti, 2 null-aware anti
    int build_empty, build_has_null;
    uint32_t *head;             // per row: its first build row, kNone; kRowsOnly: 0 an output row, kNone none
    uint32_t *cnt;              // kChains: per row, its output rows
    unsigned long long *tiles;  // per tile: its output rows, then (scanned) its first output row
    uint32_t *status;           // single_match: ST_TOO_MANY
};

__global__ void direct_build_kernel(KeysDev bk, int64_t n, DirectDev d) {
    const long long *keys = static_cast<const long long *>(bk.c[0].data);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (!key_valid(bk.c[0], i)) continue;
        const unsigned long long off = (unsigned long long)keys[i] - (unsigned long long)d.lo;
        if (off <= d.span) const_cast<uint32_t *>(d.row)[off] = (uint32_t)i;
    }
}

// NK key columns known to the compiler (0: a loop over any number), so that
// the loads of all columns and rows are in flight together.
template <int NK>
__device__ __forceinline__ void hash_rows_of(const KeysDev &K, int64_t r0, const bool (&look)[kRowsPerThread],
                                             uint64_t (&h)[kRowsPerThread]) {
    constexpr int U = kRowsPerThread, M = NK ? NK : 1;
    const int n = NK ? NK : K.n;
#pragma unroll
    for (int u = 0; u < U; u++) h[u] = 0;  // fold(SEEDLESS = 0, MIX)
    for (int c0 = 0; c0 < n; c0 += M) {
        uint64_t w0[M][U], w1[M][U];
        bool v[M][U];
#pragma unroll
        for (int c = 0; c < M; c++)
#pragma unroll
            for (int u = 0; u < U; u++) {
                w0[c][u] = w1[c][u] = 0;
                v[c][u] = look[u] && key_valid(K.c[c0 + c], r0 + u * kProbeThreads);
                if (v[c][u]) key_words(K.c[c0 + c], r0 + u * kProbeThreads, w0[c][u], w1[c][u]);
            }
#pragma unroll
        for (int c = 0; c < M; c++)
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (v[c][u]) {
                    h[u] = mix(h[u], w0[c][u]);
                    if (K.c[c0 + c].width == 16) h[u] = mix(h[u], w1[c][u]);
                } else if ((K.null_safe >> (c0 + c)) & 1u) {
                    h[u] = mix(h[u], kNullHash);
                }
            }
    }
#pragma unroll
    for (int u = 0; u < U; u++) h[u] = fold(h[u], kFinish);
}

// Whether the thread's probe rows and build rows cand[u] have equal keys (false
// where cand[u] is kNone), all rows' loads in flight together.
template <int NK>
__device__ __forceinline__ void keys_equal(const ProbeDev &A, int64_t r0, const uint32_t (&cand)[kRowsPerThread],
                                           bool (&eq)[kRowsPerThread]) {
    constexpr int U = kRowsPerThread, M = NK ? NK : 1;
    const int n = NK ? NK : A.pk.n;
#pragma unroll
    for (int u = 0; u < U; u++) eq[u] = cand[u] != kNone;
    for (int c0 = 0; c0 < n; c0 += M) {
        uint64_t b0[M][U], b1[M][U];
        bool bv[M][U];
#pragma unroll
        for (int c = 0; c < M; c++)
#pragma unroll
            for (int u = 0; u < U; u++) {
                b0[c][u] = b1[c][u] = 0;
                bv[c][u] = cand[u] != kNone && key_valid(A.bk.c[c0 + c], cand[u]);
                if (bv[c][u]) key_words(A.bk.c[c0 + c], cand[u], b0[c][u], b1[c][u]);
            }
#pragma unroll
        for (int c = 0; c < M; c++)
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (!eq[u]) continue;
                uint64_t p0 = 0, p1 = 0;
                const bool pv = key_valid(A.pk.c[c0 + c], r0 + u * kProbeThreads);
                if (pv) key_words(A.pk.c[c0 + c], r0 + u * kProbeThreads, p0, p1);
                eq[u] = pv == bv[c][u] && p0 == b0[c][u] && p1 == b1[c][u];
            }
    }
}

// The build rows that head the chains of rows r0 + u * kProbeThreads
// (kNone: no match; rows with look[u] false are not looked up), and whether
// each chain has more than its head. KEY: 1 one int64 `=` key, 2 two key
// columns, 0 any keys.
template <int KEY>
__device__ __forceinline__ void find_heads(const ProbeDev &A, int64_t r0, const bool (&look)[kRowsPerThread],
                                           uint32_t (&head)[kRowsPerThread], bool (&chained)[kRowsPerThread]) {
    constexpr int U = kRowsPerThread;
    constexpr bool FAST = KEY == 1;
    uint64_t h[U];
    long long key[U];
    const long long *bkeys = static_cast<const long long *>(A.bk.c[0].data);
    if (FAST) {
        const long long *pkeys = static_cast<const long long *>(A.pk.c[0].data);
#pragma unroll
        for (int u = 0; u < U; u++) key[u] = look[u] ? pkeys[r0 + u * kProbeThreads] : 0;
#pragma unroll
        for (int u = 0; u < U; u++) h[u] = hash_word((uint64_t)key[u]);
    } else {
        hash_rows_of<KEY>(A.pk, r0, look, h);
    }
    uint32_t tag[U];
    uint64_t pos[U];
    unsigned long long sl[U];
    bool more = false;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint64_t g = finalize(h[u], A.seed);
        tag[u] = slot_tag(g);
        pos[u] = g & A.mask;
        sl[u] = look[u] ? __ldg(A.slots + pos[u]) : 0ull;
        head[u] = kNone;
        chained[u] = false;
        more = more || look[u];
    }
    // Every row steps to a slot of its tag or to an empty one (sl is 0 then),
    // the rows of a thread side by side; then the keys are compared once. A
    // tag names another key once in 2^31 times: such a row steps on.
    for (uint64_t round = 0; more && round <= A.mask; round++) {
        bool step = true;
        for (uint64_t probes = 0; step && probes <= A.mask; probes++) {
            step = false;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (sl[u] == 0 || slot_matches(sl[u], tag[u])) continue;
                pos[u] = (pos[u] + 1) & A.mask;
                sl[u] = __ldg(A.slots + pos[u]);
                step = true;
            }
        }
        uint32_t cand[U];
        bool eq[U];
#pragma unroll
        for (int u = 0; u < U; u++) cand[u] = sl[u] != 0 ? slot_row(sl[u]) : kNone;
        if (FAST) {
            long long bkey[U];
#pragma unroll
            for (int u = 0; u < U; u++) bkey[u] = cand[u] != kNone ? __ldg(bkeys + cand[u]) : 0;
#pragma unroll
            for (int u = 0; u < U; u++) eq[u] = cand[u] != kNone && bkey[u] == key[u];
        } else {
            keys_equal<KEY>(A, r0, cand, eq);
        }
        more = false;
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (eq[u]) {
                head[u] = cand[u];
                chained[u] = (sl[u] & kSlotChained) != 0;
                sl[u] = 0;
            } else if (sl[u] != 0) {
                pos[u] = (pos[u] + 1) & A.mask;
                sl[u] = __ldg(A.slots + pos[u]);
                more = true;
            }
        }
    }
}

template <int KEY, bool FILT, int LOOK>
__global__ void __launch_bounds__(kProbeThreads, kLookupBlocks) lookup_kernel(ProbeDev A, FilterDev F) {
    constexpr int U = kRowsPerThread, kWarps = kProbeThreads / 32;
    __shared__ unsigned long long s_warp[kWarps];
    const int64_t base = (int64_t)blockIdx.x * kTileRows;
    unsigned long long total = 0;
#pragma unroll 1
    for (int step = 0; step < kTileRows / (kProbeThreads * U); step++) {
        const int64_t r0 = base + step * (kProbeThreads * U) + threadIdx.x;
        bool look[U], chained[U];
        uint32_t cur[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t r = r0 + u * kProbeThreads;
            look[u] = r < A.n && !A.build_empty && (KEY == 1 ? key_valid(A.pk.c[0], r) : matchable(A.pk, r));
            cur[u] = kNone;
        }
        if (LOOK == kDirect) {
            long long key[U];
#pragma unroll
            for (int u = 0; u < U; u++)
                key[u] = look[u] ? static_cast<const long long *>(A.pk.c[0].data)[r0 + u * kProbeThreads] : 0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const unsigned long long off = (unsigned long long)key[u] - (unsigned long long)A.dir.lo;
                if (look[u] && off <= A.dir.span) cur[u] = __ldg(A.dir.row + off);
            }
        } else {
            find_heads<KEY>(A, r0, look, cur, chained);
        }
        if (FILT)
#pragma unroll
            for (int u = 0; u < U; u++) cur[u] = first_true(F, r0 + u * kProbeThreads, cur[u], A.next);
        uint32_t cnt[U];
        if (LOOK == kChains) {
            // the chains of all rows walked together
            uint32_t w[U];
            bool more = false;
#pragma unroll
            for (int u = 0; u < U; u++) {
                cnt[u] = cur[u] != kNone ? 1 : 0;
                if (A.marks && cur[u] != kNone) A.marks[cur[u]] = 1;
                w[u] = cur[u] != kNone && chained[u] ? cur[u] : kNone;
                more = more || w[u] != kNone;
            }
            while (more) {
                more = false;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (w[u] == kNone) continue;
                    w[u] = __ldg(A.next + w[u]);
                    if (FILT) w[u] = first_true(F, r0 + u * kProbeThreads, w[u], A.next);
                    if (w[u] == kNone) continue;
                    if (A.marks) A.marks[w[u]] = 1;
                    cnt[u]++;
                    more = true;
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (A.single_match && cnt[u] > 1) atomicOr(A.status, ST_TOO_MANY);
                if (cnt[u] == 0 && A.pad && r0 + u * kProbeThreads < A.n) cnt[u] = 1;
            }
        } else if (LOOK == kRowsOnly) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const bool hit = cur[u] != kNone;
                bool ok = hit;
                if (A.kind == 1) ok = !hit;
                if (A.kind == 2) ok = A.build_empty || (!A.build_has_null && look[u] && !hit);
                cnt[u] = ok && r0 + u * kProbeThreads < A.n ? 1 : 0;
                cur[u] = cnt[u] ? 0u : kNone;
            }
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (A.marks && cur[u] != kNone) A.marks[cur[u]] = 1;
                cnt[u] = cur[u] != kNone || (A.pad && r0 + u * kProbeThreads < A.n) ? 1 : 0;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int64_t r = r0 + u * kProbeThreads;
            total += cnt[u];
            if (r >= A.n) continue;
            if (A.head) A.head[r] = cur[u];
            if (LOOK == kChains && A.cnt) A.cnt[r] = cnt[u];
        }
    }
    if (!A.tiles) return;  // only the marks are wanted (right semi / anti)
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(kFull, total, d);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kWarps; w++) total += s_warp[w];
        A.tiles[blockIdx.x] = total;
    }
}

// Every tile's first output row (an exclusive scan of the tiles' rows, in
// place); out[0] (mapped host memory): all rows, out[1]: the status word,
// out[2]: whether a tile has more than kWindow output rows.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) tile_scan_kernel(unsigned long long *tiles, int64_t n,
                                                                 const uint32_t *status, volatile unsigned long long *out) {
    __shared__ unsigned long long s_warp[kScanThreads / 32], s_run;
    constexpr int kPer = 16;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long run = 0;
    bool large = false;
    for (int64_t t0 = 0; t0 < n; t0 += kScanThreads * kPer) {
        unsigned long long v[kPer], mine = 0;
        const int64_t i0 = t0 + (int64_t)threadIdx.x * kPer;
        if (i0 + kPer <= n) {
#pragma unroll
            for (int j = 0; j < kPer; j += 2) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(tiles + i0 + j);
                v[j] = x.x, v[j + 1] = x.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < kPer; j++) v[j] = i0 + j < n ? tiles[i0 + j] : 0;
        }
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            mine += v[j];
            large = large || v[j] > kWindow;
        }
        unsigned long long incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, incl, d);
            if (lane >= d) incl += y;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const unsigned long long w = s_warp[lane];
            unsigned long long wi = w;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long y = __shfl_up_sync(kFull, wi, d);
                if (lane >= d) wi += y;
            }
            s_warp[lane] = wi - w;
            if (lane == 31) s_run = wi;
        }
        __syncthreads();
        unsigned long long at = run + s_warp[warp] + incl - mine;
#pragma unroll
        for (int j = 0; j < kPer; j++) {
            if (i0 + j < n) tiles[i0 + j] = at;
            at += v[j];
        }
        run += s_run;
        __syncthreads();  // s_warp and s_run are rewritten by the next chunk
    }
    large = __syncthreads_or(large);
    if (threadIdx.x == 0) {
        out[0] = run;
        out[1] = status ? *status : 0u;
        out[2] = large;
    }
}

// What emit_kernel reads of the lookup.
struct EmitDev {
    int64_t row0, rows;  // the probe rows of this launch (head and cnt start at row0)
    const uint32_t *head;
    const uint32_t *cnt;
    const unsigned long long *tiles;  // of the tiles from row0 on
    const uint32_t *next;
    int pad;
};

// One output column of m staged pairs (output rows first .. first + m), by N
// threads: the CTA or a warp of it. Four pairs' loads, then their stores.
// `rows`: the pairs' rows of the column's side (kNone: NULL). With validity
// words a warp starts at a multiple of 32 output rows and owns whole words but
// the ends.
template <int N, class T, class R>
__device__ __forceinline__ void emit_column(const OutColDev &c, const R *rows, int64_t base, unsigned long long first, int m) {
    constexpr int V = 4;
    const int t = (int)threadIdx.x & (N - 1);
    const T *src = static_cast<const T *>(c.src) + (c.side == 0 ? base : 0);
    T *dst = static_cast<T *>(c.dst) + first;
    if (!c.dst_valid) {
        for (int q0 = t; q0 < m; q0 += V * N) {
            T v[V];
#pragma unroll
            for (int j = 0; j < V; j++) {
                const int q = q0 + j * N;
                v[j] = T{};
                if (q >= m) continue;
                const uint32_t r = rows[q];
                if (sizeof(R) == 2 || r != kNone) v[j] = src[r];
            }
#pragma unroll
            for (int j = 0; j < V; j++)
                if (q0 + j * N < m) dst[q0 + j * N] = v[j];
        }
        return;
    }
    const int64_t voff = c.src_voff + (c.side == 0 ? base : 0);
    for (int q0 = t - (int)(first & 31); q0 - t < m; q0 += N) {
        const uint32_t r = (unsigned)q0 < (unsigned)m ? (uint32_t)rows[q0] : kNone;
        const bool some = (unsigned)q0 < (unsigned)m && (sizeof(R) == 2 || r != kNone);
        if ((unsigned)q0 < (unsigned)m) dst[q0] = some ? src[r] : T{};
        const unsigned w = __ballot_sync(kFull, some && bit_get(c.src_valid, voff, r));
        if (w && lane_id() == (unsigned)(__ffs(w) - 1)) {
            const int first_lane = q0 - (int)lane_id();  // the word's first pair
            uint32_t *p = c.dst_valid + ((unsigned long long)((long long)first + q0) >> 5);
            if (first_lane >= 0 && first_lane + 32 <= m) *p = w;
            else atomicOr(p, w);  // a word shared with other pairs (zeroed before)
        }
    }
}
template <int N, class R>
__device__ __forceinline__ void emit_by_width(const OutColDev &c, const R *rows, int64_t base, unsigned long long first, int m) {
    if (c.width == 8) emit_column<N, uint64_t>(c, rows, base, first, m);
    else if (c.width == 4) emit_column<N, uint32_t>(c, rows, base, first, m);
    else if (c.width == 16) emit_column<N, uint4>(c, rows, base, first, m);
    else emit_column<N, uint8_t>(c, rows, base, first, m);
}
// All columns of m staged pairs, by N threads.
template <int N>
__device__ __forceinline__ void emit_pairs(const OutDev &out, const uint16_t *prow, const uint32_t *brow, int64_t base,
                                           unsigned long long first, unsigned m) {
    for (int k = 0; k < out.n; k++) {
        const OutColDev c = out.c[k];
        if (c.side == 0) {
            emit_by_width<N>(c, prow, base, first, (int)m);
        } else if (c.side == 1) {
            emit_by_width<N>(c, brow, base, first, (int)m);
        } else {  // the row index itself (3 probe, 4 build)
            for (unsigned q = threadIdx.x & (N - 1); q < m; q += N)
                static_cast<long long *>(c.dst)[first + q] =
                    c.side == 3 ? (long long)(base + prow[q]) : brow[q] != kNone ? (long long)brow[q] : -1ll;
        }
    }
}

// This thread's rows of its tile (neighbours, so that output order is probe
// order): their first build rows and numbers of output rows, the output rows
// before them in the tile, and the tile's. All threads of the CTA.
template <int LOOK, class Sum>
__device__ __forceinline__ void emit_rows(const EmitDev &E, int64_t tile, uint32_t (&cur)[kEmitRows], uint32_t (&cnt)[kEmitRows],
                                          Sum *s_warp, Sum &before, Sum &total) {
    constexpr int U = kEmitRows, kWarps = kProbeThreads / 32;
    static_assert(U == 4, "heads are read four at a time");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t l0 = tile * kTileRows + threadIdx.x * U;
    if (l0 + U <= E.rows) {
        const uint4 h = *reinterpret_cast<const uint4 *>(E.head + l0);
        cur[0] = h.x, cur[1] = h.y, cur[2] = h.z, cur[3] = h.w;
        if (LOOK == kChains) {
            const uint4 n = *reinterpret_cast<const uint4 *>(E.cnt + l0);
            cnt[0] = n.x, cnt[1] = n.y, cnt[2] = n.z, cnt[3] = n.w;
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; u++) {
            cur[u] = l0 + u < E.rows ? E.head[l0 + u] : kNone;
            if (LOOK == kChains) cnt[u] = l0 + u < E.rows ? E.cnt[l0 + u] : 0;
        }
    }
    Sum mine = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (LOOK != kChains) cnt[u] = cur[u] != kNone || (E.pad && l0 + u < E.rows) ? 1 : 0;
        if (LOOK == kRowsOnly) cur[u] = kNone;
        mine += cnt[u];
    }
    Sum incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Sum y = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    total = 0;
    before = incl - mine;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const Sum c = s_warp[w];
        before += w < warp ? c : 0;
        total += c;
    }
}

// The tiles of at most kWindow output rows, each staged whole.
template <bool FILT, int LOOK>
__global__ void __launch_bounds__(kProbeThreads, kEmitBlocks) emit_kernel(EmitDev E, OutDev out, FilterDev F) {
    constexpr int U = kEmitRows;
    // a tile's output rows: at most one per probe row, or chains of any length
    using Sum = std::conditional_t<LOOK == kChains, unsigned long long, uint32_t>;
    __shared__ Sum s_warp[kProbeThreads / 32];
    __shared__ uint32_t s_brow[kWindow];
    __shared__ uint16_t s_prow[kWindow];
    const int64_t base = E.row0 + (int64_t)blockIdx.x * kTileRows;  // the tile's first probe row
    uint32_t cur[U], cnt[U];
    Sum before, total;
    emit_rows<LOOK>(E, blockIdx.x, cur, cnt, s_warp, before, total);
    if (LOOK == kChains && total > kWindow) return;  // emit_long_kernel's
    uint32_t at = (uint32_t)before;
    if (LOOK == kChains) {
        // the chains of the thread's rows side by side: each step is a
        // dependent random read
        uint32_t off[U];
        bool more = true;
#pragma unroll
        for (int u = 0; u < U; u++) {
            off[u] = at;
            at += cnt[u];
        }
        for (uint32_t k = 0; more; k++) {
            more = false;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (k >= cnt[u]) continue;
                s_prow[off[u] + k] = (uint16_t)(threadIdx.x * U + u);
                s_brow[off[u] + k] = cur[u];
                if (k + 1 >= cnt[u]) continue;
                cur[u] = __ldg(E.next + cur[u]);
                if (FILT) cur[u] = first_true(F, base + threadIdx.x * U + u, cur[u], E.next);
                more = true;
            }
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!cnt[u]) continue;
            s_prow[at] = (uint16_t)(threadIdx.x * U + u);
            s_brow[at] = cur[u];
            at++;
        }
    }
    __syncthreads();
    emit_pairs<kProbeThreads>(out, s_prow, s_brow, base, E.tiles[blockIdx.x], (unsigned)total);
}

// The tiles of more than kWindow output rows (long chains of duplicate build
// keys), kLongParts CTAs to a tile and each warp for itself: its lanes follow
// their rows' chains side by side, a step at a time, stage the pairs as they come
// and write them out whenever the warp's share of the window may not hold
// another step. Bound by the chains' dependent reads. Measured on B200, 50,000
// probe rows, chains of 1,024, 25M output rows of three columns: 0.67 ms (the
// join 1.9 ms; 2.9 with four rows to a lane). With the CTA staging a window of
// its tile at a time, only the threads whose rows fell into it followed chains,
// and the join took 92 ms; a warp per 32 rows writing each step took 2.0 ms.
constexpr int kLongParts = kTileRows / kProbeThreads;
template <bool FILT>
__global__ void __launch_bounds__(kProbeThreads) emit_long_kernel(EmitDev E, OutDev out, FilterDev F) {
    constexpr int kWarps = kProbeThreads / 32, kShare = kWindow / kWarps;
    static_assert(kShare >= 64, "a warp's share holds more than a step's pairs");
    __shared__ unsigned long long s_warp[kWarps], s_before[kProbeThreads];
    __shared__ uint32_t s_brow[kWarps][kShare];
    __shared__ uint16_t s_prow[kWarps][kShare];
    const int warp = threadIdx.x >> 5;
    const int64_t tile = blockIdx.x / kLongParts;
    const int part = blockIdx.x % kLongParts * kProbeThreads;  // this CTA's first row of the tile
    const int64_t base = E.row0 + tile * kTileRows;
    unsigned long long first;
    {
        uint32_t cur[kEmitRows], cnt[kEmitRows];
        unsigned long long before, total;
        emit_rows<kChains>(E, tile, cur, cnt, s_warp, before, total);
        if (total <= kWindow) return;  // emit_kernel's
        s_before[threadIdx.x] = before;  // the output rows before tile row threadIdx.x * kEmitRows
        __syncthreads();
        first = E.tiles[tile] + s_before[(part + warp * 32) / kEmitRows];
    }
    const int row = part + (int)threadIdx.x;
    const bool live = tile * kTileRows + row < E.rows;
    uint32_t cur = live ? E.head[tile * kTileRows + row] : kNone, left = live ? E.cnt[tile * kTileRows + row] : 0;
    unsigned want = __ballot_sync(kFull, left != 0);
    while (want) {
        unsigned m = 0;
        for (; want && m + 32 <= (unsigned)kShare; want = __ballot_sync(kFull, left != 0)) {
            if (left) {
                const unsigned q = m + __popc(want & lanemask_lt());
                s_prow[warp][q] = (uint16_t)row;
                s_brow[warp][q] = cur;
                if (--left) {
                    cur = __ldg(E.next + cur);
                    if (FILT) cur = first_true(F, base + row, cur, E.next);
                }
            }
            m += __popc(want);
        }
        __syncwarp();
        emit_pairs<32>(out, s_prow[warp], s_brow[warp], base, first, m);
        first += m;
        __syncwarp();  // the share is staged anew
    }
}

// Existence: every probe row once plus `exists` (join/mod.rs:35-45). Rows
// keep their positions; the flag of rows [base, base + 32) is one word.
template <bool FAST, bool FILT>
__global__ void __launch_bounds__(256) probe_exists_kernel(KeysDev pk, KeysDev bk, int64_t n,
                                                           const unsigned long long *slots, uint64_t mask,
                                                           uint64_t seed, uint32_t *exists, int build_empty,
                                                           const uint32_t *next, FilterDev F) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < n; base += stride) {
        const int64_t i = base + threadIdx.x;
        bool hit = false;
        if (i < n && !build_empty && matchable(pk, i)) {
            uint32_t c = lookup<FAST>(pk, i, bk, slots, mask, seed);
            if (FILT) c = first_true(F, i, c, next);
            hit = c != kNone;
        }
        const unsigned word = __ballot_sync(kFull, hit);
        if (lane_id() == 0 && (i < n)) exists[i >> 5] = word;
    }
}

// Allocates this round's output rows for the warp: returns the first row of
// the round (same on every lane) and this lane's row.
__device__ __forceinline__ unsigned long long round_alloc(unsigned long long *count, bool want,
                                                          unsigned long long &pos) {
    const unsigned ballot = __ballot_sync(kFull, want);
    unsigned long long first = 0;
    if (lane_id() == 0 && ballot) first = atomicAdd(count, (unsigned long long)__popc(ballot));
    first = __shfl_sync(kFull, first, 0);
    pos = first + __popc(ballot & lanemask_lt());
    return first;
}

// Build rows by their marks once the probe side is done (emit_build,
// join/probe.rs:610-): kind 0 right semi (marked rows with a matchable key),
// kind 1 unmatched rows (right anti, right outer, full outer).
__global__ void __launch_bounds__(256) tail_kernel(int64_t nb, const uint8_t *marks, KeysDev bk, int kind,
                                                   OutDev out, unsigned long long cap,
                                                   unsigned long long *count) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < nb; base += stride) {
        const int64_t r = base + threadIdx.x;
        bool ok = false;
        if (r < nb) ok = kind == 0 ? (marks[r] != 0 && matchable(bk, r)) : marks[r] == 0;
        unsigned long long pos;
        const unsigned long long first = round_alloc(count, ok, pos);
        emit_round(out, ok, pos, first, -1, ok ? (uint32_t)r : kNone, cap);
    }
}

void zero(Runtime *rt, void *p, size_t bytes) {
    if (bytes) KRV_CUDA(cudaMemsetAsync(p, 0, bytes, rt->stream));
}

}  // namespace

KeysDev keys_of(const DevBatch &b, const int32_t *cols, int n, const int32_t *null_safe) {
    KeysDev k{};
    k.n = n;
    for (int i = 0; i < n; i++) {
        if (cols[i] < 0 || cols[i] >= (int)b.cols.size()) fail(KRV_INVALID_ARGUMENT, "key column out of range");
        const DevCol &c = b.cols[cols[i]];
        const int w = c.type.width();
        if (w != 4 && w != 8 && w != 16) fail(KRV_UNSUPPORTED, "key column of type " + c.type.format());
        k.c[i] = KeyColDev{c.data, c.valid, c.valid_off, w, c.type.id == Type::F64 ? 1 : 0};
        if (null_safe && null_safe[i]) k.null_safe |= 1u << i;
    }
    return k;
}

namespace {
// The join's own key hash for every row, as the build and probe kernels
// compute it: h (row_hash), g = fin(h ^ seed), and the partition at `depth`
// (0: the top `radix` bits of h; d >= 1: bits [48-3d, 51-3d) of g).
__global__ void __launch_bounds__(256) hash_rows_kernel(KeysDev k, int64_t n, uint64_t seed, int depth, int radix,
                                                        uint64_t *out_h, uint64_t *out_g, int32_t *out_part) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t h = row_hash(k, i);
        const uint64_t g = finalize(h, seed);
        if (out_h) out_h[i] = h;
        if (out_g) out_g[i] = g;
        if (out_part) out_part[i] = depth == 0 ? (int32_t)(h >> (64 - radix)) : (int32_t)((g >> (48 - 3 * depth)) & 7u);
    }
}
}  // namespace

void hash_rows(Runtime *rt, const DevBatch &b, const int32_t *cols, int n, const int32_t *null_safe, uint64_t seed,
               int depth, int radix, uint64_t *out_h, uint64_t *out_g, int32_t *out_part) {
    if (n < 1 || n > KRV_MAX_KEYS) fail(KRV_INVALID_ARGUMENT, "1 to 4 key columns");
    // Hashing::partition (join/keys.rs:92-95, 118-128): radix 3..6, depth 0..6
    radix = std::min(6, std::max(3, radix));
    if (depth < 0) fail(KRV_INVALID_ARGUMENT, "negative partition depth");
    depth = std::min(depth, 6);
    const KeysDev k = keys_of(b, cols, n, null_safe);
    if (b.rows == 0) return;
    hash_rows_kernel<<<grid_for(rt, b.rows, 256, 8), 256, 0, rt->stream>>>(k, b.rows, seed, depth, radix, out_h, out_g,
                                                                          out_part);
    rt->launches++;
    check_launch("hash_rows_kernel");
}

// One int64 `=` key: hashed and compared as its value (a `<=>` key's NULL is a
// key of its own, which the general code tells from every value).
static bool fast_keys(const KeysDev &k) { return k.n == 1 && k.c[0].width == 8 && !k.c[0].is_float && !k.null_safe; }

HashJoin::HashJoin(Runtime *rt, const krv_join_spec &spec) : rt_(rt), spec_(spec) {
    if (spec.n_keys < 1 || spec.n_keys > KRV_MAX_KEYS) fail(KRV_INVALID_ARGUMENT, "join needs 1..4 keys");
    if (spec.join_type < KRV_JOIN_INNER || spec.join_type > KRV_JOIN_FULL_OUTER)
        fail(KRV_INVALID_ARGUMENT, "unknown join type");
    if (spec.has_residual_filter && spec.join_type == KRV_JOIN_NULL_AWARE_ANTI)
        fail(KRV_UNSUPPORTED, "KRISHIV_UNSUPPORTED_FEATURE: null-aware anti join with a residual condition");
    if (spec.single_match && spec.join_type != KRV_JOIN_LEFT_OUTER)
        fail(KRV_INVALID_ARGUMENT, "single_match is for left outer joins only");
    if (spec.join_type == KRV_JOIN_NULL_AWARE_ANTI && (spec.n_keys != 1 || spec.null_safe[0]))
        fail(KRV_INVALID_ARGUMENT, "a null-aware anti join has one `=` key");
    if (spec.n_probe_out > KRV_MAX_OUT_COLUMNS || spec.n_build_out > KRV_MAX_OUT_COLUMNS)
        fail(KRV_INVALID_ARGUMENT, "too many output columns");
    if (spec_.max_load <= 0.f || spec_.max_load > 0.9f) spec_.max_load = 0.5f;
    if (spec_.seed == 0) spec_.seed = 0x4B52565F4A4F494EULL;  // fixed: results never depend on it
    counters_.partitions = 1;
}

// Room for `need` build rows in the arena.
void HashJoin::grow_arena(int64_t need) {
    if (need > (int64_t)0xFFFFFFFEll) fail(KRV_UNSUPPORTED, "more than 2^32-2 build rows in one table");
    if (need > arena_cap_) {
        int64_t cap = std::max<int64_t>({need, arena_cap_ * 2, spec_.build_rows_hint, 1024});
        if (arena_var_.size() < arena_cols_.size()) arena_var_.resize(arena_cols_.size());
        for (size_t i = 0; i < arena_cols_.size(); i++) {
            const DType t = arena_cols_[i].type;
            // a string column keeps a start (int64) per row here and its length beside
            const size_t w = t.var() ? 8 : (size_t)t.width();
            const size_t bytes = t.id == Type::Bool ? (size_t)ceil_div(cap, 8) : (size_t)cap * w;
            auto nd = std::make_shared<DBuf>(rt_, bytes);
            std::shared_ptr<DBuf> nv;
            if (arena_valid_[i]) {
                nv = std::make_shared<DBuf>(rt_, (size_t)ceil_div(cap, 32) * 4 + 8);
                zero(rt_, nv->get(), nv->bytes());
            }
            std::shared_ptr<DBuf> nl;
            if (t.var()) nl = std::make_shared<DBuf>(rt_, (size_t)cap * 4);
            if (build_rows_) {
                const size_t old = t.id == Type::Bool ? (size_t)ceil_div(build_rows_, 8) : (size_t)build_rows_ * w;
                KRV_CUDA(cudaMemcpyAsync(nd->get(), arena_data_[i]->get(), old, cudaMemcpyDeviceToDevice, rt_->stream));
                if (nv)
                    KRV_CUDA(cudaMemcpyAsync(nv->get(), arena_valid_[i]->get(), (size_t)ceil_div(build_rows_, 8),
                                             cudaMemcpyDeviceToDevice, rt_->stream));
                if (nl)
                    KRV_CUDA(cudaMemcpyAsync(nl->get(), arena_var_[i].lens->get(), (size_t)build_rows_ * 4,
                                             cudaMemcpyDeviceToDevice, rt_->stream));
            }
            arena_data_[i] = nd;
            arena_valid_[i] = nv;
            if (nl) {
                arena_var_[i].starts = nd;
                arena_var_[i].lens = nl;
            }
        }
        arena_cap_ = cap;
    }
}

// Room for `rows` more build rows (no NULLs), which the caller's kernels
// write: where each column's begin. They count from build_commit on.
void HashJoin::build_reserve(int64_t rows, void **dst) {
    if (built_ || !have_schema_ || coded_) fail(KRV_INTERNAL, "build_reserve takes a plain build side's rows");
    DeviceGuard g(rt_);
    grow_arena(build_rows_ + rows);
    for (size_t i = 0; i < arena_cols_.size(); i++) {
        const DType t = arena_cols_[i].type;
        if (t.id == Type::Bool || t.var()) fail(KRV_UNSUPPORTED, "build_reserve takes fixed-width columns");
        dst[i] = arena_data_[i]->as<uint8_t>() + (size_t)build_rows_ * t.width();
    }
}

void HashJoin::build_commit(int64_t rows) {
    for (size_t i = 0; i < arena_cols_.size(); i++)
        if (arena_valid_[i]) set_bits(rt_, arena_valid_[i]->as<uint8_t>(), build_rows_, rows);
    build_rows_ += rows;
}

void HashJoin::append_arena(const DevBatch &b) {
    if (!have_schema_) {
        for (const DevCol &c : b.cols) {
            DevCol a;
            a.type = c.type;
            a.name = c.name;
            a.nullable = c.nullable;
            arena_cols_.push_back(a);
        }
        arena_data_.resize(b.cols.size());
        arena_valid_.resize(b.cols.size());
        have_schema_ = true;
    } else {
        if (b.cols.size() != arena_cols_.size()) fail(KRV_INVALID_ARGUMENT, "build batches differ in columns");
        for (size_t i = 0; i < b.cols.size(); i++)
            if (b.cols[i].type != arena_cols_[i].type) fail(KRV_INVALID_ARGUMENT, "build batches differ in types");
    }
    const int64_t need = build_rows_ + b.rows;
    grow_arena(need);
    for (size_t i = 0; i < arena_cols_.size(); i++) {
        const DevCol &c = b.cols[i];
        const DType t = c.type;
        if (t.id == Type::Bool) fail(KRV_UNSUPPORTED, "boolean build columns");
        if (c.valid) arena_cols_[i].nullable = true;
        if (b.rows == 0) continue;  // an empty batch only fixes the schema
        if (t.var()) {
            var_arena_append(rt_, arena_var_[i], c, build_rows_, b.rows);
        } else {
            const size_t w = (size_t)t.width();
            KRV_CUDA(cudaMemcpyAsync(arena_data_[i]->as<uint8_t>() + build_rows_ * w, c.data, (size_t)b.rows * w,
                                     cudaMemcpyDeviceToDevice, rt_->stream));
        }
        // a column keeps a bitmap from its first batch with one on
        if (c.valid && !arena_valid_[i]) {
            arena_valid_[i] = std::make_shared<DBuf>(rt_, (size_t)ceil_div(arena_cap_, 32) * 4 + 8);
            zero(rt_, arena_valid_[i]->get(), arena_valid_[i]->bytes());
            set_bits(rt_, arena_valid_[i]->as<uint8_t>(), 0, build_rows_);
        }
        if (arena_valid_[i]) append_bits(rt_, c.valid, c.valid_off, b.rows, arena_valid_[i]->as<uint8_t>(), build_rows_);
    }
    build_rows_ = need;
}

void HashJoin::build_adopt(DevBatch b) {
    if (built_ || have_schema_) fail(KRV_INVALID_ARGUMENT, "build_adopt takes the whole build side, before any push");
    if (b.rows > (int64_t)0xFFFFFFFEll) fail(KRV_UNSUPPORTED, "more than 2^32-2 build rows in one table");
    for (const DevCol &c : b.cols) {
        if (!c.hold_data || c.hold_data->get() != c.data) fail(KRV_INVALID_ARGUMENT, "build_adopt needs owned columns");
        if (c.type.id == Type::Bool) fail(KRV_UNSUPPORTED, "boolean build columns");
        DevCol m;
        m.type = c.type;
        m.name = c.name;
        m.nullable = c.nullable || c.valid;
        arena_cols_.push_back(m);
        arena_data_.push_back(c.hold_data);
        arena_valid_.push_back(c.valid && c.valid_off == 0 ? c.hold_valid : nullptr);
        if (c.valid && (c.valid_off != 0 || !c.hold_valid)) fail(KRV_INVALID_ARGUMENT, "build_adopt needs owned bitmaps");
    }
    have_schema_ = true;
    build_rows_ = b.rows;
    arena_cap_ = b.rows;
}

HashJoin::~HashJoin() = default;

VarSrc HashJoin::var_src(int side, int col, const DevBatch *probe) const {
    VarSrc v{};
    if (side == 0) {
        const DevCol &c = probe->cols[col];
        v.offs = static_cast<const int32_t *>(c.data);
        v.bytes = static_cast<const uint8_t *>(c.bytes);
        v.valid = c.valid;
        v.voff = c.valid_off;
        return v;
    }
    if (col >= (int)arena_var_.size() || !arena_var_[col].starts) return v;  // no build rows: never read
    const VarArena &a = arena_var_[col];
    v.starts = a.starts->as<long long>();
    v.lens = a.lens->as<int32_t>();
    v.bytes = a.heap ? a.heap->as<uint8_t>() : nullptr;
    v.valid = arena_cols_[col].nullable && arena_valid_[col] ? arena_valid_[col]->as<uint8_t>() : nullptr;
    return v;
}

DevCol HashJoin::empty_col(const DevCol &meta) const {
    if (meta.type.var()) return var_gather(rt_, VarSrc{}, nullptr, 0, meta.type, meta.nullable, meta.name);
    return make_col(rt_, meta.type, 0, meta.nullable, meta.name);
}

void HashJoin::set_filter(const krv_join_filter &f) {
    if (decided_) fail(KRV_INVALID_ARGUMENT, "krv_join_set_filter after the first build push");
    if (spec_.join_type == KRV_JOIN_NULL_AWARE_ANTI)
        fail(KRV_UNSUPPORTED, "KRISHIV_UNSUPPORTED_FEATURE: null-aware anti join with a residual condition");
    if (f.n_terms < 1 || f.n_terms > KRV_MAX_FILTER_TERMS)
        fail(KRV_INVALID_ARGUMENT, "a residual filter has 1 to 8 comparisons");
    for (int t = 0; t < f.n_terms; t++) {
        const krv_filter_term &T = f.terms[t];
        if (T.op < KRV_CMP_EQ || T.op > KRV_CMP_GE) fail(KRV_INVALID_ARGUMENT, "unknown comparison");
        for (const krv_filter_operand *o : {&T.left, &T.right})
            if (o->kind < KRV_OPERAND_PROBE || o->kind > KRV_OPERAND_CONST_F64)
                fail(KRV_INVALID_ARGUMENT, "unknown filter operand kind");
    }
    residual_ = f;
    residual_set_ = true;
    spec_.has_residual_filter = 1;
}

// The device form of the residual filter over probe batch `in` and the arena.
FilterDev HashJoin::filter_dev(const DevBatch &in) const {
    FilterDev F{};
    F.n = residual_.n_terms;
    auto operand = [&](const krv_filter_operand &o, FilterOpDev &d, DType &t) {
        d.side = o.kind == KRV_OPERAND_PROBE ? 0 : o.kind == KRV_OPERAND_BUILD ? 1 : 2;
        if (d.side == 2) {
            d.is_float = o.kind == KRV_OPERAND_CONST_F64;
            d.ci = o.i64;
            d.cf = o.f64;
            t = DType{d.is_float ? Type::F64 : Type::I64, 0, 0};
            return;
        }
        const int ncol = d.side == 0 ? (int)in.cols.size() : (int)arena_cols_.size();
        if (o.column < 0 || o.column >= ncol) fail(KRV_INVALID_ARGUMENT, "residual filter column out of range");
        const DevCol &meta = d.side == 0 ? in.cols[o.column] : arena_cols_[o.column];
        t = meta.type;
        if (t.id != Type::I32 && t.id != Type::Date32 && t.id != Type::I64 && t.id != Type::Dec64 && t.id != Type::F64)
            fail(KRV_UNSUPPORTED, "a residual filter over " + t.format() + " columns");
        d.width = t.width();
        d.is_float = t.id == Type::F64;
        if (d.side == 0) {
            d.data = meta.data;
            d.valid = meta.valid;
            d.voff = meta.valid_off;
        } else if (!arena_.cols.empty()) {
            const DevCol &c = arena_.cols[o.column];
            d.data = c.data;
            d.valid = meta.nullable ? c.valid : nullptr;
            d.voff = c.valid_off;
        }
    };
    for (int t = 0; t < F.n; t++) {
        const krv_filter_term &T = residual_.terms[t];
        FilterTermDev &D = F.t[t];
        D.op = T.op;
        DType lt, rt;
        operand(T.left, D.l, lt);
        operand(T.right, D.r, rt);
        D.as_float = D.l.is_float || D.r.is_float;
        const bool ldec = lt.id == Type::Dec64, rdec = rt.id == Type::Dec64;
        if (!D.as_float && D.l.side != 2 && D.r.side != 2 && ldec != rdec)
            fail(KRV_UNSUPPORTED, "a residual filter compares a decimal column with an integer column");
        if (ldec && rdec && lt.scale != rt.scale)
            fail(KRV_UNSUPPORTED, "a residual filter compares decimal columns of different scales");
    }
    return F;
}

// Whether the keys are coded: some key column of the first build batch is
// a string or binary column.
void HashJoin::decide(const DevBatch &b) {
    decided_ = true;
    bool var = false;
    for (int k = 0; k < spec_.n_keys; k++) {
        const int c = spec_.build_keys[k];
        if (c < 0 || c >= (int)b.cols.size()) fail(KRV_INVALID_ARGUMENT, "build key column out of range");
        var = var || b.cols[c].type.var();
    }
    if (!var) return;
    if (residual_set_) fail(KRV_UNSUPPORTED, "a residual filter on a join over string or binary keys");
    coded_.reset(new Coded());
    coded_->outer = spec_;
    std::vector<DevCol> meta;
    for (int k = 0; k < spec_.n_keys; k++) {
        const DevCol &c = b.cols[spec_.build_keys[k]];
        DevCol m;
        m.type = c.type;
        m.name = c.name;
        m.nullable = c.nullable || c.valid;
        meta.push_back(m);
    }
    coded_->dict = make_key_dict(rt_, meta);
    // the build side's columns (string key columns stay, as payload), then the code
    const krv_join_spec &o = coded_->outer;
    spec_.n_keys = 1;
    spec_.build_keys[0] = (int32_t)b.cols.size();
    spec_.null_safe[0] = 0;
    spec_.runtime_filter = 0;  // a filter over codes answers nothing outside
    const int nb = o.n_build_out < 0 ? (int)b.cols.size() : o.n_build_out;
    for (int i = 0; i < nb; i++) {
        const int c = o.n_build_out < 0 ? i : o.build_out[i];
        if (c < 0 || c >= (int)b.cols.size()) fail(KRV_INVALID_ARGUMENT, "projection column out of range");
        spec_.build_out[i] = c;
    }
    spec_.n_build_out = nb;
}

__global__ void code_valid_kernel(KeysDev k, int64_t n, uint32_t *bits) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i - (threadIdx.x & 31) < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        bool v = i < n;
        for (int c = 0; c < k.n && v; c++)
            if (!((k.null_safe >> c) & 1u) && !bit_get(k.c[c].valid, k.c[c].voff, i)) v = false;
        const unsigned w = __ballot_sync(0xFFFFFFFFu, v);
        if ((threadIdx.x & 31) == 0) bits[i >> 5] = w;
    }
}

// The batch the table sees: b's columns (string and binary ones included,
// as payload the output can carry), then the key code (NULL where an `=`
// key is NULL: such a row never matches).
DevBatch HashJoin::coded_batch(const DevBatch &b, bool build) {
    const krv_join_spec &o = coded_->outer;
    const int32_t *keys = build ? o.build_keys : o.probe_keys;
    std::vector<int> cols;
    for (int k = 0; k < o.n_keys; k++) {
        if (keys[k] < 0 || keys[k] >= (int)b.cols.size()) fail(KRV_INVALID_ARGUMENT, "key column out of range");
        cols.push_back(keys[k]);
    }
    auto codes = std::make_shared<DBuf>(key_dict_encode(coded_->dict, b, cols, build));
    DevBatch in;
    in.rows = b.rows;
    in.cols = b.cols;
    // validity of the code: every `=` key component valid
    KeysDev kd{};
    kd.n = o.n_keys;
    for (int k = 0; k < o.n_keys; k++) {
        const DevCol &c = b.cols[keys[k]];
        kd.c[k] = KeyColDev{c.data, c.valid, c.valid_off, 8, 0};
        if (o.null_safe[k]) kd.null_safe |= 1u << k;
    }
    auto bits = std::make_shared<DBuf>(rt_, (size_t)ceil_div(std::max<int64_t>(b.rows, 1), 32) * 4 + 8);
    if (b.rows > 0) {
        code_valid_kernel<<<grid_for(rt_, b.rows, 256, 8), 256, 0, rt_->stream>>>(kd, b.rows, bits->as<uint32_t>());
        rt_->launches++;
        check_launch("code_valid_kernel");
    }
    DevCol cc;
    cc.type = DType{Type::I64, 0, 0};
    cc.name = "#key";
    cc.nullable = true;
    cc.length = b.rows;
    cc.hold_data = codes;
    cc.data = codes->get();
    cc.hold_valid = bits;
    cc.valid = bits->as<uint8_t>();
    cc.valid_off = 0;
    in.cols.push_back(cc);
    if (!build && !coded_->probe_mapped) {
        coded_->probe_mapped = true;
        spec_.probe_keys[0] = (int32_t)b.cols.size();
        const int np = o.n_probe_out < 0 ? (int)b.cols.size() : o.n_probe_out;
        for (int i = 0; i < np; i++) {
            const int c = o.n_probe_out < 0 ? i : o.probe_out[i];
            if (c < 0 || c >= (int)b.cols.size()) fail(KRV_INVALID_ARGUMENT, "projection column out of range");
            spec_.probe_out[i] = c;
        }
        spec_.n_probe_out = np;
    }
    return in;
}

void HashJoin::build_push(DevBatch b) {
    if (built_) fail(KRV_INVALID_ARGUMENT, "build_push after build_finish");
    DeviceGuard g(rt_);
    if (!decided_) decide(b);
    if (coded_) b = coded_batch(b, true);
    append_arena(b);
}

DevBatch HashJoin::staged() const {
    DevBatch b;
    b.rows = build_rows_;
    for (size_t i = 0; i < arena_cols_.size(); i++) {
        DevCol c = arena_cols_[i];
        c.length = build_rows_;
        c.hold_data = arena_data_[i];
        c.data = c.hold_data ? c.hold_data->get() : nullptr;
        c.valid = nullptr;
        c.valid_off = 0;
        b.cols.push_back(c);
    }
    return b;
}

HashJoin::TableDev HashJoin::table_dev() const {
    return TableDev{slots_.as<unsigned long long>(), mask_, next_.as<uint32_t>(), spec_.seed};
}

void HashJoin::build_finish() {
    if (built_) fail(KRV_INVALID_ARGUMENT, "build_finish called twice");
    DeviceGuard g(rt_);
    arena_.rows = build_rows_;
    arena_.cols.clear();
    for (size_t i = 0; i < arena_cols_.size(); i++) {
        DevCol c = arena_cols_[i];
        c.length = build_rows_;
        c.hold_data = arena_data_[i];
        c.hold_valid = arena_valid_[i];
        c.data = c.hold_data ? c.hold_data->get() : nullptr;
        c.valid = c.hold_valid ? c.hold_valid->as<uint8_t>() : nullptr;
        c.valid_off = 0;
        arena_.cols.push_back(c);
    }
    const uint64_t want = (uint64_t)std::ceil((double)std::max<int64_t>(build_rows_, 1) / spec_.max_load);
    const uint64_t slots = std::max<uint64_t>(1024, next_pow2(want));
    mask_ = slots - 1;
    // the slots and, after them, the build's counters: one clearing
    slots_ = DBuf(rt_, slots * 8 + 64);
    zero(rt_, slots_.get(), slots * 8 + 64);
    next_ = DBuf(rt_, (size_t)std::max<int64_t>(build_rows_, 1) * 4);
    unsigned long long *ctr = slots_.as<unsigned long long>() + slots;
    const int jt = spec_.join_type;
    const bool preserved = jt == KRV_JOIN_RIGHT_SEMI || jt == KRV_JOIN_RIGHT_ANTI || jt == KRV_JOIN_RIGHT_OUTER ||
                           jt == KRV_JOIN_FULL_OUTER;
    if (preserved) {
        marks_ = DBuf(rt_, (size_t)std::max<int64_t>(build_rows_, 1));
        zero(rt_, marks_.get(), marks_.bytes());
    }
    unsigned long long host_ctr[8] = {};
    if (build_rows_ > 0) {
        if (arena_.cols.empty()) fail(KRV_INVALID_ARGUMENT, "build batches without columns");
        KeysDev k = keys_of(arena_, spec_.build_keys, spec_.n_keys, spec_.null_safe);
        const int grid = grid_for(rt_, ceil_div(build_rows_, fast_keys(k) ? kBuildRowsFast : kBuildRowsAny), kBuildThreads,
                                  fast_keys(k) ? 8 : 16);
        if (fast_keys(k))
            build_kernel<true><<<grid, kBuildThreads, 0, rt_->stream>>>(k, build_rows_, slots_.as<unsigned long long>(),
                                                                       mask_, next_.as<uint32_t>(), spec_.seed, ctr);
        else
            build_kernel<false><<<grid, kBuildThreads, 0, rt_->stream>>>(k, build_rows_, slots_.as<unsigned long long>(),
                                                                        mask_, next_.as<uint32_t>(), spec_.seed, ctr);
        rt_->launches++;
        check_launch("build_kernel");
        read_device(rt_, ctr, 64, host_ctr);
        if (host_ctr[5] & ST_CAPACITY) fail(KRV_INTERNAL, "join table full");
    }
    counters_.build_rows = build_rows_;
    counters_.build_keys = (int64_t)host_ctr[0];
    counters_.table_slots = (int64_t)slots;
    any_null_build_ = host_ctr[1] != 0;
    indexed_rows_ = (int64_t)host_ctr[4];
    // without rows: lo > hi
    key_lo_ = indexed_rows_ ? (long long)(~host_ctr[2] ^ kOrderBit) : LLONG_MAX;
    key_hi_ = indexed_rows_ ? (long long)(host_ctr[3] ^ kOrderBit) : LLONG_MIN;
    // Unique, dense int64 keys (a span of at most 4 values per row): a direct
    // index, 4 bytes per key value, for the probe of inner and left outer joins.
    direct_.reset();
    direct_span_ = 0;
    if (indexed_rows_ > 0 && counters_.build_keys == indexed_rows_ && spec_.n_keys == 1 && !spec_.null_safe[0] &&
        arena_.cols[spec_.build_keys[0]].type.id == Type::I64 &&
        (spec_.join_type == KRV_JOIN_INNER || spec_.join_type == KRV_JOIN_LEFT_OUTER)) {
        const __int128 span = (__int128)key_hi_ - (__int128)key_lo_;
        if (span >= 0 && span < ((__int128)1 << 31) && span < (__int128)4 * indexed_rows_ + 4096) {
            direct_span_ = (unsigned long long)span;
            direct_ = DBuf(rt_, (size_t)(span + 1) * 4);
            KRV_CUDA(cudaMemsetAsync(direct_.get(), 0xFF, direct_.bytes(), rt_->stream));
            KeysDev k = keys_of(arena_, spec_.build_keys, spec_.n_keys, spec_.null_safe);
            direct_build_kernel<<<grid_for(rt_, build_rows_, 256, 8), 256, 0, rt_->stream>>>(
                k, build_rows_, DirectDev{direct_.as<uint32_t>(), key_lo_, direct_span_});
            rt_->launches++;
            check_launch("direct_build_kernel");
        }
    }
    // The runtime filter of a one-key join (BuildSink::publish, join/build.rs:482).
    if (spec_.runtime_filter && spec_.n_keys == 1) {
        const DevCol &key = arena_.cols[spec_.build_keys[0]];
        if (key.type.id == Type::I64) {
            krv_key_filter_options o;
            krv_key_filter_options_default(&o);
            // The build already counted the kept rows, the distinct keys and
            // their range: the filter builder needs no pass of its own unless
            // an exact form may apply.
            KeyStats ks{(int64_t)host_ctr[4], (int64_t)host_ctr[0], key_lo_, key_hi_};
            filter_ = build_key_filter(rt_, o, key, spec_.null_safe[0] ? nullptr : &ks);
        }
    }
    built_ = true;  // only now: a call that failed (for memory, say) may be made again
}

static std::vector<int> projection(int n, const int32_t *cols, int ncols) {
    std::vector<int> v;
    if (n < 0) {
        for (int i = 0; i < ncols; i++) v.push_back(i);
    } else {
        for (int i = 0; i < n; i++) {
            if (cols[i] < 0 || cols[i] >= ncols) fail(KRV_INVALID_ARGUMENT, "projection column out of range");
            v.push_back(cols[i]);
        }
    }
    return v;
}

DevBatch HashJoin::probe(const DevBatch &outer_in) {
    if (!built_) fail(KRV_INVALID_ARGUMENT, "probe before build_finish");
    DeviceGuard g(rt_);
    DevBatch coded_in;
    if (coded_) coded_in = coded_batch(outer_in, false);
    const DevBatch &in = coded_ ? coded_in : outer_in;
    const int jt = spec_.join_type;
    const int64_t n = in.rows;
    emitting_ = n > 0;  // from here on kernels that read the batch are queued, until total() has waited
    counters_.probe_rows += n;
    if (probe_types_.empty()) {
        for (const DevCol &c : in.cols) {
            probe_types_.push_back(c.type);
            probe_names_.push_back(c.name);
            probe_nullable_.push_back(c.nullable);
        }
    }
    KeysDev pk = keys_of(in, spec_.probe_keys, spec_.n_keys, spec_.null_safe);
    KeysDev bk{};
    if (build_rows_ > 0) bk = keys_of(arena_, spec_.build_keys, spec_.n_keys, spec_.null_safe);
    else bk = pk;  // never dereferenced: the table is empty
    for (int c = 0; c < spec_.n_keys; c++) {
        const DevCol &pc = in.cols[spec_.probe_keys[c]];
        if (build_rows_ > 0 && pc.type != arena_.cols[spec_.build_keys[c]].type)
            fail(KRV_INVALID_ARGUMENT, "probe and build key types differ");
    }
    const bool fast = fast_keys(pk);
    if (spec_.has_residual_filter && !residual_set_)
        fail(KRV_INVALID_ARGUMENT, "has_residual_filter is set but no filter was given (krv_join_set_filter)");
    const bool filt = residual_set_;
    const FilterDev fd = filt ? filter_dev(in) : FilterDev{};
    // The lookup over rows [row0, row0 + rows) (row0 a multiple of kTileRows).
    auto launch_lookup = [&](int look, int64_t row0, int64_t rows, uint32_t *head, uint32_t *cnt,
                             unsigned long long *tiles, uint8_t *marks, int pad, int kind, uint32_t *status) {
        if (rows == 0) return;
        ProbeDev A{};
        A.pk = pk;
        for (int k = 0; k < pk.n; k++) {
            A.pk.c[k].data = static_cast<const uint8_t *>(pk.c[k].data) + row0 * pk.c[k].width;
            A.pk.c[k].voff += row0;
        }
        A.bk = bk;
        A.n = rows;
        A.slots = slots_.as<unsigned long long>();
        A.mask = mask_;
        A.next = next_.as<uint32_t>();
        A.seed = spec_.seed;
        A.dir = DirectDev{direct_.as<uint32_t>(), key_lo_, direct_span_};
        A.marks = marks;
        A.pad = pad;
        A.single_match = status ? spec_.single_match : 0;
        A.kind = kind;
        A.build_empty = build_rows_ == 0;
        A.build_has_null = any_null_build_;
        A.head = head;
        A.cnt = cnt;
        A.tiles = tiles;
        A.status = status;
        FilterDev f = fd;  // its probe columns from row0 on
        for (int t = 0; t < f.n; t++)
            for (FilterOpDev *o : {&f.t[t].l, &f.t[t].r})
                if (o->side == 0) {
                    o->data = static_cast<const uint8_t *>(o->data) + row0 * o->width;
                    o->voff += row0;
                }
        const int grid = (int)ceil_div(rows, kTileRows);
        auto go = [&](auto kernel) { kernel<<<grid, kProbeThreads, 0, rt_->stream>>>(A, f); };
        auto by_keys = [&](auto l) {
            constexpr int L = decltype(l)::value;
            if (fast && filt) go(lookup_kernel<1, true, L>);
            else if (fast) go(lookup_kernel<1, false, L>);
            else if (filt) go(lookup_kernel<0, true, L>);
            else if (pk.n == 2) go(lookup_kernel<2, false, L>);
            else go(lookup_kernel<0, false, L>);
        };
        if (look == kDirect) go(lookup_kernel<1, false, kDirect>);
        else if (look == kUnique) by_keys(std::integral_constant<int, kUnique>{});
        else if (look == kChains) by_keys(std::integral_constant<int, kChains>{});
        else by_keys(std::integral_constant<int, kRowsOnly>{});
        rt_->launches++;
        check_launch("lookup_kernel");
    };
    bool long_tiles = false;  // tiles of more than kWindow output rows (known once the total is)
    auto launch_emit = [&](int look, const EmitDev &E, const OutDev &od) {
        if (E.rows == 0 || od.n == 0) return;
        const int grid = (int)ceil_div(E.rows, kTileRows);
        if (long_tiles) {
            if (filt) emit_long_kernel<true><<<grid * kLongParts, kProbeThreads, 0, rt_->stream>>>(E, od, fd);
            else emit_long_kernel<false><<<grid * kLongParts, kProbeThreads, 0, rt_->stream>>>(E, od, fd);
            rt_->launches++;
            check_launch("emit_long_kernel");
        }
        if (look == kChains && filt) emit_kernel<true, kChains><<<grid, kProbeThreads, 0, rt_->stream>>>(E, od, fd);
        else if (look == kChains) emit_kernel<false, kChains><<<grid, kProbeThreads, 0, rt_->stream>>>(E, od, fd);
        else if (look == kRowsOnly) emit_kernel<false, kRowsOnly><<<grid, kProbeThreads, 0, rt_->stream>>>(E, od, fd);
        else emit_kernel<false, kUnique><<<grid, kProbeThreads, 0, rt_->stream>>>(E, od, fd);
        rt_->launches++;
        check_launch("emit_kernel");
    };
    // unique build keys: at most one output row per probe row
    const bool unique_keys = build_rows_ > 0 && counters_.build_keys == indexed_rows_;
    const int look = !unique_keys ? kChains : fast && !filt && direct_.get() ? kDirect : kUnique;
    const auto pcols = projection(spec_.n_probe_out, spec_.probe_out, (int)in.cols.size());
    const auto bcols = projection(spec_.n_build_out, spec_.build_out, (int)arena_cols_.size());
    const int threads = 256;
    const int grid = grid_for(rt_, n, threads, 8);
    const auto *slots = slots_.as<unsigned long long>();
    DevBatch out;

    if (jt == KRV_JOIN_EXISTENCE) {
        out.rows = n;
        for (int pc : pcols) {
            const DevCol &s = in.cols[pc];
            if (s.type.var()) {
                out.cols.push_back(var_gather(rt_, var_src(0, pc, &in), nullptr, n, s.type, s.nullable || s.valid, s.name));
                continue;
            }
            DevCol d = make_col(rt_, s.type, n, s.nullable || s.valid, s.name);
            const size_t bytes = s.type.id == Type::Bool ? (size_t)ceil_div(n, 8) : (size_t)n * s.type.width();
            if (bytes) KRV_CUDA(cudaMemcpyAsync(const_cast<void *>(d.data), s.data, bytes, cudaMemcpyDeviceToDevice, rt_->stream));
            if (d.valid) {
                zero(rt_, const_cast<uint8_t *>(d.valid), d.hold_valid->bytes());
                append_bits(rt_, s.valid, s.valid_off, n, const_cast<uint8_t *>(d.valid), 0);
            }
            out.cols.push_back(d);
        }
        DevCol ex = make_col(rt_, DType{Type::Bool, 0, 0}, n, false, "exists");
        zero(rt_, const_cast<void *>(ex.data), ex.hold_data->bytes());
        if (n > 0) {
            const uint32_t *nx = next_.as<uint32_t>();
            uint32_t *exw = (uint32_t *)ex.data;
            const int empty = build_rows_ == 0;
            if (fast && filt)
                probe_exists_kernel<true, true><<<grid, threads, 0, rt_->stream>>>(pk, bk, n, slots, mask_, spec_.seed,
                                                                                   exw, empty, nx, fd);
            else if (fast)
                probe_exists_kernel<true, false><<<grid, threads, 0, rt_->stream>>>(pk, bk, n, slots, mask_, spec_.seed,
                                                                                    exw, empty, nx, fd);
            else if (filt)
                probe_exists_kernel<false, true><<<grid, threads, 0, rt_->stream>>>(pk, bk, n, slots, mask_, spec_.seed,
                                                                                    exw, empty, nx, fd);
            else
                probe_exists_kernel<false, false><<<grid, threads, 0, rt_->stream>>>(pk, bk, n, slots, mask_,
                                                                                     spec_.seed, exw, empty, nx, fd);
            rt_->launches++;
            check_launch("probe_exists_kernel");
        }
        out.cols.push_back(ex);
        counters_.output_rows += n;
        remember_shape(out);
        return out;
    }

    const bool pairs = jt == KRV_JOIN_INNER || jt == KRV_JOIN_LEFT_OUTER || jt == KRV_JOIN_RIGHT_OUTER ||
                       jt == KRV_JOIN_FULL_OUTER;
    if (!pairs && (jt == KRV_JOIN_RIGHT_SEMI || jt == KRV_JOIN_RIGHT_ANTI)) {
        // Probe only marks build rows; output comes at finish.
        if (n > 0 && build_rows_ > 0) {
            launch_lookup(look, 0, n, nullptr, nullptr, nullptr, marks_.as<uint8_t>(), 0, 0, nullptr);
        }
        // Nothing is emitted by this batch: an empty batch of the output shape.
        DevBatch empty;
        for (int bc : bcols) empty.cols.push_back(empty_col(arena_cols_[bc]));
        return empty;
    }

    const bool build_nullable = jt == KRV_JOIN_LEFT_OUTER || jt == KRV_JOIN_FULL_OUTER;
    const bool probe_nullable = jt == KRV_JOIN_RIGHT_OUTER || jt == KRV_JOIN_FULL_OUTER;
    const bool pads = jt == KRV_JOIN_LEFT_OUTER || jt == KRV_JOIN_FULL_OUTER;
    const int kind = jt == KRV_JOIN_LEFT_SEMI ? 0 : jt == KRV_JOIN_LEFT_ANTI ? 1 : 2;
    const int how = pairs ? look : kRowsOnly;
    const bool none = n == 0 || (pairs && build_rows_ == 0 && !pads);  // no output rows
    uint8_t *marks = marks_.get() ? marks_.as<uint8_t>() : nullptr;
    const int64_t ntiles = ceil_div(n, (int64_t)kTileRows);
    DBuf head, cnt, tiles, status;
    int64_t chunk = n;  // rows looked up and emitted together
    bool kept = true;   // every row's lookup is kept until it is emitted
    // Otherwise rows are looked up again, a chunk at a time, when they are emitted.
    auto keep_a_chunk = [&] {
        kept = false;
        head = DBuf();
        cnt = DBuf();
        chunk = std::min(n, std::min<int64_t>(64, ceil_div(ntiles, (int64_t)64)) * kTileRows);
        head = DBuf(rt_, (size_t)chunk * 4);
        if (how == kChains) cnt = DBuf(rt_, (size_t)chunk * 4);
    };
    if (!none) {
        if (spec_.single_match) {
            status = DBuf(rt_, 8);
            zero(rt_, status.get(), 8);
        }
        tiles = DBuf(rt_, (size_t)ntiles * 8);
        try {
            head = DBuf(rt_, (size_t)n * 4);
            if (how == kChains) cnt = DBuf(rt_, (size_t)n * 4);
        } catch (const Error &e) {
            if (e.code != KRV_NEED_MEMORY) throw;
            keep_a_chunk();
        }
        launch_lookup(how, 0, n, kept ? head.as<uint32_t>() : nullptr, kept && how == kChains ? cnt.as<uint32_t>() : nullptr,
                      tiles.as<unsigned long long>(), pairs ? marks : nullptr, pads && pairs, kind, status.as<uint32_t>());
        tile_scan_kernel<<<1, kScanThreads, 0, rt_->stream>>>(
            tiles.as<unsigned long long>(), ntiles, status.as<uint32_t>(),
            reinterpret_cast<volatile unsigned long long *>(static_cast<uint8_t *>(rt_->status_host_dev) + 64));
        rt_->launches++;
        check_launch("tile_scan_kernel");
    }
    auto total = [&]() -> int64_t {  // waits for the scan
        if (none) return 0;
        KRV_CUDA(cudaStreamSynchronize(rt_->stream));
        emitting_ = false;
        volatile unsigned long long *seen =
            reinterpret_cast<volatile unsigned long long *>(static_cast<uint8_t *>(rt_->status_host) + 64);
        if (seen[1] & ST_TOO_MANY)
            fail(KRV_TOO_MANY_ROWS, "SCALAR_SUBQUERY_TOO_MANY_ROWS: a probe row matched more than one build row");
        long_tiles = seen[2] != 0;
        return (int64_t)seen[0];
    };
    // The output columns for m rows, and the kernel that fills them.
    std::vector<VarOut> vars;  // string columns, gathered once the row indexes are known
    DBuf idx[2];
    auto emit = [&](int64_t m) {
        out = DevBatch{};
        vars.clear();
        OutDev od{};
        EmitDev E{};
        auto column = [&](const DevCol &s, const DType &type, const std::string &name, const uint8_t *src_valid, int side,
                          int col, bool nullable) {
            if (type.var()) {
                DevCol meta;
                meta.type = type;
                meta.name = name;
                meta.nullable = nullable;
                vars.push_back(VarOut{(int)out.cols.size(), side, col});
                out.cols.push_back(meta);
                return;
            }
            DevCol d = make_col(rt_, type, m, nullable, name);
            if (d.valid) zero(rt_, const_cast<uint8_t *>(d.valid), d.hold_valid->bytes());
            od.c[od.n++] = OutColDev{s.data, src_valid, s.valid_off, const_cast<void *>(d.data), (uint32_t *)d.valid,
                                     type.width(), side};
            out.cols.push_back(d);
        };
        for (int pc : pcols) {
            const DevCol &s = in.cols[pc];
            if (s.type.id == Type::Bool) fail(KRV_UNSUPPORTED, "boolean probe payload columns");
            column(s, s.type, s.name, s.valid, 0, pc, s.nullable || s.valid || probe_nullable);
        }
        if (pairs)
            for (int bc : bcols) {
                const DevCol s = arena_.cols.empty() ? DevCol{} : arena_.cols[bc];
                const DevCol &meta = arena_cols_[bc];
                column(s, meta.type, meta.name, meta.nullable ? s.valid : nullptr, 1, bc, meta.nullable || build_nullable);
            }
        for (const VarOut &v : vars)
            if (!idx[v.side].get()) idx[v.side] = DBuf(rt_, (size_t)std::max<int64_t>(m, 1) * 8);
        for (int side = 0; side < 2; side++)
            if (idx[side].get()) od.c[od.n++] = OutColDev{nullptr, nullptr, 0, idx[side].get(), nullptr, 8, 3 + side};
        if (m == 0 || none) return;
        for (int64_t row0 = 0; row0 < n; row0 += chunk) {
            const int64_t rows = std::min(chunk, n - row0);
            if (!kept)
                launch_lookup(how, row0, rows, head.as<uint32_t>(), how == kChains ? cnt.as<uint32_t>() : nullptr, nullptr,
                              nullptr, pads && pairs, kind, nullptr);
            E.row0 = row0;
            E.rows = rows;
            E.head = head.as<uint32_t>();
            E.cnt = cnt.as<uint32_t>();
            E.tiles = tiles.as<unsigned long long>() + row0 / kTileRows;
            E.next = next_.as<uint32_t>();
            E.pad = pads && pairs;
            emitting_ = true;
            launch_emit(how, E, od);
        }
    };
    // Where a probe row has at most one output row, columns of n rows hold
    // the output and one wait, after everything is queued, tells its size.
    // Duplicate build keys wait for the size first.
    int64_t m = -1;
    if (how != kChains) {
        try {
            emit(n);
        } catch (const Error &e) {
            if (e.code != KRV_NEED_MEMORY) throw;
            idx[0] = DBuf();
            idx[1] = DBuf();
            m = total();  // the rows there are may still fit
        }
    } else {
        m = total();
    }
    if (m < 0) {
        m = total();
    } else {
        try {
            emit(m);
        } catch (const Error &e) {
            // the lookups' memory may be what the output lacks
            if (e.code != KRV_NEED_MEMORY || none || !kept) throw;
            out = DevBatch{};
            idx[0] = DBuf();
            idx[1] = DBuf();
            keep_a_chunk();
            emit(m);
        }
    }
    out.rows = m;
    for (DevCol &c : out.cols) c.length = m;
    for (const VarOut &v : vars) {
        const DevCol meta = out.cols[v.pos];
        emitting_ = emitting_ || (v.side == 0 && m > 0);
        out.cols[v.pos] = var_gather(rt_, var_src(v.side, v.col, &in), idx[v.side].as<long long>(), m, meta.type,
                                     meta.nullable, meta.name);
    }
    counters_.output_rows += m;
    remember_shape(out);
    return out;
}

DevBatch HashJoin::finish() {
    if (!built_) fail(KRV_INVALID_ARGUMENT, "finish before build_finish");
    DeviceGuard g(rt_);
    const int jt = spec_.join_type;
    const bool tail = jt == KRV_JOIN_RIGHT_SEMI || jt == KRV_JOIN_RIGHT_ANTI || jt == KRV_JOIN_RIGHT_OUTER ||
                      jt == KRV_JOIN_FULL_OUTER;
    if (!tail || finished_) {
        // Nothing waits for the end: an empty batch of the probe output's shape.
        finished_ = true;
        DevBatch empty;
        for (const DevCol &m : out_meta_) empty.cols.push_back(empty_col(m));
        return empty;
    }
    const bool with_probe = jt == KRV_JOIN_RIGHT_OUTER || jt == KRV_JOIN_FULL_OUTER;
    if (with_probe && probe_types_.empty())
        fail(KRV_INVALID_ARGUMENT, "an outer join's tail needs the probe schema: probe at least one batch");
    const auto bcols = projection(spec_.n_build_out, spec_.build_out, (int)arena_cols_.size());
    std::vector<int> pcols;
    if (with_probe) pcols = projection(spec_.n_probe_out, spec_.probe_out, (int)probe_types_.size());
    const unsigned long long cap = (unsigned long long)std::max<int64_t>(build_rows_, 1);
    DevBatch out;
    OutDev od{};
    std::vector<VarOut> vars;
    for (int pc : pcols) {
        if (probe_types_[pc].var()) {
            DevCol m;
            m.type = probe_types_[pc];
            m.name = probe_names_[pc];
            m.nullable = true;
            vars.push_back(VarOut{(int)out.cols.size(), 0, pc});
            out.cols.push_back(m);
            continue;
        }
        DevCol d = make_col(rt_, probe_types_[pc], (int64_t)cap, true, probe_names_[pc]);
        zero(rt_, const_cast<uint8_t *>(d.valid), d.hold_valid->bytes());
        od.c[od.n++] = OutColDev{nullptr, nullptr, 0, const_cast<void *>(d.data), (uint32_t *)d.valid,
                                 probe_types_[pc].width(), 2};
        out.cols.push_back(d);
    }
    for (int bc : bcols) {
        const DevCol &meta = arena_cols_[bc];
        const DevCol &s = arena_.cols[bc];
        const bool nullable = meta.nullable || jt == KRV_JOIN_FULL_OUTER;
        if (meta.type.var()) {
            DevCol m;
            m.type = meta.type;
            m.name = meta.name;
            m.nullable = nullable;
            vars.push_back(VarOut{(int)out.cols.size(), 1, bc});
            out.cols.push_back(m);
            continue;
        }
        DevCol d = make_col(rt_, meta.type, (int64_t)cap, nullable, meta.name);
        if (d.valid) zero(rt_, const_cast<uint8_t *>(d.valid), d.hold_valid->bytes());
        od.c[od.n++] = OutColDev{s.data, meta.nullable ? s.valid : nullptr, 0, const_cast<void *>(d.data),
                                 (uint32_t *)d.valid, meta.type.width(), 1};
        out.cols.push_back(d);
    }
    DBuf idx[2];
    for (const VarOut &v : vars)
        if (!idx[v.side].get()) {
            idx[v.side] = DBuf(rt_, (size_t)cap * 8);
            od.c[od.n++] = OutColDev{nullptr, nullptr, 0, idx[v.side].get(), nullptr, 8, 3 + v.side};
        }
    DBuf cnt(rt_, 8);
    zero(rt_, cnt.get(), 8);
    if (build_rows_ > 0) {
        KeysDev bk = keys_of(arena_, spec_.build_keys, spec_.n_keys, spec_.null_safe);
        const int threads = 256;
        tail_kernel<<<grid_for(rt_, build_rows_, threads, 8), threads, 0, rt_->stream>>>(
            build_rows_, marks_.as<uint8_t>(), bk, jt == KRV_JOIN_RIGHT_SEMI ? 0 : 1, od, cap,
            cnt.as<unsigned long long>());
        rt_->launches++;
        check_launch("tail_kernel");
    }
    out.rows = (int64_t)read_scalar<unsigned long long>(rt_, cnt.get());
    for (DevCol &c : out.cols) c.length = out.rows;
    for (const VarOut &v : vars) {
        const DevCol m = out.cols[v.pos];
        // the tail's probe side is all NULL: its string columns read nothing
        const VarSrc src = v.side == 1 ? var_src(1, v.col, nullptr) : VarSrc{};
        out.cols[v.pos] = var_gather(rt_, src, idx[v.side].as<long long>(), out.rows, m.type, m.nullable, m.name);
    }
    counters_.output_rows += out.rows;
    finished_ = true;  // only now: a call that failed may be made again
    return out;
}

}  // namespace krv
