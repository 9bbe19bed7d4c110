// star_fused.cuh -- the fact-side kernels of the star-join pipeline.
//
// Dimension B's runtime filter is first evaluated once for every value of
// its key range [lo, hi] into an answer bitmap (bit v - lo = whether the
// filter passes v: the Bloom's answer, false positives included), staged in
// shared memory when it fits; a row's B test is then one bit. Without a
// bitmap the kernels probe the filter itself (range, then Bloom block or
// exact set).
//
// A dimension with unique keys over a range of at most 2^26 values also gets a
// direct index: its attribute's group id at key - lo (one byte or two, -1 =
// absent), so a probe is one L2 read instead of a hash-slot read and a key
// read. Otherwise the join's hash table is probed.
//
// Two kernels, so neither waits on the other's latency:
//  1. star_scan_kernel streams fk_b (a warp 2 KB contiguous, each load 512
//     bytes of it, the next tile prefetched into registers), tests B's filter
//     without a branch, and appends the passing rows (row, fk_b) to its CTA's
//     region of a survivor list, a loop turn per lane and passing row. Bound by
//     its instructions until few enough are left for the memory: 300M rows, 5%
//     passing, on B200 take 0.45 ms (5.4 TB/s) at 290 instructions a warp and
//     256 rows; 0.55 ms at 434 with 64-byte lane strides and an unrolled
//     append, 0.65 ms at 523 with a ballot per row;
//  2. star_join_kernel takes one survivor per thread over many CTAs: reads
//     fk_a, tests A's filter, looks both dimensions up and adds
//     price * (1 - discount) of each joined row to its group's accumulator.
// The fact side moves all of fk_b, the 32-byte sectors of fk_a holding a row
// that passed B's filter, price/discount of joined rows, and the survivor
// list (written once, read once).
#pragma once

#include <type_traits>

#include "krv_device.cuh"
#include "krv_filter.cuh"
#include "ops.h"

namespace krv {

constexpr int kScanThreads = 1024;                        // threads per scan CTA
constexpr int kScanRows = 8;                              // rows per lane per tile
constexpr int kScanTile = kScanThreads * kScanRows;       // 8192 rows
constexpr int kJoinThreads = 512;                         // threads per join CTA
constexpr uint32_t kStarNone = 0xFFFFFFFFu;

struct StarTable {
    const unsigned long long *slots;
    uint64_t mask;
    const uint32_t *next;
    uint64_t seed;
    const long long *keys;  // build key column
    const int32_t *gid;     // dense group id of each build row's attribute
};

// key -> group id of a dimension with unique keys: gid at key - lo.
struct StarDirect {
    const void *gid;  // int8_t or int16_t per key value, -1 = no row
    long long lo;
    unsigned long long span;  // hi - lo
    int width;                // 1 or 2 (0: none)
};

struct StarArgs {
    const long long *fk_a, *fk_b, *price;
    const double *disc;
    int64_t n;
    KeyFilterDev fa, fb;
    const uint32_t *bits_b;  // B's answer bitmap over [fb.lo, fb.hi]
    int use_filters;
    int group_by;  // 0: dim A's attribute, 1: dim B's
    StarTable ta, tb;
    StarDirect da, db;
    int ngroups;
    int bits_b_smem_words;  // B's answer bitmap words staged in shared memory
    double *sum_hi, *sum_lo;
    unsigned long long *cnt;
    unsigned long long *stats;  // [0] rows passing both filters, [1] joined rows, [2] fk_a sectors read
    // Survivor list: CTA c of the scan owns entries [c * region, (c + 1) * region).
    uint32_t *surv_row;
    uint32_t *surv_kb32;   // fk_b - fb.lo (when B's range is below 2^32)
    long long *surv_kb64;  // fk_b (otherwise)
    uint64_t region;
    unsigned long long *region_count;
    // Validity bitmaps of the fact columns (null: no NULLs) and the bit of
    // row 0 in each. A NULL key never joins (join/keys.rs:17-19); a NULL
    // price or discount makes the row's value NULL, which SUM skips: the row
    // still joins and counts, and adds one to its group's `nulls`.
    const uint8_t *v_fk_a, *v_fk_b, *v_price, *v_disc;
    int64_t o_fk_a, o_fk_b, o_price, o_disc;
    unsigned long long *nulls;
};

__device__ __forceinline__ uint32_t star_lookup(const StarTable &t, long long k) {
    const uint64_t g = finalize(hash_word((uint64_t)k), t.seed);
    const uint32_t tag = slot_tag(g);
    uint64_t pos = g & t.mask;
    for (uint64_t p = 0; p <= t.mask; p++) {
        const unsigned long long s = __ldg(t.slots + pos);
        if (s == 0) return kStarNone;
        if (slot_matches(s, tag)) {
            const uint32_t o = slot_row(s);
            if (__ldg(t.keys + o) == k) return o;
        }
        pos = (pos + 1) & t.mask;
    }
    return kStarNone;
}

__device__ __forceinline__ int star_direct(const StarDirect &d, long long k) {
    const unsigned long long off = (unsigned long long)(k - d.lo);
    if (off > d.span) return -1;
    return d.width == 1 ? (int)__ldg(static_cast<const int8_t *>(d.gid) + off)
                        : (int)__ldg(static_cast<const int16_t *>(d.gid) + off);
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
    return v;
}

// A lane's rows of its warp's 256 rows from `wb` on: row 64j + 2 lane + k at
// v[2j + k], so that each load of the warp covers 512 contiguous bytes.
__device__ __forceinline__ int64_t star_row(int64_t wb, int lane, int u) { return wb + (u >> 1) * 64 + 2 * lane + (u & 1); }
template <bool VEC>
__device__ __forceinline__ void star_load_tile(const StarArgs &A, int64_t wb, int lane, long long (&v)[kScanRows]) {
    if (VEC && wb + 32 * kScanRows <= A.n) {
        const longlong2 *p = reinterpret_cast<const longlong2 *>(A.fk_b + wb) + lane;
#pragma unroll
        for (int j = 0; j < kScanRows / 2; j++) {
            const longlong2 x = __ldcs(p + 32 * j);
            v[2 * j] = x.x;
            v[2 * j + 1] = x.y;
        }
    } else {
#pragma unroll
        for (int u = 0; u < kScanRows; u++) v[u] = star_row(wb, lane, u) < A.n ? __ldcs(A.fk_b + star_row(wb, lane, u)) : 0;
    }
}

// ---- stage 1 ------------------------------------------------------------------------
// BMODE 1: B's answer bitmap in shared memory; 0: B's filter probed per row.
// KB32: survivors keep fk_b - lo in 32 bits.
// NULLS: fact columns with validity bitmaps (compiled apart, so the kernel for
// columns without NULLs tests no bits).
template <int BMODE, bool VEC, bool KB32, bool NULLS>
__global__ void __launch_bounds__(kScanThreads, 1) star_scan_kernel(StarArgs A) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t *s_bits = reinterpret_cast<uint32_t *>(smem);
    __shared__ unsigned s_fill;
    __shared__ unsigned long long s_sectors;
    const int tid = threadIdx.x, lane = tid & 31;
    if (BMODE == 1) {
        const uint4 *src = reinterpret_cast<const uint4 *>(A.bits_b);
        uint4 *dst = reinterpret_cast<uint4 *>(s_bits);
        for (int w = tid; w < A.bits_b_smem_words / 4; w += kScanThreads) dst[w] = src[w];
    }
    if (tid == 0) {
        s_fill = 0;
        s_sectors = 0;
    }
    __syncthreads();
    const long long blo = A.fb.lo;
    const unsigned long long bspan = (unsigned long long)(A.fb.hi - A.fb.lo);
    // this CTA's region of the survivor list
    uint32_t *out_row = A.surv_row + (uint64_t)blockIdx.x * A.region;
    uint32_t *out_kb32 = A.surv_kb32 + (uint64_t)blockIdx.x * A.region;
    long long *out_kb64 = A.surv_kb64 + (uint64_t)blockIdx.x * A.region;
    unsigned long long sectors = 0;

    auto take = [&](int64_t wb, const long long (&cur)[kScanRows], auto full) {
        // The rows that pass B's filter, a bit each. The bitmap's range has
        // fewer than 2^28 values: an offset outside it is clamped into it for
        // the load, so that no row branches.
        uint32_t off[kScanRows];
        unsigned m = 0;
#pragma unroll
        for (int u = 0; u < kScanRows; u++) {
            const unsigned long long d = (unsigned long long)(cur[u] - blo);
            off[u] = (uint32_t)d;
            bool p = true;
            if (BMODE == 1) {
                const uint32_t o = min(off[u], (uint32_t)bspan);
                p = (d <= bspan) & ((s_bits[o >> 5] >> (o & 31)) & 1u);
            } else if (A.use_filters) {
                p = filter_pass(A.fb, cur[u]);
            }
            m |= (unsigned)p << u;
        }
        if (!full || NULLS) {
#pragma unroll
            for (int u = 0; u < kScanRows; u++) {
                const int64_t r = star_row(wb, lane, u);
                if (r >= A.n || (NULLS && !bit_get(A.v_fk_b, A.o_fk_b, r))) m &= ~(1u << u);
            }
        }
        // fk_a's 32-byte sectors of the passing rows (4 rows: two lanes' pairs) will be read by stage 2.
        unsigned pairs = (m | (m >> 1)) & 0x55u;
        pairs |= __shfl_xor_sync(0xFFFFFFFFu, pairs, 1);
        sectors += __popc(pairs);  // by both lanes: halved at the end
        // Append the passing rows to this CTA's region: one shared atomic per warp.
        const int np = __popc(m);
        int incl = np;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += y;
        }
        unsigned base = 0;
        if (lane == 31 && incl) base = atomicAdd(&s_fill, (unsigned)incl);
        unsigned pos = __shfl_sync(0xFFFFFFFFu, base, 31) + (unsigned)(incl - np);
        while (m) {
            const int u = __ffs(m) - 1;
            m &= m - 1;
            const int64_t r = star_row(wb, lane, u);
            out_row[pos] = (uint32_t)r;
            if (KB32) {
                const uint32_t x0 = u & 1 ? off[1] : off[0], x1 = u & 1 ? off[3] : off[2];
                const uint32_t x2 = u & 1 ? off[5] : off[4], x3 = u & 1 ? off[7] : off[6];
                const uint32_t y0 = u & 2 ? x1 : x0, y1 = u & 2 ? x3 : x2;
                out_kb32[pos] = u & 4 ? y1 : y0;
            } else {
                out_kb64[pos] = A.fk_b[r];
            }
            pos++;
        }
    };
    auto step = [&](int64_t wb, const long long (&cur)[kScanRows]) {
        if (wb + 32 * kScanRows <= A.n) take(wb, cur, std::true_type());
        else take(wb, cur, std::false_type());
    };
    static_assert(kScanRows == 8, "take selects among eight offsets");

    const int64_t tstride = (int64_t)gridDim.x * kScanTile;
    int64_t wb = (int64_t)blockIdx.x * kScanTile + (tid >> 5) * (32 * kScanRows);
    long long v0[kScanRows], v1[kScanRows];  // in turn: one is taken while the other's loads are on their way
    if (wb < A.n) star_load_tile<VEC>(A, wb, lane, v0);
    while (wb < A.n) {
        if (wb + tstride < A.n) star_load_tile<VEC>(A, wb + tstride, lane, v1);
        step(wb, v0);
        wb += tstride;
        if (wb >= A.n) break;
        if (wb + tstride < A.n) star_load_tile<VEC>(A, wb + tstride, lane, v0);
        step(wb, v1);
        wb += tstride;
    }
    sectors = warp_sum(sectors) / 2;
    if (lane == 0 && sectors) atomicAdd(&s_sectors, sectors);
    __syncthreads();
    if (tid == 0) {
        A.region_count[blockIdx.x] = s_fill;
        if (s_sectors) atomicAdd(A.stats + 2, s_sectors);
    }
}

// ---- stage 2 ------------------------------------------------------------------------
// price * (1 - discount) of a row is NULL.
__device__ __forceinline__ bool star_value_null(const StarArgs &A, uint32_t row) {
    return (A.v_price && !bit_get(A.v_price, A.o_price, row)) || (A.v_disc && !bit_get(A.v_disc, A.o_disc, row));
}

// Adds v to the group of one joined pair: this warp's own accumulators in
// shared memory (lanes take turns, plain compensated adds: float64 atomics
// in shared memory are compare-and-swap loops) or, past them, the global ones.
__device__ __forceinline__ void star_add_plain(const StarArgs &A, int g, double v, double *w_hi, double *w_lo,
                                               unsigned long long *w_cnt, int G) {
    if (g < G) {
        double s, e;
        two_sum(w_hi[g], v, s, e);
        w_hi[g] = s;
        w_lo[g] = __dadd_rn(w_lo[g], e);
        w_cnt[g] += 1;
    } else {
        atomic_add_dd(A.sum_hi + g, A.sum_lo + g, v);
        atomicAdd(A.cnt + g, 1ull);
    }
}

// A's filter test of K keys at once: with a Bloom form the K block loads
// are issued together.
template <int K>
__device__ __forceinline__ void star_filterk(const KeyFilterDev &f, const long long (&k)[K], const bool (&has)[K],
                                             bool (&pass)[K]) {
    if (f.form == KRV_FILTER_BLOOM) {
        uint4 w0[K], w1[K];
        uint32_t key[K];
        bool in[K];
#pragma unroll
        for (int j = 0; j < K; j++) {
            in[j] = has[j] && !(f.has_range && (k[j] < f.lo || k[j] > f.hi));
            const uint64_t h = xxh64_u64((uint64_t)k[j]);
            key[j] = (uint32_t)h;
            const uint32_t *blk = f.bloom + (size_t)__umulhi((uint32_t)(h >> 32), (uint32_t)f.nblocks) * 8;
            if (in[j]) {
                w0[j] = __ldg(reinterpret_cast<const uint4 *>(blk));
                w1[j] = __ldg(reinterpret_cast<const uint4 *>(blk) + 1);
            }
        }
#pragma unroll
        for (int j = 0; j < K; j++) {
            const uint32_t miss = (sbbf_bit(key[j], 0) & ~w0[j].x) | (sbbf_bit(key[j], 1) & ~w0[j].y) |
                                  (sbbf_bit(key[j], 2) & ~w0[j].z) | (sbbf_bit(key[j], 3) & ~w0[j].w) |
                                  (sbbf_bit(key[j], 4) & ~w1[j].x) | (sbbf_bit(key[j], 5) & ~w1[j].y) |
                                  (sbbf_bit(key[j], 6) & ~w1[j].z) | (sbbf_bit(key[j], 7) & ~w1[j].w);
            pass[j] = in[j] && miss == 0;
        }
    } else {
#pragma unroll
        for (int j = 0; j < K; j++) pass[j] = has[j] && filter_pass(f, k[j]);
    }
}

// DIRECT: both dimensions have direct indexes; KB32 as in the scan. Each
// thread takes two survivors per step, each stage's loads issued together,
// so a thread keeps two probe chains in flight beside the loads of the next
// two steps. Bound by DRAM, which reads some 120 bytes for each sparse fk_a
// (15M survivors of 300M rows: 0.35 ms, 2.0 GB; 0.37 ms without the loads
// ahead; cache hints of the fk_a load change neither).
template <bool DIRECT, bool KB32, bool NULLS>
__global__ void __launch_bounds__(kJoinThreads, 2) star_join_kernel(StarArgs A, int regions, int slices, int G) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kWarps = kJoinThreads / 32;
    constexpr int kK = 2;
    constexpr int kStep = kK * kJoinThreads;
    double *s_hi = reinterpret_cast<double *>(smem);
    double *s_lo = s_hi + kWarps * G;
    unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(s_lo + kWarps * G);
    __shared__ unsigned long long s_stat[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kWarps * G; i += kJoinThreads) {
        s_hi[i] = 0.0;
        s_lo[i] = 0.0;
        s_cnt[i] = 0;
    }
    if (tid < 2) s_stat[tid] = 0;
    __syncthreads();
    double *w_hi = s_hi + warp * G, *w_lo = s_lo + warp * G;
    unsigned long long *w_cnt = s_cnt + warp * G;
    unsigned long long passed = 0, joined = 0;
    const int r = blockIdx.x % regions, slice = blockIdx.x / regions;
    const uint64_t base0 = (uint64_t)r * A.region;
    const unsigned long long count = A.region_count[r];
    // The list entries of the step after next and fk_a of the next step are
    // on their way while a step is worked on.
    using Off = typename std::conditional<KB32, uint32_t, long long>::type;
    const Off *list_kb;
    if constexpr (KB32) list_kb = A.surv_kb32 + base0;
    else list_kb = A.surv_kb64 + base0;
    const uint32_t *list_row = A.surv_row + base0;
    const unsigned long long stride = (unsigned long long)slices * kStep;
    uint32_t row1[kK], row2[kK];
    Off off1[kK], off2[kK];
    long long ka1[kK];
    auto entries = [&](unsigned long long b, uint32_t (&row)[kK], Off (&off)[kK]) {
#pragma unroll
        for (int j = 0; j < kK; j++) {
            const unsigned long long e = b + (unsigned long long)j * kJoinThreads + tid;
            row[j] = e < count ? __ldcs(list_row + e) : 0u;
            off[j] = e < count ? __ldcs(list_kb + e) : Off(0);
        }
    };
    auto keys_a = [&](unsigned long long b, const uint32_t (&row)[kK], long long (&ka)[kK]) {
#pragma unroll
        for (int j = 0; j < kK; j++) ka[j] = b + (unsigned long long)j * kJoinThreads + tid < count ? __ldcs(A.fk_a + row[j]) : 0;
    };
    const unsigned long long b0 = (unsigned long long)slice * kStep;
    entries(b0, row1, off1);
    entries(b0 + stride, row2, off2);
    keys_a(b0, row1, ka1);
    for (unsigned long long b = b0; b < count; b += stride) {
        bool has[kK], pa[kK], hit[kK];
        uint32_t row[kK];
        long long ka[kK], kb[kK];
        int g[kK];
        double v[kK];
#pragma unroll
        for (int j = 0; j < kK; j++) {
            has[j] = b + (unsigned long long)j * kJoinThreads + tid < count;
            row[j] = row1[j];
            ka[j] = ka1[j];
            kb[j] = !has[j] ? 0 : KB32 ? A.fb.lo + (long long)off1[j] : (long long)off1[j];
            row1[j] = row2[j];
            off1[j] = off2[j];
        }
        keys_a(b + stride, row1, ka1);
        entries(b + 2 * stride, row2, off2);
        // Loads are issued a level at a time for both entries; B's direct
        // index needs only fk_b, A's runs beside A's filter.
        int ga[kK], gb[kK];
#pragma unroll
        for (int j = 0; j < kK; j++) {
            if (DIRECT) gb[j] = has[j] ? star_direct(A.db, kb[j]) : -1;
        }
        if (DIRECT) {
#pragma unroll
            for (int j = 0; j < kK; j++) ga[j] = has[j] ? star_direct(A.da, ka[j]) : -1;
        }
        if (A.use_filters) star_filterk<kK>(A.fa, ka, has, pa);
        else {
#pragma unroll
            for (int j = 0; j < kK; j++) pa[j] = has[j];
        }
        if (NULLS) {
#pragma unroll
            for (int j = 0; j < kK; j++) pa[j] = pa[j] && bit_get(A.v_fk_a, A.o_fk_a, row[j]);
        }
        if (DIRECT) {
#pragma unroll
            for (int j = 0; j < kK; j++) {
                passed += pa[j];
                hit[j] = pa[j] && ga[j] >= 0 && gb[j] >= 0;
                g[j] = A.group_by == 0 ? ga[j] : gb[j];
                v[j] = 0.0;
                if (hit[j]) {
                    if (NULLS && star_value_null(A, row[j])) atomicAdd(A.nulls + g[j], 1ull);
                    else v[j] = __dmul_rn((double)__ldcs(A.price + row[j]), __dsub_rn(1.0, __ldcs(A.disc + row[j])));
                }
            }
#pragma unroll
            for (int j = 0; j < kK; j++) {
                // Lanes with a joined row add it in turn to the warp's accumulators.
                unsigned pend = __ballot_sync(0xFFFFFFFFu, hit[j]);
                while (pend) {
                    const int l = __ffs(pend) - 1;
                    pend &= pend - 1;
                    if (lane == l) {
                        joined++;
                        star_add_plain(A, g[j], v[j], w_hi, w_lo, w_cnt, G);
                    }
                    __syncwarp();
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < kK; j++) {
                passed += pa[j];
                uint32_t ra = kStarNone, rb0 = kStarNone;
                if (pa[j]) {
                    ra = star_lookup(A.ta, ka[j]);
                    if (ra != kStarNone) rb0 = star_lookup(A.tb, kb[j]);
                }
                const bool h = ra != kStarNone && rb0 != kStarNone;
                const bool vnull = NULLS && h && star_value_null(A, row[j]);
                double vv = 0.0;
                if (h && !vnull) vv = __dmul_rn((double)__ldcs(A.price + row[j]), __dsub_rn(1.0, __ldcs(A.disc + row[j])));
                unsigned pend = __ballot_sync(0xFFFFFFFFu, h);
                while (pend) {
                    const int l = __ffs(pend) - 1;
                    pend &= pend - 1;
                    if (lane == l) {
                        // every (a, b) match pair (chains are one long for unique keys)
                        for (int ca = 0; ra != kStarNone && ca < (1 << 20); ca++, ra = A.ta.next[ra]) {
                            int cb = 0;
                            for (uint32_t rb = rb0; rb != kStarNone && cb < (1 << 20); cb++, rb = A.tb.next[rb]) {
                                joined++;
                                const int gg = A.group_by == 0 ? A.ta.gid[ra] : A.tb.gid[rb];
                                if (vnull) atomicAdd(A.nulls + gg, 1ull);
                                star_add_plain(A, gg, vv, w_hi, w_lo, w_cnt, G);
                            }
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    passed = warp_sum(passed);
    joined = warp_sum(joined);
    if (lane == 0) {
        if (passed) atomicAdd(&s_stat[0], passed);
        if (joined) atomicAdd(&s_stat[1], joined);
    }
    __syncthreads();
    for (int gi = tid; gi < G; gi += kJoinThreads) {
        double H = 0.0, L = 0.0;
        unsigned long long C = 0;
        for (int w = 0; w < kWarps; w++) {
            const unsigned long long c = s_cnt[w * G + gi];
            if (!c) continue;
            double s, e;
            two_sum(H, s_hi[w * G + gi], s, e);
            H = s;
            L = __dadd_rn(L, __dadd_rn(e, s_lo[w * G + gi]));
            C += c;
        }
        if (C) {
            atomic_add_dd2(A.sum_hi + gi, A.sum_lo + gi, H, L);
            atomicAdd(A.cnt + gi, C);
        }
    }
    if (tid < 2 && s_stat[tid]) atomicAdd(A.stats + tid, s_stat[tid]);
}

// Evaluates a key filter for every value of [lo, lo + values) into an answer
// bitmap (bit v - lo), one value per thread, one word per warp.
__global__ void filter_bitmap_kernel(KeyFilterDev f, long long lo, uint64_t words, uint64_t values, uint32_t *out) {
    const uint64_t total = words * 32;
    for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x; base < total; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = base + threadIdx.x;
        const bool p = v < values && filter_pass(f, lo + (long long)v);
        const unsigned w = __ballot_sync(0xFFFFFFFFu, p);
        if ((threadIdx.x & 31) == 0 && v < total) out[v >> 5] = w;
    }
}

// Writes each dimension row's group id at its key's place of a direct index
// (the index starts all -1).
template <class T>
__global__ void direct_index_kernel(const long long *keys, const int32_t *gid, int64_t n, long long lo, T *out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[keys[i] - lo] = (T)gid[i];
}

// Shared memory of the scan: the staged bitmap words.
inline size_t star_scan_smem(int bits_words) { return (size_t)bits_words * 4; }
// Shared memory of the join kernel: per-warp accumulators of G groups.
inline size_t star_join_smem(int G) { return (size_t)(kJoinThreads / 32) * G * 24; }

}  // namespace krv
