// Q1 scan kernels for sm_100a: date predicate + (returnflag, linestatus) group-by with exact
// fixed-point sums, over HBM-resident columns.
//
// Replaces the 15 __global__ kernels of the reference (src/kernels/*: 5 table placements x
// {uncompressed, compressed, filter-pushdown compressed}); the per-row arithmetic is that of
// every reference kernel (e.g. src/kernels/ht_in_registers_per_thread.cuh:38-60):
//   disc_1 = 100 - disc, disc_price = disc_1 * price, charge = disc_price * (100 + tax),
//   group = (rf << 1) + ls; sums of quantity, price, disc_price, charge, disc and a count.
//
// Structure (one design for every layout and placement):
//   * persistent grid, one CTA per SM, each CTA = 1 producer warp + W consumer warps;
//   * the producer streams tiles of R rows, every column of the tile with one
//     cp.async.bulk (TMA bulk copy, evict-first L2 policy) into an S-stage shared-memory ring,
//     completion tracked on mbarriers; consumers release a stage with one arrive per warp;
//   * consumers decode the rows from shared memory in registers (predicate, group code,
//     quantity/discount/tax bytes, price) and accumulate according to the placement;
//   * one 128-bit atomic per CTA per (group, aggregate) into the caller's buffer.
// Every wait is bounded (q1_ptx.cuh, kWaitLimitNs); on expiry the kernel records
// kStatusWaitTimeout in the status word, drains its own copies and returns.
//
// Fast domain: discount <= 100 (so 100 - d >= 0), tax <= 255, extendedprice and quantity < 2^32.
// Then every per-row product fits 64 bits unsigned (charge < 2^47.2) and per-thread 64-bit
// partials cannot wrap for launches of up to 2^31 rows (the host splits longer launches).
// Compressed columns cannot leave it except by a discount above 100 or a ship offset above 32767,
// which set kStatusDomain (the host reports Q1_ERR_DOMAIN). The reference-typed (uncompressed)
// columns are int64: a passing row outside the fast domain is summed exactly by wide_row (signed
// 128-bit arithmetic, 128-bit atomics straight into the output), and only a row whose int64
// products overflow, which the reference's KernelHyPer reports through handle_overflow
// (cpu/kernel_hyper.hpp:65-91), sets kStatusDomain.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>

#include "q1_common.cuh"
#include "q1_kernels.h"
#include "q1_ptx.cuh"
#include "q1_quad.cuh"

namespace q1 {

using namespace ptx;

// ---------------------------------------------------------------------------------------------
// Layouts
// ---------------------------------------------------------------------------------------------

// Column order inside a tile: ship (or filter), qty, disc, tax, price, flags... (see q1_kernels.h)
template <int L>
struct LayoutTraits;

template <>
struct LayoutTraits<kLayPair> {
    static constexpr int kCols = 6;
    static constexpr uint64_t kBitsWord = 0x0000022008080810ull;  // bits per column, one byte each: {16, 8, 8, 8, 32, 2, 0}
    static constexpr int kRowsPerStep = 4;
    static constexpr int kCodes = 4;   // 2-bit pair dictionary
    static constexpr bool kFilter = false;
    static constexpr bool kWideQty = false;
};
template <>
struct LayoutTraits<kLayPairFilter> {
    static constexpr int kCols = 6;
    static constexpr uint64_t kBitsWord = 0x0000022008080801ull;  // bits per column, one byte each: {1, 8, 8, 8, 32, 2, 0}
    static constexpr int kRowsPerStep = 4;
    static constexpr int kCodes = 4;
    static constexpr bool kFilter = true;
    static constexpr bool kWideQty = false;
};
template <>
struct LayoutTraits<kLaySep> {
    static constexpr int kCols = 7;
    static constexpr uint64_t kBitsWord = 0x0001022008080810ull;  // bits per column, one byte each: {16, 8, 8, 8, 32, 2, 1}
    static constexpr int kRowsPerStep = 4;
    static constexpr int kCodes = 6;   // (rf << 1) + ls
    static constexpr bool kFilter = false;
    static constexpr bool kWideQty = false;
};
template <>
struct LayoutTraits<kLaySepFilter> {
    static constexpr int kCols = 7;
    static constexpr uint64_t kBitsWord = 0x0001022008080801ull;  // bits per column, one byte each: {1, 8, 8, 8, 32, 2, 1}
    static constexpr int kRowsPerStep = 4;
    static constexpr int kCodes = 6;
    static constexpr bool kFilter = true;
    static constexpr bool kWideQty = false;
};
template <>
struct LayoutTraits<kLayUncomp> {
    static constexpr int kCols = 7;
    static constexpr uint64_t kBitsWord = 0x0008084040404020ull;  // bits per column, one byte each: {32, 64, 64, 64, 64, 8, 8}
    static constexpr int kRowsPerStep = 2;
    static constexpr int kCodes = 6;
    static constexpr bool kFilter = false;
    static constexpr bool kWideQty = true;
};

template <int L>
__host__ __device__ constexpr uint32_t col_bits(int c) {
    return (uint32_t)((LayoutTraits<L>::kBitsWord >> (8 * c)) & 0xFFu);
}
template <int L>
__host__ __device__ constexpr uint32_t col_offset(int c, uint32_t R) {
    uint32_t off = 0;
    for (int i = 0; i < c; ++i) off += R * col_bits<L>(i) / 8u;
    return off;
}
template <int L>
__host__ __device__ constexpr uint32_t stage_bytes(uint32_t R) {
    return col_offset<L>(LayoutTraits<L>::kCols, R);
}

// ---------------------------------------------------------------------------------------------
// Accumulators (table placements)
// ---------------------------------------------------------------------------------------------

// Per-row decoded values handed to a placement:
//   c  group code (0..kCodes-1) of a passing row, or a value >= kCodes for a filtered row
//   q  quantity (whole units for compressed, hundredths for uncompressed)
//   d  discount, a = 100 - d, ab = a * (100 + tax), p = extendedprice

// Aggregates of one group, per thread, in registers (reference-typed rows, one at a time).
struct GroupRegs {
    uint64_t p, dp, ch, q;
    uint32_t d, cnt;

    __device__ __forceinline__ void zero() {
        p = dp = ch = q = 0;
        d = cnt = 0;
    }
    __device__ __forceinline__ void add(bool hit, uint32_t qty, uint32_t disc, uint32_t a, uint32_t ab, uint32_t pr) {
        const uint32_t pg = hit ? pr : 0u;
        q = mad_wide(hit ? qty : 0u, 1u, q);
        d += hit ? disc : 0u;
        cnt += hit ? 1u : 0u;
        p += pg;
        dp = mad_wide(a, pg, dp);
        ch = mad_wide(ab, pg, ch);
    }
    // Aggregate values in q1 order (count, qty, price, disc, disc_price, charge).
    __device__ __forceinline__ uint64_t value(int agg) const {
        switch (agg) {
            case kAggCount: return cnt;
            case kAggQty: return q;
            case kAggBasePrice: return p;
            case kAggDisc: return d;
            case kAggDiscPrice: return dp;
            default: return ch;
        }
    }
};

// Most rows a thread adds in one launch (scan_max_rows_per_launch).
constexpr uint32_t kMaxThreadRows = 1u << 15;

// Warp-wide sum of aggregate a's per-thread partials. Per thread and launch at most 2^15 rows: count
// < 2^16, quantity (compressed) < 2^23, discount < 2^22, price and reference-typed quantity < 2^47,
// disc_price < 2^53.7, charge < 2^62.2.
template <bool kWideQty>
__device__ __forceinline__ Sum128 warp_sum_agg(int a, uint64_t v) {
    switch (a) {
        case kAggCount:
        case kAggDisc: return warp_sum<27>(v);
        case kAggQty: return warp_sum<kWideQty ? 54 : 27>(v);
        case kAggCharge: return warp_sum<63>(v);
        default: return warp_sum<54>(v);
    }
}

// A warp's sums at the end of the scan: its record [codes][6] of the CTA's shared memory (written
// whole, by any of its lanes), summed over the warps by the kernel's last lines.
struct WarpRecord {
    ulonglong2* v;
    __device__ __forceinline__ void set(int code, int agg, Sum128 s) {
        v[code * kNumAggs + agg] = make_ulonglong2(s.lo, s.hi);
    }
};

// --- in_registers_per_thread: every thread owns all groups in registers; a row updates the
// matching group through predicated (select) arithmetic over all groups
// (src/kernels/ht_in_registers_per_thread.cuh:11-79).
template <int G, bool kWideQty>
struct AccPerThread {
    // With the six (returnflag, linestatus) groups of the separate flag layout, A/O and R/O (codes
    // 1 and 5) need a receipt date before the ship date and do not occur in TPC-H data: their rows
    // go straight into the CTA's 128-bit shared table (red) behind one warp vote, so that only the
    // four other groups' planes take registers (a kernel of 128 registers a thread).
    static constexpr bool kCold = (G == 6) && !kWideQty;
    static constexpr int kPlanes = kWideQty ? 1 : (kCold ? 4 : G);
    GroupRegs g[kWideQty ? G : 1];      // row-wise path (uncompressed layout)
    GroupPlanes gq[kPlanes];                      // quad path (compressed layouts)
    unsigned long long* red;                      // the CTA's [G][6][lo, hi] table (cold groups)
    // group of plane slot s: the codes themselves, or with cold groups AF, NF, NO, RF
    static __device__ __forceinline__ constexpr uint32_t group_of(int s) {
        return kCold ? (s == 0 ? 0u : (uint32_t)s + 1u) : (uint32_t)s;
    }
    static __device__ __forceinline__ constexpr bool cold(int grp) { return kCold && (grp == 1 || grp == 5); }
    __device__ __forceinline__ void init(uint32_t, uint32_t, uint8_t*, unsigned long long* cta_red) {
        red = cta_red;
#pragma unroll
        for (int i = 0; i < (kWideQty ? G : 1); ++i) g[i].zero();
#pragma unroll
        for (int i = 0; i < kPlanes; ++i) gq[i].zero();
    }
    // One passing row of a cold group, exactly, into the CTA's table: where the rows of those groups go
    // unless the caller of add() and add_quad() has a place of its own for them.
    __device__ __forceinline__ void cold_row(uint32_t grp, uint32_t q, uint32_t d, uint32_t a, uint32_t ab,
                                             uint32_t p) {
        unsigned long long* v = red + 2 * (grp * kNumAggs);
        atomic_add_u128_shared(v + 2 * kAggCount, 1, 0);
        atomic_add_u128_shared(v + 2 * kAggQty, q, 0);
        atomic_add_u128_shared(v + 2 * kAggBasePrice, p, 0);
        atomic_add_u128_shared(v + 2 * kAggDisc, d, 0);
        atomic_add_u128_shared(v + 2 * kAggDiscPrice, (uint64_t)a * p, 0);
        atomic_add_u128_shared(v + 2 * kAggCharge, (uint64_t)ab * p, 0);
    }
    struct ToCta {
        AccPerThread& acc;
        __device__ __forceinline__ void row(uint32_t grp, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) const {
            acc.cold_row(grp, q, d, a, ab, p);
        }
        __device__ __forceinline__ void quad(const Quad& x) const {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint32_t b = (x.OH >> (8 * r)) & 0x22u;
                if (b) acc.cold_row((b & 2u) ? 1u : 5u, (x.Q >> (8 * r)) & 0xFFu, (x.D >> (8 * r)) & 0xFFu, x.a[r], x.ab[r], x.p[r]);
            }
        }
    };
    __device__ __forceinline__ void add(uint32_t c, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) {
        add(c, q, d, a, ab, p, ToCta{*this});
    }
    template <class Cold>
    __device__ __forceinline__ void add(uint32_t c, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p,
                                        Cold&& cold_to) {
        if constexpr (kWideQty) {
#pragma unroll
            for (int i = 0; i < G; ++i) g[i].add(c == (uint32_t)i, q, d, a, ab, p);
        } else {
            if (kCold && (c == 1u || c == 5u)) {
                cold_to.row(c, q, d, a, ab, p);
                return;
            }
            // one row through the quad path (tail rows)
            Quad x;
            x.OH = c < (uint32_t)G ? (1u << c) : 0u;
            x.Q = q;
            x.D = d;
            x.A = a;
            x.P[0] = p & 0xFFu;
            x.P[1] = (p >> 8) & 0xFFu;
            x.P[2] = (p >> 16) & 0xFFu;
            x.P[3] = p >> 24;
            x.ABL = ab & 0xFFu;
            x.ABH = ab >> 8;
#pragma unroll
            for (int i = 0; i < kPlanes; ++i) gq[i].add_quad(x.OH, group_of(i), x);   // no warp vote: lanes diverge here
        }
    }
    // Called by all lanes of the warp.
    template <bool kTop, class Cold>
    __device__ __forceinline__ void add_quad_planes(const Quad& x, Cold&& cold_to) {
#pragma unroll
        for (int i = 0; i < kPlanes; ++i) gq[i].template add_quad<kTop>(x.OH, group_of(i), x);
        if constexpr (kCold) {
            if (__any_sync(0xffffffffu, x.OH & 0x22222222u)) cold_to.quad(x);
        }
    }
    __device__ __forceinline__ void add_quad(const Quad& x) { add_quad(x, ToCta{*this}); }
    template <class Cold>
    __device__ __forceinline__ void add_quad(const Quad& x, Cold&& cold_to) {
        if constexpr (!kWideQty) {
            // the prices' top byte plane is zero for the whole warp unless a price is >= 2^24
            if (__any_sync(0xffffffffu, x.P[3])) add_quad_planes<true>(x, cold_to);
            else add_quad_planes<false>(x, cold_to);
        }
    }
    // plane slot of group i (not called for cold groups)
    static __device__ __forceinline__ constexpr int slot_of(int i) { return kCold ? (i == 0 ? 0 : i - 1) : i; }
    // The thread's partial of group i (0 for a cold group: its rows are in the CTA table already).
    __device__ __forceinline__ uint64_t value(int i, int a) const {
        if constexpr (kWideQty) return g[i].value(a);
        else return cold(i) ? 0ull : gq[slot_of(i)].value(a);
    }
    __device__ __forceinline__ void zero_group(int i) {
        if constexpr (kWideQty) g[i].zero();
        else if (!cold(i)) gq[slot_of(i)].zero();
    }
    template <class P>
    __device__ __forceinline__ void tile_done(const P&, uint32_t) {}
    template <class P>
    __device__ __forceinline__ void finish(const P&, uint32_t) {}
    __device__ __forceinline__ void flush(WarpRecord rec, uint32_t lane) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
#pragma unroll
            for (int a = 0; a < kNumAggs; ++a) {
                const Sum128 s = cold(i) ? Sum128{0, 0} : warp_sum_agg<kWideQty>(a, value(i, a));
                if (lane == 0) rec.set(i, a, s);
            }
        }
    }
};

// A group's entry in the per-thread tables below: count, quantity and discount in one word (a thread
// adds at most 2^15 rows per launch, so count < 2^16, quantity <= 255 * 2^15 < 2^23, discount
// <= 100 * 2^15 < 2^22), then price, (100 - d) price and (100 - d)(100 + t) price. Reference-typed
// rows' quantity takes a word of its own.
template <bool kWideQty>
struct Entry {
    static constexpr int kWords = kWideQty ? 5 : 4;
    static constexpr int kQtyShift = 16, kDiscShift = kWideQty ? 16 : 39;
    static_assert(kMaxThreadRows < 1u << kQtyShift && (kWideQty || 255ull * kMaxThreadRows < 1ull << (kDiscShift - kQtyShift)) &&
                      100ull * kMaxThreadRows < 1ull << (64 - kDiscShift),
                  "the packed sums' fields");
    // word w of a group's sums
    template <class Buf>
    static __device__ __forceinline__ uint64_t word(const Buf& b, int i, int w) {
        switch (w) {
            case 0:
                return b.value(i, kAggCount) | (kWideQty ? 0ull : b.value(i, kAggQty) << kQtyShift) |
                       (b.value(i, kAggDisc) << kDiscShift);
            case 1: return b.value(i, kAggBasePrice);
            case 2: return b.value(i, kAggDiscPrice);
            case 3: return b.value(i, kAggCharge);
            default: return b.value(i, kAggQty);
        }
    }
    // One row of compressed columns added to an entry, word(j) its word j.
    template <class Word>
    static __device__ __forceinline__ void add_row(Word&& word, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) {
        word(0) = word(0) + (1ull | (uint64_t)q << kQtyShift | (uint64_t)d << kDiscShift);
        word(1) = word(1) + p;
        word(2) = mad_wide(a, p, word(2));
        word(3) = mad_wide(ab, p, word(3));
    }
    // The rows of a quad with byte r of `rows` 1 (0 in the others).
    template <class Word>
    static __device__ __forceinline__ void add_quad(Word&& word, uint32_t rows, const Quad& x) {
        uint64_t p = 0, dp = 0, ch = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t pr = (rows >> (8 * r)) & 1u ? x.p[r] : 0u;
            p += pr;
            dp = mad_wide(x.a[r], pr, dp);
            ch = mad_wide(x.ab[r], pr, ch);
        }
        word(0) = word(0) + ((uint64_t)__popc(rows) | (uint64_t)__dp4a(rows, x.Q, 0u) << kQtyShift |
                             (uint64_t)__dp4a(rows, x.D, 0u) << kDiscShift);
        word(1) = word(1) + p;
        word(2) = word(2) + dp;
        word(3) = word(3) + ch;
    }
    // aggregate a of the words w
    static __device__ __forceinline__ uint64_t value(const uint64_t w[kWords], int a) {
        switch (a) {
            case kAggCount: return w[0] & 0xFFFFull;
            case kAggQty: return kWideQty ? w[kWords - 1] : (w[0] >> kQtyShift) & ((1ull << 23) - 1);
            case kAggBasePrice: return w[1];
            case kAggDisc: return w[0] >> kDiscShift;
            case kAggDiscPrice: return w[2];
            default: return w[3];
        }
    }
    // The warp's sum of group i's entries into its record.
    static __device__ __forceinline__ void reduce(const uint64_t w[kWords], int i, WarpRecord rec, uint32_t lane) {
#pragma unroll
        for (int a = 0; a < kNumAggs; ++a) {
            const Sum128 s = warp_sum_agg<kWideQty>(a, value(w, a));
            if (lane == 0) rec.set(i, a, s);
        }
    }
};

// Where rows of the cold groups (codes 1 and 5) go in a placement with per-thread entries: word(group, j) is word j
// of the thread's entry of that group. (The groups are constants, which keeps a table that lies in local memory
// apart from the rest of its accumulator.)
template <class E, class Word>
struct ToEntries {
    Word word;
    __device__ __forceinline__ void row(uint32_t grp, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) const {
        if (grp == 1u) E::add_row([&](uint32_t j) -> auto& { return word(1u, j); }, q, d, a, ab, p);
        else E::add_row([&](uint32_t j) -> auto& { return word(5u, j); }, q, d, a, ab, p);
    }
    __device__ __forceinline__ void quad(const Quad& x) const {
        const uint32_t one = (x.OH >> 1) & 0x01010101u, five = (x.OH >> 5) & 0x01010101u;
        if (one) E::add_quad([&](uint32_t j) -> auto& { return word(1u, j); }, one, x);
        if (five) E::add_quad([&](uint32_t j) -> auto& { return word(5u, j); }, five, x);
    }
};
template <class E, class Word>
__device__ __forceinline__ ToEntries<E, Word> to_entries(Word word) { return ToEntries<E, Word>{word}; }

// The other placements keep their table elsewhere and write-combine: a thread sums its rows of some
// tiles in registers (AccPerThread, four rows an instruction), then adds the sums to the table.
// Adding every quad or row to the table directly made the table the bound: 600 M pair-layout rows
// took 1.95 ms (in_registers: every lane of a table read all of its rows), 2.13 ms
// (shared_mem_per_thread) and 3.19 ms (local_mem) against 0.88 ms in registers. Rows of the two groups that
// AccPerThread has no planes for go to entries of the thread's own, where the placement has such. (Separate flags
// with line status at random, a quarter of the rows of those groups, 4.0 M rows: 24 to 28 us; into the CTA's
// table, by 128-bit shared atomics, 270 to 296.)
template <int G, bool kWideQty>
struct AccCombining {
    AccPerThread<G, kWideQty> buf;
    uint32_t tiles;   // in buf
    __device__ __forceinline__ void init_buffer(uint32_t lane, uint32_t ctid, uint8_t* scratch, unsigned long long* red) {
        buf.init(lane, ctid, scratch, red);
        tiles = 0;
    }
    __device__ __forceinline__ void add(uint32_t c, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) {
        buf.add(c, q, d, a, ab, p);
    }
    __device__ __forceinline__ void add_quad(const Quad& x) { buf.add_quad(x); }
    // Whether the buffer goes to the table now; called by all lanes after each tile.
    __device__ __forceinline__ bool due() {
        if (++tiles < kCombineTiles) return false;
        tiles = 0;
        return true;
    }
};

// --- in_registers ("warp-lane tables", src/kernels/ht_in_registers.cuh:30-121): lane g of a warp
// holds group g's sums in registers; the warp's buffers meet there through warp reductions. (In
// the reference all lanes of a table read the same rows, each keeping those of its group.)
template <int G, bool kWideQty, uint32_t kThreads>
struct AccWarpLane : AccCombining<G, kWideQty> {
    using E = Entry<kWideQty>;
    static constexpr bool kCold = AccPerThread<G, kWideQty>::kCold;
    // lane g: group g. A launch gives a warp at most 2^20 rows: the charge sum takes 128 bits
    // (2^47.2 a row), the others 64.
    uint64_t t[kNumAggs], ch_hi;
    uint64_t* cold_tab;   // this thread's column of [word][cold group][thread]
    static constexpr uint32_t kTableBytes = kCold ? 8u * E::kWords * 2u * kThreads : 0u;
    __device__ __forceinline__ uint64_t& cold_entry(uint32_t grp, uint32_t j) {
        return cold_tab[(2u * j + (grp == 1u ? 0u : 1u)) * kThreads];
    }
    __device__ __forceinline__ void init(uint32_t lane, uint32_t ctid, uint8_t* scratch, unsigned long long* red) {
        this->init_buffer(lane, ctid, scratch, red);
#pragma unroll
        for (int a = 0; a < kNumAggs; ++a) t[a] = 0;
        ch_hi = 0;
        if constexpr (kCold) {
            cold_tab = reinterpret_cast<uint64_t*>(scratch) + ctid;
#pragma unroll
            for (uint32_t j = 0; j < 2u * E::kWords; ++j) cold_tab[j * kThreads] = 0;
        }
    }
    __device__ __forceinline__ auto cold() {
        return to_entries<E>([this](uint32_t grp, uint32_t j) -> uint64_t& { return cold_entry(grp, j); });
    }
    __device__ __forceinline__ void add(uint32_t c, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) {
        this->buf.add(c, q, d, a, ab, p, cold());
    }
    __device__ __forceinline__ void add_quad(const Quad& x) { this->buf.add_quad(x, cold()); }
    __device__ __forceinline__ void to_table(uint32_t lane) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
            if (this->buf.cold(i)) continue;
#pragma unroll
            for (int a = 0; a < kNumAggs; ++a) {
                const uint64_t v = warp_sum_agg<kWideQty>(a, this->buf.value(i, a)).lo;
                if (lane == (uint32_t)i) {
                    t[a] += v;
                    if (a == kAggCharge) ch_hi += t[a] < v ? 1u : 0u;
                }
            }
            this->buf.zero_group(i);
        }
    }
    template <class P>
    __device__ __forceinline__ void tile_done(const P&, uint32_t lane) {
        if (this->due()) to_table(lane);
    }
    template <class P>
    __device__ __forceinline__ void finish(const P&, uint32_t lane) { to_table(lane); }
    __device__ __forceinline__ void flush(WarpRecord rec, uint32_t lane) {
        if (lane < (uint32_t)G && !(kCold && this->buf.cold((int)lane))) {
#pragma unroll
            for (int a = 0; a < kNumAggs; ++a) rec.set((int)lane, a, Sum128{t[a], a == kAggCharge ? ch_hi : 0ull});
        }
        if constexpr (kCold) {
#pragma unroll
            for (int i = 1; i <= 5; i += 4) {
                uint64_t w[E::kWords];
#pragma unroll
                for (int j = 0; j < E::kWords; ++j) w[j] = cold_entry((uint32_t)i, j);
                E::reduce(w, i, rec, lane);
            }
        }
    }
};

// --- local_mem (src/kernels/ht_in_local_mem.cuh:11-74): per-thread tables in (L1-cached) local
// memory.
template <int G, bool kWideQty>
struct AccLocal : AccCombining<G, kWideQty> {
    using E = Entry<kWideQty>;
    volatile uint64_t t[G][E::kWords];   // (volatile: not in registers)
    __device__ __forceinline__ void init(uint32_t lane, uint32_t ctid, uint8_t* scratch, unsigned long long* red) {
        this->init_buffer(lane, ctid, scratch, red);
        for (int i = 0; i < G; ++i)
            for (int j = 0; j < E::kWords; ++j) t[i][j] = 0;
    }
    __device__ __forceinline__ auto cold() {
        return to_entries<E>([this](uint32_t grp, uint32_t j) -> volatile uint64_t& { return t[grp < G ? grp : 0][j]; });
    }
    __device__ __forceinline__ void add(uint32_t c, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) {
        this->buf.add(c, q, d, a, ab, p, cold());
    }
    __device__ __forceinline__ void add_quad(const Quad& x) { this->buf.add_quad(x, cold()); }
    __device__ __forceinline__ void to_table() {
#pragma unroll
        for (int i = 0; i < G; ++i) {
            if (this->buf.cold(i)) continue;
#pragma unroll
            for (int j = 0; j < E::kWords; ++j) t[i][j] = t[i][j] + E::word(this->buf, i, j);
            this->buf.zero_group(i);
        }
    }
    template <class P>
    __device__ __forceinline__ void tile_done(const P&, uint32_t) {
        if (this->due()) to_table();
    }
    template <class P>
    __device__ __forceinline__ void finish(const P&, uint32_t) { to_table(); }
    __device__ __forceinline__ void flush(WarpRecord rec, uint32_t lane) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
            uint64_t w[E::kWords];
#pragma unroll
            for (int j = 0; j < E::kWords; ++j) w[j] = t[i][j];
            E::reduce(w, i, rec, lane);
        }
    }
};

// --- shared_mem_per_thread (src/kernels/ht_in_shared_mem_per_thread.cuh:23-118): per-thread
// tables in shared memory, laid out [word][group][thread] so a warp's accesses are bank-conflict
// free. Reference-typed rows update their group's entry row by row: six groups' 64-bit sums in
// registers cost more than the table (100 M rows 0.599 ms against 0.548 ms).
template <int G, bool kWideQty, uint32_t kThreads>
struct AccSharedPerThread : AccCombining<G, kWideQty> {
    using E = Entry<kWideQty>;
    uint64_t* tab;       // this thread's column of [w0, p, dp, ch, (quantity)][group][thread]
    __device__ __forceinline__ void init(uint32_t lane, uint32_t ctid, uint8_t* scratch, unsigned long long* red) {
        this->init_buffer(lane, ctid, scratch, red);
        tab = reinterpret_cast<uint64_t*>(scratch) + ctid;
#pragma unroll
        for (int i = 0; i < E::kWords * G; ++i) tab[i * kThreads] = 0;
    }
    __device__ __forceinline__ uint64_t& entry(uint32_t i, uint32_t j) { return tab[(j * G + i) * kThreads]; }
    __device__ __forceinline__ void add(uint32_t c, uint32_t q, uint32_t d, uint32_t a, uint32_t ab, uint32_t p) {
        if constexpr (kWideQty) {
            if (c < (uint32_t)G) {
                entry(c, 0) += 1ull | ((uint64_t)d << E::kDiscShift);
                entry(c, 4) += q;
                entry(c, 1) += p;
                entry(c, 2) = mad_wide(a, p, entry(c, 2));
                entry(c, 3) = mad_wide(ab, p, entry(c, 3));
            }
        } else {
            this->buf.add(c, q, d, a, ab, p, cold());
        }
    }
    __device__ __forceinline__ auto cold() {
        return to_entries<E>([this](uint32_t grp, uint32_t j) -> uint64_t& { return entry(grp, j); });
    }
    __device__ __forceinline__ void add_quad(const Quad& x) { this->buf.add_quad(x, cold()); }
    __device__ __forceinline__ void to_table() {
        if constexpr (!kWideQty) {
#pragma unroll
            for (int i = 0; i < G; ++i) {
                if (this->buf.cold(i)) continue;
#pragma unroll
                for (int j = 0; j < E::kWords; ++j) entry(i, j) += E::word(this->buf, i, j);
                this->buf.zero_group(i);
            }
        }
    }
    template <class P>
    __device__ __forceinline__ void tile_done(const P&, uint32_t) {
        if (this->due()) to_table();
    }
    template <class P>
    __device__ __forceinline__ void finish(const P&, uint32_t) { to_table(); }
    __device__ __forceinline__ void flush(WarpRecord rec, uint32_t lane) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
            uint64_t w[E::kWords];
#pragma unroll
            for (int j = 0; j < E::kWords; ++j) w[j] = entry(i, j);
            E::reduce(w, i, rec, lane);
        }
    }
};

// --- global (src/kernels/ht_in_global_mem.hpp:11-52): no thread- or block-private table; the
// aggregates live only in the global output, updated by atomics all through the scan. The
// reference issues 6 atomics per row; here each warp issues one 128-bit atomic add per (group,
// aggregate) for its buffered rows straight into the global table.
template <int G, bool kWideQty>
struct AccGlobal : AccCombining<G, kWideQty> {
    __device__ __forceinline__ void init(uint32_t lane, uint32_t ctid, uint8_t* scratch, unsigned long long* red) {
        this->init_buffer(lane, ctid, scratch, red);
    }
    template <class P>
    __device__ __forceinline__ void tile_done(const P& prm, uint32_t lane) {
        if (this->due()) to_global(prm, lane);
    }
    template <class P>
    __device__ __forceinline__ void finish(const P&, uint32_t) {}
    template <class P>
    __device__ __forceinline__ void to_global(const P& prm, uint32_t lane) {
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const int grp = G == 4 ? prm.pair_group[i] : i;
#pragma unroll
            for (int a = 0; a < kNumAggs; ++a) {
                uint64_t v = warp_sum_agg<kWideQty>(a, this->buf.value(i, a)).lo;
                if (a == kAggQty) v *= prm.qty_scale;
                if (lane == (uint32_t)((i * kNumAggs + a) & 31)) atomic_add_u128(prm.out + 2 * (grp * kNumAggs + a), v, 0);
            }
            this->buf.zero_group(i);
        }
    }
    // What is left at the end goes through the CTA's reduction, one atomic per CTA and sum instead of
    // one per warp (60 M rows: 0.118 -> 0.107 ms).
    __device__ __forceinline__ void flush(WarpRecord rec, uint32_t lane) { this->buf.flush(rec, lane); }
};

template <int P, int G, bool W, uint32_t T>
struct AccSel;
template <int G, bool W, uint32_t T> struct AccSel<kPlaceInRegisters, G, W, T> { using A = AccWarpLane<G, W, T>; };
template <int G, bool W, uint32_t T> struct AccSel<kPlaceInRegistersPerThread, G, W, T> { using A = AccPerThread<G, W>; };
template <int G, bool W, uint32_t T> struct AccSel<kPlaceLocalMem, G, W, T> { using A = AccLocal<G, W>; };
template <int G, bool W, uint32_t T> struct AccSel<kPlaceSharedMemPerThread, G, W, T> { using A = AccSharedPerThread<G, W, T>; };
template <int G, bool W, uint32_t T> struct AccSel<kPlaceGlobal, G, W, T> { using A = AccGlobal<G, W>; };

// ---------------------------------------------------------------------------------------------
// Row decoding
// ---------------------------------------------------------------------------------------------


__device__ __forceinline__ uint32_t code_of_chars(uint32_t rf, uint32_t ls) {
    const uint32_t r = (rf == 'R' ? 2u : 0u) + (rf == 'N' ? 1u : 0u);
    return (r << 1) + (ls == 'F' ? 0u : 1u);
}

__device__ __forceinline__ bool fits_i64(__int128 v) { return v >= (__int128)INT64_MIN && v <= (__int128)INT64_MAX; }

__device__ __forceinline__ void atomic_add_i128(unsigned long long* p, __int128 v) {
    atomic_add_u128(p, (uint64_t)(unsigned __int128)v, (uint64_t)((unsigned __int128)v >> 64));
}

// One passing reference-typed row outside the fast domain, summed exactly with the reference's
// arithmetic (cpu/kernel_hyper.hpp:70-83): disc_1 = 100 - disc, tax_1 = 100 + tax,
// disc_price = disc_1 * price, charge = disc_price * tax_1, each an int64 in the reference and
// checked for overflow there; the six sums go straight into the output table as signed 128-bit
// values. A row whose int64 arithmetic would overflow is reported instead of summed.
__device__ __noinline__ void wide_row(const ScanParams& prm, uint32_t group, int64_t q, int64_t d, int64_t t,
                                      int64_t p) {
    const __int128 d1 = (__int128)100 - d, t1 = (__int128)100 + t;
    const __int128 dp = d1 * p;
    const __int128 ch = dp * t1;   // |dp| < 2^64 and |t1| < 2^64 here, so the product is exact
    if (!fits_i64(d1) || !fits_i64(t1) || !fits_i64(dp) || !fits_i64(ch)) {
        if (prm.status) atomicOr(prm.status, kStatusDomain);
        return;
    }
    unsigned long long* o = prm.out + 2 * (group * kNumAggs);
    atomic_add_i128(o + 2 * kAggCount, 1);
    atomic_add_i128(o + 2 * kAggQty, (__int128)q * prm.qty_scale);
    atomic_add_i128(o + 2 * kAggBasePrice, p);
    atomic_add_i128(o + 2 * kAggDisc, d);
    atomic_add_i128(o + 2 * kAggDiscPrice, dp);
    atomic_add_i128(o + 2 * kAggCharge, ch);
}

// One step of rows [kRowsPerStep * j, +kRowsPerStep) of the R-row tile held at shared address `base`.
template <int L, uint32_t R, class Acc>
__device__ __forceinline__ void process_step(const ScanParams& prm, uint32_t base, uint32_t j, int32_t cut,
                                             uint32_t lut, Acc& acc, uint32_t& bad) {
    using T = LayoutTraits<L>;
    if constexpr (L == kLayUncomp) {
        const uint2 sd = lds_v2(base + col_offset<L>(0, R) + 8 * j);
        const uint4 Q = lds_v4(base + col_offset<L>(1, R) + 16 * j);
        const uint4 D = lds_v4(base + col_offset<L>(2, R) + 16 * j);
        const uint4 X = lds_v4(base + col_offset<L>(3, R) + 16 * j);
        const uint4 P = lds_v4(base + col_offset<L>(4, R) + 16 * j);
        const uint32_t RF = lds_u16(base + col_offset<L>(5, R) + 2 * j);
        const uint32_t LS = lds_u16(base + col_offset<L>(6, R) + 2 * j);
        // Both rows in the fast domain (always, in TPC-H data): the placement's tables only.
        const bool fast = ((Q.y | Q.w | D.y | D.w | X.y | X.w | P.y | P.w) == 0u) & (D.x <= 100u) & (D.z <= 100u) &
                          (X.x <= 255u) & (X.z <= 255u);
        if (fast) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int32_t ship = (int32_t)(r ? sd.y : sd.x);
                const uint32_t code = code_of_chars((RF >> (8 * r)) & 0xFFu, (LS >> (8 * r)) & 0xFFu);
                const uint32_t c = ship <= cut ? code : 7u;
                const uint32_t q = r ? Q.z : Q.x;
                const uint32_t d = r ? D.z : D.x;
                const uint32_t t = r ? X.z : X.x;
                const uint32_t p = r ? P.z : P.x;
                const uint32_t a = 100u - d;
                acc.add(c, q, d, a, a * (100u + t), p);
            }
        } else {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int32_t ship = (int32_t)(r ? sd.y : sd.x);
                const uint32_t code = code_of_chars((RF >> (8 * r)) & 0xFFu, (LS >> (8 * r)) & 0xFFu);
                const uint32_t q = r ? Q.z : Q.x;
                const uint32_t d = r ? D.z : D.x;
                const uint32_t t = r ? X.z : X.x;
                const uint32_t p = r ? P.z : P.x;
                const bool wide =
                    ((r ? (Q.w | D.w | X.w | P.w) : (Q.y | D.y | X.y | P.y)) != 0u) | (d > 100u) | (t > 255u);
                const bool pass = ship <= cut;
                if (wide && pass)
                    wide_row(prm, code, (int64_t)((uint64_t)(r ? Q.w : Q.y) << 32 | q),
                             (int64_t)((uint64_t)(r ? D.w : D.y) << 32 | d),
                             (int64_t)((uint64_t)(r ? X.w : X.y) << 32 | t),
                             (int64_t)((uint64_t)(r ? P.w : P.y) << 32 | p));
                const uint32_t c = (pass && !wide) ? code : 7u;
                const uint32_t a = 100u - d;
                acc.add(c, q, d, a, a * (100u + t), p);
            }
        }
    } else {
        constexpr bool kSep = (L == kLaySep || L == kLaySepFilter);
        // pass mask of the 4 rows: byte r = 0xFF iff row r passes
        uint32_t PM;
        if constexpr (T::kFilter) {
            const uint32_t bits = (lds_u8(base + col_offset<L>(0, R) + (j >> 1)) >> ((j & 1u) * 4u)) & 0xFu;
            PM = ((bits * 0x00204081u) & 0x01010101u) * 0xFFu;
        } else {
            PM = quad_pass_mask(lds_v2(base + col_offset<L>(0, R) + 8 * j), cut, bad);
        }
        Quad x;
        x.Q = lds_u32(base + col_offset<L>(1, R) + 4 * j);
        x.D = lds_u32(base + col_offset<L>(2, R) + 4 * j);
        const uint32_t X = lds_u32(base + col_offset<L>(3, R) + 4 * j);
        const uint4 P = lds_v4(base + col_offset<L>(4, R) + 16 * j);
        const uint32_t F = lds_u8(base + col_offset<L>(5, R) + j);
        bad |= disc_out_of_domain4(x.D);
        // one-hot group bit per row byte, from a 256-entry table indexed by the 4 codes' byte
        uint32_t OH = lds_u32(lut + 4 * F);
        if constexpr (kSep) {
            // the table gives bit 2*rf; a line status of 1 doubles it to bit 2*rf+1; rf 3 -> dropped
            const uint32_t LS = (lds_u8(base + col_offset<L>(6, R) + (j >> 1)) >> ((j & 1u) * 4u)) & 0xFu;
            const uint32_t lsm = ((LS * 0x00204081u) & 0x01010101u) * 0xFFu;   // byte r = 0xFF iff ls_r
            OH = (OH + (OH & lsm)) & 0x3F3F3F3Fu;
        }
        x.OH = OH & PM;
        x.p[0] = P.x;
        x.p[1] = P.y;
        x.p[2] = P.z;
        x.p[3] = P.w;
        quad_derive(x, X);
        acc.add_quad(x);
    }
}

// One row straight from global memory (tail rows that do not fill a tile).
template <int L, class Acc>
__device__ __forceinline__ void process_row_global(const ScanParams& prm, uint64_t i, Acc& acc, uint32_t& bad) {
    if constexpr (L == kLayUncomp) {
        const int32_t ship = __ldg(reinterpret_cast<const int32_t*>(prm.col[0]) + i);
        const uint64_t q = __ldg(reinterpret_cast<const unsigned long long*>(prm.col[1]) + i);
        const uint64_t d = __ldg(reinterpret_cast<const unsigned long long*>(prm.col[2]) + i);
        const uint64_t t = __ldg(reinterpret_cast<const unsigned long long*>(prm.col[3]) + i);
        const uint64_t p = __ldg(reinterpret_cast<const unsigned long long*>(prm.col[4]) + i);
        const uint32_t rf = (uint8_t)__ldg(reinterpret_cast<const char*>(prm.col[5]) + i);
        const uint32_t ls = (uint8_t)__ldg(reinterpret_cast<const char*>(prm.col[6]) + i);
        const bool wide = ((q | p) >> 32) != 0 || d > 100u || t > 255u;
        const bool pass = ship <= prm.cutoff;
        if (wide && pass)
            wide_row(prm, code_of_chars(rf, ls), (int64_t)q, (int64_t)d, (int64_t)t, (int64_t)p);
        const uint32_t c = (pass && !wide) ? code_of_chars(rf, ls) : 7u;
        const uint32_t a = 100u - (uint32_t)d;
        acc.add(c, (uint32_t)q, (uint32_t)d, a, a * (100u + (uint32_t)t), (uint32_t)p);
    } else {
        using T = LayoutTraits<L>;
        constexpr bool kSep = (L == kLaySep || L == kLaySepFilter);
        bool pass;
        if constexpr (T::kFilter) {
            pass = (__ldg(reinterpret_cast<const uint32_t*>(prm.col[0]) + (i >> 5)) >> (i & 31)) & 1u;
        } else {
            const uint32_t ship = __ldg(reinterpret_cast<const uint16_t*>(prm.col[0]) + i);
            bad |= ship > 32767u;
            pass = (int32_t)ship <= prm.cutoff;
        }
        const uint32_t q = __ldg(prm.col[1] + i);
        const uint32_t d = __ldg(prm.col[2] + i);
        const uint32_t t = __ldg(prm.col[3] + i);
        const uint32_t p = __ldg(reinterpret_cast<const uint32_t*>(prm.col[4]) + i);
        uint32_t code;
        const uint32_t rfw = __ldg(reinterpret_cast<const uint32_t*>(prm.col[5]) + (i >> 4));
        code = (rfw >> (2 * (i & 15))) & 3u;
        if constexpr (kSep) {
            const uint32_t lsw = __ldg(reinterpret_cast<const uint32_t*>(prm.col[6]) + (i >> 5));
            code = (code << 1) | ((lsw >> (i & 31)) & 1u);
        }
        bad |= d > 100u;
        const uint32_t c = pass ? code : 7u;
        const uint32_t a = 100u - d;
        acc.add(c, q, d, a, a * (100u + t), p);
    }
}

// ---------------------------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------------------------

template <int L, int P, bool kWide>
__global__ void __launch_bounds__((kConsumerWarps<L, P, kWide> + 1) * 32, 1)
q1_scan_kernel(const __grid_constant__ ScanParams prm) {
    using T = LayoutTraits<L>;
    constexpr uint32_t R = kTileRows<L, P, kWide>;
    constexpr uint32_t S = kStages<L, P>;
    constexpr uint32_t W = kConsumerWarps<L, P, kWide>;
    constexpr uint32_t kStage = stage_bytes<L>(R);
    constexpr int G = T::kCodes;
    static_assert(kStage % 16 == 0, "stage must keep 16-byte alignment");

    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full_bar[S];
    __shared__ __align__(8) uint64_t empty_bar[S];
    __shared__ __align__(16) ulonglong2 warp_rec[W * G * kNumAggs];   // a record per consumer warp
    __shared__ __align__(16) unsigned long long red[G * kNumAggs * 2];    // the CTA's sums (and the cold groups' rows)

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t num_tiles = prm.rows / R;
    const uint32_t ring = ptx::smem_addr(smem);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(smem_addr(&full_bar[s]), 1);
            mbar_init(smem_addr(&empty_bar[s]), W);
        }
        fence_mbar_init();
    }
    for (uint32_t i = threadIdx.x; i < (uint32_t)(G * kNumAggs * 2); i += blockDim.x) red[i] = 0;
    // byte of four 2-bit codes -> one-hot bit per row byte (pair: bit code; separate: bit 2*rf)
    __shared__ uint32_t code_lut[256];
    for (uint32_t f = threadIdx.x; f < 256; f += blockDim.x) {
        uint32_t v = 0;
        for (uint32_t r = 0; r < 4; ++r) {
            const uint32_t code = (f >> (2 * r)) & 3u;
            v |= (1u << (G == 4 ? code : 2 * code)) << (8 * r);
        }
        code_lut[f] = v;
    }
    const uint32_t lut = smem_addr(code_lut);
    __syncthreads();

    if (warp == W) {
        // ----------------------------- producer warp ------------------------------------
        if (lane == 0) {
            const uint64_t pol = policy_evict_first();
            uint32_t k = 0;
            for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x, ++k) {
                const uint32_t s = k % S;
                if (!mbar_wait(smem_addr(&empty_bar[s]), ((k / S) & 1u) ^ 1u, prm.status)) break;
                const uint32_t fb = smem_addr(&full_bar[s]);
                mbar_arrive_expect_tx(fb, kStage);
                const uint32_t dst = ring + s * kStage;
#pragma unroll
                for (int c = 0; c < T::kCols; ++c) {
                    const uint32_t bytes = R * col_bits<L>(c) / 8u;
                    bulk_g2s(dst + col_offset<L>(c, R), prm.col[c] + t * (uint64_t)bytes, bytes, fb, pol);
                }
            }
            // Never leave with copies in flight: wait for the last tiles issued to land.
            for (uint32_t i = (k > S ? k - S : 0u); i < k; ++i) mbar_wait(smem_addr(&full_bar[i % S]), (i / S) & 1u, prm.status);
        }
    } else {
        // ----------------------------- consumer warps -----------------------------------
        using Acc = typename AccSel<P, G, T::kWideQty, W * 32>::A;
        const uint32_t ctid = threadIdx.x;  // 0 .. 32W-1
        Acc acc;
        acc.init(lane, ctid, smem + S * kStage, red);
        uint32_t bad = 0;
        constexpr uint32_t kSteps = R / T::kRowsPerStep;  // steps per tile
        // Rows one consumer thread adds per tile.
        constexpr uint32_t kRowsPerThreadTile = kSteps / (W * 32) * T::kRowsPerStep;
        static_assert(kSteps % (W * 32) == 0, "steps must divide evenly among consumer threads");
        // The in_registers and global placements sum a warp's buffers in 64 bits: at most 2048 rows
        // a lane of charges below 100 (2^32 - 1) 355 < 2^47.2 stays below 2^64.
        static_assert(kRowsPerThreadTile * kCombineTiles <= 2048u, "warp sums must stay below 2^64");
        // Tail rows [num_tiles * R, rows), a row a thread, while the first tiles are on their way: spread over the
        // CTAs, those with a tile less first. (One CTA taking all of them after its tiles: up to R / (32 W)
        // trips to global memory one after the other: 700,000 rows 14.5 us instead of 10.4.)
        {
            const uint32_t extra = (uint32_t)(num_tiles % gridDim.x);
            const uint32_t turn = blockIdx.x >= extra ? blockIdx.x - extra : blockIdx.x + gridDim.x - extra;
            uint64_t i = num_tiles * R + (uint64_t)turn * (W * 32);
            if (i < prm.rows) {
                for (; i < prm.rows; i += (uint64_t)gridDim.x * (W * 32))
                    if (i + ctid < prm.rows) process_row_global<L>(prm, i + ctid, acc, bad);
                acc.tile_done(prm, lane);
            }
        }
        uint32_t k = 0;
        for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x, ++k) {
            const uint32_t s = k % S;
            // Every lane waits (acquiring the bulk-copy writes); the warp proceeds only together.
            const bool landed = mbar_wait(smem_addr(&full_bar[s]), (k / S) & 1u, prm.status);
            if (!__all_sync(0xffffffffu, landed)) break;
            const uint32_t base = ring + s * kStage;
#pragma unroll
            for (uint32_t it = 0; it < kSteps / (W * 32); ++it)
                process_step<L, R>(prm, base, ctid + it * (W * 32), prm.cutoff, lut, acc, bad);
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&empty_bar[s]));
            acc.tile_done(prm, lane);
        }
        acc.finish(prm, lane);
        if (bad && prm.status) atomicOr(prm.status, kStatusDomain);
        acc.flush(WarpRecord{warp_rec + warp * (G * kNumAggs)}, lane);
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)(G * kNumAggs)) {
        uint64_t lo = red[2 * threadIdx.x], hi = red[2 * threadIdx.x + 1];
#pragma unroll
        for (uint32_t w = 0; w < W; ++w) {
            const ulonglong2 v = warp_rec[w * (G * kNumAggs) + threadIdx.x];
            lo += v.x;
            hi += v.y + (lo < v.x ? 1u : 0u);
        }
        red[2 * threadIdx.x] = lo;
        red[2 * threadIdx.x + 1] = hi;
    }
    __syncthreads();
    if (prm.records) {
        // Per-CTA record instead of atomics: one thread per (group, aggregate), summing the codes
        // that map to the group.
        unsigned long long* rec = prm.records + (uint64_t)blockIdx.x * (kNumGroups * kNumAggs * 2);
        for (uint32_t i = threadIdx.x; i < (uint32_t)(kNumGroups * kNumAggs); i += blockDim.x) {
            const uint32_t grp = i / kNumAggs, agg = i % kNumAggs;
            uint64_t lo = 0, hi = 0;
            for (uint32_t code = 0; code < (uint32_t)G; ++code) {
                if (((G == 4) ? prm.pair_group[code] : code) != grp) continue;
                uint64_t clo = red[2 * (code * kNumAggs + agg)], chi = red[2 * (code * kNumAggs + agg) + 1];
                if (agg == kAggQty && prm.qty_scale != 1u) {
                    const unsigned __int128 v = ((unsigned __int128)chi << 64 | clo) * prm.qty_scale;
                    clo = (uint64_t)v;
                    chi = (uint64_t)(v >> 64);
                }
                const uint64_t nlo = lo + clo;
                hi += chi + (nlo < lo ? 1u : 0u);
                lo = nlo;
            }
            rec[2 * i] = lo;
            rec[2 * i + 1] = hi;
        }
        return;
    }
    for (uint32_t i = threadIdx.x; i < (uint32_t)(G * kNumAggs); i += blockDim.x) {
        const uint32_t code = i / kNumAggs, agg = i % kNumAggs;
        const uint32_t grp = (G == 4) ? prm.pair_group[code] : code;
        uint64_t lo = red[2 * i], hi = red[2 * i + 1];
        if (agg == kAggQty && prm.qty_scale != 1u) {
            // 128 x 32 -> 128 multiply (sum of quantity in whole units -> hundredths)
            const uint64_t l_lo = (lo & 0xFFFFFFFFull) * prm.qty_scale;
            const uint64_t l_hi = (lo >> 32) * prm.qty_scale;
            const uint64_t nlo = l_lo + (l_hi << 32);
            hi = hi * prm.qty_scale + (l_hi >> 32) + (nlo < l_lo ? 1u : 0u);
            lo = nlo;
        }
        atomic_add_u128(prm.out + 2 * (grp * kNumAggs + agg), lo, hi);
    }
}

// ---------------------------------------------------------------------------------------------
// Host launch table
// ---------------------------------------------------------------------------------------------

template <int L, int P, bool kWide>
static cudaError_t launch_sized(const ScanParams& prm, int sm_count, int max_blocks, cudaStream_t stream) {
    constexpr uint32_t R = kTileRows<L, P, kWide>;
    constexpr uint32_t S = kStages<L, P>;
    constexpr uint32_t W = kConsumerWarps<L, P, kWide>;
    constexpr int G = LayoutTraits<L>::kCodes;
    constexpr uint32_t dyn =
        S * stage_bytes<L>(R) +
        (P == kPlaceSharedMemPerThread ? 8u * Entry<L == kLayUncomp>::kWords * G * W * 32u
         : P == kPlaceInRegisters      ? AccWarpLane<G, L == kLayUncomp, W * 32u>::kTableBytes
                                       : 0u);
    static_assert(dyn + sizeof(ulonglong2) * W * G * kNumAggs + 2048 <= 227 * 1024, "ring and tables beside the static shared memory");
    cudaError_t e = cudaFuncSetAttribute(q1_scan_kernel<L, P, kWide>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = scan_grid_blocks(L, P, prm.rows, sm_count, max_blocks);
    q1_scan_kernel<L, P, kWide><<<blocks, (W + 1) * 32, dyn, stream>>>(prm);
    return cudaGetLastError();
}

static uint32_t most_ctas(int sm_count, int max_blocks) {   // one CTA per SM (shared-memory bound)
    return max_blocks > 0 && max_blocks < sm_count ? (uint32_t)max_blocks : (uint32_t)sm_count;
}

template <int L, int P>
static cudaError_t launch_one(const ScanParams& prm, int sm_count, int max_blocks, cudaStream_t stream) {
    if constexpr (scan_has_wide(L, P))
        if (scan_is_wide(L, P, prm.rows, most_ctas(sm_count, max_blocks)))
            return launch_sized<L, P, true>(prm, sm_count, max_blocks, stream);
    return launch_sized<L, P, false>(prm, sm_count, max_blocks, stream);
}

template <int L>
static cudaError_t launch_layout(int placement, const ScanParams& prm, int sm_count, int max_blocks, cudaStream_t st) {
    switch (placement) {
        case kPlaceInRegisters: return launch_one<L, kPlaceInRegisters>(prm, sm_count, max_blocks, st);
        case kPlaceInRegistersPerThread: return launch_one<L, kPlaceInRegistersPerThread>(prm, sm_count, max_blocks, st);
        case kPlaceLocalMem: return launch_one<L, kPlaceLocalMem>(prm, sm_count, max_blocks, st);
        case kPlaceSharedMemPerThread: return launch_one<L, kPlaceSharedMemPerThread>(prm, sm_count, max_blocks, st);
        case kPlaceGlobal: return launch_one<L, kPlaceGlobal>(prm, sm_count, max_blocks, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_scan(int layout, int placement, const ScanParams& prm, int sm_count, int max_blocks,
                        cudaStream_t stream) {
    switch (layout) {
        case kLayPair: return launch_layout<kLayPair>(placement, prm, sm_count, max_blocks, stream);
        case kLayPairFilter: return launch_layout<kLayPairFilter>(placement, prm, sm_count, max_blocks, stream);
        case kLaySep: return launch_layout<kLaySep>(placement, prm, sm_count, max_blocks, stream);
        case kLaySepFilter: return launch_layout<kLaySepFilter>(placement, prm, sm_count, max_blocks, stream);
        case kLayUncomp: return launch_layout<kLayUncomp>(placement, prm, sm_count, max_blocks, stream);
        default: return cudaErrorInvalidValue;
    }
}

namespace {

struct Geometry {
    uint32_t warps, tile_rows;
};
template <int L, bool kWide>
Geometry geometry_of(int placement) {
    switch (placement) {
        case kPlaceInRegisters:
            return {kConsumerWarps<L, kPlaceInRegisters, kWide>, kTileRows<L, kPlaceInRegisters, kWide>};
        case kPlaceInRegistersPerThread:
            return {kConsumerWarps<L, kPlaceInRegistersPerThread, kWide>, kTileRows<L, kPlaceInRegistersPerThread, kWide>};
        case kPlaceLocalMem: return {kConsumerWarps<L, kPlaceLocalMem, kWide>, kTileRows<L, kPlaceLocalMem, kWide>};
        case kPlaceSharedMemPerThread:
            return {kConsumerWarps<L, kPlaceSharedMemPerThread, kWide>, kTileRows<L, kPlaceSharedMemPerThread, kWide>};
        default: return {kConsumerWarps<L, kPlaceGlobal, kWide>, kTileRows<L, kPlaceGlobal, kWide>};
    }
}
template <int L>
Geometry geometry_of(int placement, bool wide) {
    return wide ? geometry_of<L, true>(placement) : geometry_of<L, false>(placement);
}
Geometry geometry(int layout, int placement, bool wide) {
    switch (layout) {
        case kLayPair: return geometry_of<kLayPair>(placement, wide);
        case kLayPairFilter: return geometry_of<kLayPairFilter>(placement, wide);
        case kLaySep: return geometry_of<kLaySep>(placement, wide);
        case kLaySepFilter: return geometry_of<kLaySepFilter>(placement, wide);
        default: return geometry_of<kLayUncomp>(placement, wide);
    }
}

}  // namespace

uint64_t scan_max_rows_per_launch(int layout, int placement, uint32_t grid) {
    const Geometry g = geometry(layout, placement, false);   // the fewer threads
    // Whole tiles of a CTA, each thread its rows of every one, less one that leaves room for its tail rows (at
    // most a tile's).
    const uint32_t rows_per_thread = g.tile_rows / (g.warps * 32u);
    const uint64_t n = (uint64_t)grid * (kMaxThreadRows / rows_per_thread - 1u) * g.tile_rows;
    return std::min<uint64_t>(n, (1ull << 31) / g.tile_rows * g.tile_rows);
}

uint32_t scan_grid_blocks(int layout, int placement, uint64_t rows, int sm_count, int max_blocks) {
    const uint32_t cap = most_ctas(sm_count, max_blocks);
    const uint64_t tiles = rows / geometry(layout, placement, scan_is_wide(layout, placement, rows, cap)).tile_rows;
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(tiles, 1), cap);
}

uint32_t scan_tile_rows(int layout, int placement) { return geometry(layout, placement, false).tile_rows; }

}  // namespace q1
