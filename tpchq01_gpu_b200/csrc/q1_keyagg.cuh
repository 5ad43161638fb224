// Group-key aggregation engines shared by the group-key kernel (groupkey_kernels.cu) and the
// batch kernel (batch_kernels.cu): the Q1 predicate and aggregates over a 13 B/row tile
// (ship u16 | qty u8 | disc u8 | tax u8 | price u32 | key u32), grouped by key < num_groups.
// The per-row arithmetic is the reference's (src/kernels/ht_in_global_mem.hpp:31-49) with
// group = key.
//
// Engines (one per placement):
//   PlaneRegs<NG>  num_groups <= NG (4 or 8): per-thread byte-plane dot products (dp4a), four
//                  rows per instruction, as in the scan kernel, over three price byte planes (a
//                  row with a price >= 2^24 goes to the CTA's 128-bit sums); no atomics until a
//                  flush.
//   Cube3Table     num_groups <= 64: a shared-memory table per (group, discount, tax) cell; a
//                  row adds its count, its quantity and its price: three atomics.
//   FewTable       num_groups <= 4, in the batch kernel: eight of those tables, by lane, and a slot
//                  per lane and group for rows outside their domain.
//   CubeTable      num_groups <= 1024: a shared-memory table per (group, discount) cell. A row
//                  adds its count, price and tax * price to its cell and its quantity to its
//                  group's word; the discounted sums follow exactly at the flush, because the
//                  discount of a cell is known there: sum (100-d) p = sum_d (100-d) P_d and
//                  sum (100-d)(100+t) p = sum_d (100-d) (100 P_d + TP_d).
//   SlotTable      one shared-memory slot per key below the table's size (2048 in the batch
//                  kernel, 4096 in the group-key kernel): count, discount, quantity, price,
//                  discount x price, charge; disc_price follows at the flush as
//                  100 sum p - sum d p.
//   global         every row reduces straight into the scratch accumulators.
// The shared tables use only 32-bit shared atomics (64-bit shared atomics are far slower).
// Counts and quantities cannot wrap a 32-bit word between two flushes (at most 2^23 rows per
// CTA: count < 2^24, quantity <= 255 * 2^23 < 2^32), so their atomics need no result and no carry
// check. (Packing a count and 2^24 x its quantity into one word saved an atomic but wrapped about
// every tenth row of a cell, so the warp-voted carry branch ran on nearly every quad: 11.7 shared
// atomic instructions per warp and quad where 8 were needed.) Price sums can wrap: the slot table
// and the (group, discount, tax) cube keep them as (low word, carry word) pairs: the low word's
// atomic returns the old value, and a wrap adds the carry to the high word. The
// (group, discount) cube keeps only the low words of its cells, so that 1024 groups fit: a wrap of
// a price or tax-price word (a few rows in a thousand) is counted in three words of its group
// (wraps, and the cells' 100 - d summed over price and over tax-price wraps), from which the
// flush adds what the wraps are worth. (Sending each wrap's 2^32 straight to the group's scratch
// sums in global memory serialised on the L2 when one key holds many rows: Zipf keys over 1024
// groups at full pass 2.98 ms per 600 M rows, 1.57 ms without those global atomics.) Rows
// outside the tables' fast domain
// (discount > 10, tax > 8 or price >= 2^24; TPC-H data has none) take the global path, the FewTable's
// its slots, so every result is exact over the whole compressed domain.
//
// Scratch per group (8 x u64, zeroed before a launch): count, quantity (whole units), discount,
// price, disc_price = a4 + 2^32 a5, charge = a6 + 2^32 a7; folded into an int128 table later.
#pragma once

#include <stdint.h>

#include "q1_common.cuh"
#include "q1_ptx.cuh"
#include "q1_quad.cuh"

namespace q1 {
namespace ka {

using namespace ptx;

// ---------------------------------------------------------------------------------------------
// Tile layout (TR rows per tile, TR a multiple of 16, so every column offset is a multiple of 16
// bytes): ship u16 | qty u8 | disc u8 | tax u8 | price u32 | key u32
// ---------------------------------------------------------------------------------------------
template <uint32_t TR>
struct TileLayout {
    static_assert(TR % 16 == 0, "column offsets must stay 16-byte aligned");
    static constexpr uint32_t kOffShip = 0, kOffQty = 2 * TR, kOffDisc = 3 * TR, kOffTax = 4 * TR,
                              kOffPrice = 5 * TR, kOffKey = 9 * TR;
    static constexpr uint32_t kStageBytes = 13 * TR;
    static __host__ __device__ constexpr uint32_t col_bytes(int c) { return c == 0 ? 2 * TR : (c < 4 ? TR : 4 * TR); }
    static __host__ __device__ constexpr uint32_t col_off(int c) {
        return c == 0 ? kOffShip
                      : (c == 1 ? kOffQty : (c == 2 ? kOffDisc : (c == 3 ? kOffTax : (c == 4 ? kOffPrice : kOffKey))));
    }
};

// Flush cadences. Plane partials: at most 2^15 rows per thread; every consumer thread handles at
// most 8 rows of a tile (the kernels assert it), so 4032 tiles leave room for one more partial
// tile.
// Shared tables: at most 2^23 rows per CTA between flushes keeps every packed field and carry
// word below its limit (count < 2^24 per cell; carry words < 2^32).
constexpr uint32_t kPlaneFlushTiles = 4032;
constexpr uint64_t kTableFlushRows = 1ull << 23;

constexpr uint32_t kCubeMaxGroups = 1024;
constexpr uint32_t kCubeDisc = 11;          // discount 0..10
constexpr uint32_t kCubeWords = 3;          // count, price, tax * price (low words)
constexpr uint32_t kCube3MaxGroups = 64;
constexpr uint32_t kCubeTax = 9;            // tax 0..8
constexpr uint32_t kCube3Words = 4;         // count, quantity, price low, price carry
constexpr uint32_t kSlots = 2048;
constexpr uint32_t kSlotWords = 9;          // count, discount, quantity, price lo/hi, discount x price lo/hi, charge lo/hi

// cells, then (CubeTable) kCubeGroupWords words per group: quantity and three wrap counters
constexpr uint32_t kCubeGroupWords = 4;
// (the groups' words by place: CubeTable::place)
__host__ __device__ constexpr uint32_t cube_places(uint32_t num_groups) { return (num_groups + 63) & ~63u; }
__host__ __device__ constexpr uint32_t cube_bytes(uint32_t num_groups) {
    return (num_groups * kCubeDisc * kCubeWords + cube_places(num_groups) * kCubeGroupWords) * 4;
}
__host__ __device__ constexpr uint32_t cube3_bytes(uint32_t num_groups) {
    return num_groups * kCubeDisc * kCubeTax * kCube3Words * 4;
}
__host__ __device__ constexpr uint32_t slot_bytes(uint32_t slots) { return slots * kSlotWords * 4; }

// ---------------------------------------------------------------------------------------------
// Scratch updates
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void red_add(unsigned long long* p, uint64_t v) {
    if (v) asm volatile("red.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void scratch_add(unsigned long long* acc, uint32_t g, uint64_t cnt, uint64_t q, uint64_t d,
                                            uint64_t p, uint64_t dp_lo, uint64_t dp_hi, uint64_t ch_lo, uint64_t ch_hi) {
    unsigned long long* a = acc + 8ull * g;
    red_add(a + 0, cnt);
    red_add(a + 1, q);
    red_add(a + 2, d);
    red_add(a + 3, p);
    red_add(a + 4, dp_lo);
    red_add(a + 5, dp_hi);
    red_add(a + 6, ch_lo);
    red_add(a + 7, ch_hi);
}

// One passing row straight into the scratch (the global placement and the slow path).
__device__ __forceinline__ void scratch_row(unsigned long long* acc, uint32_t key, uint32_t q, uint32_t d, uint32_t t,
                                            uint32_t p) {
    const uint32_t a = 100u - d;
    const uint64_t dp = (uint64_t)a * p, ch = (uint64_t)(a * (100u + t)) * p;
    scratch_add(acc, key, 1, q, d, p, dp & 0xFFFFFFFFull, dp >> 32, ch & 0xFFFFFFFFull, ch >> 32);
}

// ---------------------------------------------------------------------------------------------
// Count and quantity in one word: rows add q + 2^16 (q <= 255). Exact for any number of rows, from the
// word and the two carries an atomic's old value shows: out of the low half (every 65536 of quantity,
// about 2,600 rows) C times and out of the word K times,
//   quantity = low half + 2^16 C     count = high half + 2^16 K - C.
// Both are counted per group, C and K and the same weighted with the cell's discount (for the sum of
// discounts), in kPackedWords words: one atomic a row instead of two, for a branch 0.04% of the rows take.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kPackedWords = 4;   // C, sum d over C, K, sum d over K
__device__ __forceinline__ uint32_t packed_row(uint32_t q) { return q + 0x10000u; }
__device__ __forceinline__ bool packed_carries(uint32_t old, uint32_t q) {
    return (old & 0xFFFFu) + q > 0xFFFFu || old > ~packed_row(q);
}
// Counts an added row's carries, if any, in the group's words gw[0], gw[stride], ...
__device__ __forceinline__ void packed_carry(uint32_t* gw, uint32_t stride, uint32_t old, uint32_t q, uint32_t d) {
    if ((old & 0xFFFFu) + q > 0xFFFFu) {
        atomicAdd(gw, 1u);
        atomicAdd(gw + stride, d);
    }
    if (old > ~packed_row(q)) {
        atomicAdd(gw + 2 * stride, 1u);
        atomicAdd(gw + 3 * stride, d);
    }
}
// A group's count, quantity and sum of discounts from its cells' words.
struct PackedSums {
    uint64_t cnt, q, disc;
    // the carries (their words are zeroed)
    __device__ __forceinline__ void start(uint32_t* gw, uint32_t stride) {
        const uint64_t C = gw[0], Cd = gw[stride], K = gw[2 * stride], Kd = gw[3 * stride];
        gw[0] = gw[stride] = gw[2 * stride] = gw[3 * stride] = 0;
        q = C << 16;
        cnt = (K << 16) - C;
        disc = (Kd << 16) - Cd;
    }
    __device__ __forceinline__ void add(uint32_t w, uint32_t d) {   // a cell's word, its discount
        q += w & 0xFFFFu;
        cnt += w >> 16;
        disc += (uint64_t)d * (w >> 16);
    }
};

// ---------------------------------------------------------------------------------------------
// A quad: four consecutive rows of a tile
// ---------------------------------------------------------------------------------------------
struct KeyQuad {
    uint32_t PM;        // byte r = 0xFF iff row r passes the predicate
    uint32_t Q, D, X;   // bytes r: quantity, discount, tax
    uint32_t p[4];
    uint32_t k[4];
};

// Rows 4j..4j+3 of the TR-row tile at shared address `base`. `bad` becomes nonzero for a value
// outside the compressed domain (ship offset > 32767, discount > 100).
template <uint32_t TR>
__device__ __forceinline__ KeyQuad load_quad(uint32_t base, uint32_t j, int32_t cut, uint32_t& bad) {
    using TL = TileLayout<TR>;
    KeyQuad x;
    x.PM = quad_pass_mask(lds_v2(base + TL::kOffShip + 8 * j), cut, bad);
    x.Q = lds_u32(base + TL::kOffQty + 4 * j);
    x.D = lds_u32(base + TL::kOffDisc + 4 * j);
    x.X = lds_u32(base + TL::kOffTax + 4 * j);
    const uint4 P = lds_v4(base + TL::kOffPrice + 16 * j);
    const uint4 K = lds_v4(base + TL::kOffKey + 16 * j);
    bad |= disc_out_of_domain4(x.D);
    x.p[0] = P.x, x.p[1] = P.y, x.p[2] = P.z, x.p[3] = P.w;
    x.k[0] = K.x, x.k[1] = K.y, x.k[2] = K.z, x.k[3] = K.w;
    return x;
}

// A quad with no passing row (for lanes past the end of a partial tile, so that every lane of
// the warp takes part in the warp votes of the table engines).
__device__ __forceinline__ KeyQuad empty_quad() {
    KeyQuad x;
    x.PM = x.Q = x.D = x.X = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) x.p[r] = x.k[r] = 0;
    return x;
}

// One row read from global memory (tail rows of a partial tile), as a quad whose rows 1..3 fail.
__device__ __forceinline__ KeyQuad load_row(const uint8_t* const col[6], uint64_t i, int32_t cut, uint32_t& bad) {
    KeyQuad x;
    const uint32_t ship = __ldg(reinterpret_cast<const uint16_t*>(col[0]) + i);
    const uint32_t d = __ldg(col[2] + i);
    bad |= (ship > 32767u || d > 100u) ? 1u : 0u;
    x.PM = (int32_t)ship <= cut ? 0xFFu : 0u;
    x.Q = __ldg(col[1] + i);
    x.D = d;
    x.X = __ldg(col[3] + i);
    x.p[0] = __ldg(reinterpret_cast<const uint32_t*>(col[4]) + i);
    x.k[0] = __ldg(reinterpret_cast<const uint32_t*>(col[5]) + i);
    x.p[1] = x.p[2] = x.p[3] = 0;
    x.k[1] = x.k[2] = x.k[3] = 0;
    return x;
}

// ---------------------------------------------------------------------------------------------
// PlaneRegs: per-thread dp4a byte planes for num_groups <= NG
// ---------------------------------------------------------------------------------------------
template <int NG>
struct PlaneRegs {
    // Three price byte planes a group: a passing row with a price >= 2^24 (none in TPC-H data) goes
    // to `slow` behind one warp vote, so that eight groups' planes fit in registers (the fourth plane
    // took 32 more a thread and made the 8-group kernel spill).
    GroupPlanesT<3> g[NG];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < NG; ++i) g[i].zero();
    }
    // Every lane of the warp calls it (warp vote). slow(key, quantity, discount, tax, price): one row.
    template <class Slow>
    __device__ __forceinline__ void add(const KeyQuad& kq, uint32_t num_groups, uint32_t& bad, Slow&& slow) {
        uint32_t OH = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t key = kq.k[r];
            const bool in = key < num_groups;
            if (!in && ((kq.PM >> (8 * r)) & 1u)) bad = 1u;
            OH |= (in ? (1u << (key & 7u)) : 0u) << (8 * r);
        }
        Quad x;
        x.OH = OH & kq.PM;
        x.Q = kq.Q;
        x.D = kq.D;
#pragma unroll
        for (int r = 0; r < 4; ++r) x.p[r] = kq.p[r];
        quad_derive(x, kq.X);
        if (__any_sync(0xffffffffu, x.P[3])) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (((x.P[3] >> (8 * r)) & 0xFFu) && ((x.OH >> (8 * r)) & 0xFFu)) {
                    slow(kq.k[r], (kq.Q >> (8 * r)) & 0xFFu, (kq.D >> (8 * r)) & 0xFFu, (kq.X >> (8 * r)) & 0xFFu,
                         kq.p[r]);
                    x.OH &= ~(0xFFu << (8 * r));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NG; ++i) g[i].template add_quad<false>(x.OH, (uint32_t)i, x);
    }
    // Warp sum of aggregate a of group i (kAgg*; quantity in whole units): at most 2^15 rows a thread and
    // prices below 2^24, so price < 2^39, disc_price < 2^46 and charge < 2^54.2 a thread, < 2^60 a warp.
    __device__ __forceinline__ uint64_t warp_total(int i, int a) const {
        const uint64_t v = g[i].value(a);
        return a == kAggCount || a == kAggQty || a == kAggDisc ? warp_sum<27>(v).lo
               : a == kAggCharge                               ? warp_sum<63>(v).lo
                                                               : warp_sum<54>(v).lo;
    }
};

// ---------------------------------------------------------------------------------------------
// CubeTable: shared (group, discount) cells
// ---------------------------------------------------------------------------------------------
// Wraps are counted in the group's shared words. (Sent straight to the group's scratch sums instead, as the
// batch kernel did: 64 instances of 1024 groups 299 us instead of 292, and frequent keys serialise.)
struct CubeTable {
    uint32_t* w;       // [kCubeWords][cells]: count, price, tax * price (low words)
    uint32_t* gw;      // [kCubeGroupWords][places]: quantity; wraps of the group's cells' price words;
                       // sum (100 - d) over those wraps; sum (100 - d) over wraps of tax * price
                       // words
    uint32_t cells, places;
    // A group's place in gw, within its 64: consecutive groups lie in consecutive banks, and groups any power of two
    // apart spread over the banks too. (By group alone, keys that are multiples of 128, 60 M rows of 1024 groups in the
    // batch kernel, took 368 us instead of 238. group ^ (group >> 5) leaves steps of 31, 33 and 62 in one bank; turning
    // every 32 groups by 21 banks spreads nearly any step, but its third instruction made 600 groups, 60 M rows in
    // the group-key kernel, 150 -> 156 us.)
    static __device__ __forceinline__ uint32_t place(uint32_t group) { return group ^ (group >> 4); }
    __device__ __forceinline__ void bind(uint8_t* base, uint32_t num_groups) {
        w = reinterpret_cast<uint32_t*>(base);
        cells = num_groups * kCubeDisc;
        places = cube_places(num_groups);
        gw = w + kCubeWords * cells;
    }
    __device__ __forceinline__ void zero(uint32_t tid, uint32_t nthreads) {
        for (uint32_t i = tid; i < kCubeWords * cells + kCubeGroupWords * places; i += nthreads) w[i] = 0;
    }
    // Rows r of a quad with bit r of `m` set (passing, key < num_groups, fast domain). All
    // atomics of the quad are issued before any carry is checked, so their latencies overlap.
    static constexpr bool kPacked = true, kSlots = false;
    // The quantity, discount and tax bytes of the four rows packed in Q, D, X. A cell's
    // count and a group's quantity cannot wrap between flushes (at most 2^23 rows per CTA:
    // count < 2^24, quantity <= 255 * 2^23 < 2^32), so their atomics need no result. A wrap of a
    // cell's price or tax * price word (a few rows in a thousand) is worth, with the cell's
    // discount d and a = 100 - d, 2^32 of price, 2^32 a of disc_price and 2^32 100 a of charge,
    // or 2^32 a of charge.
    __device__ __forceinline__ void add_quad_packed(uint32_t m, const uint32_t key[4], uint32_t Q, uint32_t D,
                                                    uint32_t X, const uint32_t p[4]) {
        uint32_t c[4], vt[4], op[4], ot[4];
        if (!__any_sync(0xffffffffu, m)) return;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            c[r] = key[r] * kCubeDisc + ((D >> (8 * r)) & 0xFFu);
            vt[r] = ((X >> (8 * r)) & 0xFFu) * p[r];                     // t p < 2^28
            op[r] = ot[r] = 0;
            if ((m >> r) & 1u) {
                atomicAdd(w + c[r], 1u);
                atomicAdd(gw + place(key[r]), (Q >> (8 * r)) & 0xFFu);
                op[r] = atomicAdd(w + cells + c[r], p[r]);
                ot[r] = atomicAdd(w + 2 * cells + c[r], vt[r]);
            }
        }
        // a word wrapped iff old > ~added (rows not added have old == 0): one predicate, and
        // the rows only in the rare branch
        bool wrap = false;
#pragma unroll
        for (int r = 0; r < 4; ++r) wrap |= (op[r] > ~p[r]) | (ot[r] > ~vt[r]);
        if (__any_sync(0xffffffffu, wrap)) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint32_t a = 100u - ((D >> (8 * r)) & 0xFFu);
                uint32_t* g = gw + place(key[r]);
                if (op[r] > ~p[r]) {
                    atomicAdd(g + places, 1u);
                    atomicAdd(g + 2 * places, a);
                }
                if (ot[r] > ~vt[r]) atomicAdd(g + 3 * places, a);
            }
        }
    }
    // Cells -> per-group sums -> scratch, from group `first` on (and round to it); the caller
    // synchronises the consumers around it.
    __device__ __forceinline__ void flush(unsigned long long* acc, uint32_t num_groups, uint32_t tid, uint32_t nthreads,
                                          uint32_t first = 0) {
        for (uint32_t i = tid; i < num_groups; i += nthreads) {
            const uint32_t g = i + first < num_groups ? i + first : i + first - num_groups;
            uint32_t* const of = gw + place(g);
            const uint64_t q = of[0], pw = of[places], aw = of[2 * places], tw = of[3 * places];
#pragma unroll
            for (uint32_t j = 0; j < kCubeGroupWords; ++j) of[j * places] = 0;
            uint64_t cnt = 0, dsum = 0, P = pw << 32;
            unsigned __int128 DP = (unsigned __int128)aw << 32, CH = (unsigned __int128)(100u * aw + tw) << 32;
#pragma unroll
            for (uint32_t d = 0; d < kCubeDisc; ++d) {
                const uint32_t c = g * kCubeDisc + d;
                const uint32_t nd = w[c], Pd = w[cells + c], TPd = w[2 * cells + c];
                cnt += nd;
                dsum += (uint64_t)d * nd;
                P += Pd;
                DP += (uint64_t)(100u - d) * Pd;
                CH += (unsigned __int128)(100u - d) * ((uint64_t)Pd * 100u + TPd);
#pragma unroll
                for (uint32_t k = 0; k < kCubeWords; ++k) w[k * cells + c] = 0;
            }
            if (cnt)
                scratch_add(acc, g, cnt, q, dsum, P, (uint64_t)DP & 0xFFFFFFFFull, (uint64_t)(DP >> 32),
                            (uint64_t)CH & 0xFFFFFFFFull, (uint64_t)(CH >> 32));
        }
    }
};

// ---------------------------------------------------------------------------------------------
// Cube3Table: shared (group, discount, tax) cells, for num_groups <= 64. A row adds only its
// count, quantity and price: three atomics, of which only the price's can wrap (into the cell's
// carry word) between flushes. At the flush the cell's discount and tax give
// sum (100-d) p = (100-d) P and sum (100-d)(100+t) p = (100-d)(100+t) P.
// ---------------------------------------------------------------------------------------------
struct Cube3Table {
    uint32_t* w;       // [kCube3Words][cells]: count, quantity, price low word, price carry word
    uint32_t cells;
    __device__ __forceinline__ void bind(uint8_t* base, uint32_t num_groups) {
        w = reinterpret_cast<uint32_t*>(base);
        cells = num_groups * kCubeDisc * kCubeTax;
    }
    __device__ __forceinline__ void zero(uint32_t tid, uint32_t nthreads) {
        for (uint32_t i = tid; i < kCube3Words * cells; i += nthreads) w[i] = 0;
    }
    static constexpr bool kPacked = true, kSlots = false;
    // Rows r of a quad with bit r of `m` set (fast domain), the quantity, discount and tax bytes
    // of the four rows packed in Q, D, X (D and X zero in rows outside the fast domain). There
    // 9 d + t < 99 fits a byte, so one shift-and-add gives the four (discount, tax) cell offsets.
    __device__ __forceinline__ void add_quad_packed(uint32_t m, const uint32_t key[4], uint32_t Q, uint32_t D,
                                                    uint32_t X, const uint32_t p[4]) {
        uint32_t c[4], op[4];
        if (!__any_sync(0xffffffffu, m)) return;
        const uint32_t DT = (D << 3) + D + X;   // bytes r: 9 d + t (garbage outside the fast domain)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            c[r] = key[r] * (kCubeDisc * kCubeTax) + ((DT >> (8 * r)) & 0xFFu);
            op[r] = 0;
            if ((m >> r) & 1u) {
                atomicAdd(w + c[r], 1u);
                atomicAdd(w + cells + c[r], (Q >> (8 * r)) & 0xFFu);
                op[r] = atomicAdd(w + 2 * cells + c[r], p[r]);
            }
        }
        // a price word wrapped iff old > ~added (rows not added have old == 0): one predicate
        // and one vote, the rows only in the branch (a cell's price word wraps every thousand
        // rows or so; its count and quantity words cannot wrap between flushes)
        bool wrap = false;
#pragma unroll
        for (int r = 0; r < 4; ++r) wrap |= op[r] > ~p[r];
        if (__any_sync(0xffffffffu, wrap)) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (op[r] > ~p[r]) atomicAdd(w + 3 * cells + c[r], 1u);
        }
    }
    // Cells -> per-group sums -> scratch, from group `first` on (and round to it); the caller
    // synchronises the consumers around it, and every lane of its warps calls. Half a warp per group, a
    // lane per discount (a thread per group ran 99 cells one after the other: 5 us, 10^6 rows of 64 groups 26 us instead of 21). At most 2^23
    // rows of prices below 2^24 lie between flushes, so a group's largest sum, the charge, is below
    // 2^47 * 100 * 108 < 2^61.
    __device__ __forceinline__ void flush(unsigned long long* acc, uint32_t num_groups, uint32_t tid, uint32_t nthreads,
                                          uint32_t first = 0) {
        static_assert(kTableFlushRows * 10800ull <= 1ull << 37, "64-bit sums");
        const uint32_t d = tid & 15u;
        for (uint32_t i0 = tid / 32 * 2; i0 < num_groups; i0 += nthreads / 16) {
            const uint32_t i = i0 + (tid >> 4 & 1u);
            const uint32_t g = i + first < num_groups ? i + first : i + first - num_groups;
            uint32_t cnt = 0, q = 0;
            uint64_t P = 0, T = 0;   // sum over the taxes of the price, and of tax * price
            if (i < num_groups && d < kCubeDisc) {
#pragma unroll
                for (uint32_t t = 0; t < kCubeTax; ++t) {
                    const uint32_t c = (g * kCubeDisc + d) * kCubeTax + t;
                    const uint64_t Pt = ((uint64_t)w[3 * cells + c] << 32) | w[2 * cells + c];
                    cnt += w[c];
                    q += w[cells + c];
                    P += Pt;
                    T += t * Pt;
#pragma unroll
                    for (uint32_t k = 0; k < kCube3Words; ++k) w[k * cells + c] = 0;
                }
            }
            uint32_t disc = d * cnt;
            uint64_t DP = (100u - d) * P, CH = (100u - d) * (100u * P + T);
#pragma unroll
            for (uint32_t o = 8; o; o >>= 1) {
                cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
                q += __shfl_xor_sync(0xffffffffu, q, o);
                disc += __shfl_xor_sync(0xffffffffu, disc, o);
                P += __shfl_xor_sync(0xffffffffu, P, o);
                DP += __shfl_xor_sync(0xffffffffu, DP, o);
                CH += __shfl_xor_sync(0xffffffffu, CH, o);
            }
            // lane j of the half adds the group's word j
            const uint64_t s01 = d & 1u ? q : cnt, s23 = d & 1u ? P : disc, s45 = d & 1u ? DP >> 32 : DP & 0xFFFFFFFFull,
                           s67 = d & 1u ? CH >> 32 : CH & 0xFFFFFFFFull;
            if (d < 8 && i < num_groups) red_add(acc + 8ull * g + d, d & 4u ? (d & 2u ? s67 : s45) : (d & 2u ? s23 : s01));
        }
    }
};

// ---------------------------------------------------------------------------------------------
// FewTable: num_groups <= kFewGroups, in the batch kernel. kFewCopies (group, discount, tax) tables: a lane adds to
// the one of its number modulo kFewCopies, so that at most four lanes of a warp meet in a cell, as they do in a bank
// for spread values. A quad with a row outside the cells' domain goes to slots instead, one per lane and group, whose
// lanes lie in all 32 banks. So the time does not hang on the values.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kFewGroups = 4, kFewCopies = 8;
// A slot's words: count, quantity, discount, then price, disc_price and charge in pieces of 16 bits (2, 3, 3), whose sums
// over a lane's rows between flushes need no carry: at most kFewFlushRows / 32 rows and, of a last tile, one more in each
// of a team's kFewTeamWarps warps.
constexpr uint32_t kFewSlotWords = 11, kFewTeamWarps = 8;
constexpr uint64_t kFewFlushRows = (1ull << 21) - 2048;
static_assert((kFewFlushRows / 32 + kFewTeamWarps) * 0xFFFFull < 1ull << 32 && kFewFlushRows < kTableFlushRows, "a word's sum");
// words from one table to the next: the tables start four banks apart
constexpr __host__ __device__ uint32_t few_stride(uint32_t num_groups) {
    const uint32_t words = cube3_bytes(num_groups) / 4;
    return words + (32u / kFewCopies + 32u - words % 32u) % 32u;
}
constexpr __host__ __device__ uint32_t few_bytes(uint32_t num_groups) {
    return 4 * (kFewCopies * few_stride(num_groups) + kFewSlotWords * num_groups * 32);
}
// Rows r of a quad with bit r of m set into the slots at slot + 32 key, n words from word to word. (A function of its
// own, and a small one: what it needs in registers is taken from the cells' path beside it.)
static __device__ __noinline__ void few_slot_rows(uint32_t* slot, uint32_t n, uint32_t m, const KeyQuad x) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (!((m >> r) & 1u)) continue;
        const uint32_t q = (x.Q >> (8 * r)) & 0xFFu, d = (x.D >> (8 * r)) & 0xFFu, t = (x.X >> (8 * r)) & 0xFFu, p = x.p[r];
        const uint32_t a = 100u - d;
        const uint64_t dp = (uint64_t)a * p, ch = (uint64_t)(a * (100u + t)) * p;   // below 2^38.7, 2^47.2
        uint32_t* const w = slot + x.k[r] * 32;
        atomicAdd(w, 1u);
        atomicAdd(w + n, q);
        atomicAdd(w + 2 * n, d);
        atomicAdd(w + 3 * n, p & 0xFFFFu);
        atomicAdd(w + 4 * n, p >> 16);
        atomicAdd(w + 5 * n, (uint32_t)dp & 0xFFFFu);
        atomicAdd(w + 6 * n, (uint32_t)dp >> 16);
        atomicAdd(w + 7 * n, (uint32_t)(dp >> 32));
        atomicAdd(w + 8 * n, (uint32_t)ch & 0xFFFFu);
        atomicAdd(w + 9 * n, (uint32_t)ch >> 16);
        atomicAdd(w + 10 * n, (uint32_t)(ch >> 32));
    }
}
struct FewTable {
    Cube3Table cells;   // the lane's
    uint32_t* slot;     // the lane's of group 0, [kFewSlotWords][groups][32 lanes]
    uint32_t groups;
    __device__ __forceinline__ void bind(uint8_t* base, uint32_t num_groups, uint32_t lane) {
        cells.bind(base, num_groups);
        slot = cells.w + kFewCopies * few_stride(num_groups) + lane;
        cells.w += lane % kFewCopies * few_stride(num_groups);
        groups = num_groups;
    }
    static constexpr bool kPacked = true, kSlots = true;
    __device__ __forceinline__ void add_quad_packed(uint32_t m, const uint32_t key[4], uint32_t Q, uint32_t D, uint32_t X,
                                                    const uint32_t p[4]) {
        cells.add_quad_packed(m, key, Q, D, X, p);
    }
    // Rows r of a quad with bit r of m set, of any values, into the lane's slots.
    __device__ __forceinline__ void slot_rows(uint32_t m, const KeyQuad& x) const { few_slot_rows(slot, groups * 32, m, x); }
    // All tables' and slots' sums -> scratch, and zero again: a warp per group, half of the tables to each half of its
    // lanes. The caller synchronises the consumers around it; all lanes of the warps call. Of kFewFlushRows
    // rows a group's price sum is below 2^53, its disc_price below 2^60.
    __device__ __forceinline__ void flush(unsigned long long* acc, uint32_t g, uint32_t lane) {
        if (g >= groups) return;
        const uint32_t d = lane & 15u, n = groups * 32, stride = few_stride(groups), per_word = cells.cells;
        uint32_t cnt = 0, q = 0;
        uint64_t P = 0, T = 0;   // of the lane's cells: sum over the taxes of the price, and of tax * price
        if (d < kCubeDisc) {
            uint32_t* const first = cells.w - lane % kFewCopies * stride + (g * kCubeDisc + d) * kCubeTax;
            for (uint32_t k = lane / 16; k < kFewCopies; k += 2) {
                uint32_t* const w = first + k * stride;
#pragma unroll
                for (uint32_t t = 0; t < kCubeTax; ++t) {
                    const uint64_t Pt = ((uint64_t)w[3 * per_word + t] << 32) | w[2 * per_word + t];
                    cnt += w[t];
                    q += w[per_word + t];
                    P += Pt;
                    T += t * Pt;
#pragma unroll
                    for (uint32_t j = 0; j < kCube3Words; ++j) w[j * per_word + t] = 0;
                }
            }
        }
        uint32_t disc = d * cnt;
        uint64_t DP = (100u - d) * P, CH = (100u - d) * (100u * P + T);
        uint64_t chl = CH & 0xFFFFFFFFull, chh = CH >> 32;
        uint32_t* const s = slot + g * 32;
        if (__any_sync(0xffffffffu, *s)) {
            uint64_t w[kFewSlotWords];
#pragma unroll
            for (uint32_t j = 0; j < kFewSlotWords; ++j) {
                w[j] = s[j * n];
                s[j * n] = 0;
            }
            cnt += (uint32_t)w[0];
            q += (uint32_t)w[1];
            disc += (uint32_t)w[2];
            P += w[3] + (w[4] << 16);
            DP += w[5] + (w[6] << 16) + (w[7] << 32);
            chl += w[8] + (w[9] << 16);
            chh += w[10];
        }
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        q = __reduce_add_sync(0xffffffffu, q);
        disc = __reduce_add_sync(0xffffffffu, disc);
        P = warp_sum<64>(P).lo, DP = warp_sum<64>(DP).lo, chl = warp_sum<54>(chl).lo, chh = warp_sum<54>(chh).lo;
        // lane j adds the group's word j
        const uint64_t s01 = lane & 1u ? q : cnt, s23 = lane & 1u ? P : disc,
                       s45 = lane & 1u ? DP >> 32 : DP & 0xFFFFFFFFull, s67 = lane & 1u ? chh : chl;
        if (lane < 8) red_add(acc + 8ull * g + lane, lane & 4u ? (lane & 2u ? s67 : s45) : (lane & 2u ? s23 : s01));
    }
};

// ---------------------------------------------------------------------------------------------
// SlotTable: shared per-group slots for keys < slots
// ---------------------------------------------------------------------------------------------
struct SlotTable {
    static constexpr bool kPacked = false, kSlots = false;
    uint32_t* w;       // [kSlotWords][slots]
    uint32_t slots;
    __device__ __forceinline__ void bind(uint8_t* base, uint32_t n) {
        w = reinterpret_cast<uint32_t*>(base);
        slots = n;
    }
    __device__ __forceinline__ void zero(uint32_t tid, uint32_t nthreads) {
        for (uint32_t i = tid; i < kSlotWords * slots; i += nthreads) w[i] = 0;
    }
    // Rows r of a quad with bit r of `m` set (passing, key < slots, fast domain); atomics first,
    // carries after.
    __device__ __forceinline__ void add_quad(uint32_t m, const uint32_t key[4], const uint32_t q[4],
                                             const uint32_t d[4], const uint32_t t[4], const uint32_t p[4]) {
        const uint32_t S = slots;
        uint32_t vd[4], cl[4], ch[4], op[4], od[4], oc[4];
        if (!__any_sync(0xffffffffu, m)) return;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t a = 100u - d[r];
            vd[r] = d[r] * p[r];         // d p < 2^28 (the discounted price follows at the flush)
            const uint64_t c64 = (uint64_t)(a * (100u + t[r])) * p[r];
            cl[r] = (uint32_t)c64;
            ch[r] = (uint32_t)(c64 >> 32);
            op[r] = od[r] = oc[r] = 0;
            if ((m >> r) & 1u) {
                const uint32_t s = key[r];
                atomicAdd(w + s, 1u);
                atomicAdd(w + S + s, d[r]);
                atomicAdd(w + 2 * S + s, q[r]);
                op[r] = atomicAdd(w + 3 * S + s, p[r]);
                od[r] = atomicAdd(w + 5 * S + s, vd[r]);
                oc[r] = atomicAdd(w + 7 * S + s, cl[r]);
            }
        }
        // a word wrapped iff old > ~added (rows not added have old == 0): one predicate, and
        // the rows only in the rare branch
        bool wrap = false;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            wrap |= (op[r] > ~p[r]) | (od[r] > ~vd[r]);
            ch[r] = ((m >> r) & 1u) ? ch[r] + (oc[r] > ~cl[r] ? 1u : 0u) : 0u;
        }
        // the charge's high word is nonzero for most rows: added per row
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (ch[r]) atomicAdd(w + 8 * S + key[r], ch[r]);
        if (__any_sync(0xffffffffu, wrap)) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (op[r] > ~p[r]) atomicAdd(w + 4 * S + key[r], 1u);
                if (od[r] > ~vd[r]) atomicAdd(w + 6 * S + key[r], 1u);
            }
        }
    }
    __device__ __forceinline__ void flush(unsigned long long* acc, uint32_t, uint32_t tid, uint32_t nthreads,
                                          uint32_t first = 0) {
        const uint32_t S = slots;
        for (uint32_t i = tid; i < S; i += nthreads) {
            const uint32_t s = i + first < S ? i + first : i + first - S;
            const uint64_t cnt = w[s];
            if (cnt) {
                const uint64_t P = ((uint64_t)w[4 * S + s] << 32) | w[3 * S + s];
                const uint64_t DP = 100u * P - (((uint64_t)w[6 * S + s] << 32) | w[5 * S + s]);   // sum (100 - d) p
                scratch_add(acc, s, cnt, w[2 * S + s], w[S + s], P, DP & 0xFFFFFFFFull, DP >> 32, w[7 * S + s],
                            w[8 * S + s]);
            }
#pragma unroll
            for (uint32_t k = 0; k < kSlotWords; ++k) w[k * S + s] = 0;
        }
    }
};

// One quad into a shared table: rows in the table's fast domain go to the table, other passing rows
// with key < num_groups straight to the scratch (a FewTable's to its slots), passing rows with
// key >= num_groups make `bad` nonzero.
// All lanes of the warp call it (the slow path, the tables' early exit when no lane of the warp
// has a row to add, and the carries use warp votes).
template <class Table>
__device__ __forceinline__ void table_quad(Table& tab, const KeyQuad& x, uint32_t num_groups, uint32_t hot,
                                           unsigned long long* acc, uint32_t& bad) {
    // rows outside the tables' fast domain: bit 7 of byte r set when d > 10, t > 8 or p >= 2^24
    const uint32_t top = __byte_perm(__byte_perm(x.p[0], x.p[1], 0x0073u), __byte_perm(x.p[2], x.p[3], 0x0073u),
                                     0x5410u);   // bytes r: top byte of p[r]
    const uint32_t outside = (((top & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | top | ((x.D & 0x7F7F7F7Fu) + 0x75757575u) |
                              x.D | ((x.X & 0x7F7F7F7Fu) + 0x77777777u) | x.X) &
                             0x80808080u;
    uint32_t m = 0, slow = 0;
    const uint32_t kmax = max(max(x.k[0], x.k[1]), max(x.k[2], x.k[3]));
    if (kmax < hot) {
        // every key of the quad in the table (hot <= num_groups): byte-parallel masks, each
        // gathered to bits 0..3 by one multiply (byte r's bit 0 lands on bit 24 + r)
        const uint32_t ob = (outside >> 7) * 0xFFu;
        m = (((x.PM & ~ob) & 0x01010101u) * 0x01020408u) >> 24;
        slow = (((x.PM & ob) & 0x01010101u) * 0x01020408u) >> 24;
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t pass = (x.PM >> (8 * r)) & 1u;
            const uint32_t key = x.k[r];
            const uint32_t in = pass & (key < num_groups ? 1u : 0u);
            bad |= pass & (key >= num_groups ? 1u : 0u);
            const uint32_t fast = in & (key < hot ? 1u : 0u) & (((outside >> (8 * r + 7)) & 1u) ^ 1u);
            m |= fast << r;
            slow |= (in & (fast ^ 1u)) << r;
        }
    }
    // rows outside the tables' fast domain (none in TPC-H data): one vote skips the path
    if (__any_sync(0xffffffffu, slow)) {
        if constexpr (Table::kSlots) {   // as good for the warp's other rows, and one path is shorter than two
            tab.slot_rows(m | slow, x);
            return;
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if ((slow >> r) & 1u)
                    scratch_row(acc, x.k[r], (x.Q >> (8 * r)) & 0xFFu, (x.D >> (8 * r)) & 0xFFu,
                                (x.X >> (8 * r)) & 0xFFu, x.p[r]);
        }
    }
    if constexpr (Table::kPacked) {
        // discount and tax bytes of in-domain rows only (d <= 10, t <= 8), so that byte-wise
        // arithmetic on them cannot carry into a neighbouring row's byte
        const uint32_t inb = ((~outside & 0x80808080u) >> 7) * 0xFFu;
        tab.add_quad_packed(m, x.k, x.Q, x.D & inb, x.X & inb, x.p);
    } else {
        uint32_t q[4], d[4], t[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            q[r] = (x.Q >> (8 * r)) & 0xFFu;
            d[r] = (x.D >> (8 * r)) & 0xFFu;
            t[r] = (x.X >> (8 * r)) & 0xFFu;
        }
        tab.add_quad(m, x.k, q, d, t, x.p);
    }
}

// Barrier of the consumer warps only (the producer keeps streaming): one arrive per warp on an
// mbarrier initialised with the warp count, bounded wait. Every consumer passes the same sequence
// of barriers, so a local phase counter tracks the parity.
struct ConsumerBarrier {
    uint32_t addr;
    uint32_t phase;
    __device__ __forceinline__ void sync(uint32_t lane, uint32_t* status) {
        __syncwarp();
        if (lane == 0) mbar_arrive(addr);
        mbar_wait(addr, phase & 1u, status);
        ++phase;
    }
};

}  // namespace ka
}  // namespace q1
