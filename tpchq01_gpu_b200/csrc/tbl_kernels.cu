// lineitem text ingestion on the GPU: the reference's lineitem::FromFile (cpu/tpch_kit.cpp:155-172
// with the TableReader tokenizer at :10-99) as one kernel over a device copy of the text.
//
// Format (dbgen .tbl): one row per '\n'-terminated line (the last line may lack the '\n'), fields
// separated by '|'. Fields 5-11 (1-based) are read, the others skipped:
//   quantity, extendedprice, discount, tax   decimals "[+-]digits[.digits]" -> 100 * int + frac
//                                             (Decimal<15,2>::ToValue, cpu/tpch_kit.hpp:52-54;
//                                             the fraction's digits are read as an integer, as
//                                             the reference's parser does)
//   returnflag, linestatus                    exactly one character (Char, cpu/tpch_kit.hpp:15-23)
//   shipdate                                  "year-month-day" -> day number counted the MonetDB
//                                             way (Date, cpu/tpch_kit.cpp:142-153): 1992-01-01 is
//                                             727563
// A line that does not match is counted as malformed (its row is written as zeros) and the host
// reports the count and the first malformed line's byte offset.
//
// Kernels:
//   tbl_count_kernel  newlines of the whole text, where only they are asked for (16-byte loads, byte
//                     compares on 32-bit words)
//   tbl_parse_kernel  one pass over the text. One persistent CTA per SM takes 63 KB tiles in ticket
//                     order and streams them into shared memory with bulk copies (three stages).
//                     Workers find the next tile's newlines with word compares and rank them by
//                     ballots, then parse the current tile's lines, a line a lane, word by word from
//                     shared memory (parse_fast; any other form goes to the byte-wise parse_line,
//                     which reads shared memory too unless the line ends beyond the stage).
//                     A control warp meanwhile sums the newlines before the tile from the counts the
//                     other CTAs published (decoupled look-back, bounded).
//
// What bounds it: instructions, 28 warp instructions a line at half of the issue slots. 6.0 M rows of
// dbgen text (757 MB, 1.0 GB with the columns, 0.15 ms at the copy bandwidth) take 0.31 ms a call;
// counting, scanning the counts and parsing byte by byte in three kernels took 1.62 ms (142 warp
// instructions a line, the text read twice). 10,000 rows: 91 -> 37 us. Lines of other forms, 1.0 M rows: a sign
// before every price 217 us (read again from the text instead of from shared memory 348, three kernels 352),
// 40 characters in the first two fields 341 (542, 389), all as dbgen writes them 88 (354). Measured on the way: tiles of
// 30 KB with two CTAs an SM 0.36 to 0.59 ms (twice the tiles to order), a look-back step of 256 tiles
// 0.1 ms more than one of 64, the newline search with 512 bytes a load across the warp 0.39 ms.
#include <cuda_runtime.h>
#include <stdint.h>

#include "q1_kernels.h"
#include "q1_ptx.cuh"

namespace q1 {

namespace tbl {

using namespace ptx;

// A CTA is 18 worker warps and one control warp, one CTA per SM (16 workers 0.336 ms, 17 0.324 ms,
// 18 0.311 ms: as many as three stages leave room for). Text positions are counted from the 16-byte
// boundary at or before the first byte, so that every tile starts on a boundary. A worker's part of a
// tile is 3.5 KB: long enough to spread what each tile costs beside the search (barriers, sums),
// and at 120 to 130 bytes a line just under 32 lines, so that a tile's lines make about one batch of
// 32 for every worker.
constexpr uint32_t kWorkers = 18;
constexpr uint32_t kThreads = (kWorkers + 1) * 32;
constexpr uint32_t kSubs = 7;                        // 16-byte pieces a lane
constexpr uint32_t kLaneBytes = kSubs * 16;
constexpr uint32_t kWords = (kSubs + 1) / 2;         // words of a lane's newline bits
constexpr uint32_t kWarpBytes = 32 * kLaneBytes;
constexpr uint32_t kTile = kWorkers * kWarpBytes;
constexpr uint32_t kAhead = 128;                     // bytes after the tile kept with it: a line's window
constexpr uint32_t kFront = 16;                      // room before the tile for right-aligned field loads
constexpr uint32_t kStageBytes = kFront + kTile + kAhead;
constexpr uint32_t kRing = 3;                        // tiles in flight or in use a CTA
constexpr uint32_t kWarpList = 192;                  // line starts listed a part (about 28 in dbgen text)
static_assert(kStageBytes % 16 == 0, "stages stay 16-byte aligned");
static_assert(kSubs % 2 == 1, "conflict-free loads of a lane's consecutive bytes");
// The shortest line that parses is four empty fields, "1|1|1|1|A|F|1-1-1" and a newline. (Lists of 96, which left lines
// of 25 bytes to the walk without a list: 1.0 M of them 2,630 us instead of 126.)
static_assert(kWarpList >= 64 && kWarpList > kWarpBytes / 22, "every line that parses is listed");
static_assert(kRing == 3, "a tile reloads the stage of the tile before it");
static_assert(kTile + kAhead + 1 <= 65535, "a tile's newlines and line starts fit 16 bits");

// Bit 7 of byte i set iff byte i of w equals the byte repeated in c4 (below 128; exact for every w).
__device__ __forceinline__ uint32_t equal_bytes(uint32_t w, uint32_t c4) {
    return ~((((w ^ c4) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;
}
// 16 bits, bit i set iff byte i of v equals the byte. The multiply gathers a word's four flags
// into its top four bits (no two partial products meet), a funnel shift appends them.
__device__ __forceinline__ uint32_t match16(const uint4& v, uint32_t c4) {
    uint32_t m = __funnelshift_l(equal_bytes(v.w, c4) * 0x00204081u, 0u, 4);
    m = __funnelshift_l(equal_bytes(v.z, c4) * 0x00204081u, m, 4);
    m = __funnelshift_l(equal_bytes(v.y, c4) * 0x00204081u, m, 4);
    return __funnelshift_l(equal_bytes(v.x, c4) * 0x00204081u, m, 4);
}

// Day number of a civil date counted the MonetDB way (days since a year 0, years >= 1 here);
// -1 for a date that does not exist.
__device__ __forceinline__ int32_t days_before_month(int32_t m) {   // non-leap year, m in 1..13
    return (367 * m - 362) / 12 - (m > 2 ? 2 : 0);
}
__device__ __forceinline__ int32_t day_number(int32_t y, int32_t m, int32_t d) {
    const bool leap = (y % 4 == 0) && (y % 100 != 0 || y % 400 == 0);
    if (y < 1 || y > 999999 || m < 1 || m > 12 || d < 1) return -1;
    const int32_t len = (m == 12 ? 31 : days_before_month(m + 1) - days_before_month(m)) + ((m == 2 && leap) ? 1 : 0);
    if (d > len) return -1;
    const int32_t p = y - 1;
    return 365 * y + (p / 4 - p / 100 + p / 400 + 1) + days_before_month(m) + ((m > 2 && leap) ? 1 : 0) + d - 1;
}

// Reads a line through a 16-byte window: one aligned 16-byte load per 16 bytes of the line
// (lanes of a warp read different lines, so every load touches a different cache line; byte
// loads would cost one L1 wavefront per byte). Offsets are 32-bit and relative to the line's
// start (a line whose first eleven fields span more than 2^31 bytes reads as malformed).
// kStaged: the line lies in a tile's stage in shared memory, which may be read to its last block.
// Else it lies in the text, whose last, partial 16-byte block is read bytewise so that no load goes
// past its end.
template <bool kStaged>
struct Cursor {
    const char* __restrict__ line;   // the line's first byte
    const uint4* __restrict__ blk;   // 16-byte blocks from the one holding line[0]
    uint32_t off;                    // line's offset inside its first block
    uint32_t p, end;                 // cursor and end of the buffer, relative to line
    uint32_t full;                   // blocks [0, full) lie wholly inside the buffer
    uint32_t wi = 0xFFFFFFFFu;       // block in the window
    uint4 win;
    __device__ __forceinline__ Cursor(const char* __restrict__ first, uint64_t rest) {
        line = first;
        const uintptr_t a = reinterpret_cast<uintptr_t>(line);
        off = (uint32_t)(a & 15u);
        blk = reinterpret_cast<const uint4*>(a - off);
        end = rest < 0x7FFFFFFFull ? (uint32_t)rest : 0x7FFFFFFFu;
        full = (uint32_t)(((uint64_t)off + end) >> 4);
        p = 0;
    }
    __device__ __forceinline__ int peek() {
        if (p >= end) return -1;
        const uint32_t a = off + p, bi = a >> 4;
        if (!kStaged && bi >= full) return (int)(unsigned char)line[p];
        if (bi != wi) {
            win = kStaged ? blk[bi] : __ldg(blk + bi);
            wi = bi;
        }
        const uint32_t o = a & 15u;
        const uint32_t w = o < 8 ? (o < 4 ? win.x : win.y) : (o < 12 ? win.z : win.w);
        return (int)((w >> (8 * (o & 3u))) & 0xFFu);
    }
    // skips to just after the next '|' of this line; false at '\n' or the end
    __device__ __forceinline__ bool skip_field() {
        for (;;) {
            const int c = peek();
            if (c < 0 || c == '\n') return false;
            ++p;
            if (c == '|') return true;
        }
    }
    __device__ __forceinline__ bool sep() {
        if (peek() != '|') return false;
        ++p;
        return true;
    }
    // "[+-]digits" (at most 18 digits)
    __device__ __forceinline__ bool integer(int64_t& v) {
        bool neg = false;
        int c = peek();
        if (c == '+' || c == '-') {
            neg = c == '-';
            ++p;
        }
        int64_t x = 0;
        uint32_t nd = 0;
        while ((c = peek()) >= '0' && c <= '9') {
            if (++nd > 18) return false;
            x = x * 10 + (c - '0');
            ++p;
        }
        if (!nd) return false;
        v = neg ? -x : x;
        return true;
    }
    // "[+-]digits[.digits]" -> 100 * int + frac
    __device__ __forceinline__ bool decimal(int64_t& v) {
        int64_t i = 0, f = 0;
        if (!integer(i)) return false;
        if (peek() == '.') {
            ++p;
            if (!integer(f)) return false;
        }
        v = 100 * i + f;
        return true;
    }
    __device__ __forceinline__ bool chr(char& c) {
        const int x = peek();
        if (x < 0 || x == '|' || x == '\n') return false;
        ++p;
        c = (char)x;
        return true;
    }
    __device__ __forceinline__ bool date(int32_t& day) {
        int64_t y, m, d;
        if (!integer(y) || peek() != '-') return false;
        ++p;
        if (!integer(m) || peek() != '-') return false;
        ++p;
        if (!integer(d)) return false;
        const int c = peek();
        if (!(c < 0 || c == '|' || c == '\n')) return false;
        if (y < 1 || y > 999999 || m < 1 || m > 12 || d < 1 || d > 31) return false;
        day = day_number((int32_t)y, (int32_t)m, (int32_t)d);
        return day >= 0;
    }
};

struct Out {
    int32_t* ship;
    int64_t *qty, *price, *disc, *tax;
    char *rf, *ls;
};

struct Row {
    int64_t qty, price, disc, tax;
    int32_t ship;
    char rf, ls;
};

// Parses the line at `first`, any form, with `rest` bytes up to the end of the text (kStaged: of the line); false (row
// zeroed) if malformed.
template <bool kStaged>
__device__ __noinline__ bool parse_line(const char* __restrict__ first, uint64_t rest, Row& r) {
    Cursor<kStaged> c(first, rest);
    r = Row{0, 0, 0, 0, 0, 0, 0};
    bool ok = c.skip_field() && c.skip_field() && c.skip_field() && c.skip_field();
    ok = ok && c.decimal(r.qty) && c.sep() && c.decimal(r.price) && c.sep() && c.decimal(r.disc) && c.sep() &&
         c.decimal(r.tax) && c.sep();
    ok = ok && c.chr(r.rf) && c.sep() && c.chr(r.ls) && c.sep() && c.date(r.ship);
    if (!ok) r = Row{0, 0, 0, 0, 0, 0, 0};
    return ok;
}

// A line of the usual form: every value but the price fits 32 bits.
struct FastRow {
    int64_t price;
    uint32_t qty, disc, tax;
    int32_t ship;
    uint32_t flags;   // return flag, line status << 8
};

// n words of the byte stream from any offset (at least -16), realigned.
template <int n>
__device__ __forceinline__ void load_bytes(const uint8_t* buf, int32_t at, uint32_t out[n]) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(buf + (at & ~3));
    const uint32_t sh = (uint32_t)(at & 3) * 8;
    uint32_t lo = w[0];
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const uint32_t hi = w[i + 1];
        out[i] = __funnelshift_r(lo, hi, sh);
        lo = hi;
    }
}
// The last n (0..4) bytes of a word of four characters; x: digits, 0 in the bytes before them.
__device__ __forceinline__ uint32_t last_bytes(int32_t n) {
    return __funnelshift_lc(0u, 0xFFFFFFFFu, n >= 4 ? 0 : 8 * (4 - n));
}
// Four digit values, the first character's in byte 0, as a number.
__device__ __forceinline__ uint32_t four_digits(uint32_t x) {
    return __dp4a((x * 10u + (x >> 8)) & 0x00FF00FFu, 0x00010064u, 0u);
}
// Any byte above 9: bit 7 of a byte of the result (other bits are noise).
__device__ __forceinline__ uint32_t not_digits(uint32_t x) { return (x + 0x76767676u) | x; }

// Days before each month of a non-leap year | its days << 16 (0: no such month).
__device__ __forceinline__ uint32_t month_entry(uint32_t m) {
    if (m < 1 || m > 12) return 0;
    return (uint32_t)days_before_month((int32_t)m) |
           (uint32_t)(m == 12 ? 31 : days_before_month((int32_t)m + 1) - days_before_month((int32_t)m)) << 16;
}

// Parses a line of the form dbgen writes, held in shared memory, a word at a time: four fields, a
// quantity of up to four digits with two decimals or none, a price of up to eight digits with two
// decimals (all of them within 49 characters), then the 25 characters "d.dd|d.dd|R|L|yyyy-mm-dd|".
// p: the line's first byte in buf, next: the next line's; months: month_entry of 0..15. False: not
// of this form (the caller parses the line with parse_line; every line accepted here gets the
// values that parse_line gives).
__device__ __forceinline__ bool parse_fast(const uint8_t* buf, uint32_t p, uint32_t next, const uint32_t* months,
                                           FastRow& r) {
    // the '|' of the 49 or more bytes from p, as bits
    const uint4* w = reinterpret_cast<const uint4*>(buf + (p & ~15u));
    const uint32_t bar = 0x7C7C7C7Cu;
    const uint32_t m0 = match16(w[0], bar) | match16(w[1], bar) << 16;
    const uint32_t m1 = match16(w[2], bar) | match16(w[3], bar) << 16;
    const uint32_t s = p & 15u;
    const uint32_t l0 = __funnelshift_r(m0, m1, s), l1 = m1 >> s;
    uint32_t a = l0 & (l0 - 1u);
    a &= a - 1u;
    a &= a - 1u;
    const uint32_t e4 = (uint32_t)__ffs((int)a) - 1u;             // fourth '|' (there is one if a != 0)
    const uint32_t n0 = __funnelshift_rc(l0, l1, e4 + 1u);
    const uint32_t b = n0 & (n0 - 1u);
    const uint32_t e5 = (uint32_t)__ffs((int)n0) - 1u, e6 = (uint32_t)__ffs((int)b) - 1u;   // from field 5 on
    const uint32_t c = p + e4 + e6 + 2u;                          // field 7
    if (!a || !b || c + 25u >= next) return false;
    // "d.dd|d.dd|R|L|yyyy-mm-dd|"; wrong: not a digit, off: not the character expected
    uint32_t A[7];
    load_bytes<7>(buf, (int32_t)c, A);
    const uint32_t xd = A[0] ^ 0x30302E30u, xt = __byte_perm(A[1], A[2], 0x4321u) ^ 0x30302E30u;
    uint32_t wrong = not_digits(xd) | not_digits(xt);
    uint32_t off = (xd | xt) & 0x0000FF00u;
    r.disc = __dp4a(xd, 0x010A0064u, 0u);
    r.tax = __dp4a(xt, 0x010A0064u, 0u);
    off |= ((A[1] ^ 0x7Cu) & 0xFFu) | ((A[2] ^ 0x7C007C00u) & 0xFF00FF00u) | ((A[3] ^ 0x7C00u) & 0xFF00u) |
           ((A[6] ^ 0x7Cu) & 0xFFu);
    r.flags = __byte_perm(A[2], A[3], 0x0042u);
    const bool blank = (r.flags & 0xFFu) == '|' || (r.flags & 0xFF00u) == ('|' << 8);   // an empty flag field
    const uint32_t xy = __byte_perm(A[3], A[4], 0x5432u) ^ 0x30303030u;
    const uint32_t xm = __byte_perm(A[4], A[5], 0x5432u) ^ 0x2D30302Du, xx = (A[5] >> 16) ^ 0x3030u;
    wrong |= not_digits(xy) | not_digits(xm) | not_digits(xx);
    off |= xm & 0xFF0000FFu;
    // the day number of yyyy = 100 yh + yl (day_number's steps, the centuries from the digits)
    const uint32_t yp = xy * 10u + (xy >> 8), yh = yp & 0xFFu, yl = (yp >> 16) & 0xFFu, year = 100u * yh + yl;
    const uint32_t month = __dp4a(xm, 0x00010A00u, 0u), day = __dp4a(xx, 0x0000010Au, 0u);
    const uint32_t me = months[month & 15u];
    const uint32_t leap = ((yl ? yl : yh) & 3u) == 0u ? 1u : 0u, cent = yh - (yl ? 0u : 1u);
    const uint32_t in_month = (me >> 16) + (month == 2u ? leap : 0u);
    const bool no_day = day - 1u >= in_month || year == 0u || month > 15u;
    r.ship = (int32_t)(365u * year + ((year - 1u) >> 2) - cent + (cent >> 2) + (me & 0xFFFFu) +
                       (month > 2u ? leap : 0u) + day);
    // price: ".dd|" ends at the '|' before field 7, up to eight digits before it
    uint32_t D[3];
    load_bytes<3>(buf, (int32_t)c - 12, D);
    const int32_t pd = (int32_t)(e6 - e5) - 4;                    // digits before the point
    const uint32_t x0 = (D[0] ^ 0x30303030u) & last_bytes(pd - 4 < 0 ? 0 : pd - 4);
    const uint32_t x1 = (D[1] ^ 0x30303030u) & last_bytes(pd < 0 ? 0 : pd);
    const uint32_t xc = D[2] ^ 0x7C30302Eu;
    wrong |= not_digits(x0) | not_digits(x1) | not_digits(xc);
    off |= xc & 0xFF0000FFu;
    r.price = (int64_t)(four_digits(x0) * 10000u + four_digits(x1)) * 100 + __dp4a(xc, 0x00010A00u, 0u);
    // quantity: with ".dd" or whole
    uint32_t Q[2];
    load_bytes<2>(buf, (int32_t)(p + e4 + e5) - 6, Q);             // the eight bytes up to its '|'
    const bool point = (Q[1] & 0xFFu) == '.' && e5 >= 4u;
    const int32_t qd = (int32_t)e5 - (point ? 3 : 0);
    const uint32_t xq = ((point ? Q[0] : __byte_perm(Q[0], Q[1], 0x6543u)) ^ 0x30303030u) & last_bytes(qd);
    const uint32_t xf = point ? (Q[1] ^ 0x7C30302Eu) : 0u;
    wrong |= not_digits(xq) | not_digits(xf);
    r.qty = four_digits(xq) * 100u + __dp4a(xf, 0x00010A00u, 0u);
    return ((wrong & 0x80808080u) | off) == 0u && (uint32_t)(pd - 1) < 8u && (uint32_t)(qd - 1) < 4u && !no_day && !blank;
}

// Published state of a tile: flag in the top two bits, value below.
constexpr uint64_t kFlagCount = 1ull << 62;    // value: newlines of the tile
constexpr uint64_t kFlagPrefix = 2ull << 62;   // value: newlines of the tiles up to this one
constexpr uint64_t kValueMask = (1ull << 62) - 1;
constexpr uint32_t kStatePad = 64;             // zeroed states before tile 0's (a look-back step's reach)

__device__ __forceinline__ void store_state(unsigned long long* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Newlines before tile k: sums the published counts of the tiles before it, two a lane and 64 a
// step, down to the nearest published prefix. A step is kept short: the control warp gets one
// warp's share of the issue slots (eight tiles a lane, 256 a step, took 0.1 ms longer in all).
// Every tile before k was taken by a running CTA (tickets), so the wait ends; it is bounded all the
// same. All lanes of one warp call it. state: 16-byte aligned, kStatePad zeroed states before it.
__device__ __forceinline__ bool look_back(const unsigned long long* state, uint64_t k, uint32_t lane, uint64_t& prefix,
                                          uint32_t* status) {
    prefix = 0;
    const unsigned long long* at = state + 2 * ((int64_t)((k - 1) / 2) - (int64_t)lane);
    bool skip = lane == 0 && (k & 1u);   // lane 0's second tile is k itself
    uint64_t t0 = 0;
    for (uint32_t spin = 0;;) {
        uint64_t a, b;
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(at) : "memory");
        if (skip) b = kFlagCount;
        const uint32_t fa = (uint32_t)(a >> 62), fb = (uint32_t)(b >> 62);
        const uint32_t pre = __ballot_sync(0xffffffffu, fb == 2 || (fb == 1 && fa == 2));
        const uint32_t known = __ballot_sync(0xffffffffu, fb == 2 || (fb == 1 && fa != 0));
        const uint32_t last = pre ? (uint32_t)__ffs((int)pre) - 1u : 31u;
        if ((~known & (0xFFFFFFFFu >> (31u - last))) == 0u) {
            const uint64_t sum = (b & kValueMask) + (fb == 2 ? 0ull : a & kValueMask);
            prefix += __reduce_add_sync(0xffffffffu, (lane < last || !pre) ? (uint32_t)sum : 0u);
            if (pre) {
                prefix += __shfl_sync(0xffffffffu, sum, (int)last);
                return true;
            }
            at -= 64;
            skip = false;
            continue;
        }
        __nanosleep(64);
        if ((++spin & 63u) == 0) {
            const uint64_t now = globaltimer();
            if (!t0) t0 = now;
            if (__any_sync(0xffffffffu, now - t0 > kWaitLimitNs)) {
                if (lane == 0) atomicOr(status, kStatusWaitTimeout);
                return false;
            }
        }
    }
}

}  // namespace tbl

// Newlines of the text, added to *total.
__global__ void __launch_bounds__(256) tbl_count_kernel(const char* __restrict__ text, uint64_t bytes,
                                                        unsigned long long* __restrict__ total) {
    using namespace tbl;
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(text) & 15u);
    const uint4* blk = reinterpret_cast<const uint4*>(text - off);
    const uint64_t end = off + bytes, pieces = (end + 15) / 16;
    uint32_t n = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pieces; i += (uint64_t)gridDim.x * blockDim.x) {
        if (16 * i >= off && 16 * i + 16 <= end) {
            const uint4 v = __ldg(blk + i);
            n += __popc(equal_bytes(v.x, 0x0A0A0A0Au)) + __popc(equal_bytes(v.y, 0x0A0A0A0Au)) +
                 __popc(equal_bytes(v.z, 0x0A0A0A0Au)) + __popc(equal_bytes(v.w, 0x0A0A0A0Au));
        } else {
            for (uint64_t x = 16 * i < off ? off : 16 * i; x < 16 * i + 16 && x < end; ++x)
                n += text[x - off] == '\n' ? 1u : 0u;
        }
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31u) == 0 && n) atomicAdd(&sum, n);
    __syncthreads();
    if (threadIdx.x == 0 && sum) atomicAdd(total, (unsigned long long)sum);
}

__global__ void __launch_bounds__(tbl::kThreads, 1) tbl_parse_kernel(const char* __restrict__ text, uint64_t bytes,
                                                                     tbl::Out o, uint64_t capacity, uint64_t tiles,
                                                                     uint64_t full_tiles,
                                                                     unsigned long long* __restrict__ state,
                                                                     TblResult* __restrict__ res) {
    using namespace tbl;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full_bar[kRing];
    __shared__ __align__(8) uint64_t prefix_bar;
    __shared__ unsigned long long tile_of[kRing];
    __shared__ uint16_t starts[kWorkers * kWarpList + 2];   // line starts in the tile, in text order, then the next one
    __shared__ uint16_t warp_starts[kWorkers][kWarpList];   // the line starts of each worker's part, in order
    __shared__ uint32_t warp_lines[2][32];       // newlines of each worker's part, by tile parity
    __shared__ uint64_t prefix_s[2];             // newlines before the tile, by tile parity
    __shared__ uint32_t months[16];
    __shared__ uint32_t counted_s;               // workers done counting << 16 | their newlines
    __shared__ uint32_t failed_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(text) & 15u);
    const uint8_t* base = reinterpret_cast<const uint8_t*>(text) - off;   // position 0
    const uint64_t end = off + bytes;
    uint32_t* const status = &res->status;

    // bytes of tile k and what is kept after it
    auto tile_bytes = [&](uint64_t k) -> uint32_t {
        const uint64_t left = end - k * kTile;
        return left < kTile + kAhead ? (uint32_t)left : kTile + kAhead;
    };
    auto start_load = [&](uint32_t s, uint64_t k) {   // one thread
        tile_of[s] = k;
        if (k >= tiles) return;
        const uint32_t n = tile_bytes(k) & ~15u, bar = smem_addr(&full_bar[s]);
        if (n) {
            mbar_arrive_expect_tx(bar, n);
            bulk_g2s(smem_addr(smem) + s * kStageBytes + kFront, base + k * kTile, n, bar, policy_evict_first());
        } else {
            mbar_arrive(bar);
        }
    };
    if (tid < 16) months[tid] = month_entry(tid);
    if (tid < 32) warp_lines[0][tid] = warp_lines[1][tid] = 0;
    if (tid == 0) {
        failed_s = counted_s = 0;
        for (uint32_t s = 0; s < kRing; ++s) mbar_init(smem_addr(&full_bar[s]), 1);
        mbar_init(smem_addr(&prefix_bar), 1);
        fence_mbar_init();
        for (uint32_t s = 1; s < kRing; ++s) tile_of[s] = ~0ull;
        start_load(0, atomicAdd(&res->ticket, 1ull));
    }
    __syncthreads();

    // Newlines of this worker's part of the tile in stage s.
    auto scan = [&](uint32_t s, uint32_t ph, uint64_t k, uint32_t parity) {
        uint8_t* const buf = smem + s * kStageBytes + kFront;
        if (!mbar_wait(smem_addr(&full_bar[s]), ph, status)) failed_s = 1;
        // a lane takes 112 consecutive bytes (an odd multiple of 16: its loads meet no bank conflict)
        const uint32_t at0 = warp * kWarpBytes + lane * kLaneBytes;
        if (k >= full_tiles) {
            // the last tiles: the bytes after the bulk copy, then zeros
            const uint32_t n_here = tile_bytes(k), from = n_here & ~15u;
            if (warp == 0)
                for (uint32_t i = kTile + lane; i < kTile + kAhead; i += 32)
                    if (i >= from) buf[i] = i < n_here ? base[k * kTile + i] : 0;
            for (uint32_t i = at0; i < at0 + kLaneBytes; ++i)
                if (i >= from) buf[i] = i < n_here ? base[k * kTile + i] : 0;
        }
        uint32_t m[kWords];   // bit i: byte at0 + i is a newline
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) {
            m[j] = match16(*reinterpret_cast<const uint4*>(buf + at0 + j * 32), 0x0A0A0A0Au);
            if (2 * j + 1 < kSubs)
                m[j] |= match16(*reinterpret_cast<const uint4*>(buf + at0 + j * 32 + 16), 0x0A0A0A0Au) << 16;
        }
        if (k == 0 && at0 < off) m[0] &= 0xFFFFFFFFu << off;   // the bytes before the text
        uint32_t c = 0;
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) c += __popc(m[j]);
        const uint32_t one = __ballot_sync(0xffffffffu, c >= 1u), two = __ballot_sync(0xffffffffu, c >= 2u);
        uint32_t run = __popc(one) + __popc(two);
        if (!__any_sync(0xffffffffu, c > 2u)) {   // lines of 56 bytes or more: at most two newlines a lane
            const uint32_t lt = (1u << lane) - 1u;
            const uint32_t at = __popc(one & lt) + __popc(two & lt);
            if (c) {
                uint32_t w = m[kWords - 1], lo = (kWords - 1) * 32;
#pragma unroll
                for (int j = (int)kWords - 2; j >= 0; --j) lo = m[j] ? j * 32u : lo, w = m[j] ? m[j] : w;
                warp_starts[warp][at] = at0 + lo + (uint32_t)__ffs((int)w);
            }
            if (c == 2u) {
                uint32_t w = m[0], hi = 32;
#pragma unroll
                for (uint32_t j = 1; j < kWords; ++j) hi = m[j] ? j * 32u + 32u : hi, w = m[j] ? m[j] : w;
                warp_starts[warp][at + 1u] = at0 + hi - (uint32_t)__clz((int)w);
            }
        } else {
            uint32_t inc = c;
#pragma unroll 1
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += u;
            }
            run = __shfl_sync(0xffffffffu, inc, 31);
            uint32_t at = inc - c;
#pragma unroll
            for (uint32_t j = 0; j < kWords; ++j)
#pragma unroll 1
                for (uint32_t x = m[j]; x; x &= x - 1u, ++at)
                    if (at < kWarpList) warp_starts[warp][at] = at0 + j * 32 + (uint32_t)__ffs((int)x);
        }
        if (lane == 0) {
            warp_lines[parity][warp] = run;
            // the last worker publishes the tile's count, long before anyone needs it
            const uint32_t c = atomicAdd(&counted_s, 1u << 16 | run) + (1u << 16 | run);
            if (c >> 16 == kWorkers) {
                counted_s = 0;
                store_state(state + k, (k == 0 ? kFlagPrefix : kFlagCount) | (c & 0xFFFFu));
            }
        }
    };
    // The line at byte `at` of the text, of any form, into row i (newlines before it); counted when
    // malformed or past the capacity. staged, size: the line in shared memory, if it lies there whole.
    auto put_any = [&](uint64_t i, uint64_t at, const uint8_t* staged = nullptr, uint32_t size = 0) {
        Row row;
        const bool good = staged ? parse_line<true>(reinterpret_cast<const char*>(staged), size, row)
                                 : parse_line<false>(text + at, bytes - at, row);
        if (i < capacity) {
            o.ship[i] = row.ship;
            o.qty[i] = row.qty;
            o.price[i] = row.price;
            o.disc[i] = row.disc;
            o.tax[i] = row.tax;
            o.rf[i] = row.rf;
            o.ls[i] = row.ls;
        }
        if (i >= capacity || !good) {
            atomicAdd(&res->malformed, 1ull);
            atomicMax(&res->first_malformed, ~(unsigned long long)at);
        }
    };

    // Tile by tile: the workers list tile i's lines (between two barriers), then find the newlines of
    // tile i + 1 and parse tile i while the control warp looks back.
    const bool control = warp == kWorkers;
    uint32_t s = 0, ph = 0, parity = 0;
    // Tickets are taken one at a time, as the CTA gets to them, so that the tiles before a tile are
    // counted earlier than it: three tickets at the start left every CTA waiting for the third tile
    // of the CTA before it.
    if (tile_of[0] < tiles) {
        if (!control) {
            scan(0, 0, tile_of[0], 0);
        } else if (lane == 0) {
            mbar_wait(smem_addr(&full_bar[0]), 0, status);
            start_load(1, atomicAdd(&res->ticket, 1ull));
        }
    }
    for (;;) {
        const uint64_t k = tile_of[s];
        if (k >= tiles) break;
        unsigned long long ticket = 0;
        if (control && lane == 0) ticket = atomicAdd(&res->ticket, 1ull);
        __syncthreads();   // newlines of tile i counted; tile i - 1 done
        if (failed_s) break;
        uint8_t* const buf = smem + s * kStageBytes + kFront;
        const uint32_t wl = warp_lines[parity][lane];
        const uint32_t newlines = __reduce_add_sync(0xffffffffu, wl);
        // the text's first line has no newline before it: it comes first in tile 0
        const uint32_t extra = k == 0 ? 1u : 0u, lines = newlines + extra;
        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? wl : 0u) + extra;
        const bool listed = !__any_sync(0xffffffffu, wl > kWarpList);   // (the same in every warp)
        if (control) {
            if (lane == 0) {
                fence_proxy_async();
                start_load(s == 0 ? kRing - 1 : s - 1, ticket);   // tile i - 1's stage
                if (extra) starts[0] = off;
            }
            if (listed) {
                // the end of the tile's last line: the first newline after the tile, if it is near
                const uint32_t x = lane < kAhead / 16
                                       ? match16(*reinterpret_cast<const uint4*>(buf + kTile + lane * 16), 0x0A0A0A0Au)
                                       : 0u;
                const uint32_t any = __ballot_sync(0xffffffffu, x != 0u);
                const uint32_t from = any ? (uint32_t)__ffs((int)any) - 1u : 0u;
                const uint32_t xf = __shfl_sync(0xffffffffu, x, (int)from);
                if (lane == 0)
                    starts[lines] = any ? kTile + from * 16 + (uint32_t)__ffs((int)xf) : kTile + kAhead + 1u;
            }
        } else if (listed) {
            const uint32_t n = warp_lines[parity][warp];
            for (uint32_t j = lane; j < n; j += 32) starts[before + j] = warp_starts[warp][j];
        }
        __syncthreads();   // tile i's lines listed
        uint32_t ns = s + 1, nph = ph;
        if (ns == kRing) ns = 0, nph ^= 1u;
        if (control) {
            uint64_t pre = 0;
            const bool ok = k == 0 || look_back(state, k, lane, pre, status);
            if (lane == 0) {
                if (ok && k) store_state(state + k, kFlagPrefix | (pre + newlines));
                if (!ok) failed_s = 1;
                prefix_s[parity] = pre;
                if (k + 1 == tiles) {
                    res->newlines = pre + newlines;
                    res->last_is_newline = buf[tile_bytes(k) - 1] == '\n' ? 1u : 0u;
                }
                mbar_arrive(smem_addr(&prefix_bar));
            }
        } else {
            bool known = false;
            auto prefix = [&]() -> uint64_t {   // the look-back's result
                if (!known && !mbar_wait(smem_addr(&prefix_bar), parity, status)) failed_s = 1;
                known = true;
                return prefix_s[parity] + 1u - extra;
            };
            if (!listed) {
                // very short lines: the worker walks its part, a byte a lane, without a list
                const uint64_t first = prefix();
                if (extra && tid == 0) put_any(0, 0);
                uint64_t i = first + before;
#pragma unroll 1
                for (uint32_t j = 0; j < kWarpBytes / 32; ++j) {
                    const uint32_t p = warp * kWarpBytes + j * 32 + lane;   // a byte a lane
                    const bool nl = buf[p] == '\n' && k * kTile + p >= off;
                    const uint32_t b = __ballot_sync(0xffffffffu, nl);
                    const uint64_t at = k * kTile + p + 1;
                    if (nl && at < end) put_any(i + __popc(b & ((1u << lane) - 1u)), at - off);
                    i += __popc(b);
                }
            }
            if (tile_of[ns] < tiles) scan(ns, nph, tile_of[ns], parity ^ 1u);
            if (listed) {
                for (uint32_t j = warp * 32 + lane; j - lane < lines; j += kWorkers * 32) {
                    FastRow row;
                    bool fast = false;
                    if (j < lines && k * kTile + starts[j] < end) fast = parse_fast(buf, starts[j], starts[j + 1], months, row);
                    const uint64_t i = prefix() + j;
                    fast &= i < capacity;
                    if (fast) {
                        o.ship[i] = row.ship;
                        o.qty[i] = row.qty;
                        o.price[i] = row.price;
                        o.disc[i] = row.disc;
                        o.tax[i] = row.tax;
                        o.rf[i] = (char)row.flags;
                        o.ls[i] = (char)(row.flags >> 8);
                    } else if (j < lines) {
                        const uint64_t at = k * kTile + starts[j];
                        const uint32_t next = starts[j + 1];
                        if (at < end) put_any(i, at - off, next <= kTile + kAhead ? buf + starts[j] : nullptr, next - starts[j]);
                    }
                }
            }
        }
        s = ns, ph = nph, parity ^= 1u;
    }
    // Never leave with copies in flight (only after a failed wait are there any).
    if (tid == 0 && failed_s)
        for (uint32_t i = 0; i < kRing; ++i) {
            if (tile_of[s] < tiles) mbar_wait(smem_addr(&full_bar[s]), ph, status);
            if (++s == kRing) s = 0, ph ^= 1u;
        }
}

cudaError_t launch_tbl_count(const char* text, uint64_t bytes, unsigned long long* total, int sm_count,
                             cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(total, 0, 8, stream);
    if (e != cudaSuccess || !bytes) return e;
    const uint64_t blocks = (bytes + 31) / 16 / 256 + 1, cap = (uint64_t)sm_count * 16;
    tbl_count_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, stream>>>(text, bytes, total);
    return cudaGetLastError();
}

static uint64_t tbl_tiles(const char* text, uint64_t bytes) {
    return ((reinterpret_cast<uintptr_t>(text) & 15u) + bytes + tbl::kTile - 1) / tbl::kTile;
}

uint64_t tbl_scratch_bytes(const char* text, uint64_t bytes) {
    static_assert(sizeof(TblResult) % 16 == 0, "states start on a 16-byte boundary");
    return sizeof(TblResult) + 8 * (tbl::kStatePad + ((tbl_tiles(text, bytes) + 1) & ~1ull));
}

cudaError_t launch_tbl_parse(const char* text, uint64_t bytes, void* scratch, int32_t* ship, int64_t* qty,
                             int64_t* price, int64_t* disc, int64_t* tax, char* rf, char* ls, uint64_t capacity,
                             int sm_count, cudaStream_t stream) {
    using namespace tbl;
    const uint64_t tiles = tbl_tiles(text, bytes);
    cudaError_t e = cudaMemsetAsync(scratch, 0, tbl_scratch_bytes(text, bytes), stream);
    if (e != cudaSuccess || !bytes) return e;
    const uint32_t dyn = kRing * kStageBytes;
    if ((e = cudaFuncSetAttribute(tbl_parse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn)) != cudaSuccess)
        return e;
    TblResult* res = static_cast<TblResult*>(scratch);
    Out o{ship, qty, price, disc, tax, rf, ls};
    const uint64_t end = (reinterpret_cast<uintptr_t>(text) & 15u) + bytes;
    const uint64_t full_tiles = end < kAhead ? 0 : (end - kAhead) / kTile;   // those with all of their kAhead bytes
    const uint64_t cap = (uint64_t)sm_count;
    tbl_parse_kernel<<<(unsigned)(tiles < cap ? tiles : cap), kThreads, dyn, stream>>>(
        text, bytes, o, capacity, tiles, full_tiles, reinterpret_cast<unsigned long long*>(res + 1) + kStatePad, res);
    return cudaGetLastError();
}

}  // namespace q1
