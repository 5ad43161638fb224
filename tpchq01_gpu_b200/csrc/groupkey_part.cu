// High-cardinality group-key aggregation for sm_100a (shared_mem_per_thread placement,
// num_groups > 4096, when the sample-based choice in groupkey_kernels.cu picks it): a radix
// partition of the passing rows by key, then shared-memory cells per partition.
//
// A shared-memory table holds at most a few thousand groups, and sending the other rows straight to
// global accumulators is bound by L2 atomic throughput (at G = 65,536 with uniform keys, 97% of the
// rows). Instead, per segment of at most 6 * 2^24 rows, with 64 partitions (key mod 64, so that
// neighbouring, for skewed keys frequent, keys spread over the partitions):
//
//   pass 1  q1_gk_partition_kernel: two CTAs per SM stream the 13 B/row tiles in like the group-key
//           kernel (cp.async.bulk, 3072 rows a tile, 12 consumer warps). A round sorts one tile: every
//           passing row in the tables' fast domain becomes an 8-byte record (price 24 bits, quantity 8 |
//           discount 4, tax 4, key 16, valid bit) whose rank in its partition comes from one shared
//           atomic; a scan of the 64 counts gives the partitions' places in a staging buffer, the
//           records are put there, and during the next round's scan the buffer goes out in runs, each
//           to the CTA's open chunk (256 records, 2 KB) of its partition in a global pool. Rows
//           outside the fast domain reduce straight into the scratch accumulators.
//   lists   q1_gk_lists_kernel: directory of chunks -> chunk list per partition (counting sort).
//   pass 2  q1_gk_partagg_kernel: the concatenated lists are split evenly over the CTAs and walked in
//           stages of 24 chunks of one partition; every thread loads eight records a stage ahead
//           and adds them to (group, discount) cells (CellTable, at most 1024 groups), flushed into the scratch accumulators whenever the partition changes.
//
// What bounds it: 29 B of traffic a row (13 read, 8 written, 8 read), 0.89 ms per 200 M rows at the copy
// bandwidth, and in both passes the shared-memory pipe (65 to 75%: scattered 8-byte stores and atomics
// whose random addresses meet four to a bank). 200 M uniform rows over 65,536 groups: 1.26 ms, 0.82 of
// it pass 1. Before: a 64-record ring per warp and partition in pass 1 and one slot of nine words per
// group in pass 2, 1.76 ms. With 128 partitions (half as long runs) 1.40 ms; three CTAs of 8 warps per
// SM in pass 1 1.53, one of 24 1.64; count and quantity in words of their own in pass 2 1.47.
//
// The arithmetic per row is the reference's (src/kernels/ht_in_global_mem.hpp:31-49), grouped
// by key; results are bit-identical to the single-pass placements.
#include <cuda_runtime.h>
#include <stdint.h>

#include "q1_common.cuh"
#include "q1_keyagg.cuh"
#include "q1_kernels.h"
#include "q1_ptx.cuh"

namespace q1 {

using namespace ptx;

namespace gp {

constexpr uint32_t kPartLog = 6, kParts = 1u << kPartLog;
constexpr uint32_t kWidth = 65536u >> kPartLog;   // groups of a partition at most
constexpr uint32_t kChunk = 256;                  // records per chunk (2 KB)
constexpr uint32_t kGrab = 128;                   // chunks a CTA reserves at a time
constexpr uint64_t kSegRows = 6ull << 24;         // rows per segment (bounds the pool)
constexpr uint32_t kP1Ctas = 2;                   // CTAs of pass 1 per SM
constexpr uint32_t kMaxGrid = kP1Ctas * 152;      // CTAs of pass 1 (bounds the pool's slack)
constexpr uint32_t kNone = 0xFFFFFFFFu;

// pass 1
constexpr uint32_t kP1Warps = 12, kP1Consumers = kP1Warps * 32;
constexpr uint32_t kP1Rows = 256 * kP1Warps;      // a tile: two quads a consumer thread
constexpr uint32_t kP1Stages = 2;
using P1Tile = ka::TileLayout<kP1Rows>;
constexpr uint32_t kP1Smem = kP1Stages * P1Tile::kStageBytes + kP1Rows * 8;
static_assert(kP1Ctas * (kP1Smem + 6144) <= 227 * 1024, "CTAs per SM");
static_assert(kP1Rows == kP1Consumers * 8, "two quads per thread");
static_assert(kParts % 32 == 0 && kParts <= kP1Consumers, "a thread per partition, whole warps");
// pass 2
constexpr uint32_t kP2Warps = 24, kP2Threads = kP2Warps * 32;
constexpr uint32_t kP2Ctas = 1;                   // CTAs of pass 2 per SM
constexpr uint32_t kQuads = 2;                    // times four records per thread and stage
constexpr uint32_t kStageChunks = kQuads * kP2Threads * 4 / kChunk;

// Most chunks the CTAs of a segment reserve. A partition's list takes its records' chunks and, in every CTA,
// an open one. Of every grab but a CTA's last, fewer than kRun chunks stay unused (a partition's chunks of one
// round stay together), and all of the last may.
constexpr uint32_t kRun = kP1Rows / kChunk;       // chunks one partition takes in a round at most
static_assert(kP1Rows % kChunk == 0 && kParts + kRun <= kGrab, "a grab holds any round's chunks");
__host__ __device__ constexpr uint64_t max_chunks(uint64_t rows, uint64_t ctas) {
    const uint64_t used = rows / kChunk + ctas * kParts, of_grab = kGrab - (kRun - 1);
    return (used * kGrab + of_grab - 1) / of_grab + ctas * kGrab;
}
constexpr uint64_t kPoolChunks = max_chunks(kSegRows, kMaxGrid);
static_assert(kPoolChunks < (1u << 20), "a chunk id takes 20 bits of a list entry");

struct Ctl {
    uint32_t pool_next;              // chunks reserved
    uint32_t part_chunks[kParts];    // chunks written per partition
    uint32_t list_cursor[kParts];    // list entries placed per partition
};

__host__ __device__ constexpr uint64_t align256(uint64_t x) { return (x + 255) & ~255ull; }

// Workspace after the accumulators: 256 bytes (the mode word at 192) | ctl | dir (2 B a chunk:
// partition + 1 << 8 | records - 1; 0: unused) | lists (4 B: chunk | records - 1 << 20) | pool.
constexpr uint64_t kOffCtl = 256;
constexpr uint64_t kOffDir = kOffCtl + align256(sizeof(Ctl));
constexpr uint64_t kOffLists = kOffDir + align256(2 * kPoolChunks);
constexpr uint64_t kOffPool = kOffLists + align256(4 * kPoolChunks);
constexpr uint64_t kWorkspaceBytes = kOffPool + kPoolChunks * kChunk * 8;

__device__ __forceinline__ void bar_sync(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// ---------------------------------------------------------------------------------------------
// Pass 2's table: (group, discount) cells like ka::CubeTable, with the quantity in the cell too (a
// partition of skewed keys can be almost all one group: its rows then spread over eleven words).
// ---------------------------------------------------------------------------------------------
struct CellTable {
    static constexpr uint32_t kCells = kWidth * ka::kCubeDisc;
    static constexpr uint32_t kGroupWords = 3 + ka::kPackedWords;
    static constexpr uint32_t kWords = 3 * kCells + kGroupWords * kWidth;
    uint32_t* w;   // [3][cells]: packed count and quantity (ka::packed_row), price, tax * price (low words); then
                   // per group, word-major: wraps of its cells' price words, sum (100 - d) over them and over
                   // those of tax * price, and the packed words' carries
    __device__ __forceinline__ void zero(uint32_t tid, uint32_t n) {
        for (uint32_t i = tid; i < kWords; i += n) w[i] = 0;
    }
    // Rows r with bit r of m set, in the fast domain. All lanes of the warp call it.
    __device__ __forceinline__ void add_quad(uint32_t m, const uint32_t g[4], const uint32_t q[4], const uint32_t d[4],
                                             const uint32_t t[4], const uint32_t p[4]) {
        uint32_t vt[4], oq[4], op[4], ot[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t c = g[r] * ka::kCubeDisc + d[r];
            vt[r] = t[r] * p[r];
            oq[r] = op[r] = ot[r] = 0;
            if ((m >> r) & 1u) {
                oq[r] = atomicAdd(w + c, ka::packed_row(q[r]));
                op[r] = atomicAdd(w + kCells + c, p[r]);
                ot[r] = atomicAdd(w + 2 * kCells + c, vt[r]);
            }
        }
        bool wrap = false;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            wrap |= (op[r] > ~p[r]) | (ot[r] > ~vt[r]) | ka::packed_carries(oq[r], q[r]);
        if (__any_sync(0xffffffffu, wrap)) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                uint32_t* gw = w + 3 * kCells + g[r];
                const uint32_t a = 100u - d[r];
                if (op[r] > ~p[r]) {
                    atomicAdd(gw, 1u);
                    atomicAdd(gw + kWidth, a);
                }
                if (ot[r] > ~vt[r]) atomicAdd(gw + 2 * kWidth, a);
                ka::packed_carry(gw + 3 * kWidth, kWidth, oq[r], q[r], d[r]);
            }
        }
    }
    // Groups of partition `part` -> scratch, and zero again; the caller synchronises around it.
    __device__ __forceinline__ void flush(unsigned long long* acc, uint32_t part, uint32_t tid, uint32_t n) {
        for (uint32_t g = tid; g < kWidth; g += n) {
            uint32_t* gw = w + 3 * kCells + g;
            const uint64_t pw = gw[0], aw = gw[kWidth], tw = gw[2 * kWidth];
            gw[0] = gw[kWidth] = gw[2 * kWidth] = 0;
            ka::PackedSums s;
            s.start(gw + 3 * kWidth, kWidth);
            uint64_t P = pw << 32;
            unsigned __int128 DP = (unsigned __int128)aw << 32, CH = (unsigned __int128)(100u * aw + tw) << 32;
#pragma unroll
            for (uint32_t d = 0; d < ka::kCubeDisc; ++d) {
                const uint32_t c = g * ka::kCubeDisc + d;
                const uint32_t Pd = w[kCells + c], Td = w[2 * kCells + c];
                s.add(w[c], d);
                P += Pd;
                DP += (uint64_t)(100u - d) * Pd;
                CH += (unsigned __int128)(100u - d) * ((uint64_t)Pd * 100u + Td);
                w[c] = w[kCells + c] = w[2 * kCells + c] = 0;
            }
            if (s.cnt)
                ka::scratch_add(acc, g << kPartLog | part, s.cnt, s.q, s.disc, P, (uint64_t)DP & 0xFFFFFFFFull,
                                (uint64_t)(DP >> 32), (uint64_t)CH & 0xFFFFFFFFull, (uint64_t)(CH >> 32));
        }
    }
};
constexpr uint32_t kP2Smem = CellTable::kWords * 4;
static_assert(kP2Ctas * (kP2Smem + 4096) <= 227 * 1024, "CTAs per SM");

}  // namespace gp

struct PartParams {
    const uint8_t* col[6];          // ship, qty, disc, tax, price, key (16-byte aligned)
    uint64_t rows;                  // rows of this segment (<= kSegRows)
    int32_t cutoff;                 // cutoff_day - 727563
    uint32_t num_groups;
    unsigned long long* acc;        // scratch accumulators: num_groups x 8 u64
    uint32_t* status;
    const uint32_t* mode;           // when set, the kernels run only if *mode == kModePartitioned
    gp::Ctl* ctl;
    uint32_t max_chunks;            // of the segment: directory entries cleared
    uint16_t* dir;
    uint32_t* lists;
    uint2* pool;
};

// ---------------------------------------------------------------------------------------------
// Pass 1: partition
// ---------------------------------------------------------------------------------------------

// A quad's records: fast-domain passing rows (lo = price | quantity << 24, hi = discount | tax << 4 |
// key << 8 | valid bit; hi 0: none). Other passing rows with key < num_groups reduce into the
// scratch; passing rows with key >= num_groups set `bad`. All lanes call it.
__device__ __forceinline__ void quad_records(const ka::KeyQuad& x, const PartParams& prm, uint2 rec[4], uint32_t& bad) {
    const uint32_t G = prm.num_groups;
    // rows outside the fast domain: bit 7 of byte r set when d > 10, t > 8 or p >= 2^24
    const uint32_t top = __byte_perm(__byte_perm(x.p[0], x.p[1], 0x0073u), __byte_perm(x.p[2], x.p[3], 0x0073u),
                                     0x5410u);
    const uint32_t outside = (((top & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | top | ((x.D & 0x7F7F7F7Fu) + 0x75757575u) |
                              x.D | ((x.X & 0x7F7F7F7Fu) + 0x77777777u) | x.X) &
                             0x80808080u;
    const uint32_t ob = (outside >> 7) * 0xFFu;
    const uint32_t DT = (x.D & ~ob) | ((x.X & ~ob) << 4);   // bytes r: d | t << 4 (in-domain rows)
    uint32_t fast, slow;   // byte r = 0xFF: row r becomes a record; bit r: row r to the scratch
    if (max(max(x.k[0], x.k[1]), max(x.k[2], x.k[3])) < G) {
        // every key of the quad in range: byte-parallel masks, the slow rows gathered to bits
        // 0..3 by one multiply (byte r's bit 0 lands on bit 24 + r)
        fast = x.PM & ~ob;
        slow = (((x.PM & ob) & 0x01010101u) * 0x01020408u) >> 24;
    } else {
        fast = slow = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t pass = (x.PM >> (8 * r)) & 1u;
            const uint32_t in = pass & (x.k[r] < G ? 1u : 0u);
            bad |= pass & (in ^ 1u);
            const uint32_t f = in & (((outside >> (8 * r + 7)) & 1u) ^ 1u);
            slow |= (in & (f ^ 1u)) << r;
            fast |= (f * 0xFFu) << (8 * r);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        rec[r].x = __byte_perm(x.p[r], x.Q, 0x0210u | ((4u + (uint32_t)r) << 12));   // p | q << 24
        rec[r].y = (fast >> (8 * r)) & 1u ? ((DT >> (8 * r)) & 0xFFu) | x.k[r] << 8 | 0x80000000u : 0u;
    }
    if (__any_sync(0xffffffffu, slow)) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if ((slow >> r) & 1u)
                ka::scratch_row(prm.acc, x.k[r], (x.Q >> (8 * r)) & 0xFFu, (x.D >> (8 * r)) & 0xFFu,
                                (x.X >> (8 * r)) & 0xFFu, x.p[r]);
    }
}

__device__ __forceinline__ uint32_t part_of(uint32_t hi) { return (hi >> 8) & (gp::kParts - 1u); }

__global__ void __launch_bounds__((gp::kP1Warps + 1) * 32, gp::kP1Ctas)
    q1_gk_partition_kernel(const __grid_constant__ PartParams prm) {
    using namespace gp;
    constexpr uint32_t S = kP1Stages, R = kP1Rows, kStage = P1Tile::kStageBytes;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full_bar[S];
    __shared__ __align__(8) uint64_t empty_bar[S];
    __shared__ uint32_t hist[kParts];                    // records of the round per partition
    // per partition: place in the staging buffer, and, by round parity, where its records go: those
    // before split at (index + head) of the pool, the others (a new chunk's) at (index + rest)
    __shared__ uint32_t place[kParts];
    __shared__ __align__(8) uint2 dest[2][kParts];       // split, head
    __shared__ uint32_t dest_rest[2][kParts];
    __shared__ uint32_t total_s[2];                      // records of the round, by parity
    __shared__ uint32_t warp_sum[kParts / 32];
    __shared__ uint32_t grab_s, fit_s, failed_s;
    if (prm.mode && *prm.mode != kModePartitioned) return;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint64_t num_tiles = prm.rows / R;
    const uint32_t ring = smem_addr(smem);
    uint2* const stage = reinterpret_cast<uint2*>(smem + S * kStage);

    if (tid == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(smem_addr(&full_bar[s]), 1);
            mbar_init(smem_addr(&empty_bar[s]), kP1Warps);
        }
        fence_mbar_init();
        failed_s = fit_s = 0;
        total_s[0] = total_s[1] = 0;
    }
    for (uint32_t i = tid; i < kParts; i += blockDim.x) hist[i] = 0;
    __syncthreads();

    if (warp == kP1Warps) {
        if (lane == 0) {
            const uint64_t pol = policy_evict_first();
            uint32_t k = 0;
            for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x, ++k) {
                const uint32_t s = k % S;
                if (!mbar_wait(smem_addr(&empty_bar[s]), ((k / S) & 1u) ^ 1u, prm.status)) break;
                const uint32_t fb = smem_addr(&full_bar[s]);
                mbar_arrive_expect_tx(fb, kStage);
#pragma unroll
                for (int c = 0; c < 6; ++c)
                    bulk_g2s(ring + s * kStage + P1Tile::col_off(c), prm.col[c] + t * (uint64_t)P1Tile::col_bytes(c),
                             P1Tile::col_bytes(c), fb, pol);
            }
            for (uint32_t i = (k > S ? k - S : 0u); i < k; ++i) mbar_wait(smem_addr(&full_bar[i % S]), (i / S) & 1u, prm.status);
        }
        return;
    }

    // Thread p < kParts: partition p's open chunk (next and end record of the pool) and its chunks; the
    // chunks reserved by the CTA, [free, free_end), are the same in all of those threads.
    uint32_t next = 0, end = 0, chunks = 0, free = 0, free_end = 0;
    // Scan of the round's counts: places in the staging buffer and chunks for what the open ones
    // cannot take (the first warps; named barrier 1).
    auto scan_counts = [&](uint32_t parity) {
        const uint32_t p = tid, n = hist[p];
        hist[p] = 0;
        const uint32_t room = end - next, head = min(n, room), rest = n - head;
        const uint32_t want = (rest + kChunk - 1) / kChunk;
        const uint32_t v = n | want << 16;   // both sums stay below 2^16
        uint32_t inc = v;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += u;
        }
        if (lane == 31) warp_sum[warp] = inc;
        bar_sync(1, kParts);
        uint32_t before = inc - v, all = 0;
#pragma unroll
        for (uint32_t i = 0; i < kParts / 32; ++i) {
            const uint32_t t = warp_sum[i];
            before += i < warp ? t : 0u;
            all += t;
        }
        const uint32_t at = before & 0xFFFFu, c0 = before >> 16, need = all >> 16;
        uint32_t first = free + c0;          // the partition's first new chunk
        if (need > free_end - free) {        // (the same in all of those threads)
            // the partitions whose chunks fit take the rest of the grab, the others a new one
            const bool fits = c0 + want <= free_end - free;
            if (want && fits) atomicMax(&fit_s, c0 + want);
            bar_sync(1, kParts);
            const uint32_t fit = fit_s, more = max(need - fit, kGrab);
            if (p == 0) grab_s = atomicAdd(&prm.ctl->pool_next, more);
            bar_sync(1, kParts);
            if (p == 0) fit_s = 0;
            if (!fits) first = grab_s + c0 - fit;
            free = grab_s + need - fit;
            free_end = grab_s + more;
        } else {
            free += need;
        }
        if (first + want > prm.max_chunks) {   // (gp::max_chunks is such that this cannot be)
            if (prm.status) atomicOr(prm.status, kStatusInternal);
            first = 0;
        }
        place[p] = at;
        dest[parity][p] = make_uint2(at + head, next - at);
        dest_rest[parity][p] = first * kChunk - at - head;
        if (want) {
            for (uint32_t c = first; c < first + want; ++c) prm.dir[c] = (uint16_t)((p + 1) << 8 | (kChunk - 1));
            next = first * kChunk + rest;
            end = (first + want) * kChunk;
            chunks += want;
        } else {
            next += n;
        }
        if (p == 0) total_s[parity] = all & 0xFFFFu;
        bar_sync(1, kParts);   // warp_sum is free again
    };
    // The round's staged records to the pool, in runs (consecutive records of a partition); four at a
    // time, so that their shared-memory loads overlap.
    auto write_out = [&](uint32_t parity) {
        const uint32_t n = total_s[parity];
        for (uint32_t i0 = tid; i0 < n; i0 += 4 * kP1Consumers) {
            uint2 r[4], d[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) r[j] = i0 + j * kP1Consumers < n ? stage[i0 + j * kP1Consumers] : make_uint2(0, 0);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) d[j] = dest[parity][part_of(r[j].y)];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t i = i0 + j * kP1Consumers;
                uint32_t at = d[j].y;
                if (i >= d[j].x) at = dest_rest[parity][part_of(r[j].y)];
                if (i < n) prm.pool[i + at] = r[j];
            }
        }
    };

    uint32_t bad = 0, k = 0, parity = 0;
    bool staged = false;   // a round's records wait in the staging buffer
    // One round: the thread's two quads, quad(0) and quad(1), then release() once they are read; false
    // after an expired wait.
    auto round = [&](auto&& quad, auto&& release) -> bool {
        uint2 rec[8];
        uint32_t rank[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) quad_records(quad(h), prm, rec + 4 * h, bad);
        release();
#pragma unroll
        for (int r = 0; r < 8; ++r) rank[r] = rec[r].y ? atomicAdd(&hist[part_of(rec[r].y)], 1u) : 0u;
        bar_sync(2, kP1Consumers);   // counted; the round before staged
        if (failed_s) return false;
        if (warp < kParts / 32) scan_counts(parity);
        if (staged) write_out(parity ^ 1u);
        bar_sync(2, kP1Consumers);   // places known, the staging buffer empty
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (rec[r].y) stage[place[part_of(rec[r].y)] + rank[r]] = rec[r];
        staged = true;
        parity ^= 1u;
        return true;
    };
    for (uint64_t t = blockIdx.x; t < num_tiles; t += gridDim.x, ++k) {
        const uint32_t s = k % S;
        if (!mbar_wait(smem_addr(&full_bar[s]), (k / S) & 1u, prm.status)) failed_s = 1;
        const uint32_t base = ring + s * kStage;
        const bool ok = round([&](int h) { return ka::load_quad<R>(base, tid + h * kP1Consumers, prm.cutoff, bad); },
                              [&]() {
                                  __syncwarp();
                                  if (lane == 0) mbar_arrive(smem_addr(&empty_bar[s]));
                              });
        if (!ok) return;
    }
    // the rows after the last full tile, by one CTA straight from global memory
    if (blockIdx.x == (uint32_t)(num_tiles % gridDim.x) && num_tiles * R < prm.rows) {
        round(
            [&](int h) {
                ka::KeyQuad x = ka::empty_quad();
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint64_t i = num_tiles * R + (uint32_t)(4 * h + r) * kP1Consumers + tid;
                    if (i < prm.rows) {
                        const ka::KeyQuad y = ka::load_row(prm.col, i, prm.cutoff, bad);
                        x.PM |= y.PM << (8 * r), x.Q |= y.Q << (8 * r), x.D |= y.D << (8 * r), x.X |= y.X << (8 * r);
                        x.p[r] = y.p[0], x.k[r] = y.k[0];
                    }
                }
                return x;
            },
            []() {});
    }
    bar_sync(2, kP1Consumers);
    if (staged) write_out(parity ^ 1u);
    if (tid < kParts) {
        // the records of the open chunk
        if (next < end && (next & (kChunk - 1)) && next / kChunk < prm.max_chunks)
            prm.dir[next / kChunk] = (uint16_t)((tid + 1) << 8 | ((next & (kChunk - 1)) - 1));
        if (chunks) atomicAdd(&prm.ctl->part_chunks[tid], chunks);
    }
    if (bad && prm.status) atomicOr(prm.status, kStatusDomain);
}

// ---------------------------------------------------------------------------------------------
// Lists: directory -> per-partition chunk lists, laid out partition after partition
// ---------------------------------------------------------------------------------------------
// off[p]: list entries of the partitions before p; off[kParts]: all. Threads below kParts call it.
__device__ __forceinline__ void list_offsets(const PartParams& prm, uint32_t tid, uint32_t* off, uint32_t* part_sum) {
    using namespace gp;
    const uint32_t lane = tid & 31u, n = prm.ctl->part_chunks[tid];
    uint32_t inc = n;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += u;
    }
    if (lane == 31) part_sum[tid >> 5] = inc;
    bar_sync(1, kParts);
    for (uint32_t i = 0; i < (tid >> 5); ++i) inc += part_sum[i];
    off[tid + 1] = inc;
    if (tid == 0) off[0] = 0;
}

__global__ void __launch_bounds__(256) q1_gk_lists_kernel(const __grid_constant__ PartParams prm) {
    using namespace gp;
    constexpr uint32_t kPer = 8, kTile = 256 * kPer;
    __shared__ uint32_t hist[kParts], base[kParts], off[kParts + 1], part_sum[kParts / 32];
    if (prm.mode && *prm.mode != kModePartitioned) return;
    const uint32_t tid = threadIdx.x;
    const uint32_t n = min(prm.ctl->pool_next, prm.max_chunks);
    if (tid < kParts) list_offsets(prm, tid, off, part_sum);
    for (uint64_t t0 = (uint64_t)blockIdx.x * kTile; t0 < n; t0 += (uint64_t)gridDim.x * kTile) {
        if (tid < kParts) hist[tid] = 0;
        __syncthreads();
        uint32_t e[kPer], rk[kPer];
#pragma unroll
        for (uint32_t j = 0; j < kPer; ++j) {
            const uint64_t i = t0 + j * 256 + tid;
            e[j] = i < n ? prm.dir[i] : 0u;
            rk[j] = e[j] ? atomicAdd(&hist[(e[j] >> 8) - 1], 1u) : 0u;
        }
        __syncthreads();
        if (tid < kParts && hist[tid]) base[tid] = off[tid] + atomicAdd(&prm.ctl->list_cursor[tid], hist[tid]);
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < kPer; ++j) {
            if (e[j]) {
                const uint32_t at = base[(e[j] >> 8) - 1] + rk[j];
                if (at < prm.max_chunks) prm.lists[at] = (uint32_t)(t0 + j * 256 + tid) | (e[j] & 0xFFu) << 20;
                else if (prm.status) atomicOr(prm.status, kStatusInternal);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Pass 2: per-partition cells
// ---------------------------------------------------------------------------------------------

// 16 bytes of a chunk the first pass wrote (read once).
__device__ __forceinline__ uint4 ldg_nc_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// One stage of a CTA's walk: its partition (kNone: past the end), first list entry and chunks.
struct P2Stage {
    uint32_t p, first, n;
};

__global__ void __launch_bounds__(gp::kP2Threads, gp::kP2Ctas) q1_gk_partagg_kernel(const __grid_constant__ PartParams prm) {
    using namespace gp;
    constexpr uint32_t T = kP2Threads;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t off_s[kParts + 1], part_sum[kParts / 32];
    if (prm.mode && *prm.mode != kModePartitioned) return;

    const uint32_t tid = threadIdx.x;
    CellTable cells{reinterpret_cast<uint32_t*>(smem)};
    if (tid < kParts) list_offsets(prm, tid, off_s, part_sum);
    cells.zero(tid, T);
    __syncthreads();

    // The CTA's share [pos, hi) of the concatenated lists, in stages of at most kStageChunks chunks that
    // never cross a partition boundary.
    const uint64_t entries = off_s[kParts];
    uint32_t pos = (uint32_t)(entries * blockIdx.x / gridDim.x), part = 0;
    const uint32_t hi = (uint32_t)(entries * (blockIdx.x + 1) / gridDim.x);
    auto next = [&]() -> P2Stage {
        if (pos >= hi) return P2Stage{kNone, 0, 0};
        while (part + 1 < kParts && off_s[part + 1] <= pos) ++part;
        P2Stage st{part, pos, min(kStageChunks, min(hi, off_s[part + 1]) - pos)};
        pos += st.n;
        return st;
    };
    // The thread's list entries in stage st (kNone: none), and its records of those chunks: two pairs of
    // each, 64 records apart, so that a warp's 16-byte loads are consecutive.
    const uint32_t my_chunk = tid / (kChunk / 4), my_pair = (tid / 32) % 2 * 128 + tid % 32 * 2;
    auto entry_of = [&](const P2Stage& st, uint32_t h) -> uint32_t {
        const uint32_t i = my_chunk + h * (kStageChunks / kQuads);
        return i < st.n ? prm.lists[st.first + i] : kNone;
    };
    auto load = [&](uint32_t e, uint4& a, uint4& b) {
        a = b = make_uint4(0, 0, 0, 0);
        // pairs past the chunk's records are not read (they were never written)
        if (e != kNone) {
            const uint2* src = prm.pool + (uint64_t)(e & 0xFFFFFu) * kChunk + my_pair;
            if (my_pair <= (e >> 20)) a = ldg_nc_v4(src);
            if (my_pair + 64 <= (e >> 20)) b = ldg_nc_v4(src + 64);
        }
    };
    // records of the pairs below the chunk's count: bits 0..3
    auto mask_of = [&](uint32_t e) -> uint32_t {
        if (e >> 20 == kChunk - 1) return 15u;
        if (e == kNone) return 0u;
        const uint32_t last = e >> 20;
        return (my_pair <= last ? 1u : 0u) | (my_pair + 1 <= last ? 2u : 0u) | (my_pair + 64 <= last ? 4u : 0u) |
               (my_pair + 65 <= last ? 8u : 0u);
    };

    // software pipeline: records of the next stage and list entries of the one after
    P2Stage s0 = next(), s1 = next(), s2 = next();
    uint32_t e0[kQuads], e1[kQuads], e2[kQuads];
    uint4 a0[kQuads], b0[kQuads], a1[kQuads], b1[kQuads];
#pragma unroll
    for (uint32_t h = 0; h < kQuads; ++h) {
        e0[h] = entry_of(s0, h);
        e1[h] = entry_of(s1, h);
        load(e0[h], a0[h], b0[h]);
    }
    uint32_t cur = kNone;
    uint64_t rows_since = 0;
    while (s0.p != kNone) {
#pragma unroll
        for (uint32_t h = 0; h < kQuads; ++h) {
            load(e1[h], a1[h], b1[h]);
            e2[h] = entry_of(s2, h);
        }
        if (s0.p != cur || rows_since + s0.n * kChunk > ka::kTableFlushRows) {
            if (cur != kNone) {
                __syncthreads();
                cells.flush(prm.acc, cur, tid, T);
                __syncthreads();
            }
            cur = s0.p;
            rows_since = 0;
        }
        rows_since += s0.n * kChunk;
#pragma unroll
        for (uint32_t h = 0; h < kQuads; ++h) {
            uint32_t g[4], q[4], d[4], t[4], pr[4];
            const uint32_t lo[4] = {a0[h].x, a0[h].z, b0[h].x, b0[h].z}, hw[4] = {a0[h].y, a0[h].w, b0[h].y, b0[h].w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                pr[r] = lo[r] & 0xFFFFFFu;
                q[r] = lo[r] >> 24;
                d[r] = hw[r] & 0xFu;
                t[r] = (hw[r] >> 4) & 0xFu;
                g[r] = (hw[r] >> (8 + kPartLog)) & (kWidth - 1);
            }
            cells.add_quad(mask_of(e0[h]), g, q, d, t, pr);
        }
        s0 = s1, s1 = s2, s2 = next();
#pragma unroll
        for (uint32_t h = 0; h < kQuads; ++h) {
            e0[h] = e1[h], e1[h] = e2[h];
            a0[h] = a1[h], b0[h] = b1[h];
        }
    }
    __syncthreads();
    if (cur != kNone) cells.flush(prm.acc, cur, tid, T);
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
uint64_t groupkey_part_workspace_bytes() { return gp::kWorkspaceBytes; }

// more groups than the single pass's slot table holds
uint32_t groupkey_part_min_groups() { return 4097; }

uint64_t groupkey_part_mode_offset() { return 192; }

uint64_t groupkey_part_max_chunks(uint64_t rows, uint32_t ctas) { return gp::max_chunks(rows, ctas); }

cudaError_t launch_groupkey_part(const uint8_t* const cols[6], uint64_t rows, int32_t cutoff_rel,
                                 uint32_t num_groups, unsigned long long* acc, uint8_t* workspace,
                                 const uint32_t* mode, uint32_t* status, int sm_count, int max_blocks,
                                 cudaStream_t stream) {
    using namespace gp;
    if (num_groups > kWidth * kParts) return cudaErrorInvalidValue;
    cudaError_t e =
        cudaFuncSetAttribute(q1_gk_partition_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP1Smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(q1_gk_partagg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kP2Smem);
    if (e != cudaSuccess) return e;
    auto grid_of = [&](uint32_t ctas) {
        const uint32_t most = max_blocks > 0 ? (uint32_t)max_blocks : ~0u;
        return min(min(ctas * (uint32_t)sm_count, kMaxGrid), most);
    };
    const uint32_t grid = grid_of(kP1Ctas), grid2 = grid_of(kP2Ctas);
    PartParams prm{};
    prm.cutoff = cutoff_rel;
    prm.num_groups = num_groups;
    prm.acc = acc;
    prm.status = status;
    prm.mode = mode;
    prm.ctl = reinterpret_cast<Ctl*>(workspace + kOffCtl);
    prm.dir = reinterpret_cast<uint16_t*>(workspace + kOffDir);
    prm.lists = reinterpret_cast<uint32_t*>(workspace + kOffLists);
    prm.pool = reinterpret_cast<uint2*>(workspace + kOffPool);
    const uint32_t bytes[6] = {2, 1, 1, 1, 4, 4};
    for (uint64_t off = 0; off < rows; off += kSegRows) {
        const uint64_t n = rows - off < kSegRows ? rows - off : kSegRows;
        for (int c = 0; c < 6; ++c) prm.col[c] = cols[c] + off * bytes[c];
        prm.rows = n;
        const uint64_t tiles = n / kP1Rows;
        const uint32_t g1 = (uint32_t)(tiles == 0 ? 1 : (tiles < grid ? tiles : grid));
        prm.max_chunks = (uint32_t)max_chunks(n, g1);
        e = cudaMemsetAsync(prm.ctl, 0, kOffDir - kOffCtl + 2ull * prm.max_chunks, stream);
        if (e != cudaSuccess) return e;
        q1_gk_partition_kernel<<<g1, (kP1Warps + 1) * 32, kP1Smem, stream>>>(prm);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        uint64_t gl = (prm.max_chunks + 2047) / 2048;
        if (gl > 4ull * (uint64_t)sm_count) gl = 4ull * (uint64_t)sm_count;
        q1_gk_lists_kernel<<<(unsigned)gl, 256, 0, stream>>>(prm);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        q1_gk_partagg_kernel<<<grid2, kP2Threads, kP2Smem, stream>>>(prm);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace q1
