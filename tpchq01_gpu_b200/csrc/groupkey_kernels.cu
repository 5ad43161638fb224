// Group-key aggregation for sm_100a: the Q1 predicate and aggregates, grouped by a synthetic
// uint32 key (up to 65,536 groups) instead of the (returnflag, linestatus) pair.
//
// The per-row arithmetic is the reference's (src/kernels/ht_in_global_mem.hpp:31-49); only the
// group index changes: group = key[i] (< num_groups) instead of (rf << 1) + ls.
//
// Input tiles (1024 to 3840 rows by placement and table): ship u16 | qty u8 | disc u8 | tax u8 |
// price u32 | key u32 (13 B/row), streamed with one cp.async.bulk per column into a shared-memory
// ring like the scan kernel's (scan_kernels.cu); the consumer warps decode 4 rows per step
// (q1_keyagg.cuh).
//
// Placements:
//   in_registers_per_thread  num_groups <= 8: per-thread dp4a byte planes (PlaneRegs<4|8>)
//   shared_mem_per_thread    num_groups <= 64: shared (group, discount, tax) cells
//                            (Cube3Table); <= 1024: shared (group, discount) cells (CubeTable);
//                            <= 4096: shared per-group slots (SlotTable), both in three teams over
//                            1024-row tiles where three stages of 3072 rows do not fit beside the
//                            table; or, above 4096, this kernel with keys < 4096 in slots and
//                            larger keys reduced straight into the global
//                            accumulators, or the two-pass partitioned path of
//                            groupkey_part.cu; above 4096 groups, and above about 3100 on a large
//                            table, the path is chosen on the device from a sample of the rows
//                            (q1_groupkey_choose), which may be the global placement's, when few
//                            rows pass over spread keys
//   global                   every passing row reduces into the global accumulators
//
// Accumulators live in scratch memory (per launch, zeroed first): per group 8 x u64 (see
// q1_keyagg.cuh); a finalize kernel folds them into the caller's int128 table [group][6] with
// 128-bit atomics (so, like the reference kernels, results accumulate into a caller-zeroed
// buffer). Launches are capped at 2^31 rows so every u64 scratch sum stays exact. The register
// placement needs neither: its warps leave records in shared memory and each CTA adds its sums to the
// caller's table, one 128-bit atomic per (group, aggregate). (Every warp reducing into the scratch
// made 1,184 same-address atomics per word: 4 groups, 1.0 M rows with the zeroed output 35 us, 8 groups
// 47 us.)
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdlib>
#include <cstring>

#include "q1_common.cuh"
#include "q1_keyagg.cuh"
#include "q1_kernels.h"
#include "q1_ptx.cuh"

namespace q1 {

using namespace ptx;

namespace gk {

constexpr uint32_t kMaxStages = 10;   // ring stages
constexpr uint32_t kWideSlots = 4096; // slot-table keys of the single-pass kernel
constexpr uint32_t kMaxDynSmem = 227 * 1024;
// Consumer warps. Register planes: 8, or 15 for four groups' planes on a large table (kWide: their 115
// registers a thread fit the 128 that 16 warps leave, and four warps per scheduler hide more of the
// planes' issue latency: 100 M rows 206 us with 12, 188 with 15). Eight groups' planes take 168 registers,
// which 11 consumer warps would leave too (100 M rows 322 -> 316 us, but 6 M 27.4 -> 28.8). Global
// placement: 16. Shared tables: 24, whose atomics need many warps in flight to hide their latency (64
// groups, 100 M rows: 237 us with 16, 199 with 24).
template <int P, int NG, bool kWide>
__host__ __device__ constexpr uint32_t consumer_warps() {
    return P == kPlaceInRegistersPerThread ? (kWide ? 15u : 8u)
                                           : (P == kPlaceSharedMemPerThread ? 24u : 16u);
}
// Rows per tile: two quads of a tile for every consumer thread of the register planes (at most 8
// rows, which their flush cadence assumes), one for the others. The shared tables' consumers may
// form teams that take the tiles in turn, each with a producer warp of its own (one producer feeding
// three teams' small tiles was the bound: 283 us): the tiles are smaller, so that the ring beside a large
// table still holds several.
template <int P, int NG, bool kWide, uint32_t kTeams>
__host__ __device__ constexpr uint32_t tile_rows() {
    return consumer_warps<P, NG, kWide>() / kTeams * 128u * (P == kPlaceInRegistersPerThread ? 2u : 1u);
}
template <int P, int NG, bool kWide, uint32_t kTeams>
__host__ __device__ constexpr uint32_t stage_bytes() {
    return ka::TileLayout<tile_rows<P, NG, kWide, kTeams>()>::kStageBytes;
}

// Table engine of the shared_mem_per_thread placement.
enum TableKind : uint32_t { kTableNone = 0, kTableCube = 1, kTableSlots = 2, kTableCube3 = 3 };

__host__ __device__ constexpr uint32_t table_kind(int placement, uint32_t num_groups) {
    return placement != kPlaceSharedMemPerThread
               ? kTableNone
               : (num_groups <= ka::kCube3MaxGroups ? kTableCube3
                                                    : (num_groups <= ka::kCubeMaxGroups ? kTableCube : kTableSlots));
}
__host__ __device__ constexpr uint32_t table_bytes(uint32_t kind, uint32_t num_groups) {
    return kind == kTableCube3 ? ka::cube3_bytes(num_groups)
                               : (kind == kTableCube ? ka::cube_bytes(num_groups)
                                                     : (kind == kTableSlots ? ka::slot_bytes(num_groups < kWideSlots
                                                                                                 ? num_groups
                                                                                                 : kWideSlots)
                                                                            : 0u));
}
// Stages of the ring in `bytes` of shared memory: at most 4 of 2048 rows and more, the same number for
// each team.
template <int P, int NG, bool kWide, uint32_t kTeams>
__host__ constexpr uint32_t stages_in(uint32_t bytes) {
    const uint32_t fit = bytes / stage_bytes<P, NG, kWide, kTeams>();
    const uint32_t most = kTeams == 1 ? 4u : kMaxStages;
    return (fit < most ? fit : most) / kTeams * kTeams;
}
// As many as fit beside the table and the static shared memory (the register placement's records: less
// than 4 KB; the others' barriers: less than 1 KB, which leaves six stages beside the cells of 1024
// groups, where three took 600 M rows 2.35 ms instead of 1.49).
template <int P, int NG, bool kWide, uint32_t kTeams>
__host__ constexpr uint32_t ring_stages(uint32_t kind, uint32_t num_groups) {
    return stages_in<P, NG, kWide, kTeams>(kMaxDynSmem - (P == kPlaceInRegistersPerThread ? 4096 : 1024) -
                                           table_bytes(kind, num_groups));
}
// Teams of the shared tables. One while three stages of its 3072-row tiles fit beside the table, then
// three (100 M rows, 600 groups: 238 us with one team, 244 with two or three; 1000 groups: 303, 280 and
// 273; 2500 groups: 326, 337, 337; 4096 groups, 60 M rows: 279, 270, 270). The (group, discount, tax)
// cells have two throughout (64 groups: 203, 199, 199).
constexpr uint32_t kSmallTeams = 3;
static uint32_t table_teams(uint32_t kind, uint32_t num_groups) {
    if (kind == kTableCube3) return 2;
    return ring_stages<kPlaceSharedMemPerThread, 4, false, 1>(kind, num_groups) >= 3 ? 1 : kSmallTeams;
}
static_assert(ring_stages<kPlaceSharedMemPerThread, 4, false, kSmallTeams>(kTableCube, ka::kCubeMaxGroups) >= 2 * kSmallTeams &&
                  ring_stages<kPlaceSharedMemPerThread, 4, false, kSmallTeams>(kTableSlots, kWideSlots) >= 2 * kSmallTeams,
              "two stages for every team beside the largest tables");

}  // namespace gk

struct GroupKeyParams {
    const uint8_t* col[6];          // ship, qty, disc, tax, price, key (16-byte aligned)
    uint64_t rows;
    int32_t cutoff;                 // cutoff_day - 727563
    uint32_t num_groups;
    uint32_t stages;                // ring stages
    uint32_t stages_no_table;       // and where the global path leaves the table's room free
    unsigned long long* acc;        // scratch: num_groups x 8 u64, zeroed (shared and global placements)
    unsigned long long* out;        // [num_groups][6][lo, hi] (register placement)
    uint32_t* status;
    const uint32_t* mode;           // when set, the path chosen on the device (GroupKeyMode)
};

// P: placement; NG: plane groups of in_registers_per_thread (4 or 8); kWide: 15 consumer warps
// over 3840-row tiles for four groups' planes; kTab: table engine of shared_mem_per_thread. (Each engine
// its own kernel: one kernel with all of them behind a launch parameter ran 64 groups, 100 M rows, in
// 255 us instead of 240 once the global path was a fourth alternative.)
template <uint32_t kTab>
struct TableOf { using T = ka::SlotTable; };
template <> struct TableOf<gk::kTableCube> { using T = ka::CubeTable; };
template <> struct TableOf<gk::kTableCube3> { using T = ka::Cube3Table; };

template <int P, int NG, bool kWide = false, uint32_t kTab = gk::kTableNone, uint32_t kTeams = 1>
__global__ void __launch_bounds__((gk::consumer_warps<P, NG, kWide>() + kTeams) * 32, 1)
    q1_groupkey_kernel(const __grid_constant__ GroupKeyParams prm) {
    using namespace gk;
    constexpr uint32_t W = consumer_warps<P, NG, kWide>();
    constexpr uint32_t R = tile_rows<P, NG, kWide, kTeams>();
    constexpr uint32_t kStage = stage_bytes<P, NG, kWide, kTeams>();
    constexpr uint32_t kSteps = R / 4;   // 4 rows per consumer step
    constexpr uint32_t WT = W / kTeams;   // warps of a team
    static_assert(W % kTeams == 0 && kSteps % (WT * 32) == 0 && kSteps / (WT * 32) * 4 <= 8,
                  "two quads per consumer thread at most");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full_bar[kMaxStages];
    __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
    __shared__ __align__(8) uint64_t cons_bar;
    // the register placement's warp records, and the rows its planes do not take (128-bit sums)
    constexpr uint32_t kRegValues = P == kPlaceInRegistersPerThread ? NG * kNumAggs : 1;
    __shared__ uint64_t warp_rec[P == kPlaceInRegistersPerThread ? W : 1][kRegValues];
    __shared__ __align__(16) unsigned long long wide[2 * kRegValues];
    // a path chosen on the device: this kernel (its table, or no table: the global path) unless partitioned
    constexpr bool kChosen = kTab == kTableSlots && kTeams > 1;
    bool no_table = false;
    if (kChosen && prm.mode) {
        const uint32_t mode = *prm.mode;
        if (mode == kModePartitioned) return;
        no_table = mode == kModeGlobalPath;
    }
    const uint32_t S = no_table ? prm.stages_no_table : prm.stages;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint64_t num_tiles = prm.rows / R;
    const uint32_t ring = smem_addr(smem);
    const uint32_t G = prm.num_groups;
    const uint32_t hot = kTab == kTableSlots && G > kWideSlots ? kWideSlots : G;   // keys the table takes
    typename TableOf<kTab>::T tab;
    if (kTab != kTableNone) tab.bind(smem + S * kStage, hot);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(smem_addr(&full_bar[s]), 1);
            mbar_init(smem_addr(&empty_bar[s]), WT);
        }
        mbar_init(smem_addr(&cons_bar), W);
        fence_mbar_init();
    }
    if (kTab != kTableNone && !no_table) tab.zero(threadIdx.x, blockDim.x);
    if (P == kPlaceInRegistersPerThread)
        for (uint32_t i = threadIdx.x; i < 2 * kRegValues; i += blockDim.x) wide[i] = 0;
    __syncthreads();

    if (warp >= W) {
        // a producer warp per team: its tiles, into every kTeams-th stage. Beside the larger tables lane c
        // issues column c's copies (100 M rows: 600 groups 238 -> 232 us, 1000 273 -> 264, 4096 358 -> 349);
        // elsewhere one lane issues all six (register planes, 4 groups 206 -> 217 with a lane per column; 64
        // groups 200 either way).
        constexpr bool kLanes = kTab == kTableCube || kTab == kTableSlots;
        if (kLanes || lane == 0) {
            const uint64_t pol = policy_evict_first();
            const uint32_t c = lane < 6 ? lane : 5;
            const uint32_t dst = ring + ka::TileLayout<R>::col_off((int)c), bytes = ka::TileLayout<R>::col_bytes((int)c);
            // stage s and phase ph of the tile, stepped rather than divided (S is a launch parameter)
            uint32_t s = warp - W, ph = 0;
            auto next = [&]() {
                s += kTeams;
                if (s >= S) {
                    s -= S;
                    ph ^= 1u;
                }
            };
            const uint64_t step = (uint64_t)kTeams * gridDim.x;
            uint64_t t = blockIdx.x + (uint64_t)(warp - W) * gridDim.x;
            const uint8_t* src = prm.col[c] + t * bytes;
            for (; t < num_tiles; t += step, src += step * bytes) {
                const bool empty = mbar_wait(smem_addr(&empty_bar[s]), ph ^ 1u, prm.status);
                const uint32_t fb = smem_addr(&full_bar[s]);
                if constexpr (kLanes) {
                    if (!__all_sync(0xffffffffu, empty)) break;
                    if (lane == 0) mbar_arrive_expect_tx(fb, kStage);
                    __syncwarp();
                    if (lane < 6) bulk_g2s(dst + s * kStage, src, bytes, fb, pol);
                } else {
                    if (!empty) break;
                    mbar_arrive_expect_tx(fb, kStage);
#pragma unroll
                    for (int k = 0; k < 6; ++k)
                        bulk_g2s(ring + s * kStage + ka::TileLayout<R>::col_off(k),
                                 prm.col[k] + t * (uint64_t)ka::TileLayout<R>::col_bytes(k),
                                 ka::TileLayout<R>::col_bytes(k), fb, pol);
                }
                next();
            }
            // Never leave with copies in flight: wait for the last tiles issued to land.
            for (uint32_t i = 0; i < S; i += kTeams) {
                mbar_wait(smem_addr(&full_bar[s]), ph ^ 1u, prm.status);
                next();
            }
        }
    } else {
        const uint32_t ctid = threadIdx.x;
        ka::PlaneRegs<NG> regs;
        if (P == kPlaceInRegistersPerThread) regs.zero();
        ka::ConsumerBarrier cb{smem_addr(&cons_bar), 0};
        uint32_t bad = 0;
        uint32_t tiles_since = 0;
        uint64_t rows_since = 0;

        // every passing row of a quad straight into the global accumulators
        auto add_global = [&](const ka::KeyQuad& x) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!((x.PM >> (8 * r)) & 1u)) continue;
                const uint32_t key = x.k[r];
                if (key >= G) {
                    bad = 1u;
                    continue;
                }
                ka::scratch_row(prm.acc, key, (x.Q >> (8 * r)) & 0xFFu, (x.D >> (8 * r)) & 0xFFu,
                                (x.X >> (8 * r)) & 0xFFu, x.p[r]);
            }
        };
        // one decoded quad into the placement's engine
        auto add_quad = [&](const ka::KeyQuad& x) {
            if constexpr (P == kPlaceInRegistersPerThread) {
                regs.add(x, G, bad, [&](uint32_t key, uint32_t q, uint32_t d, uint32_t t, uint32_t p) {
                    unsigned long long* v = wide + 2 * (key * kNumAggs);
                    const uint32_t a = 100u - d;
                    atomic_add_u128_shared(v + 2 * kAggCount, 1, 0);
                    atomic_add_u128_shared(v + 2 * kAggQty, q, 0);
                    atomic_add_u128_shared(v + 2 * kAggBasePrice, p, 0);
                    atomic_add_u128_shared(v + 2 * kAggDisc, d, 0);
                    atomic_add_u128_shared(v + 2 * kAggDiscPrice, (uint64_t)a * p, 0);
                    atomic_add_u128_shared(v + 2 * kAggCharge, (uint64_t)(a * (100u + t)) * p, 0);
                });
            } else if constexpr (kTab != kTableNone) {
                ka::table_quad(tab, x, G, hot, prm.acc, bad);
            } else {
                add_global(x);
            }
        };
        auto table_flush = [&]() {
            cb.sync(lane, prm.status);
            tab.flush(prm.acc, hot, ctid, W * 32);
            cb.sync(lane, prm.status);
        };

        // all of this CTA's rows through `add`
        auto add_rows = [&](auto&& add, bool flushes) {
            bool ok = true;
            uint32_t s = warp / WT, ph = 0;   // stage and phase of the team's tile
            // a round is a tile for every team (the last one's may be past the end: the flushes below
            // are barriers of all consumer warps)
            for (uint64_t t0 = blockIdx.x; t0 < num_tiles; t0 += (uint64_t)kTeams * gridDim.x) {
                if (P == kPlaceInRegistersPerThread && tiles_since >= ka::kPlaneFlushTiles) {
#pragma unroll
                    for (int i = 0; i < NG; ++i)
#pragma unroll
                        for (int a = 0; a < kNumAggs; ++a) {
                            const uint64_t v = regs.warp_total(i, a) * (a == kAggQty ? 100u : 1u);
                            if (lane == 0 && (uint32_t)i < G) atomic_add_u128(prm.out + 2 * (i * kNumAggs + a), v, 0);
                        }
                    regs.zero();
                    tiles_since = 0;
                }
                if (flushes && rows_since + kTeams * R > ka::kTableFlushRows) {
                    table_flush();
                    rows_since = 0;
                }
                ++tiles_since;
                rows_since += kTeams * R;
                if (t0 + (uint64_t)(warp / WT) * gridDim.x >= num_tiles) continue;
                const bool landed = mbar_wait(smem_addr(&full_bar[s]), ph, prm.status);
                if (!__all_sync(0xffffffffu, landed)) {
                    ok = false;
                    break;
                }
                const uint32_t base = ring + s * kStage;
#pragma unroll
                for (uint32_t it = 0; it < kSteps / (WT * 32); ++it)
                    add(ka::load_quad<R>(base, ctid % (WT * 32) + it * (WT * 32), prm.cutoff, bad));
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_addr(&empty_bar[s]));
                s += kTeams;
                if (s >= S) {
                    s -= S;
                    ph ^= 1u;
                }
            }
            // the rows after the last full tile, straight from global memory: spread over the CTAs, those with
            // a tile less first (register planes, whose loop that made 2% slower: by one CTA)
            constexpr bool kSpread = P != kPlaceInRegistersPerThread;
            const uint32_t extra = (uint32_t)(num_tiles % gridDim.x);
            const uint32_t turn = blockIdx.x >= extra ? blockIdx.x - extra : blockIdx.x + gridDim.x - extra;
            uint64_t i0 = kSpread || turn == 0 ? num_tiles * R + (uint64_t)turn * (W * 32) : prm.rows;
            if (ok && i0 < prm.rows) {
                if (flushes && rows_since + kTeams * R > ka::kTableFlushRows) table_flush();
                // every lane runs every round (the table engines vote across the warp)
                for (; i0 < prm.rows; i0 += (uint64_t)(kSpread ? gridDim.x : 1u) * (W * 32)) {
                    const uint64_t i = i0 + ctid;
                    add(i < prm.rows ? ka::load_row(prm.col, i, prm.cutoff, bad) : ka::empty_quad());
                }
            }
        };
        if (kChosen && no_table) add_rows(add_global, false);
        else add_rows(add_quad, kTab != kTableNone);
        if (bad && prm.status) atomicOr(prm.status, kStatusDomain);
        if constexpr (P == kPlaceInRegistersPerThread) {
#pragma unroll
            for (int i = 0; i < NG; ++i)
#pragma unroll
                for (int a = 0; a < kNumAggs; ++a) {
                    const uint64_t v = regs.warp_total(i, a);
                    if (lane == 0) warp_rec[warp][i * kNumAggs + a] = v;
                }
        }
    }
    __syncthreads();
    if constexpr (P == kPlaceInRegistersPerThread) {
        // the CTA's sums (below 2^64 over its warps) and the rows kept out of the planes
        if (threadIdx.x < G * kNumAggs) {
            uint64_t lo = 0;
#pragma unroll
            for (uint32_t w = 0; w < W; ++w) lo += warp_rec[w][threadIdx.x];
            unsigned __int128 v = ((unsigned __int128)wide[2 * threadIdx.x + 1] << 64 | wide[2 * threadIdx.x]) + lo;
            if (threadIdx.x % kNumAggs == kAggQty) v *= 100u;
            atomic_add_u128(prm.out + 2 * threadIdx.x, (uint64_t)v, (uint64_t)(v >> 64));
        }
    }
    // CTAs start at different groups, so that they do not all add to the same words at once (6.0 M rows,
    // 4096 groups 91 -> 81 us, 1000 groups 62.5 -> 59 us)
    if (kTab != kTableNone && !no_table)
        tab.flush(prm.acc, hot, threadIdx.x, blockDim.x, (uint32_t)((uint64_t)blockIdx.x * hot / gridDim.x));
}

// acc (num_groups x 8 u64) -> out[group][6] int128 (+=), quantity scaled to hundredths.
__global__ void __launch_bounds__(256) q1_groupkey_finalize(const unsigned long long* __restrict__ acc,
                                                            uint32_t num_groups, unsigned long long* out) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= num_groups) return;
    const unsigned long long* a = acc + 8ull * g;
    if (!a[0]) return;
    unsigned long long* o = out + 12ull * g;
    atomic_add_u128(o + 2 * kAggCount, a[0], 0);
    const unsigned __int128 q = (unsigned __int128)a[1] * 100u;
    atomic_add_u128(o + 2 * kAggQty, (uint64_t)q, (uint64_t)(q >> 64));
    atomic_add_u128(o + 2 * kAggBasePrice, a[3], 0);
    atomic_add_u128(o + 2 * kAggDisc, a[2], 0);
    const unsigned __int128 dp = (unsigned __int128)a[4] + ((unsigned __int128)a[5] << 32);
    atomic_add_u128(o + 2 * kAggDiscPrice, (uint64_t)dp, (uint64_t)(dp >> 64));
    const unsigned __int128 ch = (unsigned __int128)a[6] + ((unsigned __int128)a[7] << 32);
    atomic_add_u128(o + 2 * kAggCharge, (uint64_t)ch, (uint64_t)(ch >> 64));
}

template <int P, int NG, bool kWide = false, uint32_t kTab = gk::kTableNone, uint32_t kTeams = 1>
static cudaError_t launch_gk(GroupKeyParams prm, int sm_count, int max_blocks, cudaStream_t st) {
    using namespace gk;
    constexpr uint32_t R = tile_rows<P, NG, kWide, kTeams>();
    prm.stages = ring_stages<P, NG, kWide, kTeams>(kTab, prm.num_groups);
    const uint32_t dyn = prm.stages * stage_bytes<P, NG, kWide, kTeams>() + table_bytes(kTab, prm.num_groups);
    prm.stages_no_table = stages_in<P, NG, kWide, kTeams>(dyn);
    cudaError_t e = cudaFuncSetAttribute(q1_groupkey_kernel<P, NG, kWide, kTab, kTeams>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    const uint64_t tiles = prm.rows / R;
    uint64_t blocks = tiles ? tiles : 1;
    uint64_t cap = (uint64_t)sm_count;
    if (max_blocks > 0 && (uint64_t)max_blocks < cap) cap = (uint64_t)max_blocks;
    if (blocks > cap) blocks = cap;
    q1_groupkey_kernel<P, NG, kWide, kTab, kTeams><<<(unsigned)blocks, (consumer_warps<P, NG, kWide>() + kTeams) * 32, dyn, st>>>(prm);
    return cudaGetLastError();
}

static cudaError_t launch_table(uint32_t table, uint32_t teams, const GroupKeyParams& prm, int sm_count, int max_blocks,
                                cudaStream_t st) {
    constexpr int P = kPlaceSharedMemPerThread;
    using namespace gk;
    if (table == kTableCube3) return launch_gk<P, 4, false, kTableCube3, 2>(prm, sm_count, max_blocks, st);
    if (table == kTableCube)
        return teams == 1 ? launch_gk<P, 4, false, kTableCube, 1>(prm, sm_count, max_blocks, st)
                          : launch_gk<P, 4, false, kTableCube, kSmallTeams>(prm, sm_count, max_blocks, st);
    return teams == 1 ? launch_gk<P, 4, false, kTableSlots, 1>(prm, sm_count, max_blocks, st)
                      : launch_gk<P, 4, false, kTableSlots, kSmallTeams>(prm, sm_count, max_blocks, st);
}

static uint64_t acc_bytes(uint32_t num_groups) { return 64ull * num_groups; }
// Whether the kernel of the shared placement takes a path chosen on the device (the largest tables').
static bool takes_choice(int placement, uint32_t num_groups) {
    const uint32_t table = gk::table_kind(placement, num_groups);
    return table == gk::kTableSlots && gk::table_teams(table, num_groups) > 1;
}
// Whether the path is chosen, by rows of the launch; elsewhere it is the single pass. The choice costs a
// launch (10 us, 20 us before the partition's kernels) and the global path gains little on the tables:
// with 1% of the rows passing, 200 M rows, 1030 groups 485 us against 406 with the table, 2500 groups 482
// and 432, 4096 groups 396 and 497, where 25 M rows take 81 and 80. Above 4096 groups a key without a slot
// may hold most of the rows, 4.3 ns each in the single pass: it is chosen from 4096 rows on, where that is 18 us.
static bool chosen_on_device(int placement, uint32_t num_groups, uint64_t rows) {
    return takes_choice(placement, num_groups) &&
           rows >= (num_groups >= groupkey_part_min_groups() ? 1ull << 12 : 1ull << 25);
}

// Chooses the path of the shared placement's largest tables (takes_choice) from 8192 evenly spaced
// sample rows and writes it to *mode (every path gives identical results):
//   kModeGlobalPath   every passing row straight into the global accumulators, when fewer than
//                     2% of the rows pass and no key occurs more than 3 times among the sampled
//                     passing rows (global atomics on spread keys do not contend: 1.29 ms per
//                     600 M rows at 1% pass, against 2.0 ms for the slot table; frequent keys make
//                     them contend, 11.7 ms for Zipf keys at 1% pass);
//   kModeSinglePass   the group-key kernel: keys < 4096 in a shared slot table, passing rows of
//                     larger ("cold") keys straight into the global accumulators;
//   kModePartitioned  (more than 4096 groups) the two-pass radix partition (groupkey_part.cu).
// Between the last two, a cost model fitted to both paths on a B200 (ms per 200 M rows; c = fraction of
// the rows that pass with a cold key, p = fraction that pass): single pass 0.73 + 3.5 c + 0.35 p (Zipf
// keys over 5,000 to 65,536 groups 1.08, 1.49, 1.90 at full pass; uniform ones, all cold, 6.1 to 6.8),
// partitioned 0.56 + 0.75 p and 8 us for its three kernels (1.26 and 1.35 uniform and Zipf at full
// pass, 0.65 at 7%). Rows of one cold key wait for each other in the single pass, 860 ms for 200 M (1.0 M rows, all
// of one cold key, 4.38 ms): h is the fullest of 8192 bins of the sampled cold keys, less 12 samples that spread
// keys put in one, as a fraction. The single pass wins when (0.17 + 3.5 c - 0.4 p + 860 h) x rows < 1.5 M.
// All loads of a thread's eight samples are in flight together: one block of 256 threads taking them
// one after another was 31 us, two thirds of a launch on 100,000 rows.
__global__ void __launch_bounds__(1024) q1_groupkey_choose(const uint16_t* __restrict__ ship,
                                                           const uint32_t* __restrict__ keys, uint64_t rows,
                                                           int32_t cutoff, uint32_t hot, uint32_t allow_part,
                                                           uint32_t force, uint32_t* mode) {
    constexpr uint32_t K = 8192, kPer = K / 1024, kList = 512;
    if (force) {
        if (threadIdx.x == 0) *mode = force;
        return;
    }
    __shared__ uint32_t cnt[4];       // passing, cold, listed, largest key multiplicity
    __shared__ uint32_t list[kList];  // keys of the sampled passing rows
    __shared__ uint32_t bins[K];      // sampled cold keys by hash
    __shared__ uint32_t fullest;
    if (threadIdx.x < 4) cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) fullest = 0;
#pragma unroll
    for (uint32_t e = 0; e < kPer; ++e) bins[e * 1024 + threadIdx.x] = 0;
    uint32_t day[kPer], key[kPer];
#pragma unroll
    for (uint32_t e = 0; e < kPer; ++e) {
        const uint64_t i = (uint64_t)(e * 1024 + threadIdx.x) * rows / K;
        day[e] = __ldg(ship + i);
        key[e] = __ldg(keys + i);
    }
    __syncthreads();
    uint32_t pass = 0, cold = 0, most = 0;
#pragma unroll
    for (uint32_t e = 0; e < kPer; ++e) {
        const bool in = (int32_t)day[e] <= cutoff;
        pass += in ? 1u : 0u;
        if (in && key[e] >= hot) {
            ++cold;
            most = max(most, atomicAdd(&bins[key[e] * 0x9E3779B1u >> 19], 1u) + 1u);
        }
    }
    static_assert(K == 1u << (32 - 19), "a bin of 13 bits");
    pass = __reduce_add_sync(0xffffffffu, pass);
    cold = __reduce_add_sync(0xffffffffu, cold);
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&cnt[0], pass);
        atomicAdd(&cnt[1], cold);
        atomicMax(&fullest, most);
    }
    __syncthreads();
    const uint32_t P = cnt[0], C = cnt[1];
    const bool few = (uint64_t)P * 50 < K;   // fewer than 164: they fit the list
    static_assert(K / 50 < kList, "the few passing rows' keys fit the list");
    if (few) {
#pragma unroll
        for (uint32_t e = 0; e < kPer; ++e)
            if ((int32_t)day[e] <= cutoff) list[atomicAdd(&cnt[2], 1u)] = key[e];
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < P; e += blockDim.x) {
            uint32_t m = 0;
            for (uint32_t x = 0; x < P; ++x) m += list[x] == list[e] ? 1u : 0u;
            atomicMax(&cnt[3], m);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (few && cnt[3] <= 3) {
            *mode = kModeGlobalPath;
        } else if (!allow_part) {
            *mode = kModeSinglePass;
        } else {
            // 1000 x (0.17 + 3.5 c - 0.4 p + 860 h) x K, within 2^32, so that its product with the rows is exact
            const int64_t score = min(170ll * K + 3500ll * C - 400ll * P + 860000ll * (fullest > 12 ? fullest - 12 : 0),
                                      4000000000ll);
            *mode = score * (int64_t)rows < 1500000000ll * K ? kModeSinglePass : kModePartitioned;
        }
    }
}

cudaError_t launch_groupkey(int placement, const uint8_t* const cols[6], uint64_t rows, int32_t cutoff_rel,
                            uint32_t num_groups, unsigned long long* scratch, unsigned long long* out,
                            uint32_t* status, int sm_count, int max_blocks, cudaStream_t stream) {
    const bool direct = placement == kPlaceInRegistersPerThread;   // no scratch: straight into `out`
    cudaError_t e = direct ? cudaSuccess : cudaMemsetAsync(scratch, 0, acc_bytes(num_groups), stream);
    if (e != cudaSuccess) return e;
    uint8_t* workspace = reinterpret_cast<uint8_t*>(scratch) + ((acc_bytes(num_groups) + 255) & ~255ull);
    const bool part = num_groups >= groupkey_part_min_groups();
    // Q1_GROUPKEY_PATH=single|partitioned|global overrides the sample-based choice (tests, tuning)
    uint32_t force = 0;
    if (const char* env = std::getenv("Q1_GROUPKEY_PATH")) {
        if (!std::strcmp(env, "single")) force = kModeSinglePass;
        else if (!std::strcmp(env, "partitioned") && part) force = kModePartitioned;
        else if (!std::strcmp(env, "global")) force = kModeGlobalPath;
    }
    const uint64_t kMaxRows = 1ull << 31;
    for (uint64_t off = 0; off < rows; off += kMaxRows) {
        GroupKeyParams prm{};
        const uint64_t n = rows - off < kMaxRows ? rows - off : kMaxRows;
        const uint32_t bytes[6] = {2, 1, 1, 1, 4, 4};
        for (int c = 0; c < 6; ++c) prm.col[c] = cols[c] + off * bytes[c];
        prm.rows = n;
        prm.cutoff = cutoff_rel;
        prm.num_groups = num_groups;
        const uint32_t table = gk::table_kind(placement, num_groups);
        uint32_t* mode = nullptr;   // the path, when it is not the single pass throughout
        if (force ? force != kModeSinglePass && takes_choice(placement, num_groups)
                  : chosen_on_device(placement, num_groups, n))
            mode = reinterpret_cast<uint32_t*>(workspace + groupkey_part_mode_offset());
        const bool forced_global = force == kModeGlobalPath && num_groups > 256 && !mode;
        prm.acc = scratch;
        prm.out = out;
        prm.status = status;
        if (mode) {
            q1_groupkey_choose<<<1, 1024, 0, stream>>>(reinterpret_cast<const uint16_t*>(prm.col[0]),
                                                      reinterpret_cast<const uint32_t*>(prm.col[5]), n, cutoff_rel,
                                                      gk::kWideSlots, part ? 1u : 0u, force, mode);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            prm.mode = mode;
        }
        switch (placement) {
            case kPlaceInRegistersPerThread: {
                // The wide tiles on a table of at least 32 tiles per CTA of the grid (18.2 M rows on
                // 148 SMs): one such scan is up to 20% faster (with 12 warps, 50 M rows 136 -> 115 us), but a queue
                // of launches on tables of a few million rows ran slower with them (256 launches on
                // 10^4..5*10^7 rows: 10.72 ms with 2048-row tiles throughout, 11.56 ms with the wide
                // ones from 2 tiles per CTA, 10.78 ms from 32).
                const uint64_t grid = (max_blocks > 0 && max_blocks < sm_count) ? (uint64_t)max_blocks : (uint64_t)sm_count;
                const bool wide = n >= 32 * grid * gk::tile_rows<kPlaceInRegistersPerThread, 4, true, 1>();
                e = num_groups > 4 ? launch_gk<kPlaceInRegistersPerThread, 8>(prm, sm_count, max_blocks, stream)
                    : wide         ? launch_gk<kPlaceInRegistersPerThread, 4, true>(prm, sm_count, max_blocks, stream)
                                   : launch_gk<kPlaceInRegistersPerThread, 4>(prm, sm_count, max_blocks, stream);
                break;
            }
            case kPlaceSharedMemPerThread:
                e = forced_global ? launch_gk<kPlaceGlobal, 4>(prm, sm_count, max_blocks, stream)
                                 : launch_table(table, gk::table_teams(table, num_groups), prm, sm_count, max_blocks, stream);
                break;
            case kPlaceGlobal: e = launch_gk<kPlaceGlobal, 4>(prm, sm_count, max_blocks, stream); break;
            default: return cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) return e;
        if (mode && part) {
            e = launch_groupkey_part(prm.col, n, cutoff_rel, num_groups, scratch, workspace, mode, status, sm_count,
                                     max_blocks, stream);
            if (e != cudaSuccess) return e;
        }
        if (direct) continue;
        // fold after every 2^31-row launch so the scratch sums stay exact
        q1_groupkey_finalize<<<(num_groups + 255) / 256, 256, 0, stream>>>(scratch, num_groups, out);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (off + kMaxRows < rows) {
            e = cudaMemsetAsync(scratch, 0, acc_bytes(num_groups), stream);
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

// The accumulators; for the largest tables also the mode word of the shared placement's path choice (room for it
// from 257 on), and above 4096 groups the partition workspace (which holds that word).
uint64_t groupkey_scratch_bytes(uint32_t num_groups) {
    const uint64_t a = (acc_bytes(num_groups) + 255) & ~255ull;
    if (num_groups >= groupkey_part_min_groups()) return a + groupkey_part_workspace_bytes();
    if (num_groups > 256) return a + 256;   // the path choice's mode word
    return acc_bytes(num_groups);
}

// Group keys of the seeded generator: uniform over [0, G) (cdf == nullptr) or by inverse CDF.
__global__ void __launch_bounds__(256) generate_keys_kernel(uint64_t key, uint64_t first_row, uint64_t rows,
                                                            uint32_t num_groups, const uint32_t* __restrict__ cdf,
                                                            uint32_t* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    out[i] = cdf ? gen_group_key_cdf(key, first_row + i, cdf, num_groups)
                 : gen_group_key_uniform(key, first_row + i, num_groups);
}

cudaError_t launch_generate_keys(uint64_t seed, uint64_t first_row, uint64_t rows, uint32_t num_groups,
                                 const uint32_t* dev_cdf, uint32_t* dev_keys, cudaStream_t stream) {
    if (!rows) return cudaSuccess;
    generate_keys_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, stream>>>(gen_key(seed), first_row, rows, num_groups,
                                                                          dev_cdf, dev_keys);
    return cudaGetLastError();
}

}  // namespace q1
