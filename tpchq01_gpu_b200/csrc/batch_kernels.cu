// Batched Q1 aggregation: many independent instances (each its own table, cutoff and group count)
// in ONE persistent kernel over a device-side queue of row tiles.
//
// Each instance is a group-key table (ship u16, qty u8, disc u8, tax u8, price u32, key u32;
// 13 B/row) aggregated exactly as q1_launch_groupkey does (groupkey_kernels.cu): the per-row
// arithmetic is the reference's (src/kernels/ht_in_global_mem.hpp:31-49) with group = key.
//
// Work queue: the host splits every instance into items of at most `chunk` tiles of 2048 rows
// (the autotuner chooses the chunk); CTAs claim items with an atomic cursor, so small and large
// instances balance across the GPU without one launch per instance.
//
// Per CTA: 24 consumer warps in three teams, each with a producer warp. The producers go through the
// items that the first of them claims, and stream the column slices of their team's tiles (1024 rows,
// in turn) with cp.async.bulk into a shared-memory ring of 6 to 9 stages (a partial last tile is read by
// the consumers straight from global memory instead). The teams aggregate into one table; when the
// instance changes all of them flush it into the instance's scratch (red.global.add), according to
// the instance's placement mode:
//   kModeShared     num_groups <= 4: (group, discount, tax) cells and slots by lane (ka::FewTable); <= 64:
//                   shared (group, discount, tax) cells (ka::Cube3Table); <= 1024: shared (group,
//                   discount) cells (ka::CubeTable); more groups: shared slots for keys < 2048
//                   (ka::SlotTable), the rest spilled
//   kModeGlobal     every passing row reduces straight into the scratch accumulators
// Few groups: 100 M rows of 4 groups 210 us, of one group 216 (byte planes in registers, in a kernel of their
// own, 299 and 290: in this one they spill). Eight tables by lane instead of one: 4.0 M rows of one group with one
// discount and tax 29 us instead of 72 (planes 29). Slots by lane instead of the scratch for rows outside the
// cells' domain: with taxes up to 19, 35 us instead of 9,480 (planes 29); prices of 2^24 and more 35 us instead of
// 19,800 (planes 19,400). Sums of every thread's own in shared memory, for rows of any values, took 257 us per
// 100 M rows.
// Bound: 64 instances as above take 245 us, their bytes 191 at the copy rate; with 64 groups all, 217: the
// shared atomics of a row and the last pieces. 16 consumer warps in one team with one producer: 291.
// (engines in q1_keyagg.cuh). Scratch per instance: num_groups x 8 u64, folded into the
// caller's int128 table by batch_finalize.
// All waits are bounded (q1_ptx.cuh); on expiry the kernel records a status bit and leaves.
#include <cuda_runtime.h>
#include <stdint.h>

#include "q1_batch.h"
#include "q1_common.cuh"
#include "q1_keyagg.cuh"
#include "q1_ptx.cuh"

namespace q1 {

using namespace ptx;

namespace bk {

// Consumer warps in teams that take the ring's tiles in turn: the shared-memory atomics need many warps
// in flight, and a large table leaves room for a few small tiles.
constexpr uint32_t kWarps = 24, kTeams = 3, kTeamWarps = kWarps / kTeams;
constexpr uint32_t R = kTeamWarps * 128;   // rows of a ring tile: one quad per consumer thread
static_assert(kBatchTileRows % R == 0, "whole ring tiles in a work item's tile");
// Rows of a run, between two flushes of an engine's table.
__host__ __device__ constexpr uint32_t flush_rows(uint32_t engine) {
    return (uint32_t)(engine == kEngFew ? ka::kFewFlushRows : ka::kTableFlushRows);
}
static_assert((uint64_t)kBatchMaxItemTiles * kBatchTileRows <= flush_rows(kEngGlobal) &&
                  (uint64_t)kBatchMaxFewItemTiles * kBatchTileRows <= flush_rows(kEngFew), "an item in one run");
static_assert(kTeamWarps <= ka::kFewTeamWarps, "rows of a lane");
using Tile = ka::TileLayout<R>;
constexpr uint32_t kStage = Tile::kStageBytes;
constexpr uint32_t kMaxStages = 9;         // of the ring
constexpr uint32_t kStaticBytes = 1024;    // at most, of static shared memory
constexpr uint32_t kDynBytes = 227 * 1024 - kStaticBytes;   // ring, then table
constexpr uint32_t kKindFull = 0, kKindPartial = 1, kKindEnd = 2;

constexpr uint32_t table_bytes(uint32_t engine, uint32_t groups) {
    return engine == kEngFew     ? ka::few_bytes(groups)
           : engine == kEngCube3 ? ka::cube3_bytes(groups)
           : engine == kEngCube ? ka::cube_bytes(groups)
           : engine == kEngSlots ? ka::slot_bytes(groups < ka::kSlots ? groups : ka::kSlots)
                                 : 0;
}
// As many stages as fit beside the table, the same number for each team.
constexpr uint32_t stages_beside(uint32_t bytes) {
    const uint32_t fit = (kDynBytes - bytes) / kStage;
    return (fit < kMaxStages ? fit : kMaxStages) / kTeams * kTeams;
}
static_assert(stages_beside(table_bytes(kEngFew, ka::kFewGroups)) == 9 &&
                  stages_beside(table_bytes(kEngCube3, ka::kCube3MaxGroups)) == 9 &&
                  stages_beside(table_bytes(kEngCube, ka::kCubeMaxGroups)) == 6 &&
                  stages_beside(table_bytes(kEngSlots, ka::kSlots)) == 9,
              "ring beside the largest tables");

struct __align__(16) StageMeta {
    uint32_t tag;        // kind | run << 2: the run of tiles (Run) it belongs to; kKindEnd: the runs so far
    uint32_t instance;   // kKindEnd: the engine to go on with, kEngines when the work is done
    uint32_t tile;       // ring tile of the instance, low word
    uint32_t rows;       // rows | the tile's high word << 16
};

// A run: consecutive tiles of one instance in this CTA, at most flush_rows() of them; the table
// is flushed at its end. Every team's producer numbers all runs alike and writes their descriptors for
// its own team before the next stage that it posts. A team's next stage is at most a few of its tiles
// past the last one it released (a ring's worth and one), and so many times three of the CTA's, each of
// which may begin a run.
constexpr uint32_t kRuns = kMaxStages + kTeams + 1;
struct __align__(16) Run {
    unsigned long long* acc;   // the instance's scratch accumulators
    uint32_t num_groups;
    int32_t cutoff;
};

// Work items on their way from the claiming producer to the others.
constexpr uint32_t kClaims = 2;
static_assert(sizeof(BatchItem) == 16, "claims");

// A consumer warp's place: the stage its team reads next and its phase, the runs flushed so far.
struct Place {
    uint32_t s, ph, run;
};

// Consumer side of one engine: processes the team's stages until the producer's end-of-engine
// marker, flushing the table at the end of every run (a barrier of all consumer warps: each team goes
// through all runs, also those none of its tiles belong to). Returns the engine to go on with, kEngines
// at the end or if a bounded wait expired (the kernel then stops). (A function of its own for each engine: inlined
// in one, 64 instances of 64 groups took 218 us instead of 215, of 1024 groups 302 instead of 292.)
template <int E>
static __device__ __noinline__ uint32_t consume_engine(const BatchParams& prm, uint32_t ring, uint8_t* smem,
                                                       uint64_t* full_bar, uint64_t* empty_bar, const StageMeta* meta,
                                                       const Run* runs, Place& at_, ka::ConsumerBarrier& cb_,
                                                       uint32_t& bad_) {
    Place at = at_;
    ka::ConsumerBarrier cb = cb_;
    uint32_t bad = bad_;
    auto leave = [&](uint32_t e) {
        at_ = at, cb_ = cb, bad_ = bad;
        return e;
    };
    const uint32_t S = prm.stages[E];
    uint8_t* const tab = smem + S * kStage;   // all zero between runs
    const uint32_t lane = threadIdx.x & 31u, ctid = threadIdx.x, ttid = ctid % (kTeamWarps * 32);
    ka::FewTable few;
    ka::Cube3Table cube3;
    ka::CubeTable cube;
    ka::SlotTable slots;
    unsigned long long* acc = nullptr;
    uint32_t num_groups = 0, hot = 0;   // hot: keys below it go to the shared table
    int32_t cutoff = 0;

    auto bind = [&]() {
        const Run& r = runs[at.run % kRuns];
        acc = r.acc;
        num_groups = r.num_groups;
        cutoff = r.cutoff;
        hot = (E == kEngSlots && num_groups > ka::kSlots) ? ka::kSlots : num_groups;
        if constexpr (E == kEngFew) few.bind(tab, num_groups, lane);
        if constexpr (E == kEngCube3) cube3.bind(tab, num_groups);
        if constexpr (E == kEngCube) cube.bind(tab, num_groups);
        if constexpr (E == kEngSlots) slots.bind(tab, hot);
    };
    auto add = [&](const ka::KeyQuad& x) {
        if constexpr (E == kEngFew) {
            ka::table_quad(few, x, num_groups, hot, acc, bad);
        } else if constexpr (E == kEngCube3) {
            ka::table_quad(cube3, x, num_groups, hot, acc, bad);
        } else if constexpr (E == kEngCube) {
            ka::table_quad(cube, x, num_groups, hot, acc, bad);
        } else if constexpr (E == kEngSlots) {
            ka::table_quad(slots, x, num_groups, hot, acc, bad);
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!((x.PM >> (8 * r)) & 1u)) continue;
                const uint32_t key = x.k[r];
                if (key >= num_groups) {
                    bad = 1u;
                    continue;
                }
                ka::scratch_row(acc, key, (x.Q >> (8 * r)) & 0xFFu, (x.D >> (8 * r)) & 0xFFu, (x.X >> (8 * r)) & 0xFFu,
                                x.p[r]);
            }
        }
    };

    constexpr uint32_t kUnbound = 0xFFFFFFFFu;
    uint32_t current = kUnbound;   // tag of a full tile of run at.run, once the fields above are that run's
    for (;;) {
        const bool landed = mbar_wait(smem_addr(&full_bar[at.s]), at.ph, prm.status);
        if (!__all_sync(0xffffffffu, landed)) return leave(kEngines);
        const uint32_t tag = meta[at.s].tag;
        uint32_t n = 0, next = kEngines;   // rows of a partial tile, engine after this one
        if (tag != current) {
            for (; at.run < tag >> 2; ++at.run) {
                if constexpr (E != kEngGlobal) {
                    if (current == kUnbound) bind();
                    cb.sync(lane, prm.status);
                    if constexpr (E == kEngFew) few.flush(acc, ctid >> 5, lane);
                    else if constexpr (E == kEngCube3) cube3.flush(acc, num_groups, ctid, kWarps * 32);
                    else if constexpr (E == kEngCube) cube.flush(acc, num_groups, ctid, kWarps * 32);
                    else slots.flush(acc, hot, ctid, kWarps * 32);
                    cb.sync(lane, prm.status);
                }
                current = kUnbound;
            }
            if ((tag & 3u) == kKindEnd) {
                next = meta[at.s].instance;
            } else {
                if (current == kUnbound) bind();
                current = at.run << 2 | kKindFull;
                if ((tag & 3u) == kKindPartial) n = meta[at.s].rows & 0xFFFFu;
            }
        }
        if (tag == current) {
            add(ka::load_quad<R>(ring + at.s * kStage, ttid, cutoff, bad));
        } else if (n) {
            // every lane runs every round (the table engines vote across the warp)
            const uint8_t* const* col = prm.inst[meta[at.s].instance].col;
            const uint64_t row0 = ((uint64_t)(meta[at.s].rows >> 16) << 32 | meta[at.s].tile) * R;
            for (uint32_t i0 = 0; i0 < n; i0 += kTeamWarps * 32) {
                const uint32_t i = i0 + ttid;
                add(i < n ? ka::load_row(col, row0 + i, cutoff, bad) : ka::empty_quad());
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_addr(&empty_bar[at.s]));
        at.s += kTeams;
        if (at.s >= S) {
            at.s -= S;
            at.ph ^= 1u;
        }
        if ((tag & 3u) == kKindEnd) return leave(next);
    }
}

// Engine queue processed at step `step` of a CTA: it starts at its role's queue (grid ranges
// role_end) and visits the others in turn.
__device__ __forceinline__ uint32_t queue_at(const BatchParams& prm, uint32_t step) {
    uint32_t e0 = 0;
    while (e0 + 1 < kEngines && blockIdx.x >= prm.role_end[e0]) ++e0;
    return (e0 + step) % kEngines;
}

__device__ __forceinline__ void zero_table(const BatchParams& prm, uint8_t* smem, uint32_t e, uint32_t tid, uint32_t n) {
    uint32_t* const w = reinterpret_cast<uint32_t*>(smem + prm.stages[e] * kStage);
    for (uint32_t i = tid; i < prm.table_words[e]; i += n) w[i] = 0;
}

}  // namespace bk

__global__ void __launch_bounds__((bk::kWarps + bk::kTeams) * 32, 1)
    q1_batch_kernel(const __grid_constant__ BatchParams prm) {
    using namespace bk;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full_bar[kMaxStages];
    __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
    __shared__ StageMeta meta[kMaxStages];
    __shared__ Run runs[kTeams][kRuns];
    __shared__ __align__(16) BatchItem claim[kClaims];
    __shared__ __align__(8) uint64_t claim_full[kClaims];
    __shared__ __align__(8) uint64_t claim_empty[kClaims];
    __shared__ __align__(8) uint64_t consumers_bar;   // barrier of the consumer warps (bounded wait)
    __shared__ __align__(8) uint64_t engine_bar;      // the next engine's table is in place
    static_assert(sizeof(full_bar) + sizeof(empty_bar) + sizeof(meta) + sizeof(runs) + sizeof(claim) +
                          2 * sizeof(claim_full) + 32 <= kStaticBytes, "static shared memory");

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t ring = smem_addr(smem);
    const uint32_t first_engine = queue_at(prm, 0);

    auto init_ring = [&]() {
        for (uint32_t s = 0; s < kMaxStages; ++s) {
            mbar_init(smem_addr(&full_bar[s]), 1);
            mbar_init(smem_addr(&empty_bar[s]), kTeamWarps);
        }
    };
    if (threadIdx.x == 0) {
        init_ring();
        for (uint32_t i = 0; i < kClaims; ++i) {
            mbar_init(smem_addr(&claim_full[i]), 1);
            mbar_init(smem_addr(&claim_empty[i]), kTeams);
        }
        mbar_init(smem_addr(&consumers_bar), kWarps);
        mbar_init(smem_addr(&engine_bar), 1);
        fence_mbar_init();
    }
    zero_table(prm, smem, first_engine, threadIdx.x, blockDim.x);
    __syncthreads();

    if (warp >= kWarps) {
        // ------------------------------ producers ---------------------------------------
        // One for each team. They go through the items that team 0's producer claims (and passes
        // on), queue after queue, and post the tiles that are their team's; between engines, and at
        // the end, a marker. Lane c issues column c's copies: beside 24 busy warps a producer's
        // instructions are what bounds it (one lane for all columns, stepping through every tile of an item:
        // 64 instances of 10^4 to 10^7 rows 285 us instead of 245).
        const uint64_t pol = policy_evict_first();
        const uint32_t team = warp - kWarps;
        const uint32_t c6 = lane < 6 ? lane : 5;             // the lane's column
        const uint32_t dst = ring + Tile::col_off((int)c6), bytes = Tile::col_bytes((int)c6);
        Run* const desc = runs[team];
        uint32_t engine = first_engine, S = prm.stages[engine], switches = 0, step = 0;
        uint32_t s = team, ph = 1, posted = 0;       // stage, the parity of its emptiness, stages posted
        uint32_t turn = 0;                           // team of the next tile
        uint32_t run = 0xFFFFFFFFu, run_rows = 0;    // the last run begun
        uint32_t run_instance = 0xFFFFFFFFu;
        uint32_t c = 0, cph = 0;                     // claim slot and its phase
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            return __all_sync(0xffffffffu, mbar_wait(smem_addr(bar), parity, prm.status));
        };
        auto step_stage = [&]() {
            __syncwarp();
            ++posted;
            s += kTeams;
            if (s >= S) {
                s -= S;
                ph ^= 1u;
            }
        };
        for (bool ok = true; ok;) {
            if (team == 0) {
                if (!wait(&claim_empty[c], cph ^ 1u)) break;
                if (lane == 0) {
                    BatchItem it;
                    it.num_tiles = 0;   // every queue is empty
                    for (; step < kEngines; ++step) {
                        const uint32_t e = queue_at(prm, step), count = prm.item_begin[e + 1] - prm.item_begin[e];
                        const uint32_t idx = count ? atomicAdd(prm.cursor + e, 1u) : 0;
                        if (idx < count) {
                            it = prm.items[prm.item_begin[e] + idx];
                            it.pad = e;
                            break;
                        }
                    }
                    claim[c] = it;
                    mbar_arrive(smem_addr(&claim_full[c]));
                }
            }
            if (!wait(&claim_full[c], cph)) break;
            const BatchItem it = claim[c];
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&claim_empty[c]));
            if (++c == kClaims) {
                c = 0;
                cph ^= 1u;
            }
            const uint32_t next = it.num_tiles ? it.pad : (uint32_t)kEngines;
            if (next != engine) {
                if (!wait(&empty_bar[s], ph)) break;
                if (lane == 0) {
                    meta[s] = StageMeta{(run + 1) << 2 | kKindEnd, next, 0, 0};
                    mbar_arrive(smem_addr(&full_bar[s]));
                }
                step_stage();
                // the engine's ring may lie where the last one's table was, and its barriers begin anew
                if (next == kEngines || !wait(&engine_bar, switches++ & 1u)) break;
                engine = next;
                S = prm.stages[engine];
                s = team;
                ph = 1;
                posted = 0;
                run_instance = 0xFFFFFFFFu;   // an engine begins with a run of its own
            }
            const BatchInstanceDev& in = prm.inst[it.instance];
            const uint64_t row0 = (uint64_t)it.first_tile * kBatchTileRows;
            const uint64_t left = in.rows - row0;   // an item has at most flush_rows(engine) rows
            const uint32_t rows = left < it.num_tiles * kBatchTileRows ? (uint32_t)left : it.num_tiles * kBatchTileRows;
            if (it.instance != run_instance || run_rows + rows > flush_rows(engine)) {
                ++run;
                run_instance = it.instance;
                run_rows = 0;
                if (lane == 0) desc[run % kRuns] = Run{in.acc, in.num_groups, in.cutoff};
            }
            run_rows += rows;
            // the team's tiles: every kTeams-th from its next turn on
            const uint32_t full = rows / R, tiles = (rows + R - 1) / R;
            uint32_t t = team >= turn ? team - turn : team + kTeams - turn;
            turn = (turn + tiles) % kTeams;
            const uint8_t* src = in.col[c6] + (row0 + (uint64_t)t * R) * (bytes / R);
            for (; t < full; t += kTeams) {
                if (!(ok = wait(&empty_bar[s], ph))) break;
                const uint32_t fb = smem_addr(&full_bar[s]);
                if (lane == 0) {
                    meta[s].tag = run << 2 | kKindFull;
                    mbar_arrive_expect_tx(fb, kStage);
                }
                __syncwarp();
                if (lane < 6) bulk_g2s(dst + s * kStage, src, bytes, fb, pol);
                src += kTeams * bytes;
                step_stage();
            }
            if (ok && t == full && t < tiles) {   // the instance's last, partial tile
                if (!(ok = wait(&empty_bar[s], ph))) break;
                const uint64_t tile = row0 / R + t;
                if (lane == 0) {
                    meta[s] = StageMeta{run << 2 | kKindPartial, it.instance, (uint32_t)tile,
                                        (rows - full * R) | (uint32_t)(tile >> 32) << 16};
                    mbar_arrive(smem_addr(&full_bar[s]));
                }
                step_stage();
            }
        }
        // never leave with copies in flight: wait for the last fill of each of the team's stages
        for (uint32_t own = S / kTeams, i = posted > own ? posted - own : 0u; i < posted; ++i)
            mbar_wait(smem_addr(&full_bar[team + i % own * kTeams]), i / own & 1u, prm.status);
    } else {
        // ------------------------------ consumers ---------------------------------------
        // The same engines in the same order; each engine's loop keeps only its own table live.
        ka::ConsumerBarrier cb{smem_addr(&consumers_bar), 0};
        uint32_t bad = 0;
        const uint32_t team = warp / kTeamWarps;
        Place at{team, 0, 0};
        for (uint32_t e = first_engine;;) {
            switch (e) {
                case kEngFew: e = consume_engine<kEngFew>(prm, ring, smem, full_bar, empty_bar, meta, runs[team], at, cb, bad); break;
                case kEngCube3: e = consume_engine<kEngCube3>(prm, ring, smem, full_bar, empty_bar, meta, runs[team], at, cb, bad); break;
                case kEngCube: e = consume_engine<kEngCube>(prm, ring, smem, full_bar, empty_bar, meta, runs[team], at, cb, bad); break;
                case kEngSlots: e = consume_engine<kEngSlots>(prm, ring, smem, full_bar, empty_bar, meta, runs[team], at, cb, bad); break;
                default: e = consume_engine<kEngGlobal>(prm, ring, smem, full_bar, empty_bar, meta, runs[team], at, cb, bad); break;
            }
            if (e >= kEngines) break;
            // every team is past its marker: the next engine's table goes where ring or table was
            cb.sync(lane, prm.status);
            if (threadIdx.x == 0) {
                for (uint32_t s = 0; s < kMaxStages; ++s) {
                    mbar_inval(smem_addr(&full_bar[s]));
                    mbar_inval(smem_addr(&empty_bar[s]));
                }
                init_ring();
                fence_mbar_init();
            }
            zero_table(prm, smem, e, threadIdx.x, kWarps * 32);
            fence_proxy_async();   // table words of the last engine before copies into the ring there
            cb.sync(lane, prm.status);
            if (threadIdx.x == 0) mbar_arrive(smem_addr(&engine_bar));
            at.s = team;
            at.ph = 0;
        }
        if (bad && prm.status) atomicOr(prm.status, kStatusDomain);
    }
    __syncthreads();
}

// scratch of every instance -> its int128 table, added to it or (overwrite) stored, empty groups
// too, so that the tables need no zeroing first; one thread per (instance, group).
template <bool kOverwrite>
__global__ void __launch_bounds__(256) q1_batch_finalize(const BatchInstanceDev* __restrict__ inst,
                                                         const uint64_t* __restrict__ group_base, uint32_t ninst,
                                                         uint64_t total_groups) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total_groups) return;
    uint32_t lo = 0, hi = ninst;   // instance with group_base[i] <= t < group_base[i+1]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (group_base[mid] <= t) lo = mid; else hi = mid;
    }
    const BatchInstanceDev& in = inst[lo];
    const uint32_t g = (uint32_t)(t - group_base[lo]);
    const unsigned long long* a = in.acc + 8ull * g;
    unsigned long long* o = in.out + 12ull * g;
    if (!kOverwrite && !a[0]) return;
    auto put = [&](int agg, unsigned __int128 v) {
        if (kOverwrite) {   // 8-byte stores: the tables need no more alignment than the 64-bit atomics do
            o[2 * agg] = (uint64_t)v;
            o[2 * agg + 1] = (uint64_t)(v >> 64);
        } else {
            atomic_add_u128(o + 2 * agg, (uint64_t)v, (uint64_t)(v >> 64));
        }
    };
    put(kAggCount, a[0]);
    put(kAggQty, (unsigned __int128)a[1] * 100u);
    put(kAggBasePrice, a[3]);
    put(kAggDisc, a[2]);
    put(kAggDiscPrice, (unsigned __int128)a[4] + ((unsigned __int128)a[5] << 32));
    put(kAggCharge, (unsigned __int128)a[6] + ((unsigned __int128)a[7] << 32));
}

void batch_tables(const uint32_t max_groups[kEngines], BatchParams& prm) {
    for (uint32_t e = 0; e < kEngines; ++e) {
        const uint32_t bytes = bk::table_bytes(e, max_groups[e]);
        prm.table_words[e] = bytes / 4;
        prm.stages[e] = bk::stages_beside(bytes);
    }
}

cudaError_t batch_prepare_launch() {
    return cudaFuncSetAttribute(q1_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bk::kDynBytes);
}

cudaError_t launch_batch(const BatchParams& prm, cudaStream_t stream) {
    q1_batch_kernel<<<prm.grid, (bk::kWarps + bk::kTeams) * 32, bk::kDynBytes, stream>>>(prm);
    return cudaGetLastError();
}

cudaError_t launch_batch_finalize(const BatchInstanceDev* inst, const uint64_t* group_base, uint32_t ninst,
                                  uint64_t total_groups, bool overwrite, cudaStream_t stream) {
    if (!total_groups) return cudaSuccess;
    const unsigned grid = (unsigned)((total_groups + 255) / 256);
    if (overwrite) q1_batch_finalize<true><<<grid, 256, 0, stream>>>(inst, group_base, ninst, total_groups);
    else q1_batch_finalize<false><<<grid, 256, 0, stream>>>(inst, group_base, ninst, total_groups);
    return cudaGetLastError();
}

}  // namespace q1
