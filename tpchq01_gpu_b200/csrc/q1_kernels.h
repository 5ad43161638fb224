// Internal interface between the host runtime (C++) and the CUDA kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace q1 {

// Input layouts the scan kernel understands (column order inside a tile in brackets).
enum ScanLayout : int {
    kLayPair = 0,        // [ship u16, qty u8, disc u8, tax u8, price u32, pair code 2b]
    kLayPairFilter = 1,  // [filter 1b, qty, disc, tax, price, pair code 2b]
    kLaySep = 2,         // [ship u16, qty, disc, tax, price, rf 2b, ls 1b]
    kLaySepFilter = 3,   // [filter 1b, qty, disc, tax, price, rf 2b, ls 1b]
    kLayUncomp = 4,      // [ship i32, qty i64, disc i64, tax i64, price i64, rf char, ls char]
    kNumScanLayouts = 5
};

// Table placements (same numbering as q1_placement in include/q1.h).
enum ScanPlacement : int {
    kPlaceInRegisters = 0,
    kPlaceInRegistersPerThread = 1,
    kPlaceLocalMem = 2,
    kPlaceSharedMemPerThread = 3,
    kPlaceGlobal = 4,
};

// Consumer warps per CTA (plus one producer warp), per input layout, as measured on the 600 M-row
// table (100 M uncompressed). More warps per SM sub-partition hide more of the decode's issue latency
// where the registers allow. The register file is given out four warps at a time: 15 consumer warps (or 12:
// 13 warps take the room of 16) leave 128 registers a thread, and the compressed layouts' kernels fit, the
// separate-flag ones by keeping only four groups' planes in registers (A/O and R/O go to the CTA's shared
// table). Separate flags took 1.129 ms with 8 warps and six planes, 1.044 with 10, 0.980 with 12.
// kWide, 15 warps: large tables (scan_is_wide): 600 M rows, pair 871 -> 832 us, separate flags
// 1005 -> 920, with filter 1205 -> 1084; 14 warps 886, 1000, 1156. Their larger tile (a small table is a
// few tiles per CTA) costs 60,175 rows 2 us. The shared placement's tables leave no room for it.
// The uncompressed layout and in_registers over separate flags need up to 168 registers: 11 warps with
// the producer's 12 (10: uncompressed 100 M rows per-thread 582 us instead of 536; the shared
// placement's table again leaves no room).
constexpr bool scan_needs_168(int L, int P) {
    return L == kLayUncomp || ((L == kLaySep || L == kLaySepFilter) && P == kPlaceInRegisters);
}
constexpr bool scan_has_wide(int L, int P) { return !scan_needs_168(L, P) && P != kPlaceSharedMemPerThread; }
template <int L, int P, bool kWide>
inline constexpr uint32_t kConsumerWarps =
    scan_needs_168(L, P) ? (P == kPlaceSharedMemPerThread ? 10u : 11u) : (kWide && scan_has_wide(L, P) ? 15u : 12u);
// Rows of the launch for each CTA it may have from which on a wide kernel runs (148 CTAs: 12 M rows take
// 27.1 us with 12 warps and 28.1 with 15, 25 M rows 46.9 and 45.9; separate flags with filter 35.1 and
// 35.0, 60.9 and 59.1).
inline constexpr uint64_t kWideRowsPerCta = 1u << 17;
constexpr bool scan_is_wide(int L, int P, uint64_t rows, uint32_t ctas) {
    return scan_has_wide(L, P) && rows >= kWideRowsPerCta * ctas;
}
// Rows per tile (one bulk copy per column per tile): a multiple of 128, so that every column slice
// of every tile starts on a 16-byte boundary down to 1-bit columns, and of the consumer threads x
// the rows of a step, so that a tile's steps divide evenly among the consumer threads.
template <int L, int P, bool kWide>
inline constexpr uint32_t kTileRows =
    (L == kLayUncomp ? 128u : 384u) * kConsumerWarps<L, P, kWide>;
// Shared-memory ring depth: 3 where the shared placement's tables take the room of the fourth.
template <int L, int P>
inline constexpr uint32_t kStages = (P == kPlaceSharedMemPerThread && L != kLayPair && L != kLayPairFilter) ? 3u : 4u;
// Tiles a thread sums in registers before its sums go to the table of a placement that keeps it
// elsewhere (12 rows a thread and tile, 4 of the uncompressed layout: 49,152 rows a warp between
// two flushes, a few per warp over 600 M rows). The global placement sets it: 600 M rows (8 warps,
// 4096-row tiles) took 12.94 ms with 1 tile (same-address L2 atomics serialise), 4.05 ms with 4,
// 1.95 ms with 16, 1.22 ms with 64 and 1.08 ms with 128. A 64-bit warp sum bounds the rows a thread
// may buffer (the kernel's static_assert).
#ifndef Q1_COMBINE_TILES
#define Q1_COMBINE_TILES 128
#endif
inline constexpr uint32_t kCombineTiles = Q1_COMBINE_TILES;

struct ScanParams {
    const uint8_t* col[7];      // column base pointers in tile order; 16-byte aligned
    uint64_t rows;              // rows to aggregate (<= 2^31 per launch)
    int32_t cutoff;             // compressed: cutoff_day - 727563; uncompressed: cutoff_day
    uint32_t qty_scale;         // 100 when quantity is stored in whole units, else 1
    uint8_t pair_group[4];      // pair layouts: code -> group
    unsigned long long* out;    // [6 groups][6 aggregates][lo, hi]
    uint32_t* status;           // device status word (kStatus* bits); may be null
    unsigned long long* records;  // null: atomics into `out`. Otherwise each CTA writes its own
                                  // [6][6][lo, hi] record at records[blockIdx.x] and leaves `out`
                                  // alone (used by the allocation-free entry point)
};

// Launch the scan kernel for one layout x placement. max_blocks <= 0: one CTA per SM.
cudaError_t launch_scan(int layout, int placement, const ScanParams& prm, int sm_count, int max_blocks,
                        cudaStream_t stream);
// Rows per tile of the layout x placement's kernel for small tables (a multiple of 128).
uint32_t scan_tile_rows(int layout, int placement);
// Grid size launch_scan uses for `rows` rows of the layout x placement.
uint32_t scan_grid_blocks(int layout, int placement, uint64_t rows, int sm_count, int max_blocks);
// Most rows one launch may take so that no consumer thread adds more than 2^15 rows (which keeps
// its 32-bit and 64-bit partial sums exact) and per-launch sums stay below 2^31 rows.
uint64_t scan_max_rows_per_launch(int layout, int placement, uint32_t grid);

// Group-key aggregation (groupkey_kernels.cu). cols: ship, qty, disc, tax, price, key.
cudaError_t launch_groupkey(int placement, const uint8_t* const cols[6], uint64_t rows, int32_t cutoff_rel,
                            uint32_t num_groups, unsigned long long* scratch, unsigned long long* out,
                            uint32_t* status, int sm_count, int max_blocks, cudaStream_t stream);
uint64_t groupkey_scratch_bytes(uint32_t num_groups);
// High-cardinality path of the shared_mem_per_thread placement (groupkey_part.cu): a radix
// partition by key, then per-partition shared-memory cells. acc: num_groups x 8 u64
// (zeroed by the caller); workspace: groupkey_part_workspace_bytes(), 256-byte aligned. When
// `mode` is set, every kernel of the path returns at once unless *mode == kModePartitioned.
enum GroupKeyMode : uint32_t { kModeSinglePass = 1, kModePartitioned = 2, kModeGlobalPath = 3 };
cudaError_t launch_groupkey_part(const uint8_t* const cols[6], uint64_t rows, int32_t cutoff_rel,
                                 uint32_t num_groups, unsigned long long* acc, uint8_t* workspace,
                                 const uint32_t* mode, uint32_t* status, int sm_count, int max_blocks,
                                 cudaStream_t stream);
uint64_t groupkey_part_workspace_bytes();
// byte offset of a spare word in the workspace (the mode word of launch_groupkey)
uint64_t groupkey_part_mode_offset();
// fewest groups for which the shared placement has the partitioned path
uint32_t groupkey_part_min_groups();
// most chunks of 256 records that `ctas` CTAs reserve for a segment of `rows` rows
uint64_t groupkey_part_max_chunks(uint64_t rows, uint32_t ctas);
cudaError_t launch_generate_keys(uint64_t seed, uint64_t first_row, uint64_t rows, uint32_t num_groups,
                                 const uint32_t* dev_cdf, uint32_t* dev_keys, cudaStream_t stream);

// lineitem text parsing (tbl_kernels.cu). launch_tbl_count: the newlines of the text into *total.
cudaError_t launch_tbl_count(const char* text, uint64_t bytes, unsigned long long* total, int sm_count,
                             cudaStream_t stream);
// What launch_tbl_parse leaves at the start of its scratch (16-byte aligned, tbl_scratch_bytes).
struct alignas(16) TblResult {
    unsigned long long newlines;
    unsigned long long malformed;         // malformed lines and lines past the capacity
    unsigned long long first_malformed;   // ~(byte offset of the first of them), 0 if none
    unsigned long long ticket;            // tiles handed out
    uint32_t last_is_newline;
    uint32_t status;                      // kStatus* bits
};
uint64_t tbl_scratch_bytes(const char* text, uint64_t bytes);
cudaError_t launch_tbl_parse(const char* text, uint64_t bytes, void* scratch, int32_t* ship, int64_t* qty,
                             int64_t* price, int64_t* disc, int64_t* tax, char* rf, char* ls, uint64_t capacity,
                             int sm_count, cudaStream_t stream);

// Utility kernels (util_kernels.cu).
struct GenCompressedOut {
    uint16_t* shipdate;
    uint8_t* discount;
    uint32_t* extendedprice;
    uint8_t* tax;
    uint8_t* quantity;
    uint32_t* flags;        // pair codes (may be null)
    uint32_t* returnflag;   // separate containers (may be null)
    uint32_t* linestatus;
};
cudaError_t launch_generate_compressed(uint64_t seed, uint64_t first_row, uint64_t rows, const GenCompressedOut& out,
                                       cudaStream_t stream);
// One thread waits on an mbarrier nothing completes, bounded by limit_ns; on expiry it records
// kStatusWaitTimeout in *status and returns (the bounded-wait self-test).
cudaError_t launch_wait_selftest(uint64_t limit_ns, uint32_t* status, cudaStream_t stream);
cudaError_t launch_precompute_filter(const uint16_t* shipdate, uint64_t rows, int32_t cutoff_rel, uint32_t* bitmap,
                                     cudaStream_t stream);

}  // namespace q1
