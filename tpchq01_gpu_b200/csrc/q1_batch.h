// Internal interface of the batched (persistent, work-queue) aggregation.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace q1 {

constexpr uint32_t kBatchTileRows = 2048;
constexpr uint32_t kBatchMaxItemTiles = 4096;   // 2^23 rows: what a table takes between flushes
constexpr uint32_t kBatchMaxFewItemTiles = 1023;   // and what the one of few groups does

// Placement of one instance inside the batch kernel.
enum BatchMode : uint32_t {
    kModeShared = 1,      // shared-memory table: cells for <= 1024 groups, else slots for keys < 2048
                          // with the rest spilled to scratch
    kModeGlobal = 2,      // reductions straight into scratch
};

struct BatchInstanceDev {
    const uint8_t* col[6];        // ship, qty, disc, tax, price, key (16-byte aligned, device)
    uint64_t rows;
    int32_t cutoff;               // cutoff_day - 727563, clamped to [-1, 32767]
    uint32_t num_groups;
    uint32_t mode;                // BatchMode
    uint32_t pad;
    unsigned long long* acc;      // scratch: num_groups x 8 u64
    unsigned long long* out;      // caller's int128 table [num_groups][6][lo, hi]
};

struct BatchItem {
    uint32_t instance;
    uint32_t first_tile;
    uint32_t num_tiles;
    uint32_t pad;
};

// Engine that aggregates an instance inside the batch kernel (q1_keyagg.cuh).
enum BatchEngine : uint32_t {
    kEngFew = 0,         // (group, discount, tax) cells and slots by lane, <= 4 groups
    kEngCube3 = 1,       // (group, discount, tax) cells, <= 64 groups
    kEngCube = 2,        // (group, discount) cells, <= 1024 groups
    kEngSlots = 3,       // slots for keys < 2048, larger keys spilled
    kEngGlobal = 4,      // straight into scratch
    kEngines = 5,
};
uint32_t batch_engine(uint32_t mode, uint32_t num_groups);

struct BatchParams {
    const BatchInstanceDev* inst;
    const BatchItem* items;             // grouped by engine: [item_begin[e], item_begin[e + 1])
    uint32_t item_begin[kEngines + 1];
    uint32_t role_end[kEngines];        // CTAs [role_end[e-1], role_end[e]) start with queue e
    uint32_t grid;                      // CTAs
    uint32_t stages[kEngines];          // ring stages beside the engine's table
    uint32_t table_words[kEngines];     // the table of the engine's largest instance, in 32-bit words
    uint32_t* cursor;                   // kEngines claim counters, zeroed before every launch
    uint32_t* status;
};

// Cuts every instance (host descriptors) into items of at most `chunk` tiles (0: of falling size, see
// plan_items), groups them by engine (largest first inside an engine) and splits at most `grid` CTAs among the
// queues in proportion to estimated cost.
void batch_plan(const BatchInstanceDev* inst, uint32_t n, uint32_t chunk, uint32_t grid, std::vector<BatchItem>& items,
                BatchParams& prm);

// Table sizes and ring stages, from the most groups an instance of each engine has.
void batch_tables(const uint32_t max_groups[kEngines], BatchParams& prm);
cudaError_t batch_prepare_launch();
cudaError_t launch_batch(const BatchParams& prm, cudaStream_t stream);
// Scratch of every instance into its result table: stored (every group, empty ones too) or added.
cudaError_t launch_batch_finalize(const BatchInstanceDev* inst, const uint64_t* group_base, uint32_t ninst,
                                  uint64_t total_groups, bool overwrite, cudaStream_t stream);

}  // namespace q1
