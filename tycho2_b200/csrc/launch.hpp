// Host-safe declarations of the wavefront launch (no device code): the
// per-level argument block and the launcher, instantiated for double (in
// device_ops.cu, FMA contraction off) and float (sweep_f32.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace tycho {

// The 4x4 solvers of gaussElim4 (deck key GaussElim, src/Global.hh:99-105),
// numbered as tycho_gauss_elim.  Each one factors the group-independent
// matrix once per item into 16 numbers (and, for Original, a row order) and
// applies them to every group's right-hand side in the reference's order.
enum SolveKind : uint32_t { kSolveOriginal = 0, kSolveNoPivot = 1, kSolveCramerGlu = 2, kSolveCramerIntel = 3 };

struct LevelArgs {
    const uint32_t *items;   // cell*A + angle, level-sorted
    const void *abar;        // Real4 per item: face area * omega.n, faces 0..3
    const int4 *adj;         // per cell: neighbour across face f, -1 on the boundary
    const uint32_t *nbrmap;  // per cell: 2 bits per (face f, vertex j): neighbour's vertex at j
    const void *cellk;       // Real[3] per cell: V/20, sigma_t V/20, 2 sigma_t V/20
    const void *iso;         // Real, phi layout: isotropic total source (nullable)
    const double *qang;      // angular source, psi layout, FP64 only (nullable)
    void *psi;               // Real, psi layout
    uint32_t A, G;
    uint32_t gmagic;         // ceil(2^32 / G): pair -> item in the warp-tile variant (0 when G == 1)
    uint32_t vg;             // record variant: groups per vector access (divides G)
    uint32_t vmagic;         // ceil(2^32 / (G / vg)): task -> item (0 when G == vg)
    uint32_t solver;         // 4x4 solver (deck key GaussElim), numbered as tycho_gauss_elim
    uint32_t zero_row;       // psi row of zeros (in rows of the sweep's precision)
    uint32_t scalar;         // default FP32 form: group by group, not packed (an odd group count)
};

// Record variant's group vector width: 16-byte accesses where G allows.
constexpr uint32_t record_vg(bool fp32, uint32_t G)
{
    return fp32 ? (G % 4 == 0 ? 4 : (G % 2 == 0 ? 2 : 1)) : (G % 2 == 0 ? 2 : 1);
}

// Per-sweep state of the persistent (dataflow) schedule.
struct DataflowArgs {
    uint32_t *done;       // per cell*A + angle: epoch of the sweep that finished it
    uint32_t *err;        // [0] error code (0 = none), [1] item, [2] face
    uint32_t *abort;      // raised on the first failure; every warp drains
    const uint32_t *epoch;  // device word: this sweep's epoch (never 0)
    uint64_t n_items;     // padded item count, a multiple of 32
    uint32_t spin_limit;  // polls of one upwind flag before giving up
};
constexpr uint32_t kErrTimeoutCode = 1;

// Launches the wavefront kernel over items [begin, end) with `tpi` threads
// per item (1, 2, 4, 8 or 16).
template <typename Real>
cudaError_t launch_level(int tpi, const LevelArgs &p, uint64_t begin, uint64_t end, cudaStream_t s);

// The whole sweep as one cooperative launch of `grid` 256-thread blocks
// (at most the co-resident count from dataflow_blocks_per_sm).
template <typename Real>
cudaError_t launch_dataflow(int tpi, const LevelArgs &p, const DataflowArgs &df, unsigned grid,
                            cudaStream_t s);
template <typename Real>
cudaError_t dataflow_blocks_per_sm(int tpi, int *blocks);

// Warp-tile variant (sweep_tiles.cuh): 32 items per warp, `wpb` warps per
// block (1, 2 or 4); same contracts as the launchers above.
template <typename Real>
cudaError_t launch_level_tile(int wpb, const LevelArgs &p, uint64_t begin, uint64_t end, cudaStream_t s);
template <typename Real>
cudaError_t launch_dataflow_tile(int wpb, const LevelArgs &p, const DataflowArgs &df, unsigned grid,
                                 cudaStream_t s);
template <typename Real>
cudaError_t tile_dataflow_blocks_per_sm(int wpb, int *blocks);

// Record variant (sweep_records.cuh): per-item factors precomputed once per
// cross-section set into `rec` (128 B per item for float, 256 B for double).
constexpr size_t record_bytes(bool fp32) { return fp32 ? 128 : 256; }
template <typename Real>
cudaError_t launch_item_records(const LevelArgs &p, uint64_t n, void *rec, cudaStream_t s);
template <typename Real>
cudaError_t launch_level_record(int wpb, const LevelArgs &p, const void *rec, uint64_t begin, uint64_t end,
                                cudaStream_t s);
template <typename Real>
cudaError_t launch_dataflow_record(int wpb, const LevelArgs &p, const void *rec, const DataflowArgs &df,
                                   unsigned grid, cudaStream_t s);
template <typename Real>
cudaError_t record_dataflow_blocks_per_sm(int ipw, int vg, int *blocks);
// Direct record variant (level schedule only): one thread per (item, group
// vector), `bs` threads per block (64, 128 or 256).
template <typename Real>
cudaError_t launch_direct_level(int bs, const LevelArgs &p, const void *rec, uint64_t begin, uint64_t end,
                                cudaStream_t s, bool compact);
// Direct variants on the dataflow schedule: one cooperative launch, a
// completion flag per (item, group vector) in df.done (n_cells * A * G/vg
// words, G/vg a power of two <= 32).
template <typename Real>
cudaError_t launch_direct_dataflow(const LevelArgs &p, const void *rec, bool compact, const DataflowArgs &df,
                                   unsigned grid, cudaStream_t s);
template <typename Real>
cudaError_t direct_dataflow_blocks_per_sm(int vg, bool compact, int *blocks);
// Direct kernel (compact records, NoPivot, p.vg 1 or 2) over the schedule
// positions pos[begin, end).
template <typename Real>
cudaError_t launch_direct_subset(const LevelArgs &p, const void *rec, const uint32_t *pos, uint64_t begin,
                                 uint64_t end, cudaStream_t s);
// Compact records (64 B per item for float, 112 B for double): the inputs of
// each item's matrix, from which the direct kernels rebuild its factors.
constexpr size_t compact_record_bytes(bool fp32) { return fp32 ? 64 : 112; }
template <typename Real>
cudaError_t launch_compact_records(const LevelArgs &p, uint64_t n, const uint32_t *pos, void *rec, cudaStream_t s);
// The default level kernel (sweep_block.cuh): compact records, NoPivot.  FP64:
// p.vg = record_vg, rows as they are.  FP32: rows (psi, and the source p.iso) are
// kept as blocks of p.vg groups, p.G groups in all.
template <typename Real>
cudaError_t launch_block_level(const LevelArgs &p, const void *rec, uint64_t begin, uint64_t end, cudaStream_t s);
// How the default form keeps FP32 rows: blocks of record_vg groups, or (pad) of
// 4 with the last one padded.
struct BlockRows {
    uint32_t vg, groups;
    constexpr BlockRows(uint32_t G = 1, bool pad = false)
        : vg(pad ? 4 : record_vg(true, G)), groups(pad ? (G + 3) / 4 * 4 : G)
    {
    }
};
// Batched passes: blocks of record_vg groups, never padded (0: the plain row).
constexpr uint32_t block_width(uint32_t G) { return record_vg(true, G) == G ? 0u : record_vg(true, G); }
// Batched level launches: whether a member's rows stay plain with each thread
// loading its record itself, instead of blocks and records by the warp's stage.
// FP64 rows of several pairs (which are no blocks either way): pass in ms, staged /
// direct, one 24^3 S4 member of 8 / 4 groups 1.14 / 1.08 and 0.905 / 0.837, four of 8
// 3.29 / 3.05, one 24^3 S8 G=16 5.73 / 5.25; rows that are one block 28^3 S4 G=1 0.73 /
// 0.99.
// FP32 rows of three and more blocks: a face of four takes 32 lines of a warp's accesses as
// blocks (two of 32 bytes a task), 24 plain (three of 16, the tasks of an item side
// by side), of two blocks 32 and 48; two 24^3 S2 G=16 members 1.13 / 0.98, one 24^3 S4
// G=16 1.18 / 1.06, one 24^3 S4 G=12 1.12 / 1.06; of two blocks 24^3 S6 G=8 1.14 / 1.18.
constexpr bool level_direct(bool fp32, uint32_t G)
{
    return fp32 ? record_vg(true, G) == 4 && G >= 12 : record_vg(false, G) == 2 && G >= 4;
}
// Direction chains (sweep_chains.cuh): one sweep of n_dir directions of the
// chain records, each walked by one block; off: n_levels + 2 record offsets
// per direction.  Rows as in the default level kernel.
struct ChainShape {
    int threads = 0;     // of a direction's block (0: level launches instead)
    bool turns = false;  // its warps in two groups that take the levels in turn
};
template <typename Real>
cudaError_t launch_chains(ChainShape sh, const LevelArgs &p, const void *rec, const uint32_t *off, uint32_t n_levels,
                          uint32_t n_dir, cudaStream_t s);
// The default form of a problem with so many tasks per level and direction;
// one_block: rows of one block; wide: FP32 rows of three and more blocks of 4.
ChainShape chain_shape(bool fp32, bool one_block, double tasks, int directions, bool wide = false);
// Persistent levels: one cooperative launch, a bounded grid barrier between
// levels (level_off: device copy of the n_levels + 1 level offsets).
template <typename Real>
cudaError_t launch_persist_record(int ipw, const LevelArgs &p, const void *rec, const uint64_t *level_off,
                                  uint32_t n_levels, unsigned long long *barrier, const DataflowArgs &df,
                                  unsigned grid, cudaStream_t s);
template <typename Real>
cudaError_t record_persist_blocks_per_sm(int ipw, int vg, int *blocks);

}  // namespace tycho
