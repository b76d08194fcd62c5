// Batched sweep of many independent instances (uneven mesh size, group
// count and SN order) in one set of launches.  There is no counterpart in
// the reference, which sweeps one problem per process.
//
// Each pass (one operator application of every active member, in one
// precision) is one CUDA graph:
//   plan        device work list over (member, wavefront level): per level,
//               the active members' record ranges as segments with chunk
//               prefixes; per member, its phi chunks
//   accept      phi += delta for members that finished an inner solve
//   scatter     iso = [Q] + M S phi_in                   (per phi element)
//   chains      every direction of every active member walked by one block
//               (sweep_chains.cuh), longest first; the default while no
//               direction outlasts the levels as launches (batch.cpp), else
//   level L     one launch per global level L = 0..max levels - 1: every
//               warp takes IPW-item chunks of the level's work list, finds
//               its member by binary search over the segments, and runs the
//               record kernel's per-(item, group) arithmetic for that member
//   psi->phi    phi_out = sum_a w_a psi
//   post        per member operation (SI change, residual, inner update)
//               with per-chunk partial L1 sums
//   finish      per member: its partials in chunk order -> two norms
// Chunks are member-local (kChunk phi elements of one member), so every
// member's arithmetic and reductions are the same alone and in any mix.
#pragma once

#include "batch_types.hpp"
#include "sweep_chains.cuh"
#include "stream_ops.cuh"

namespace tycho {

constexpr int kBatchPlanThreads = 256;

__device__ __forceinline__ uint32_t batch_class(const BatchSlot &s)
{
    return s.direct ? kDirectClass : s.vg == 4 ? 2u : s.vg == 2 ? 1u : 0u;
}

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t warp_tot[kBatchPlanThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    uint32_t base = 0, all = 0;
    for (uint32_t k = 0; k < kBatchPlanThreads / 32; ++k) {
        if (k < w) base += warp_tot[k];
        all += warp_tot[k];
    }
    __syncthreads();
    *total = all;
    return base + x - v;
}

// Whether a level launch of so many 128-thread blocks is deep: the shallow
// form's blocks (4 per SM) are not resident at once.
inline bool batch_deep(const BatchCuts &cut) { return cut.c[kBatchClasses] > 4u * (unsigned)device_sm_count(); }

// Grid: max levels + 1 blocks of kBatchPlanThreads.  Block L < max levels
// builds level L's segments, one list per vector-width class (members of a
// class run the same kernel body); the last block lists the active members
// and their phi chunk prefix.
template <int IPW>
__global__ void __launch_bounds__(kBatchPlanThreads)
batch_plan_kernel(const BatchSlot *__restrict__ slots, uint32_t n_slots, uint32_t max_levels, uint32_t rec_bytes,
                  BatchPlan pl)
{
    const uint32_t L = blockIdx.x;
    if (L < max_levels) {
        for (uint32_t cls = 0; cls < kBatchClasses; ++cls) {
            uint32_t chunk_run = 0, seg_run = 0;
            BatchSeg *segs = pl.segs + ((size_t)L * kBatchClasses + cls) * pl.seg_stride;
            for (uint32_t base = 0; base < n_slots; base += kBatchPlanThreads) {
                const uint32_t j = base + threadIdx.x;
                uint32_t nch = 0;
                uint64_t lo = 0;
                const uint32_t sh = j < n_slots ? slots[j].level_shift : 0u;
                if (j < n_slots && slots[j].active && L >= sh && L - sh < slots[j].n_levels &&
                    batch_class(slots[j]) == cls) {
                    lo = slots[j].level_off[L - sh];
                    const uint64_t items = slots[j].level_off[L - sh + 1] - lo;
                    // IPW items per chunk; IPW == 0 (direct kernel): 32 (item, group vector) tasks
                    nch = IPW ? (uint32_t)(items / IPW) : (uint32_t)(items / 32 * (slots[j].G / slots[j].vg));
                }
                uint32_t tot_c, tot_s;
                const uint32_t ex_c = block_exclusive_scan(nch, &tot_c);
                const uint32_t ex_s = block_exclusive_scan(nch ? 1u : 0u, &tot_s);
                if (nch) {
                    const BatchSlot &sl = slots[j];
                    BatchSeg sg;
                    sg.rec = (const char *)sl.rec + lo * rec_bytes;
                    sg.psi = sl.psi;
                    sg.iso = sl.iso32 ? (const void *)sl.iso32 : (const void *)sl.iso;
                    sg.item_begin = lo;
                    sg.slot = j;
                    sg.chunk_begin = chunk_run + ex_c;
                    sg.G = sl.G;
                    sg.vmagic = sl.vmagic;
                    sg.solver = sl.solver;
                    sg.zero_row = sl.zero_row;
                    segs[seg_run + ex_s] = sg;
                    pl.seg_first[((size_t)L * kBatchClasses + cls) * pl.seg_stride + seg_run + ex_s] = sg.chunk_begin;
                }
                chunk_run += tot_c;
                seg_run += tot_s;
            }
            if (threadIdx.x == 0) {
                pl.level_nchunk[L * kBatchClasses + cls] = chunk_run;
                pl.level_nseg[L * kBatchClasses + cls] = seg_run;
            }
        }
        return;
    }
    uint32_t chunk_run = 0, act_run = 0;
    for (uint32_t base = 0; base < n_slots; base += kBatchPlanThreads) {
        const uint32_t j = base + threadIdx.x;
        uint32_t nch = 0, on = 0;
        if (j < n_slots && slots[j].active) {
            on = 1;
            const uint64_t n = slots[j].nc * 4 * slots[j].G;
            nch = (uint32_t)((n + kBatchChunk - 1) / kBatchChunk);
        }
        uint32_t tot_c, tot_a;
        const uint32_t ex_c = block_exclusive_scan(nch, &tot_c);
        const uint32_t ex_a = block_exclusive_scan(on, &tot_a);
        if (on) {
            pl.act[act_run + ex_a] = j;
            pl.chunk_prefix[act_run + ex_a] = chunk_run + ex_c;
        }
        chunk_run += tot_c;
        act_run += tot_a;
    }
    if (threadIdx.x == 0) {
        pl.chunk_prefix[act_run] = chunk_run;
        *pl.n_act = act_run;
    }
}

// Largest k in [0, n) with key(k) <= x (key(0) <= x is given).
template <typename KeyFn>
__device__ __forceinline__ uint32_t upper_index(uint32_t n, uint32_t x, KeyFn key)
{
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (key(mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <typename Real>
__device__ __forceinline__ LevelArgs slot_args(const BatchSlot &s)
{
    LevelArgs p = {};
    p.iso = s.iso32 ? (const void *)s.iso32 : (const void *)s.iso;
    p.qang = nullptr;
    p.psi = s.psi;
    p.G = s.G;
    p.vg = s.vg;
    p.vmagic = s.vmagic;
    p.solver = s.solver;
    p.zero_row = s.zero_row;
    return p;
}

// The chunks of one class at one level, taken by this block's warps with a
// stride of the class's block count.  The first chunk's records are staged
// before waiting on the previous level (programmatic dependent launch).
template <typename Real, int IPW, int VG>
__device__ __forceinline__ void batch_class_body(const BatchSlot *__restrict__ slots, const BatchPlan &pl,
                                                 uint32_t L, uint32_t cls, uint32_t blk, uint32_t nblk,
                                                 RecordTile<Real, IPW> &T, bool &waited)
{
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t nchunk = pl.level_nchunk[L * kBatchClasses + cls];
    const uint32_t nseg = pl.level_nseg[L * kBatchClasses + cls];
    const BatchSeg *__restrict__ segs = pl.segs + ((size_t)L * kBatchClasses + cls) * pl.seg_stride;
    for (uint32_t ch = blk * 4u + w; ch < nchunk; ch += nblk * 4u) {
        const uint32_t k = upper_index(nseg, ch, [&](uint32_t m) { return segs[m].chunk_begin; });
        const BatchSeg sg = segs[k];
        const BatchSlot &s = slots[sg.slot];
        const ItemRecord<Real> *rec = (const ItemRecord<Real> *)s.rec;
        tile_fill<Real, IPW>(T, rec + sg.item_begin + (uint64_t)(ch - sg.chunk_begin) * IPW + lane, lane, true);
        if (!waited) {
            pdl_wait_prerequisites();
            waited = true;
        }
        __syncwarp();
        record_pairs<Real, IPW, VG, kLoadPlain>(slot_args<Real>(s), T, lane);
        __syncwarp();
    }
}

// Direct form (compact records rebuilt into registers): chunk = 32 (item,
// group vector) tasks of one member at one level (a level's item count is a
// multiple of 32, so chunks never straddle members), one task per lane.  The
// block stages its class's segments of the level in shared memory before the
// wait on the previous level (up to kBatchSegSmem of them; more are searched
// in global memory), so a warp's member lookup is a shared-memory search.
constexpr uint32_t kBatchSegSmem = 256, kBatchSegWhole = 32;

// One chunk (32 tasks of one member at one level) of the direct form: the
// member's segment found by binary search, its compact record rebuilt in
// registers, the source loaded, then (after `wait`, which the caller uses to
// wait for the previous level) the upwind rows (read as MODE says; of all four
// faces at once) and the solve.
template <typename Real, int VG, bool ANY, int MODE, bool FACTOR, typename Wait>
__device__ __forceinline__ void batch_direct_chunk(const BatchSeg *segs, uint32_t nseg, uint32_t ch, uint32_t lane,
                                                   Wait wait)
{
    const uint32_t k = upper_index(nseg, ch, [&](uint32_t m) { return segs[m].chunk_begin; });
    const BatchSeg &sg = segs[k];
    LevelArgs p = {};
    p.psi = sg.psi;
    p.iso = sg.iso;
    p.G = sg.G;
    p.vg = VG;
    p.vmagic = sg.vmagic;
    p.solver = sg.solver;
    p.zero_row = sg.zero_row;
    const uint32_t gpv = p.G / VG;
    const uint32_t task = (ch - sg.chunk_begin) * 32u + lane;
    const uint32_t itl = gpv == 1u ? task : __umulhi(task, p.vmagic);
    const uint32_t g = (task - itl * gpv) * VG;
    RegRecord<Real> R;
    // NoPivot: the LU is rebuilt after the first upwind loads are issued, in
    // their latency; FACTOR false: with the record, before them.
    constexpr bool kLate = !ANY && FACTOR;
    if constexpr (kLate) load_compact_raw((const CompactRecord<Real> *)sg.rec + itl, R);
    else load_record((const CompactRecord<Real> *)sg.rec + itl, R, ANY ? p.solver : (uint32_t)kSolveNoPivot);
    const bool live = R.u(0) != kSentinel;
    PairIn<Real, VG> in;
    if (live) pair_load_source<Real, VG>(p, R, g, in);
    wait();
    if (!live) return;
    if constexpr (ANY) {
        pair_load_upwind<Real, VG, MODE>(p, R, g, in);
        pair_solve_store_any<Real, VG, RegRecord<Real>, ANY>(p, R, g, in);
    } else {
        auto source = [&](Real (&q)[4][VG]) {
#pragma unroll
            for (int v = 0; v < 4; ++v)
#pragma unroll
                for (int e = 0; e < VG; ++e) q[v][e] = in.q[v][e];
        };
        sweep_task<Real, VG, MODE, FACTOR, true, false>(p, R, g, source);
    }
}

// The same chunk in the default form (NoPivot; sweep_block.cuh): the records
// copied by the warp as one run, FP32 rows as blocks (slot.blk), FP64 rows as
// blocks when they hold one vector of groups.  DEEP as there.
template <typename Real, int VG, bool BLK, bool DEEP, typename Wait>
__device__ __forceinline__ void batch_block_chunk(const BatchSeg &sg, uint32_t ch, uint32_t lane,
                                                  RecordStage<Real> &S, Wait wait)
{
    LevelArgs p = {};
    p.psi = sg.psi;
    p.iso = sg.iso;
    p.G = sg.G;
    p.vg = VG;
    p.vmagic = sg.vmagic;
    p.zero_row = sg.zero_row;
    const uint32_t gpv = p.G / VG;
    auto item_of = [&](uint32_t t) { return gpv == 1u ? t : __umulhi(t, p.vmagic); };
    const uint32_t w = (ch - sg.chunk_begin) * 32u, first = item_of(w), it = item_of(w + lane);
    const uint32_t g = (w + lane - it * gpv) * VG;
    S.fill((const CompactRecord<Real> *)sg.rec + first, item_of(w + 31u) - first + 1u, lane);
    S.wait();
    RegRecord<Real> R;
    S.take(it - first, R);
    __syncwarp();  // every lane has its record: the stage may be refilled
    const bool live = R.u(0) != kSentinel;
    Real q[4][VG];
    if (live) {
        task_source<Real, VG, BLK>(p, R, g, q);
        if constexpr (!DEEP) compact_factor_nopivot(R);
    }
    wait();
    if (live)
        sweep_task<Real, VG, kLoadPlain, DEEP, !DEEP || sizeof(Real) == 8, BLK>(p, R, g, [&](Real (&x)[4][VG]) {
#pragma unroll
            for (int v = 0; v < 4; ++v)
#pragma unroll
                for (int e = 0; e < VG; ++e) x[v][e] = q[v][e];
        });
}

// Stages a (level, class) list of segments in shared memory when it fits
// (block-wide); returns the list to search.
__device__ __forceinline__ const BatchSeg *batch_stage_segs(const BatchPlan &pl, uint32_t L, uint32_t cls,
                                                            BatchSeg *sseg, uint32_t &nseg)
{
    nseg = pl.level_nseg[L * kBatchClasses + cls];
    const BatchSeg *gsegs = pl.segs + ((size_t)L * kBatchClasses + cls) * pl.seg_stride;
    const bool staged = nseg <= kBatchSegSmem;
    if (staged)
        for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) sseg[i] = gsegs[i];
    __syncthreads();
    return staged ? sseg : gsegs;
}

// The chunks of one class at one level, taken by this block's warps with a
// stride of the class's block count.  Before the wait on the previous level
// a few segments (kBatchSegWhole) are staged whole in shared memory; of more
// only the first chunks (up to kBatchSegSmem, beyond that they are searched in
// global memory), and the segment found is read from global memory, where the
// blocks of an SM share it in L1.
// DIRECT: the members of class kDirectClass.
template <typename Real, int VG, bool ANY, bool DEEP, bool DIRECT>
__device__ __forceinline__ void batch_level_body(const BatchPlan &pl, uint32_t L, uint32_t cls, uint32_t blk,
                                                 uint32_t nblk, BatchSeg *sseg, RecordStage<Real> &S, bool &waited)
{
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t at = L * kBatchClasses + cls;
    const uint32_t nchunk = pl.level_nchunk[at], nseg = pl.level_nseg[at];
    const BatchSeg *segs = pl.segs + (size_t)at * pl.seg_stride;
    const uint32_t *gfirst = pl.seg_first + (size_t)at * pl.seg_stride;
    uint32_t *sfirst = reinterpret_cast<uint32_t *>(sseg);
    const bool whole = nseg <= kBatchSegWhole, staged = nseg <= kBatchSegSmem;
    if (whole)
        for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) sseg[i] = segs[i];
    else if (staged)
        for (uint32_t i = threadIdx.x; i < nseg; i += blockDim.x) sfirst[i] = gfirst[i];
    __syncthreads();
    const uint32_t *begin = staged ? sfirst : gfirst;
    auto wait = [&] {
        if (!waited) {
            pdl_wait_prerequisites();
            waited = true;
        }
    };
    for (uint32_t ch = blk * 4u + w; ch < nchunk; ch += nblk * 4u) {
        const BatchSeg &sg =
            whole ? sseg[upper_index(nseg, ch, [&](uint32_t m) { return sseg[m].chunk_begin; })]
                  : segs[upper_index(nseg, ch, [&](uint32_t m) { return begin[m]; })];
        if constexpr (ANY || DIRECT) batch_direct_chunk<Real, VG, ANY, kLoadPlain, true>(&sg, 1, ch, lane, wait);
        else if (sizeof(Real) == 4 || sg.G == VG) batch_block_chunk<Real, VG, true, DEEP>(sg, ch, lane, S, wait);
        else batch_block_chunk<Real, VG, false, DEEP>(sg, ch, lane, S, wait);
    }
}

// ANY: some member solves with Original or a Cramer solver (each member's
// own p.solver); otherwise every member uses NoPivot.
// DEEP: more tasks than are resident at once (FP64: always, its shallow form
// spills at 128 registers).  MINB: blocks per SM the
// register allocation must allow (NoPivot: 4, at most 128 registers; FP32 deep
// launches 5, at most 96).
// SET: the classes it may meet, 1 those by vector width, 2 the direct one, 3 both
// (together they take each other's registers).
template <typename Real, bool ANY, int MINB = 1, bool DEEP = true, int SET = 1>
__global__ void __launch_bounds__(128, MINB)
batch_direct_level_kernel(const BatchSlot *__restrict__ slots, BatchPlan pl, uint32_t L, BatchCuts cut)
{
    __shared__ BatchSeg sseg[kBatchSegWhole];
    static_assert(sizeof(sseg) >= sizeof(uint32_t) * kBatchSegSmem, "first chunks fit the staged segments' space");
    constexpr bool kStaged = !ANY && (SET & 1);
    __shared__ RecordStage<Real> stages[kStaged ? 4 : 1];
    RecordStage<Real> &S = stages[kStaged ? threadIdx.x >> 5 : 0];
    pdl_launch_dependents();
    bool waited = false;
    const uint32_t b = blockIdx.x;
    if ((SET & 2) && (SET == 2 || b >= cut.c[kDirectClass])) {
        constexpr int kVG = sizeof(Real) == 4 ? 4 : 2;
        batch_level_body<Real, kVG, ANY, DEEP, true>(pl, L, kDirectClass, b - cut.c[kDirectClass],
                                                     cut.c[kDirectClass + 1] - cut.c[kDirectClass], sseg, S, waited);
    } else if constexpr (SET & 1) {
        if (b < cut.c[1])
            batch_level_body<Real, 1, ANY, DEEP, false>(pl, L, 0, b, cut.c[1], sseg, S, waited);
        else if (b < cut.c[2])
            batch_level_body<Real, 2, ANY, DEEP, false>(pl, L, 1, b - cut.c[1], cut.c[2] - cut.c[1], sseg, S, waited);
        else if constexpr (sizeof(Real) == 4)
            batch_level_body<Real, 4, ANY, DEEP, false>(pl, L, 2, b - cut.c[2], cut.c[3] - cut.c[2], sseg, S, waited);
    }
    if (!waited) pdl_wait_prerequisites();
    (void)slots;
}

// The NoPivot level kernel for the classes with blocks at this level.
template <typename Real>
const void *batch_level_fn(const BatchCuts &cut)
{
    constexpr bool f = sizeof(Real) == 4;
    const bool direct = cut.c[kDirectClass + 1] > cut.c[kDirectClass], others = cut.c[kDirectClass] > 0;
    if (direct && !others) return (const void *)batch_direct_level_kernel<Real, false, 4, true, 2>;
    if constexpr (f) {
        if (direct) return (const void *)batch_direct_level_kernel<Real, false, 4, false, 3>;
        return batch_deep(cut) ? (const void *)batch_direct_level_kernel<Real, false, 5, true, 1>
                               : (const void *)batch_direct_level_kernel<Real, false, 4, false, 1>;
    } else {
        return direct ? (const void *)batch_direct_level_kernel<Real, false, 4, true, 3>
                      : (const void *)batch_direct_level_kernel<Real, false, 4, true, 1>;
    }
}

template <typename Real, int VG, bool BLK, int NT, bool LEAN>
__device__ __forceinline__ void batch_walk(const BatchSlot &s, const LevelArgs &p,
                                           const CompactRecord<Real> *__restrict__ rec,
                                           const uint32_t *__restrict__ o, RecordStage<Real> &S)
{
    if (s.turns) chain_walk_turns<Real, VG, BLK, NT, LEAN>(p, rec, o, s.n_levels, S);
    else chain_walk<Real, VG, BLK, NT, LEAN>(p, rec, o, s.n_levels, S);
}

// The chains of a pass: block b walks chain table[b] = (slot, direction), the
// longest first; nothing to do for a member that the pass leaves out.
template <typename Real, int NT, int MINB, bool LEAN>
__global__ void __launch_bounds__(NT, MINB)
batch_chain_kernel(const BatchSlot *__restrict__ slots, const uint2 *__restrict__ table)
{
    extern __shared__ uint4 chain_smem[];
    RecordStage<Real> &S = reinterpret_cast<RecordStage<Real> *>(chain_smem)[threadIdx.x >> 5];
    const uint2 t = table[blockIdx.x];
    const BatchSlot &s = slots[t.x];
    if (!s.active) return;
    const LevelArgs p = slot_args<Real>(s);
    const CompactRecord<Real> *rec = (const CompactRecord<Real> *)s.rec;
    const uint32_t *o = s.chain_off + (size_t)t.y * (s.n_levels + 2);
    if constexpr (sizeof(Real) == 4) {
        if (p.vg == 4) batch_walk<Real, 4, true, NT, LEAN>(s, p, rec, o, S);
        else if (p.vg == 2) batch_walk<Real, 2, true, NT, LEAN>(s, p, rec, o, S);
        else batch_walk<Real, 1, true, NT, LEAN>(s, p, rec, o, S);
    } else {
        if (p.G == 1) batch_walk<Real, 1, true, NT, LEAN>(s, p, rec, o, S);
        else if (p.G == 2) batch_walk<Real, 2, true, NT, LEAN>(s, p, rec, o, S);
        else if (p.vg == 2) batch_walk<Real, 2, false, NT, LEAN>(s, p, rec, o, S);
        else batch_walk<Real, 1, false, NT, LEAN>(s, p, rec, o, S);
    }
}

template <typename Real>
cudaError_t batch_chain_launch(int nt, const BatchSlot *slots, const uint2 *table, unsigned n, cudaStream_t s)
{
    constexpr bool f = sizeof(Real) == 4;
    const void *fn = nt == 512   ? (const void *)batch_chain_kernel<Real, 512, 1, false>
                     : nt == 256 ? (const void *)batch_chain_kernel<Real, 256, f ? 3 : 2, f>
                                 : nullptr;
    if (!fn) return cudaErrorInvalidValue;
    if (n == 0) return cudaSuccess;
    const size_t smem = sizeof(RecordStage<Real>) * (nt / 32);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    void *args[] = {(void *)&slots, (void *)&table};
    return cudaLaunchKernel(fn, dim3(n), dim3(nt), args, smem, s);
}

// Persistent form of a pass's wavefront: one cooperative launch walks every
// global level.  Within a level, for each vector-width class, the warps take
// chunks from a device work queue (one counter per level and class, zeroed
// before the launch) until the level's chunks run out; then every block
// meets at a bounded grid barrier before the next level.  The per-chunk
// arithmetic is the level kernels' (bit-identical results); upwind rows are
// read around L1, since other SMs wrote them during this launch.
template <typename Real, int VG, bool ANY>
__device__ __noinline__ void batch_persist_class(const BatchPlan &pl, const BatchPersistArgs &a, uint32_t L,
                                                    uint32_t cls, BatchSeg *sseg)
{
    const uint32_t nchunk = pl.level_nchunk[L * kBatchClasses + cls];
    if (nchunk == 0) return;  // the same for every thread of the block
    uint32_t nseg;
    const BatchSeg *segs = batch_stage_segs(pl, L, cls, sseg, nseg);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t *q = a.queue + L * kBatchClasses + cls;
    for (;;) {
        uint32_t ch = 0;
        if (lane == 0) ch = atomicAdd(q, 1u);
        ch = __shfl_sync(0xffffffffu, ch, 0);
        if (ch >= nchunk) break;
        // all four faces at once, so that a chunk waits for the L2 once after its
        // record; FP32 with the LU before them.  Pass of 256 uneven members by pairs
        // of faces / so: FP32 58.2 / 49.4 ms, FP64 62.0 / 50.0 (51-65 from run to
        // run); FP64 with the LU first 61.5, 24 members 3.99 / 3.96 and 4.65.
        constexpr bool f = sizeof(Real) == 4;
        batch_direct_chunk<Real, VG, ANY, kLoadL2, !f>(segs, nseg, ch, lane, [] {});
    }
    __syncthreads();  // the segment list is restaged for the next class
}

template <typename Real, bool ANY, int MINB = 1>
__global__ void __launch_bounds__(128, MINB)
batch_persist_kernel(const BatchSlot *__restrict__ slots, BatchPlan pl, BatchPersistArgs a)
{
    __shared__ BatchSeg sseg[kBatchSegSmem];
    for (uint32_t L = 0; L < a.max_levels; ++L) {
        batch_persist_class<Real, 1, ANY>(pl, a, L, 0, sseg);
        batch_persist_class<Real, 2, ANY>(pl, a, L, 1, sseg);
        if constexpr (sizeof(Real) == 4) batch_persist_class<Real, 4, ANY>(pl, a, L, 2, sseg);
        if (L + 1 < a.max_levels &&
            !grid_barrier(a.barrier, (unsigned long long)(L + 1) * gridDim.x, a.df, L))
            return;
    }
    (void)slots;
}

// One global level of the batched sweep, 4 warps per block, IPW items per
// chunk.  Blocks [cut[c], cut[c+1]) serve vector-width class c (1, 2, 4
// groups per access), so each block runs one kernel body.  The work list was
// built by the plan kernel, which completed before the first level started.
template <typename Real, int IPW>
__global__ void __launch_bounds__(128)
batch_level_kernel(const BatchSlot *__restrict__ slots, BatchPlan pl, uint32_t L, BatchCuts cut)
{
    __shared__ RecordTile<Real, IPW> tiles[4];
    pdl_launch_dependents();
    RecordTile<Real, IPW> &T = tiles[threadIdx.x >> 5];
    bool waited = false;
    const uint32_t b = blockIdx.x;
    if (b < cut.c[1]) {
        batch_class_body<Real, IPW, 1>(slots, pl, L, 0, b, cut.c[1], T, waited);
    } else if (b < cut.c[2]) {
        batch_class_body<Real, IPW, 2>(slots, pl, L, 1, b - cut.c[1], cut.c[2] - cut.c[1], T, waited);
    } else if constexpr (sizeof(Real) == 4) {
        batch_class_body<Real, IPW, 4>(slots, pl, L, 2, b - cut.c[2], cut.c[3] - cut.c[2], T, waited);
    }
    if (!waited) pdl_wait_prerequisites();
}

}  // namespace tycho

namespace tycho {

// Cooperative launch of the persistent form with as many blocks as can be
// resident at once.
template <typename Real, bool ANY, int MINB>
cudaError_t batch_persist_launch(const BatchSlot *slots, const BatchPlan &pl, const BatchPersistArgs &a,
                                 cudaStream_t s)
{
    const void *fn = (const void *)batch_persist_kernel<Real, ANY, MINB>;
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 128, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(per_sm * sms));
    cfg.blockDim = dim3(128);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BatchPlan plc = pl;
    BatchPersistArgs ac = a;
    void *args[] = {(void *)&slots, (void *)&plc, (void *)&ac};
    return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace tycho
