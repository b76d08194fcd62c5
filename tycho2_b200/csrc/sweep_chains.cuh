// Direction chains: the sweep of one direction is a chain of wavefront levels
// that no other direction waits for or feeds, so one block walks one
// direction's levels from first to last with a block barrier between levels.
// One launch per sweep instead of one per level and octant group: a level
// costs a barrier (0.8 us with its upwind loads and solve, taken in turns)
// instead of a launch's hand-off (1.8 us), which is most of the time of a small
// problem.
//
// Records are compact records in (direction, level) order (chain records,
// no padding); off[a * (n_levels + 2) + l] is the first record of direction
// a's level l, with the direction's end repeated from its last level on.
//
// A warp takes 32 tasks (item, VG groups) of a level at a time; the next 32
// tasks' records, in the next level too, are on their way meanwhile: records
// do not depend on psi.  The source is requested and the LU rebuilt before
// the barrier, so what follows a barrier is the upwind loads, the sums, the
// solve and the store.
#pragma once

#include "sweep_block.cuh"

namespace tycho {

// One direction's levels by a block of NT threads.  LEAN: for several blocks
// per SM, two faces' rows live at a time and the LU in the first loads'
// latency; otherwise the LU before the barrier and all four faces at once.
template <typename Real, int VG, bool BLK, int NT, bool LEAN, bool SC = false>
__device__ __forceinline__ void chain_walk(const LevelArgs &p, const CompactRecord<Real> *__restrict__ rec,
                                           const uint32_t *__restrict__ o, const uint32_t n_levels,
                                           RecordStage<Real> &S)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t gpv = p.G / VG;
    // the warp's first task of every level; then every `stride`-th
    const uint32_t w0 = threadIdx.x & ~31u, stride = NT;
    const uint32_t last = o[n_levels];
    auto item_of = [&](uint32_t t) { return gpv == 1u ? t : __umulhi(t, p.vmagic); };
    uint32_t first = 0;  // item of the requested tasks' first one
    auto request = [&](uint32_t base, uint32_t w, uint32_t nt) {
        if (w >= nt) return;
        first = item_of(w);
        S.fill(rec + base + first, item_of(min(w + 31u, nt - 1u)) - first + 1u, lane);
    };
    uint32_t b = o[0], e = o[1];
    request(b, w0, (e - b) * gpv);
    for (uint32_t l = 0; b < last; ++l) {
        const uint32_t e2 = o[l + 2];
        const uint32_t nt = (e - b) * gpv, nt2 = (e2 - e) * gpv;
        RegRecord<Real> R;
        Real q[4][VG];
        uint32_t g = 0;
        bool live = false;
        // the requested record into registers, the warp's next ones on their
        // way, the task's source and factors
        auto take = [&](uint32_t w) {
            S.wait();
            const uint32_t t = w + lane, it = item_of(t);
            live = t < nt;
            if (live) S.take(it - first, R);
            __syncwarp();  // every lane has its record: the stage may be refilled
            if (w + stride < nt) request(b, w + stride, nt);
            else request(e, w0, nt2);
            if (live) {
                g = (t - it * gpv) * VG;
                task_source<Real, VG, BLK>(p, R, g, q);
                if constexpr (!LEAN) compact_factor_nopivot(R);
            }
        };
        if (w0 < nt) take(w0);
        else request(e, w0, nt2);
        if (l) __syncthreads();
        for (uint32_t w = w0; w < nt;) {
            if (live)
                sweep_task<Real, VG, kLoadShared, LEAN, !LEAN, BLK, SC>(p, R, g, [&](Real (&x)[4][VG]) {
#pragma unroll
                    for (int v = 0; v < 4; ++v)
#pragma unroll
                        for (int k = 0; k < VG; ++k) x[v][k] = q[v][k];
                });
            w += stride;
            if (w < nt) take(w);
        }
        b = e;
        e = e2;
    }
}

// The same with the block's warps in two groups that take the levels in
// turn: while one group sweeps a level, the other takes its records, sources
// and factors of the next, so that a level costs a barrier, the upwind loads
// and the solve alone.
template <typename Real, int VG, bool BLK, int NT, bool LEAN, bool SC = false>
__device__ __forceinline__ void chain_walk_turns(const LevelArgs &p, const CompactRecord<Real> *__restrict__ rec,
                                                 const uint32_t *__restrict__ o, const uint32_t n_levels,
                                                 RecordStage<Real> &S)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t gpv = p.G / VG;
    const uint32_t grp = threadIdx.x / (NT / 2), w0 = threadIdx.x % (NT / 2) & ~31u, stride = NT / 2;
    const uint32_t last = o[n_levels];
    auto item_of = [&](uint32_t t) { return gpv == 1u ? t : __umulhi(t, p.vmagic); };
    uint32_t first = 0;  // item of the requested tasks' first one
    auto request = [&](uint32_t base, uint32_t w, uint32_t nt) {
        if (w >= nt) return;
        first = item_of(w);
        S.fill(rec + base + first, item_of(min(w + 31u, nt - 1u)) - first + 1u, lane);
    };
    RegRecord<Real> R;
    Real q[4][VG];
    uint32_t g = 0;
    bool live = false;
    // tasks w of a level's nt: the requested records into registers, the next
    // ones (of this level, else the group's next level) on their way, the
    // sources and factors
    auto take = [&](uint32_t w, uint32_t base, uint32_t nt, uint32_t base2, uint32_t nt2) {
        if (w >= nt) {
            live = false;
            request(base2, w0, nt2);
            return;
        }
        S.wait();
        const uint32_t t = w + lane, it = item_of(t);
        live = t < nt;
        if (live) S.take(it - first, R);
        __syncwarp();  // every lane has its record: the stage may be refilled
        if (w + stride < nt) request(base, w + stride, nt);
        else request(base2, w0, nt2);
        if (live) {
            g = (t - it * gpv) * VG;
            task_source<Real, VG, BLK>(p, R, g, q);
            if constexpr (!LEAN) compact_factor_nopivot(R);
        }
    };
    auto off = [&](uint32_t l) { return o[min(l, n_levels)]; };
    uint32_t b0 = off(0), b1 = off(1), b2 = off(2), b3 = off(3);  // levels l, l + 1, l + 2, l + 3
    if (grp == 0) {
        request(b0, w0, (b1 - b0) * gpv);
        take(w0, b0, (b1 - b0) * gpv, b2, (b3 - b2) * gpv);
    } else {
        request(b1, w0, (b2 - b1) * gpv);
    }
    for (uint32_t l = 0; b0 < last; ++l) {
        const uint32_t b4 = off(l + 4);
        if (l) __syncthreads();
        if (grp == (l & 1u)) {
            const uint32_t nt = (b1 - b0) * gpv;
            for (uint32_t w = w0; w < nt;) {
                if (live)
                    sweep_task<Real, VG, kLoadShared, LEAN, !LEAN, BLK, SC>(p, R, g, [&](Real (&x)[4][VG]) {
#pragma unroll
                        for (int v = 0; v < 4; ++v)
#pragma unroll
                            for (int k = 0; k < VG; ++k) x[v][k] = q[v][k];
                    });
                w += stride;
                if (w < nt) take(w, b0, nt, b2, (b3 - b2) * gpv);
            }
        } else {
            take(w0, b1, (b2 - b1) * gpv, b3, (b4 - b3) * gpv);
        }
        b0 = b1; b1 = b2; b2 = b3; b3 = b4;
    }
}

template <typename Real, int VG, bool BLK, int NT, bool SC = false>
__global__ void __launch_bounds__(NT, 512 / NT)
sweep_turns_kernel(const LevelArgs p, const CompactRecord<Real> *__restrict__ rec, const uint32_t *__restrict__ off,
                   const uint32_t n_levels)
{
    extern __shared__ uint4 chain_smem[];
    pdl_launch_dependents();
    pdl_wait_prerequisites();
    RecordStage<Real> &S = reinterpret_cast<RecordStage<Real> *>(chain_smem)[threadIdx.x >> 5];
    chain_walk_turns<Real, VG, BLK, NT, false, SC>(p, rec, off + (size_t)blockIdx.x * (n_levels + 2), n_levels, S);
}

template <typename Real, int VG, bool BLK, int NT, bool SC = false>
__global__ void __launch_bounds__(NT, 512 / NT)
sweep_chain_kernel(const LevelArgs p, const CompactRecord<Real> *__restrict__ rec, const uint32_t *__restrict__ off,
                   const uint32_t n_levels)
{
    extern __shared__ uint4 chain_smem[];
    pdl_launch_dependents();
    pdl_wait_prerequisites();
    RecordStage<Real> &S = reinterpret_cast<RecordStage<Real> *>(chain_smem)[threadIdx.x >> 5];
    chain_walk<Real, VG, BLK, NT, false, SC>(p, rec, off + (size_t)blockIdx.x * (n_levels + 2), n_levels, S);
}

template <typename Real, int NT>
static const void *turns_fn(const LevelArgs &p)
{
    if constexpr (sizeof(Real) == 4)
        return p.scalar    ? (const void *)sweep_turns_kernel<float, 4, true, NT, true>
               : p.vg == 4 ? (const void *)sweep_turns_kernel<float, 4, true, NT>
               : p.vg == 2 ? (const void *)sweep_turns_kernel<float, 2, true, NT>
                           : (const void *)sweep_turns_kernel<float, 1, true, NT>;
    else
        return p.G == 1    ? (const void *)sweep_turns_kernel<double, 1, true, NT>
               : p.G == 2  ? (const void *)sweep_turns_kernel<double, 2, true, NT>
               : p.vg == 2 ? (const void *)sweep_turns_kernel<double, 2, false, NT>
                           : (const void *)sweep_turns_kernel<double, 1, false, NT>;
}

// One sweep of n_dir directions, one block each.
template <typename Real>
cudaError_t launch_chains(ChainShape sh, const LevelArgs &p, const void *rec, const uint32_t *off, uint32_t n_levels,
                          uint32_t n_dir, cudaStream_t s)
{
    if (n_dir == 0) return cudaSuccess;
    const void *fn = nullptr;
    if (sh.turns)
        fn = sh.threads == 512   ? turns_fn<Real, 512>(p)
             : sh.threads == 256 ? turns_fn<Real, 256>(p)
             : sh.threads == 128 ? turns_fn<Real, 128>(p)
                                 : nullptr;
    else if constexpr (sizeof(Real) == 4)
        if (sh.threads == 512)
            fn = p.scalar    ? (const void *)sweep_chain_kernel<float, 4, true, 512, true>
                 : p.vg == 4 ? (const void *)sweep_chain_kernel<float, 4, true, 512>
                 : p.vg == 2 ? (const void *)sweep_chain_kernel<float, 2, true, 512>
                             : (const void *)sweep_chain_kernel<float, 1, true, 512>;
    if (!fn || p.solver != kSolveNoPivot) return cudaErrorInvalidValue;
    const size_t smem = sizeof(RecordStage<Real>) * (sh.threads / 32);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const CompactRecord<Real> *r = (const CompactRecord<Real> *)rec;
    void *args[] = {(void *)&p, (void *)&r, (void *)&off, (void *)&n_levels};
    // launched while the source kernel ends, and lets the scalar flux's blocks
    // in before it ends itself (both wait for the whole kernel before them):
    // 6^3 S4 65.0 -> 60.9 us an application, 15^3 S6 G=5 FP32 367.6 -> 363.5
    return launch_programmatic(fn, n_dir, sh.threads, smem, args, s);
}

// tasks: (item, group vector) tasks per level and direction on average; the
// whole sweep must fit one wave of blocks.  Measured on B200, sweep in us at
// (tasks, directions), level launches / one group of warps / turns: FP64 one
// block a row (22, 32) 112 / 70 / 45, (38, 32) 159 / 96 / 63, (84, 72) 258 / 167 /
// 114, (84, 128) 350 / 264 / 230, (327, 128) 716 / 694 / 665; FP64 several (84,
// 128) - / 102 / 78, (120, 128) - / 211 / 153, (297, 72) 426 / 526 / 561; FP32 (168,
// 128) 283 / 197 / 189, (252, 72) 247 / 150 / 167, (327, 128) 643-674 / 531-566 /
// 533-607, (640, 72) 352 / 349 / -, (655, 128) 909 / 1044 / 1261.  Up to 64 tasks 256
// threads are as fast as 512 (128 a little slower), and more directions fit.
// Wide FP32 rows: (343, 32) 255 / 281 / -, (343, 8) 234 / 280, (345, 32) 344 / 390,
// (303, 128) 188 / 166, (290, 72) 244 / 226.
inline ChainShape chain_shape_rule(bool fp32, bool one_block, double tasks, int directions, bool wide)
{
    const int sms = device_sm_count();
    ChainShape sh;
    if (tasks <= 64) {
        sh.threads = directions <= 2 * sms ? 256 : directions <= 4 * sms ? 128 : 0;
        sh.turns = true;
    } else if (directions <= sms && tasks <= (wide ? 320 : fp32 ? 450 : one_block ? 340 : 200)) {
        sh.threads = 512;
        sh.turns = !fp32 || tasks <= 170;
    }
    return sh;
}

}  // namespace tycho
