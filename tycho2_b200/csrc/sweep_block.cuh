// The default level kernel: 64-thread blocks, one (item, VG groups) task per
// lane, compact records.
//
// What bounds a level kernel is its dependent loads through the L1, which takes
// the up to 32 different lines of an instruction one after the other: a mid-sweep
// FP32 launch keeps the L1 busy in 48% of the SM's cycles and waits for global
// loads in 8 of 13.6 cycles per instruction; leaving the LU out of a sweep changes
// it by less than 2%, the upwind loads by 30%.  So this kernel makes fewer and
// wider accesses than the direct ones (sweep_records.cuh):
//   * the warp copies its items' records, which are consecutive, as one run
//     into shared memory (8 lines for 16 FP32 records against 32, 7 for 8 FP64
//     records against 49);
//   * BLK: a task's values of a row, four vertices of VG groups, are one
//     contiguous block, read and written by 32-byte accesses (two for 4 FP32
//     groups instead of three per face and four per store; one for 1 or 2
//     FP32 groups or 1 FP64 group).  FP32 psi and source are laid out block
//     by block for it; FP64 rows keep the reference's layout and are blocks
//     when they hold 1 or 2 groups.
// The arithmetic is the direct kernels', task for task.  Measured on B200,
// sweep in us, direct kernel -> this: FP32 32^3 S8 G=8 2062 -> 1833, 24^3 S8
// G=1 / 2 / 4 / 8 784 -> 671, 817 -> 638, 1103 -> 930, 1043 -> 911, 48^3 S8 G=8
// 6929 -> 6339; FP64 32^3 S8 G=8 4139 -> 3984, 24^3 S8 G=1 / 4 862 -> 714, 1137 ->
// 1079.
#pragma once

#include <algorithm>

#include "stream_ops.cuh"
#include "sweep_records.cuh"

namespace tycho {

template <typename Real>
constexpr int kRecordChunks = sizeof(CompactRecord<Real>) / 16;

// A launch whose blocks may start before the kernel before it ends; they wait
// for it (griddepcontrol.wait) before they read or write what it touches.
inline cudaError_t launch_programmatic(const void *fn, unsigned grid, unsigned threads, size_t smem, void **args,
                                       cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

// A warp's stage for the records of 32 consecutive tasks.
template <typename Real>
struct RecordStage {
    static constexpr int N = kRecordChunks<Real>;
    uint4 chunk[32 * N];

    // Slot of chunk k of item i: FP32 records are swizzled so that eight
    // lanes reading one chunk of eight items hit 32 different banks (the
    // 112-byte FP64 records already do).
    static __device__ __forceinline__ uint32_t slot(uint32_t i, uint32_t k)
    {
        return N == 4 ? i * 4u + (k ^ ((i >> 1) & 3u)) : i * (uint32_t)N + k;
    }

    // Requests the n records from `src` on; all lanes of the warp.
    __device__ __forceinline__ void fill(const CompactRecord<Real> *__restrict__ src, uint32_t n, uint32_t lane)
    {
        const uint4 *s = reinterpret_cast<const uint4 *>(src);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const uint32_t c = lane + 32u * j;
            if (c < n * (uint32_t)N) cp_async16(&chunk[N == 4 ? slot(c >> 2, c & 3u) : c], s + c);
        }
    }

    // The requested records are there; all lanes of the warp.
    __device__ __forceinline__ void wait() const
    {
        cp_async_wait_all();
        __syncwarp();
    }

    __device__ __forceinline__ void take(uint32_t i, RegRecord<Real> &R) const
    {
        uint4 v[N];
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = chunk[slot(i, k)];
        compact_raw(v, R);
    }
};

// The task's sources, in the layout its psi has.
template <typename Real, int VG, bool BLK>
__device__ __forceinline__ void task_source(const LevelArgs &p, const RegRecord<Real> &R, uint32_t g, Real (&q)[4][VG])
{
    if constexpr (BLK) {
        const Real *iso = reinterpret_cast<const Real *>(p.iso);
        const uint32_t rowG = 4u * p.G;
        if (sizeof(Real) == 8 && p.qang) {  // angular sources are FP64 only
            block_load<Real, VG>(reinterpret_cast<const Real *>(p.qang) + (uint64_t)R.u(1) * rowG + 4u * g, q);
            if (iso) {
                Real x[4][VG];
                block_load<Real, VG>(iso + (uint64_t)R.u(0) * rowG + 4u * g, x);
#pragma unroll
                for (int v = 0; v < 4; ++v)
#pragma unroll
                    for (int e = 0; e < VG; ++e) q[v][e] = q[v][e] + x[v][e];
            }
        } else if (iso) {
            block_load<Real, VG>(iso + (uint64_t)R.u(0) * rowG + 4u * g, q);
        } else {
#pragma unroll
            for (int v = 0; v < 4; ++v)
#pragma unroll
                for (int e = 0; e < VG; ++e) q[v][e] = Real(0);
        }
    } else {
        PairIn<Real, VG> in;
        pair_load_source<Real, VG>(p, R, g, in);
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
            for (int e = 0; e < VG; ++e) q[v][e] = in.q[v][e];
    }
}

// Blocks per SM that the registers are bound for: deep launches at most 73 /
// 102 registers, shallow ones 128.
template <typename Real, bool DEEP>
constexpr int kBlockMin = DEEP ? (sizeof(Real) == 4 ? 14 : 10) : 8;

// DEEP: the launch has more tasks than the shallow form keeps resident, and
// residency sets its rate: two faces' rows are live at a time and the LU is
// rebuilt after the wait, in the first loads' latency.  A shallow launch
// lasts as long as one task's chain after the wait: its LU is rebuilt before
// it and all four faces' rows are requested at once.
// PF: several resident waves deep (record prefetch).
template <typename Real, int VG, bool BLK, bool DEEP, bool PF, bool SC = false>
__global__ void __launch_bounds__(64, (kBlockMin<Real, DEEP>))
sweep_block_kernel(const LevelArgs p, const CompactRecord<Real> *__restrict__ rec, const uint64_t begin,
                   const uint64_t end)
{
    __shared__ RecordStage<Real> stage[2];
    pdl_launch_dependents();
    const uint32_t gpv = p.G / VG, lane = threadIdx.x & 31u;
    const uint32_t t = blockIdx.x * 64u + threadIdx.x;
    const uint32_t n = (uint32_t)(end - begin);
    auto item_of = [&](uint32_t task) { return gpv == 1u ? task : __umulhi(task, p.vmagic); };
    const uint32_t itl = item_of(t), first = item_of(t - lane);
    const uint32_t g = (t - itl * gpv) * VG;
    bool live = itl < n;
    RegRecord<Real> R;
    Real q[4][VG];
    if constexpr (PF) prefetch_record_ahead<CompactRecord<Real>, 64, kBlockMin<Real, DEEP>>(rec, t, gpv, p.vmagic, begin, end);
    if (first < n) {  // the same for the whole warp
        RecordStage<Real> &S = stage[threadIdx.x >> 5];
        S.fill(rec + begin + first, min(item_of(t - lane + 31u), n - 1u) - first + 1u, lane);
        S.wait();
        if (live) {
            S.take(itl - first, R);
            live = R.u(0) != kSentinel;
        }
        if (live) {
            task_source<Real, VG, BLK>(p, R, g, q);
            if constexpr (!DEEP) compact_factor_nopivot(R);
        }
    }
    pdl_wait_prerequisites();
    if (!live) return;
    sweep_task<Real, VG, kLoadPlain, DEEP, !DEEP, BLK, SC>(p, R, g, [&](Real (&x)[4][VG]) {
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
            for (int e = 0; e < VG; ++e) x[v][e] = q[v][e];
    });
}

// Deep FP64 launches of rows of four and more group vectors: as many blocks as
// are resident at 128 registers, each warp walking several runs of 32 tasks
// with the next run's records on their way and all four faces' rows in flight.
// Sweep in us, without -> with: 32^3 S8 G=8 3950 -> 3800, 24^3 S8 G=12 2490 -> 2390,
// 28^3 S6 G=16 2876 -> 2837; fewer vectors are slower this way (24^3 S8 G=4 1075 ->
// 1107, 40^3 S8 G=2 3360 -> 3508), and so is FP32 (32^3 S8 G=8 1831 -> 1972 at best).
template <typename Real, int VG, bool BLK>
__global__ void __launch_bounds__(64, (kBlockMin<Real, false>))
sweep_pipe_kernel(const LevelArgs p, const CompactRecord<Real> *__restrict__ rec, const uint64_t begin,
                  const uint64_t end)
{
    __shared__ RecordStage<Real> stage[2];
    pdl_launch_dependents();
    const uint32_t gpv = p.G / VG, lane = threadIdx.x & 31u;
    const uint32_t nt = (uint32_t)(end - begin) * gpv, stride = gridDim.x * 64u;
    const CompactRecord<Real> *base = rec + begin;
    RecordStage<Real> &S = stage[threadIdx.x >> 5];
    auto item_of = [&](uint32_t t) { return gpv == 1u ? t : __umulhi(t, p.vmagic); };
    uint32_t first = 0;
    auto request = [&](uint32_t w) {
        if (w >= nt) return;
        first = item_of(w);
        S.fill(base + first, item_of(min(w + 31u, nt - 1u)) - first + 1u, lane);
    };
    uint32_t w = blockIdx.x * 64u + (threadIdx.x & ~31u);
    RegRecord<Real> R;
    Real q[4][VG];
    uint32_t g = 0;
    bool live = false;
    auto take = [&]() {
        S.wait();
        const uint32_t t = w + lane, it = item_of(t);
        live = t < nt;
        if (live) {
            S.take(it - first, R);
            live = R.u(0) != kSentinel;
        }
        __syncwarp();
        request(w + stride);
        if (live) {
            g = (t - it * gpv) * VG;
            task_source<Real, VG, BLK>(p, R, g, q);
        }
    };
    request(w);
    if (w < nt) take();
    pdl_wait_prerequisites();
    while (w < nt) {
        if (live)
            sweep_task<Real, VG, kLoadPlain, true, true, BLK>(p, R, g, [&](Real (&x)[4][VG]) {
#pragma unroll
                for (int v = 0; v < 4; ++v)
#pragma unroll
                    for (int e = 0; e < VG; ++e) x[v][e] = q[v][e];
            });
        w += stride;
        if (w < nt) take();
    }
}

template <typename Real, int VG, bool BLK, bool SC = false>
static const void *block_fn(bool deep, bool pf)
{
    if (!deep) return (const void *)sweep_block_kernel<Real, VG, BLK, false, false, SC>;
    return pf ? (const void *)sweep_block_kernel<Real, VG, BLK, true, true, SC>
              : (const void *)sweep_block_kernel<Real, VG, BLK, true, false, SC>;
}

template <typename Real>
cudaError_t launch_block_level(const LevelArgs &p, const void *rec, uint64_t begin, uint64_t end, cudaStream_t s)
{
    if (end <= begin) return cudaSuccess;
    const uint64_t tasks = (end - begin) * (p.G / p.vg);
    if (tasks >= (1ull << 26) || p.solver != kSolveNoPivot) return cudaErrorInvalidValue;
    const uint64_t sms = (uint64_t)device_sm_count();
    // the shallow form while its blocks are resident at once (75,776 tasks on
    // 148 SMs): against 0 / 40,000 / 75,776 / 120,000 the FP32 sweep takes 963 /
    // 925 / 911 / 970 us at 24^3 S8 G=8 and 1897 / 1840 / 1833 / 1890 at 32^3
    const bool deep = tasks > sms * kBlockMin<Real, false> * 64;
    unsigned grid = (unsigned)((tasks + 63) / 64);
    const bool pf = sms && tasks >= sms * kBlockMin<Real, true> * 64 * 2;
    const void *fn = nullptr;
    if constexpr (sizeof(Real) == 4)
        fn = p.scalar    ? block_fn<float, 4, true, true>(deep, pf)
             : p.vg == 4 ? block_fn<float, 4, true>(deep, pf)
             : p.vg == 2 ? block_fn<float, 2, true>(deep, pf)
                         : block_fn<float, 1, true>(deep, pf);
    else
        fn = p.G == 1    ? block_fn<double, 1, true>(deep, pf)
             : p.G == 2  ? block_fn<double, 2, true>(deep, pf)
             : p.vg == 2 ? block_fn<double, 2, false>(deep, pf)
                         : block_fn<double, 1, false>(deep, pf);
    if constexpr (sizeof(Real) == 8)
        if (deep && sms && p.vg == 2 && p.G >= 8) {
            fn = (const void *)sweep_pipe_kernel<double, 2, false>;
            grid = std::min(grid, (unsigned)(sms * kBlockMin<Real, false>));
        }
    void *args[] = {(void *)&p, (void *)&rec, (void *)&begin, (void *)&end};
    return launch_programmatic(fn, grid, 64, 0, args, s);
}

}  // namespace tycho
