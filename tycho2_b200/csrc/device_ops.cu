// Streaming kernels around the wavefront sweep, and deterministic vector
// kernels for the outer solvers.  This translation unit is compiled with
// -fmad=false: the FP64 wavefront kernel, the per-item face terms, the
// scalar flux and the scattering source keep the reference's rounding.
#include "device_ops.hpp"

#include <cstring>
#include "devmem.hpp"
#include "sweep_kernels.cuh"
#include "sweep_tiles.cuh"
#include "sweep_records.cuh"
#include "sweep_block.cuh"
#include "sweep_chains.cuh"
#include "stream_ops.cuh"

namespace tycho {

template cudaError_t launch_level<double>(int, const LevelArgs &, uint64_t, uint64_t, cudaStream_t);
template cudaError_t launch_dataflow<double>(int, const LevelArgs &, const DataflowArgs &, unsigned, cudaStream_t);
template cudaError_t dataflow_blocks_per_sm<double>(int, int *);
template cudaError_t launch_level_tile<double>(int, const LevelArgs &, uint64_t, uint64_t, cudaStream_t);
template cudaError_t launch_dataflow_tile<double>(int, const LevelArgs &, const DataflowArgs &, unsigned, cudaStream_t);
template cudaError_t tile_dataflow_blocks_per_sm<double>(int, int *);
template cudaError_t launch_item_records<double>(const LevelArgs &, uint64_t, void *, cudaStream_t);
template cudaError_t launch_level_record<double>(int, const LevelArgs &, const void *, uint64_t, uint64_t, cudaStream_t);
template cudaError_t launch_dataflow_record<double>(int, const LevelArgs &, const void *, const DataflowArgs &, unsigned,
                                               cudaStream_t);
template cudaError_t record_dataflow_blocks_per_sm<double>(int, int, int *);
template cudaError_t launch_persist_record<double>(int, const LevelArgs &, const void *, const uint64_t *, uint32_t,
                                                   unsigned long long *, const DataflowArgs &, unsigned, cudaStream_t);
template cudaError_t record_persist_blocks_per_sm<double>(int, int, int *);
template cudaError_t launch_direct_subset<double>(const LevelArgs &, const void *, const uint32_t *, uint64_t, uint64_t,
                                                   cudaStream_t);
template cudaError_t launch_direct_level<double>(int, const LevelArgs &, const void *, uint64_t, uint64_t, cudaStream_t,
                                                  bool);
template cudaError_t launch_block_level<double>(const LevelArgs &, const void *, uint64_t, uint64_t, cudaStream_t);
template cudaError_t launch_compact_records<double>(const LevelArgs &, uint64_t, const uint32_t *, void *, cudaStream_t);
template cudaError_t launch_chains<double>(ChainShape, const LevelArgs &, const void *, const uint32_t *, uint32_t, uint32_t,
                                             cudaStream_t);
template cudaError_t launch_direct_dataflow<double>(const LevelArgs &, const void *, bool, const DataflowArgs &,
                                                     unsigned, cudaStream_t);
template cudaError_t direct_dataflow_blocks_per_sm<double>(int, bool, int *);

namespace {

__global__ void item_abar_kernel(const uint32_t *__restrict__ items, uint64_t n, uint32_t A,
                                 const double *__restrict__ normal, const double *__restrict__ area,
                                 const double *__restrict__ omega, double4 *abar64, float4 *abar32)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t ca = items[i];
    if (ca == kSentinel) {  // level padding: never read by the sweep
        abar64[i] = make_double4(0.0, 0.0, 0.0, 0.0);
        if (abar32) abar32[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    const uint32_t c = ca / A, a = ca - c * A;
    const double xi = omega[a], eta = omega[A + a], mu = omega[2 * A + a];
    double ab[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const double *nrm = normal + ((size_t)c * 4 + f) * 3;
        // TychoMesh.cc:219-221 then Transport.cc:694-701
        const double odn = xi * nrm[0] + eta * nrm[1] + mu * nrm[2];
        ab[f] = area[(size_t)c * 4 + f] * odn;
    }
    abar64[i] = make_double4(ab[0], ab[1], ab[2], ab[3]);
    if (abar32) abar32[i] = make_float4((float)ab[0], (float)ab[1], (float)ab[2], (float)ab[3]);
}

// blk: 0 for rows [v][g]; else FP32 rows are blocks of blk groups, Gp groups
// with the padding (the default FP32 form), and a row's elements go where they
// stand in phi's.
template <typename Real, typename Form>
__global__ void __launch_bounds__(Form::kThreads)
psi_to_phi_kernel(const Real *__restrict__ psi, const double *__restrict__ w, double *__restrict__ phi, uint64_t nc,
                  uint32_t A, uint32_t G, uint32_t blk, uint32_t Gp, PhiPlan plan)
{
    extern __shared__ __align__(16) unsigned char stages[];
    pdl_wait_prerequisites();
    const uint64_t c0 = (uint64_t)blockIdx.x * plan.cells;
    const uint32_t row = 4 * Gp, n = (uint32_t)min((uint64_t)plan.cells, nc - c0);
    phi_of_tiles<Real, Form, true>(psi + c0 * A * row, w, n, A, row, plan, stages,
                             [&](uint32_t, uint32_t, const double (&s)[Form::kElems]) {
#pragma unroll
        for (int k = 0; k < Form::kElems; ++k) {
            const uint32_t e = Form::kElems * threadIdx.x + k;
            if (e >= n * row) return;
            const uint32_t cl = e / row, q = e - cl * row;
            uint32_t v = q / G, g = q - v * G;
            if (blk) {
                const uint32_t b = q / (4 * blk), r = q - b * 4 * blk;
                v = r / blk;
                g = b * blk + (r - v * blk);
            }
            if (g < G) phi[(c0 + cl) * 4 * G + v * G + g] = s[k];
        }
    });
}

// One thread per (cell, group): the group's four vertex elements (groups
// fastest, so a warp writes runs of G consecutive elements per vertex).
__global__ void scatter_source_kernel(const double *__restrict__ phi, const double *__restrict__ q,
                                      const double *__restrict__ sigma_s,
                                      const double *__restrict__ scat, double *__restrict__ iso,
                                      float *__restrict__ iso32, uint64_t nc, uint32_t G, uint32_t blk,
                                      uint32_t Gp)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nc * G) return;
    const uint64_t c = t < (1ull << 32) ? (uint64_t)((uint32_t)t / G) : t / G;
    const uint32_t g = (uint32_t)(t - c * G);
    double s[4];
    scatter_cell_group(phi, q, sigma_s, scat, c, g, G, s);
    const uint64_t base = c * 4 * G + g;
#pragma unroll
    for (int v = 0; v < 4; ++v) iso[base + v * G] = s[v];
    if (iso32) {
#pragma unroll
        for (int v = 0; v < 4; ++v)
            iso32[c * 4 * (blk ? Gp : G) + source_pos(v, g, G, blk)] = (float)s[v];
    }
}

// Where block b of a reduction leaves its sum of result j: a result's
// partial sums side by side, so that the blocks that add them up read whole
// lines.
__device__ __forceinline__ size_t partial_at(int j, int b) { return (size_t)j * kReduceBlocks + b; }

// The block's K sums over its threads into the partial sums j0 ... of b.
template <int K>
__device__ __forceinline__ void store_partials(const double (&acc)[K], int j0, int k, double *partials)
{
    __shared__ double sh[8][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const double v = warp_sum(acc[j]);
        if (lane == 0) sh[warp][j] = v;
    }
    __syncthreads();
    if (threadIdx.x < K && j0 + (int)threadIdx.x < k) {
        double s = 0.0;
        for (int q = 0; q < 8; ++q) s += sh[q][threadIdx.x];
        partials[partial_at(j0 + threadIdx.x, blockIdx.x)] = s;
    }
}

// One thread's share of the sum of p[0 .. nb) over 128 threads: t, t + 128,
// ... in order.  L2: read past the L1 (written by this launch's other blocks).
template <bool L2 = false>
__device__ __forceinline__ double partial_share(const double *p, int nb, int t)
{
    constexpr int kMax = (kReduceBlocks + 127) / 128;
    double v[kMax];
#pragma unroll
    for (int q = 0; q < kMax; ++q) {
        const int b = t + 128 * q;
        v[q] = b < nb ? (L2 ? __ldcg(p + b) : p[b]) : 0.0;
    }
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kMax; ++q) s += v[q];
    return s;
}

// The sums of k <= 8 results over nb blocks, by one block of 256 threads,
// into h[0 .. k): each half of the block takes every other result.
__device__ __forceinline__ void sum_partials8(const double *partials, int nb, int k, double *h)
{
    __shared__ double part[8][4];
    const int half = threadIdx.x >> 7, t = threadIdx.x & 127, lane = threadIdx.x & 31, warp = t >> 5;
    double s[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        s[q] = half + 2 * q < k ? partial_share(partials + partial_at(half + 2 * q, 0), nb, t) : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double v = warp_sum(s[q]);
        if (lane == 0) part[half + 2 * q][warp] = v;
    }
    __syncthreads();
    if ((int)threadIdx.x < k)
        h[threadIdx.x] = (part[threadIdx.x][0] + part[threadIdx.x][1]) + (part[threadIdx.x][2] + part[threadIdx.x][3]);
    __syncthreads();
}

// Inner products <w, V_j>, j0 <= j < k, on 16-byte pairs: each thread issues
// U x (K + 1) pair loads before its FMAs, so that the few-vector passes of an
// Arnoldi step keep enough loads in flight to stream at HBM rate.  Per
// thread: the pairs it visits in grid-stride order, the first element of each
// pair before the second.
template <int K, int U>
__global__ void __launch_bounds__(256)
multi_dot_kernel(const double2 *__restrict__ w, const double2 *__restrict__ V, size_t ld2, int k, int j0,
                  uint64_t n2, double *__restrict__ partials)
{
    double acc[K];
#pragma unroll
    for (int j = 0; j < K; ++j) acc[j] = 0.0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n2; i0 += stride * U) {
        double2 wv[U], v[U][K];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + u * stride;
            if (i < n2) {
                wv[u] = w[i];
#pragma unroll
                for (int j = 0; j < K; ++j)
                    if (j0 + j < k) v[u][j] = V[(size_t)(j0 + j) * ld2 + i];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u * stride >= n2) break;
#pragma unroll
            for (int j = 0; j < K; ++j)
                if (j0 + j < k) {
                    acc[j] = __fma_rn(wv[u].x, v[u][j].x, acc[j]);
                    acc[j] = __fma_rn(wv[u].y, v[u][j].y, acc[j]);
                }
        }
    }
    store_partials<K>(acc, j0, k, partials);
}

// The fixed point's change, sum |x - y| and sum |x|, and y = x for the next
// one.  The block that finishes last adds the partial sums up (in block
// order, whichever block that is) and writes the pair to the host, so one
// launch takes the place of a copy, two kernels and a copy to the host: a
// step of 8^3 S4 87 -> 81 us.
__global__ void __launch_bounds__(256)
l1_kernel(const double *__restrict__ x, double *__restrict__ y, uint64_t n, double *__restrict__ partials,
          unsigned *__restrict__ ticket, double *__restrict__ host)
{
    double acc[2] = {0.0, 0.0};
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const double xi = x[i];
        acc[0] += fabs(xi - y[i]);
        acc[1] += fabs(xi);
        y[i] = xi;
    }
    store_partials<2>(acc, 0, 2, partials);
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    __shared__ double part[8];
    const int j = threadIdx.x >> 7, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double v = warp_sum(partial_share<true>(partials + partial_at(j, 0), (int)gridDim.x, threadIdx.x & 127));
    if (lane == 0) part[warp] = v;
    __syncthreads();
    if (threadIdx.x < 2) {
        const double *q = part + 4 * threadIdx.x;
        host[threadIdx.x] = (q[0] + q[1]) + (q[2] + q[3]);
    }
}

// out[j] and host[j] = the sum over blocks b of the partial sums of result j:
// one block per result, each thread its blocks in order, then a fixed tree.
// One thread per result walking every partial took 27 us (592 dependent loads
// and adds), as long as ten wavefront levels of a small problem; this takes
// about 3.
__global__ void __launch_bounds__(128)
reduce_partials_kernel(const double *__restrict__ partials, int nblocks, double *__restrict__ out,
                       double *__restrict__ host)
{
    __shared__ double sh[4];
    const int j = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double s = warp_sum(partial_share(partials + partial_at(j, 0), nblocks, threadIdx.x));
    if (lane == 0) sh[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) out[j] = host[j] = (sh[0] + sh[1]) + (sh[2] + sh[3]);
}

// One pass of the twice-applied Gram-Schmidt step over w and k basis vectors.
//   PASS 0: w = V_{k-1} - w (the operator I - K), then <w, V_j>;
//   PASS 1: w -= sum_j h[j] V_j, then <w, V_j>;
//   PASS 2: w -= sum_j h[j] V_j, then <w, w>.
// The update and the inner products of the new w share one read of w and, for
// the first K vectors, of V: 3 reads of the basis a step in place of 4, and 8
// fewer passes over w.  k <= 8 (MANY false): every block adds up the last
// pass's partial sums itself (28 KB from L2 at k = 8, about 1 us) where a
// launch between the two would cost 2-3; beyond 8 vectors that read grows
// past the launch, and h is read as reduce_partials_kernel left it.  Bound by
// the bytes of V and w on large problems and by the launches (4 a step) on
// small ones: after each sweep of 16^3 S6 G=4, 10 launches and a copy to the
// host before, now 4 (10 steps 5.78 -> 5.74 ms; 24^3 S8 G=8 mixed, 9 steps,
// 14.05 -> 13.75).  The operations of each element and of each sum, and their
// order, are those of separate passes.
template <int K, int U, int PASS, bool MANY>
__global__ void __launch_bounds__(256)
arnoldi_pass_kernel(double2 *__restrict__ w, const double2 *__restrict__ V, size_t ld2, int k, uint64_t n2,
                    const double *__restrict__ h_in, int nb_in, double *__restrict__ h_host,
                    double *__restrict__ partials)
{
    __shared__ double h[MANY ? 64 : 8];
    if (PASS > 0) {
        if (MANY) {
            if ((int)threadIdx.x < k) h[threadIdx.x] = h_in[threadIdx.x];
            __syncthreads();
        } else {
            sum_partials8(h_in, nb_in, k, h);
            if (blockIdx.x == 0 && (int)threadIdx.x < k) h_host[threadIdx.x] = h[threadIdx.x];
        }
    }
    constexpr int KD = PASS == 2 ? 1 : K;
    double acc[KD];
#pragma unroll
    for (int j = 0; j < KD; ++j) acc[j] = 0.0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n2; i0 += stride * U) {
        double2 wv[U], v[U][K];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + u * stride;
            if (i < n2) {
                wv[u] = w[i];
#pragma unroll
                for (int j = 0; j < K; ++j)
                    if (j < k) v[u][j] = V[(size_t)j * ld2 + i];
                if (PASS == 0) {
                    const double2 x = V[(size_t)(k - 1) * ld2 + i];
                    wv[u].x = x.x - wv[u].x;
                    wv[u].y = x.y - wv[u].y;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint64_t i = i0 + u * stride;
            if (i >= n2) break;
            double2 s = wv[u];
            if (PASS > 0) {
#pragma unroll
                for (int j = 0; j < K; ++j)
                    if (j < k) {
                        s.x = __fma_rn(-h[j], v[u][j].x, s.x);
                        s.y = __fma_rn(-h[j], v[u][j].y, s.y);
                    }
                if (MANY) {
                    for (int j0 = K; j0 < k; j0 += 8) {
                        double2 x[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (j0 + j < k) x[j] = V[(size_t)(j0 + j) * ld2 + i];
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (j0 + j < k) {
                                s.x = __fma_rn(-h[j0 + j], x[j].x, s.x);
                                s.y = __fma_rn(-h[j0 + j], x[j].y, s.y);
                            }
                    }
                }
            }
            w[i] = s;
            if (PASS == 2) {
                acc[0] = __fma_rn(s.x, s.x, acc[0]);
                acc[0] = __fma_rn(s.y, s.y, acc[0]);
            } else {
#pragma unroll
                for (int j = 0; j < KD; ++j)
                    if (j < k) {
                        acc[j] = __fma_rn(s.x, v[u][j].x, acc[j]);
                        acc[j] = __fma_rn(s.y, v[u][j].y, acc[j]);
                    }
            }
        }
    }
    store_partials<KD>(acc, 0, PASS == 2 ? 1 : k, partials);
}

// w /= ||w|| (left as is when that is 0); *norm = ||w||, from the partial
// sums of <w, w>, which every block adds up.
__global__ void __launch_bounds__(256)
scale_by_norm_kernel(double2 *__restrict__ w, uint64_t n2, const double *__restrict__ partials, int nb,
                     double *__restrict__ norm)
{
    __shared__ double sq;
    sum_partials8(partials, nb, 1, &sq);
    const double hn = sqrt(sq);
    if (blockIdx.x == 0 && threadIdx.x == 0) *norm = hn;
    if (!(hn > 0.0)) return;
    const double inv = 1.0 / hn;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += (uint64_t)gridDim.x * blockDim.x) {
        double2 s = w[i];
        s.x *= inv;
        s.y *= inv;
        w[i] = s;
    }
}

// w -= sum_j h[j] V_j on 16-byte pairs, eight basis vectors' loads issued
// before their FMAs.
__global__ void multi_axpy_kernel(double2 *__restrict__ w, const double2 *__restrict__ V, size_t ld2,
                                   const double *__restrict__ h, int k, uint64_t n2)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n2) return;
    double2 s = w[i];
    for (int j0 = 0; j0 < k; j0 += 8) {
        double2 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j0 + j < k) v[j] = V[(size_t)(j0 + j) * ld2 + i];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j0 + j < k) {
                const double hj = h[j0 + j];
                s.x = __fma_rn(-hj, v[j].x, s.x);
                s.y = __fma_rn(-hj, v[j].y, s.y);
            }
    }
    w[i] = s;
}

__global__ void axpby_kernel(double alpha, const double *__restrict__ x, double beta,
                             double *__restrict__ y, uint64_t n)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __fma_rn(alpha, x[i], beta * y[i]);
}

__global__ void sub_from_kernel(const double *__restrict__ x, double *__restrict__ y, uint64_t n)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = x[i] - y[i];
}

__global__ void bump_epoch_kernel(uint32_t *epoch)
{
    const uint32_t v = *epoch + 1u;
    *epoch = v == 0u ? 1u : v;
}

inline unsigned blocks_for(uint64_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace

ChainShape chain_shape(bool fp32, bool one_block, double tasks, int directions, bool wide)
{
    return chain_shape_rule(fp32, one_block, tasks, directions, wide);
}

cudaError_t launch_item_abar(const uint32_t *items, uint64_t n, uint32_t A, const double *normal,
                             const double *area, const double *omega, double4 *abar64,
                             float4 *abar32, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    item_abar_kernel<<<blocks_for(n), 256, 0, s>>>(items, n, A, normal, area, omega, abar64, abar32);
    return cudaGetLastError();
}

template <typename Real, typename Form>
static cudaError_t launch_phi(const Real *psi, const double *w, double *phi, uint64_t nc, uint32_t A, uint32_t G,
                       uint32_t blk, uint32_t Gp, cudaStream_t s)
{
    // tiles of an element or two per thread; fewer cells a tile where those would not give
    // every SM four blocks (8^3 of 4 elements: 512 tiles of 6 cells, not 48 of 64)
    const uint64_t blocks = 4 * (uint64_t)std::max(device_sm_count(), 1);
    const uint64_t even = (nc + blocks - 1) / blocks;
    const uint32_t tile = (uint32_t)Form::kElems * Form::kThreads;
    const PhiPlan plan = phi_plan<Form>((uint32_t)std::min<uint64_t>(tile / (4 * Gp), even),
                                        4 * Gp * (uint32_t)sizeof(Real), A);
    const unsigned grid = (unsigned)((nc + plan.cells - 1) / plan.cells);
    void *args[] = {(void *)&psi, (void *)&w, (void *)&phi, (void *)&nc,  (void *)&A,
                    (void *)&G,   (void *)&blk, (void *)&Gp, (void *)&plan};
    return launch_programmatic((const void *)psi_to_phi_kernel<Real, Form>, grid, Form::kThreads,
                               Form::kStages * plan.cells * plan.stride, args, s);
}

cudaError_t launch_psi_to_phi(const void *psi, bool psi_fp32, const double *w, double *phi,
                              uint64_t nc, uint32_t A, uint32_t G, uint32_t blk, uint32_t Gp, cudaStream_t s)
{
    if (nc == 0) return cudaSuccess;
    const uint32_t row = 4 * (psi_fp32 && blk ? Gp : G);
    const bool wide = row > 128 && row <= 160;
    if (!psi_fp32 && wide) return launch_phi<double, PhiWide>((const double *)psi, w, phi, nc, A, G, 0, G, s);
    if (!psi_fp32) return launch_phi<double, PhiOne>((const double *)psi, w, phi, nc, A, G, 0, G, s);
    if (G == 1) return launch_phi<float, PhiOne>((const float *)psi, w, phi, nc, A, G, blk, blk ? Gp : G, s);
    if (wide) return launch_phi<float, PhiWide>((const float *)psi, w, phi, nc, A, G, blk, blk ? Gp : G, s);
    return launch_phi<float, PhiTwo>((const float *)psi, w, phi, nc, A, G, blk, blk ? Gp : G, s);
}

cudaError_t launch_scatter_source(const double *phi_in, const double *q_fixed, const double *sigma_s,
                                  const double *scatter, double *iso, float *iso32, uint64_t nc,
                                  uint32_t G, uint32_t blk, uint32_t Gp, cudaStream_t s)
{
    const uint64_t n = nc * G;
    if (n == 0) return cudaSuccess;
    scatter_source_kernel<<<blocks_for(n), 256, 0, s>>>(phi_in, q_fixed, sigma_s, scatter, iso, iso32, nc, G,
                                                         blk, Gp);
    return cudaGetLastError();
}

cudaError_t launch_bump_epoch(uint32_t *epoch, cudaStream_t s)
{
    bump_epoch_kernel<<<1, 1, 0, s>>>(epoch);
    return cudaGetLastError();
}

cudaError_t reducer_init(Reducer &r, cudaStream_t s)
{
    cudaError_t e = dev_malloc(&r.partials, sizeof(double) * kReduceBlocks * 64 * 2, s);
    if (e == cudaSuccess) e = dev_malloc(&r.result, sizeof(double) * kReduceSlots, s);
    if (e == cudaSuccess) e = dev_malloc(&r.ticket, sizeof(unsigned), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(r.ticket, 0, sizeof(unsigned), s);
    if (e == cudaSuccess) e = cudaMallocHost(&r.host, sizeof(double) * kReduceSlots);
    if (e == cudaSuccess) std::memset(r.host, 0, sizeof(double) * kReduceSlots);
    return e;
}

void reducer_free(Reducer &r, cudaStream_t s)
{
    dev_free(r.partials, s);
    dev_free(r.result, s);
    dev_free(r.ticket, s);
    if (r.host) cudaFreeHost(r.host);
    r = Reducer();
}

// Vectors that the kernels read as pairs of doubles.
static bool in_pairs(const double *a, const double *b, uint64_t n)
{
    return n % 2 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}

// The blocks of a pass over n2 pairs: a small problem's further blocks would
// only add zeros.
static int dot_blocks(uint64_t n2)
{
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(kDotBlocks, (n2 + 255) / 256));
}

// The inner products <w, V_j>, j0 <= j < k, into per-block partials, in
// passes of at most 8 basis vectors.
static void launch_multi_dot(const double2 *w2, const double2 *V2, size_t ld2, int j0, int k, uint64_t n2,
                             double *partials, cudaStream_t s)
{
    const int nb = dot_blocks(n2);
    while (j0 < k) {
        const int rem = k - j0;
        if (rem <= 2) {
            multi_dot_kernel<2, 4><<<nb, 256, 0, s>>>(w2, V2, ld2, k, j0, n2, partials);
            j0 += 2;
        } else if (rem <= 4) {
            multi_dot_kernel<4, 2><<<nb, 256, 0, s>>>(w2, V2, ld2, k, j0, n2, partials);
            j0 += 4;
        } else {
            multi_dot_kernel<8, 1><<<nb, 256, 0, s>>>(w2, V2, ld2, k, j0, n2, partials);
            j0 += 8;
        }
    }
}

template <int PASS>
static void launch_arnoldi_pass(double2 *w, const double2 *V, int k, uint64_t n2, const double *h_in, double *h_host,
                                double *partials, cudaStream_t s)
{
    const int nb = dot_blocks(n2);
    if (k <= 2) arnoldi_pass_kernel<2, 4, PASS, false><<<nb, 256, 0, s>>>(w, V, n2, k, n2, h_in, nb, h_host, partials);
    else if (k <= 4)
        arnoldi_pass_kernel<4, 2, PASS, false><<<nb, 256, 0, s>>>(w, V, n2, k, n2, h_in, nb, h_host, partials);
    else if (k <= 8)
        arnoldi_pass_kernel<8, 1, PASS, false><<<nb, 256, 0, s>>>(w, V, n2, k, n2, h_in, nb, h_host, partials);
    else arnoldi_pass_kernel<8, 1, PASS, true><<<nb, 256, 0, s>>>(w, V, n2, k, n2, h_in, nb, h_host, partials);
}

cudaError_t arnoldi_step(double *V, int k, uint64_t n, Reducer &r, cudaStream_t s)
{
    if (k < 1 || k > 64 || !in_pairs(V, V, n)) return cudaErrorInvalidValue;
    const uint64_t n2 = n / 2;
    const int nb = dot_blocks(n2);
    const double2 *V2 = reinterpret_cast<const double2 *>(V);
    double2 *w = reinterpret_cast<double2 *>(V) + (size_t)k * n2;
    double *pa = r.partials, *pb = r.partials + (size_t)kReduceBlocks * 64, *res = r.result;
    launch_arnoldi_pass<0>(w, V2, k, n2, nullptr, nullptr, pa, s);
    if (k > 8) {
        launch_multi_dot(w, V2, n2, 8, k, n2, pa, s);
        reduce_partials_kernel<<<k, 128, 0, s>>>(pa, nb, res, r.host);
        launch_arnoldi_pass<1>(w, V2, k, n2, res, nullptr, pb, s);
        launch_multi_dot(w, V2, n2, 8, k, n2, pb, s);
        reduce_partials_kernel<<<k, 128, 0, s>>>(pb, nb, res + 64, r.host + 64);
        launch_arnoldi_pass<2>(w, V2, k, n2, res + 64, nullptr, pa, s);
    } else {
        launch_arnoldi_pass<1>(w, V2, k, n2, pa, r.host, pb, s);
        launch_arnoldi_pass<2>(w, V2, k, n2, pb, r.host + 64, pa, s);
    }
    scale_by_norm_kernel<<<nb, 256, 0, s>>>(w, n2, pa, nb, r.host + 128);
    return cudaGetLastError();
}

cudaError_t dot(const double *x, const double *y, uint64_t n, Reducer &r, cudaStream_t s)
{
    if (!in_pairs(x, y, n)) return cudaErrorInvalidValue;
    launch_multi_dot(reinterpret_cast<const double2 *>(x), reinterpret_cast<const double2 *>(y), n / 2, 0, 1, n / 2,
                     r.partials, s);
    reduce_partials_kernel<<<1, 128, 0, s>>>(r.partials, dot_blocks(n / 2), r.result, r.host);
    cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

cudaError_t l1_change(const double *x, double *y, uint64_t n, Reducer &r, cudaStream_t s)
{
    const unsigned nb = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(kReduceBlocks, (n + 255) / 256));
    l1_kernel<<<nb, 256, 0, s>>>(x, y, n, r.partials, r.ticket, r.host);
    return cudaGetLastError();
}

cudaError_t multi_axpy(double *w, const double *V, const double *h, int k, uint64_t n, cudaStream_t s)
{
    if (n == 0 || k == 0) return cudaSuccess;
    if (!in_pairs(w, V, n)) return cudaErrorInvalidValue;
    multi_axpy_kernel<<<blocks_for(n / 2), 256, 0, s>>>(reinterpret_cast<double2 *>(w),
                                                        reinterpret_cast<const double2 *>(V), n / 2, h, k, n / 2);
    return cudaGetLastError();
}

cudaError_t axpby(double alpha, const double *x, double beta, double *y, uint64_t n, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    axpby_kernel<<<blocks_for(n), 256, 0, s>>>(alpha, x, beta, y, n);
    return cudaGetLastError();
}

cudaError_t sub_from(const double *x, double *y, uint64_t n, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    sub_from_kernel<<<blocks_for(n), 256, 0, s>>>(x, y, n);
    return cudaGetLastError();
}

}  // namespace tycho
