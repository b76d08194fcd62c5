// Element arithmetic of the streaming passes around the sweep, shared by the
// single-instance kernels (device_ops.cu) and the batched ones (batch_ops.cu)
// so that a batch member computes bit for bit what it computes alone.  Both
// translation units are compiled with -fmad=false.
#pragma once

#include <cstdint>

namespace tycho {

constexpr double kFourPi = 4.0 * 3.14159265358979323846;

// Isotropic total source of phi element i = (c*4 + v)*G + g:
//   [q_i +] sum_g' sigma_s[c] * scat[g][g'] / (4 pi) * phi_(c,v,g')
// (within-group when scat is null: Util.cc:126-128).  phi == nullptr gives
// q_i (or 0).
__device__ __forceinline__ double scatter_elem(const double *__restrict__ phi, const double *__restrict__ q,
                                               const double *__restrict__ sigma_s,
                                               const double *__restrict__ scat, uint64_t i, uint32_t G)
{
    const uint64_t c = i / ((uint64_t)4 * G);
    double s;
    if (phi) {
        if (!scat) {
            s = sigma_s[c] / kFourPi * phi[i];
        } else {
            const uint32_t g = (uint32_t)(i % G);
            const double *pv = phi + (i - g);
            s = 0.0;
            for (uint32_t gp = 0; gp < G; ++gp) {
                const double k = scat[g * G + gp];
                if (k == 0.0) continue;
                s += sigma_s[c] * k / kFourPi * pv[gp];
            }
        }
        if (q) s = q[i] + s;
    } else {
        s = q ? q[i] : 0.0;
    }
    return s;
}

// The four vertex elements (c, v, g), v = 0..3, of the total isotropic
// source, with the arithmetic of scatter_elem term by term (the same
// coefficient sigma_s[c] * k / 4pi, the same summation order over g'), so
// the results are bit-identical; the coefficient is formed once for the four
// vertices instead of once per element.
__device__ __forceinline__ void scatter_cell_group(const double *__restrict__ phi, const double *__restrict__ q,
                                                   const double *__restrict__ sigma_s,
                                                   const double *__restrict__ scat, uint64_t c, uint32_t g,
                                                   uint32_t G, double (&s)[4])
{
    const uint64_t base = c * 4 * G;
    if (phi) {
        if (!scat) {
            const double k = sigma_s[c] / kFourPi;
#pragma unroll
            for (int v = 0; v < 4; ++v) s[v] = k * phi[base + v * G + g];
        } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) s[v] = 0.0;
            for (uint32_t gp = 0; gp < G; ++gp) {
                const double k = scat[g * G + gp];
                if (k == 0.0) continue;
                const double kc = sigma_s[c] * k / kFourPi;
#pragma unroll
                for (int v = 0; v < 4; ++v) s[v] += kc * phi[base + v * G + gp];
            }
        }
        if (q) {
#pragma unroll
            for (int v = 0; v < 4; ++v) s[v] = q[base + v * G + g] + s[v];
        }
    } else {
#pragma unroll
        for (int v = 0; v < 4; ++v) s[v] = q ? q[base + v * G + g] : 0.0;
    }
}

// FP32 rows kept as blocks of `blk` groups: [g / blk][v][g % blk] instead of
// [v][g].  Position of (v, g) in a row (blk 0: plain):
__device__ __forceinline__ uint32_t source_pos(uint32_t v, uint32_t g, uint32_t G, uint32_t blk)
{
    return blk ? (g / blk * 4u + v) * blk + g % blk : v * G + g;
}
// and the plain element of the one at block-layout position i (c*4G + j).
__device__ __forceinline__ uint64_t block_to_plain(uint64_t i, uint32_t G, uint32_t blk)
{
    const uint32_t row = 4u * G, j = (uint32_t)(i % row);
    const uint32_t b = j / (4u * blk), r = j - b * 4u * blk, v = r / blk;
    return i - j + v * G + b * blk + (r - v * blk);
}

// Asynchronous 16-byte copy into shared memory.
__device__ __forceinline__ void cp_async16(void *smem, const void *global)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(global) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Scalar flux, phi(c, v, g) = sum_a w_a psi(c, a, v, g), angles in increasing
// order in FP64 (Util::psiToPhi, Util.cc:85-97), for tiles of whole cells (at
// most 256 elements, wide ones 512).  Bound by the bytes of psi, which a block streams
// through shared-memory stages, each some angles of each of its cells.  Loads
// into registers, eight angles ahead of their sums, waited a memory latency
// per eight angles: 32^3 S8, FP64 G=8 923 -> 906 us (7.1 TB/s), 24^3 G=3
// 240 -> 172, G=1 S4 30 -> 21; FP32 G=8 588 -> 493 (6.5 TB/s).
// Two forms: one element per thread with 3 stages of 12 KB in flight in each
// of 4 blocks of an SM; and for FP32 rows of two and more groups, whose
// conversions and sums otherwise bound it (G=8 560 us), two elements per
// thread of blocks of half as many threads, in 9 blocks with 2 stages of 8 KB.
// At G=1 the second form's stages are a few angles of 64 cells: 169 us
// against 105.  Rows of 132 to 160 elements leave up to half of a 256-element
// tile's threads idle; with two elements per thread of 256 a tile has three of
// them (24^3 S4 G=33: FP32 405 -> 351 us, FP64 591 -> 487; G=40 at 20^3 FP64 375 -> 346;
// G=48, rows of 192, FP32 20^3 S6 472 -> 499).
struct PhiOne { static constexpr int kElems = 1, kThreads = 256, kStages = 4, kBytes = 12288; };
struct PhiTwo { static constexpr int kElems = 2, kThreads = 128, kStages = 3, kBytes = 8192; };
struct PhiWide { static constexpr int kElems = 2, kThreads = 256, kStages = 4, kBytes = 12288; };
constexpr int kPhiTile = 256;

struct PhiPlan {
    uint32_t cells;   // of a tile
    uint32_t angles;  // of a stage
    uint32_t stride;  // bytes from a cell to the next in a stage
    uint32_t shift;   // log2 of the threads that copy a cell
};

// row_bytes: of one (cell, angle) row, a multiple of 16 and at most 2 KB.  A
// cell's part of a stage is followed by as much padding as makes the next
// cell's rows continue in the banks where its own end.
template <typename Form>
__host__ __device__ inline PhiPlan phi_plan(uint32_t cells, uint32_t row_bytes, uint32_t A)
{
    PhiPlan p;
    p.cells = cells;
    uint32_t n = Form::kBytes / (cells * row_bytes);
    n = n < A ? n : A;
    for (;; --n) {
        p.stride = n * row_bytes + ((row_bytes - n * row_bytes) & 127u);
        if (n == 1 || cells * p.stride <= (uint32_t)Form::kBytes) break;
    }
    const uint32_t stages = (A + n - 1) / n;
    p.angles = (A + stages - 1) / stages;
    p.stride = p.angles * row_bytes + ((row_bytes - p.angles * row_bytes) & 127u);
    p.shift = 0;
    while ((cells << p.shift) * 2 <= (uint32_t)Form::kThreads) ++p.shift;
    return p;
}

// The elements of n cells from `psi` on, rows of `row` values, in tiles of
// p.cells: emit(first cell of the tile, its cells, s) with the thread's elements
// E * threadIdx.x ... of the tile's (garbage beyond its end).  The stages of all
// tiles are one sequence, so a tile's first ones are on their way while the tile
// before is summed.  smem: the stages, each p.cells * p.stride bytes, 16-byte
// aligned.  ONE: n <= p.cells.  All threads of a block of Form::kThreads must
// call it.
template <typename Real, typename Form, bool ONE, typename Emit>
__device__ __forceinline__ void phi_of_tiles(const Real *__restrict__ psi, const double *__restrict__ w, uint32_t n,
                                             uint32_t A, uint32_t row, const PhiPlan &p, unsigned char *smem, Emit emit)
{
    constexpr int E = Form::kElems, NS = Form::kStages;
    struct alignas(E * sizeof(Real)) Vec { Real x[E]; };
    const uint32_t rb = row * (uint32_t)sizeof(Real), cell = threadIdx.x >> p.shift;
    const uint32_t lane = threadIdx.x & ((1u << p.shift) - 1u);
    const uint32_t stage_bytes = p.cells * p.stride;
    const size_t tile_bytes = (size_t)p.cells * A * rb;
    const unsigned char *src = reinterpret_cast<const unsigned char *>(psi) + (size_t)cell * A * rb;
    uint32_t ld_c0 = 0, ld_a0 = 0, ld_slot = 0;  // the next stage to load: its tile's first cell, first angle, place
    auto load = [&] {
        if (ONE ? ld_a0 < A : ld_c0 < n) {
            if (ONE ? cell < n : cell < p.cells && ld_c0 + cell < n) {
                const uint32_t bytes = min(p.angles, A - ld_a0) * rb;
                unsigned char *d = smem + ld_slot * stage_bytes + cell * p.stride;
                const unsigned char *q = src + (size_t)ld_a0 * rb;
                for (uint32_t x = lane * 16; x < bytes; x += 16u << p.shift) cp_async16(d + x, q + x);
            }
            ld_slot = ld_slot + 1 == NS ? 0 : ld_slot + 1;
            ld_a0 += p.angles;
            if (!ONE && ld_a0 >= A) {
                ld_a0 = 0;
                ld_c0 += p.cells;
                src += tile_bytes;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) load();
    const uint32_t e = E * threadIdx.x < p.cells * row ? E * threadIdx.x : 0, ec = e / row;
    const unsigned char *mine = smem + ec * p.stride + (e - ec * row) * sizeof(Real);
    uint32_t slot = 0;
    for (uint32_t c0 = 0; c0 < n; c0 += p.cells) {
        double s[E];
#pragma unroll
        for (int k = 0; k < E; ++k) s[k] = 0.0;
        for (uint32_t a0 = 0; a0 < A; a0 += p.angles) {
            asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
            __syncthreads();  // the stage is there; all threads are done with the one before
            load();           // into the latter's place
            const uint32_t na = min(p.angles, A - a0);
            const unsigned char *q = mine + slot * stage_bytes;
            slot = slot + 1 == NS ? 0 : slot + 1;
#pragma unroll 4
            for (uint32_t a = 0; a < na; ++a, q += rb) {
                const Vec v = *reinterpret_cast<const Vec *>(q);
                const double wa = w[a0 + a];
#pragma unroll
                for (int k = 0; k < E; ++k) s[k] += (double)v.x[k] * wa;
            }
        }
        emit(c0, ONE ? n : min(p.cells, n - c0), s);
        if (ONE) break;
    }
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace tycho
