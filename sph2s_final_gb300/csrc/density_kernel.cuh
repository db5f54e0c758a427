// density_kernel.cuh -- the density pass of the single-scale step.
//
// computeDensitiesPressuresD + computeDensityCell (SPH2S_FINAL_SINGLE_SCALE/
// Solver.cu:536-599, 198-229): rho_i = m sum_j W_poly6(r_ij) over the stencil
// [cell(x - h), cell(x + h)] with r < h (self included), p_i = K (rho_i - rho0).
//
// Besides rho and the factors the force pass needs from every neighbour
// (p/rho^2, 1/rho, in aux), it writes the force pass's per-neighbour records:
// xa[i] = (x, y, z, p/rho^2) and the w slot of the step's velocity,
// svel[i].w = 1/rho, so the force pass gathers two 16-byte records per
// neighbour instead of three loads.  It also emits the neighbour list: every j with
// 0 < r2 < T, in stencil order.  Lists are stored transposed in groups of
// four, group g of particle i at nbr4[g * n + i], so the force pass reads 512
// contiguous bytes per warp instruction; the density pass stores each index
// as it is found (one 4-byte store into its slot, cheaper per hit than
// assembling groups in registers: 0.68 -> 0.58 ms at 2M particles on GB300).
// The list traffic (~136 bytes per particle, read once by the force pass) is
// stored and loaded with streaming (evict-first) cache hints, so it displaces
// less of the force records the force pass gathers from L2 (2M step
// 0.837 -> 0.830 ms).
// A count beyond the list (above kMaxNbr) has the force pass rescan the stencil for
// that particle.
//
// One thread per particle, particles in Morton order (a warp's particles
// share most of their stencil cells, so candidate loads hit in L1).  Measured
// alternatives that were slower on GB300 at 2M particles: a warp-cooperative
// scan of the warp's union stencil through shared memory (Morton order puts
// about a quarter of all warps across octant jumps, whose union boxes hold
// hundreds of cells), Morton-contiguous multi-cell runs (parity-dependent
// control flow diverges inside a warp), and branch-free hit masks with
// deferred list appends.
#pragma once
#include "common.cuh"

namespace sph {

constexpr int kDensityThreads = 256;

// Density of particle i of the sorted array (n particles, indices in `cells`
// refer to that array); the batched solver calls this with per-scene P and
// cell table.
template <bool DEBUG, class LISTS>
__device__ __forceinline__ void density_one(uint32_t i, const float4* __restrict__ pos,
                                            const uint2* __restrict__ cells, uint32_t n,
                                            const SimParams& P, float* __restrict__ rho,
                                            float2* __restrict__ aux, uint4* __restrict__ nbr4,
                                            uint32_t* __restrict__ nbr_count, LISTS lists,
                                            uint32_t* __restrict__ dbg_count,
                                            float4* __restrict__ xa, float4* __restrict__ svel) {
    uint32_t k = 0, zero = 0;
    float sum = 0.0f;
    const float4 xi = pos[i];
    // next list slot: element k & 3 of group k >> 2, i.e. u32 offset 4 (g n + i) + (k & 3)
    uint32_t* out = reinterpret_cast<uint32_t*>(nbr4) + 4 * (size_t)i;
    const uint32_t next_group = 4u * n - 3u;  // fits 32 bits: n <= 2^30
    const Stencil s = stencil(P.g, xi.x, xi.y, xi.z, P.h);
    for (int cz = s.z0; cz <= s.z1; ++cz)
        for (int cy = s.y0; cy <= s.y1; ++cy) {
            const uint32_t row = linear_cell(P.g, 0, cy, cz);
            for (int cx = s.x0; cx <= s.x1; ++cx) {
                const uint2 r = __ldg(&cells[row + cx]);
                const uint32_t e = min(r.y, n);
                for (uint32_t j = r.x; j < e; ++j) {
                    const float4 xj = __ldg(&pos[j]);
                    float dx, dy, dz;
                    const float r2 = dist2(xi.x, xi.y, xi.z, xj.x, xj.y, xj.z, dx, dy, dz);
                    if (r2 < P.T) {
                        const float a = P.h2 - r2;
                        sum = fmaf(a * a, a, sum);
                        if (r2 != 0.0f) {
                            if (lists.holds(k)) __stcs(out, j);  // evict-first
                            out += (k & 3u) == 3u ? next_group : 1u;
                            ++k;
                        } else {
                            ++zero;
                        }
                    }
                }
            }
        }
    const float rh = P.dens_coef * sum;
    const float p = P.bulk * (rh - P.rho0);
    const float inv = 1.0f / rh;
    rho[i] = rh;
    aux[i] = make_float2(p * inv * inv, inv);
    xa[i] = make_float4(xi.x, xi.y, xi.z, p * inv * inv);
    reinterpret_cast<float*>(svel + i)[3] = inv;
    nbr_count[i] = lists.count(k);
    if (DEBUG) dbg_count[i] = k + zero;
}

template <bool DEBUG, class LISTS>
__global__ void __launch_bounds__(kDensityThreads) density_kernel(
    const float4* __restrict__ pos, const uint2* __restrict__ cells, uint32_t n, SimParams P,
    float* __restrict__ rho, float2* __restrict__ aux, uint4* __restrict__ nbr4,
    uint32_t* __restrict__ nbr_count, LISTS lists, uint32_t* __restrict__ dbg_count,
    float4* __restrict__ xa, float4* __restrict__ svel) {
    grid_wait();
    const uint32_t i = after_wait(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    density_one<DEBUG>(i, pos, cells, n, P, rho, aux, nbr4, nbr_count, lists, dbg_count, xa, svel);
}

// Below this many particles the density pass takes nine lanes to one: 4,096
// particles are 16 blocks otherwise, and the pass is one lane's chain of ~100
// candidates.  Us per step alone, and of three solvers in turn, one lane and nine:
// 4,096 particles 64 and 39, 25 and 17; 8,000 68 and 44, 27 and 20; 13,824 70 and
// 52, 28 and 25; 21,952 72 and 62, but 29 and 34: nine lanes are more work, which
// pays while the chip has room.  (The first hundred steps of a dam break.)
constexpr uint32_t kDensitySplitMost = 16384;
constexpr uint32_t kSplitLanes = 9, kSplitPer = 32 / kSplitLanes, kSplitWarps = 4;
// Neighbours that a lane keeps; one with more scans its share again, for the list
// and for the sum.  A lane has one row of three cells, which hold 27 each where
// particles lie closest: 39 us per step at 4,096 with 40, 43 with 24.
constexpr uint32_t kSplitHits = 40;

struct SplitScratch {  // of one warp
    float a[kSplitHits][32];
    uint32_t j[kSplitHits][32];
};

// The density pass with nine lanes to a particle, each scanning its share of the
// stencil's cell rows.  Lane 0 adds the terms in the scan's order, and the list is
// written in it: the results are density_one's bit for bit.  The neighbours
// of a lane that the scratch does not hold are found again.
template <bool DEBUG, class LISTS>
__global__ void __launch_bounds__(32 * kSplitWarps) density_split_kernel(
    const float4* __restrict__ pos, const uint2* __restrict__ cells, uint32_t n, SimParams P,
    float* __restrict__ rho, float2* __restrict__ aux, uint4* __restrict__ nbr4,
    uint32_t* __restrict__ nbr_count, LISTS lists, uint32_t* __restrict__ dbg_count,
    float4* __restrict__ xa, float4* __restrict__ svel) {
    constexpr uint32_t kAll = 0xFFFFFFFFu, L = kSplitLanes;
    __shared__ SplitScratch scratch[kSplitWarps];
    SplitScratch& S = scratch[threadIdx.x >> 5];
    grid_wait();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t g = lane / L, q = lane % L;
    const uint32_t i =
        after_wait((blockIdx.x * kSplitWarps + (threadIdx.x >> 5)) * kSplitPer + g);
    const bool on = g < kSplitPer && i < n;
    const float4 xi = pos[min(i, n - 1u)];
    uint32_t hits = 0, listed = 0;
    // f(j, r2) for the neighbours in lane l's share of the rows
    auto scan = [&](uint32_t l, auto&& f) {
        const Stencil s = stencil(P.g, xi.x, xi.y, xi.z, P.h);
        const int ny = s.y1 - s.y0 + 1, rows = ny * (s.z1 - s.z0 + 1);
        const int last = ((int)l + 1) * rows / (int)L;
        for (int r = (int)l * rows / (int)L; r < last; ++r) {
            const uint32_t row = linear_cell(P.g, 0, s.y0 + r % ny, s.z0 + r / ny);
            for (int cx = s.x0; cx <= s.x1; ++cx) {
                const uint2 c = __ldg(&cells[row + cx]);
                const uint32_t e = min(c.y, n);
                for (uint32_t j = c.x; j < e; ++j) {
                    const float4 xj = __ldg(&pos[j]);
                    float dx, dy, dz;
                    const float r2 = dist2(xi.x, xi.y, xi.z, xj.x, xj.y, xj.z, dx, dy, dz);
                    if (r2 < P.T) f(j, r2);
                }
            }
        }
    };
    if (on)
        scan(q, [&](uint32_t j, float r2) {
            if (hits < kSplitHits) {
                S.a[hits][lane] = P.h2 - r2;
                S.j[hits][lane] = r2 != 0.0f ? j : 0xFFFFFFFFu;  // not itself
            }
            ++hits;
            listed += r2 != 0.0f;
        });
    __syncwarp();
    uint32_t at = listed, all = hits;
#pragma unroll
    for (uint32_t d = 1; d < L; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, at, d), z = __shfl_up_sync(kAll, all, d);
        if (q >= d) {
            at += y;
            all += z;
        }
    }
    const int end = (int)min(L * g + L - 1u, 31u);
    const uint32_t total = __shfl_sync(kAll, at, end);
    all = __shfl_sync(kAll, all, end);
    at -= listed;
    if (on && lists.fits(total)) {  // a longer list is not read
        uint32_t k = at;
        uint32_t* out =
            reinterpret_cast<uint32_t*>(nbr4) + 4 * ((size_t)(k >> 2) * n + i) + (k & 3u);
        const uint32_t next_group = 4u * n - 3u;
        auto put = [&](uint32_t j) {
            __stcs(out, j);
            out += (k & 3u) == 3u ? next_group : 1u;
            ++k;
        };
        if (hits <= kSplitHits) {
            for (uint32_t t = 0; t < hits; ++t)
                if (S.j[t][lane] != 0xFFFFFFFFu) put(S.j[t][lane]);
        } else {
            scan(q, [&](uint32_t j, float r2) {
                if (r2 != 0.0f) put(j);
            });
        }
    }
    float sum = 0.0f;
#pragma unroll
    for (uint32_t l = 0; l < L; ++l) {
        const uint32_t from = min(L * g + l, 31u), m = __shfl_sync(kAll, hits, (int)from);
        if (on && q == 0) {
            if (m <= kSplitHits) {
#pragma unroll 4
                for (uint32_t t = 0; t < m; ++t) {
                    const float a = S.a[t][from];
                    sum = fmaf(a * a, a, sum);
                }
            } else {
                scan(l, [&](uint32_t, float r2) {
                    const float a = P.h2 - r2;
                    sum = fmaf(a * a, a, sum);
                });
            }
        }
    }
    if (!on || q != 0) return;
    const float rh = P.dens_coef * sum;
    const float p = P.bulk * (rh - P.rho0);
    const float inv = 1.0f / rh;
    rho[i] = rh;
    aux[i] = make_float2(p * inv * inv, inv);
    xa[i] = make_float4(xi.x, xi.y, xi.z, p * inv * inv);
    reinterpret_cast<float*>(svel + i)[3] = inv;
    nbr_count[i] = lists.count(total);
    if (DEBUG) dbg_count[i] = all;
}

}  // namespace sph
