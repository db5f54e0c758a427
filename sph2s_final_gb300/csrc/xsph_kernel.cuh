// xsph_kernel.cuh -- the XSPH integrator variant of the single-scale step.
//
// integrateXSPHD + computeVelXSPHCell (SPH2S_FINAL_SINGLE_SCALE/Solver.cu:
// 345-395, 757-853; its launch is commented out in Solver::Advance,
// Solver.cu:1185-1196):
//   v'_i  = v_i + dt a_i
//   dv_i  = sum_{j: r_ij < h} (v'_j - v'_i) m / rho_j W_poly6(r_ij)
//   v''_i = v'_i + eps dv_i        (per component; the reference adds dv.x to
//                                   all three components, fixed here)
//   x'_i  = x_i + dt v''_i
// v'' is stored as the new velocity.  The self term vanishes (v'_i - v'_i is
// exactly 0); neighbours come from the density pass's list (0 < r < h), the
// force pass having written (v'_i, 1/rho_i), so that a neighbour costs two
// 16-byte gathers (what bounds the pass is their latency; with position, 1/rho,
// velocity and three accelerations it was six, and the whole step of 65,536
// particles took 78 us with three solvers side by side against 54 now, of which
// the boundary scan inside the force pass was most: it now has its own pass
// beside density, as in the Euler step); partners at distance 0 other than i itself
// (flagged by the density pass's full count) are picked up from the home
// cell, and particles whose list overflowed rescan the stencil.
#pragma once
#include "common.cuh"

namespace sph {

struct XsphAcc {
    float x = 0.f, y = 0.f, z = 0.f;
};

// vj: (v'_j, 1 / rho_j)
__device__ __forceinline__ void xsph_pair(XsphAcc& S, const SimParams& P, float r2,
                                          const float4& vi, const float4& vj) {
    const float a = P.h2 - r2;
    const float w = a * a * a * vj.w;
    S.x = fmaf(vj.x - vi.x, w, S.x);
    S.y = fmaf(vj.y - vi.y, w, S.y);
    S.z = fmaf(vj.z - vi.z, w, S.z);
}

static __global__ void __launch_bounds__(256) xsph_integrate_kernel(
    const float4* __restrict__ pos, const float4* __restrict__ vel1,
    const uint2* __restrict__ cells, const uint4* __restrict__ nbr4,
    const uint32_t* __restrict__ nbr_count, const uint32_t* __restrict__ nbr_all, uint32_t n,
    SimParams P, float dt, float eps, float4* __restrict__ pos_out, float4* __restrict__ vel_out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 xi = pos[i];
    const float4 vi = vel1[i];  // (v', 1 / rho)
    XsphAcc S;
    const uint32_t kc = nbr_count[i];
    if (kc <= (uint32_t)kMaxNbr) {
        for (uint32_t t = 0; t < kc; t += 4) {
            const uint4 g = __ldg(&nbr4[(size_t)(t >> 2) * n + i]);
            const uint32_t js[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (t + u < kc) {
                    const uint32_t j = min(js[u], n - 1);
                    const float4 xj = __ldg(&pos[j]);
                    float dx, dy, dz;
                    const float r2 = dist2(xi.x, xi.y, xi.z, xj.x, xj.y, xj.z, dx, dy, dz);
                    xsph_pair(S, P, r2, vi, __ldg(&vel1[j]));
                }
            }
        }
        if (nbr_all[i] > kc + 1u) {  // coincident partners: same position, same cell
            const uint32_t home = linear_cell(P.g, cell_coord(xi.x, P.g.ox, P.g.spacing, P.g.dx),
                                              cell_coord(xi.y, P.g.oy, P.g.spacing, P.g.dy),
                                              cell_coord(xi.z, P.g.oz, P.g.spacing, P.g.dz));
            const uint2 r = __ldg(&cells[home]);
            const uint32_t e = min(r.y, n);
            for (uint32_t j = r.x; j < e; ++j) {
                const float4 xj = __ldg(&pos[j]);
                float dx, dy, dz;
                const float r2 = dist2(xi.x, xi.y, xi.z, xj.x, xj.y, xj.z, dx, dy, dz);
                if (j != i && r2 == 0.0f)
                    xsph_pair(S, P, r2, vi, __ldg(&vel1[j]));
            }
        }
    } else {
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
                        if (r2 < P.T && j != i)
                            xsph_pair(S, P, r2, vi, __ldg(&vel1[j]));
                    }
                }
            }
    }
    const float c = eps * P.dens_coef;  // dens_coef = m * 315 / (64 pi h^9)
    const float nvx = fmaf(c, S.x, vi.x), nvy = fmaf(c, S.y, vi.y), nvz = fmaf(c, S.z, vi.z);
    pos_out[i] = make_float4(fmaf(dt, nvx, xi.x), fmaf(dt, nvy, xi.y), fmaf(dt, nvz, xi.z), xi.w);
    vel_out[i] = make_float4(nvx, nvy, nvz, 0.0f);
}

}  // namespace sph
