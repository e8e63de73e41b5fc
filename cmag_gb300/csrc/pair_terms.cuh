// pair_terms.cuh -- the force of one candidate pair, without branches on its distance,
// for the three-launch step of small planar scenes (small_step.cu).  Every particle of such
// a scene has the same z and no z velocity, so each z term is an exact zero and is left out.
//
// The same operations as the scalar pair of the force pass (force.cu), so that terms
// added in the same order give the same bits.  The force pass keeps its own form,
// which reads a neighbour's velocity and aux data only after the distance test: a
// shared function cost it 2.3 % (2-D dam break, 528,382 particles, 163.1 -> 166.9 us).
#pragma once

#include "neighbor_walk.cuh"

namespace cmag {

// What the pairs of one particle have in common.
struct PairSelf {
    uint32_t i;
    float4 pos, vel;
    float2 aux;    // p/rho^2, and rho (DamBreak) or 1/rho
    float nmass;   // -mass: pressure factor
    float visc_i;  // viscous factor of the particle
    bool lists;    // take the pairs that interaction lists hold
};

// DamBreak: sum += a r.  Poiseuille: sum += a r, then b v.  Peristalsis: pressure
// sum += a r, viscous sum += b v.
struct PairTerms {
    float a, rx, ry;
    float b, vx, vy;
};

// Lennard-Jones wall force over r (fluid_kernel.cu:199-207).
__device__ __forceinline__ float wall_factor(const DevParams &p, float d2)
{
    const float inv_d2 = __frcp_rn(d2);
    const float a2 = p.lj_a2 * inv_d2;
    const float a6 = a2 * a2 * a2;
    return p.lj_D * __fmaf_rn(a6, a6, -a6) * inv_d2;
}

// The terms of an interacting fluid pair (Poiseuille, Peristalsis: any pair) at
// distance (t.rx, t.ry), squared d2, from candidate values pj, vj, aj.
template <int SYS>
__device__ __forceinline__ void pair_factors(const DevParams &p, const PairSelf &s, const float4 &pj, float d2,
                                             const float4 &vj, const float2 &aj, PairTerms &t)
{
    const float inv_d = rsqrtf(d2);
    const float g = kernel_dw_over_r(p, d2 * inv_d, inv_d);  // dW/dr / r
    if (SYS == CMAG_DAMBREAK) {
        // pressure + Monaghan viscosity (fluid_kernel.cu:221-237)
        float q = s.aux.x + aj.x;
        const float vij = __fmaf_rn(s.vel.y - vj.y, t.ry, (s.vel.x - vj.x) * t.rx);
        if (vij < 0.0f) {
            // viscosity 2 alpha h c0 v_ij / ((rho_i + rho_j)(r^2 + eps^2))
            q -= __fdividef(p.av_coeff * vij, (s.aux.y + aj.y) * (d2 + p.av_eps2));
        }
        t.a = q * (s.nmass * g);
        return;
    }
    t.vx = s.vel.x - vj.x;
    t.vy = s.vel.y - vj.y;
    if (SYS == CMAG_POISEUILLE && pj.w == 1.0f && (pj.y > p.wall_top || pj.y < p.wall_bottom)) {
        // Morris viscosity with wall extrapolation (poiseuilleFlowKernel.cu:184-208)
        const bool top = pj.y > p.wall_top;
        const float da = top ? p.wall_top - s.pos.y : s.pos.y - p.wall_bottom;
        const float db = top ? pj.y - p.wall_top : p.wall_bottom - pj.y;
        const float beta = fminf(1000.0f, 1.0f + __fdividef(db, da));
        t.vx = beta * s.vel.x;
        t.vy = beta * s.vel.y;
    }
    // pressure (poiseuilleFlowKernel.cu:236-245, PeristalsisPressureForce.cu:39-43)
    // and viscous (PeristalsisViscousForce.cu:206-213) factors
    t.a = s.nmass * g * (s.aux.x + aj.x);
    t.b = s.visc_i * aj.y * g;
}

// Squared distance of the particle from candidate pj seen through image shift (sx, sy);
// the relative position in t.
template <int SYS>
__device__ __forceinline__ float pair_distance(const PairSelf &s, const float4 &pj, float sx, float sy, PairTerms &t)
{
    const float3 rv = walk::rel<SYS>(s.pos, pj, sx, sy, 0.0f);
    t.rx = rv.x;
    t.ry = rv.y;
    return __fmaf_rn(t.ry, t.ry, t.rx * t.rx);
}

// The terms of candidate j with its position, velocity and aux data at hand (loaded
// together, so that several candidates' loads are in flight); zeros and false when
// the pair contributes nothing.
template <int SYS, bool TRIM>
__device__ __forceinline__ bool pair_terms(const DevParams &p, const PairSelf &s, uint32_t j, const float4 &pj,
                                           const float4 &vj, const float2 &aj, float sx, float sy, PairTerms &t)
{
    const float d2 = pair_distance<SYS>(s, pj, sx, sy, t);
    // (a coincident pair has no direction: it contributes nothing)
    const bool wall = SYS == CMAG_DAMBREAK && pj.w != (float)CMAG_FLUID;
    // a wall without cut-off at a distance that is not a number: the walk takes it, lists
    // do not hold it
    const bool hit = j != s.i && d2 != 0.0f && (d2 < p.support2 || (wall && !TRIM && (!s.lists || d2 > 0.0f)));
    pair_factors<SYS>(p, s, pj, d2, vj, aj, t);
    if (wall) t.a = wall_factor(p, d2);
    if (!hit) t = PairTerms{};
    return hit;
}

}  // namespace cmag
