// particle_motion.cuh -- time integration of one particle and the Peristalsis
// phase machine, shared by the integration kernels (integrate.cu) and the
// three-launch step of small scenes (small_step.cu).
//
//   integrate                    DamBreak.Core/fluid_kernel.cu:323-366
//   integratePoiseuilleSystemD   Poiseuille.Core/poiseuilleFlowKernel.cu:311-348
//   computeCoordinatesD          Peristalsis.Core/PeristalsisIntegrate.cu:1-66
#pragma once

#include "sph_common.cuh"

namespace cmag {

// The phase block after one boundary-configuration phase, exactly as the host
// mirror advances it (separately rounded adds and multiplies, no contraction).
__device__ __forceinline__ PhaseState next_phase(const DevParams &p, PhaseState s, float k_milli)
{
    s.configure = 0;
    if (s.is_bc) {
        s.time_shift = __fadd_rn(s.time_shift, p.dt);
        if (s.wave_height < p.amplitude) {
            s.configure = 1;
            s.configure_height = s.wave_height;
            s.wave_height = __fadd_rn(s.wave_height, __fmul_rn(p.dt, k_milli));
        } else {
            s.time_relax = __fsub_rn(s.time_relax, p.dt);
            if (s.time_relax < 0.0f) s.is_bc = 0;
        }
    }
    s.t = s.is_bc ? 0.0f : __fsub_rn(s.elapsed, s.time_shift);
    s.elapsed = __fadd_rn(s.elapsed, p.dt);
    return s;
}

// A Peristalsis wall particle (q.w != 0) on the moving wall at time t; false while
// the boundary is being configured (walls frozen).
__device__ __forceinline__ bool move_wall(const DevParams &p, int is_bc, float t, float4 &q)
{
    if (is_bc) return false;
    const float wave = get_wave(p, q.x, t);
    if (q.w > 0.0f) q.y = -p.half_fluid_h + p.amplitude * wave - p.r * (q.w - 1.0f);
    else q.y = p.half_fluid_h - p.amplitude * wave + p.r * (-q.w - 1.0f);
    return true;
}

// Position, velocity and leap-frog velocity of a fluid particle after a step with
// acceleration a (gravity added here), with the family's walls and periodic ends.
__device__ __forceinline__ void integrate_fluid(const DevParams &p, float ax, float ay, float az,
                                                float4 &q, float4 &v, float4 &lf)
{
    const float nvx = v.x + (p.gvx + ax) * p.dt;
    const float nvy = v.y + (p.gvy + ay) * p.dt;
    const float nvz = v.z + (p.gvz + az) * p.dt;
    lf = make_float4((v.x + nvx) * 0.5f, (v.y + nvy) * 0.5f, (v.z + nvz) * 0.5f, lf.w);
    v.x = nvx; v.y = nvy; v.z = nvz;
    q.x += v.x * p.dt; q.y += v.y * p.dt; q.z += v.z * p.dt;
    if (p.system == CMAG_DAMBREAK) {
        if (q.x < p.left_border) { q.x = p.left_border; v.x *= p.damping; }
        if (q.x > p.right_boundary) { q.x = p.right_boundary; v.x *= p.damping; }
        if (q.y < p.bottom_border) { q.y = p.bottom_border; v.y *= p.damping; }
        if (p.clamp_z) {
            if (q.z < p.z_min_border) { q.z = p.z_min_border; v.z *= p.damping; }
            if (q.z > p.z_max_border) { q.z = p.z_max_border; v.z *= p.damping; }
        }
    } else {
        if (q.x > p.half_world_x) q.x -= 2.0f * p.half_world_x;
        if (p.system == CMAG_PERISTALSIS && q.x < -p.half_world_x) q.x += 2.0f * p.half_world_x;
    }
}

}  // namespace cmag
