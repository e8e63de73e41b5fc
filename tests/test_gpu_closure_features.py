"""The 16 closure features against 64-bit sums over all pairs, for both kernels, planar and
3-D (the pair walk takes two candidates at a time and evaluates each kernel in its own
form); and the interpolation next to a particle that holds NaN or infinity.

Tolerances: a 64-bit sum of the same FP32 positions, velocities and densities differs from
the walk's by the rounding of about ten operations in each term (2^-24 each: under 1e-6 of
the sum of the terms' magnitudes, with the sum's own 150 additions under 1e-5) and, near
the edge of the support where a weight is a small difference, by 2^-22 of the largest
weight in each of the candidates: 2^-20 allows for its later operations."""
import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi, presets
from test_gpu_closure_walks import state

pytestmark = pytest.mark.gpu

CASES = [(False, _abi.KERNEL_WENDLAND), (False, _abi.KERNEL_CUBIC_SPLINE), (True, _abi.KERNEL_WENDLAND),
         (True, _abi.KERNEL_CUBIC_SPLINE)]


def scene(planar, kernel):
    if not (planar and kernel == _abi.KERNEL_CUBIC_SPLINE):
        return state(planar, kernel)
    p = presets.dambreak_params((24, 48, 1), 1, (96, 48, 4), 1.0 / 48)
    p.particle_mass = np.float32(float(p.particle_mass) * (128.0 / 24) ** 2)
    p.delta_time = np.float32(1e-4)
    p.kernel = kernel
    s = cm.DamBreakSystem(params=p)
    s.reset()
    s.update_n(5)
    s.run_stages(_abi.STAGE_FORCE)
    return p, s


def kernels(planar, kernel, h):
    if kernel == _abi.KERNEL_WENDLAND:
        wn = 7 / (4 * np.pi * h ** 2) if planar else 21 / (16 * np.pi * h ** 3)
        return (wn, 2 * wn / h, lambda q: wn * (1 - q / 2) ** 4 * (2 * q + 1),
                lambda q: -5 * wn / h * q * (1 - q / 2) ** 3)
    wn = 10 / (7 * np.pi * h ** 2) if planar else 1 / (np.pi * h ** 3)
    return (wn, wn / h, lambda q: wn * np.where(q < 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2 - q) ** 3),
            lambda q: wn / h * np.where(q < 1, -3 * q + 2.25 * q ** 2, -0.75 * (2 - q) ** 2))


@pytest.mark.parametrize("planar,kernel", CASES)
def test_features(gpu, planar, kernel):
    import torch
    p, s = scene(planar, kernel)
    n = s.getNumParticles()
    pos, vel = (s.getArray(a).astype(np.float64) for a in (cm.POSITION, cm.VELOCITYLEAPFROG))
    acc, meas, idx = s.getArray(cm.ACCELERATION).astype(np.float64), s.getArray(cm.MEASURES), s.getUintArray(_abi.INDEX)
    rho, pres = np.empty(n), np.empty(n)
    rho[idx], pres[idx] = meas[:, 0], meas[:, 1]
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    h, mass, c0, rho0, B = f32(p.smoothing_radius), f32(p.particle_mass), f32(p.soundspeed), f32(p.rest_density), f32(p.B)
    w_max, dw_max, w_of, dw_of = kernels(planar, kernel, h)
    g = np.linalg.norm([p.gravity[0], p.gravity[1], p.gravity[2]])
    out = torch.full((n + 1, 16), 7.0, device="cuda")
    torch.cuda.synchronize()
    s.closure_features(out.data_ptr())
    got = out.cpu().numpy().astype(np.float64)
    assert (got[n] == 7.0).all()
    fluid = np.flatnonzero(pos[:, 3] == _abi.FLUID)
    wall = pos[:, 3] != _abi.FLUID
    assert (got[:n][wall] == 7.0).all()  # walls are left alone
    walls_seen = 0
    for i in fluid[:: max(1, len(fluid) // 300)]:
        r = pos[:, :3] - pos[i, :3]
        d = np.sqrt((r * r).sum(1))
        nb = np.flatnonzero(d < 2 * h)
        r, d, vol, dv = r[nb], d[nb], mass / rho[nb], vel[nb, :3] - vel[i, :3]
        walls_seen += int(wall[nb].sum())
        q = d / h
        vw = vol * w_of(q)
        floor = len(nb) * 2.0 ** -20 * vol.max() * w_max

        def near(k, terms, scale, factor):
            """Feature k is scale * sum of the terms; factor: a term over its weight."""
            tol = scale * (1e-5 * np.abs(terms).sum() + floor * np.abs(factor).max())
            assert abs(got[i, k] - scale * terms.sum()) <= tol, (i, k, got[i, k], scale * terms.sum(), tol)

        for a in range(3):
            near(2 + a, vw * r[:, a], 1 / h, r[:, a])
            near(5 + a, vw * dv[:, a], 1 / c0, dv[:, a])
            assert abs(got[i, 11 + a] - acc[i, a] / g) <= 1e-6 * np.linalg.norm(acc[i, :3]) / g
        near(8, vw, 1.0, np.ones(1))
        near(9, vw * d ** 2, 1 / h ** 2, d ** 2)
        near(10, vw * wall[nb], 1.0, np.ones(1))
        nz = d > 0
        dot = (dv[nz] * r[nz]).sum(1)
        terms = -vol[nz] * dw_of(q[nz]) / d[nz] * dot
        speed = np.linalg.norm(dv, axis=1).max()
        tol = h / c0 * (1e-5 * np.abs(terms).sum() + 1e-5 * (vol[nz] * np.abs(dw_of(q[nz]))).sum() * speed
                        + len(nb) * 2.0 ** -20 * vol.max() * dw_max * speed)
        assert abs(got[i, 14] - h / c0 * terms.sum()) <= tol, (i, got[i, 14], h / c0 * terms.sum(), tol)
        assert abs(got[i, 0] - (rho[i] / rho0 - 1)) <= 2.0 ** -22 * rho[i] / rho0
        assert abs(got[i, 1] - pres[i] / B) <= 1e-6 * abs(pres[i] / B)
        assert abs(got[i, 15] - np.linalg.norm(vel[i, :3]) / c0) <= 1e-6 * np.linalg.norm(vel[i, :3]) / c0
    assert walls_seen > 0
    s.close()


@pytest.mark.parametrize("planar,kernel", CASES)
def test_interpolation_outside_the_support_adds_nothing(gpu, planar, kernel):
    import torch
    p, s = scene(planar, kernel)
    pos = s.getArray(cm.POSITION)
    h = float(np.float32(p.smoothing_radius))
    fluid = np.flatnonzero(pos[:, 3] == _abi.FLUID)
    bad = int(fluid[len(fluid) // 2])
    pts = pos[fluid].copy()
    points = torch.from_numpy(pts).cuda()

    def interpolated():
        out = torch.full((len(pts), 4), 7.0, device="cuda")
        torch.cuda.synchronize()
        s.interpolate(_abi.VELOCITY, points.data_ptr(), len(pts), out.data_ptr())
        return out.cpu().numpy()

    want = interpolated()
    far = np.linalg.norm(pts[:, :3] - pos[bad, :3], axis=1) > 2.001 * h
    vel = s.getArray(cm.VELOCITY)
    for value in (np.nan, np.inf):
        holds = vel.copy()
        holds[bad, :2] = value
        s.setArray(cm.VELOCITY, holds)
        got = interpolated()
        assert np.array_equal(got[far].view(np.uint32), want[far].view(np.uint32))
        assert not np.isfinite(got[pts[:, :3].tolist().index(pos[bad, :3].tolist()), :2]).any()
    s.close()
