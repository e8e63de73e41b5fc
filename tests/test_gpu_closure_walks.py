"""The feature and interpolation walks (two candidates at a time; four lanes to an
interpolation point) against 64-bit sums over all pairs: both kernels, planar and 3-D,
point counts at the edges of a block (32 points) and away from the particles; and a
candidate outside a particle's support adds nothing to it, whatever it holds.

Tolerances: a 64-bit sum of the same FP32 positions, densities and accelerations
differs from the walk by the rounding of a weight (about ten operations, each 2^-24 of
it, near the edge of the support 2^-22 of W(0)) and of a sum of at most 300 terms: under
1e-5 of the sum of the weights, and of that times the largest value.  A result of weights
below 1e-3 (a point that touches the fluid at the edge of its support) is not compared."""
import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi, presets

pytestmark = pytest.mark.gpu


def state(planar, kernel):
    if planar:
        p = presets.dambreak_params((24, 48, 1), 1, (96, 48, 4), 1.0 / 48)
        p.particle_mass = np.float32(float(p.particle_mass) * (128.0 / 24) ** 2)
        p.delta_time = np.float32(1e-4)
        s = cm.DamBreakSystem(params=p)
        s.reset()
    else:
        p, n, tank, layers = presets.dambreak3d(fluid=(9, 14, 7), tank=(20, 18, 7), layers=3, dt=1e-4, kernel=kernel)
        s = cm.DamBreakSystem(params=p, num_particles=n)
        s.scene3d(tank, layers, 0.05, 5)
    s.update_n(5)
    s.run_stages(_abi.STAGE_FORCE)
    return p, s


def weight(kernel, q, w_norm):
    if kernel == _abi.KERNEL_WENDLAND:
        return w_norm * (1 - q / 2) ** 4 * (2 * q + 1)
    return w_norm * np.where(q < 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2 - q) ** 3)


@pytest.mark.parametrize("planar,kernel", [(False, _abi.KERNEL_WENDLAND), (False, _abi.KERNEL_CUBIC_SPLINE),
                                           (True, _abi.KERNEL_WENDLAND)])
def test_interpolation(gpu, planar, kernel):
    import torch
    p, s = state(planar, kernel)
    pos, acc = s.getArray(cm.POSITION).astype(np.float64), s.getArray(cm.ACCELERATION).astype(np.float64)
    idx, meas = s.getUintArray(_abi.INDEX), s.getArray(cm.MEASURES)
    rho = np.empty(len(pos))
    rho[idx] = meas[:, 0]
    h = float(np.float32(p.smoothing_radius))
    if kernel == _abi.KERNEL_WENDLAND:
        w_norm = 7 / (4 * np.pi * h ** 2) if planar else 21 / (16 * np.pi * h ** 3)
    else:
        w_norm = 1 / (np.pi * h ** 3)
    fluid = np.flatnonzero(pos[:, 3] == _abi.FLUID)
    lo, hi = pos[fluid, :3].min(0) - 3 * h, pos[fluid, :3].max(0) + 3 * h
    if planar:
        lo[2] = hi[2] = pos[fluid[0], 2]
    for n in (1, 31, 32, 33, 500):
        rng = np.random.default_rng(n)
        pts = np.zeros((n, 4), np.float32)
        pts[:, :3] = rng.uniform(lo, hi, (n, 3))
        pts[0] = pos[fluid[len(fluid) // 2]]  # on a particle
        out = torch.full((n + 1, 4), 7.0, device="cuda")
        s.interpolate(_abi.ACCELERATION, torch.from_numpy(pts).cuda().data_ptr(), n, out.data_ptr())
        got = out.cpu().numpy()
        assert (got[n] == 7.0).all()
        for k in range(n):
            d = np.sqrt(((pos[fluid, :3] - pts[k, :3].astype(np.float64)) ** 2).sum(1))
            nb = np.flatnonzero(d < 2 * h)
            w = float(np.float32(p.particle_mass)) / rho[fluid[nb]] * weight(kernel, d[nb] / h, w_norm)
            a, sw = acc[fluid[nb], :3], w.sum()
            assert abs(got[k, 3] - sw) <= 1e-5 * max(sw, 1e-2)
            if sw > 1e-3:
                want = (w[:, None] * a).sum(0) / sw
                assert np.abs(got[k, :3] - want).max() <= 2e-5 * np.abs(a).max()
            elif sw == 0.0 and got[k, 3] == 0.0:
                assert (got[k] == 0.0).all()
    s.close()


def test_outside_the_support_adds_nothing(gpu):
    import torch
    p, s = state(False, _abi.KERNEL_WENDLAND)
    pos = s.getArray(cm.POSITION)
    h = float(np.float32(p.smoothing_radius))
    fluid = pos[:, 3] == _abi.FLUID
    bad = int(np.flatnonzero(fluid)[400])

    def features():
        s.run_stages(_abi.STAGE_FORCE)
        f = torch.full((len(pos), 16), 0.0, device="cuda")
        s.closure_features(f.data_ptr())
        return f.cpu().numpy()

    want = features()
    for value in (np.nan, np.inf):
        vel = s.getArray(cm.VELOCITYLEAPFROG)
        keep = vel.copy()
        vel[bad, :3] = value
        s.setArray(cm.VELOCITYLEAPFROG, vel)
        got = features()
        s.setArray(cm.VELOCITYLEAPFROG, keep)
        far = fluid & (np.linalg.norm(pos[:, :3] - pos[bad, :3], axis=1) > 2.001 * h)
        assert not np.isfinite(got[bad]).all()
        assert np.array_equal(got[far], want[far])
    s.close()
