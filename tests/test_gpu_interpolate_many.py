"""Interpolation at more than 2^30 points in one call: every point gets its own result.
The points repeat a pattern of a prime length, so a result that lands at another point, or
a point that is left out, shows.  Needs 36 GB of device memory for points and results."""
import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi, presets

pytestmark = pytest.mark.gpu


def test_more_than_a_billion_points(gpu):
    import torch
    n = (1 << 30) + 12345
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("needs 48 GB of free device memory")
    p = presets.dambreak_params((24, 48, 1), 1, (96, 48, 4), 1.0 / 48)
    p.particle_mass = np.float32(float(p.particle_mass) * (128.0 / 24) ** 2)
    p.delta_time = np.float32(1e-4)
    s = cm.DamBreakSystem(params=p)
    s.reset()
    s.update_n(5)
    s.run_stages(_abi.STAGE_FORCE)
    pos = s.getArray(cm.POSITION)
    fluid = np.flatnonzero(pos[:, 3] == _abi.FLUID)
    rng = np.random.default_rng(3)
    period = 65521
    few = np.zeros((period, 4), np.float32)
    few[:, 2] = pos[fluid[0], 2]
    far = pos[:, :2].max(0) + 10 * float(p.smoothing_radius)
    few[:, :2] = far  # most lie away from the fluid: quick
    few[::16, :2] = rng.uniform(pos[fluid, :2].min(0), pos[fluid, :2].max(0), (len(few[::16]), 2))
    few = torch.from_numpy(few).cuda()
    want = torch.full((period, 4), 7.0, device="cuda")
    s.interpolate(_abi.ACCELERATION, few.data_ptr(), period, want.data_ptr())
    assert bool((want[::16, 3] > 0).any())
    points = torch.empty((n, 4), device="cuda")
    whole = n // period
    points[:whole * period].view(whole, period, 4)[:] = few
    points[whole * period:] = few[:n - whole * period]
    out = torch.full((n, 4), 7.0, device="cuda")
    torch.cuda.synchronize()
    s.interpolate(_abi.ACCELERATION, points.data_ptr(), n, out.data_ptr())
    del points
    for k in range(0, whole, 256):  # in pieces: little further memory
        part = out[k * period:min(k + 256, whole) * period].view(-1, period, 4)
        assert bool((part == want).all())
    assert bool((out[whole * period:] == want[:n - whole * period]).all())
    s.close()
    del out
    torch.cuda.empty_cache()
