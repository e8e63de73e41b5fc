"""Several host threads query one dam-break system at once (interpolation of different
arrays at different points, closure features): every call gives what it gives alone,
although the calls share the system's stream and scratch."""
import threading

import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi, presets

pytestmark = pytest.mark.gpu


def test_queries_from_several_threads(gpu):
    import torch
    p, n, tank, layers = presets.dambreak3d(fluid=(9, 14, 7), tank=(20, 18, 7), layers=3, dt=1e-4)
    s = cm.DamBreakSystem(params=p, num_particles=n)
    s.scene3d(tank, layers, 0.05, 5)
    s.update_n(5)
    s.run_stages(_abi.STAGE_FORCE)
    pos = s.getArray(cm.POSITION)
    fluid = pos[:, 3] == _abi.FLUID
    lo, hi = pos[fluid, :3].min(0), pos[fluid, :3].max(0)
    arrays = (_abi.ACCELERATION, _abi.VELOCITY, _abi.POSITION, _abi.VELOCITYLEAPFROG)
    calls = []
    for k, array in enumerate(arrays):
        m = 100 + 57 * k
        pts = np.zeros((m, 4), np.float32)
        pts[:, :3] = np.random.default_rng(k).uniform(lo, hi, (m, 3))
        pts = torch.from_numpy(pts).cuda()
        calls.append((torch.zeros((m, 4), device="cuda"),
                      lambda out, array=array, pts=pts, m=m: s.interpolate(array, pts.data_ptr(), m, out.data_ptr())))
    calls.append((torch.zeros((n, 16), device="cuda"), lambda out: s.closure_features(out.data_ptr())))
    torch.cuda.synchronize()
    want = []
    for out, call in calls:
        call(out)
        want.append(out.clone())
    torch.cuda.synchronize()
    start = threading.Barrier(len(calls))
    wrong = []

    def work(k):
        out, call = calls[k]
        start.wait()
        for _ in range(300):
            call(out)  # returns when its result is there
            if not np.array_equal(out.cpu().numpy(), expect[k]):
                wrong.append(k)

    expect = [w.cpu().numpy() for w in want]
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, "%d results differ" % len(wrong)
    s.close()
