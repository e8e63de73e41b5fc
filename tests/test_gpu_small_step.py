"""The three-launch step of small planar scenes (csrc/small_step.cu) against the staged
step (graphs off: one launch a stage): the same bits in every array, because both add
the same pair terms in the same order.  Sizes at the edges: a few particles, blocks
and warps that end inside a scene, rows that wrap, crowded rows (a column at rest
pressed into its corner, the parked gate on one point), the largest scene that takes
the path and the smallest that does not."""
import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi, presets

pytestmark = pytest.mark.gpu


def jittered(s, seed, amplitude=0.1):
    rng = np.random.default_rng(seed)
    p = s.params
    pos = s.getArray(cm.POSITION)
    fluid = pos[:, 3] == (_abi.FLUID if p.system == _abi.DAMBREAK else 0)
    dx = 2 * float(p.particle_radius)
    pos[fluid, :2] += (amplitude * dx * rng.uniform(-1, 1, (fluid.sum(), 2))).astype(np.float32)
    vel = np.zeros_like(pos)
    vel[fluid, :2] = (0.05 * float(p.soundspeed) * rng.normal(size=(fluid.sum(), 2))).astype(np.float32)
    vel[~fluid, 3] = 0.0
    s.setArrays({cm.POSITION: pos, cm.VELOCITY: vel, cm.VELOCITYLEAPFROG: (0.999 * vel).astype(np.float32)})


def dambreak(num, cut=False, gate=True):
    p = presets.dambreak_params((num, 2 * num, 1), 1, (4 * num, 2 * num, 4), 1.0 / (2 * num))
    p.particle_mass = np.float32(float(p.particle_mass) * (128.0 / num) ** 2)
    p.delta_time = np.float32(1e-4 * 64 / num)
    p.lj_cutoff = int(cut)
    s = cm.DamBreakSystem(params=p)
    s.reset()
    if gate:  # the gate's particles parked on one point
        s.removeRightBoundary()
    return s


def poiseuille(fx, fy, spline=False):
    r = 1.0 / (2 * fy * 1000)
    p = presets.poiseuille_params((fx, fy, 1), 3, (max(fx, 7), fy + 12, 4), r)
    p.particle_mass = np.float32(float(p.particle_mass) * (58.0 / fy) ** 2)
    if spline:
        p.kernel, p.smoothing_radius = _abi.KERNEL_CUBIC_SPLINE, np.float32(2.6 * r)
    s = cm.PoiseuilleFlowSystem(params=p)
    s.reset()
    return s


def peristalsis(fx, fy, released=True):
    p = presets.peristalsis_c3(fluid=(fx, fy))
    s = cm.PeristalsisSystem(params=p)
    s.reset()
    if released:
        p = s.params
        p.is_boundary_configuration = 0
        s.set_params(p)
    return s


def crowded(s):
    """Three particles to a cell: every row holds more candidates than its slots."""
    pos = s.getArray(cm.POSITION)
    fluid = pos[:, 3] == _abi.FLUID
    lo = pos[fluid, :2].min(0)
    pos[fluid, :2] = lo + (pos[fluid, :2] - lo) / np.float32(1.7)
    s.setArray(cm.POSITION, pos)
    return s


SCENES = {
    "dambreak 16": lambda: dambreak(16),
    "dambreak 64": lambda: dambreak(64),
    "dambreak 64 gate": lambda: dambreak(64, gate=False),
    "dambreak 64 cut": lambda: dambreak(64, cut=True),
    "dambreak 64 crowded": lambda: crowded(dambreak(64)),
    "dambreak 74": lambda: dambreak(74),   # 11,542 particles, and
    "dambreak 76": lambda: dambreak(76),   # 12,158: either side of 8 and 4 lanes
    "dambreak 86 cut": lambda: dambreak(86, cut=True),
    "dambreak 86 crowded": lambda: crowded(dambreak(86)),
    "dambreak 92": lambda: dambreak(92),   # 17,662 particles: of the largest
    "dambreak 94": lambda: dambreak(94),   # 18,422: staged
    "poiseuille 7x1": lambda: poiseuille(7, 1),
    "poiseuille 37x28": lambda: poiseuille(37, 28),
    "poiseuille 64x58": lambda: poiseuille(64, 58),
    "poiseuille 171x97": lambda: poiseuille(171, 97),
    "poiseuille spline 64x64": lambda: poiseuille(64, 64, True),
    "poiseuille spline 150x101": lambda: poiseuille(150, 101, True),
    "peristalsis 128x24": lambda: peristalsis(128, 24),
    "peristalsis 128x58": lambda: peristalsis(128, 58),
    "peristalsis 256x58 configuring": lambda: peristalsis(256, 58, False),
    "peristalsis 256x58": lambda: peristalsis(256, 58),
}


@pytest.mark.parametrize("lists", [0, 1])
@pytest.mark.parametrize("name", list(SCENES))
def test_three_launch_steps_equal_staged_steps(gpu, name, lists):
    a, b = SCENES[name](), SCENES[name]()
    b.set_graphs(False)
    for s in (a, b):
        jittered(s, 11)
        if lists:
            s.set_neighbor_lists(True)
    for calls in (lambda s: s.update(), lambda s: s.update_n(7), lambda s: s.update(0.5 * float(s.params.delta_time))):
        calls(a)
        calls(b)
        a.synchronize()
        b.synchronize()
        x, y = a.state(), b.state()
        for k in x:
            assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), (name, k)
    assert a.getElapsedTime() == b.getElapsedTime()
    # the staged step continues where the three-launch steps ended, and back
    a.set_graphs(False)
    a.update()
    b.set_graphs(True)
    b.update()
    x, y = a.state(), b.state()
    for k in x:
        assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), (name, k)


@pytest.mark.parametrize("make,one_lane", [(lambda: poiseuille(64, 64), True), (lambda: dambreak(64), True),
                                           (lambda: poiseuille(160, 100), None)])
def test_autotuned_scene(gpu, make, one_lane):
    """The autotuner keeps one lane where the three launches are the fastest step, and
    what it then steps has the untuned system's bits."""
    a, b = make(), make()
    for s in (a, b):
        jittered(s, 4)
    lanes = tuple(b.autotune(2))
    if one_lane:
        assert lanes == (1, 1, False)
    a.update_n(20)
    b.update_n(20)
    if lanes == (1, 1, False):
        for array in (cm.POSITION, cm.VELOCITY, cm.MEASURES):
            assert np.array_equal(a.getArray(array), b.getArray(array))
    a.close()
    b.close()
