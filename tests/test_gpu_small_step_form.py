"""Which scenes take the step of three launches, and that step where rows are crowded.

The form is asked of the library, so that a comparison with the staged step does not
compare the staged step with itself.  Crowded rows: the fluid pressed together towards the
periodic ends (or the far corner of a dam break), until a row holds more terms than its
slots, then more candidates than one lane takes; for both kernels and on either side of
the line between 8 and 4 lanes."""
import ctypes

import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi
from cmag_gb300._lib import lib
from test_gpu_small_step import SCENES, dambreak, jittered, peristalsis, poiseuille

pytestmark = pytest.mark.gpu


def blocks(s):
    b = ctypes.c_uint32(99)
    assert lib().cmag_testing_small_step_blocks(s._h, ctypes.byref(b)) == 0
    return b.value


@pytest.mark.parametrize("name", list(SCENES))
def test_form(gpu, name):
    s = SCENES[name]()
    want = s.getNumParticles() <= 18000
    assert want == (name != "dambreak 94")
    assert (blocks(s) >= 8) == want and (blocks(s) == 0) == (not want)
    s.set_graphs(False)
    assert blocks(s) == 0
    s.set_graphs(True)
    s.set_groups(2, 1)
    assert blocks(s) == 0
    s.close()


@pytest.mark.parametrize("fx,n", [(180, 18000), (181, 18100)])
def test_form_at_the_limit(gpu, fx, n):
    a, b = poiseuille(fx, 94), poiseuille(fx, 94)
    assert a.getNumParticles() == n
    assert (blocks(a) > 0) == (n <= 18000)
    b.set_graphs(False)
    assert blocks(b) == 0
    for s in (a, b):
        jittered(s, 3)
        s.update_n(3)
    x, y = a.state(), b.state()
    for k in x:
        assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), k
    a.close()
    b.close()


def press(s, factor):
    """Fluid pressed towards x = -L and x = L (dam break: its lowest corner), and 1.5 in y."""
    p = s.params
    pos = s.getArray(cm.POSITION)
    fluid = pos[:, 3] == (_abi.FLUID if p.system == _abi.DAMBREAK else 0)
    x, y = pos[fluid, 0].astype(np.float64), pos[fluid, 1].astype(np.float64)
    if p.system == _abi.DAMBREAK:
        x = x.min() + (x - x.min()) / factor
    else:
        end = float(s.getHalfWorldXSize()) if p.system == _abi.POISEUILLE else np.abs(x).max() * 1.0001
        x = np.where(x < 0, -end + (x + end) / factor, end - (end - x) / factor)
    pos[fluid, 0], pos[fluid, 1] = x.astype(np.float32), (y.min() + (y - y.min()) / 1.5).astype(np.float32)
    s.setArray(cm.POSITION, pos)


def longest_row(s):
    """Most particles in 2 c + 1 neighbouring cells of a row (wrapped) of the layer."""
    p = s.params
    c, (gx, gy, gz) = int(p.cell_count), tuple(p.grid_size)
    cells = np.bincount(s.getUintArray(_abi.HASH), minlength=gx * gy * gz).reshape(gz, gy, gx).max(0)
    return int(sum(np.roll(cells, k, 1) for k in range(-c, c + 1)).max())


@pytest.mark.parametrize("lists", [0, 1])
@pytest.mark.parametrize("factor,least,most", [(2.0, 16, 32), (6.0, 33, 10000)])
@pytest.mark.parametrize("name,make", [
    ("poiseuille 64x58", lambda: poiseuille(64, 58)),
    ("poiseuille 171x97", lambda: poiseuille(171, 97)),
    ("poiseuille spline 64x64", lambda: poiseuille(64, 64, True)),
    ("poiseuille spline 150x101", lambda: poiseuille(150, 101, True)),
    ("peristalsis 128x24", lambda: peristalsis(128, 24)),
    ("peristalsis 256x58", lambda: peristalsis(256, 58)),
    ("dambreak 64 cut", lambda: dambreak(64, cut=True, gate=False)),
    ("dambreak 86", lambda: dambreak(86, gate=False)),
])
def test_crowded_rows_equal_staged_steps(gpu, name, make, factor, least, most, lists):
    a, b = make(), make()
    b.set_graphs(False)
    for s in (a, b):
        jittered(s, 8)
        press(s, factor)
        if lists:
            s.set_neighbor_lists(True)
    assert blocks(a) > 0 and blocks(b) == 0
    for step in range(2):
        a.update()
        b.update()
        if step == 0:
            assert least <= longest_row(a) <= most, longest_row(a)
        x, y = a.state(), b.state()
        for k in x:
            assert np.array_equal(x[k], y[k], equal_nan=x[k].dtype == np.float32), (name, step, k)
            if step == 0:
                assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), (name, k)
    a.close()
    b.close()


def test_autotuned_scene_of_the_chosen_lanes(gpu):
    """Above the size where the autotuner leaves one lane, its choice steps like a system
    set to it."""
    a, b = poiseuille(160, 100), poiseuille(160, 100)
    for s in (a, b):
        jittered(s, 4)
    density, force, lists = b.autotune(2)
    a.set_groups(density, force)
    a.set_neighbor_lists(lists)
    assert blocks(a) == blocks(b)
    a.update_n(20)
    b.update_n(20)
    for array in (cm.POSITION, cm.VELOCITY, cm.MEASURES):
        assert np.array_equal(a.getArray(array).view(np.uint32), b.getArray(array).view(np.uint32))
    a.close()
    b.close()
