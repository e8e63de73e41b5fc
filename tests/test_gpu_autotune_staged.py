"""What the autotuner finds for the staged step of a small scene is used when its steps
become staged, and one lane again when they are three launches."""
import numpy as np
import pytest

import cmag_gb300 as cm
from test_gpu_small_step import jittered, poiseuille

pytestmark = pytest.mark.gpu

ARRAYS = (cm.POSITION, cm.VELOCITY, cm.MEASURES)


def lanes(s):
    return s.groups() + (s.neighbor_lists()[0],)


def same(a, b):
    for array in ARRAYS:
        assert np.array_equal(a.getArray(array).view(np.uint32), b.getArray(array).view(np.uint32))


def staged(s, on, how):
    if how == "graphs":
        s.set_graphs(not on)
    else:
        s.set_stage_timing(on)


@pytest.mark.parametrize("how", ["graphs", "timing"])
def test_tuned_lanes_of_staged_steps(gpu, how):
    a, b = poiseuille(64, 64), poiseuille(64, 64)
    for s in (a, b):
        jittered(s, 4)
    # one thread a particle leaves most of the GPU idle here: several lanes, or lists, win
    assert a.autotune(5) == (1, 1, False)
    staged(a, True, how)
    a.update_n(3)
    found = lanes(a)
    assert found != (1, 1, False)
    b.set_groups(*found[:2])
    b.set_neighbor_lists(found[2])
    b.set_graphs(False)
    b.update_n(3)
    same(a, b)
    staged(a, False, how)
    a.update_n(3)
    assert lanes(a) == (1, 1, False)
    b.set_groups(1, 1)
    b.set_neighbor_lists(False)
    b.update_n(3)
    same(a, b)
    staged(a, True, how)
    a.update()
    assert lanes(a) == found
    a.close()
    b.close()


def test_chosen_lanes_stay(gpu):
    """Lanes or lists that the user sets after autotuning are not replaced."""
    for choose, want in ((lambda s: s.set_groups(1, 1), (1, 1, False)), (lambda s: s.set_groups(2, 1), (2, 1, False)),
                         (lambda s: s.set_neighbor_lists(True), (1, 1, True))):
        s = poiseuille(64, 64)
        s.autotune(3)
        choose(s)
        s.set_graphs(False)
        s.update()
        assert lanes(s) == want
        s.close()


def test_kept_lists_after_autotuning(gpu):
    """Lists kept over steps are not touched by what the autotuner found."""
    a, b = poiseuille(64, 64), poiseuille(64, 64)
    for s in (a, b):
        jittered(s, 4)
    a.autotune(3)
    for s in (a, b):
        s.set_verlet(0.5)
        s.update_n(4)
    same(a, b)
    for s in (a, b):
        s.set_graphs(False)
        s.update_n(2)
    same(a, b)
    assert a.neighbor_lists() == b.neighbor_lists()
    a.close()
    b.close()
