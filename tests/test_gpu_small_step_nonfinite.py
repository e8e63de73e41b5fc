"""The three-launch step with particles whose position is not finite: every array is the
staged step's, NaN where that has NaN (0 * NaN of an out-of-reach candidate included),
whichever way candidates pair up.  Particles at NaN share cell 0, so each step brings
further ones there: rows of one, then of many."""
import numpy as np
import pytest

import cmag_gb300 as cm
from test_gpu_small_step import SCENES, jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("lists", [0, 1])
@pytest.mark.parametrize("name", ["dambreak 64", "dambreak 64 cut", "dambreak 64 crowded", "dambreak 76",
                                  "poiseuille 37x28", "poiseuille 171x97", "poiseuille spline 64x64",
                                  "peristalsis 128x24", "peristalsis 256x58"])
def test_nonfinite_positions_equal_staged_steps(gpu, name, lists, value):
    a, b = SCENES[name](), SCENES[name]()
    b.set_graphs(False)
    for s in (a, b):
        jittered(s, 5)
        if lists:
            s.set_neighbor_lists(True)
        pos = s.getArray(cm.POSITION)
        rng = np.random.default_rng(2)
        for i, axes in zip(rng.choice(len(pos), 6, replace=False), ((0,), (1,), (0, 1)) * 2):
            pos[i, list(axes)] = value
        s.setArray(cm.POSITION, pos)
    for _ in range(3):
        a.update()
        b.update()
        x, y = a.state(), b.state()
        for k in x:
            assert np.array_equal(x[k], y[k], equal_nan=x[k].dtype == np.float32), (name, k)
    a.close()
    b.close()
