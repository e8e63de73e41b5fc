"""The per-cell ordering at crowded cells (above 64 particles a cell is read in wide
loads from its first aligned word): whole cells of every size around the limit, starting
at every alignment, keep their particles by original index."""
import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import _abi, presets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lead", [0, 1, 2, 3])
def test_crowded_cells_keep_the_original_order(gpu, lead):
    p = presets.dambreak_params((128, 256, 1), 1, (512, 256, 4), 1.0 / 256)
    s = cm.DamBreakSystem(params=p)
    s.reset()
    pos = s.getArray(cm.POSITION)
    n = len(pos)
    dx = 2 * float(p.particle_radius)
    rng = np.random.default_rng(lead)
    # piles of these sizes, one cell each, in cells between the lattice and the far wall
    free = list(rng.permutation(np.flatnonzero(pos[:, 3] == _abi.FLUID)))
    sizes = [lead] + [1, 5, 63, 64, 65, 66, 67, 68, 79, 80, 81, 96, 97, 1023]
    for k, size in enumerate(sizes):
        for _ in range(size):
            pos[free.pop(), :2] = ((300 + 3 * k + 0.5) * dx + float(p.world_origin[0]),
                                   (20.5) * dx + float(p.world_origin[1]))
    s.setArray(cm.POSITION, pos)
    s.run_stages(_abi.STAGE_DENSITY)
    key, idx = s.getUintArray(_abi.HASH)[:n], s.getUintArray(_abi.INDEX)[:n]
    assert np.array_equal(np.sort(idx), np.arange(n))
    assert (np.diff(key.astype(np.int64)) >= 0).all()
    same = key[1:] == key[:-1]
    assert (idx[1:][same] > idx[:-1][same]).all()
    count = np.unique(key, return_counts=True)[1]
    assert set(sizes[1:]) <= set(count.tolist())
    s.close()
