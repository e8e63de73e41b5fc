"""The radix sort at the edges of its tiling (1,024 threads, 1 to 8 pairs each, a tile for
each of 152 SMs, look-back groups of 16 tiles) and of its odd and even numbers of passes:
both entry points against a stable host sort, exactly, one size after another on the
same cached workspace."""
import ctypes

import numpy as np
import pytest

from cmag_gb300._lib import c_u32p, check, lib

pytestmark = pytest.mark.gpu

TILE, SMS = 1024, 152


@pytest.mark.parametrize("bits", [8, 23, 32])
def test_sort_sizes(gpu, bits):
    import torch
    rng = np.random.default_rng(bits)
    sizes = [1, TILE - 1, TILE, TILE + 1, 16 * TILE, 16 * TILE + 1, SMS * TILE, SMS * TILE + 1, 2 * SMS * TILE + 7,
             8 * SMS * TILE, 8 * SMS * TILE + 1, 33 * 16 * 8 * TILE - 5, 5000]
    for n in sizes:
        keys = rng.integers(0, 1 << bits, size=n, dtype=np.uint64).astype(np.uint32)
        if n > 3:
            keys[: n // 3] = keys[0]  # a crowded digit
        vals = rng.permutation(n).astype(np.uint32)
        order = np.argsort(keys, kind="stable")
        for entry in ("cmag_sort_particles", "cmag_sort_particles_noalloc"):
            if entry.endswith("noalloc") and n > 1 << 20:
                continue
            k = torch.from_numpy(keys.view(np.int32).copy()).cuda()
            v = torch.from_numpy(vals.view(np.int32).copy()).cuda()
            check(getattr(lib(), entry)(ctypes.cast(k.data_ptr(), c_u32p), ctypes.cast(v.data_ptr(), c_u32p), n, bits,
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
            assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[order]), (entry, n)
            assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[order]), (entry, n)
