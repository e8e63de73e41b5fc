"""A step on a caller's stream that is being captured is refused, for small scenes (three
launches) as for large ones (a graph of its own): it would be recorded, not run, while
the host's clock moves on.  After the capture the solver goes on where it was."""
import ctypes

import numpy as np
import pytest

import cmag_gb300 as cm
from cmag_gb300 import presets
from cmag_gb300._lib import LIB_PATH

pytestmark = pytest.mark.gpu


def scene(fluid):
    p = presets.poiseuille_params((fluid, fluid, 1), 3, (fluid, fluid + 12, 4), 1.0 / (2 * fluid * 1000))
    s = cm.PoiseuilleFlowSystem(params=p)
    s.reset()
    return s


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("fluid", [16, 160])
def test_update_under_capture_is_refused(gpu, fluid, warm):
    rt = ctypes.CDLL(LIB_PATH)  # resolves the CUDA runtime the library links
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    a, b = scene(fluid), scene(fluid)
    a.set_stream(stream.value)
    if warm:
        a.update()
        b.update()
    a.synchronize()
    elapsed = a.getElapsedTime()
    assert rt.cudaStreamBeginCapture(stream, 1) == 0  # thread-local
    for step in (a.update, lambda: a.update_n(3)):
        with pytest.raises(cm.CmagError):
            step()
    rt.cudaStreamEndCapture(stream, ctypes.byref(graph))  # (an invalidated capture ends with an error code)
    rt.cudaGetLastError()
    assert a.getElapsedTime() == elapsed
    a.update_n(4)
    b.update_n(4)
    for array in (cm.POSITION, cm.VELOCITY, cm.MEASURES):
        assert np.array_equal(a.getArray(array).view(np.uint32), b.getArray(array).view(np.uint32))
    assert a.getElapsedTime() == b.getElapsedTime()
    a.close()
    b.close()
    assert rt.cudaStreamDestroy(stream) == 0
