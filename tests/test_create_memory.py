"""A dam-break system made where device memory is short: the kept wall densities need no
room for the scratch of the interpolation, which is then asked for on first use.  On the
host, with a fake of the CUDA runtime that has a given amount of memory."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = r"""
import ctypes
from cmag_gb300 import _abi, presets
from cmag_gb300._lib import lib
fake, L = ctypes.CDLL(None), lib()
fake.fake_used.restype = ctypes.c_longlong
fake.fake_memory.argtypes = [ctypes.c_longlong]
p = presets.dambreak_params((16, 32, 1), 1, (64, 64, 4), 1 / 256)
n = 5000

def create():
    h, on = ctypes.c_void_p(), ctypes.c_int32(-1)
    assert L.cmag_system_create(ctypes.byref(p), n, ctypes.byref(h)) == 0, L.cmag_last_error()
    assert L.cmag_system_get_wall_cache(h, ctypes.byref(on)) == 0
    return h, on.value

def interpolate(h):  # the stage check passes: a new system counts as stepped
    pts, out = (ctypes.c_float * 4)(), (ctypes.c_float * 4)()
    return L.cmag_system_interpolate(h, _abi.VELOCITY, pts, 1, out)

h, on = create()
whole = fake.fake_used()
assert on == 1 and interpolate(h) == 0 and fake.fake_used() == whole
assert L.cmag_system_destroy(h) == 0 and fake.fake_used() == 0
for short, kept in ((1, 1), (16 * n, 1), (16 * n + 1, 0)):
    fake.fake_memory(whole - short)
    h, on = create()
    assert on == kept, (short, on)
    assert fake.fake_pending() == 0
    used = fake.fake_used()
    if kept:
        assert used == whole - 16 * n
        fake.fake_memory(used)  # no room for the scratch: reported, and had later
        assert interpolate(h) == _abi.CMAG_ERR_NOMEM
        fake.fake_memory(-1)
        assert interpolate(h) == 0 and fake.fake_used() == whole
    assert L.cmag_system_destroy(h) == 0 and fake.fake_used() == 0
"""


def test_wall_densities_are_kept_without_the_scratch(built, tmp_path):
    fake = str(tmp_path / "libfake_cudart.so")
    subprocess.run(["gcc", "-std=gnu17", "-O1", "-shared", "-fPIC", os.path.join(HERE, "fake_cudart", "fake_cudart.c"),
                    "-o", fake], check=True)
    run = subprocess.run([sys.executable, "-c", CHILD], cwd=os.path.dirname(HERE),
                         env=dict(os.environ, LD_PRELOAD=fake), capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr[-2000:]
