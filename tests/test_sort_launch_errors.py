"""The sort reports a launch that the CUDA runtime rejects, and a kernel attribute that it
does not grant, instead of returning unsorted pairs as sorted.  On the host: the failing
calls come from a fake of the runtime that is loaded before the real one."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = r"""
import ctypes, sys
fake, lib = ctypes.CDLL(None), ctypes.CDLL(sys.argv[1])
lib.cmag_last_error.restype = lib.cmag_sort_particles_noalloc_error.restype = ctypes.c_char_p
keys, vals = (ctypes.c_uint32 * 5000)(), (ctypes.c_uint32 * 5000)()
for entry, message in ((lib.cmag_sort_particles, lib.cmag_last_error),
                       (lib.cmag_sort_particles_noalloc, lib.cmag_sort_particles_noalloc_error)):
    for bits in (8, 12, 30):
        passes = (bits + 7) // 8
        call = lambda: entry(keys, vals, 5000, bits, None)
        fake.fake_fail(-1, 0, 0)
        assert call() == 0, message()
        for k in range(passes + 1):  # the histogram's launch, then each pass's
            fake.fake_fail(k, 0, 0)
            assert call() == 2, (entry, bits, k)  # CMAG_ERR_CUDA
            assert b"resources" in message(), message()
            if entry is lib.cmag_sort_particles:
                assert fake.fake_pending() == 0  # its own error is cleared
                assert fake.fake_waits() == 1  # and its workspace idle
        fake.fake_fail(-1, 1, 0)
        assert call() == 2, (entry, bits)
# an error that the caller's earlier work left is not the sort's
fake.fake_fail(-1, 0, 1)
assert lib.cmag_sort_particles(keys, vals, 5000, 12, None) == 0
assert fake.fake_pending() == 1
"""


def test_rejected_launches_are_reported(built, tmp_path):
    from cmag_gb300._lib import LIB_PATH
    fake = str(tmp_path / "libfake_cudart.so")
    subprocess.run(["gcc", "-std=gnu17", "-O1", "-shared", "-fPIC", os.path.join(HERE, "fake_cudart", "fake_cudart.c"),
                    "-o", fake], check=True)
    run = subprocess.run([sys.executable, "-c", CHILD, LIB_PATH], env=dict(os.environ, LD_PRELOAD=fake),
                         capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr[-2000:]
