"""A mode-0 term launch that fails adds nothing to bigSum: no entry counts as a sum then."""
import os
import subprocess
import sys

from conftest import ROOT

SCRIPT = r"""
import ctypes
import clbellard_gb300 as C
lib = C.load()
fn = getattr(lib, "_ZN3cbl15launch_dd_termsEiP5uint2iPimmmijjmiP11CUstream_st")
u64, u32, c_int, vp = ctypes.c_uint64, ctypes.c_uint32, ctypes.c_int, ctypes.c_void_p
fn.argtypes = [c_int, vp, c_int, ctypes.POINTER(c_int), u64, u64, u64, c_int, u32, u32, u64, c_int, vp]
fn.restype = c_int
used = c_int(3)
rc = fn(0, None, 1368, ctypes.byref(used), 0, 100000, 200001, 1, 4, 1, 200001, 0, None)
print("rc", rc, "used", used.value)
"""


def test_failed_term_launch_leaves_the_entries_as_they_were():
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")          # no device: the launch fails in the runtime
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rc, used = int(r.stdout.split()[1]), int(r.stdout.split()[3])
    assert rc != 0 and used == 3
