"""mfgb_operator_create where the host has no memory for its marks of constrained
DoFs (one bit each): a status comes back through the C ABI, no exception."""
import os
import subprocess
import sys

CALL = """
import ctypes, resource
L = ctypes.CDLL({lib!r})
with open("/proc/self/statm") as f:
    used = int(f.read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (200 << 20), resource.RLIM_INFINITY))
n = 2 ** 32 - 2  # the largest operator: 512 MB of marks
dof_map = (ctypes.c_uint32 * 8)(*range(8))
G = (ctypes.c_double * 48)()
constrained = (ctypes.c_int64 * 1)(n - 1)
op = ctypes.c_void_p()
st = L.mfgb_operator_create(1, ctypes.c_int64(n), ctypes.c_int64(1), dof_map, G, ctypes.c_int64(1),
                            constrained, ctypes.byref(op))
print("status", st)
"""


def test_no_exception_leaves_the_c_abi():
    from benchmarks_gb300 import build
    if not os.path.exists(build.LIB):
        build.build()
    r = subprocess.run([sys.executable, "-c", CALL.format(lib=build.LIB)], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)
    assert r.stdout.startswith("status ")
