"""bhSurrogateGenerate when the host has no memory for the views' parameters: an error, not an exception out of a
C function, and the set from before stays.  In a child process with a limit on its address space."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, resource, sys
sys.path[:0] = [%r, %r, %r]
import numpy as np
from test_gpu_surrogate import Net
rays = 1 << 22
net = Net(3)
assert net.L.bhSurrogateGenerate(net.h, C.c_longlong(rays), 64, C.c_uint(5)) == 0
row = np.zeros((2, 8), np.float32)
def first():
    assert net.L.bhSurrogateDatasetCopy(net.h, row[0].ctypes.data_as(C.c_void_p), row[1].ctypes.data_as(C.c_void_p),
                                        C.c_longlong(0), C.c_longlong(1)) == 0
    return row.copy()
before = first()
size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (size + (64 << 20), resource.RLIM_INFINITY))
code = net.L.bhSurrogateGenerate(net.h, C.c_longlong(rays), rays, C.c_uint(6))   # some 350 MB of views
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
n = C.c_longlong()
assert net.L.bhSurrogateDataset(net.h, None, None, C.byref(n)) == 0
assert code == 2 and n.value == rays, (code, n.value)    # cudaErrorMemoryAllocation
assert np.array_equal(first(), before)
assert net.L.bhSurrogateGenerate(net.h, C.c_longlong(rays), 64, C.c_uint(5)) == 0
assert np.array_equal(first(), before)
print("done")
"""


def test_out_of_host_memory_is_an_error(cuda):
    p = subprocess.run([sys.executable, "-c", CHILD % (ROOT + "/black-hole_b200", ROOT + "/oracle", ROOT + "/tests")],
                       capture_output=True, text=True, timeout=300, cwd=ROOT + "/tests")
    assert p.returncode == 0 and "done" in p.stdout, (p.returncode, p.stdout[-500:], p.stderr[-1500:])
